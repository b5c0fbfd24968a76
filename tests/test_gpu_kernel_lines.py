"""The device kernels at the lines where their work is split differently: row widths of the SELL
and lane-group visits, tile counts of the reductions, row lengths of the setup's products and
sorts. Each against the oracle or the host build; whole numbers and fixed-order sums bit for bit,
reordered FP64 sums within their round-off bound."""
import numpy as np
import pytest

import oracle as O
from cfd_b200 import workloads as W

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _banded(n, half, seed=3):
    """Symmetric, diagonally dominant matrix with 2 half + 1 entries in the rows away from the ends."""
    i = np.arange(n)
    pairs = np.concatenate([np.stack([i[:n - k], i[k:]], 1) for k in range(1, half + 1)])
    pairs = pairs[np.lexsort((pairs[:, 1], pairs[:, 0]))]
    own, nei = pairs[:, 0].astype(np.int32), pairs[:, 1].astype(np.int32)
    rng = np.random.default_rng(seed)
    w = rng.uniform(0.5, 1.5, len(own))
    diag = np.bincount(own, w, n) + np.bincount(nei, w, n) + 0.05
    return own, nei, -w, -w.copy(), diag, rng.standard_normal(n)


def _pressure(case):
    up, lo, dg, dv = O.assemble(case.n, case.owner, case.neighbour, case.flux, case.gamma,
                                case.delta, 0.0)
    diag, src = case.finalize(up, lo, dg, dv)
    return up, lo, diag, src


def _csr(n, own, nei, diag, up, lo):
    return O.ldu_to_csr(O.build_pattern(n, own, nei), diag, up, lo)


@pytest.mark.parametrize("n", [33, 255, 257, 20001])
@pytest.mark.parametrize("half", [1, 2, 3, 4, 7, 24])
def test_row_widths_of_the_operator_kernels(gpu, n, half):
    """One FP64 V-cycle on rows of 3 to 49 entries, tiles with a last partial warp or one row more
    than a block. In the oracle's order (SELL throughout, one row at a time and the next row loaded
    ahead) bit for bit; by default and with lane groups throughout (wide_row) the row sums differ
    in order: a few hundred additions deep over all levels, each within EPS of its magnitude."""
    cb = gpu
    own, nei, up, lo, diag, src = _banded(n, half)
    ds = cb.DeviceSolver(cb.build_csr_pattern(n, own, nei))
    settings = cb.AmgSettings(strength_threshold=0.04, coarse_size=16)
    a = _csr(n, own, nei, diag, up, lo)
    h = O.Hierarchy(a, theta=0.04, coarse_size=16)
    ds.setup_amg(diag, up, lo, settings)
    r = np.random.default_rng(8).standard_normal(n)
    zr = O.vcycle_apply(h.a, h.p, h.r, h.coarse_inverse, r, 2, 0.7)
    x = np.zeros(n)
    ds.set_ordered(True)
    for pair in (0, 1):
        ds.set_tuning(cb.Tuning(vcycle_pair=pair))
        ds.solve(diag, up, lo, src, x, cb.Method.Cg, True, cb.SolveControl(1e300, 1))
        assert np.array_equal(ds.apply_amg(r), zr)
    ds.set_ordered(False)
    for t in (cb.Tuning(), cb.Tuning(wide_row=2), cb.Tuning(wide_row=2, lanes_div=4)):
        ds.set_tuning(t)
        ds.solve(diag, up, lo, src, x, cb.Method.Cg, True, cb.SolveControl(1e300, 1))
        z = ds.apply_amg(r)
        assert np.linalg.norm(z - zr) <= 1e3 * EPS * np.linalg.norm(zr)
    ds.close()


@pytest.mark.parametrize("half", [2, 3, 4, 9])
def test_norms_of_the_ldu_solve_by_row_width(gpu, half):
    """Residual and reference norms summed on the SELL operator: rows of 5, 7, 9 and 19 entries. All
    terms are positive, so the two orders of the sums differ by less than n EPS of the result."""
    cb = gpu
    n = 3001
    own, nei, up, lo, diag, src = _banded(n, half)
    ds = cb.DeviceSolver(cb.build_csr_pattern(n, own, nei))
    x = np.random.default_rng(4).standard_normal(n)
    want = O.normalised_residual(own, nei, diag, up, lo, src, x)
    r = ds.solve_ldu(diag, up, lo, src, x, cb.LduSettings(tolerance=1e-12, rel_tolerance=1e-6),
                     cb.AmgSettings(strength_threshold=0.04))
    assert abs(r.initial_residual - want) <= n * EPS * want
    ds.close()


@pytest.mark.parametrize("tiles", [1, 31, 32, 33, 444, 1184, 0])
def test_reductions_over_any_number_of_tiles(gpu, tiles):
    """Level-0 sums over one tile, the 32 that one warp adds in order, whole waves, and more than one
    group (0: 2050 tiles of 256 rows, the last of one row): CG and BiCGStab to 1e-10 and the
    norms of solve_ldu. The sums differ in order only: iterations within 1 (2), residuals at the
    target."""
    cb = gpu
    n = 2049 * 256 + 1
    own, nei, up, lo, diag, src = _banded(n, 1)
    diag = diag + 1.0
    ds = cb.DeviceSolver(cb.build_csr_pattern(n, own, nei))
    ds.set_tuning(cb.Tuning(target_tiles=tiles))
    a = _csr(n, own, nei, diag, up, lo)
    tol = 1e-10 * np.linalg.norm(src)
    xo, so = O.krylov(a, src, method=0, abs_tol=tol, max_iterations=500)
    x = np.zeros(n)
    st = ds.solve(diag, up, lo, src, x, cb.Method.Cg, False, cb.SolveControl(tol, 500))
    assert st.converged and abs(st.iterations - so["iterations"]) <= 1
    assert np.linalg.norm(src - a.matvec(x)) <= 1.05 * tol
    xb = np.zeros(n)
    xo, so = O.krylov(a, src, method=1, abs_tol=tol, max_iterations=500)
    st = ds.solve(diag, up, lo, src, xb, cb.Method.BiCgStab, False, cb.SolveControl(tol, 500))
    assert st.converged and abs(st.iterations - so["iterations"]) <= 2
    assert np.linalg.norm(src - a.matvec(xb)) <= 1.05 * tol
    want = O.normalised_residual(own, nei, diag, up, lo, src, x)
    r = ds.solve_ldu(diag, up, lo, src, x, cb.LduSettings(tolerance=1.0))
    # x is nearly the solution: the residual itself carries the cancellation of b - A x
    assert r.iterations == 0 and abs(r.initial_residual - want) <= 1e-4 * want
    ds.close()


@pytest.mark.parametrize("max_it", [1, 2, 3])
def test_bicgstab_limit_and_half_step(gpu, max_it):
    """The iteration limit is reported as the oracle reports it; a diagonal matrix is solved by the
    first half step."""
    cb = gpu
    case = W.cavity(8)
    up, lo, diag, src = _pressure(case)
    a = _csr(case.n, case.owner, case.neighbour, diag, up, lo)
    ds = cb.DeviceSolver(cb.build_csr_pattern(case.n, case.owner, case.neighbour))
    tol = 1e-10 * np.linalg.norm(src)
    xo, so = O.krylov(a, src, method=1, abs_tol=tol, max_iterations=max_it)
    x = np.zeros(case.n)
    st = ds.solve(diag, up, lo, src, x, cb.Method.BiCgStab, False, cb.SolveControl(tol, max_it))
    assert not st.converged and st.iterations == so["iterations"] == max_it
    # three iterations from the same start: sums of 512 terms in another order, not yet amplified
    assert np.linalg.norm(x - xo) <= 1e-9 * np.linalg.norm(xo)
    z = np.zeros_like(up)
    d = 4.0 * np.ones(case.n)
    xd = np.zeros(case.n)
    st = ds.solve(d, z, z, src, xd, cb.Method.BiCgStab, False, cb.SolveControl(tol, max_it))
    assert st.converged and st.iterations == 1
    assert np.linalg.norm(src - d * xd) <= tol
    ds.close()


@pytest.mark.parametrize("tol", [1e-6, 1e-12, 1e-18])
def test_mixed_precision_reports_the_checked_residual(gpu, tol):
    """Mixed precision: a system at its target is checked in FP64 and goes on if the check fails.
    `converged` and `true_residual` are those of the returned x, also where the target is out of
    reach."""
    cb = gpu
    case = W.tet(8)
    up, lo, diag, src = _pressure(case)
    a = _csr(case.n, case.owner, case.neighbour, diag, up, lo)
    ds = cb.DeviceSolver(cb.build_csr_pattern(case.n, case.owner, case.neighbour))
    ds.set_precision(cb.Precision.MIXED)
    ds.setup_amg(diag, up, lo, cb.AmgSettings(strength_threshold=0.04, coarse_size=50))
    t = tol * np.linalg.norm(src)
    x = np.zeros(case.n)
    st = ds.solve(diag, up, lo, src, x, cb.Method.Cg, True, cb.SolveControl(t, 60))
    got = np.linalg.norm(src - a.matvec(x))
    mag = np.linalg.norm(np.abs(src) + _abs_matvec(a, x))
    assert abs(got - st.true_residual) <= 64 * EPS * mag
    assert st.iterations <= 60
    if st.converged:
        assert st.true_residual <= t
    assert st.converged or tol < 1e-15
    ds.close()


def _abs_matvec(a, x):
    return np.add.reduceat(np.abs(a.va) * np.abs(x)[a.ci], a.rp[:-1])


@pytest.mark.parametrize("n", [4095, 4097, 9000, 70000])
@pytest.mark.parametrize("half", [3, 4, 7, 8, 9, 10, 15, 16])
def test_setup_at_the_row_lengths_of_its_kernels(gpu, n, half):
    """Rows of 2 half + 1 entries: products of 7 to 33 contributions (8, 16 and 32 lanes, then
    tables), sorts of up to 32 entries and more, aggregation on the device (70000 rows, up to 20 strong
    entries a row) and on the host. Every level equals the host build bit for bit."""
    cb = gpu
    own, nei, up, lo, diag, _ = _banded(n, half, seed=half)
    a = _csr(n, own, nei, diag, up, lo)
    view = cb.CsrView(a.n_rows, a.rp, a.ci, a.va)
    for theta in (0.0, 0.02):
        s = cb.AmgSettings(strength_threshold=theta)
        d, h = cb.AmgHierarchy(view, s, device=True), cb.AmgHierarchy(view, s)
        assert d.levels() == h.levels()
        for l in range(h.levels()):
            pairs = [(d.level_matrix(l), h.level_matrix(l))]
            if l + 1 < h.levels():
                assert np.array_equal(d.aggregates(l)[0], h.aggregates(l)[0])
                pairs += [(d.level_prolongation(l), h.level_prolongation(l)),
                          (d.level_restriction(l), h.level_restriction(l))]
            for g, w in pairs:
                assert np.array_equal(g.row_ptr, w.row_ptr) and np.array_equal(g.col, w.col)
                assert np.array_equal(g.val, w.val)
        assert np.array_equal(d.coarse_inverse(), h.coarse_inverse())


@pytest.mark.parametrize("n,nc", [(6, 2), (96, 32), (1248, 416), (1251, 417), (1500, 500)])
def test_dense_coarse_solve_by_size(gpu, n, nc):
    """Two levels: the dense inverse's rows up to 13 x 32 entries are loaded ahead, the rest behind
    them. Bit for bit in the oracle's order, else sums of nc terms in another order."""
    cb = gpu
    own, nei, up, lo, diag, src = _banded(n, 1)
    a = _csr(n, own, nei, diag, up, lo)
    h = O.Hierarchy(a, theta=0.04, max_levels=2, coarse_size=3)
    assert h.levels == 2 and h.a[1].n_rows == nc
    ds = cb.DeviceSolver(cb.build_csr_pattern(n, own, nei))
    ds.setup_amg(diag, up, lo, cb.AmgSettings(strength_threshold=0.04, max_levels=2, coarse_size=3))
    r = np.random.default_rng(8).standard_normal(n)
    zr = O.vcycle_apply(h.a, h.p, h.r, h.coarse_inverse, r, 2, 0.7)
    for ordered in (True, False):
        ds.set_ordered(ordered)
        x = np.zeros(n)
        ds.solve(diag, up, lo, src, x, cb.Method.Cg, True, cb.SolveControl(1e300, 1))
        z = ds.apply_amg(r)
        assert np.linalg.norm(z - zr) <= (0.0 if ordered else nc * EPS * np.linalg.norm(zr))
    ds.close()


@pytest.mark.parametrize("n_sys", [1, 167, 168, 300])
def test_batches_around_the_state_block(gpu, n_sys):
    """The states of up to 167 systems (96 bytes each) travel in the engine's page-locked block, more
    in a buffer of their own: every system of a batch reaches its own target."""
    import torch
    cb = gpu
    n = 24
    own, nei, up, lo, diag, _ = _banded(n, 2)
    a = _csr(n, own, nei, diag, up, lo)
    rng = np.random.default_rng(n_sys)
    b = cb.Batch([n] * n_sys, [len(own)] * n_sys, np.tile(own, n_sys), np.tile(nei, n_sys))
    rep = lambda v: np.tile(v, n_sys)  # noqa: E731
    src = rng.standard_normal(n * n_sys)
    b.setup_amg(rep(diag), rep(up), rep(lo))
    T = lambda v: torch.as_tensor(v, dtype=torch.float64, device="cuda")  # noqa: E731
    x = torch.zeros(n * n_sys, dtype=torch.float64, device="cuda")
    tol = [10.0 ** -(4 + k % 7) * np.linalg.norm(src[k * n:(k + 1) * n]) for k in range(n_sys)]
    for _ in range(2):
        x.zero_()
        stats = b.solve_device(T(rep(diag)), T(rep(up)), T(rep(lo)), T(src), x, [cb.SolveControl(t, 100) for t in tol])
        got = x.cpu().numpy()
        for k in range(n_sys):
            r = np.linalg.norm(src[k * n:(k + 1) * n] - a.matvec(got[k * n:(k + 1) * n]))
            assert stats[k].converged and r <= 1.05 * tol[k]


def _scattered(n, per_row, seed):
    """Symmetric, diagonally dominant CSR matrix of a sparse graph (two rows seldom share more than one
    column) whose off-diagonal entries are each held twice with probability 1/2, the second copies at
    the row's end."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), per_row)
    j = i + rng.integers(1, 400, len(i))
    i, j = i[j < n], j[j < n]
    pairs = np.unique(np.stack([i, j], 1), axis=0)
    w = rng.uniform(0.5, 1.5, len(pairs))
    rows = np.concatenate([pairs[:, 0], pairs[:, 1]])
    cols = np.concatenate([pairs[:, 1], pairs[:, 0]])
    vals = -np.concatenate([w, w])
    diag = np.bincount(rows, -vals, n) + 0.05
    rows, cols, vals = (np.concatenate([v, d]) for v, d in
                        ((rows, np.arange(n)), (cols, np.arange(n)), (vals, diag)))
    o = np.lexsort((cols, rows))
    rows, cols, vals = rows[o], cols[o], vals[o]
    twice = (rows != cols) & (rng.random(len(rows)) < 0.5)
    r2 = np.concatenate([rows, rows[twice]])
    c2 = np.concatenate([cols, cols[twice]])
    v2 = np.concatenate([vals * np.where(twice, 0.625, 1.0), vals[twice] * 0.375])
    o = np.argsort(r2, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(r2, minlength=n))])
    return rp.astype(np.int32), c2[o].astype(np.int32), v2[o]


def _same_hierarchies(d, h):
    assert d.levels() == h.levels()
    for l in range(h.levels()):
        pairs = [(d.level_matrix(l), h.level_matrix(l))]
        if l + 1 < h.levels():
            assert np.array_equal(d.aggregates(l)[0], h.aggregates(l)[0])
            pairs += [(d.level_prolongation(l), h.level_prolongation(l)),
                      (d.level_restriction(l), h.level_restriction(l))]
        for g, w in pairs:
            assert np.array_equal(g.row_ptr, w.row_ptr) and np.array_equal(g.col, w.col)
            assert np.array_equal(g.val, w.val)
    assert np.array_equal(d.coarse_inverse(), h.coarse_inverse())


@pytest.mark.parametrize("n,per_row", [(66000, 1), (70000, 1), (33000, 2), (36000, 2), (16000, 4), (20000, 4),
                                       (11000, 6), (14000, 6), (9000, 12)])
def test_setup_with_repeated_columns(gpu, n, per_row):
    """A CSR matrix whose rows (of about 4 to 40 entries) hold some columns twice, of 190K to 250K strong
    entries and so on either side of the device aggregation's line: the device setup treats the copies as
    separate entries, as the host build does, and equals it bit for bit, every time."""
    cb = gpu
    view = cb.CsrView(n, *_scattered(n, per_row, seed=per_row))
    s = cb.AmgSettings(strength_threshold=0.0)
    h = cb.AmgHierarchy(view, s)
    for _ in range(2):
        _same_hierarchies(cb.AmgHierarchy(view, s, device=True), h)


@pytest.mark.parametrize("tiles", [1, 32, 33, 444, 0])
def test_each_norm_of_the_ldu_solve_over_any_number_of_tiles(gpu, tiles):
    """The three norms over one tile to more than one group (0: 2050 tiles, the second group of two),
    from a random x. Residual and reference norm are sums of positive terms (n EPS between two
    orders); the squared norm sets the target of the solve, which then takes the oracle's iterations
    (within 2, the order of BiCGStab's sums) and ends at the target. Every repetition is the same."""
    cb = gpu
    n = 2049 * 256 + 1
    own, nei, up, lo, diag, src = _banded(n, 1)
    diag = diag + 1.0
    ds = cb.DeviceSolver(cb.build_csr_pattern(n, own, nei))
    ds.set_tuning(cb.Tuning(target_tiles=tiles))
    a = _csr(n, own, nei, diag, up, lo)
    x0 = np.random.default_rng(6).standard_normal(n)
    want = O.normalised_residual(own, nei, diag, up, lo, src, x0)
    r0 = np.linalg.norm(src - a.matvec(x0))
    rel = 1e-7
    xo, so = O.krylov(a, src, x0, method=1, abs_tol=rel * r0, max_iterations=500)
    s = cb.LduSettings(method=cb.Method.BiCgStab, tolerance=1e-14, rel_tolerance=rel)
    first = None
    for _ in range(4):
        x = x0.copy()
        r = ds.solve_ldu(diag, up, lo, src, x, s)
        assert abs(r.initial_residual - want) <= n * EPS * want
        assert abs(r.iterations - so["iterations"]) <= 2
        assert np.linalg.norm(src - a.matvec(x)) <= 1.05 * rel * r0
        if first is None:
            first = (r.initial_residual, r.final_residual, r.iterations, x)
        assert (r.initial_residual, r.final_residual, r.iterations) == first[:3] and np.array_equal(x, first[3])
    ds.close()


@pytest.mark.parametrize("limit", [2 ** 31 - 2, 2 ** 31 - 1])
def test_largest_iteration_limits(gpu, limit):
    """A limit at the end of the int range is no limit: every method takes the iterations it takes
    under a limit of 1000."""
    cb = gpu
    case = W.cavity(8)
    up, lo, diag, src = _pressure(case)
    tol = 1e-8 * np.linalg.norm(src)
    ds = cb.DeviceSolver(cb.build_csr_pattern(case.n, case.owner, case.neighbour))
    for method, amg, precision in ((cb.Method.BiCgStab, False, cb.Precision.FP64),
                                   (cb.Method.Cg, False, cb.Precision.FP64),
                                   (cb.Method.Cg, True, cb.Precision.FP64),
                                   (cb.Method.Cg, True, cb.Precision.MIXED)):
        ds.set_precision(precision)
        if amg:
            ds.setup_amg(diag, up, lo, cb.AmgSettings(strength_threshold=0.04, coarse_size=50))
        got = []
        for m in (1000, limit):
            x = np.zeros(case.n)
            st = ds.solve(diag, up, lo, src, x, method, amg, cb.SolveControl(tol, m))
            assert st.converged
            got.append((st.iterations, x))
        assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
    ds.close()


def _with_hub(n, half, degree, seed=9):
    """_banded with row n // 2 connected to `degree` further rows."""
    own, nei, up, lo, diag, _ = _banded(n, half, seed)
    hub = n // 2
    far = np.setdiff1d(np.arange(n), np.arange(hub - half, hub + half + 1))
    far = np.sort(np.random.default_rng(seed).permutation(far)[:degree])
    w = np.random.default_rng(seed + 1).uniform(0.5, 1.5, degree)
    diag = diag.copy()
    np.add.at(diag, far, w)
    diag[hub] += w.sum()
    own = np.concatenate([own, np.minimum(far, hub).astype(np.int32)])
    nei = np.concatenate([nei, np.maximum(far, hub).astype(np.int32)])
    o = np.lexsort((nei, own))
    v = np.concatenate([up, -w])[o]
    return _csr(n, own[o], nei[o], diag, v, v.copy())


@pytest.mark.parametrize("n,degree", [(40000, 300), (40000, 2800), (40000, 3600), (40000, 39000), (150000, 149000)])
def test_setup_with_a_hub_row(gpu, n, degree):
    """One row strongly connected to many: its rows conflict pairwise (degree^2 / 2), which the device
    aggregates up to 24 conflicts a strong entry (degrees to about 3200 of 40000 rows) and the host beyond.
    Equal to the host build, within memory in proportion to the matrix."""
    import torch
    cb = gpu
    a = _with_hub(n, 3, degree)
    view = cb.CsrView(a.n_rows, a.rp, a.ci, a.va)
    s = cb.AmgSettings(strength_threshold=0.0)
    h = cb.AmgHierarchy(view, s)
    free = torch.cuda.mem_get_info()[0]
    _same_hierarchies(cb.AmgHierarchy(view, s, device=True), h)
    assert free - torch.cuda.mem_get_info()[0] <= (256 << 20) + 1000 * a.va.nbytes


def _cg(cb, ds, diag, up, lo, src, tiles, method=0, pair=1):
    """Solution of a Jacobi-preconditioned solve; its bits depend on how the sums are cut into tiles."""
    ds.set_tuning(cb.Tuning(target_tiles=tiles, krylov_pair=pair))
    x = np.zeros(len(diag))
    ds.solve(diag, up, lo, src, x, method, False, cb.SolveControl(1e-10 * np.linalg.norm(src), 500))
    return x


def test_target_above_the_default_gives_shorter_tiles(gpu):
    """524545 rows of 3 entries: the default takes one wave of CTAs, 2368 four waves, which is tiles of
    256 rows here, as 0 asks for."""
    cb = gpu
    n = 2049 * 256 + 1
    own, nei, up, lo, diag, src = _banded(n, 1)
    diag = diag + 1.0
    ds = cb.DeviceSolver(cb.build_csr_pattern(n, own, nei))
    x = {t: _cg(cb, ds, diag, up, lo, src, t) for t in (0, 592, 148 * 8, 148 * 16)}
    assert np.array_equal(x[148 * 16], x[0])
    assert np.array_equal(x[148 * 8], x[592]) and not np.array_equal(x[592], x[0])
    ds.close()


@pytest.mark.parametrize("method", [0, 1])
def test_tiles_are_planned_for_the_kernels_that_run(gpu, method):
    """300000 rows of 3 entries, every 16th of 9: its slices are 9 wide, so the kernels for 7 entries a
    row run, with 3 CTAs per SM loading ahead and 6 one row at a time. The default tiles are one wave of
    those (444 and 888); BiCGStab (method 1) takes rows as CG does, with the same bits either way."""
    cb = gpu
    n = 300000
    own, nei, up, lo, diag, src = _banded(n, 1)
    hub = np.arange(8, n - 8, 16)
    far = np.concatenate([np.stack([np.minimum(hub, hub + k), np.maximum(hub, hub + k)], 1) for k in (-7, -5, -3, 2, 4, 6)])
    pairs = np.concatenate([np.stack([own, nei], 1), far])
    w = np.concatenate([-up, np.full(len(far), 0.25)])
    o = np.lexsort((pairs[:, 1], pairs[:, 0]))
    pairs, w = pairs[o].astype(np.int32), w[o]
    own, nei = np.ascontiguousarray(pairs[:, 0]), np.ascontiguousarray(pairs[:, 1])
    diag = np.bincount(own, w, n) + np.bincount(nei, w, n) + 1.0
    up, lo = -w, -w.copy()
    ds = cb.DeviceSolver(cb.build_csr_pattern(n, own, nei))
    a = _csr(n, own, nei, diag, up, lo)
    assert len(a.va) / n < 5.25
    x = {(t, p): _cg(cb, ds, diag, up, lo, src, t, method, p) for t in (148 * 8, 444, 888) for p in (0, 1)}
    assert np.linalg.norm(src - a.matvec(x[444, 1])) <= 1.05e-10 * np.linalg.norm(src)
    assert np.array_equal(x[148 * 8, 1], x[444, 1]) and np.array_equal(x[148 * 8, 0], x[888, 0])
    assert np.array_equal(x[444, 0], x[444, 1]) and not np.array_equal(x[888, 0], x[444, 0])
    ds.close()


def test_mixed_batch_with_a_target_out_of_reach(gpu):
    """Three systems in mixed precision: one whose target lies below the FP64 floor, so that its FP64 check
    fails and it goes on alone, round after round, and two that reach theirs. Those keep the iterations
    and the solution that they have without it (the same plan), and every true residual is that of
    the returned x."""
    import torch
    cb = gpu
    case = W.cavity(12)
    up, lo, diag, src = _pressure(case)
    a = _csr(case.n, case.owner, case.neighbour, diag, up, lo)
    n, k = case.n, 3
    b = cb.Batch([n] * k, [case.n_faces] * k, np.tile(case.owner[:case.n_faces], k), np.tile(case.neighbour, k))
    rep = lambda v: np.tile(v, k)  # noqa: E731
    b.set_precision(cb.Precision.MIXED)
    b.setup_amg(rep(diag), rep(up), rep(lo), cb.AmgSettings(strength_threshold=0.04, coarse_size=50))
    T = lambda v: torch.as_tensor(v, dtype=torch.float64, device="cuda")  # noqa: E731
    rng = np.random.default_rng(2)
    rhs = np.concatenate([src, rng.standard_normal(n), rng.standard_normal(n)])
    norm = [np.linalg.norm(rhs[i * n:(i + 1) * n]) for i in range(k)]
    mag = np.linalg.norm
    out = {}
    for far in (1e-8, 1e-18):
        x = torch.zeros(n * k, dtype=torch.float64, device="cuda")
        rel = [1e-6, far, 1e-10]
        st = b.solve_device(T(rep(diag)), T(rep(up)), T(rep(lo)), T(rhs), x,
                            [cb.SolveControl(r * v, 40) for r, v in zip(rel, norm)])
        got = x.cpu().numpy()
        for i in range(k):
            xi, bi = got[i * n:(i + 1) * n], rhs[i * n:(i + 1) * n]
            res = mag(bi - a.matvec(xi))
            assert abs(res - st[i].true_residual) <= 64 * EPS * mag(np.abs(bi) + _abs_matvec(a, xi))
            assert st[i].converged == (rel[i] > 1e-15) and st[i].iterations <= 40
            if st[i].converged:
                assert st[i].true_residual <= rel[i] * norm[i]
        assert st[1].iterations == 40 or far > 1e-15
        out[far] = (got, [s.iterations for s in st])
    for i in (0, 2):
        assert out[1e-8][1][i] == out[1e-18][1][i]
        assert np.array_equal(out[1e-8][0][i * n:(i + 1) * n], out[1e-18][0][i * n:(i + 1) * n])


@pytest.mark.parametrize("shape", [(150000, 1, 1), (3, 3, 9000), (9000, 3, 3), (300, 300, 1), (40, 40, 40)])
def test_setup_of_long_thin_meshes(gpu, shape):
    """Meshes whose rows decide one after another along their length, for which the device leaves the
    aggregation to the host after some sweeps, and two that settle on the device: equal to the host build."""
    cb = gpu
    m = cb.Mesh.box(*shape)
    ni, n = m.n_internal_faces, m.n_cells
    own, nei = np.ascontiguousarray(m.owner[:ni]), m.neighbour
    w = np.random.default_rng(1).uniform(0.5, 1.5, ni)
    diag = np.bincount(own, w, n) + np.bincount(nei, w, n) + 0.01
    a = _csr(n, own, nei, diag, -w, -w.copy())
    view = cb.CsrView(a.n_rows, a.rp, a.ci, a.va)
    s = cb.AmgSettings(strength_threshold=0.04)
    _same_hierarchies(cb.AmgHierarchy(view, s, device=True), cb.AmgHierarchy(view, s))
