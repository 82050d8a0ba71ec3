"""Edges of the cell-index lookup (scoring, refinement, assignment): rows of
cells holding more g than a warp lists at once, more rows than it lists, indexes
split into slabs, and the starting drlv2 values of the assignment -- against the
oracle.  Counts, labels and drlv2 must be identical; refined UBIs are FP64 sums
in another order: 1e-11 of the UBI's largest element, as for the index's other
refinement tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    from imaged11_b200 import synth
    ps = synth.simulate(60, "Al", gmax=1.3, seed=91, noise_frac=0.10)
    rng = np.random.default_rng(92)
    u = synth.trial_ubis(ps.ubis, 60, 0.5, 0.2, rng)
    u[3] = 0.0                      # singular: plain scan
    u[7] = u[5]                     # a tie
    return ps.gv, u


# cell side, x cells per side, g kept: one row of 24,000 g (longer than the
# marks), few long rows, many rows of few g (three boxes' rows fill the list),
# 65M cells (eight slabs) and a ragged 1,000-g index
@pytest.mark.parametrize("cell,xsub,n", [(10.0, 1, None), (1.0, 1, None), (0.3, 2, 20001),
                                         (0.006, 1, None), (0.0275, 16, None), (0.05, 4, 1000)])
@pytest.mark.parametrize("tol", [0.03, 0.25])
def test_rows_and_slabs(scene, oracle, cell, xsub, n, tol, cuda):
    from imaged11_b200 import batch
    gv, u = scene
    g = gv[:n]
    grid = batch.GvecGrid(g, cell=cell, xsub=xsub)
    assert np.array_equal(
        batch.score_grid(u, grid, [tol, 0.6], method="walk").cpu().numpy(),
        oracle.score_many(u, g, [tol, 0.6]))
    d = np.zeros(len(g)) + 2
    lab = np.zeros(len(g), np.int32) - 1
    rd, rl = d.copy(), lab.copy()
    for i, x in enumerate(u):
        _, rd, rl = oracle.score_and_assign(x, g, tol, rd, rl, i)
    batch.score_and_assign_grid(u, grid, tol, d, lab)
    assert np.array_equal(lab, rl) and np.array_equal(d, rd)
    ur, npk, mean = (t.cpu().numpy() for t in batch.refine_grid(u[4:12].copy(), grid, tol))
    for i in range(8):
        k, m, x = oracle.score_and_refine(u[4 + i], g, tol)
        assert npk[i] == k and abs(mean[i] - m) <= 1e-12 * m
        assert np.abs(ur[i] - x).max() <= 1e-11 * np.abs(x).max()


@pytest.mark.parametrize("two", [True, False])
def test_second_slab_with_many_ubis(scene, oracle, two, cuda):
    """An index past the size from which every UBI gets a second item, 38,000 UBIs:
    with the workspace the size functions give, and with one that holds one item
    each (the least a call takes)."""
    import torch
    from imaged11_b200 import batch, synth
    from imaged11_b200._lib import lib
    g = scene[0]
    grid = batch.GvecGrid(g, cell=0.0115, xsub=4)
    assert 20 * grid.n + 4 * grid.nx ** 3 * grid.xsub > 60 << 20
    m = 38000
    u = np.repeat(scene[1], m // 60 + 1, 0)[:m] * np.linspace(0.9, 1.1, m)[:, None, None]
    tols = np.array([0.1, 0.3])
    ub = torch.as_tensor(u, device=cuda).reshape(-1, 9).contiguous()
    cnt = torch.zeros((m, 2), dtype=torch.int32, device=cuda)
    al = lambda b: (b + 255) // 256 * 256
    ws = lib.id11b_grid_score_workspace_bytes(m, 2) if two else al(16 * m) + al(32 * m)
    buf = torch.empty(ws, dtype=torch.uint8, device=cuda)
    args = (ub.data_ptr(), m, grid.gv.data_ptr(), grid.n, grid.nx, grid.xsub, grid.buf.data_ptr())

    def score(size):
        return lib.id11b_dev_score_grid(*args, tols.ctypes.data, 2, cnt.data_ptr(), None,
                                        buf.data_ptr(), size, None)
    assert score(al(16 * m) + al(32 * m) - 256) == 4     # ID11B_ERR_SIZE
    assert score(ws) == 0
    torch.cuda.synchronize()
    assert grid.stats()["fallback_ubis"] == np.count_nonzero(~u.any((1, 2)))
    assert np.array_equal(cnt.cpu().numpy(), oracle.score_many(u, g, tols))
    npk = torch.zeros(m, dtype=torch.int32, device=cuda)
    mean = torch.zeros(m, dtype=torch.float64, device=cuda)
    ws = lib.id11b_grid_refine_workspace_bytes(m) if two else al(136 * m)
    buf = torch.empty(ws, dtype=torch.uint8, device=cuda)

    def refine(size):
        return lib.id11b_dev_refine_grid(*args, 0.1, 1, npk.data_ptr(), mean.data_ptr(),
                                         buf.data_ptr(), size, None)
    assert refine(al(136 * m) - 256) == 4
    assert refine(ws) == 0
    torch.cuda.synchronize()
    assert np.array_equal(npk.cpu().numpy(), oracle.score_many(u, g, [0.1])[:, 0])
    ur = ub.cpu().numpy().reshape(-1, 3, 3)
    for i in range(0, m, 997):
        k, mn, x = oracle.score_and_refine(u[i], g, 0.1)
        assert npk[i] == k and abs(float(mean[i]) - mn) <= 1e-12 * mn
        assert np.abs(ur[i] - x).max() <= 1e-11 * np.abs(x).max()


def test_assignment_starting_values(scene, oracle, cuda):
    """drlv2 on entry: NaN, infinities, zeros of both signs, negative, above
    tol^2, and exactly a grain's drlv2 (not below it: the label stays)."""
    from imaged11_b200 import batch
    gv, u = scene
    n = len(gv)
    exact = np.zeros(n) + 2
    _, exact, _ = oracle.score_and_assign(u[5], gv, 0.1, exact, np.zeros(n, np.int32), 1)
    rng = np.random.default_rng(93)
    d = rng.choice([np.nan, np.inf, -np.inf, 0.0, -0.0, -1.0, 0.01, 2.0, 1e-9], n)
    d[::3] = exact[::3]
    lab = rng.integers(-1, 70, n).astype(np.int32)
    rd, rl = d.copy(), lab.copy()
    for i, x in enumerate(u):
        _, rd, rl = oracle.score_and_assign(x, gv, 0.1, rd, rl, i)
    batch.score_and_assign_grid(u, batch.GvecGrid(gv), 0.1, d, lab)
    assert np.array_equal(lab, rl) and np.array_equal(d, rd, equal_nan=True)


@pytest.mark.parametrize("copies", [1, 3, 33, 70])
@pytest.mark.parametrize("ntol", [1, 3, 4])
def test_binned_sums_of_dense_boxes(oracle, copies, ntol, cuda):
    """Every g of a run inside every box (up to 32 x 32 pairs of one step, many
    more than a warp lists at once) and odd tiles: counts identical, sums equal
    to FP64 rounding and the fixed-point step of each term."""
    from imaged11_b200 import batch
    rng = np.random.default_rng(94 + copies)
    a = 4.0
    hkl = np.stack(np.meshgrid(*[np.arange(-3, 4)] * 3), -1).reshape(-1, 3)[1:].astype(float)
    g = np.repeat(hkl / a, copies, 0) + rng.normal(size=(len(hkl) * copies, 3)) * 1e-3
    u = a * np.eye(3)[None] * (1 + rng.normal(size=(101, 1, 1)) * 1e-3)
    tols = [0.3, 0.01, 0.1, 0.03][:ntol]
    c, s = batch.score_grid(u, batch.GvecGrid(g), tols, sums=True, method="bins")
    assert np.array_equal(c.cpu().numpy(), oracle.score_many(u, g, tols))
    step = 2.0 ** -(62 - np.ceil(np.log2(len(g) * max(tols) ** 2)))
    s = s.cpu().numpy()
    for i in range(0, len(u), 7):
        for j, t in enumerate(tols):
            n, mean, _ = oracle.score_and_refine(u[i], g, t)
            assert abs(s[i, j] - n * mean) <= 1e-12 * n * mean + n * step


@pytest.mark.parametrize("n", [0, 1, 4095, 4096, 4097, 30000])
@pytest.mark.parametrize("cell", [None, 0.6])
def test_build_is_repeatable(scene, n, cell, cuda):
    """The index's layout depends on the g alone, whatever order the build's
    atomics ran in: two builds and a rebuild refine to the same bits (g repeated,
    outside the regular range, and cells of one and of hundreds of g)."""
    import torch
    from imaged11_b200 import batch
    gv, u = scene
    g = gv[:n].copy()
    g[5:n:7] = g[4:n - 1:7][:len(g[5:n:7])]
    g[3:n:101] = np.nan
    grids = [batch.GvecGrid(g, cell=cell), batch.GvecGrid(g, cell=cell)]
    out = [batch.refine_grid(u.copy(), x, 0.1) for x in grids]
    grids[0].refresh()
    out.append(batch.refine_grid(u.copy(), grids[0], 0.1))
    st = grids[0].stats()
    assert st["special"] == int(np.isnan(g[:, 0]).sum())
    assert st["regular"] + st["special"] == len(g)
    for o in out[1:]:
        assert all(torch.equal(a, b) for a, b in zip(o, out[0]))


@pytest.mark.parametrize("grains", [1, 6, 12, 60])
@pytest.mark.parametrize("m", [1, 37, 3000])
def test_binned_join_of_crowded_trials(scene, oracle, grains, m, cuda):
    """Trials that crowd around a few orientations: streams that are counted
    first, that overflow the room they are given, and that fit; one to several
    work items a UBI; a UBI the join does not take among them."""
    from imaged11_b200 import batch, synth
    gv, _ = scene
    rng = np.random.default_rng(95)
    base = np.linalg.inv(synth.random_rotations(grains, rng) / 4.05)
    u = synth.perturb_ubis(base[np.arange(m) % grains], 0.3, 0.001, rng)
    if m > 20:
        u[11] = 0.0
    grid = batch.GvecGrid(gv)
    tols = [0.05, 0.15]
    c, s = batch.score_grid(u, grid, tols, sums=True, method="bins")
    ref = oracle.score_many(u, gv, tols)
    assert np.array_equal(c.cpu().numpy(), ref)
    assert np.array_equal(batch.score_grid(u, grid, tols, method="bins").cpu().numpy(), ref)
    w = batch.score_grid(u, grid, tols, sums=True, method="walk")[1]
    step = 2.0 ** -(62 - np.ceil(np.log2(len(gv) * max(tols) ** 2)))
    assert np.all((s - w).abs().cpu().numpy() <= 1e-12 * w.cpu().numpy() + ref * step)


@pytest.mark.parametrize("m", [1, 33, 1025])
def test_box_estimate(m, cuda):
    """The expected number of boxes against numpy, with UBIs that count none:
    singular, NaN, infinite, and more points than g.  Near singular UBIs lose digits in
    numpy's inverse: 1e-9."""
    import torch
    from imaged11_b200 import batch
    rng = np.random.default_rng(m)
    g = batch.GvecGrid(torch.from_numpy(rng.uniform(-1, 1, (4000, 3))).cuda())
    u = rng.normal(size=(m, 3, 3)) * 4
    if m > 8:
        u[1] = 0
        u[2, 1, 1] = np.nan
        u[3, 0, 0] = np.inf
        u[4] *= 1e3
    tol = 0.05
    want = 0.0
    for k in range(m):
        det = abs(np.linalg.det(u[k])) if np.isfinite(u[k]).all() else 0.0
        if det > 0:
            r = g.rmax + (tol + 1e-6) * np.linalg.norm(np.linalg.inv(u[k]))
            est = 4 / 3 * np.pi * r ** 3 * det
            want += est if est <= g.n else 0.0
    got = batch.bins_box_estimate(torch.from_numpy(u).cuda(), g, tol)
    assert abs(got - (1.25 * want + 64 * m)) <= 1 + 1e-9 * want


@pytest.mark.parametrize("tols", [[0.05], [0.0], [1e-5, 0.05], [0.05, 0.05], [0.1, 0.05, 0.03],
                                  [0.39, 1e-4, 0.05, np.nextafter(0.05, 1)]])
@pytest.mark.parametrize("n", [4000, 4001])
def test_binned_counts_at_the_thresholds(oracle, tols, n, cuda):
    """Most g lie one tolerance from a lattice point to within rounding, so their
    FP32 values fall into the bands that are evaluated exactly (and into several at
    once for equal tolerances); the counts must be the oracle's."""
    import torch
    from imaged11_b200 import batch
    rng = np.random.default_rng(n)
    ub = np.linalg.qr(rng.normal(size=(3, 3)))[0] / 4.05
    hkl = rng.integers(-5, 6, (n, 3))
    d = rng.normal(size=(n, 3))
    d *= rng.choice(tols, n)[:, None] / np.linalg.norm(d, axis=1, keepdims=True)
    g = (hkl + d) @ ub.T
    u = np.linalg.inv(ub)[None] + rng.normal(size=(40, 3, 3)) * 1e-6
    u[0] = np.linalg.inv(ub)
    grid = batch.GvecGrid(torch.from_numpy(g).cuda())
    want = oracle.score_many(u, g, tols)
    for sums in (False, True):
        got = batch.score_grid(u, grid, tols, method="bins", sums=sums)
        got = got[0] if sums else got
        assert np.array_equal(got.cpu().numpy(), want)
