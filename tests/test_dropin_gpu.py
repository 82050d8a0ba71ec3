"""Parity of the drop-in module (imaged11_b200.cImageD11) with the reference.

Every call goes through the C ABI: numpy arguments take the reference-
signature host entry points, CUDA tensors take the device entry points.
Decisions (counts, labels, hkl) are bit-exact; floating-point results carry
the tolerance written in each test.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# compute_gv: CUDA's sincos is within 2 ulp of the reference's libm, the rest
# of the arithmetic is operation-for-operation identical, so g agrees to a few
# ulp of its largest component.
GV_ULPS = 64


def _close_ulps(a, b, ulps):
    scale = np.maximum(np.abs(b).max(axis=-1, keepdims=True), 1e-300)
    return np.all(np.abs(a - b) <= ulps * np.spacing(scale))


@pytest.fixture(scope="module")
def cim():
    from imaged11_b200 import cImageD11
    return cImageD11


def test_verify_rounding(cim, cuda):
    for n in (0, 1, 20, 12345, -7):
        assert cim.verify_rounding(n) == 0


def test_compute_gv_host_and_device(cim, golden, cuda):
    import torch
    d = golden["compute_gv"]
    for i in range(int(d["gv_ncases"])):
        osg, wl, w, c, tx, ty, tz = d["gv%d_params" % i]
        gv = np.empty((len(d["gv_omega"]), 3))
        cim.compute_gv(d["gv_xlylzl"], d["gv_omega"], osg, wl, w, c, [tx, ty, tz], gv)
        assert _close_ulps(gv, d["gv%d_out" % i], GV_ULPS), np.abs(gv - d["gv%d_out" % i]).max()
        assert np.allclose(gv, d["gv%d_numpy" % i])
        out = np.empty((len(gv), 6))
        cim.compute_geometry(d["gv_xlylzl"], d["gv_omega"], osg, wl, w, c, [tx, ty, tz], out)
        ref = d["gv%d_geometry" % i]
        assert np.abs(out[:, :2] - ref[:, :2]).max() < 1e-11      # degrees
        assert _close_ulps(out[:, 3:], ref[:, 3:], GV_ULPS)
        assert np.allclose(out[:, 2], ref[:, 2], rtol=1e-14, atol=0)
    osg, wl, w, c, tx, ty, tz = d["rand_params"]
    x = torch.tensor(d["rand_xlylzl"], device=cuda)
    om = torch.tensor(d["rand_omega"], device=cuda)
    g = torch.empty_like(x)
    cim.compute_gv(x, om, osg, wl, w, c, [tx, ty, tz], g)
    assert _close_ulps(g.cpu().numpy(), d["rand_gv"], GV_ULPS)


def test_compute_xlylzl_bitexact(cim, golden, cuda):
    d = golden["compute_xlylzl"]
    for r, ref in zip(d["xl_r"], d["xl_out"]):
        out = np.empty((len(d["xl_s"]), 3))
        cim.compute_xlylzl(d["xl_s"], d["xl_f"], d["xl_p"], r, d["xl_dist"], out)
        assert np.array_equal(out, ref)


def test_score_bitexact(cim, golden, cuda):
    import torch
    d = golden["scoring"]
    gv_dev = torch.tensor(d["sc_gv"], device=cuda)
    for i, u in enumerate(d["sc_ubis"]):
        for j, t in enumerate(d["sc_tols"]):
            assert cim.score(u, d["sc_gv"], t) == d["sc_counts"][i, j]
            assert cim.score(u, gv_dev, t) == d["sc_counts"][i, j]


# Least squares: the GPU sums R = sum ih g^T in a fixed tree instead of the
# reference's sequential order; n and H are exact, UBI and mean drlv2 agree to
# rounding of that order.
UBI_RTOL = 1e-12
DRLV2_RTOL = 1e-12


def test_score_and_refine(cim, golden, cuda):
    import torch
    d = golden["scoring"]
    gv = d["sc_gv"]
    gv_dev = torch.tensor(gv, device=cuda)
    for i, u in enumerate(d["sc_ubis"]):
        for j, t in enumerate(d["sc_tols"]):
            uu = np.array(u, order="C")
            n, m = cim.score_and_refine(uu, gv, t)
            assert n == d["sar_n"][i, j]
            assert abs(m - d["sar_drlv2"][i, j]) <= DRLV2_RTOL * abs(d["sar_drlv2"][i, j])
            ref = d["sar_ubi"][i, j]
            assert np.abs(uu - ref).max() <= UBI_RTOL * np.abs(ref).max()
            ud = torch.tensor(u, device=cuda).contiguous()
            n2, m2 = cim.score_and_refine(ud, gv_dev, t)
            assert n2 == n and m2 == m
            assert np.array_equal(ud.cpu().numpy(), uu)      # same kernels, same order


def test_score_and_refine_iterated(cim, golden, cuda):
    d = golden["scoring"]
    for i, u in enumerate(d["sc_ubis"][:20]):
        uu = np.array(u, order="C")
        for _ in range(3):
            cim.score_and_refine(uu, d["sc_gv"], 0.05)
        ref = d["sar3_ubi"][i]
        assert np.abs(uu - ref).max() <= 1e-11 * np.abs(ref).max()


def test_refine_assigned(cim, golden, cuda):
    d = golden["scoring"]
    for gi in range(8):
        u = np.array(d["sc_ubis"][gi], order="C")
        n, m = cim.refine_assigned(u, d["sc_gv"], d["ra_labels"], gi)
        assert n == d["ra_n"][gi]
        assert abs(m - d["ra_drlv2"][gi]) <= DRLV2_RTOL * abs(d["ra_drlv2"][gi])
        ref = d["ra_ubi"][gi]
        assert np.abs(u - ref).max() <= UBI_RTOL * np.abs(ref).max()


def test_refine_assigned_fortran_ubi_not_modified(cim, golden, cuda):
    d = golden["scoring"]
    u = np.asfortranarray(d["sc_ubis"][0])
    before = u.copy()
    cim.refine_assigned(u, d["sc_gv"], d["ra_labels"], 0)
    assert np.array_equal(u, before)


def test_score_and_assign_bitexact(cim, golden, cuda):
    import torch
    d = golden["scoring"]
    gv = d["sc_gv"]
    drl = np.full(len(gv), 2.0)
    lab = np.full(len(gv), -1, np.int32)
    gd = torch.tensor(gv, device=cuda)
    drl_d = torch.full((len(gv),), 2.0, dtype=torch.float64, device=cuda)
    lab_d = torch.full((len(gv),), -1, dtype=torch.int32, device=cuda)
    for i, u in enumerate(d["sc_ubis"][:24]):
        assert cim.score_and_assign(u, gv, 0.05, drl, lab, i) == d["sa_n"][i]
        assert cim.score_and_assign(u, gd, 0.05, drl_d, lab_d, i) == d["sa_n"][i]
    assert np.array_equal(drl, d["sa_drlv2"]) and np.array_equal(lab, d["sa_labels"])
    assert np.array_equal(drl_d.cpu().numpy(), d["sa_drlv2"])
    assert np.array_equal(lab_d.cpu().numpy(), d["sa_labels"])


def test_adversarial_edges_bitexact(cim, golden, cuda):
    d = golden["scoring"]
    u0, g = d["adv_ubi"], d["adv_gv"]
    for j, t in enumerate(d["sc_tols"]):
        assert cim.score(u0, g, t) == d["adv_counts"][j]
        uu = np.array(u0, order="C")
        n, m = cim.score_and_refine(uu, g[:-6], t)
        assert n == d["adv_sar_n"][j]
        ref = d["adv_sar_ubi"][j]
        assert np.abs(uu - ref).max() <= UBI_RTOL * np.abs(ref).max()


def test_singular_leaves_ubi_unchanged(cim, golden, cuda):
    d = golden["scoring"]
    u0 = d["adv_ubi"]
    for i, row in enumerate(d["sing_results"]):
        uu = np.array(u0, order="C")
        n, m = cim.score_and_refine(uu, d["sing%d_gv" % i], 0.05)
        assert n == row[0] and m == row[1]
        assert np.array_equal(uu.ravel(), row[2:])


def test_empty_inputs(cim, cuda):
    u = np.eye(3) * 4.05
    g = np.zeros((0, 3))
    assert cim.score(u, g, 0.1) == 0
    uu = u.copy()
    assert cim.score_and_refine(uu, g, 0.1) == (0, 0.0)
    assert np.array_equal(uu, u)
    out = np.zeros((0, 3))
    cim.compute_gv(np.zeros((0, 3)), np.zeros(0), 1., 0.3, 0., 0., [0, 0, 0], out)


def test_compute_gv_specialisations_and_nonfinite(cim, oracle, cuda):
    """Every host-chosen kernel variant (t zero or not, chi.wedge identity or
    not), with NaN / inf omega and lab positions mixed in: NaN positions match
    the reference exactly, finite values agree to GV_ULPS."""
    import torch
    rng = np.random.default_rng(77)
    n = 5000
    x = np.stack([rng.uniform(1.4e5, 1.6e5, n), rng.uniform(-8e4, 8e4, n),
                  rng.uniform(-8e4, 8e4, n)], 1)
    om = rng.uniform(0, 360, n)
    om[::97] = np.nan
    om[5::101] = np.inf
    x[7::103, 1] = np.nan
    x[9::107, 0] = np.inf
    for wedge, chi, t in [(0., 0., [0., 0., 0.]), (0., 0., [5., -3., 2.]),
                          (0.01, 0.02, [0., 0., 0.]), (0.01, 0.02, [5., -3., 2.])]:
        ref = oracle.compute_gv(x, om, 1.0, 0.2846, wedge, chi, t)
        xd = torch.tensor(x, device=cuda)
        od = torch.tensor(om, device=cuda)
        g = torch.empty_like(xd)
        cim.compute_gv(xd, od, 1.0, 0.2846, wedge, chi, t, g)
        got = g.cpu().numpy()
        assert np.array_equal(np.isnan(got), np.isnan(ref)), (wedge, chi, t)
        fin = np.isfinite(ref).all(1)
        assert np.array_equal(np.isinf(got), np.isinf(ref))
        assert _close_ulps(got[fin], ref[fin], GV_ULPS)


def test_host_calls_small_large_and_threads(cim, oracle, cuda):
    """Host-buffer calls stage through buffers kept per host thread (calls up to
    64 MB) or the stream-ordered pool (larger): alternate small and large
    calls, then run calls from four host threads at once; every result equals
    the oracle's (counts exact, UBIs 1e-12)."""
    from concurrent.futures import ThreadPoolExecutor
    from imaged11_b200 import synth
    rng = np.random.default_rng(71)
    nb = 1_600_000                                     # 38 MB of g, > 64 MB staged
    big = np.stack([150000.0 + rng.normal(0, 100, nb), rng.uniform(-1e5, 1e5, nb),
                    rng.uniform(-1e5, 1e5, nb)], axis=1)  # lab positions (um)
    om = rng.uniform(-180, 180, nb)
    ps = synth.simulate(4, "Al", gmax=1.0, seed=72)
    ubis = [np.array(u, order="C") for u in ps.ubis]
    g_big = np.empty_like(big)
    cim.compute_gv(big, om, 1.0, 0.2846, 0.01, -0.02, [10.0, -20.0, 5.0], g_big)
    ref = oracle.compute_gv(big, om, 1.0, 0.2846, 0.01, -0.02, np.array([10.0, -20.0, 5.0]))
    assert _close_ulps(g_big, ref, GV_ULPS)
    small = np.ascontiguousarray(g_big[:5000])
    for g in (small, g_big, small, ps.gv):
        for u in ubis:
            assert cim.score(u, g, 0.05) == oracle.score(u, g, 0.05)
            uu = u.copy()
            n, m = cim.score_and_refine(uu, g, 0.05)
            n2, m2, u2 = oracle.score_and_refine(u, g, 0.05)
            assert n == n2 and abs(m - m2) <= 1e-12 * abs(m2)
            assert np.abs(uu - u2).max() <= 1e-12 * np.abs(u2).max()

    def work(k):
        out = []
        for rep in range(20):
            u = ubis[(k + rep) % len(ubis)].copy()
            out.append((cim.score_and_refine(u, ps.gv, 0.05), u))
        return out

    with ThreadPoolExecutor(4) as ex:
        results = list(ex.map(work, range(4)))
    for k, res in enumerate(results):
        for rep, ((n, m), u) in enumerate(res):
            n2, m2, u2 = oracle.score_and_refine(ubis[(k + rep) % len(ubis)], ps.gv, 0.05)
            assert n == n2 and abs(m - m2) <= 1e-12 * abs(m2)
            assert np.abs(u - u2).max() <= 1e-12 * np.abs(u2).max()


@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 511, 513, 1535, 2047, 2049, 8191, 8192,
                               8193, 16383, 16384, 16385])
def test_least_squares_sizes(oracle, n, cuda):
    """Sizes around the CTAs, shares and tiles of the one-cluster launch and past
    it, from host arrays, device arrays and a device array that is not 16-byte
    aligned: counts exact, UBI and mean drlv2 to the rounding of sums in another
    order (1e-12)."""
    import torch
    from imaged11_b200 import cImageD11 as cim
    rng = np.random.default_rng(n)
    ubi = 4.05 * np.linalg.qr(rng.normal(size=(3, 3)))[0]
    gv = rng.integers(-5, 6, size=(n, 3)) @ np.linalg.inv(ubi).T + rng.normal(size=(n, 3)) * 4e-3
    labels = rng.integers(0, 3, n).astype(np.int32)
    labels[-1] = 1
    kept = gv[labels == 1]
    want = (oracle.score_and_refine(ubi, gv, 0.05), oracle.score_and_refine(ubi, kept, 1.0))
    dev = torch.tensor(np.concatenate([gv[:1], gv]), device=cuda)
    forms = ((gv, labels), (dev[1:].clone(), torch.tensor(labels, device=cuda)),
             (dev[1:], torch.tensor(labels, device=cuda)))
    assert forms[2][0].data_ptr() % 16 == 8
    for g, lab in forms:
        for mode, (rn, rmean, ru) in enumerate(want):
            host = isinstance(g, np.ndarray)
            u = ubi.copy() if host else torch.tensor(ubi, device=cuda)
            k, mean = cim.score_and_refine(u, g, 0.05) if mode == 0 else \
                cim.refine_assigned(u, g, lab, 1)
            u = u if host else u.cpu().numpy()
            assert k == rn
            if k > 3:       # (up to three peaks the normal matrix is singular to rounding)
                assert abs(mean - rmean) <= 1e-12 * rmean
                assert np.abs(u - np.asarray(ru)).max() <= 1e-12 * np.abs(ru).max() * \
                    max(1.0, 1e3 / k)
