"""Fused detector -> lab -> geometry pass (Ctransform.sf2geometry) against the
two separate drop-in calls (bit for bit) and against the oracle's
compute_xlylzl + compute_geometry (xyz bit for bit; angles and g within the
sin/cos tolerance of the other geometry tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GV_ULPS = 64


def _close_ulps(a, b, ulps):
    scale = np.abs(b).max(axis=-1, keepdims=True)
    return np.all(np.abs(a - b) <= ulps * np.spacing(scale))


def _pars(rng, tilt=True):
    return {"y_center": 1024.3, "z_center": 1021.7, "y_size": 75.0, "z_size": 75.2,
            "distance": 152300.0, "wavelength": 0.2846, "omegasign": -1.0,
            "tilt_x": 0.004 if tilt else 0.0, "tilt_y": -0.002 if tilt else 0.0,
            "tilt_z": 0.006 if tilt else 0.0, "o11": 1, "o12": 0, "o21": 0, "o22": -1,
            "wedge": 0.01 if tilt else 0.0, "chi": 0.02 if tilt else 0.0}


@pytest.mark.parametrize("tilt,t", [(True, (5.0, -3.0, 2.0)), (False, (0.0, 0.0, 0.0))])
def test_sf2geometry(oracle, tilt, t, cuda):
    import torch
    from imaged11_b200 import transform
    rng = np.random.default_rng(71)
    n = 100_003                                 # ragged final tile
    sc = rng.uniform(0, 2048, n)
    fc = rng.uniform(0, 2048, n)
    om = rng.uniform(-180, 360, n)
    sc[:3] = [1021.7, np.nan, 0.0]              # on the beam centre row, NaN, edge
    ct = transform.Ctransform(_pars(rng, tilt))
    xyz, out = ct.sf2geometry(sc, fc, om, *t)
    xyz2 = ct.sf2xyz(sc, fc)
    out2 = ct.xyz2geometry(xyz2, om, *t)
    assert np.array_equal(xyz, xyz2, equal_nan=True)
    assert np.array_equal(out, out2, equal_nan=True)
    ref_x = oracle.compute_xlylzl(sc, fc, ct.cen, ct.rmat, ct.distance_vec)
    assert np.array_equal(xyz, ref_x, equal_nan=True)
    p = ct.pars
    ref = oracle.compute_geometry(ref_x, om, p["omegasign"], p["wavelength"], p["wedge"],
                                  p["chi"], np.array(t))
    fin = np.isfinite(ref).all(1)
    assert np.array_equal(np.isfinite(out).all(1), fin)
    assert np.abs(out[fin, :2] - ref[fin, :2]).max() < 1e-11
    assert _close_ulps(out[fin, 3:], ref[fin, 3:], GV_ULPS)
    assert np.allclose(out[fin, 2], ref[fin, 2], rtol=1e-14, atol=0)
    # device tensors in, device tensors out, without the lab positions
    xd, od = ct.sf2geometry(torch.tensor(sc, device=cuda), torch.tensor(fc, device=cuda),
                            torch.tensor(om, device=cuda), *t, xyz=False)
    assert xd is None and od.is_cuda
    assert np.array_equal(od.cpu().numpy(), out, equal_nan=True)


def test_ctransform_methods_match_drop_in(cuda):
    from imaged11_b200 import transform
    rng = np.random.default_rng(72)
    ct = transform.Ctransform(_pars(rng))
    sc, fc, om = rng.uniform(0, 2048, 999), rng.uniform(0, 2048, 999), rng.uniform(0, 360, 999)
    g = ct.sf2gv(sc, fc, om, 1.0, 2.0, 3.0)
    out = ct.xyz2geometry(ct.sf2xyz(sc, fc), om, 1.0, 2.0, 3.0)
    assert np.array_equal(g, out[:, 3:])
    with pytest.raises(ValueError):
        ct.sf2geometry(sc, fc[:10], om)


def test_inverse_root_rounds_as_root_and_division(oracle, cuda):
    """With no rotation g is ds (d / |d| - beam) in the reference's operations, exactly
    but for 1 / |d|, which the kernel takes in one go: every bit as the IEEE root and
    division give it, but for values within 2^-80 of halfway between two doubles.
    Of 4 million two roundings at odds of some 2^-27 each make 0.06; at most two may
    differ, by a last place of 1 / |d|."""
    from imaged11_b200 import cImageD11
    rng = np.random.default_rng(75)
    n = 4_000_000
    x = rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-6, 9, (n, 1))
    x[: n // 2, 0] = 10.0 ** rng.uniform(3, 6, n // 2)         # near the direct beam
    x[: n // 2, 1:] *= 1e-3
    om, t, wvln = np.zeros(n), np.zeros(3), 0.2846
    g = np.empty((n, 3))
    cImageD11.compute_gv(x, om, 1.0, wvln, 0.0, 0.0, t, g)
    ref = oracle.compute_gv(x, om, 1.0, wvln, 0.0, 0.0, t)
    diff = np.abs(g - ref).max(1)
    assert np.count_nonzero(diff) <= 2
    assert np.all(diff <= 2.0 ** -51 / wvln)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 255, 256, 257, 700])
def test_positions_off_16_bytes(n, cuda):
    """Positions and omega that are 8 bytes off a 16-byte boundary (a slice of a larger
    table) take another kernel: the same bits, nothing read past the end."""
    import torch
    from imaged11_b200._lib import lib, check
    rng = np.random.default_rng(74)
    xyz = torch.tensor(rng.uniform(-1e5, 1e5, 3 * n + 1), device=cuda)
    om = torch.tensor(rng.uniform(0, 360, n + 1), device=cuda)
    t = np.array([5.0, -3.0, 2.0])
    out = torch.full((2, 6 * n + 1), -7.0, dtype=torch.float64, device=cuda)
    for row, x, w in ((0, xyz[1:], om[1:]), (1, xyz[1:].clone(), om[1:].clone())):
        assert (x.data_ptr() % 16, w.data_ptr() % 16) == ((8, 8) if row == 0 else (0, 0))
        check(lib.id11b_dev_compute_geometry(x.data_ptr(), w.data_ptr(), -1.0, 0.28, 0.01, 0.02,
                                             t.ctypes.data, out[row].data_ptr(), n, None),
              "compute_geometry")
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1]) and bool((out[:, -1] == -7.0).all())


@pytest.mark.parametrize("kind", ["nodes", "tiny", "special"])
def test_angles(kind, cuda):
    """Two-theta and eta of given positions (no rotation, no translation, so the
    diffraction vector is the position) in every octant: ratios at and between the
    arctangent table's nodes, tiny ratios, and what goes to the library's function.
    Against numpy with 64-bit mantissas: the root before (1/2 ulp), the arctangent
    (1 ulp) and the degrees (1/2 ulp and the constant's 1/2), each up to doubled by
    the next one's spacing: 5 ulp."""
    from imaged11_b200 import transform
    rng = np.random.default_rng(73)
    if kind == "nodes":
        r = (np.arange(0, 129)[:, None] / 128.0 + [0.0, 1e-16, -1e-9, 1e-9, 3e-3]).ravel()
        r = np.abs(r)
        y, z = np.r_[r, np.ones_like(r)] * 1e4, np.r_[np.ones_like(r), r] * 1e4
    elif kind == "tiny":
        r = 10.0 ** rng.uniform(-40, -2, 3000)
        y, z = np.r_[r, np.ones_like(r)] * 37.0, np.r_[np.ones_like(r), r] * 37.0
    else:
        v = np.array([0.0, 1.0, np.inf, np.nan, 2.0 ** -101, 2.0 ** -100, 2.0 ** 100, 2.0 ** 101,
                      1e-160, 1e150])
        y, z = (a.ravel() for a in np.meshgrid(v, v))
    y, z = np.r_[y, -y, y, -y], np.r_[z, z, -z, -z]
    xyz = np.stack([rng.choice(z, len(z)), y, z], axis=1)
    p = dict(_pars(rng, False), wedge=0.0, chi=0.0)
    out = transform.Ctransform(p).xyz2geometry(xyz, np.zeros(len(xyz)), 0.0, 0.0, 0.0)
    d = xyz.astype(np.longdouble)
    deg = np.longdouble(180) / np.arctan2(np.longdouble(0), np.longdouble(-1))
    with np.errstate(all="ignore"):
        q = np.sqrt(xyz[:, 1] ** 2 + xyz[:, 2] ** 2)      # overflows where the kernel's does
        mid = (q > 1e-100) & (q < 1e150)
        q = np.where(mid, np.sqrt(d[:, 1] ** 2 + d[:, 2] ** 2), q)
        want = np.stack([np.arctan2(q, d[:, 0]), np.arctan2(-d[:, 1], d[:, 2])], axis=1) * deg
    near = want.astype(np.float64)
    assert np.array_equal(np.isnan(out[:, :2]), np.isnan(near))
    ok = np.isfinite(near)
    assert np.all(np.abs(out[:, :2].astype(np.longdouble) - want)[ok] <=
                  5 * np.spacing(np.abs(near[ok])))
    assert np.array_equal(np.signbit(out[:, 1][ok[:, 1]]), np.signbit(near[:, 1][ok[:, 1]]))
