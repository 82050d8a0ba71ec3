"""Measured cases: what a program built on this package has it do.

A case names an operation and its sizes.  The sizes are those of the package's
benchmark configurations (a 6k-peak drop-in sequence, a 1.1M-peak scan with
20,000 trial orientations, 2,000 unevenly filled grains, 500 grains for the
geometry gradient, a 10M-peak scan with 20,000 grains) and, for drawn cases,
log-uniform ranges below them.  Inputs are simulated on the GPU from the seed:
grains uniform on SO(3), every allowed reflection below |g| <= gmax seen twice
(the two rotation angles), centroid noise, and noise peaks uniform over the
detector and the rotation, as imaged11_b200.synth makes them on the host.
"""
import math

import numpy as np
import torch

from imaged11_b200 import adjoint, batch, synth, transform
from imaged11_b200 import cImageD11 as cim

F64 = torch.float64
TOLS = [0.02, 0.05, 0.1]
NOISE_G = 8e-4       # 1/Angstrom per component: 0.5 px and 0.05 degrees
TRUTH = dict(distance=152300., y_center=1027.7, z_center=1021.9, tilt_x=0.004, tilt_y=-0.002,
             tilt_z=0.006, wedge=0.01, chi=0.02, t_x=5., t_y=-3., t_z=2.)
# an experiment's first estimate of that geometry
ESTIMATE = dict(TRUTH, distance=152600., y_center=1028.1, z_center=1021.6, tilt_y=-0.0016,
                tilt_z=0.0057, wedge=0.015)


def listed():
    return [
        # an unchanged refinegrains caller: host arrays, one small call at a time
        {"name": "dropin_6k", "op": "dropin", "grains": 50},
        # one indexer.scorethem: a new index over a small scan, its trial
        # orientations scored at one tolerance
        {"name": "index_60k", "op": "index", "grains": 107, "gmax": 1.5, "trials": 1500,
         "tol": 0.05},
        # candidate scoring of a scan: index rebuilt from the g-vectors, 20,000
        # trials at three tolerances
        {"name": "score_1M", "op": "score", "grains": 2000, "gmax": 1.5, "trials": 20000,
         "sums": False},
        # the same with the summed drlv2 reported beside the counts
        {"name": "score_sums_560k", "op": "score", "grains": 1000, "gmax": 1.5, "trials": 5003,
         "sums": True},
        # fight_over_peaks on a full scan: every peak to the best of 20,000 grains
        {"name": "assign_10M", "op": "assign", "grains": 20000, "gmax": 1.27, "tol": 0.05},
        # the grains found in a scan refined against all of its peaks
        {"name": "refine_index_1M", "op": "refine_index", "grains": 2000, "gmax": 1.5,
         "tol": 0.05, "iters": 3},
        # grains with their own peaks, 20 to 2,000 each, five rounds
        {"name": "refine_grains_2k", "op": "refine_grains", "grains": 2000, "least": 20,
         "most": 2000, "tol": 0.05, "iters": 5},
        # refinepositions: every grain's translation, 30 iterations
        {"name": "translations_500", "op": "translations", "grains": 500, "cell": "Al",
         "gmax": 1.75, "least": 420, "most": 560, "iters": 30},
        # one gradient of a joint refinement (12 geometry parameters, every UBI)
        {"name": "gradient_500", "op": "gradient", "grains": 500, "cell": "Al", "gmax": 1.75,
         "least": 420, "most": 560},
        # one evaluation of a full scan's geometry refinement, UBIs eliminated
        {"name": "projected_20k", "op": "projected", "grains": 20000, "cell": "Ti_hcp",
         "gmax": 1.27, "least": 300, "most": 480},
        # updateGeometry: detector positions to tth, eta, ds and g
        {"name": "geometry_10M", "op": "geometry", "peaks": 10000001, "tilted": True},
        # compute_gv of a scan
        {"name": "gv_10M", "op": "gv", "peaks": 10000000, "tilted": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["dropin", "index", "score", "score", "assign", "refine_index",
                     "refine_grains", "translations", "gradient", "projected", "geometry", "gv"])
    if op == "dropin":
        return {"op": op, "grains": _log(rng, 3, 50)}
    if op == "index":
        return {"op": op, "grains": _log(rng, 10, 300), "gmax": rng.choice([1.27, 1.5]),
                "trials": _log(rng, 100, 5000), "tol": round(rng.uniform(0.02, 0.1), 4)}
    if op == "score":
        return {"op": op, "grains": _log(rng, 100, 2000), "gmax": 1.5,
                "trials": _log(rng, 300, 20000), "sums": rng.random() < 0.3}
    if op == "assign":
        return {"op": op, "grains": _log(rng, 100, 20000), "gmax": 1.27,
                "tol": round(rng.uniform(0.02, 0.1), 4)}
    if op == "refine_index":
        return {"op": op, "grains": _log(rng, 50, 2000), "gmax": 1.5,
                "tol": round(rng.uniform(0.02, 0.08), 4), "iters": rng.choice([1, 3, 5])}
    if op == "refine_grains":
        return {"op": op, "grains": _log(rng, 50, 8000), "least": 20,
                "most": _log(rng, 100, 2000), "tol": 0.05, "iters": rng.choice([1, 3, 5])}
    if op == "translations":
        return {"op": op, "grains": _log(rng, 20, 500), "cell": "Al", "gmax": 1.75,
                "least": _log(rng, 50, 420), "most": _log(rng, 421, 560),
                "iters": rng.choice([20, 30])}
    if op == "gradient":
        return {"op": op, "grains": _log(rng, 50, 5000), "cell": "Al", "gmax": 1.75,
                "least": _log(rng, 50, 420), "most": _log(rng, 421, 560)}
    if op == "projected":
        return {"op": op, "grains": _log(rng, 100, 20000), "cell": "Ti_hcp", "gmax": 1.27,
                "least": _log(rng, 30, 300), "most": _log(rng, 301, 480)}
    return {"op": op, "peaks": _log(rng, 20000, 10000000), "tilted": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs --

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, dtype=F64, device="cuda")


def _randn(g, *shape):
    return torch.randn(shape, generator=g, dtype=F64, device="cuda")


def _rotations(n, g):
    q = _randn(g, n, 4)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)],
                       1).view(n, 3, 3)


def _small_rotations(n, degrees, g):
    a = _randn(g, n, 3)
    x, y, z = (a / a.norm(dim=1, keepdim=True)).unbind(1)
    c, s = math.cos(math.radians(degrees)), math.sin(math.radians(degrees))
    d = 1 - c
    return torch.stack([c + x * x * d, x * y * d - z * s, x * z * d + y * s,
                        y * x * d + z * s, c + y * y * d, y * z * d - x * s,
                        z * x * d - y * s, z * y * d + x * s, c + z * z * d], 1).view(n, 3, 3)


def _lattice(cell, gmax):
    hkl, B = synth.hkl_list(cell, gmax)
    return torch.tensor(hkl, device="cuda"), torch.tensor(B, device="cuda")


def _perturbed(ub, degrees, strain, g):
    """UBIs of these UBs rotated by `degrees` and strained."""
    n = ub.shape[0]
    e = _randn(g, n, 3, 3) * strain
    eye = torch.eye(3, dtype=F64, device="cuda")
    return torch.linalg.inv(_small_rotations(n, degrees, g) @
                            (eye + 0.5 * (e + e.transpose(1, 2))) @ ub).contiguous()


def _wedgechi(wedge, chi):
    w, c = wedge * (math.pi / 180), chi * (math.pi / 180)
    sw, cw = (torch.sin(w), torch.cos(w)) if torch.is_tensor(w) else (math.sin(w), math.cos(w))
    sc, cc = (torch.sin(c), torch.cos(c)) if torch.is_tensor(c) else (math.sin(c), math.cos(c))
    W = _matrix([[cw, 0., -sw], [0., 1., 0.], [sw, 0., cw]])
    C = _matrix([[1., 0., 0.], [0., cc, -sc], [0., sc, cc]])
    return W @ C


def _matrix(rows):
    return torch.stack([torch.stack([v if torch.is_tensor(v) else
                                     torch.tensor(float(v), dtype=F64, device="cuda")
                                     for v in r]) for r in rows])


def _detector(p):
    """r = R3(tilt_x).R2(tilt_y).R1(tilt_z).flip of tensors or numbers."""
    def sc(a):
        a = a if torch.is_tensor(a) else torch.tensor(float(a), dtype=F64, device="cuda")
        return torch.sin(a), torch.cos(a)
    (sx, cx), (sy, cy), (sz, cz) = sc(p["tilt_x"]), sc(p["tilt_y"]), sc(p["tilt_z"])
    R1 = _matrix([[cz, -sz, 0.], [sz, cz, 0.], [0., 0., 1.]])
    R2 = _matrix([[cy, 0., sy], [0., 1., 0.], [-sy, 0., cy]])
    R3 = _matrix([[1., 0., 0.], [0., cx, -sx], [0., sx, cx]])
    return R3 @ R2 @ R1 @ _matrix([[1., 0., 0.], [0., p["o22"], p["o21"]],
                                   [0., p["o12"], p["o11"]]])


def _lab(p, s, f):
    r = _detector(p)
    v1 = (f - p["y_center"]) * p["y_size"]
    v2 = (s - p["z_center"]) * p["z_size"]
    x = v1[:, None] * r[:, 1] + v2[:, None] * r[:, 2]
    return torch.cat([x[:, :1] + p["distance"], x[:, 1:]], 1)


def _k_of(p, xyz, omega, t):
    """(d, k, so, co) of lab positions; t: (3,) or one translation per peak."""
    M = _wedgechi(p["wedge"], p["chi"])
    a = omega * (p["omegasign"] * math.pi / 180)
    so, co = torch.sin(a), torch.cos(a)
    t = t.expand(len(so), 3)
    u = torch.stack([co * t[:, 0] - so * t[:, 1], so * t[:, 0] + co * t[:, 1], t[:, 2]], 1)
    d = xyz - u @ M.T
    dh = d / d.norm(dim=1, keepdim=True)
    k = torch.cat([dh[:, :1] - 1.0, dh[:, 1:]], 1) / p["wavelength"]
    return d, k, so, co, M


def _g_of(p, xyz, omega, t):
    d, k, so, co, M = _k_of(p, xyz, omega, t)
    v = k @ M
    return torch.stack([co * v[:, 0] + so * v[:, 1], co * v[:, 1] - so * v[:, 0], v[:, 2]], 1)


def _translation(p):
    return torch.stack([v if torch.is_tensor(v) else torch.tensor(float(v), dtype=F64,
                                                                  device="cuda")
                        for v in (p["t_x"], p["t_y"], p["t_z"])])


def _noise_g(n, p, g):
    """g-vectors of peaks uniform over the detector and the rotation."""
    s, f, om = _rand(g, n) * p["dim"], _rand(g, n) * p["dim"], _rand(g, n) * 360.
    return _g_of(p, _lab(p, s, f), om, _translation(p))


def _scene(cells, gmax, noise, g):
    """(gv shuffled, UBs) of a scan: cells is [(cell, grains), ...]."""
    gv, ubs = [], []
    for cell, n in cells:
        hkl, B = _lattice(cell, gmax)
        ub = _rotations(n, g) @ B
        x = torch.einsum("nij,hj->nhi", ub, hkl).reshape(-1, 3).repeat(2, 1)
        gv.append(x + _randn(g, *x.shape) * NOISE_G)
        ubs.append(ub)
    gv = torch.cat(gv)
    gv = torch.cat([gv, _noise_g(int(noise * len(gv)), synth.default_geometry(), g)])
    return gv[torch.randperm(len(gv), generator=g, device="cuda")].contiguous(), torch.cat(ubs)


def _trials(ub, m, g):
    """10% true orientations 0.5 degrees off, the rest uniform on SO(3)."""
    near = max(1, m // 10)
    pick = torch.randint(0, len(ub), (near,), generator=g, device="cuda")
    a = _perturbed(ub[pick], 0.5, 0.0, g)
    B = torch.tensor(synth.hkl_list("Al", 0.5)[1], device="cuda")
    b = torch.linalg.inv(_rotations(m - near, g) @ B)
    u = torch.cat([a, b])
    return u[torch.randperm(m, generator=g, device="cuda")].contiguous()


def _spots(case, p, g, spread=0.0):
    """Peaks of grains on the detector, sorted by grain: dict of s, f, omega,
    hkl, grain, offsets, ub, translations."""
    n = case["grains"]
    hkl, B = _lattice(case["cell"], case["gmax"])
    ub = _rotations(n, g) @ B
    t = _translation(p) + (2 * _rand(g, n, 3) - 1) * spread
    M = _wedgechi(p["wedge"], p["chi"])
    r = _detector(p)
    dist = torch.tensor([p["distance"], 0., 0.], dtype=F64, device="cuda")
    nrm = torch.linalg.cross(r[:, 1], r[:, 2])
    H = len(hkl)
    G = torch.einsum("nij,hj->nhi", ub, hkl)
    lam = p["wavelength"]
    A = M[0, 0] * G[..., 0] + M[0, 1] * G[..., 1]
    C = M[0, 1] * G[..., 0] - M[0, 0] * G[..., 1]
    q = (-0.5 * lam * (G * G).sum(-1) - M[0, 2] * G[..., 2]) / torch.hypot(A, C)
    phi, dw = torch.atan2(C, A), torch.acos(q.clamp(-1, 1))
    w = torch.cat([phi + dw, phi - dw], 1)                       # (n, 2H)
    G = torch.cat([G, G], 1)
    co, so = torch.cos(w), torch.sin(w)
    v = torch.stack([co * G[..., 0] - so * G[..., 1], so * G[..., 0] + co * G[..., 1],
                     G[..., 2]], -1)
    dh = lam * (v @ M.T) + torch.tensor([1., 0., 0.], dtype=F64, device="cuda")
    tt = t[:, None, :]
    o = torch.stack([co * tt[..., 0] - so * tt[..., 1], so * tt[..., 0] + co * tt[..., 1],
                     tt[..., 2].expand_as(co)], -1) @ M.T
    rel = o + ((dist - o) @ nrm / (dh @ nrm))[..., None] * dh - dist
    f = (rel @ r[:, 1]) / p["y_size"] + p["y_center"]
    s = (rel @ r[:, 2]) / p["z_size"] + p["z_center"]
    on = (torch.cat([q, q], 1).abs() <= 1) & (f >= 0) & (f < p["dim"]) & (s >= 0) & (s < p["dim"])
    # of each grain's spots on the detector, a random count[i]
    key = _rand(g, n, 2 * H) + torch.where(on, 0.0, 2.0)
    order = key.argsort(1)
    span = case["most"] - case["least"] + 1
    count = case["least"] + (torch.arange(n, device="cuda") * 7919) % span
    keep = torch.arange(2 * H, device="cuda")[None, :] < count[:, None]
    grain = torch.arange(n, device="cuda")[:, None].expand(n, 2 * H)[keep]
    at = order[keep]
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = count.cumsum(0)
    m = len(at)
    return {"s": s[grain, at] + 0.5 * _randn(g, m), "f": f[grain, at] + 0.5 * _randn(g, m),
            "omega": torch.rad2deg(w[grain, at]) % 360. + 0.05 * _randn(g, m),
            "hkl": hkl[at % H].contiguous(), "grain": grain, "offsets": off, "ub": ub, "t": t}


def _segments(case, g):
    """Grains of hexagonal Ti with their shortest reflections, log-uniform counts."""
    n, lo, hi = case["grains"], case["least"], case["most"]
    gmax = (3.2 * hi / (4.1888 * 35.27)) ** (1 / 3) + 0.2
    hkl, B = _lattice("Ti_hcp", gmax)
    # the counts' distribution is the case's, their order the seed's
    q = (torch.arange(n, dtype=F64, device="cuda") + 0.5) / n
    count = torch.exp(math.log(lo) + q * math.log(hi / lo)).long()
    count = count[torch.randperm(n, generator=g, device="cuda")]
    ub = _rotations(n, g) @ B
    grain = torch.repeat_interleave(torch.arange(n, device="cuda"), count)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = count.cumsum(0)
    rank = torch.arange(len(grain), device="cuda") - off[grain]
    gv = torch.einsum("nij,nj->ni", ub[grain], hkl[rank])
    return (gv + _randn(g, *gv.shape) * 5e-4).contiguous(), off, grain, \
        _perturbed(ub, 0.2, 0.002, g)


def _inputs(case, seed):
    """The case's inputs as plain tensors, with none of the package's plans."""
    g = _gen(seed)
    op = case["op"]
    if op == "dropin":
        p = synth.default_geometry()
        d = _spots({"grains": case["grains"], "cell": "Al", "gmax": 1.0, "least": 100,
                    "most": 118}, p, g)
        m = len(d["s"]) // 10
        s = torch.cat([d["s"], _rand(g, m) * p["dim"]])
        f = torch.cat([d["f"], _rand(g, m) * p["dim"]])
        om = torch.cat([d["omega"], _rand(g, m) * 360.])
        o = torch.randperm(len(s), generator=g, device="cuda")
        return {"p": p, "xyz": _lab(p, s[o], f[o]), "omega": om[o],
                "ubis": _perturbed(d["ub"], 0.1, 0.001, g)}
    if op in ("index", "score"):
        gv, ub = _scene([("Al", case["grains"])], case["gmax"], 0.10, g)
        return {"gv": gv, "ubis": _trials(ub, case["trials"], g)}
    if op == "assign":
        a = int(0.7 * case["grains"])
        gv, ub = _scene([("Ti_hcp", a), ("Ti_beta", case["grains"] - a)], case["gmax"], 0.15, g)
        return {"gv": gv, "ubis": _perturbed(ub, 0.2, 0.002, g)}
    if op == "refine_index":
        gv, ub = _scene([("Al", case["grains"])], case["gmax"], 0.10, g)
        return {"gv": gv, "ubis": _perturbed(ub, 0.1, 0.001, g)}
    if op == "refine_grains":
        gv, off, grain, ubis = _segments(case, g)
        return {"gv": gv, "offsets": off, "grain": grain, "ubis": ubis}
    if op in ("translations", "gradient", "projected"):
        p = synth.default_geometry(**TRUTH)
        d = _spots(case, p, g, 60.0 if op == "translations" else 0.0)
        d["p"] = p
        d["ubis"] = torch.linalg.inv(d["ub"]) if op == "translations" else \
            _perturbed(d["ub"], 0.05, 0.0005, g)
        if op == "translations":
            d["xyz"] = _lab(p, d["s"], d["f"])
        return d
    p = synth.default_geometry(**(dict(TRUTH, wedge=0.01) if case["tilted"] else {}))
    n = case["peaks"]
    return {"p": p, "s": _rand(g, n) * p["dim"], "f": _rand(g, n) * p["dim"],
            "omega": _rand(g, n) * 360.}


# --------------------------------------------------------------------- run --

def prepare(case, seed):
    x = _inputs(case, seed)
    op = case["op"]
    st = {"case": case, "x": x}
    if op == "dropin":
        st["xyz"], st["omega"] = x["xyz"].cpu().numpy(), x["omega"].cpu().numpy()
        st["ubis"] = x["ubis"].cpu().numpy()
    elif op == "score":
        st["grid"] = batch.GvecGrid(x["gv"])
        st["ws"] = batch.BinsWorkspace(len(x["ubis"]), st["grid"], batch.bins_box_estimate(
            x["ubis"], st["grid"], max(TOLS)))
    elif op == "assign":
        st["grid"] = batch.GvecGrid(x["gv"])
        n = len(x["gv"])
        st["d"] = torch.empty(n, dtype=F64, device="cuda")
        st["lab"] = torch.empty(n, dtype=torch.int32, device="cuda")
    elif op == "refine_index":
        st["grid"] = batch.GvecGrid(x["gv"])
    elif op == "refine_grains":
        st["grains"] = batch.GrainSet(x["gv"], x["offsets"], x["ubis"])
        st["u0"] = st["grains"].ubis.clone()
    elif op == "translations":
        st["t0"] = torch.zeros((case["grains"], 3), dtype=F64, device="cuda")
    elif op in ("gradient", "projected"):
        st["peaks"] = adjoint.PeakTable(x["s"], x["f"], x["omega"], x["hkl"], x["offsets"], x["p"])
        st["params"] = adjoint.params_tensor(dict(x["p"], **ESTIMATE))
    elif op == "geometry":
        st["ct"] = transform.Ctransform(x["p"])
    elif op == "gv":
        st["xyz"] = _lab(x["p"], x["s"], x["f"]).contiguous()
        st["gv"] = torch.empty_like(st["xyz"])
    return st


def run(st):
    case, x = st["case"], st["x"]
    op = case["op"]
    if op == "dropin":
        p = x["p"]
        gv = np.empty_like(st["xyz"])
        cim.compute_gv(st["xyz"], st["omega"], p["omegasign"], p["wavelength"], p["wedge"],
                       p["chi"], [0., 0., 0.], gv)
        us, ns, ds = [], [], []
        for u in st["ubis"]:
            u = np.array(u, order="C")
            for _ in range(3):
                n, d = cim.score_and_refine(u, gv, 0.05)
            us.append(u)
            ns.append(n)
            ds.append(d)
        return {"gv": gv, "ubis": np.array(us), "n": np.array(ns), "mean": np.array(ds)}
    if op == "index":
        return batch.score_grid(x["ubis"], batch.GvecGrid(x["gv"]), [case["tol"]])
    if op == "score":
        st["grid"].refresh()
        return batch.score_grid(x["ubis"], st["grid"], TOLS, sums=case["sums"],
                                workspace=st["ws"])
    if op == "assign":
        st["d"].fill_(2.0)
        st["lab"].fill_(-1)
        batch.score_and_assign_grid(x["ubis"], st["grid"], case["tol"], st["d"], st["lab"])
        return {"drlv2": st["d"], "labels": st["lab"]}
    if op == "refine_index":
        u, n, d = batch.refine_grid(x["ubis"].clone(), st["grid"], case["tol"], case["iters"])
        return {"ubis": u, "n": n, "mean": d}
    if op == "refine_grains":
        st["grains"].ubis.copy_(st["u0"])
        u, n, d = st["grains"].refine(case["tol"], case["iters"])
        return {"ubis": u, "n": n, "mean": d}
    if op == "translations":
        p = x["p"]
        t, cost, n = batch.refine_translations(x["xyz"], x["omega"], x["offsets"], x["ubis"],
                                               st["t0"], p["omegasign"], p["wavelength"],
                                               p["wedge"], p["chi"], iters=case["iters"])
        return {"t": t, "cost": cost, "n": n}
    if op == "gradient":
        a = st["params"].clone().requires_grad_(True)
        u = x["ubis"].clone().requires_grad_(True)
        value = adjoint.loss(a, u, st["peaks"])
        value.backward()
        return {"loss": value.detach(), "params": a.grad, "ubis": u.grad}
    if op == "projected":
        a = st["params"].clone().requires_grad_(True)
        ubis = torch.empty((case["grains"], 3, 3), dtype=F64, device="cuda")
        value = adjoint.projected_loss(a, st["peaks"], ubis)
        value.backward()
        return {"loss": value.detach(), "params": a.grad, "ubis": ubis}
    if op == "geometry":
        p = x["p"]
        xyz, out = st["ct"].sf2geometry(x["s"], x["f"], x["omega"], p["t_x"], p["t_y"], p["t_z"])
        return {"xyz": xyz, "out": out}
    p = x["p"]
    cim.compute_gv(st["xyz"], x["omega"], p["omegasign"], p["wavelength"], p["wedge"], p["chi"],
                   [p["t_x"], p["t_y"], p["t_z"]], st["gv"])
    return st["gv"]


# -------------------------------------------------------------------- work --

def _reflections(cell, gmax):
    return len(synth.hkl_list(cell, gmax)[0])


def _volume(cell):
    return 1.0 / abs(np.linalg.det(synth.b_matrix(*synth.CELLS[cell][:6])))


def _scan_peaks(case):
    if case["op"] == "assign":
        a = int(0.7 * case["grains"])
        n = 2 * (a * _reflections("Ti_hcp", case["gmax"]) +
                 (case["grains"] - a) * _reflections("Ti_beta", case["gmax"]))
        return n + int(0.15 * n)
    n = 2 * case["grains"] * _reflections("Al", case["gmax"])
    return n + int(0.10 * n)


def _lookup_flops(m, n, tol, cell):
    """m orientations against n g-vectors through their lattice points: each
    point once (20), each g within tol of one by chance once (30)."""
    points = 4.2 * 2.17 ** 3 * _volume(cell)
    return m * (20 * points + 30 * n * 4.2 * tol ** 3)


def work(case):
    """Inputs read once, outputs written once; FP32 or FP64 operations that the
    result takes."""
    op = case["op"]
    if op == "dropin":
        n = int(120 * case["grains"])
        return {"bytes": 56 * n + 3 * case["grains"] * 24 * n,
                "flops": 90 * n + 3 * case["grains"] * 60 * n}
    if op in ("index", "score"):
        n, m = _scan_peaks(case), case["trials"]
        tols = [case["tol"]] if op == "index" else TOLS
        wide = 12 if case.get("sums") else 4
        return {"bytes": 24 * n + 72 * m + wide * len(tols) * m,
                "flops": _lookup_flops(m, n, max(tols), "Al")}
    if op == "assign":
        n, m = _scan_peaks(case), case["grains"]
        own = 60 * 2 * _reflections("Ti_hcp", case["gmax"]) * m
        return {"bytes": 36 * n + 72 * m, "flops": _lookup_flops(m, n, case["tol"], "Ti_hcp") + own}
    if op == "refine_index":
        n, m = _scan_peaks(case), case["grains"]
        own = 90 * 2 * _reflections("Al", case["gmax"]) * m
        return {"bytes": 24 * n + 156 * m,
                "flops": case["iters"] * (_lookup_flops(m, n, case["tol"], "Al") + own)}
    if op == "refine_grains":
        r = case["most"] / case["least"]
        n = case["grains"] * case["least"] * (r - 1) / math.log(r)
        return {"bytes": 24 * n + 156 * case["grains"], "flops": 75 * n * case["iters"]}
    if op in ("translations", "gradient", "projected"):
        n = 0.5 * (case["least"] + case["most"]) * case["grains"]
        each = {"translations": 400 * (case.get("iters", 0) + 1), "gradient": 400,
                "projected": 550}[op]
        row = {"translations": 32, "gradient": 48, "projected": 48}[op]
        return {"bytes": row * n + 144 * case["grains"], "flops": each * n}
    n = case["peaks"]
    return {"bytes": (96 if op == "geometry" else 56) * n, "flops": (250 if op == "geometry"
                                                                       else 110) * n}


# ------------------------------------------------------------------- exact --

def _inv3(m):
    """Cofactor inverse of (n,3,3)."""
    r0, r1, r2 = m.unbind(1)
    c = torch.stack([torch.linalg.cross(r1, r2), torch.linalg.cross(r2, r0),
                     torch.linalg.cross(r0, r1)], 2)
    return c / (r0 * torch.linalg.cross(r1, r2)).sum(1)[:, None, None]


def _refit(R, H, u):
    """UBI = (R H^-1)^-1 where both inverses exist, else as it was."""
    ok = torch.linalg.det(H) != 0
    eye = torch.eye(3, dtype=F64, device="cuda")
    UB = R @ _inv3(torch.where(ok[:, None, None], H, eye))
    ok = ok & (torch.linalg.det(UB) != 0)
    return torch.where(ok[:, None, None], _inv3(torch.where(ok[:, None, None], UB, eye)), u)


def _dense_round(u, gv, tol):
    """One score_and_refine of every UBI against every g: (UBIs, n, mean)."""
    out, ns, ds = [], [], []
    step = max(1, int(4e7 // len(gv)))
    for i in range(0, len(u), step):
        h = torch.einsum("mij,nj->mni", u[i:i + step], gv)
        ih = h.round()
        d = ((h - ih) ** 2).sum(2)
        w = (d < tol * tol).to(F64)
        hw = ih * w[..., None]
        R = torch.einsum("mni,nj->mji", hw, gv)
        H = torch.einsum("mni,mnj->mij", hw, ih)
        n = w.sum(1)
        out.append(_refit(R, H, u[i:i + step]))
        ns.append(n)
        ds.append((d * w).sum(1) / n.clamp(min=1))
    return torch.cat(out), torch.cat(ns), torch.cat(ds)


def _by_grain(v, off):
    """Sums of v's rows (last dimensions kept) over the grains' ranges."""
    return torch.segment_reduce(v.reshape(len(v), -1).contiguous(), "sum", offsets=off,
                                axis=0).reshape(-1, *v.shape[1:])


def _grain_sums(u, gv, grain, off, tol2):
    h = torch.einsum("nij,nj->ni", u[grain], gv)
    ih = h.round()
    d = ((h - ih) ** 2).sum(1)
    w = (d < tol2).to(F64)
    hw = ih * w[:, None]
    return (_by_grain(gv[:, :, None] * hw[:, None, :], off),
            _by_grain(ih[:, :, None] * hw[:, None, :], off), _by_grain(d * w, off),
            _by_grain(w, off))


def _translations_exact(x, iters):
    """The damped Gauss-Newton of refine_translations, all grains at once; the
    Jacobian by forward-mode differentiation of the residuals."""
    p, grain, off, u0 = x["p"], x["grain"], x["offsets"], x["ubis"]
    n = len(u0)
    t = torch.zeros((n, 3), dtype=F64, device="cuda")
    best = None
    lam = torch.full((n,), 1e-3, dtype=F64, device="cuda")
    for it in range(iters + 1):
        gv = _g_of(p, x["xyz"], x["omega"], t[grain])
        R, H, _, _ = _grain_sums(u0, gv, grain, off, 1.0)
        u1 = _refit(R, H, u0)
        h = torch.einsum("nij,nj->ni", u1[grain], gv)
        r = h - h.round()
        cost = _by_grain((r * r).sum(1), off)
        J = torch.stack([torch.func.jvp(
            lambda s: torch.einsum("nij,nj->ni", u1[grain],
                                   _g_of(p, x["xyz"], x["omega"], s[grain])),
            (t,), (torch.eye(3, dtype=F64, device="cuda")[j].expand(n, 3).contiguous(),))[1]
            for j in range(3)], 2)
        new = {"H": _by_grain(J.transpose(1, 2) @ J, off),
               "b": _by_grain((J * r[:, :, None]).sum(1), off), "t": t, "cost": cost}
        if best is None:
            best = new
        else:
            ok = cost < best["cost"]
            lam = torch.where(ok, (lam * 0.3).clamp(min=1e-9), (lam * 10).clamp(max=1e9))
            best = {k: torch.where(ok.view(-1, *[1] * (v.dim() - 1)), v, best[k])
                    for k, v in new.items()}
        A = best["H"] + torch.diag_embed(torch.diagonal(best["H"], dim1=1, dim2=2) * lam[:, None])
        t = best["t"] - (_inv3(A) @ best["b"][:, :, None])[:, :, 0]
    return {"t": best["t"], "cost": best["cost"], "n": None}


def _params_of(a, p):
    return dict(p, **{k: a[i] for i, k in enumerate(adjoint.PARAMS)})


def exact(case, seed):
    op = case["op"]
    if op in ("index", "assign") or (op == "score" and not case["sums"]):
        return None                 # whole numbers, or drlv2 over 2e11 pairs
    x = _inputs(case, seed)
    if op == "dropin":
        gv = _g_of(x["p"], x["xyz"], x["omega"], torch.zeros(3, dtype=F64, device="cuda"))
        u = x["ubis"]
        for _ in range(3):
            u, _, d = _dense_round(u, gv, 0.05)
        return {"gv": gv, "ubis": u, "n": None, "mean": d}
    if op == "score":
        u, gv = x["ubis"], x["gv"]
        if len(u) * len(gv) > 1.2e10:
            return None
        sums = []
        step = max(1, int(6e7 // len(gv)))
        for i in range(0, len(u), step):
            h = torch.einsum("mij,nj->mni", u[i:i + step], gv)
            d = ((h - h.round()) ** 2).sum(2)
            del h
            sums.append(torch.stack([torch.where(d < t * t, d, 0.0).sum(1) for t in TOLS], 1))
        return [None, torch.cat(sums)]
    if op == "refine_index":
        if case["iters"] * len(x["ubis"]) * len(x["gv"]) > 1.2e10:
            return None
        u = x["ubis"]
        for _ in range(case["iters"]):
            u, _, d = _dense_round(u, x["gv"], case["tol"])
        return {"ubis": u, "n": None, "mean": d}
    if op == "refine_grains":
        u = x["ubis"]
        for _ in range(case["iters"]):
            R, H, d, n = _grain_sums(u, x["gv"], x["grain"], x["offsets"], case["tol"] ** 2)
            u = _refit(R, H, u)
        return {"ubis": u, "n": None, "mean": d / n.clamp(min=1)}
    if op == "translations":
        return _translations_exact(x, case["iters"])
    if op in ("gradient", "projected"):
        p = x["p"]
        a = torch.tensor([float(dict(p, **ESTIMATE)[k]) for k in adjoint.PARAMS], dtype=F64,
                         device="cuda", requires_grad=True)
        q = _params_of(a, p)
        gv = _g_of(q, _lab(q, x["s"], x["f"]), x["omega"], _translation(q))
        if op == "gradient":
            u = x["ubis"].clone().requires_grad_(True)
        else:
            gd = gv.detach()
            u = _by_grain(x["hkl"][:, :, None] * gd[:, None, :], x["offsets"]) @ \
                _inv3(_by_grain(gd[:, :, None] * gd[:, None, :], x["offsets"]))
        value = 0.5 * ((torch.einsum("nij,nj->ni", u[x["grain"]], gv) - x["hkl"]) ** 2).sum()
        value.backward()
        return {"loss": value.detach(), "params": a.grad,
                "ubis": u.grad if op == "gradient" else u}
    p = x["p"]
    xyz, t = _lab(p, x["s"], x["f"]), _translation(p)
    if op == "gv":
        return _g_of(p, xyz, x["omega"], t)
    d, k, so, co, M = _k_of(p, xyz, x["omega"], t)
    v = k @ M
    out = torch.stack([torch.rad2deg(torch.atan2(torch.hypot(d[:, 1], d[:, 2]), d[:, 0])),
                       torch.rad2deg(torch.atan2(-d[:, 1], d[:, 2])), k.norm(dim=1),
                       co * v[:, 0] + so * v[:, 1], co * v[:, 1] - so * v[:, 0], v[:, 2]], 1)
    return {"xyz": xyz, "out": out}
