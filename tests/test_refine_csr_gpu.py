"""Per-grain CSR refinement (persistent kernel, CUDA graph, plain baseline)
against the oracle's loop of score_and_refine calls over each grain's peaks.

n per grain is exact; refined UBIs agree to the rounding of the summation
order (UBI_RTOL, as the other refinement tests); mean drlv2 to 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UBI_RTOL = 1e-11
DRLV2_RTOL = 1e-12


@pytest.fixture(scope="module")
def grains():
    from imaged11_b200 import synth
    rng = np.random.default_rng(41)
    ng = 120
    counts = np.exp(rng.uniform(np.log(20), np.log(2000), ng)).astype(int)
    ps = synth.simulate(ng, "Ti_hcp", gmax=2.2, seed=42, noise_frac=0.0,
                        per_grain_counts=counts)
    idx, off = ps.grain_offsets()
    gv = ps.gv[idx]
    u0 = synth.perturb_ubis(ps.ubis, 0.2, 0.002, rng)
    # a few edge cases: an empty grain, a grain with 2 peaks (singular H)
    off = np.concatenate([off, [off[-1], off[-1] + 2]])
    gv = np.concatenate([gv, gv[:2]])
    u0 = np.concatenate([u0, ps.ubis[:2]])
    return gv, off, u0


def _check(u, npk, mean, ref_u, ref_n, ref_m):
    assert np.array_equal(npk, ref_n)
    assert np.all(np.abs(mean - ref_m) <= DRLV2_RTOL * np.abs(ref_m))
    scale = np.abs(ref_u).reshape(len(ref_u), -1).max(1)
    err = np.abs(u - ref_u).reshape(len(ref_u), -1).max(1)
    assert np.all(err <= UBI_RTOL * scale), err.max()


@pytest.mark.parametrize("persistent", [True, False])
def test_refine_csr_matches_oracle(grains, oracle, persistent, cuda):
    from imaged11_b200 import batch
    gv, off, u0 = grains
    ref_u, ref_n, ref_m = oracle.refine_csr(u0, gv, off, 0.05, 5)
    gs = batch.GrainSet(gv, off, u0)
    u, npk, mean = gs.refine(0.05, 5, persistent=persistent)
    _check(u.cpu().numpy(), npk.cpu().numpy(), mean.cpu().numpy(), ref_u, ref_n, ref_m)


def test_refine_csr_graph_replay(grains, oracle, cuda):
    import torch
    from imaged11_b200 import batch
    gv, off, u0 = grains
    gs = batch.GrainSet(gv, off, u0)
    graph = gs.capture(0.05, 2)
    assert np.array_equal(gs.ubis.cpu().numpy().reshape(-1, 3, 3), u0)
    graph.replay()
    graph.replay()                    # 2 + 2 rounds
    torch.cuda.synchronize()
    ref_u, ref_n, ref_m = oracle.refine_csr(u0, gv, off, 0.05, 4)
    _check(gs.ubis.cpu().numpy().reshape(-1, 3, 3), gs.npk.cpu().numpy(),
           gs.mean.cpu().numpy(), ref_u, ref_n, ref_m)


def test_refine_csr_deterministic(grains, cuda):
    from imaged11_b200 import batch
    gv, off, u0 = grains
    a = batch.GrainSet(gv, off, u0).refine(0.05, 3)[0].cpu().numpy()
    b = batch.GrainSet(gv, off, u0).refine(0.05, 3)[0].cpu().numpy()
    assert np.array_equal(a, b)


def test_refine_csr_compensated_fp32(grains, oracle, cuda):
    """The compensated-FP32 variant: FP32 screening inside the proven band
    with an FP64 recheck (peak membership exact), normal equations summed as
    compensated FP32 pairs (about FP64 accuracy), FP64 3x3 solves.  UBIs to
    1e-9 relative."""
    from imaged11_b200 import batch
    gv, off, u0 = grains
    ref_u, ref_n, ref_m = oracle.refine_csr(u0, gv, off, 0.05, 5)
    gs = batch.GrainSet(gv, off, u0)
    u, npk, mean = gs.refine(0.05, 5, precision="f32c")
    u, npk, mean = u.cpu().numpy(), npk.cpu().numpy(), mean.cpu().numpy()
    assert np.array_equal(npk, ref_n)
    scale = np.abs(ref_u).reshape(len(ref_u), -1).max(1)
    err = np.abs(u - ref_u).reshape(len(ref_u), -1).max(1)
    assert np.all(err <= 1e-9 * scale), err.max()
    # the mean drlv2 is a sum of FP32 per-peak values (each within the
    # screening band of the exact one): about 1e-6 relative here
    assert np.all(np.abs(mean - ref_m) <= 1e-4 * np.abs(ref_m) + 1e-18)


@pytest.mark.parametrize("threads", [32, 64, 128, 256, 512])
@pytest.mark.parametrize("ordered", [True, False])
def test_refine_csr_more_grains_than_ctas(oracle, threads, ordered, cuda):
    """More grains than resident CTAs: grains on both sides of the size one warp
    takes, empty and tiny ones, in order of size and not (a large grain met by a
    warp working alone): the oracle's rounds, and the same bits in both orders."""
    import torch
    from imaged11_b200 import batch, synth
    from imaged11_b200._lib import lib, check
    rng = np.random.default_rng(43)
    counts = rng.integers(20, 41, 5200)
    counts[:12] = [0, 1, 2, 31, 32, 33, 767, 768, 769, 1537, 2000, 770]
    rng.shuffle(counts)
    gv, off, ubis = synth.grain_gvectors(counts, "Ti_hcp", rng)
    u0 = synth.perturb_ubis(ubis, 0.2, 0.002, rng)
    ref_u, ref_n, ref_m = oracle.refine_csr(u0, gv, off, 0.05, 3)
    gs = batch.GrainSet(gv, off, u0, threads=threads)
    u, npk, mean = gs.refine(0.05, 3)
    u = u.cpu().numpy()
    if not ordered:
        other = torch.tensor(u0, device=cuda).contiguous()
        check(lib.id11b_dev_refine_csr(other.data_ptr(), gs.gv.data_ptr(), gs.offsets.data_ptr(),
                                       None, gs.ngrains, 0.05, 3, 1, threads, npk.data_ptr(),
                                       mean.data_ptr(), gs.ws.data_ptr(), gs.ws.numel(), None),
              "refine_csr")
        torch.cuda.synchronize()
        assert np.array_equal(other.cpu().numpy(), u)
    big = ref_n > 3     # (up to three peaks the normal matrix is singular to rounding)
    _check(u[big], npk.cpu().numpy()[big], mean.cpu().numpy()[big], ref_u[big], ref_n[big],
           ref_m[big])
    assert np.array_equal(npk.cpu().numpy(), ref_n)


@pytest.mark.parametrize("threads", [32, 128])
def test_refine_csr_grain_alone_and_among_many(threads, cuda):
    """The same grains in a call of 16 and among 5,200: the same peaks, and the same
    bits where the sums' order is the same -- with 32 threads always, with more for
    the grains that a whole CTA refines in both (above 768 peaks).  The others
    differ by the order of their sums."""
    from imaged11_b200 import batch, synth
    rng = np.random.default_rng(45)
    counts = rng.integers(20, 41, 5200)
    counts[:16] = [20, 31, 32, 33, 64, 127, 128, 129, 500, 767, 768, 769, 800, 1537, 2000, 2600]
    gv, off, ubis = synth.grain_gvectors(counts, "Ti_hcp", rng)
    u0 = synth.perturb_ubis(ubis, 0.2, 0.002, rng)
    many = [t.cpu().numpy()[:16] for t in batch.GrainSet(gv, off, u0, threads=threads).refine(0.05, 3)]
    few = [t.cpu().numpy() for t in
           batch.GrainSet(gv[:off[16]], off[:17], u0[:16], threads=threads).refine(0.05, 3)]
    assert np.array_equal(many[1], few[1])
    same = (counts[:16] > 768) | (threads == 32)
    assert np.array_equal(many[0][same], few[0][same])
    assert np.array_equal(many[2][same], few[2][same])
    scale = np.abs(few[0]).reshape(16, -1).max(1)
    assert np.all(np.abs(many[0] - few[0]).reshape(16, -1).max(1) <= UBI_RTOL * scale)


@pytest.mark.parametrize("ordered", [True, False])
def test_compensated_more_grains_than_ctas(oracle, ordered, cuda):
    """The same for the compensated-FP32 variant, whose one-warp grains end at 384
    peaks; grains of 20 peaks and more, with that variant's tolerances above."""
    import torch
    from imaged11_b200 import batch, synth
    from imaged11_b200._lib import lib, check
    rng = np.random.default_rng(44)
    counts = rng.integers(20, 41, 5200)
    counts[:9] = [0, 1, 31, 383, 384, 385, 769, 2000, 386]
    rng.shuffle(counts)
    gv, off, ubis = synth.grain_gvectors(counts, "Ti_hcp", rng)
    u0 = synth.perturb_ubis(ubis, 0.2, 0.002, rng)
    ref_u, ref_n, ref_m = oracle.refine_csr(u0, gv, off, 0.05, 3)
    gs = batch.GrainSet(gv, off, u0)
    u, npk, mean = gs.refine(0.05, 3, precision="f32c")
    if not ordered:
        other = torch.tensor(u0, device=cuda).contiguous()
        check(lib.id11b_dev_refine_csr_f32c(other.data_ptr(), gs.gv.data_ptr(),
                                            gs.offsets.data_ptr(), None, gs.ngrains, 0.05, 3,
                                            gs.gmax, npk.data_ptr(), mean.data_ptr(),
                                            gs.ws.data_ptr(), gs.ws.numel(), None), "f32c")
        torch.cuda.synchronize()
        assert torch.equal(other.view(-1, 3, 3), u)
    big = counts >= 20
    u, npk, mean = u.cpu().numpy()[big], npk.cpu().numpy()[big], mean.cpu().numpy()[big]
    assert np.array_equal(npk, ref_n[big])
    scale = np.abs(ref_u[big]).reshape(len(u), -1).max(1)
    assert np.all(np.abs(u - ref_u[big]).reshape(len(u), -1).max(1) <= 1e-9 * scale)
    assert np.all(np.abs(mean - ref_m[big]) <= 1e-4 * np.abs(ref_m[big]) + 1e-18)


@pytest.mark.parametrize("ngrains,edge", [(1000, 384), (5200, 1024)])
def test_compensated_one_warp_sizes(oracle, ngrains, edge, cuda):
    """The compensated variant on both sides of the size that one warp takes, with
    few grains per CTA and with many; that variant's tolerances above."""
    from imaged11_b200 import batch, synth
    rng = np.random.default_rng(47)
    counts = rng.integers(20, 41, ngrains)
    counts[:8] = [edge - 1, edge, edge + 1, edge + 31, edge + 128, 1800, 127, 128]
    rng.shuffle(counts)
    gv, off, ubis = synth.grain_gvectors(counts, "Ti_hcp", rng)
    u0 = synth.perturb_ubis(ubis, 0.2, 0.002, rng)
    ref_u, ref_n, ref_m = oracle.refine_csr(u0, gv, off, 0.05, 3)
    u, npk, mean = (t.cpu().numpy() for t in
                    batch.GrainSet(gv, off, u0).refine(0.05, 3, precision="f32c"))
    assert np.array_equal(npk, ref_n)
    scale = np.abs(ref_u).reshape(ngrains, -1).max(1)
    assert np.all(np.abs(u - ref_u).reshape(ngrains, -1).max(1) <= 1e-9 * scale)
    assert np.all(np.abs(mean - ref_m) <= 1e-4 * np.abs(ref_m) + 1e-18)


def test_refine_csr_grain_longer_than_2_31(oracle, cuda):
    """One grain of 2^31 + 300 peaks (its length, and a peak's index in it, need 64
    bits): its peaks are at the start, around 2^30 and 2^31 and at the end, NaN
    between them."""
    import torch
    from imaged11_b200 import batch, synth
    n = (1 << 31) + 300
    if torch.cuda.mem_get_info(cuda)[0] < 3 * 8 * n + (4 << 30):
        pytest.skip("51.5 GB of g")
    rng = np.random.default_rng(46)
    gv, off, ubis = synth.grain_gvectors(np.array([900]), "Ti_hcp", rng)
    u0 = synth.perturb_ubis(ubis, 0.2, 0.002, rng)
    where = np.concatenate([np.arange(100), (1 << 30) - 250 + np.arange(500),
                            (1 << 31) - 150 + np.arange(250), n - 50 + np.arange(50)])
    g = torch.full((n, 3), float("nan"), dtype=torch.float64, device=cuda)
    g[torch.as_tensor(where, device=cuda)] = torch.as_tensor(gv, device=cuda)
    u, npk, mean = batch.GrainSet(g, np.array([0, n]), u0, threads=512).refine(0.05, 2)
    ref_u, ref_n, ref_m = oracle.refine_csr(u0, gv, off, 0.05, 2)
    _check(u.cpu().numpy(), npk.cpu().numpy(), mean.cpu().numpy(), ref_u, ref_n, ref_m)
