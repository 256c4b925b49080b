"""The few-token form of the GEMM (what the launchers take by themselves for short prompts) at its edges: token counts around its
chunks of eight and the row gathers' groups of four, tiles of more than one chunk, the shortest K and an odd number of stage
pairs, one and several items a CTA, weight segments, residual add.  Bit for bit against the CPU checker; the fused SwiGLU form
against the CUDA-core form (itself checked in test_gpu_prefill.py)."""
import ctypes

import numpy as np
import pytest

from helpers import act_floats, dev, host, nan_f32, rand_q4

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MAX_TILES = 66                                          # what a caller passes for a few tokens: one tile per expert, one per 64 slots
COUNTS = [1, 2, 3, 4, 5, 7, 8, 9, 0, 12, 16, 17, 38, 66]   # 188 slots: the most this form takes


@pytest.fixture(params=[0, 1], ids=["exact", "fold"])
def L(request, lkb, orc):
    lkb.init(0)
    lkb.pf_gemm_arith(request.param)
    orc.set_gemm_fold(request.param)
    lkb.pf_gemm_config(-1)
    yield lkb
    lkb.pf_gemm_config(-1)
    lkb.pf_gemm_arith(1)
    orc.set_gemm_fold(1)
    assert lkb.lib.lkb_pf_gemm_status() == 0


def _plan(rng):
    idx = rng.permutation(np.repeat(np.arange(len(COUNTS)), COUNTS)).astype(np.int32)
    perm = np.argsort(idx, kind="stable").astype(np.int32)
    tiles, off = [], 0
    for e, c in enumerate(COUNTS):
        tiles += [[e, off + k, min(64, c - k), 0] for k in range(0, c, 64)]
        off += c
    assert perm.size == 188
    return perm, np.array(tiles, np.int32)


def _takes(L, g, max_tiles=MAX_TILES):
    return L.lib.lkb_debug_gemm_few_better(ctypes.byref(g), max_tiles) == 1


@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("N,ends,bpr", [(256, (256,) * 3, 8), (1024, (512, 640, 1024), 24)])
def test_dense(L, orc, m, N, ends, bpr):
    rng = np.random.default_rng(7 * m + N)
    qs, d = rand_q4(rng, N, bpr, "ref")
    cut = [slice(a, b) for a, b in zip((0,) + ends[:2], ends) if b > a]
    aq, asc = orc.pf_quant_rows(act_floats(rng, m * bpr * 32).reshape(m, bpr * 32), bpr)
    o0 = rng.uniform(-1, 1, size=(m, N)).astype(np.float32)
    out = dev(o0)
    g = L.make_pf_gemm([(dev(qs[c]), dev(d[c])) for c in cut], list(ends), N, bpr, dev(aq), dev(asc), ntok=m, out=out, out_ld=N, add=1)
    assert _takes(L, g)
    L.pf_gemm_dense(g)
    ref = orc.pf_gemm([(qs[c], d[c]) for c in cut], list(ends), N, bpr, aq, asc, ntok=m, out_init=o0, add=1)
    assert np.array_equal(host(out), ref)


@pytest.mark.parametrize("N,bpr", [(256, 8), (2048, 24)])
def test_grouped(L, orc, N, bpr):
    rng = np.random.default_rng(N)
    perm, tiles = _plan(rng)
    ns, E = perm.size, len(COUNTS)
    qs, d = rand_q4(rng, E * N, bpr, "ref")
    aq, asc = orc.pf_quant_rows(act_floats(rng, ns * bpr * 32).reshape(ns, bpr * 32), bpr)
    out = nan_f32(ns, N)
    g = L.make_pf_gemm([(dev(qs), dev(d))], [N] * 3, N, bpr, dev(aq), dev(asc), ntok=ns, exp_stride=N * bpr, perm=dev(perm), tiles=dev(tiles),
                       ntiles=dev(np.array([len(tiles)], np.int32)), out=out, out_ld=N)
    assert _takes(L, g)
    L.pf_gemm_moe(g, MAX_TILES)
    ref = orc.pf_gemm([(qs, d)], [N] * 3, N, bpr, aq, asc, exp_stride=N * bpr, perm=perm, tiles=tiles, out_rows=ns)
    assert np.array_equal(host(out), ref)


@pytest.mark.parametrize("I,bpr", [(128, 8), (384, 24), (1536, 64)])
def test_swiglu(L, orc, I, bpr):
    rng = np.random.default_rng(I)
    perm, tiles = _plan(rng)
    ns, E = perm.size, len(COUNTS)
    w = [tuple(dev(x) for x in rand_q4(rng, E * I, bpr, "ref")) for _ in range(2)]
    m = (ns + 3) // 4
    x = act_floats(rng, m * bpr * 32).reshape(m, bpr * 32)
    x[5] = 0.0                                                       # a row of all-zero blocks
    aq, asc = (dev(v) for v in orc.pf_quant_rows(x, bpr))
    scale = dev(rng.uniform(0.01, 0.05, size=m).astype(np.float32))
    dperm, dtiles, dnt = dev(perm), dev(tiles), dev(np.array([len(tiles)], np.int32))
    got = []
    for cfg in (0, -1):
        L.pf_gemm_config(cfg)
        oqs, osc = torch.full((ns, I), 0x5A, dtype=torch.int8, device="cuda"), nan_f32(ns, I // 32, 2)
        g = L.make_pf_gemm(w, [I] * 3, I, bpr, aq, asc, ntok=ns, exp_stride=I * bpr, perm=dperm, tiles=dtiles, ntiles=dnt,
                           a_shift=2, scale=scale, oqs=oqs, osc=osc, okb=I // 32)
        assert _takes(L, g)
        L.pf_gemm_swiglu(g, MAX_TILES)
        got.append((oqs, osc))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert int(got[1][0].float().abs().max()) > 0


@pytest.mark.parametrize("m", [3, 20, 60])
def test_short_stack_replays_from_a_graph(lkb, m):
    """A short chunk through the MoE stack (few-token GEMMs up to 47 tokens, clustered router): a captured step replays to the
    residual of an eager one, bit for bit."""
    import importlib
    lkb.init(0)
    ps = importlib.import_module("lfm2-ampere_b200.prefill").PrefillStack(importlib.import_module("lfm2-ampere_b200.synth").make_model(2, seed=41, zipf_s=0.7), m)
    x0 = torch.randn(m, 2048, device="cuda", generator=torch.Generator("cuda").manual_seed(9))
    ps.X.copy_(x0); ps.step(); torch.cuda.synchronize()
    ref = ps.X.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ps.step()
    for _ in range(2):
        ps.X.copy_(x0); g.replay(); torch.cuda.synchronize()
        assert torch.isfinite(ref).all() and torch.equal(ps.X, ref)
