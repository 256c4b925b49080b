"""The few-token form of the GEMM beyond its first 47 tokens, at its edges: plan tiles cut into parts of 16 or 32 tokens, the MMA's groups of
eight tokens, one stage of K and an odd number, more items than the stages hold, more parts than its list holds, dense chunks of every width, last
waves cut into halves and quarters of rows, alone and behind whole ones.
Bit for bit against the oracle; the fused SwiGLU form against the CUDA-core form (itself checked in test_gpu_prefill.py)."""
import ctypes

import numpy as np
import pytest

from helpers import act_floats, dev, host, nan_f32, rand_q4

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MAX_TILES = 90
COUNTS = {16: [1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 48, 0, 64], 32: [24, 25, 31, 32, 33, 40, 63, 64, 65, 129, 1, 200, 128]}      # 281 and 835 slots


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


def _plan(rng, counts, tile=64):
    perm = np.argsort(rng.permutation(np.repeat(np.arange(len(counts)), counts)), kind="stable").astype(np.int32)
    tiles, off = [], 0
    for e, c in enumerate(counts):
        tiles += [[e, off + k, min(tile, c - k), 0] for k in range(0, c, tile)]
        off += c
    return perm, np.array(tiles, np.int32)


def _width(L, g, max_tiles=MAX_TILES):
    return L.lib.lkb_debug_gemm_few_width(ctypes.byref(g), max_tiles, L.sm_count())


@pytest.mark.parametrize("width", [16, 32])
@pytest.mark.parametrize("N,bpr", [(256, 8), (1024, 24), (1280, 8), (2048, 8)])       # 22 to 256 items on 148 SMs
def test_grouped(L, orc, N, bpr, width):
    rng = np.random.default_rng(N + width)
    perm, tiles = _plan(rng, COUNTS[width])
    ns, E = perm.size, len(COUNTS[width])
    qs, d = rand_q4(rng, E * N, bpr, "ref")
    aq, asc = orc.pf_quant_rows(act_floats(rng, ns * bpr * 32).reshape(ns, bpr * 32), bpr)
    out = nan_f32(ns, N)
    g = L.make_pf_gemm([(dev(qs), dev(d))], [N] * 3, N, bpr, dev(aq), dev(asc), ntok=ns, exp_stride=N * bpr, perm=dev(perm), tiles=dev(tiles),
                       ntiles=dev(np.array([len(tiles)], np.int32)), out=out, out_ld=N)
    assert _width(L, g) == width
    L.pf_gemm_moe(g, MAX_TILES)
    ref = orc.pf_gemm([(qs, d)], [N] * 3, N, bpr, aq, asc, exp_stride=N * bpr, perm=perm, tiles=tiles, out_rows=ns)
    assert np.array_equal(host(out), ref)


def test_more_parts_than_are_listed(L, orc):
    """2100 tiles of one token: the parts are walked instead, empty ones too.  (Slots stated low, as only the choice of the form reads them.)"""
    rng = np.random.default_rng(5)
    N, bpr, E, ns = 256, 8, 3, 2100
    perm, tiles = _plan(rng, [ns // E] * E, tile=1)
    qs, d = rand_q4(rng, E * N, bpr, "ref")
    aq, asc = orc.pf_quant_rows(act_floats(rng, ns * bpr * 32).reshape(ns, bpr * 32), bpr)
    out = nan_f32(ns, N)
    g = L.make_pf_gemm([(dev(qs), dev(d))], [N] * 3, N, bpr, dev(aq), dev(asc), ntok=300, exp_stride=N * bpr, perm=dev(perm), tiles=dev(tiles),
                       ntiles=dev(np.array([ns], np.int32)), out=out, out_ld=N)
    assert _width(L, g, ns) == 16
    L.pf_gemm_moe(g, ns)
    ref = orc.pf_gemm([(qs, d)], [N] * 3, N, bpr, aq, asc, exp_stride=N * bpr, perm=perm, tiles=tiles, out_rows=ns)
    assert np.array_equal(host(out), ref)


def test_more_parts_than_are_listed_swiglu(L, orc):
    """As above with three row tiles, so that a block meets empty parts between others."""
    rng = np.random.default_rng(6)
    I, bpr, E, ns = 384, 8, 3, 2100
    perm, tiles = _plan(rng, [ns // E] * E, tile=1)
    w = [tuple(dev(x) for x in rand_q4(rng, E * I, bpr, "ref")) for _ in range(2)]
    aq, asc = (dev(v) for v in orc.pf_quant_rows(act_floats(rng, ns * bpr * 32).reshape(ns, bpr * 32), bpr))
    dperm, dtiles, dnt = dev(perm), dev(tiles), dev(np.array([ns], np.int32))
    got = []
    for cfg in (0, -1):
        L.pf_gemm_config(cfg)
        oqs, osc = torch.full((ns, I), 0x5A, dtype=torch.int8, device="cuda"), nan_f32(ns, I // 32, 2)
        g = L.make_pf_gemm(w, [I] * 3, I, bpr, aq, asc, ntok=300, exp_stride=I * bpr, perm=dperm, tiles=dtiles, ntiles=dnt, oqs=oqs, osc=osc, okb=I // 32)
        assert _width(L, g, ns) == 16
        L.pf_gemm_swiglu(g, ns)
        got.append((oqs, osc))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1].view(torch.int32), got[1][1].view(torch.int32))


@pytest.mark.parametrize("width", [16, 32])
@pytest.mark.parametrize("I,bpr", [(128, 8), (384, 40), (640, 8), (1024, 8)])          # 22 to 256 items
@pytest.mark.parametrize("off", [0, 1])
def test_swiglu(L, orc, I, bpr, width, off):
    """off: the quants' plane starts on an odd byte, which this form's stores cannot take; the call is served all the same."""
    rng = np.random.default_rng(I + width)
    perm, tiles = _plan(rng, COUNTS[width])
    ns, E = perm.size, len(COUNTS[width])
    w = [tuple(dev(x) for x in rand_q4(rng, E * I, bpr, "ref")) for _ in range(2)]
    m = (ns + 3) // 4
    x = act_floats(rng, m * bpr * 32).reshape(m, bpr * 32)
    x[5], x[7, 32:64], x[9, 3] = 0.0, 3e4, np.nan                     # all-zero blocks, large ones, a NaN
    aq, asc = (dev(v) for v in orc.pf_quant_rows(x, bpr))
    scale = dev(rng.uniform(0.01, 0.05, size=m).astype(np.float32))
    dperm, dtiles, dnt = dev(perm), dev(tiles), dev(np.array([len(tiles)], np.int32))
    got = []
    for cfg in (0, -1):
        L.pf_gemm_config(cfg)
        oqs, osc = torch.full((ns * I + 16,), 0x5A, dtype=torch.int8, device="cuda"), nan_f32(ns, I // 32, 2)
        g = L.make_pf_gemm(w, [I] * 3, I, bpr, aq, asc, ntok=ns, exp_stride=I * bpr, perm=dperm, tiles=dtiles, ntiles=dnt,
                           a_shift=2, scale=scale, oqs=oqs[off:], osc=osc, okb=I // 32)
        assert _width(L, g) == width
        L.pf_gemm_swiglu(g, MAX_TILES)
        got.append((oqs, osc))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1].view(torch.int32), got[1][1].view(torch.int32))
    assert int(got[1][0].float().abs().max()) > 0 and torch.isfinite(got[1][1][:, 0, 0]).any()


@pytest.mark.parametrize("m,N,ends,bpr,width", [(5, 256, (256,) * 3, 64, 8), (37, 1024, (512, 640, 1024), 40, 8), (130, 2048, (2048,) * 3, 64, 8), (64, 2048, (1024, 1152, 2048), 64, 8), (3, 38912, (38912,) * 3, 8, 8), (160, 2304, (2304,) * 3, 64, 16), (251, 2048, (2048,) * 3, 64, 16),
                                                (90, 6144, (6144,) * 3, 64, 16), (97, 6144, (6144,) * 3, 64, 24), (143, 6144, (2048, 4096, 6144), 64, 24), (300, 2048, (2048,) * 3, 64, 24), (145, 6144, (6144,) * 3, 64, 0), (37, 256, (256,) * 3, 8, 0)])
def test_dense(L, orc, m, N, ends, bpr, width):
    rng = np.random.default_rng(7 * m + N)
    qs, d = rand_q4(rng, N, bpr, "ref")
    cut = [slice(a, b) for a, b in zip((0,) + ends[:2], ends) if b > a]
    aq, asc = orc.pf_quant_rows(act_floats(rng, m * bpr * 32).reshape(m, bpr * 32), bpr)
    o0 = rng.uniform(-1, 1, size=(m, N)).astype(np.float32)
    out = dev(o0)
    g = L.make_pf_gemm([(dev(qs[c]), dev(d[c])) for c in cut], list(ends), N, bpr, dev(aq), dev(asc), ntok=m, out=out, out_ld=N, add=1)
    assert L.sm_count() != 148 or _width(L, g) == width
    L.pf_gemm_dense(g)
    ref = orc.pf_gemm([(qs[c], d[c]) for c in cut], list(ends), N, bpr, aq, asc, ntok=m, out_init=o0, add=1)
    assert np.array_equal(host(out), ref)
