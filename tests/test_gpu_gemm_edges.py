"""The tensor-core GEMM at the edges of its tiles: token counts around the 16-column steps of an MMA and the 64-token plan
tile, row counts that leave half a tile or a single tile, the shortest K.  Bit for bit against the CPU checker; the fused
SwiGLU form against the CUDA-core form of the same entry point (itself checked in test_gpu_prefill.py)."""
import ctypes

import numpy as np
import pytest

from helpers import act_floats, dev, host, nan_f32, rand_q4

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 0, 129]


@pytest.fixture(params=[0, 1], ids=["exact", "fold"])
def L(request, lkb, orc):
    lkb.init(0)
    lkb.pf_gemm_arith(request.param)
    orc.set_gemm_fold(request.param)
    lkb.pf_gemm_config(1)
    yield lkb
    lkb.pf_gemm_config(-1)
    lkb.pf_gemm_arith(1)
    orc.set_gemm_fold(1)
    assert lkb.lib.lkb_pf_gemm_status() == 0


def _plan(rng):
    """Slots of 16 experts with COUNTS[e] slots each, in a random order: (slots' experts, off-ordered slots, plan tiles)."""
    idx = rng.permutation(np.repeat(np.arange(len(COUNTS)), COUNTS)).astype(np.int32)
    perm = np.argsort(idx, kind="stable").astype(np.int32)
    tiles, off = [], 0
    for e, c in enumerate(COUNTS):
        tiles += [[e, off + k, min(64, c - k), 0] for k in range(0, c, 64)]
        off += c
    return idx, perm, np.array(tiles, np.int32)


@pytest.mark.parametrize("m", [1, 16, 17, 48, 49, 64, 65])
@pytest.mark.parametrize("N,bpr", [(128, 8), (384, 16)])
def test_dense(L, orc, m, N, bpr):
    rng = np.random.default_rng(7 * m + N)
    qs, d = rand_q4(rng, N, bpr, "ref")
    aq, asc = orc.pf_quant_rows(act_floats(rng, m * bpr * 32).reshape(m, bpr * 32), bpr)
    o0 = rng.uniform(-1, 1, size=(m, N)).astype(np.float32)
    out = dev(o0)
    L.pf_gemm_dense(L.make_pf_gemm([(dev(qs), dev(d))], [N] * 3, N, bpr, dev(aq), dev(asc), ntok=m, out=out, out_ld=N, add=1))
    ref = orc.pf_gemm([(qs, d)], [N] * 3, N, bpr, aq, asc, ntok=m, out_init=o0, add=1)
    assert np.array_equal(host(out), ref)


@pytest.mark.parametrize("item,N,ends,m,bpr", [
    ((16, 256), 2176, (2176,) * 3, 161, 24), ((32, 128), 1152, (1152,) * 3, 497, 8), ((32, 256), 2176, (2176,) * 3, 305, 8),
    ((32, 256), 3072, (2048, 2560, 3072), 289, 16), ((48, 256), 3072, (2048, 2560, 3072), 401, 8), ((48, 256), 2176, (2176,) * 3, 593, 24),
    ((64, 256), 3072, (2048, 2560, 3072), 577, 8), ((64, 256), 6272, (6272,) * 3, 289, 8)])
def test_dense_items(L, orc, item, N, ends, m, bpr):
    """The items that a dense problem is cut into to fill the waves: each width and height, with the last token item short, a last row item of
    one tile where N has an odd number of them, and weight segments that end inside and between row items."""
    assert L.sm_count() != 148 or L.lib.lkb_debug_gemm_dense_item(m, N) == item[0] * 1000 + item[1]
    rng = np.random.default_rng(m + N)
    qs, d = rand_q4(rng, N, bpr, "ref")
    cut = [slice(a, b) for a, b in zip((0,) + ends[:2], ends) if b > a]
    aq, asc = orc.pf_quant_rows(act_floats(rng, m * bpr * 32).reshape(m, bpr * 32), bpr)
    out = nan_f32(m, N)
    L.pf_gemm_dense(L.make_pf_gemm([(dev(qs[c]), dev(d[c])) for c in cut], list(ends), N, bpr, dev(aq), dev(asc), ntok=m, out=out, out_ld=N))
    assert np.array_equal(host(out), orc.pf_gemm([(qs[c], d[c]) for c in cut], list(ends), N, bpr, aq, asc, ntok=m))


@pytest.mark.parametrize("N,bpr", [(128, 8), (384, 24), (2560, 8)])
def test_grouped(L, orc, N, bpr):
    rng = np.random.default_rng(N)
    idx, perm, tiles = _plan(rng)
    ns, E = idx.size, len(COUNTS)
    qs, d = rand_q4(rng, E * N, bpr, "ref")
    aq, asc = orc.pf_quant_rows(act_floats(rng, ns * bpr * 32).reshape(ns, bpr * 32), bpr)
    out = nan_f32(ns, N)
    g = L.make_pf_gemm([(dev(qs), dev(d))], [N] * 3, N, bpr, dev(aq), dev(asc), exp_stride=N * bpr, perm=dev(perm), tiles=dev(tiles),
                       ntiles=dev(np.array([len(tiles)], np.int32)), out=out, out_ld=N)
    L.pf_gemm_moe(g, len(tiles))
    ref = orc.pf_gemm([(qs, d)], [N] * 3, N, bpr, aq, asc, exp_stride=N * bpr, perm=perm, tiles=tiles, out_rows=ns)
    assert np.array_equal(host(out), ref)


def test_registered_workspace_is_left_alone(L, orc):
    """A caller that sizes and registers one as the header allows gets the same rows, and its buffer back untouched."""
    rng = np.random.default_rng(11)
    idx, perm, tiles = _plan(rng)
    ns, E, N, bpr = idx.size, len(COUNTS), 128, 8
    qs, d = rand_q4(rng, E * N, bpr, "ref")
    aq, asc = orc.pf_quant_rows(act_floats(rng, ns * bpr * 32).reshape(ns, bpr * 32), bpr)
    args = [dev(v) for v in (qs, d, aq, asc, perm, tiles, np.array([len(tiles)], np.int32))]
    buf = torch.full((L.pf_gemm_workspace_bytes(len(tiles), bpr * 32),), 0x5A, dtype=torch.uint8, device="cuda")
    got = []
    for ws in (None, buf):
        L.pf_gemm_set_workspace(ws)
        out = nan_f32(ns, N)
        L.pf_gemm_moe(L.make_pf_gemm([(args[0], args[1])], [N] * 3, N, bpr, args[2], args[3], exp_stride=N * bpr, perm=args[4],
                                     tiles=args[5], ntiles=args[6], out=out, out_ld=N), len(tiles))
        got.append(out)
    L.pf_gemm_set_workspace(None)
    assert torch.equal(got[0], got[1]) and bool(got[0].isfinite().all()) and bool((buf == 0x5A).all())


@pytest.mark.parametrize("I,bpr", [(64, 8), (192, 16), (256, 64)])
def test_swiglu(L, orc, I, bpr):
    rng = np.random.default_rng(I)
    idx, perm, tiles = _plan(rng)
    ns, E = idx.size, len(COUNTS)
    w = [tuple(dev(x) for x in rand_q4(rng, E * I, bpr, "ref")) for _ in range(2)]
    x = act_floats(rng, ns * bpr * 32).reshape(ns, bpr * 32)
    x[5] = 0.0                                                       # a row of all-zero blocks
    aq, asc = (dev(v) for v in orc.pf_quant_rows(x, bpr))
    scale = dev(rng.uniform(0.01, 0.05, size=ns).astype(np.float32))
    dperm, dtiles, dnt = dev(perm), dev(tiles), dev(np.array([len(tiles)], np.int32))
    got = []
    for cfg in (0, 1):
        L.pf_gemm_config(cfg)
        oqs, osc = torch.full((ns, I), 0x5A, dtype=torch.int8, device="cuda"), nan_f32(ns, I // 32, 2)
        L.pf_gemm_swiglu(L.make_pf_gemm(w, [I] * 3, I, bpr, aq, asc, exp_stride=I * bpr, perm=dperm, tiles=dtiles, ntiles=dnt,
                                        scale=scale, oqs=oqs, osc=osc, okb=I // 32), len(tiles))
        got.append((oqs, osc))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert int(got[1][0].float().abs().max()) > 0


def _past(a, off):
    """The array's bytes on the device, `off` bytes past an aligned address."""
    raw = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
    buf = torch.zeros(raw.size + off, dtype=torch.uint8, device="cuda")
    buf[off:] = torch.from_numpy(raw.copy()).cuda()
    return buf[off:]


@pytest.mark.parametrize("off", [0, 8])
def test_scale_planes_on_8_byte_boundaries(L, orc, off):
    """Every entry point of the tensor-core form takes weight-scale planes that start on an 8-byte boundary: dense with three
    segments, grouped with row targets, SwiGLU from planar rows and from packed ones (192 rows: half a tile is missing)."""
    rng = np.random.default_rng(5 + off)
    N, bpr, m = 640, 16, 70
    qs, d = rand_q4(rng, N, bpr, "ref")
    aq, asc = orc.pf_quant_rows(act_floats(rng, m * bpr * 32).reshape(m, bpr * 32), bpr)
    cut, ends = [slice(0, 256), slice(256, 384), slice(384, N)], [256, 384, N]
    out = nan_f32(m, N)
    L.pf_gemm_dense(L.make_pf_gemm([(dev(qs[c]), _past(d[c], off)) for c in cut], ends, N, bpr, dev(aq), dev(asc), ntok=m, out=out, out_ld=N))
    assert np.array_equal(host(out), orc.pf_gemm([(qs[c], d[c]) for c in cut], ends, N, bpr, aq, asc, ntok=m))

    idx, perm, tiles = _plan(rng)
    ns, E, I = idx.size, len(COUNTS), 192
    dperm, dtiles, dnt = dev(perm), dev(tiles), dev(np.array([len(tiles)], np.int32))
    aq, asc = orc.pf_quant_rows(act_floats(rng, ns * bpr * 32).reshape(ns, bpr * 32), bpr)
    daq, dasc = dev(aq), dev(asc)
    plan = dict(perm=dperm, tiles=dtiles, ntiles=dnt)
    qs, d = rand_q4(rng, E * 256, bpr, "ref")
    order = torch.from_numpy(rng.permutation(ns).astype(np.int64)).cuda()      # row s of the result goes to row order[s] of the buffer
    back = nan_f32(ns, 256)
    rows = back.data_ptr() + order * 1024
    g = L.make_pf_gemm([(dev(qs), _past(d, off))], [256] * 3, 256, bpr, daq, dasc, exp_stride=256 * bpr, out=back, out_ld=256, **plan)
    L.pf_gemm_moe_rows(g, len(tiles), rows)
    ref = orc.pf_gemm([(qs, d)], [256] * 3, 256, bpr, aq, asc, exp_stride=256 * bpr, perm=perm, tiles=tiles, out_rows=ns)
    assert np.array_equal(host(back)[host(order)], ref)

    w = [rand_q4(rng, E * I, bpr, "ref") for _ in range(2)]
    pitch = bpr * 40 + 16
    packed = torch.full((ns, pitch), 0x5A, dtype=torch.uint8, device="cuda")
    packed[:, :bpr * 32] = daq.view(torch.uint8)
    packed[:, bpr * 32:bpr * 40] = dasc.reshape(ns, bpr * 2).view(torch.uint8)
    got = []
    for form, planes_off in ((0, 0), (1, off), (2, off)):                       # the CUDA-core form; planar; packed
        L.pf_gemm_config(min(form, 1))
        oqs, osc = torch.full((ns, I), 0x5A, dtype=torch.int8, device="cuda"), nan_f32(ns, I // 32, 2)
        g = L.make_pf_gemm([(dev(q), _past(s, planes_off)) for q, s in w], [I] * 3, I, bpr, packed if form == 2 else daq, dasc,
                           exp_stride=I * bpr, oqs=oqs, osc=osc, okb=I // 32, **plan)
        if form == 2:
            L.pf_gemm_swiglu_packed(g, len(tiles), pitch)
        else:
            L.pf_gemm_swiglu(g, len(tiles))
        got.append((oqs, osc))
    for a, b in got[1:]:
        assert torch.equal(got[0][0], a) and torch.equal(got[0][1], b)


@pytest.mark.parametrize("cfg", [-1, 0])
def test_misaligned_planes_are_refused(L, orc, cfg):
    """Planes off the boundary that both forms' loads need are an error of the call, not of the device."""
    L.pf_gemm_config(cfg)
    rng = np.random.default_rng(3)
    N, bpr, m = 128, 8, 5
    qs, d = rand_q4(rng, N, bpr, "ref")
    aq, asc = orc.pf_quant_rows(act_floats(rng, m * bpr * 32).reshape(m, bpr * 32), bpr)
    buf = torch.zeros(m * N * 4 + 8, dtype=torch.uint8, device="cuda")
    offs = {"qs": 8, "d": 1, "aqs": 8, "asc": 4, "out": 2}
    for wrong in [None, *offs]:
        o = {k: v if k == wrong else 0 for k, v in offs.items()}
        keep = [_past(qs, o["qs"]), _past(d, o["d"]), _past(aq, o["aqs"]), _past(asc, o["asc"]), buf[o["out"]:]]
        g = L.make_pf_gemm([(keep[0], keep[1])], [N] * 3, N, bpr, keep[2], keep[3], ntok=m, out=keep[4], out_ld=N)
        assert L.lib.lkb_pf_gemm_dense(ctypes.byref(g), None) == (0 if wrong is None else -10001), wrong
    torch.cuda.synchronize()
