"""The fused SwiGLU form on consecutive tokens (no routing): each width of the few-token form's items, last waves cut and whole, and the tensor-core
form's, bit for bit against the CUDA-core form (itself checked in test_gpu_prefill.py)."""
import ctypes

import pytest

from helpers import act_floats, dev, nan_f32, rand_q4

np = pytest.importorskip("numpy")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fold", [0, 1], ids=["exact", "fold"])
@pytest.mark.parametrize("m,I,bpr,width", [(1, 128, 8, 8), (4, 384, 24, 8), (5, 128, 64, 8), (37, 1536, 64, 8), (100, 1536, 16, None), (130, 1536, 64, 16), (200, 1536, 64, 24), (203, 640, 24, None), (300, 1536, 64, 0), (509, 192, 8, 0)])
def test_dense_swiglu(lkb, orc, m, I, bpr, width, fold):
    lkb.init(0)
    rng = np.random.default_rng(m + I)
    w = [tuple(dev(x) for x in rand_q4(rng, I, bpr, "ref")) for _ in range(2)]
    x = act_floats(rng, m * bpr * 32).reshape(m, bpr * 32)
    x[m // 2] = 0.0
    aq, asc = (dev(v) for v in orc.pf_quant_rows(x, bpr))
    scale = dev(rng.uniform(0.01, 0.05, size=m).astype(np.float32))
    got = []
    try:
        lkb.pf_gemm_arith(fold)
        for cfg in (0, -1, 1):
            lkb.pf_gemm_config(cfg)
            oqs, osc = torch.full((m, I), 0x5A, dtype=torch.int8, device="cuda"), nan_f32(m, I // 32, 2)
            g = lkb.make_pf_gemm(w, [I] * 3, I, bpr, aq, asc, ntok=m, scale=scale, oqs=oqs, osc=osc, okb=I // 32)
            if width is not None and I % 128 == 0:
                assert lkb.sm_count() != 148 or lkb.lib.lkb_debug_gemm_few_width(ctypes.byref(g), 0, 148) == width
            lkb.pf_gemm_swiglu(g, 0)
            got.append((oqs, osc))
    finally:
        lkb.pf_gemm_config(-1)
        lkb.pf_gemm_arith(1)
    assert lkb.lib.lkb_pf_gemm_status() == 0
    for q, s in got[1:]:
        assert torch.equal(q, got[0][0]) and torch.equal(s.view(torch.int32), got[0][1].view(torch.int32))
    assert (int(got[0][0].float().abs().max()) > 0) == (m > 1)         # one token is the row of zeros


@pytest.mark.parametrize("m", [1, 3, 7, 8, 9, 15, 17, 23, 31, 33, 47, 63, 64, 65])
def test_last_token_beyond_the_fast_silu(lkb, orc, m):
    """A last token, alone in its pair or not, whose gates are far below -88, where the branch-free SiLU has no result (NaN): the other way must be taken for
    it although the sums beside it are of no token.  (Its block scales are beyond fp16's range, so infinite, in every form.)"""
    lkb.init(0)
    I, bpr = 256, 64
    rng = np.random.default_rng(m)
    w = [tuple(dev(x) for x in rand_q4(rng, I, bpr, "ref")) for _ in range(2)]
    aq, asc = (dev(v) for v in orc.pf_quant_rows(act_floats(rng, m * bpr * 32).reshape(m, bpr * 32), bpr))
    s = np.full(m, 0.02, dtype=np.float32)
    s[-1] = 1e4
    scale, got = dev(s), []
    try:
        for cfg in (0, -1, 1):
            lkb.pf_gemm_config(cfg)
            oqs, osc = torch.full((m, I), 0x5A, dtype=torch.int8, device="cuda"), nan_f32(m, I // 32, 2)
            lkb.pf_gemm_swiglu(lkb.make_pf_gemm(w, [I] * 3, I, bpr, aq, asc, ntok=m, scale=scale, oqs=oqs, osc=osc, okb=I // 32), 0)
            got.append((oqs, osc))
    finally:
        lkb.pf_gemm_config(-1)
    assert lkb.lib.lkb_pf_gemm_status() == 0
    assert not bool(torch.isnan(got[0][1][-1, :, 0]).any()) and int(got[0][0][-1].float().abs().max()) == 127
    for q, o in got[1:]:
        assert torch.equal(q, got[0][0]) and torch.equal(o.view(torch.int32), got[0][1].view(torch.int32))
