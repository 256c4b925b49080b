"""Which calls of the Q4_0 x Q8_1 GEMM take the few-token form by themselves, on the CPU: the rule is about tokens and slots, not about the
tiles a caller allows for (an upper bound that a full plan may meet exactly)."""
import ctypes

import pytest


def _better(lkb, *, ntok, perm, max_tiles=0):
    g = lkb.PfGemm()
    g.ntok, g.perm, g.N, g.bpr = ntok, perm, 2048, 64
    return lkb.lib.lkb_debug_gemm_few_better(ctypes.byref(g), max_tiles) == 1


@pytest.mark.parametrize("slots,max_tiles,few", [
    (4096, 64, False),                   # 64 experts, a full tile each, bounded exactly
    (4096, 66, False),
    (0, 65, False),                      # slots not stated
    (4, 64, True), (148, 66, True), (188, 66, True), (189, 66, False),
    (148, 320, True),                    # the bound of a longer chunk's buffers
    (100, 8, False),                     # a plan of a few experts: its tiles are fuller than the slots let expect
])
def test_grouped(lkb, slots, max_tiles, few):
    assert _better(lkb, ntok=slots, perm=64, max_tiles=max_tiles) == few


@pytest.mark.parametrize("m", range(1, 10))
def test_dense(lkb, m):
    assert _better(lkb, ntok=m, perm=None) == (m <= 4)


@pytest.mark.parametrize("slots,max_tiles,width", [(4, 64, 16), (188, 66, 16), (189, 66, 16), (800, 76, 16), (801, 76, 32), (1920, 94, 32), (1921, 94, 0), (4096, 128, 0), (0, 66, 0), (400, 63, 0)])
def test_width_of_grouped_items(lkb, slots, max_tiles, width):
    g = lkb.PfGemm()
    g.ntok, g.perm, g.N, g.bpr = slots, 64, 2048, 64
    assert lkb.lib.lkb_debug_gemm_few_width(ctypes.byref(g), max_tiles, 148) == width


@pytest.mark.parametrize("slots,max_tiles,width", [
    (4096, 64, 0), (1921, 320, 0), (1920, 320, 32), (800, 320, 16), (148, 320, 16), (1, 64, 16),       # the bound on the tiles decides nothing
    (100, 8, 0), (1920, 63, 0),          # a plan of a few experts
    (0, 65, 0), (-4, 65, 0),             # slots not stated
])
def test_grouped_calls_that_take_the_form(lkb, slots, max_tiles, width):
    """The launcher's own rule, over its whole range of slots (test_grouped: the sizes where the form is the better one whatever the routing)."""
    g = lkb.PfGemm()
    g.ntok, g.perm, g.N, g.bpr = slots, 64, 2048, 64
    assert lkb.lib.lkb_debug_gemm_few_width(ctypes.byref(g), max_tiles, 148) == width
    assert not _better(lkb, ntok=slots, perm=64, max_tiles=max_tiles) or width


@pytest.mark.parametrize("m,N,bpr,width", [(1, 2048, 64, 8), (4, 6144, 8, 8), (5, 2048, 8, 0), (37, 6144, 64, 8), (64, 6144, 64, 16), (96, 6144, 64, 16), (97, 6144, 64, 24), (144, 6144, 64, 24), (145, 6144, 64, 0),
                                           (144, 2048, 64, 8), (180, 2048, 64, 16), (289, 2048, 64, 24), (432, 2048, 64, 24), (433, 2048, 64, 0), (4096, 6144, 64, 0)])
def test_width_of_dense_items(lkb, m, N, bpr, width):
    """By the waves of items over 148 SMs in either form."""
    g = lkb.PfGemm()
    g.ntok, g.N, g.bpr = m, N, bpr
    assert lkb.lib.lkb_debug_gemm_few_width(ctypes.byref(g), 0, 148) == width


@pytest.mark.parametrize("m,N,bpr,width", [(5, 128, 64, 8), (37, 1536, 64, 8), (100, 1536, 64, 16), (130, 1536, 64, 16), (200, 1536, 64, 24), (300, 1536, 64, 0)])
def test_width_of_dense_swiglu_items(lkb, m, N, bpr, width):
    """An item of the SwiGLU form is 128 output rows (128 gate and 128 up rows): N / 128 of them a width of tokens, in either form."""
    g = lkb.PfGemm()
    g.ntok, g.N, g.bpr, g.oqs = m, N, bpr, 64
    assert lkb.lib.lkb_debug_gemm_few_width(ctypes.byref(g), 0, 148) == width
