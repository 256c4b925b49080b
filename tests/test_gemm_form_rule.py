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
