"""The branch-free SiLU of the SwiGLU stores against the division it stands for, over every float there is."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _counts(lkb, first, count):
    lkb.init(0)
    f = lkb.lib.lkb_debug_silu
    f.argtypes = [ctypes.c_uint, ctypes.c_ulonglong, ctypes.c_void_p, ctypes.c_void_p]
    n = torch.zeros(2, dtype=torch.int64, device="cuda")
    assert f(first, count, n.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    return n.tolist()


@pytest.mark.parametrize("first", [k << 29 for k in range(8)], ids=hex)
def test_sure_of_the_division_s_result_alone(lkb, first):
    assert _counts(lkb, first, 1 << 29)[0] == 0


@pytest.mark.parametrize("lo,hi", [(0x24000000, 0x7F000000), (0xA4000000, 0xC2180000)], ids=["2^-55 to 2^127", "-2^-55 to -38"])
def test_sure_wherever_it_matters(lkb, lo, hi):
    assert _counts(lkb, lo, hi - lo) == [0, 0]
