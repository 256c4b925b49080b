"""The native bindings: what they refuse, and the descriptors they fill, against the fields set one by one."""
import ctypes
import importlib

import pytest

torch = pytest.importorskip("torch")


def test_refusals(lkb):
    api, fast = importlib.import_module("lfm2-ampere_b200.api"), importlib.import_module("lfm2-ampere_b200._fast")
    assert api.ptr(None) is None
    with pytest.raises(AssertionError):
        api.ptr(torch.zeros(4))                                            # host memory
    with pytest.raises(TypeError):
        api.ptr(1234)
    with pytest.raises(TypeError):
        fast.pf_gemm_dense(lkb.PfAct())                                    # a structure of another type
    with pytest.raises(TypeError):
        fast.pf_gemm_dense()
    with pytest.raises((TypeError, AssertionError)):
        fast.pf_moe_route(None, 1.5, None, None, None, None, None)
    with pytest.raises(IndexError):
        fast.fill_pf_gemm(lkb.PfGemm(), [], [1], *range(17))


def _buffer(n):
    return pytest.importorskip("numpy").zeros(n, "uint8")


@pytest.mark.parametrize("wrong", [lambda lkb: lkb.StepScratch(), lambda lkb: (ctypes.c_void_p * 2)(), lambda lkb: _buffer(16), lambda lkb: bytearray(16),
                                   lambda lkb: ctypes.byref(lkb.PfAct()), lambda lkb: None, lambda lkb: 0])
def test_an_activation_is_a_pf_act(lkb, wrong):
    """Sixteen writable bytes of another kind are refused, with the exception that a ctypes call raises."""
    for call in (lambda a: lkb.k_pf_norm(None, None, 0, a, None, None, 4), lambda a: lkb.k_pf_quant_rows(None, 2048, 64, a, 4),
                 lambda a: lkb.k_pf_conv_next(None, None, None, a, 4), lambda a: lkb.k_pf_moe_combine_norm(None, None, None, None, a, None, 4),
                 lambda a: lkb.k_pf_norm_router_select(None, None, a, None, None, 4, 1, None, None, None, None, None, None)):
        with pytest.raises(ctypes.ArgumentError):
            call(wrong(lkb))


def test_a_gemm_descriptor_is_a_ctypes_object(lkb):
    """As ctypes.byref has it: no other buffer, and nothing shorter than the descriptor."""
    n = ctypes.sizeof(lkb.PfGemm)
    for g in (_buffer(n), bytearray(n), None, ctypes.byref(lkb.PfGemm()), lkb.PfAct(), (ctypes.c_byte * (n - 1))()):
        for call in (lkb.pf_gemm_dense, lambda g: lkb.pf_gemm_moe(g, 4), lambda g: lkb.pf_gemm_swiglu(g, 4)):
            with pytest.raises(TypeError):
                call(g)


def test_numbers_as_ctypes_takes_them(lkb):
    """An argument of another type raises ctypes' exception; whole numbers are masked to the field, as in a ctypes structure."""
    for bad in (None, "4", 4.0):
        with pytest.raises(ctypes.ArgumentError):
            lkb.k_pf_moe_route(None, bad, None, None, None, None, None)
    with pytest.raises(ctypes.ArgumentError):
        lkb.k_gemv_q4_0(None, None, None, 32, 64, None, eps="1e-5")
    g, wide = lkb.make_pf_gemm([(None, None)], [(1 << 70) + 5, -3], 1 << 32 | 7, 64, None, None, ntok=True, exp_stride=-(1 << 63)), lkb.PfGemm()
    wide.N, wide.bpr, wide.ntok, wide.exp_stride = 1 << 32 | 7, 64, True, -(1 << 63)
    wide.seg_end[:] = [(1 << 70) + 5, -3, -3]
    assert bytes(g) == bytes(wide)


def test_subclasses_and_arrays_are_taken(lkb):
    """What ctypes took: a subclass by value, and whatever starts with a descriptor by reference.  Without a GPU the call ends at the stream or at
    the entry point, behind its arguments."""
    class Act(lkb.PfAct):
        _fields_ = [("more", ctypes.c_int)]
    for call in (lambda: lkb.k_pf_norm(None, None, 0, Act(), None, None, 4), lambda: lkb.pf_gemm_dense((lkb.PfGemm * 2)())):
        try:
            call()
        except (TypeError, ctypes.ArgumentError):
            raise
        except Exception:
            pass


@pytest.mark.gpu
@pytest.mark.parametrize("n_seg", [1, 2, 3])
def test_descriptor_fields(lkb, n_seg):
    new = lambda n, d: torch.zeros(n, dtype=d, device="cuda")
    segs = [(new(64, torch.uint8), new(8, torch.float16)) for _ in range(n_seg)]
    ends = [128, 256, 384][:n_seg]
    t = {k: new(16, torch.int32) for k in ("aqs", "asc", "perm", "tiles", "ntiles", "scale", "out", "oqs", "osc")}
    g = lkb.make_pf_gemm(segs, ends, 384, 24, t["aqs"], t["asc"], ntok=7, exp_stride=1 << 40, perm=t["perm"], tiles=t["tiles"], ntiles=t["ntiles"], a_shift=2,
                         scale=t["scale"], out=t["out"], out_ld=5, add=1, oqs=t["oqs"], osc=t["osc"], okb=9)
    last = n_seg - 1
    for i in range(3):
        q, d = segs[min(i, last)]
        assert (g.qs[i], g.d[i], g.seg_end[i]) == (q.data_ptr(), d.data_ptr(), ends[min(i, last)])
    assert all(getattr(g, k) == v.data_ptr() for k, v in t.items())
    assert (g.N, g.bpr, g.ntok, g.exp_stride, g.a_shift, g.out_ld, g.add, g.okb) == (384, 24, 7, 1 << 40, 2, 5, 1, 9)
    assert importlib.import_module("lfm2-ampere_b200._fast").pf_moe_route(None, 4, None, None, None, None, None) != 0       # the entry point's refusal
    h = lkb.make_pf_gemm(segs, ends, 384, 24, t["aqs"], t["asc"])
    assert h.perm is None and h.out is None and h.ntok == 0 and ctypes.sizeof(h) == ctypes.sizeof(g)
    with pytest.raises(AssertionError):
        lkb.make_pf_gemm([(segs[0][0][::2], segs[0][1])], ends, 384, 24, t["aqs"], t["asc"])        # not contiguous


class _Memory:
    """What a wrapper of device memory shows of a tensor."""
    is_cuda = True

    def __init__(self, at, whole=True):
        self.at, self.whole = at, whole

    def is_contiguous(self):
        return self.whole

    def data_ptr(self):
        return self.at


class _Subclass(torch.Tensor):
    is_cuda = property(lambda self: True)

    def data_ptr(self):
        return 4096


def test_whatever_has_a_tensor_s_address(lkb):
    """An address is asked for through is_cuda, is_contiguous() and data_ptr(), which subclasses and wrappers may have of their own."""
    api = importlib.import_module("lfm2-ampere_b200.api")
    assert api.ptr(_Memory(1 << 40)) == 1 << 40 and api.ptr(torch.zeros(4).as_subclass(_Subclass)) == 4096
    assert api.pf_act(_Memory(64), _Memory(128)).sc == 128
    g = lkb.make_pf_gemm([(_Memory(16), _Memory(32))], [128], 128, 8, _Memory(48), None)
    assert (g.qs[0], g.d[2], g.aqs, g.asc) == (16, 32, 48, None)
    assert api.ptr(_Memory(0)) == 0
    for refused in (_Memory(64, whole=False), torch.zeros(4, 4).t(), torch.nn.Parameter(torch.zeros(4))):
        with pytest.raises(AssertionError):
            api.ptr(refused)
    with pytest.raises(TypeError):
        api.ptr("64")
    with pytest.raises(ZeroDivisionError):
        api.ptr(_Memory(64, whole=type("", (), {"__bool__": lambda self: 1 // 0})()))
