"""The persistent decode kernels' exchange: whatever the caller's scratch holds on entry, whatever NaN the residual holds, and
wherever the position falls in the groups of the attention slices (the new row's group is requested later than the rest), the
results are those of the kernel sequence, bit for bit."""
import ctypes
import importlib
import time

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

H = 2048


def _fill(t, pattern):
    t.view(torch.int32).fill_(pattern)


@pytest.mark.parametrize("pattern", [0, -1, 0x3F800000], ids=["zeros", "due", "ones"])
def test_stack_takes_any_scratch(lkb, pattern):
    lkb.init(0)
    synth = importlib.import_module("lfm2-ampere_b200.synth")
    st = importlib.import_module("lfm2-ampere_b200.decode").DecodeStack(synth.make_model(3, seed=19, zipf_s=1.1))
    x0 = torch.randn(H, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    st.x.copy_(x0); st.step(); ref = st.x.clone()
    for t in (st.gu, st.logits, st.sync):
        _fill(t, pattern)
    for _ in range(2):                                     # the second launch finds what the first one left
        st.x.copy_(x0); st.step_fused(); torch.cuda.synchronize()
        assert st.status() == 0 and torch.isfinite(ref).all() and torch.equal(st.x, ref)


def test_stack_takes_any_nan(lkb):
    """A residual with the bit pattern that marks words still due: an input, never waited for."""
    lkb.init(0)
    synth = importlib.import_module("lfm2-ampere_b200.synth")
    st = importlib.import_module("lfm2-ampere_b200.decode").DecodeStack(synth.make_model(2, seed=23))
    st.x.normal_()
    st.x.view(torch.int32)[77] = -1
    st.step_fused(); torch.cuda.synchronize()
    assert st.status() == 0 and torch.isnan(st.x).any()


@pytest.mark.parametrize("pos0", [0, 31, 254, 255, 256, 543, 4605])
def test_step_at_group_edges(lkb, pos0):
    """4 layers (conv, conv, attention, conv), three steps from pos0 on: one launch for all layers == one launch per kernel."""
    lkb.init(0)
    model = importlib.import_module("lfm2-ampere_b200.model")
    net = model.make_full_model(n_layers=4, seed=7, vocab=4096)
    out = []
    for impl in ("kernels", "mega"):
        ds = model.DecodeStep(net, max_seq=pos0 + 8, moe_impl=impl)
        if pos0:
            ds.fill_kv(pos0, 3)
        ds.d_token.fill_(11)
        for t in (ds.gu, ds.logits, ds.mxbuf, ds.part) if impl == "mega" else ():
            _fill(t, 0x3F800000)
        xs = []
        for _ in range(3):
            ds.step(); torch.cuda.synchronize()
            xs.append(ds.x.clone())
        assert ds.status() == 0
        out.append((torch.stack(xs), ds.kc.clone(), ds.vc.clone(), ds.hist.clone(), ds.logits_v.clone()))
    assert torch.isfinite(out[0][0]).all()
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_logits_scratch_holds_the_last_layers_logits(lkb):
    """After a launch `scratch->logits` holds what the kernel sequence leaves there: the last layer's router logits."""
    lkb.init(0)
    synth = importlib.import_module("lfm2-ampere_b200.synth")
    st = importlib.import_module("lfm2-ampere_b200.decode").DecodeStack(synth.make_model(3, seed=29, zipf_s=1.1))
    x0 = torch.randn(H, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    st.x.copy_(x0); st.step(); ref = st.logits.clone()
    for prefetch in (0, 1):
        lkb.decode_set_expert_prefetch(prefetch)
        try:
            st.logits.zero_(); st.x.copy_(x0); st.step_fused(); torch.cuda.synchronize()
        finally:
            lkb.decode_set_expert_prefetch(0)
        assert st.status() == 0 and ref.abs().max() > 0 and torch.equal(st.logits, ref)
    net = importlib.import_module("lfm2-ampere_b200.model").make_full_model(n_layers=4, seed=7, vocab=4096)
    left = []
    for impl in ("kernels", "mega"):
        ds = importlib.import_module("lfm2-ampere_b200.model").DecodeStep(net, max_seq=16, moe_impl=impl)
        ds.d_token.fill_(11); ds.step(); torch.cuda.synchronize()
        left.append(ds.logits.clone())
    assert left[0].abs().max() > 0 and torch.equal(*left)


@pytest.fixture
def withheld(lkb):
    """lkb_debug_fused_withheld(layer, expert, polls): that logit is not published."""
    lkb.init(0)
    f = lkb.lib.lkb_debug_fused_withheld
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_uint]
    yield f
    f(-1, 0, 0)


@pytest.mark.parametrize("form", ["stack", "step"])
def test_wait_for_a_word_is_bounded(lkb, withheld, form):
    """A word that never comes, behind a barrier that everyone has reached: the launch ends with that barrier's code after the caller's
    limit of polls (16384 are some 10 ms, the default 4 M some seconds), and the next one is right again."""
    layer = 2
    if form == "stack":
        synth = importlib.import_module("lfm2-ampere_b200.synth")
        st = importlib.import_module("lfm2-ampere_b200.decode").DecodeStack(synth.make_model(4, seed=31))
        go = st.step_fused
    else:
        model = importlib.import_module("lfm2-ampere_b200.model")
        st = model.DecodeStep(model.make_full_model(n_layers=4, seed=9, vocab=2048), max_seq=16, moe_impl="mega")
        go = st.step
    x0 = torch.randn(H, device="cuda", generator=torch.Generator("cuda").manual_seed(6))

    def launch():
        st.x.copy_(x0)
        if form == "step":
            st.d_token.fill_(11); st.d_pos.zero_(); st.hist.zero_()
        torch.cuda.synchronize()
        t = time.perf_counter()
        go()
        torch.cuda.synchronize()
        return time.perf_counter() - t
    launch()
    good = st.x.clone()
    assert st.status() == 0 and torch.isfinite(good).all()
    withheld(layer, 37, 1 << 14)
    assert launch() < 1.0 and st.status() == 1000 + 10 * layer + 1
    left = st.x.clone()                                        # the residual as that layer's FFN found it: nothing still due
    withheld(-1, 0, 0)
    launch()
    assert st.status() == 0 and torch.equal(st.x, good) and torch.isfinite(left).all()
    if form == "stack":
        st.x.copy_(x0)
        for i in range(layer):
            lkb.moe_ffn_decode(st._descs[i], st.x, None, None, None, st._scratch)
        torch.cuda.synchronize()
        assert torch.equal(left, st.x)
