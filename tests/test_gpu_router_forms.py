"""The tiled router's CTA shapes at their edges: token counts around a CTA's four, eight and sixteen tokens and around the counts at
which the launcher goes to the next shape, against one chunk in the largest shape, bit for bit (every logit is the same chain)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_pieces_of_every_shape_equal_one_chunk(lkb):
    lkb.init(0)
    sms = lkb.lib.lkb_sm_count()
    m = 16 * sms + 1                                                 # 32-token CTAs
    gen = torch.Generator("cuda").manual_seed(31)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    H, W, bias, inv = rnd(m, 2048), 0.03 * rnd(64, 2048), 0.1 * rnd(64), 0.5 + torch.rand(m, device="cuda", generator=gen)
    out = lambda n: (torch.full((n, 64), float("nan"), device="cuda"), torch.full((n, 64), float("nan"), device="cuda"))
    sel, sig = out(m)
    lkb.k_pf_router_tiled(H, m, W, bias, inv, sel, sig)
    assert bool(torch.isfinite(sel).all())
    for n in (1, 3, 4, 5, 7, 8, 9, 4 * sms, 4 * sms + 1, 8 * sms, 8 * sms + 1, 16 * sms):
        sel2, sig2 = out(n)
        lkb.k_pf_router_tiled(H, n, W, bias, inv, sel2, sig2)
        assert torch.equal(sel2, sel[:n]) and torch.equal(sig2, sig[:n]), n


def test_cluster_form_equals_token_form(lkb):
    """The short router's two forms, alone and with the selection in the launch, around the count at which the launcher changes."""
    lkb.init(0)
    m, gen = 256, torch.Generator("cuda").manual_seed(32)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    H, W, bias, inv = rnd(m, 2048), 0.03 * rnd(64, 2048), 0.1 * rnd(64), 0.5 + torch.rand(m, device="cuda", generator=gen)
    new = lambda n: [torch.full((n, 64), float("nan"), device="cuda") for _ in range(2)] + [torch.full((n, 4), -1, dtype=torch.int32, device="cuda"),
                                                                                         torch.full((n, 4), float("nan"), device="cuda")]
    ref = new(m)
    lkb.k_pf_router_select(H, m, True, W, bias, inv, *ref)                # 256 tokens: a CTA per token
    assert all(bool(torch.isfinite(t.float()).all()) for t in ref) and int(ref[2].min()) >= 0
    for n in (1, 2, 37, 159, 160, 161):
        got = new(n)
        lkb.k_pf_router_select(H, n, True, W, bias, inv, *got)
        assert all(torch.equal(a, b[:n]) for a, b in zip(got, ref)), n
        alone = new(n)
        lkb.k_pf_router_small(H, n, W, bias, inv, alone[0], alone[1])
        assert torch.equal(alone[0], ref[0][:n]) and torch.equal(alone[1], ref[1][:n]), n


def test_norm_and_router_in_one_launch_equal_two(lkb):
    """Up to 160 tokens the norm shares the short router's launch: activations, 1 / rms, gates and selection, bit for bit; and the counts behind."""
    lkb.init(0)
    m, gen = 300, torch.Generator("cuda").manual_seed(33)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    X, nw, W, bias = rnd(m, 2048) * torch.exp(rnd(m, 1)), 1 + 0.1 * rnd(2048), 0.03 * rnd(64, 2048), 0.1 * rnd(64)
    X[3], X[5, :32] = 0.0, 0.0                                         # a row and a block of zeros
    def new(n):
        full = lambda *s, **k: torch.full(s, k.pop("fill", float("nan")), device="cuda", **k)
        return (full(n, 2048, fill=0x55, dtype=torch.int8), full(n, 64, 2), full(n), full(n, 64), full(n, 64), full(n, 4, fill=-1, dtype=torch.int32), full(n, 4), full(n, 2048))
    for n in (1, 2, 37, 159, 160, 161, 256, 300):
        qs, sc, inv, sel, sig, idx, w, h = new(n)
        lkb.k_pf_norm(X, nw, 0, lkb.pf_act(qs, sc), inv, h, n)
        lkb.k_pf_router_select(h, n, n <= 256, W, bias, inv, sel, sig, idx, w)
        got = new(n)
        lkb.k_pf_norm_router_select(X, nw, lkb.pf_act(*got[:2]), got[2], got[7], n, n <= 256, W, bias, *got[3:7])
        assert all(torch.equal(a, b) for a, b in zip(got[:7], (qs, sc, inv, sel, sig, idx, w))), n
        assert bool(torch.isnan(got[7]).all()) == (n <= 160)
