"""Chunk attention around the edges of its tiles (32 or 64 query positions, 128 keys, one or two tiles per block) and with
rows whose maximum keeps growing along the keys, against float64.  Rows of the cache past the chunk are NaN."""
import numpy as np
import pytest

from helpers import host, nan_f32

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,P,grow", [(31, 97, 0.0), (32, 96, 0.0), (33, 95, 0.0), (65, 63, 0.0), (1, 127, 0.0), (1, 128, 0.0),
                                      (129, 0, 0.0), (1153, 0, 0.0), (1200, 511, 0.0), (40, 600, 0.02), (1217, 130, 0.01)])
def test_pf_attn_edges(lkb, orc, m, P, grow):
    lkb.init(0)
    rng = np.random.default_rng(m + 31 * P)
    S = P + m
    K = rng.standard_normal((S + 1, 8, 64)) * 1.5
    K *= (1.0 + grow * np.arange(S + 1))[:, None, None]               # later keys score higher: the running maximum moves
    K = K.astype(np.float16)
    V = rng.standard_normal((S + 1, 8, 64)).astype(np.float16)
    Q = (rng.standard_normal((m, 2048)) * 1.5 * 0.125).astype(np.float16)
    K[S:] = np.nan
    V[S:] = np.nan
    f16 = lambda a: torch.from_numpy(a.view(np.int16).copy()).cuda().view(torch.float16)
    o = nan_f32(m, 2048)
    lkb.k_pf_attn(f16(Q), m, P, f16(K), f16(V), o)
    ref = orc.pf_attn_f64(Q.view(np.uint16), m, P, K.view(np.uint16), V.view(np.uint16))
    assert float(np.max(np.abs(host(o) - ref))) < 2e-3
    assert lkb.lib.lkb_pf_gemm_status() == 0


@pytest.mark.parametrize("m,P", [(33, 95), (1217, 130)])
@pytest.mark.parametrize("q_off,o_off", [(2, 0), (4, 1), (0, 2), (6, 3)])
def test_pf_attn_alignment(lkb, m, P, q_off, o_off):
    """Q on any 4-byte boundary (q_off halfs past an aligned one) and the output on any float's: the same bits."""
    lkb.init(0)
    g = torch.Generator(device="cuda").manual_seed(m)
    f16 = lambda n: torch.randn(n, device="cuda", generator=g).half()
    K, V, Q = f16((P + m) * 512), f16((P + m) * 512), f16(m * 2048)
    want, qb, ob = nan_f32(m, 2048), torch.empty(m * 2048 + 8, dtype=torch.float16, device="cuda"), nan_f32(m * 2048 + 8)
    lkb.k_pf_attn(Q, m, P, K, V, want)
    qb[q_off:q_off + m * 2048] = Q
    lkb.k_pf_attn(qb[q_off:], m, P, K, V, ob[o_off:])
    assert torch.equal(ob[o_off:o_off + m * 2048].view(m, 2048), want)
    assert bool(ob[:o_off].isnan().all()) and bool(ob[o_off + m * 2048:].isnan().all())
    assert lkb.lib.lkb_pf_gemm_status() == 0


def _inputs(m, P, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    f16 = lambda n, w: torch.randn(n, w, 64, device="cuda", generator=g).half()
    return f16(m, 32), f16(P + m, 8), f16(P + m, 8)


@pytest.mark.parametrize("m,row", [(40, 3), (200, 131), (1217, 700)])
def test_pf_attn_row_of_minus_infinities(lkb, m, row):
    """A query whose every visible score is -inf has no softmax: NaN, and never an average of the keys it may not see."""
    lkb.init(0)
    Q, K, V = _inputs(m, 0, m)
    want, got = nan_f32(m, 32, 64), nan_f32(m, 32, 64)
    K[:, 0, 0] = -1.0
    lkb.k_pf_attn(Q, m, 0, K, V, want)
    Q[row, 0, 0] = float("inf")                                       # head 0 reads KV head 0
    lkb.k_pf_attn(Q, m, 0, K, V, got)
    assert bool(got[row, 0].isnan().all())
    got[row, 0] = want[row, 0]
    assert torch.equal(got, want)


@pytest.mark.parametrize("m,key", [(200, 100), (1217, 1000)])
def test_pf_attn_reach_of_an_infinite_value(lkb, m, key):
    """An infinite V of a later token leaves the rows of earlier 32-position tiles alone (0 x inf would be NaN there)."""
    lkb.init(0)
    Q, K, V = _inputs(m, 0, m + 1)
    want, got = nan_f32(m, 32, 64), nan_f32(m, 32, 64)
    lkb.k_pf_attn(Q, m, 0, K, V, want)
    V[key, 5, 7] = float("inf")
    lkb.k_pf_attn(Q, m, 0, K, V, got)
    first = key // 32 * 32
    assert torch.equal(got[:first], want[:first])
    assert not bool(got[key:, 20:24, 7].isfinite().any())              # heads 20..23 read KV head 5
