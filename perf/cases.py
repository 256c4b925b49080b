"""The work a user of this framework has it do, as cases that can be timed: token generation, prompt prefill, the
mixture-of-experts stack by itself, the output projection and a single projection, each through the package's public
entry points, with seeded synthetic weights of the shapes and value distributions that the rest of the repository uses.

Kinds:
  generate    a few tokens of greedy decoding through the whole model at some context length.  As the C++ host does it:
              one CUDA graph per token, captured when the model is loaded; token id and position live on the device.
  prefill     one chunk of m prompt tokens at positions P .. P+m-1 through the whole model (`PrefillChunk`), which leaves
              the conv histories and the KV cache where decoding continues.
  moe_prefill one chunk through the stack of MoE layers alone (`PrefillStack`, the benchmark's headline workload).
  moe_decode  one token through the stack of MoE layers alone, one persistent launch (`DecodeStack.step_fused`).
  lm_head     the decode tail: Q6_K output projection over the vocabulary and the argmax.
  projection  a norm and the Q4_0 projection behind it, batch 1: the smallest calls of the C ABI.
"""
from __future__ import annotations

import importlib

import torch

_pkg = importlib.import_module("lfm2-ampere_b200")
_synth = importlib.import_module("lfm2-ampere_b200.synth")
_decode = importlib.import_module("lfm2-ampere_b200.decode")
_prefill = importlib.import_module("lfm2-ampere_b200.prefill")
_model = importlib.import_module("lfm2-ampere_b200.model")

H, E, TOPK, I = _synth.H, _synth.E, _synth.TOPK, _synth.I
KV_ROW = _model.N_KV * _model.HEAD_DIM              # K (or V) values of one position and attention layer
VOCAB, SBPR = _model.VOCAB, _model.SBPR
LAYERS = 40


def listed():
    return [
        # One projection of one layer (the benchmark's configuration 0 shape): the shortest call, all latency.
        {"name": "projection 2048x2048", "kind": "projection", "rows": 2048, "bpr": 64, "residual": True},
        # One MoE layer at batch 1 (configuration 1), for a host that drives the layers itself.
        {"name": "moe layer, one token", "kind": "moe_decode", "layers": 1, "zipf": 0.0},
        # The MoE stack at batch 1, all layers in one launch (configuration 2), skewed routing as in the benchmark.
        {"name": "moe stack, one token", "kind": "moe_decode", "layers": LAYERS, "zipf": 1.1},
        # Scoring the vocabulary for one token.
        {"name": "lm_head 65536", "kind": "lm_head", "vocab": VOCAB},
        # Chat-length context: every decoded token of an ordinary conversation.
        {"name": "generate at 4096", "kind": "generate", "layers": LAYERS, "ctx": 4096, "tokens": 4},
        # A long document in the context (configuration 4).
        {"name": "generate at 131000", "kind": "generate", "layers": LAYERS, "ctx": 131000, "tokens": 2},
        # A short question: the whole prompt is one small chunk.
        {"name": "prefill 37", "kind": "prefill", "layers": LAYERS, "m": 37, "P": 0},
        # The next turn of a conversation: a few hundred new tokens behind an existing context.
        {"name": "prefill 509 at 1234", "kind": "prefill", "layers": LAYERS, "m": 509, "P": 1234},
        # The chunk size of the host, first chunk of a long prompt.
        {"name": "prefill 4096", "kind": "prefill", "layers": LAYERS, "m": 4096, "P": 0},
        # A late chunk of a 32768-token prompt in 8192-token chunks (configuration 4): attention over a long history.
        {"name": "prefill 8192 at 24576", "kind": "prefill", "layers": LAYERS, "m": 8192, "P": 24576},
        # The benchmark's headline (configuration 3): a 4096-token chunk through the MoE stack, skewed routing.
        {"name": "moe prefill 4096", "kind": "moe_prefill", "layers": LAYERS, "m": 4096, "zipf": 1.1},
        # The ragged last chunk of a prompt through the MoE stack, balanced routing.
        {"name": "moe prefill 1237", "kind": "moe_prefill", "layers": LAYERS, "m": 1237, "zipf": 0.0},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm, odd ones as likely as even ones."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["generate", "generate", "prefill", "prefill", "prefill", "moe_prefill", "moe_decode", "lm_head", "projection"])
    layers = rng.choice([4, 8, 16, 24, 40])
    zipf = rng.choice([0.0, 1.1, round(rng.uniform(0.0, 1.3), 2)])
    if kind == "generate":
        return {"kind": kind, "layers": layers, "ctx": _log(rng, 1, 131000), "tokens": rng.randint(1, 6)}
    if kind == "prefill":
        m = _log(rng, 2, 8192)
        return {"kind": kind, "layers": layers, "m": m, "P": rng.choice([0, _log(rng, 1, 24576)])}
    if kind == "moe_prefill":
        return {"kind": kind, "layers": layers, "m": _log(rng, 2, 8192), "zipf": zipf}
    if kind == "moe_decode":
        return {"kind": kind, "layers": rng.randint(1, 40), "zipf": zipf}
    if kind == "lm_head":
        return {"kind": kind, "vocab": _log(rng, 1000, VOCAB)}
    return {"kind": kind, "rows": _log(rng, 32, 65536), "bpr": 64, "residual": rng.random() < 0.5}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(seed, *shape):
    return torch.randn(*shape, device="cuda", generator=_gen(seed))


def prepare(case, seed):
    _pkg.init(torch.cuda.current_device())
    kind, seed = case["kind"], 7919 * seed + 17
    if kind == "generate":
        ctx, n = case["ctx"], case["tokens"]
        net = _model.make_full_model(case["layers"], seed=seed)
        ds = _model.DecodeStep(net, max_seq=ctx + n + 8, moe_impl="mega")
        toks = torch.randint(0, VOCAB, (1,), dtype=torch.int32, device="cuda", generator=_gen(seed + 1))
        hist = 0.5 * _normal(seed + 2, *ds.hist.shape)
        ds.d_token.copy_(toks)
        ds.hist.copy_(hist)
        ds.fill_kv(ctx, seed + 3)
        pos = ds.d_pos.clone()
        ds.step()                                    # loads every kernel before the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode="thread_local"):
            ds.step()
        return {"kind": kind, "ds": ds, "graph": graph, "first": toks, "pos": pos, "hist": hist, "n": n,
                "out": torch.zeros(n, dtype=torch.int32, device="cuda")}
    if kind == "prefill":
        m, P = case["m"], case["P"]
        net = _model.make_full_model(case["layers"], seed=seed)
        ds = _model.DecodeStep(net, max_seq=P + m + 64, moe_impl="mega")
        hist = 0.5 * _normal(seed + 2, *ds.hist.shape) if P else torch.zeros_like(ds.hist)
        if P:
            ds.fill_kv(P, seed + 3)
        pf = _model.PrefillChunk(net, m, ds)
        pf.toks.copy_(torch.randint(0, VOCAB, (m,), dtype=torch.int32, device="cuda", generator=_gen(seed + 1)))
        return {"kind": kind, "pf": pf, "ds": ds, "hist": hist, "P": P}
    if kind == "moe_prefill":
        ps = _prefill.PrefillStack(_synth.make_model(case["layers"], seed=seed, zipf_s=case["zipf"]), case["m"])
        return {"kind": kind, "ps": ps, "X": _normal(seed + 1, case["m"], H)}
    if kind == "moe_decode":
        st = _decode.DecodeStack(_synth.make_model(case["layers"], seed=seed, zipf_s=case["zipf"]))
        return {"kind": kind, "st": st, "x": _normal(seed + 1, H)}
    if kind == "lm_head":
        n = case["vocab"]
        planes = _model.make_q6(_gen(seed), n, "cuda")
        x, w = _normal(seed + 1, H), 1.0 + 0.05 * _normal(seed + 2, H)
        xq = torch.zeros(64 * 36, dtype=torch.uint8, device="cuda")
        ssq = torch.zeros(64, device="cuda")
        _pkg.norm_produce(x, H, _pkg.norm_prod(w, None, xq, ssq))
        nb = (n + 1023) // 1024
        return {"kind": kind, "planes": planes, "n": n, "xq": xq, "ssq": ssq, "y": torch.zeros(n, device="cuda"),
                "pv": torch.zeros(nb, device="cuda"), "pi": torch.zeros(nb, dtype=torch.int32, device="cuda"),
                "token": torch.zeros(1, dtype=torch.int32, device="cuda")}
    qs, d = _synth._q4(_gen(seed), case["rows"], case["bpr"], "cuda")
    return {"kind": kind, "qs": qs, "d": d, "rows": case["rows"], "bpr": case["bpr"], "add": int(case["residual"]),
            "x": _normal(seed + 1, H), "w": 1.0 + 0.05 * _normal(seed + 2, H), "res": _normal(seed + 3, case["rows"]),
            "xq": torch.zeros(64 * 36, dtype=torch.uint8, device="cuda"), "y": torch.zeros(case["rows"], device="cuda")}


def run(s):
    kind = s["kind"]
    if kind == "generate":
        ds, out = s["ds"], s["out"]
        ds.d_token.copy_(s["first"])
        ds.d_pos.copy_(s["pos"])
        ds.hist.copy_(s["hist"])
        for i in range(s["n"]):
            s["graph"].replay()
            out[i:i + 1].copy_(ds.d_token)
        return {"tokens": out, "logits": ds.logits_v, "x": ds.x, "hist": ds.hist, "kc": ds.kc, "vc": ds.vc, "pos": ds.d_pos}
    if kind == "prefill":
        pf, ds = s["pf"], s["ds"]
        ds.hist.copy_(s["hist"])
        pf.step(s["P"])
        return {"x": pf.X, "inv": pf.inv, "hist": ds.hist, "kc": ds.kc, "vc": ds.vc, "pos": ds.d_pos}
    if kind == "moe_prefill":
        ps = s["ps"]
        ps.X.copy_(s["X"])
        ps.step()
        return {"x": ps.X, "inv": ps.n_inv}
    if kind == "moe_decode":
        st = s["st"]
        st.x.copy_(s["x"])
        st.step_fused()
        return {"x": st.x, "w": st.sel_w, "idx": st.sel_idx}
    if kind == "lm_head":
        _pkg.k_gemv_q6_K(*s["planes"], s["xq"], s["n"], SBPR, s["y"], s["ssq"], 1e-5)
        _pkg.k_argmax_part(s["y"], s["n"], s["pv"], s["pi"])
        _pkg.k_argmax_final(s["pv"], s["pi"], s["pv"].numel(), s["token"])
        return {"logits": s["y"], "token": s["token"]}
    if s["add"]:
        s["y"].copy_(s["res"])
    _pkg.k_rmsnorm_q8_1(s["x"], s["w"], H, 1e-5, None, None, s["xq"])
    _pkg.k_gemv_q4_0(s["qs"], s["d"], s["xq"], s["rows"], s["bpr"], s["y"], s["add"])
    return s["y"]


def _q4_bytes(rows, k):
    return rows * (k // 32) * 18


def _mixer(i):
    """(weight rows of H inputs, whether it is an attention layer) of layer i's sequence mixer."""
    return (H + 2 * KV_ROW + H, True) if i % 4 == 2 else (3 * H + H, False)


def _moe_weights(n_experts):
    return E * H * 4 + n_experts * (_q4_bytes(2 * I, H) + _q4_bytes(H, I))


def work(case):
    kind = case["kind"]
    if kind == "projection":
        r = case["rows"]
        return {"bytes": _q4_bytes(r, H) + 2 * H * 4 + r * 4 * (2 if case["residual"] else 1), "flops": 2.0 * r * H}
    if kind == "lm_head":
        n = case["vocab"]
        return {"bytes": n * SBPR * 210 + n * 4, "flops": 2.0 * n * H}
    n = case["layers"]
    expert_macs = 3 * I * H
    if kind == "moe_decode":
        return {"bytes": n * (_moe_weights(TOPK) + 3 * H * 4), "flops": 2.0 * n * (E * H + TOPK * expert_macs)}
    if kind == "generate":
        ctx, t = case["ctx"], case["tokens"]
        b, f = VOCAB * SBPR * 210 + VOCAB * 4, VOCAB * H
        for i in range(n):
            rows, attn = _mixer(i)
            b += _q4_bytes(rows, H) + _moe_weights(TOPK)
            f += rows * H + E * H + TOPK * expert_macs
            if attn:
                b += ctx * KV_ROW * 4
                f += 2 * ctx * H
        return {"bytes": t * b, "flops": 2.0 * t * f}
    m = case["m"]
    hit = E * (1.0 - (1.0 - TOPK / E) ** m)                       # experts that some token of the chunk selects, on average
    b, f = 2 * m * H * 4, 0.0
    for i in range(n):
        b += _moe_weights(hit)
        f += m * (E * H + TOPK * expert_macs)
        if kind == "prefill":
            rows, attn = _mixer(i)
            b += _q4_bytes(rows, H)
            f += m * rows * H
            if attn:
                b += (case["P"] + 2 * m) * KV_ROW * 4
                f += 2.0 * m * (case["P"] + (m + 1) / 2) * H
    return {"bytes": b, "flops": 2.0 * f}


def tolerance(case):
    kind = case["kind"]
    if kind in ("projection", "lm_head"):
        return {"rel": 1e-5}                                      # integer block dots, fp32 sums in another order
    if kind == "moe_decode" and case["layers"] == 1:
        return {"rel": 1e-3, "max": 0.05}                         # an activation at a rounding tie of Q8_1 may fall either way
    return {"rel": 1e-2, "max": 0.5}                              # the same, layer after layer
