#!/usr/bin/env python3
"""Benchmark of the Q4_0 x Q8_1 MoE hot path on B200.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

One JSON line on stdout (rank 0).  The same metric at every N:
  metric  "4k prefill tok/s": one step = a 4096-token chunk through the 40 MoE-FFN layers of the synthetic model
          (benchmark configuration 3, Zipf(1.1)-skewed routing): per layer norm -> batched router -> top-4 -> count /
          plan / scatter -> grouped gate|up GEMM with the SwiGLU + Q8_1 epilogue -> grouped down GEMM -> rank-order
          combine + next norm.  13.6 GB of expert weights are streamed per step (inputs larger than L2).
          N > 1: expert-parallel (64/N experts and 4096/N tokens per GPU, token exchange over NVLink), strong scaling;
          before timing every rank compares a 2-layer 512-token expert-parallel run with the single-GPU path bit for
          bit (config.ep_parity) and the run exits non-zero on a mismatch.
  value   tokens/s with the chunk's hidden states resident in HBM (CUDA-event time over exactly K steps, max over ranks).
  e2e     the same steps through the public API with the hidden states copied host->device from pinned memory and
          the result copied back inside the timed region.
  roofline  the dominant kernel (the tcgen05 grouped GEMM): int8 operations of the useful slots per launch / its
          CUDA-event duration, against the int8 tensor peak measured on the spot with a library GEMM; under
          roofline.decode the batch-1 decode step (configuration 2) against the measured HBM peak.
  config.decode  the other half of the metric, measured at N = 1 (batch-1 decode does not shard): the full-model
          step (configuration 2), the 40-layer MoE stack (configuration 1 x 40), the single GEMV (configuration 0),
          the lm_head, and the long-context figures (configuration 4).
  cpu_baseline  the CPU checker's restatement of the reference formulas on a 256-token slice of one layer of
          configuration 3, all host cores, extrapolated linearly in tokens and layers.
Data are seeded synthetic tensors with the configurations' shapes and value distributions.
"""
import argparse
import importlib
import json
import os
import pathlib
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = pathlib.Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

N_LAYERS = 40
H, E, TOPK, I = 2048, 64, 4, 1536
LAYER_BYTES = E * H * 4 + 2 * TOPK * I * (H // 32) * 18 + TOPK * H * (I // 32) * 18 + 3 * H * 4   # 21,782,528
METRIC = "4k prefill tok/s"
UNIT = "tok/s"
DTYPE = "int4 x int8 -> int32 block sums (exact), fp32 accumulate"


def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured", d
    return 6650.0, "fallback", {}


class ClockSampler:
    """Samples SM clock and throttle reasons with nvidia-smi while a timed region runs."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.idx, self.proc, self.lines = gpu_index, None, []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.idx}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "50"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=lambda: self.lines.extend(self.proc.stdout), daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.15)
        self.proc.terminate()
        self.t.join(timeout=2)
        mhz, mx, reasons = [], None, set()
        for ln in self.lines:
            f = [v.strip() for v in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                mhz.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for name, v in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"), f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": float(np.median(mhz)) if mhz else None, "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(mhz)}


# --------------------------------------------------------------------------- CPU baseline
_HOST_LAYER = {}


def host_layer(seed=4321):
    """One MoE layer on the host with the benchmark's value distributions (numpy, seeded)."""
    if seed in _HOST_LAYER:
        return _HOST_LAYER[seed]
    rng = np.random.default_rng(seed)

    def q4(rows, bpr):
        qs = rng.integers(0, 256, size=(rows, bpr, 16), dtype=np.uint8)
        d = np.abs(rng.normal(0, 0.02, size=(rows, bpr))).astype(np.float16).view(np.uint16)
        return qs, d
    _HOST_LAYER[seed] = dict(gate=q4(E * I, H // 32), up=q4(E * I, H // 32), down=q4(E * H, I // 32),
                             router=(0.02 * rng.standard_normal((E, H))).astype(np.float32),
                             bias=(0.01 * rng.standard_normal(E)).astype(np.float32),
                             nw=(1 + 0.05 * rng.standard_normal(H)).astype(np.float32))
    return _HOST_LAYER[seed]


def cpu_layer_token(orc, L, x):
    """The checker's statement of one batch-1 MoE FFN layer (the reference's CPU-side formulas)."""
    h32, act, ssq = orc.norm_prod(x, L["nw"])
    inv = orc.norm_inv(ssq)
    logits = orc.router_dot(h32, L["router"], ninv=inv)
    sel, sig = orc.router_gate(logits, L["bias"])
    idx, w = orc.router_select(sel, sig)
    g = orc.gemv_q4_0_exp(L["gate"][0], L["gate"][1], act, I, H // 32, I, 0, idx, ninv=inv)
    u = orc.gemv_q4_0_exp(L["up"][0], L["up"][1], act, I, H // 32, I, 0, idx, ninv=inv)
    act2 = orc.quantize_q8_1(orc.swiglu(g, u))
    xo, _, _, _ = orc.moe_down_accum(L["down"][0], L["down"][1], act2, H, I // 32, H, I // 32, idx, w, x, None)
    return xo


def host_threads():
    """Host cores this process may use (its CPU affinity): the CPU legs pin their OpenMP team to it, so that a
    launcher's OMP_NUM_THREADS=1 does not decide the baseline."""
    try:
        return max(1, len(os.sched_getaffinity(0)))
    except AttributeError:
        return max(1, os.cpu_count() or 1)


def cpu_decode_baseline(target_s=4.0):
    """Batch-1 MoE layer passes on the host (the CPU side of the decode figures under config.decode)."""
    orc = importlib.import_module("oracle.lkb_oracle")
    orc.set_num_threads(host_threads())
    L = host_layer()
    rng = np.random.default_rng(1)
    x = rng.standard_normal(H).astype(np.float32)
    t0 = time.perf_counter()
    x1 = cpu_layer_token(orc, L, x)
    t1 = time.perf_counter() - t0
    n = max(2, int(target_s / max(t1, 1e-4)))
    t0 = time.perf_counter()
    for i in range(n):
        x1 = cpu_layer_token(orc, L, x if i % 2 else x1 * 0.5)
    per_layer = (time.perf_counter() - t0) / n
    return {"value": 1.0 / (per_layer * N_LAYERS), "unit": UNIT, "cores": orc.num_threads(), "kind": "port",
            "sample": f"{n} batch-1 MoE-layer passes on the host, {per_layer * 1e3:.2f} ms per layer, x{N_LAYERS} layers per token"}


PF_SLICE = 256           # tokens of the CPU leg's slice of configuration 3


def cpu_prefill_layer(orc, L, X):
    """The checker's statement of one prefill MoE layer over the rows of X (the reference's CPU-side formulas)."""
    m = X.shape[0]
    aq, asc, inv, h32 = orc.pf_norm(X, L["nw"], plain=False, want_h32=True)
    logits = orc.pf_router_logits(h32, L["router"], inv, 0 if m <= 256 else 1)
    sel, sig = orc.pf_gate(logits, L["bias"])
    idx, w = orc.pf_select(sel, sig)
    cnt, off, tiles, perm = orc.moe_plan(idx.reshape(-1))
    a2q, a2s, _ = orc.pf_gemm_swiglu(L["gate"], L["up"], I, H // 32, aq, asc, exp_stride=I * (H // 32), perm=perm, tiles=tiles,
                                     a_shift=2, scale=inv, out_rows=m * TOPK)
    D = orc.pf_gemm([L["down"]], [H, H, H], H, I // 32, a2q, a2s, exp_stride=H * (I // 32), perm=perm, tiles=tiles, a_shift=0,
                    out_rows=m * TOPK)
    return orc.pf_combine(X, D, w)


def cpu_baseline(target_s=12.0):
    """Configuration 3 on the host: a PF_SLICE-token slice of one layer (router, plan, both grouped GEMMs in the
    reference's arithmetic, combine), repeated for about target_s seconds, extrapolated linearly in tokens and layers
    (the work is linear in both: 9.4 MMAC per token and layer)."""
    orc = importlib.import_module("oracle.lkb_oracle")
    orc.set_num_threads(host_threads())
    L = host_layer()
    rng = np.random.default_rng(2)
    X = rng.standard_normal((PF_SLICE, H)).astype(np.float32)
    t0 = time.perf_counter()
    Y = cpu_prefill_layer(orc, L, X)
    t1 = time.perf_counter() - t0
    n = max(1, int(target_s / max(t1, 1e-3)))
    t0 = time.perf_counter()
    for i in range(n):
        Y = cpu_prefill_layer(orc, L, X if i % 2 == 0 else (Y * 0.5).astype(np.float32))
    per_slice = (time.perf_counter() - t0) / n
    tok_s = PF_SLICE / (per_slice * N_LAYERS)
    return {"value": tok_s, "unit": UNIT, "cores": orc.num_threads(), "kind": "port",
            "sample": f"{n} passes of one MoE layer over a {PF_SLICE}-token slice of configuration 3 (the CPU checker's restatement "
                      f"of the reference formulas, OpenMP over slots): {per_slice * 1e3:.0f} ms per slice and layer; extrapolated "
                      f"linearly to {N_LAYERS} layers ({4096 // PF_SLICE} slices per 4096-token chunk)"}, per_slice


def run_reference(args):
    """The reference's CPU implementation of the path = the CPU checker (the reference has no CPU inference path; its CPU
    code for this path is its test oracles), all host cores, on a bounded sample of the same workload."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    for _ in range(min(args.warmup, 2)):
        cpu_baseline(target_s=0.5)
    per = []
    t0 = time.perf_counter()
    steps = max(1, args.steps)
    for _ in range(steps):
        cb, per_slice = cpu_baseline(target_s=min(15.0, 60.0 / steps))
        per.append(per_slice)
    wall = time.perf_counter() - t0
    per_slice = float(np.mean(per))
    val = PF_SLICE / (per_slice * N_LAYERS)
    cb["value"] = val
    out = {"impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": args.gpus,
           "steps": args.steps, "warmup": args.warmup, "ms_per_step": 4096 / val * 1e3,
           "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": DTYPE,
           "data": "synthetic (seeded; shapes and distributions of the benchmark configuration)",
           "config": {"workload": WORKLOAD, "tokens": 4096, "layers": N_LAYERS, "cpu_threads": cb["cores"], "wall_s": wall,
                      "note": "each step is a bounded sample of the workload on the host cores (see cpu_baseline.sample)"},
           "cpu_baseline": cb,
           "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
           "gpu_launches": 0}
    print(json.dumps(out), flush=True)


WORKLOAD = ("config 3: 4096-token batched prefill through the 40 MoE-FFN layers (64 experts, top-4, hidden 2048, inter 1536, "
            "Q4_0 weights x Q8_1 activations, sigmoid + Zipf(1.1) bias router; per-expert counts, 64-slot tile plan, "
            "fixed-order scatter, grouped int8 GEMMs)")


# --------------------------------------------------------------------------- GPU arm
def ab_reference_kernels(ps, layers, api, rounds=5):
    """A/B on this GPU against the kernels to beat: the reference's own grouped-GEMM kernels, compiled unchanged for
    sm_100a (oracle/_ref/libref_kernels.so; absent where the reference checkout was not at hand when the tree was
    built -> null).  Same plan, same activations, same weights; the two layers' weight sets alternate so that neither
    side finds its weights in L2; ours and theirs interleaved, medians.  Outputs are compared byte for byte.
    Two routings: the benchmark's own Zipf-skewed plan, and the uniform 4-distinct-experts routing of the reference's
    own GEMM benchmark (tests/test_prefill.cu:605-638)."""
    import torch
    try:
        rk = importlib.import_module("oracle.ref_kernels")
        if not rk.available():
            return None
    except Exception:
        return None
    from importlib import import_module
    synth = import_module("lfm2-ampere_b200.synth")
    Hh, Ii, Ee = synth.H, synth.I, synth.E

    def timed(fn):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) * 1e3

    beq = lambda a, b: bool(torch.equal(a.view(torch.uint8), b.view(torch.uint8)))      # bytes: NaN-safe
    med = lambda v: float(np.median(v))

    def one_routing(perm, tiles, ntiles):
        def descs(li):
            l = layers[li]
            g = api.make_pf_gemm([(l.gate_qs, l.gate_d), (l.up_qs, l.up_d)], [Ii, Ii, Ii], Ii, Hh // 32, ps.a_qs, ps.a_sc,
                                 exp_stride=Ii * (Hh // 32), perm=perm, tiles=tiles, ntiles=ntiles,
                                 a_shift=2, scale=ps.inv, oqs=ps.a2_qs, osc=ps.a2_sc, okb=Ii // 32)
            dn = api.make_pf_gemm([(l.down_qs, l.down_d)], [Hh, Hh, Hh], Hh, Ii // 32, ps.a2_qs, ps.a2_sc,
                                  exp_stride=Hh * (Ii // 32), perm=perm, tiles=tiles, ntiles=ntiles,
                                  a_shift=0, out=ps.D, out_ld=Hh)
            return g, dn
        ours, theirs = {"swiglu": [], "down": []}, {"swiglu": [], "down": []}
        # parity first (untimed): same plan and inputs through both, outputs byte for byte
        g, dn = descs(0)
        api.pf_gemm_swiglu(g, ps.max_tiles)
        q_ours, s_ours = ps.a2_qs.clone(), ps.a2_sc.clone()
        rk.pf_gemm_swiglu(g, ps.max_tiles)
        same = beq(q_ours, ps.a2_qs) and beq(s_ours, ps.a2_sc)
        api.pf_gemm_moe(dn, ps.max_tiles)
        d_ours = ps.D.clone()
        rk.pf_gemm_moe(dn, ps.max_tiles)
        same = same and beq(d_ours, ps.D)
        del q_ours, s_ours, d_ours
        nl = min(2, len(layers))
        for r in range(rounds):
            # each call's weights were last read two calls earlier (a layer's gate|up planes alone are 226 MB: L2 is cold for both)
            for which, form in (("swiglu", 0), ("down", 1)):
                for order in ((r % nl, (r + 1) % nl), ((r + 1) % nl, r % nl)):
                    for k, li in enumerate(order):
                        gd = descs(li)
                        lib_ = api if k == 0 else rk
                        fn = (lambda: lib_.pf_gemm_swiglu(gd[0], ps.max_tiles)) if form == 0 else (lambda: lib_.pf_gemm_moe(gd[1], ps.max_tiles))
                        (ours if k == 0 else theirs)[which].append(timed(fn))
        o, t = med(ours["swiglu"]) + med(ours["down"]), med(theirs["swiglu"]) + med(theirs["down"])
        return {"ours_us": {"swiglu": med(ours["swiglu"]), "down": med(ours["down"])},
                "reference_kernel_us": {"swiglu": med(theirs["swiglu"]), "down": med(theirs["down"])},
                "speedup": t / o, "outputs_identical": bool(same), "timed_calls_each": 2 * rounds}

    out = {"what": "one layer's two grouped GEMMs on the same plan: this library vs the reference's kernels compiled unchanged for sm_100a"}
    out.update(one_routing(ps.perm, ps.tiles, ps.ntiles))                      # the benchmark's Zipf-skewed routing
    # uniform routing: four distinct experts per token, uniformly at random (seeded)
    m = ps.m
    gen = torch.Generator(device="cuda").manual_seed(4242)
    idx_u = torch.rand(m, Ee, device="cuda", generator=gen).topk(4, dim=1).indices.to(torch.int32).contiguous()
    cnt = torch.zeros(Ee, dtype=torch.int32, device="cuda")
    off = torch.zeros(Ee, dtype=torch.int32, device="cuda")
    tiles = torch.zeros_like(ps.tiles)
    ntiles = torch.zeros(1, dtype=torch.int32, device="cuda")
    perm = torch.zeros_like(ps.perm)
    api.k_pf_moe_count(idx_u, m * 4, cnt)
    api.k_pf_moe_plan(cnt, off, tiles, ntiles)
    api.k_pf_moe_scatter(idx_u, m * 4, off, perm)
    out["uniform_routing"] = one_routing(perm, tiles, ntiles)
    return out


def profile_traffic(name):
    """DRAM bytes per launch recorded in a profiles/ summary (a line `traffic_bytes_per_launch: N`), or None when the
    summary is missing: the figure belongs to the kernel build it was captured from, so it is read, never hard-coded."""
    p = ROOT / "profiles" / name
    if not p.exists():
        return None
    for ln in p.read_text().splitlines():
        if ln.strip().startswith("traffic_bytes_per_launch:"):
            try:
                return float(ln.split(":", 1)[1].split()[0])
            except ValueError:
                return None
    return None


def run_ours(args):
    import torch
    import torch.distributed as dist
    lkb = importlib.import_module("lfm2-ampere_b200")
    synth = importlib.import_module("lfm2-ampere_b200.synth")
    decode = importlib.import_module("lfm2-ampere_b200.decode")
    prefill = importlib.import_module("lfm2-ampere_b200.prefill")

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device: there is no CPU fallback for this path "
                         "(use --impl reference for the host-side baseline)")
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    lkb.init(local)
    lkb.set_pdl(False)
    hbm_peak, peak_kind, _ = peaks()
    st = torch.cuda.current_stream()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    decode_sections = world == 1                # batch-1 decode does not shard: measured once, at N = 1
    dsteps = max(200, args.decode_steps)        # timed decode steps
    fsteps = 3                                  # timed full-model prefill chunks

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    def max_over_ranks(ms):
        if world == 1:
            return ms
        t = torch.tensor([ms], device="cuda", dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    layers = synth.make_model(args.layers, seed=1234, zipf_s=1.1)       # the same model on every rank
    sampler = ClockSampler(local)
    if rank == 0:
        sampler.start()

    # ================================================================ prefill, configuration 3 (the headline)
    m = args.pf_tokens
    ep = world > 1
    ep_note, ep_parity = None, None
    if ep:
        # ---- parity first: 2 layers, 512 tokens, expert-parallel against the single-GPU path, bit for bit
        mp_, lp_ = 512, layers[:2]
        gen = torch.Generator(device="cuda").manual_seed(9)
        Xp = torch.randn(mp_, H, device="cuda", generator=gen)
        disp = args.ep_dispatch
        good = torch.ones(1, device="cuda")
        epp = None
        if disp == "peer":
            try:
                epp = prefill.PrefillStackEP(lp_, mp_, rank, world, dispatch="peer")
                epp.prepare()
            except Exception as exc:                                         # noqa: BLE001 - reported in the JSON line
                good.zero_()
                ep_note = f"peer exchange unavailable ({type(exc).__name__}: {exc}); NCCL exchange used"
            dist.all_reduce(good, op=dist.ReduceOp.MIN)
            if float(good.item()) == 0.0:
                epp, disp = None, "nccl"
                ep_note = ep_note or "peer exchange unavailable on another rank; NCCL exchange used"
        args.ep_dispatch = disp
        if epp is None:
            epp = prefill.PrefillStackEP(lp_, mp_, rank, world, dispatch="nccl")
        mlp = mp_ // world
        epp.X.copy_(Xp[rank * mlp:(rank + 1) * mlp])
        epp.step()
        refp = prefill.PrefillStack(lp_, mp_)
        refp.X.copy_(Xp)
        refp.step()
        torch.cuda.synchronize()
        same = torch.equal(epp.X, refp.X[rank * mlp:(rank + 1) * mlp]) and bool(torch.isfinite(epp.X).all())
        okp = torch.tensor([1 if (same and epp.status() == 0) else 0], device="cuda")
        dist.all_reduce(okp, op=dist.ReduceOp.MIN)
        ep_parity = {"bitwise_equal_to_1gpu": bool(int(okp.item())), "dispatch": disp, "tokens": mp_, "layers": 2,
                     "checked_on": f"{world} ranks, every rank's token slice, all_reduce(MIN)"}
        del epp, refp
        if not ep_parity["bitwise_equal_to_1gpu"]:
            if rank == 0:
                print(json.dumps({"metric": METRIC, "error": "expert-parallel prefill differs from the single-GPU path",
                                  "config": {"ep_parity": ep_parity}}), flush=True)
            dist.destroy_process_group()
            raise SystemExit(3)
        ps = prefill.PrefillStackEP(layers, m, rank, world, dispatch=disp)
        ps.prepare()
    else:
        ps = prefill.PrefillStack(layers, m)
    ml = m // world
    Xall = np.random.default_rng(5).standard_normal((m, H)).astype(np.float32)
    Xh = torch.from_numpy(Xall[rank * ml:(rank + 1) * ml].copy()).pin_memory()       # this rank's tokens
    Xd = Xh.cuda()
    Yh = torch.empty(ml, H, dtype=torch.float32).pin_memory()
    pf_graph = None

    def pf_step(e2e=False):
        ps.X.copy_(Xh if e2e else Xd, non_blocking=True)
        if pf_graph is not None:
            pf_graph.replay()
        else:
            ps.step()
        if e2e:
            Yh.copy_(ps.X, non_blocking=True)
            st.synchronize()
    pf_step()
    # per-launch durations of the dominant kernel: one eager step with CUDA events around every grouped-GEMM launch
    # (a graph replay hides individual launches from events); the timed region below replays the graph
    ps.gemm_events = []
    ps.step()
    torch.cuda.synchronize()
    gemm_ms = [a.elapsed_time(b) for a, b in ps.gemm_events]
    ps.gemm_events = None
    vs_ref_kernel = ab_reference_kernels(ps, layers, lkb) if not ep else None
    if (not ep or args.ep_dispatch == "peer") and not args.no_graph:
        # one CUDA graph for the step's launches (the NCCL exchange has a host sync per layer and cannot be captured)
        barrier()
        pf_graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(pf_graph, capture_error_mode="thread_local"):
            ps.step()
    for _ in range(max(3, args.warmup)):
        pf_step()
    barrier()
    ev0.record()
    for _ in range(args.steps):
        pf_step()
    ev1.record()
    barrier()
    pms = max_over_ranks(ev0.elapsed_time(ev1)) / args.steps
    for _ in range(2):
        pf_step(e2e=True)
    barrier()
    ev0.record()
    for _ in range(args.steps):
        pf_step(e2e=True)
    ev1.record()
    barrier()
    pms_e2e = max_over_ranks(ev0.elapsed_time(ev1)) / args.steps
    gstat = lkb.lib.lkb_pf_gemm_status()
    if gstat != 0:
        raise SystemExit(f"tensor-core GEMM reported status {gstat} (a bounded wait expired)")
    # int8 tensor peak of this GPU, measured with a library GEMM (timing only): MEASURED_PEAKS.json has no int8 figure
    int8_peak = None
    try:
        A8 = torch.randint(-8, 8, (8192, 8192), dtype=torch.int8, device="cuda")
        B8 = torch.randint(-8, 8, (8192, 8192), dtype=torch.int8, device="cuda")
        for _ in range(3):
            torch._int_mm(A8, B8)
        torch.cuda.synchronize()
        best = 1e9
        for _ in range(5):
            ev0.record()
            torch._int_mm(A8, B8)
            ev1.record()
            torch.cuda.synchronize()
            best = min(best, ev0.elapsed_time(ev1))
        int8_peak = 2 * 8192 ** 3 / (best * 1e-3) / 1e12
        del A8, B8
    except Exception:
        int8_peak = None
    macs = args.layers * m * TOPK * (2 * I * H + H * I)
    if ep:
        est = torch.tensor([ps.status()], device="cuda")
        dist.all_reduce(est, op=dist.ReduceOp.MAX)                       # every rank leaves together
        if int(est.item()) != 0:
            raise SystemExit(f"expert-parallel exchange reported status {int(est.item())} (a bounded wait expired)")
        mine = torch.as_tensor(ps.recv_slots).sum().to("cuda", torch.float64).reshape(1)
        mx, sm = mine.clone(), mine.clone()
        dist.all_reduce(mx, op=dist.ReduceOp.MAX)
        dist.all_reduce(sm, op=dist.ReduceOp.SUM)
        imbalance = float(mx.item() / (sm.item() / world))
        my_macs = float(mine.item()) * (2 * I * H + H * I)               # slots this rank's experts received, all layers
        launches = args.steps * ps.launches_per_step * world
    else:
        cnt = ps.cnt.cpu().numpy()
        imbalance = float(cnt.max() / max(1.0, cnt.mean()))
        my_macs = float(macs)
        launches = args.steps * ps.launches_per_step
    # dominant kernel: k_pf_gemm_tc (two launches per layer).  Algorithmic int8 operations of this rank's useful slots per
    # launch / the launches' average CUDA-event duration.
    n_gemm = max(1, len(gemm_ms))
    avg_launch_ms = float(np.mean(gemm_ms)) if gemm_ms else None
    ops_per_launch = 2.0 * my_macs / n_gemm
    ach = ops_per_launch / (avg_launch_ms * 1e-3) / 1e12 if avg_launch_ms else None
    peak8 = int8_peak or 4500.0
    roofline = {"bound": "tensor", "kernel": "k_pf_gemm_tc (tcgen05.mma.kind::i8, TMEM accumulators, operands by bulk tensor copies)",
                "achieved": ach, "peak": peak8, "unit": "TOP/s", "frac": (ach / peak8) if ach else None,
                "peak_kind": ("of measured here: torch._int_mm 8192^3, best of 5 (MEASURED_PEAKS.json records no int8 figure)"
                              if int8_peak else "of nominal dense int8 (MEASURED_PEAKS.json records no int8 figure)"),
                "nominal_int8_tops": 4500.0, "launches_per_step": n_gemm, "avg_launch_ms": avg_launch_ms,
                "algorithmic_ops_per_launch": ops_per_launch,
                "gemm_share_of_step": (float(np.sum(gemm_ms)) / pms) if gemm_ms else None,
                "traffic": profile_traffic("k_pf_gemm_tc_prefill_4096tok.txt"),
                "vs_ref_kernel": vs_ref_kernel,
                "co_bound": "the exact per-block scale arithmetic and the constants it reads: two fp32 FMAs per int32 block sum on the CUDA cores are "
                            "128 packed FMAs a scheduler for a block of 256 rows x 64 tokens, 2.9 cycles each, and the block's 128 shared loads of "
                            "constants 512 cycles of the SM's return path, of 600 or so a block, with the tensor pipe 19 to 20 % busy (profiles/)",
                "whole_step_TMACs": macs / (pms * 1e-3) / 1e12}
    pf_cfg = {"workload": WORKLOAD, "tokens": m, "layers": args.layers, "resident_weight_bytes": args.layers * 339738624,
              "cold_cache": "each step streams the whole 13.6 GB expert set (inputs larger than L2)",
              "parallelism": (f"expert-parallel x{world}: {E // world} experts and {ml} tokens per GPU, token exchange before and after "
                              "the grouped GEMMs, " + ("NCCL all_to_all_single with one host sync per layer" if args.ep_dispatch == "nccl"
                                                       else "peer-memory stores over NVLink with device-side flags, no host sync")) if ep else "single GPU",
              "cuda_graph": pf_graph is not None, "gemm_arith": "reference's shipped per-block term (folded offset): bit-identical to the reference kernel",
              ("slots_per_gpu_max_over_mean" if ep else "last_layer_max_over_mean_slots_per_expert"): imbalance,
              "gemm_TMACs": macs / (pms * 1e-3) / 1e12, "note": ep_note, "ep_parity": ep_parity,
              "published_reference": {"value": 21188.0, "unit": UNIT, "hardware": "RTX 3090 Ti, real weights, full model incl. attention, 4096 tokens",
                                      "note": "not this metric (full model): see config.full_prefill for the like-for-like chunk"}}
    del pf_graph

    # ---- long prompts through the expert-parallel MoE stack (configuration 4 at N > 1): 8192-token chunks, a 32768-token
    #      prompt = 4 chunks, a 131072-token prompt = 16 (the MoE stack has no state across chunks: same chunk, repeated)
    if ep and disp == "peer" and not args.no_long_ctx and not args.no_graph:
        try:
            del ps
            torch.cuda.empty_cache()
            m8 = 8192
            ps8 = prefill.PrefillStackEP(layers, m8, rank, world, dispatch="peer")
            ps8.prepare()
            ps8.X.copy_(torch.randn(m8 // world, H, device="cuda", generator=torch.Generator(device="cuda").manual_seed(77 + rank)))
            ps8.step()
            torch.cuda.synchronize()
            barrier()
            g8 = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g8, capture_error_mode="thread_local"):
                ps8.step()
            for _ in range(3):
                g8.replay()
            barrier()
            ev0.record()
            for _ in range(16):
                g8.replay()
            ev1.record()
            barrier()
            ms16 = max_over_ranks(ev0.elapsed_time(ev1))
            est = torch.tensor([ps8.status()], device="cuda")
            dist.all_reduce(est, op=dist.ReduceOp.MAX)
            pf_cfg["long_context_ep"] = {
                "workload": "configuration 4 through the expert-parallel MoE stack: 8192-token chunks (a 32768-token prompt = 4, a 131072-token prompt = 16)",
                "chunk_ms": ms16 / 16, "tok_s": 16 * m8 / (ms16 * 1e-3), "prompt_32768_ms": ms16 / 4, "prompt_131072_ms": ms16,
                "exchange_status": int(est.item())}
            del g8, ps8
        except Exception as exc:                       # reported, not fatal: the headline is measured above
            pf_cfg["long_context_ep"] = {"unavailable": f"{type(exc).__name__}: {exc}"}

    # ================================================================ decode (N = 1 only): configurations 0, 1, 2, 4
    dec = None
    if decode_sections:
        stack = decode.DecodeStack(layers)
        rng = np.random.default_rng(99 + rank)
        n_in = 64
        x_host = torch.from_numpy(rng.standard_normal((n_in, H)).astype(np.float32)).pin_memory()
        y_host = torch.empty(H, dtype=torch.float32).pin_memory()
        x_pool = x_host.cuda()
        x_in = torch.zeros(H, device="cuda")
        # parity inside the bench: the fused persistent kernel against the five-kernel sequence on one seeded token
        stack.x.copy_(x_pool[0]); stack.step(); torch.cuda.synchronize(); xa = stack.x.clone()
        stack.x.copy_(x_pool[0]); stack.step_fused(); torch.cuda.synchronize()
        dec_parity = bool(torch.equal(xa, stack.x))

        def one_step(i, e2e=False):
            if e2e:
                x_in.copy_(x_host[i % n_in], non_blocking=True)
            else:
                x_in.copy_(x_pool[i % n_in])
            stack.x.copy_(x_in)
            stack.step_fused()
            if e2e:
                y_host.copy_(stack.x, non_blocking=True)
                st.synchronize()
        for i in range(5):
            one_step(i)
        torch.cuda.synchronize()
        ev0.record()
        for i in range(dsteps):
            one_step(i)
        ev1.record()
        torch.cuda.synchronize()
        ms = ev0.elapsed_time(ev1)
        ev0.record()
        for i in range(dsteps):
            one_step(i, e2e=True)
        ev1.record()
        torch.cuda.synchronize()
        ms_e2e = ev0.elapsed_time(ev1)
        if stack.status() != 0:
            raise SystemExit(f"fused decode kernel reported status {stack.status()} (a bounded wait expired)")
        # the optional expert prefetch (off by default: measured slower), timed the same way, with its hit count
        pf_rec = None
        if args.layers > 1:
            lkb.decode_set_expert_prefetch(1)
            try:
                for i in range(5):
                    one_step(i)
                torch.cuda.synchronize()
                ev0.record()
                for i in range(dsteps):
                    one_step(i)
                ev1.record()
                torch.cuda.synchronize()
                hits, guesses = lkb.decode_expert_prefetch_hits(stack._scratch, args.layers)
                pf_rec = {"default": "off", "ms_per_step_on": ev0.elapsed_time(ev1) / dsteps, "ms_per_step_off": ms / dsteps,
                          "guesses_chosen": hits, "guesses": guesses, "hit_rate": hits / guesses, "status": stack.status()}
            finally:
                lkb.decode_set_expert_prefetch(0)
        k_ms = ms / dsteps
        ach_d = args.layers * LAYER_BYTES / (k_ms * 1e-3) / 1e9
        dec = {"moe_stack": {"metric": "bs1 decode tok/s, 40-layer MoE-FFN stack (configuration 1 x 40)", "value": dsteps / (ms * 1e-3),
                             "unit": UNIT, "ms_per_step": k_ms, "steps": dsteps, "parity_fused_equals_kernel_sequence": dec_parity, "expert_prefetch": pf_rec,
                             "e2e": {"value": dsteps / (ms_e2e * 1e-3), "unit": UNIT, "h2d_bytes_per_step": H * 4, "d2h_bytes_per_step": H * 4},
                             "roofline": {"bound": "hbm", "kernel": f"k_moe_ffn_stack (persistent, {args.layers} MoE layers per launch)",
                                          "achieved": ach_d, "peak": hbm_peak, "unit": "GB/s", "frac": ach_d / hbm_peak,
                                          "peak_kind": f"of {peak_kind}", "algorithmic_bytes_per_launch": args.layers * LAYER_BYTES,
                                          "traffic": (lambda t: t * args.layers / 4 if t else None)(profile_traffic("k_moe_ffn_stack_decode_4layers.txt")),
                                          "traffic_note": "ncu capture of a 4-layer launch, scaled by layers (traffic grows in proportion)"}}}
        del stack

    # ---------------------------------------------------------------- output projection + argmax (decode tail)
    lm = None
    if decode_sections and not args.no_lmhead:
        V, SB, NCOPY = 65536, 8, 3                      # three weight copies in rotation: 330 MB > L2
        gen = torch.Generator(device="cuda").manual_seed(77)
        copies = []
        for _ in range(NCOPY):
            copies.append((torch.randint(0, 256, (V * SB * 128,), dtype=torch.uint8, device="cuda", generator=gen),
                           torch.randint(0, 256, (V * SB * 64,), dtype=torch.uint8, device="cuda", generator=gen),
                           torch.randint(-128, 128, (V * SB * 16,), dtype=torch.int8, device="cuda", generator=gen),
                           (torch.rand(V * SB, device="cuda", generator=gen) * 4e-4).half()))
        xv = torch.randn(H, device="cuda", generator=gen)
        xq8 = torch.empty(H // 32 * 36, dtype=torch.uint8, device="cuda")
        lkb.k_quantize_q8_1(xv, xq8, H // 32)
        yl = torch.empty(V, dtype=torch.float32, device="cuda")
        pv, pi = torch.empty(V // 1024, device="cuda"), torch.empty(V // 1024, dtype=torch.int32, device="cuda")
        tok = torch.zeros(1, dtype=torch.int32, device="cuda")

        def lm_step(i, tail=True):
            lkb.k_gemv_q6_K(*copies[i % NCOPY], xq8, V, SB, yl, None, 0.0)
            if tail:
                lkb.k_argmax_part(yl, V, pv, pi)
                lkb.k_argmax_final(pv, pi, V // 1024, tok, None)
        # Timed as CUDA-graph replays (30 launches per graph) so that the host's launch rate is not in the figure.
        # GEMV alone: no programmatic overlap between launches.  GEMV + argmax chain: with programmatic dependent
        # launch, as the decode loop runs it (the next GEMV's weight stream starts under the argmax kernels).
        res = []
        for tail in (False, True):
            lkb.set_pdl(tail and not args.no_pdl)
            for i in range(3):
                lm_step(i, tail)
            torch.cuda.synchronize()
            gl = torch.cuda.CUDAGraph()
            with torch.cuda.graph(gl):
                for i in range(30):
                    lm_step(i, tail)
            nrep = max(1, args.lm_steps // 30)
            gl.replay()
            barrier()
            ev0.record()
            for _ in range(nrep):
                gl.replay()
            ev1.record()
            barrier()
            res.append(max_over_ranks(ev0.elapsed_time(ev1)) / (30 * nrep))
            del gl
        lkb.set_pdl(False)
        if lkb.gemv_q6_K_status() != 0:
            raise SystemExit("Q6_K streaming GEMV: a bounded wait expired")
        lm_bytes = V * SB * 210 + H // 32 * 36 + V * 4
        gbs = lm_bytes / (res[0] * 1e-3) / 1e9
        lm = {"metric": "lm_head: Q6_K 65536 x 2048 GEMV (+ two-stage argmax)", "gemv_us": res[0] * 1e3,
              "gemv_argmax_us": res[1] * 1e3, "launches_per_token": 3, "cold_cache": f"{NCOPY} weight copies in rotation (330 MB > L2)",
              "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm_peak, "unit": "GB/s", "frac": gbs / hbm_peak,
                           "peak_kind": f"of {peak_kind}", "algorithmic_bytes": lm_bytes,
                           "traffic": profile_traffic("k_gemv_q6_K_stream_lmhead_65536rows.txt") if V == 65536 else None}}
        del copies

    # ---------------------------------------------------------------- Q4_0 x Q8_1 GEMV size sweep (configuration 0 and up)
    sweep = None
    if decode_sections and not args.no_sweep:
        gen2 = torch.Generator(device="cuda").manual_seed(9)
        xq_s = torch.empty(H // 32 * 36, dtype=torch.uint8, device="cuda")
        lkb.k_quantize_q8_1(torch.randn(H, device="cuda", generator=gen2), xq_s, H // 32)
        lkb.set_pdl(False)
        sweep = []
        for rows in (2048, 6144, 65536, 262144):
            nbytes = rows * (H // 32) * 18 + H // 32 * 36 + rows * 4
            ncopy = min(160, max(2, (400 << 20) // nbytes + 1))            # rotate >= 400 MB of weights: every launch streams from HBM
            ws = [(torch.randint(0, 256, (rows * (H // 32) * 16,), dtype=torch.uint8, device="cuda", generator=gen2),
                   (torch.rand(rows * (H // 32), device="cuda", generator=gen2) * 0.02).half()) for _ in range(ncopy)]
            ys = torch.empty(rows, device="cuda")
            nl = max(ncopy, 24)
            for i in range(3):
                lkb.k_gemv_q4_0(ws[i % ncopy][0], ws[i % ncopy][1], xq_s, rows, H // 32, ys)
            torch.cuda.synchronize()
            gs = torch.cuda.CUDAGraph()
            with torch.cuda.graph(gs):
                for i in range(nl):
                    lkb.k_gemv_q4_0(ws[i % ncopy][0], ws[i % ncopy][1], xq_s, rows, H // 32, ys)
            gs.replay()
            barrier()
            ev0.record()
            gs.replay()
            ev1.record()
            barrier()
            us = max_over_ranks(ev0.elapsed_time(ev1)) / nl * 1e3
            sweep.append({"rows": rows, "k": H, "bytes": nbytes, "us": us, "GBs": nbytes / us / 1e3, "frac": nbytes / us / 1e3 / hbm_peak})
            del ws, gs

    # ---------------------------------------------------------------- full decode step (configuration 2)
    full = None
    if decode_sections and not args.no_full:
        model_mod = importlib.import_module("lfm2-ampere_b200.model")
        ctx = args.ctx
        fm = model_mod.make_full_model(n_layers=args.layers, seed=4321, moe_layers=layers)
        tok_h = torch.zeros(1, dtype=torch.int32).pin_memory()
        out_h = torch.zeros(1, dtype=torch.int32).pin_memory()
        res = {}
        for impl in ("mega", "kernels"):
            ds = model_mod.DecodeStep(fm, max_seq=ctx + 2 * (dsteps + 8) + 8, moe_impl=impl)
            ds.fill_kv(ctx)
            ds.d_token.fill_(11)
            lkb.set_pdl(impl == "kernels" and not args.no_pdl)
            ds.step()                                         # warm the launch path before capture
            torch.cuda.synchronize()
            gf = torch.cuda.CUDAGraph()
            with torch.cuda.graph(gf):
                ds.step()
            ds.d_pos.fill_(ctx)
            for _ in range(3):
                gf.replay()
            barrier()
            ev0.record()
            for _ in range(dsteps):
                gf.replay()
            ev1.record()
            barrier()
            t_dev = max_over_ranks(ev0.elapsed_time(ev1)) / dsteps
            # end to end: the token id arrives from pinned host memory, the chosen token goes back, every step
            ev0.record()
            for i in range(dsteps):
                tok_h[0] = 11 + i
                ds.d_token.copy_(tok_h, non_blocking=True)
                gf.replay()
                out_h.copy_(ds.d_token, non_blocking=True)
                st.synchronize()
            ev1.record()
            barrier()
            t_e2e = max_over_ranks(ev0.elapsed_time(ev1)) / dsteps
            if ds.status() != 0 or lkb.gemv_q6_K_status() != 0:
                raise SystemExit("full decode step: a bounded device-side wait expired")
            res[impl] = (t_dev, t_e2e, ds.launches_per_step, ds.bytes_per_step(ctx))
            del gf, ds
        lkb.set_pdl(False)
        best = min(res, key=lambda k: res[k][0])
        t_dev, t_e2e, nl, nbytes = res[best]
        gbs = nbytes / (t_dev * 1e-3) / 1e9
        full = {"metric": "bs1 decode tok/s, full model step at context %d" % ctx, "value": world * 1e3 / t_dev, "unit": UNIT,
                "ms_per_step": t_dev, "impl": best,
                "by_impl_ms": {k: v[0] for k, v in res.items()},
                "workload": ("embedding row -> %d layers [short conv (3 of 4) | GQA attention 32/8x64 over an fp16 KV cache (1 of 4)] + "
                             "64-expert top-4 MoE FFN -> Q6_K lm_head (vocab 65536) -> argmax; one CUDA graph per token, token id and "
                             "position device-resident; impl mega = all layers in one persistent launch (6 launches per token), "
                             "kernels = one launch per reference kernel with programmatic dependent launch" % args.layers),
                "e2e": {"value": world * 1e3 / t_e2e, "unit": UNIT, "h2d_bytes_per_step": 4, "d2h_bytes_per_step": 4},
                "gpu_launches_per_step": nl, "bytes_per_step": nbytes,
                "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm_peak, "unit": "GB/s", "frac": gbs / hbm_peak,
                             "peak_kind": f"of {peak_kind}", "traffic": None},
                "published_reference": {"value": 424.65, "unit": UNIT, "hardware": "RTX 3090 Ti, real weights, context 4096",
                                        "ratio": (1e3 / t_dev) / 424.65,
                                        "note": "the reference's model has vocab 128000 and two dense FFN layers: 1.467 GB per token "
                                                "against %.3f GB here" % (nbytes / 1e9)} if (ctx == 4096 and args.layers == 40) else None}
        del fm

    # ---------------------------------------------------------------- full-model prefill chunk
    fpf = None
    if decode_sections and not args.no_full:
        model_mod = importlib.import_module("lfm2-ampere_b200.model")
        m = args.pf_tokens
        fm = model_mod.make_full_model(n_layers=args.layers, seed=4321, moe_layers=layers)
        stt = model_mod.DecodeStep(fm, max_seq=m + 8, moe_impl="kernels")
        pc = model_mod.PrefillChunk(fm, m, stt)
        tok_hm = torch.randint(0, 65536, (m,), dtype=torch.int32).pin_memory()
        nxt_h = torch.zeros(1, dtype=torch.int32).pin_memory()
        pc.toks.copy_(tok_hm)

        def fpf_step(e2e=False):
            if e2e:
                pc.toks.copy_(tok_hm, non_blocking=True)
            stt.hist.zero_()
            pc.step(P=0)
            if e2e:                                            # the new position comes back to the host
                nxt_h.copy_(stt.d_pos, non_blocking=True)
                st.synchronize()
        fpf_step()
        torch.cuda.synchronize()
        ev0.record()
        for _ in range(fsteps):
            fpf_step()
        ev1.record()
        torch.cuda.synchronize()
        t_pf = ev0.elapsed_time(ev1) / fsteps
        ev0.record()
        for _ in range(fsteps):
            fpf_step(e2e=True)
        ev1.record()
        torch.cuda.synchronize()
        t_pf_e2e = ev0.elapsed_time(ev1) / fsteps
        if lkb.lib.lkb_pf_gemm_status() != 0:
            raise SystemExit("full-model prefill: a bounded wait of the tensor-core GEMM expired")
        attn_macs = sum(mx.is_attn for mx in fm.mixers) * 32 * 64 * 2 * (m * (m + 1) // 2)
        fpf = {"metric": "%dk prefill tok/s, full model chunk" % (m // 1024), "tokens": m, "value": m / (t_pf * 1e-3), "unit": UNIT,
               "ms_per_step": t_pf,
               "workload": "embedding rows -> %d layers [dense Q4_0 x Q8_1 GEMMs + chunk conv | causal GQA flash attention] + "
                           "MoE grouped GEMMs; KV caches and conv histories left ready for decoding" % args.layers,
               "e2e": {"value": m / (t_pf_e2e * 1e-3), "unit": UNIT, "h2d_bytes_per_step": 4 * m, "d2h_bytes_per_step": 4},
               "gemm_tmacs": pc.macs_per_step() / (t_pf * 1e-3) / 1e12, "attention_tmacs_total": attn_macs / 1e12,
               "gpu_launches_per_step": pc.launches_per_step,
               "published_reference": {"value": 21188.0, "unit": UNIT, "hardware": "RTX 3090 Ti, real weights, 4096 tokens",
                                       "ratio": (m / (t_pf * 1e-3)) / 21188.0} if (m == 4096 and args.layers == 40) else None}
        del pc, stt, fm

    # ---------------------------------------------------------------- long context (configuration 4)
    longc = None
    if decode_sections and not args.no_long_ctx and not args.no_full:
        model_mod = importlib.import_module("lfm2-ampere_b200.model")
        fm = model_mod.make_full_model(n_layers=args.layers, seed=4321, moe_layers=layers)
        LC = 131072
        ds = model_mod.DecodeStep(fm, max_seq=LC + 64, moe_impl="mega")
        # chunked prefill: 32768 tokens in 8192-token chunks, timed per chunk (attention cost grows with the prefix)
        CH = 8192
        pc = model_mod.PrefillChunk(fm, CH, ds)
        pc.toks.copy_(torch.randint(0, 65536, (CH,), dtype=torch.int32, device="cuda"))
        pc.step(P=0)
        ds.hist.zero_()
        torch.cuda.synchronize()
        chunk_ms = []
        ev_all0, ev_all1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev_all0.record()
        for c in range(4):
            ev0.record()
            pc.step(P=c * CH)
            ev1.record()
            torch.cuda.synchronize()
            chunk_ms.append(ev0.elapsed_time(ev1))
        ev_all1.record()
        torch.cuda.synchronize()
        pf32 = 4 * CH / (sum(chunk_ms) * 1e-3)
        del pc
        # decode at 131072 positions of context
        ds.fill_kv(LC)
        ds.d_token.fill_(11)
        ds.step()
        torch.cuda.synchronize()
        gL = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gL):
            ds.step()
        ds.d_pos.fill_(LC)
        for _ in range(3):
            gL.replay()
        torch.cuda.synchronize()
        nst = 40
        ev0.record()
        for _ in range(nst):
            gL.replay()
        ev1.record()
        torch.cuda.synchronize()
        t_l = ev0.elapsed_time(ev1) / nst
        nb = ds.bytes_per_step(LC)
        longc = {"decode_ctx_131072": {"value": 1e3 / t_l, "unit": UNIT, "ms_per_step": t_l, "bytes_per_step": nb,
                                       "roofline": {"bound": "hbm", "achieved": nb / (t_l * 1e-3) / 1e9, "peak": hbm_peak, "unit": "GB/s",
                                                    "frac": nb / (t_l * 1e-3) / 1e9 / hbm_peak, "peak_kind": f"of {peak_kind}"},
                                       "published_reference": {"value": 184.94, "unit": UNIT, "hardware": "RTX 3090 Ti, context 131040"}},
                 "prefill_32768_in_8192_chunks": {"value": pf32, "unit": UNIT, "chunk_ms": chunk_ms,
                                                  "published_reference": {"value": 18190.0, "unit": UNIT, "hardware": "RTX 3090 Ti"}}}
        if ds.status() != 0:
            raise SystemExit("long-context decode: a bounded device-side wait expired")
        del gL, ds, fm

    if rank == 0:
        clocks = sampler.stop()          # sampled over every timed region above
        cb = None
        if world == 1 and not args.no_cpu:
            cb, _ = cpu_baseline()
        if dec is not None:
            dec["full_step"] = full
            dec["lm_head"] = lm
            dec["gemv_sweep_config0"] = sweep
            dec["long_context"] = longc
            dec["cpu_baseline_decode"] = cpu_decode_baseline() if not args.no_cpu else None
            pf_cfg["decode"] = dec
            pf_cfg["full_prefill"] = fpf
            if full is not None:
                roofline["decode"] = dict(full["roofline"], kernel="full-model batch-1 decode step (configuration 2), one CUDA graph per token",
                                          tok_s=full["value"], ms_per_step=full["ms_per_step"], e2e_tok_s=full["e2e"]["value"])
        else:
            pf_cfg["decode"] = "measured at N = 1: batch-1 decode does not shard (replicas only)"
        out = {"metric": METRIC, "value": m / (pms * 1e-3), "unit": UNIT, "n_gpus": world, "steps": args.steps,
               "warmup": max(3, args.warmup), "ms_per_step": pms, "higher_is_better": True,
               "scaling": "strong", "vs_baseline": None, "dtype": DTYPE,
               "data": "synthetic (seeded; shapes and distributions of the benchmark configurations)",
               "config": pf_cfg,
               "e2e": {"value": m / (pms_e2e * 1e-3), "unit": UNIT, "h2d_bytes_per_step": m * H * 4, "d2h_bytes_per_step": m * H * 4},
               "gpu_launches": launches, "roofline": roofline, "cpu_baseline": cb, "clocks": clocks}
        print(json.dumps(out), flush=True)
    if world > 1:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10, help="timed prefill steps (one step = one 4096-token chunk through 40 layers)")
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--decode-steps", type=int, default=200, help="timed steps of the batch-1 decode sections (at least 200)")
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--layers", type=int, default=N_LAYERS)
    ap.add_argument("--pf-tokens", type=int, default=4096)
    ap.add_argument("--ep-dispatch", choices=["nccl", "peer"], default="peer",
                    help="token exchange of the expert-parallel prefill (N > 1): NCCL all-to-all, or this library's peer-memory kernels")
    ap.add_argument("--no-lmhead", action="store_true")
    ap.add_argument("--no-sweep", action="store_true", help="skip the GEMV size sweep")
    ap.add_argument("--no-long-ctx", action="store_true", help="skip decode at 131072 positions of context and the chunked 32768-token prefill")
    ap.add_argument("--no-full", action="store_true", help="skip the full-model decode step (configuration 2)")
    ap.add_argument("--ctx", type=int, default=4096, help="KV positions pre-filled for the full decode step")
    ap.add_argument("--lm-steps", type=int, default=90)
    ap.add_argument("--no-graph", action="store_true")
    ap.add_argument("--no-pdl", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
