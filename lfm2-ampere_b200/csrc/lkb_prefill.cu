// lkb_prefill.cu - batched-prefill kernels around the grouped GEMM (sm_100a):
// per-token RMSNorm -> planar Q8_1, row quantiser, SwiGLU quantiser, the batched
// router, top-4 selection, the deterministic expert count / tile plan / scatter,
// the rank-order combine, and a CUDA-core (dp4a) form of the Q4_0 x Q8_1 GEMM that
// serves as the always-available configuration (the tensor-core form lives in
// lkb_gemm_tc.cu).  Each kernel evaluates the per-token formula of its decode
// twin, so per-token results are bit-identical to the decode kernels.
#include "lkb_tc.cuh"
#include <cstdlib>

#define LKB_REQUIRE_INIT() do { if (!lkb_context().inited) return LKB_ERR_NOT_INIT; } while (0)

// ---------------------------------------------------------------------------
// Per-token kernels.  Warps own contiguous 512-byte runs: four elements per lane through 128-bit loads, four
// 32-element blocks per step (lkb_quad_quant), several tokens per CTA and no CTA-wide barrier.  The arithmetic per
// element, per block and per token is that of the decode kernels (reference semantics: src/prefill.cu:871-932 norm,
// :1574-1594 row quantisers), so outputs compare byte for byte.
// ---------------------------------------------------------------------------
#ifndef PF_TOK_SPLIT
#define PF_TOK_SPLIT 4                   // warps sharing one token in k_pf_token_norm
#endif
#define PF_TOK_WARPS (PF_TOK_SPLIT > 4 ? PF_TOK_SPLIT : 4)        // warps per CTA of the per-token kernels
#define PF_TOK_PER_CTA (PF_TOK_WARPS / PF_TOK_SPLIT)

// MODE 0: norm of X.  MODE 1: X += sum_k w[4t+k] * D[4t+k] first (rank-order chain), then the norm.
// MODE 2: as 1 with the row of slot 4t+k found through pos[].  PF_TOK_SPLIT warps share a token (consecutive runs of blocks): each quantises u = x * nw per block and leaves each block's sum of squares of x in shared memory;
// after a named barrier over the token's warps the first warp of the token ends with 1/rms from the 64 partials in the decode
// kernels' order ((ssq[l] + ssq[l+32]) butterflied over l).
template <int MODE>
__global__ void __launch_bounds__(PF_TOK_WARPS * 32) k_pf_token_norm(float * __restrict__ X, const float * __restrict__ D,
                                                                      const int * __restrict__ pos, const float * __restrict__ wts,
                                                                      const float * __restrict__ nw, int8_t * __restrict__ aqs,
                                                                      float2 * __restrict__ asc, float * __restrict__ inv_out,
                                                                      float * __restrict__ h32, int m) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    __shared__ float s_sq[PF_TOK_PER_CTA][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tl = warp / PF_TOK_SPLIT, part = warp % PF_TOK_SPLIT;
    const int t = blockIdx.x * PF_TOK_PER_CTA + tl;
    if (t >= m) return;                                   // all warps of the token leave together
    float4 * x4 = reinterpret_cast<float4 *>(X + (size_t) t * LKB_HIDDEN);
    const float4 * w4 = reinterpret_cast<const float4 *>(nw);
    unsigned * q4 = reinterpret_cast<unsigned *>(aqs + (size_t) t * LKB_HIDDEN);
    float2 * sc = asc + (size_t) t * (LKB_HIDDEN / 32);
    float4 * h4 = (MODE == 0 && h32) ? reinterpret_cast<float4 *>(h32 + (size_t) t * LKB_HIDDEN) : nullptr;
    const float4 * d4[LKB_TOP_K]; float wk[LKB_TOP_K];
    if (MODE) {
#pragma unroll
        for (int k = 0; k < LKB_TOP_K; ++k) {
            wk[k] = wts[t * 4 + k];
            const int row = (MODE == 2) ? pos[t * 4 + k] : t * 4 + k;
            d4[k] = reinterpret_cast<const float4 *>(D + (size_t) row * LKB_HIDDEN);
        }
    }
    constexpr int STEPS = LKB_HIDDEN / 128 / PF_TOK_SPLIT;
#pragma unroll
    for (int s = part * STEPS; s < part * STEPS + STEPS; ++s) {
        const int i4 = s * 32 + lane;
        float4 xv = x4[i4];
        if (MODE) {
            float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < LKB_TOP_K; ++k) {
                const float4 dv = d4[k][i4];
                a.x = fmaf(wk[k], dv.x, a.x); a.y = fmaf(wk[k], dv.y, a.y);
                a.z = fmaf(wk[k], dv.z, a.z); a.w = fmaf(wk[k], dv.w, a.w);
            }
            xv = make_float4(__fadd_rn(xv.x, a.x), __fadd_rn(xv.y, a.y), __fadd_rn(xv.z, a.z), __fadd_rn(xv.w, a.w));
            x4[i4] = xv;
        }
        const float4 wv = __ldg(w4 + i4);
        const float4 u = make_float4(__fmul_rn(xv.x, wv.x), __fmul_rn(xv.y, wv.y), __fmul_rn(xv.z, wv.z), __fmul_rn(xv.w, wv.w));
        if (h4) h4[i4] = u;
        float2 s2;
        q4[i4] = lkb_quad_quant(u, lane, s2);
        const float sq = lkb_quad_sum(__fmul_rn(xv.x, xv.x), __fmul_rn(xv.y, xv.y), __fmul_rn(xv.z, xv.z), __fmul_rn(xv.w, xv.w));
        if ((lane & 7) == 0) { sc[s * 4 + (lane >> 3)] = s2; s_sq[tl][s * 4 + (lane >> 3)] = sq; }
    }
    asm volatile("bar.sync %0, %1;" :: "r"(1 + tl), "n"(32 * PF_TOK_SPLIT) : "memory");
    if (part == 0) {
        const float sv = lkb_warp_sum(__fadd_rn(s_sq[tl][lane], s_sq[tl][lane + 32]));
        if (lane == 0) inv_out[t] = rsqrtf(fmaf(sv, 1.0f / (float) LKB_HIDDEN, LKB_EPS));
    }
}

// Layer-0 form: normalise first (x * inv) * w, quantise that, report scale 1.  The sum of squares keeps the
// order of a 256-wide reduction (element i in chain i mod 256, chains folded 128 / 64 / 32 apart, then the
// butterfly): lane l runs the eight chains l + 32g and folds them in registers.
__global__ void __launch_bounds__(PF_TOK_WARPS * 32) k_pf_token_norm_plain(const float * __restrict__ X, const float * __restrict__ nw,
                                                                            int8_t * __restrict__ aqs, float2 * __restrict__ asc,
                                                                            float * __restrict__ inv_out, int m) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * PF_TOK_WARPS + (threadIdx.x >> 5);
    if (t >= m) return;
    const float * x = X + (size_t) t * LKB_HIDDEN;
    float S[8];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        S[g] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) { const float xv = x[lane + 32 * g + 256 * j]; S[g] = fmaf(xv, xv, S[g]); }
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) S[g] = __fadd_rn(S[g], S[g + 4]);
    S[0] = __fadd_rn(S[0], S[2]); S[1] = __fadd_rn(S[1], S[3]);
    const float ss = lkb_warp_sum(__fadd_rn(S[0], S[1]));
    const float inv = rsqrtf(fmaf(ss, 1.0f / (float) LKB_HIDDEN, LKB_EPS));
    const float4 * x4 = reinterpret_cast<const float4 *>(x);
    const float4 * w4 = reinterpret_cast<const float4 *>(nw);
    unsigned * q4 = reinterpret_cast<unsigned *>(aqs + (size_t) t * LKB_HIDDEN);
    float2 * sc = asc + (size_t) t * (LKB_HIDDEN / 32);
#pragma unroll 4
    for (int s = 0; s < LKB_HIDDEN / 128; ++s) {
        const int i4 = s * 32 + lane;
        const float4 xv = x4[i4], wv = __ldg(w4 + i4);
        const float4 u = make_float4(__fmul_rn(__fmul_rn(xv.x, inv), wv.x), __fmul_rn(__fmul_rn(xv.y, inv), wv.y),
                                     __fmul_rn(__fmul_rn(xv.z, inv), wv.z), __fmul_rn(__fmul_rn(xv.w, inv), wv.w));
        float2 s2;
        q4[i4] = lkb_quad_quant(u, lane, s2);
        if ((lane & 7) == 0) sc[s * 4 + (lane >> 3)] = s2;
    }
    if (lane == 0) inv_out[t] = 1.0f;
}

// Row quantisers: a warp takes four adjacent blocks of one row (SWIGLU: of silu(gate) * up, the two halves of a
// row up_off apart).  Rows x ceil(kb / 4) warps, 8 per CTA.
template <int SWIGLU>
__global__ void __launch_bounds__(256) k_pf_rows_q8(const float * __restrict__ Y, int ld, int up_off, int kb, int rows,
                                                    int8_t * __restrict__ aqs, float2 * __restrict__ asc) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    const int lane = threadIdx.x & 31;
    const int gpr = (kb + 3) >> 2;
    const long long wid = (long long) blockIdx.x * 8 + (threadIdx.x >> 5);
    if (wid >= (long long) rows * gpr) return;
    const int r = (int) (wid / gpr), g = (int) (wid - (long long) r * gpr);
    const int b = g * 4 + (lane >> 3);
    const bool live = b < kb;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (live) {
        const float * y = Y + (size_t) r * ld + b * 32 + (lane & 7) * 4;
        v = *reinterpret_cast<const float4 *>(y);
        if (SWIGLU) {
            const float4 up = *reinterpret_cast<const float4 *>(y + up_off);
            v = make_float4(__fmul_rn(lkb_silu(v.x), up.x), __fmul_rn(lkb_silu(v.y), up.y),
                            __fmul_rn(lkb_silu(v.z), up.z), __fmul_rn(lkb_silu(v.w), up.w));
        }
    }
    float2 s2;
    const unsigned pk = lkb_quad_quant(v, lane, s2);
    if (live) {
        reinterpret_cast<unsigned *>(aqs + (size_t) r * kb * 32 + b * 32)[lane & 7] = pk;
        if ((lane & 7) == 0) asc[(size_t) r * kb + b] = s2;
    }
}

// ---------------------------------------------------------------------------
// Router.  Short form for a few tokens: a CTA per token keeps the token's activation in registers (64 per lane)
// and each warp walks eight expert rows over it; a logit is the decode router's sum (lane l chains elements
// l, l+32, ... ascending, then the butterfly), so it is bit-identical to it.  ref semantics: src/prefill.cu:1668-1693
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_pf_router_token(const float * __restrict__ H, const float * __restrict__ Wr,
                                                         const float * __restrict__ bias, const float * __restrict__ inv,
                                                         float * __restrict__ sel, float * __restrict__ sig,
                                                         int4 * __restrict__ idx, float4 * __restrict__ wout) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    __shared__ float s_sel[LKB_N_EXPERTS], s_sig[LKB_N_EXPERTS];
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float * h = H + (size_t) t * LKB_HIDDEN;
    float hv[LKB_HIDDEN / 32];
#pragma unroll
    for (int j = 0; j < LKB_HIDDEN / 32; ++j) hv[j] = h[j * 32 + lane];
    float mine = 0.0f;
    for (int q = 0; q < 8; ++q) {
        const float * row = Wr + (size_t) (warp * 8 + q) * LKB_HIDDEN;
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < LKB_HIDDEN / 32; ++j) acc = fmaf(__ldg(row + j * 32 + lane), hv[j], acc);
        acc = lkb_warp_sum(acc);
        if (lane == q) mine = acc;
    }
    if (lane < 8) {
        const int e = warp * 8 + lane;
        const float l = __fmul_rn(mine, inv[t]);
        const float gv = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-l)));
        const float sv = __fadd_rn(gv, bias[e]);
        sig[(size_t) t * 64 + e] = gv;
        sel[(size_t) t * 64 + e] = sv;
        s_sig[e] = gv; s_sel[e] = sv;
    }
    if (idx) {                                             // the selection in the same launch (lkb_pf_select's result)
        __syncthreads();
        if (warp == 0) {
            int ord[LKB_TOP_K]; float wv[LKB_TOP_K];
            lkb_router_select(s_sel, s_sig, lane, ord, wv);
            if (lane == 0) { idx[t] = make_int4(ord[0], ord[1], ord[2], ord[3]); wout[t] = make_float4(wv[0], wv[1], wv[2], wv[3]); }
        }
    }
}

// The same for fewer tokens still: a cluster of eight CTAs per token, a warp per expert.  The selection needs all 64 logits: they meet in
// the shared memory of the cluster's first CTA.  Bound by the latency of a warp's two rows; see router_small for where it pays.
#define RC_CTAS 8
__global__ void __cluster_dims__(RC_CTAS, 1, 1) __launch_bounds__(256) k_pf_router_cluster(const float * __restrict__ H, const float * __restrict__ Wr,
                                                         const float * __restrict__ bias, const float * __restrict__ inv,
                                                         float * __restrict__ sel, float * __restrict__ sig,
                                                         int4 * __restrict__ idx, float4 * __restrict__ wout) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    __shared__ float s_sel[LKB_N_EXPERTS], s_sig[LKB_N_EXPERTS];
    if (idx) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");       // the first CTA runs before its memory is written
    const int t = blockIdx.x / RC_CTAS, rank = blockIdx.x % RC_CTAS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = rank * 8 + warp;
    const float * h = H + (size_t) t * LKB_HIDDEN, * row = Wr + (size_t) e * LKB_HIDDEN;
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < LKB_HIDDEN / 32; ++j) acc = fmaf(__ldg(row + j * 32 + lane), h[j * 32 + lane], acc);
    acc = lkb_warp_sum(acc);
    if (idx) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (lane == 0) {
        const float l = __fmul_rn(acc, inv[t]);
        const float gv = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-l)));
        const float sv = __fadd_rn(gv, bias[e]);
        sig[(size_t) t * 64 + e] = gv;
        sel[(size_t) t * 64 + e] = sv;
        if (idx) {
            unsigned a, b;
            asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"((unsigned) __cvta_generic_to_shared(&s_sig[e])));
            asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(b) : "r"((unsigned) __cvta_generic_to_shared(&s_sel[e])));
            asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(a), "f"(gv) : "memory");
            asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(b), "f"(sv) : "memory");
        }
    }
    if (idx) {                                             // the selection in the same launch (lkb_pf_select's result)
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (rank == 0 && warp == 0) {
            int ord[LKB_TOP_K]; float wv[LKB_TOP_K];
            lkb_router_select(s_sel, s_sig, lane, ord, wv);
            if (lane == 0) { idx[t] = make_int4(ord[0], ord[1], ord[2], ord[3]); wout[t] = make_float4(wv[0], wv[1], wv[2], wv[3]); }
        }
    }
}

// ffn_norm (k_pf_token_norm<0>) and the router above in one launch, while a cluster of eight CTAs a token is the form: each CTA forms u = x * w itself for
// its eight experts' rows, quantises an eighth of it, and the first one gets logits and blocks' sums of squares through its shared memory and
// ends with 1 / rms, the gates and the selection.  Same sums in the same order.  Two launches took 5.5 + 8.5 us at 9 tokens and 5.7 + 8.2 at 37 (ncu), this 5.9 and 8.4.
__global__ void __cluster_dims__(RC_CTAS, 1, 1) __launch_bounds__(256) k_pf_norm_router_cluster(const float * __restrict__ X, const float * __restrict__ nw,
                                                         int8_t * __restrict__ aqs, float2 * __restrict__ asc, float * __restrict__ inv_out,
                                                         const float * __restrict__ Wr, const float * __restrict__ bias,
                                                         float * __restrict__ sel, float * __restrict__ sig,
                                                         int4 * __restrict__ idx, float4 * __restrict__ wout) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    __shared__ float s_u[LKB_HIDDEN], s_acc[LKB_N_EXPERTS], s_sq[LKB_HIDDEN / 32], s_sel[LKB_N_EXPERTS], s_sig[LKB_N_EXPERTS];
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");                // the first CTA runs before its memory is written
    const int t = blockIdx.x / RC_CTAS, rank = blockIdx.x % RC_CTAS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = rank * 8 + warp;
    const float4 * x4 = reinterpret_cast<const float4 *>(X + (size_t) t * LKB_HIDDEN), * w4 = reinterpret_cast<const float4 *>(nw);
    const float * row = Wr + (size_t) e * LKB_HIDDEN;
    auto to_first = [](float * p, float v) {
        unsigned a;
        asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"((unsigned) __cvta_generic_to_shared(p)));
        asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(a), "f"(v) : "memory");
    };
    float r[LKB_HIDDEN / 32];
#pragma unroll
    for (int j = 0; j < LKB_HIDDEN / 32; ++j) r[j] = __ldg(row + j * 32 + lane);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float4 xv = x4[threadIdx.x + 256 * j], wv = __ldg(w4 + threadIdx.x + 256 * j);
        reinterpret_cast<float4 *>(s_u)[threadIdx.x + 256 * j] = make_float4(__fmul_rn(xv.x, wv.x), __fmul_rn(xv.y, wv.y), __fmul_rn(xv.z, wv.z), __fmul_rn(xv.w, wv.w));
    }
    float sq = 0.0f;
    if (warp < 2) {                                        // the CTA's eight blocks, four a warp
        const int i4 = (rank * 8 + warp * 4) * 8 + lane;
        const float4 xv = x4[i4], wv = __ldg(w4 + i4);
        float2 s2;
        reinterpret_cast<unsigned *>(aqs + (size_t) t * LKB_HIDDEN)[i4] = lkb_quad_quant(make_float4(__fmul_rn(xv.x, wv.x), __fmul_rn(xv.y, wv.y), __fmul_rn(xv.z, wv.z), __fmul_rn(xv.w, wv.w)), lane, s2);
        sq = lkb_quad_sum(__fmul_rn(xv.x, xv.x), __fmul_rn(xv.y, xv.y), __fmul_rn(xv.z, xv.z), __fmul_rn(xv.w, xv.w));
        if ((lane & 7) == 0) asc[(size_t) t * (LKB_HIDDEN / 32) + rank * 8 + warp * 4 + (lane >> 3)] = s2;
    }
    __syncthreads();
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < LKB_HIDDEN / 32; ++j) acc = fmaf(r[j], s_u[j * 32 + lane], acc);
    acc = lkb_warp_sum(acc);
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (lane == 0) to_first(&s_acc[e], acc);
    if (warp < 2 && (lane & 7) == 0) to_first(&s_sq[rank * 8 + warp * 4 + (lane >> 3)], sq);
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank == 0 && warp == 0) {
        const float sv = lkb_warp_sum(__fadd_rn(s_sq[lane], s_sq[lane + 32])), inv = rsqrtf(fmaf(sv, 1.0f / (float) LKB_HIDDEN, LKB_EPS));
#pragma unroll
        for (int q = lane; q < LKB_N_EXPERTS; q += 32) {
            const float l = __fmul_rn(s_acc[q], inv);
            const float gv = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-l)));
            const float v = __fadd_rn(gv, bias[q]);
            sig[(size_t) t * 64 + q] = gv;
            sel[(size_t) t * 64 + q] = v;
            s_sig[q] = gv; s_sel[q] = v;
        }
        __syncwarp();
        int ord[LKB_TOP_K]; float wv[LKB_TOP_K];
        lkb_router_select(s_sel, s_sig, lane, ord, wv);
        if (lane == 0) { idx[t] = make_int4(ord[0], ord[1], ord[2], ord[3]); wout[t] = make_float4(wv[0], wv[1], wv[2], wv[3]); inv_out[t] = inv; }
    }
}

// Tiled form.  Each (token, expert) logit is one FMA chain over k = 0..2047 ascending (reference semantics:
// src/prefill.cu:1606-1666, same per-logit order), so a CTA runs a long sequential k loop and the kernel is bound by
// (a) how well the loads of the next k-tiles hide behind the FMAs of the current one and (b) how many FMAs each
// shared-memory wavefront feeds.  CTA = NW warps = 2 NW token groups x 16 expert lanes; a thread owns TPT tokens x the
// four experts (lane, lane + 16, + 32, + 48): 4 * TPT independent chains.  Tiles of RT_KT k-values of the CTA's token
// rows and of all 64 router rows travel global -> shared by 16-byte asynchronous copies through a ring of RT_STAGES
// buffers (rows keep their [row][k] layout, pitch RT_KT + 4 floats: nothing is transposed and 128-bit loads of 16 different
// rows are conflict-free); the multiply loop reads four k-values per load.  Instantiated for 4-token CTAs
// (TPT = 1: up to 592 tokens, one wave); larger ones take k_pf_router_tma below.  One CTA barrier per tile.
// A tile holds KT k-values, the ring STAGES of them: what a tile costs beside its FMAs (a barrier, the copies' issue) is paid
// less often with wide tiles, which small CTAs have the shared memory for (see router_tiled).
__device__ __forceinline__ void rt_cp16(float * dst, const float * src, bool live) {
    const unsigned d = (unsigned) __cvta_generic_to_shared(dst);
    const int n = live ? 16 : 0;                          // 0: the 16 bytes are zero-filled, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d), "l"(src), "r"(n) : "memory");
}
template <int TPT, int NW, int RT_KT, int RT_STAGES>
__global__ void __launch_bounds__(32 * NW) k_pf_router_pipe(const float * __restrict__ H, int m, const float * __restrict__ Wr,
                                                        const float * __restrict__ bias, const float * __restrict__ inv,
                                                        float * __restrict__ sel, float * __restrict__ sig,
                                                        int4 * __restrict__ idx, float4 * __restrict__ wout) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    constexpr int RT_PITCH = RT_KT + 4, RT_CPR = RT_KT / 4;            // floats and 16-byte copies per staged row
    constexpr int TT = 2 * NW * TPT, ROWS = TT + LKB_N_EXPERTS, NTILES = LKB_HIDDEN / RT_KT;
    extern __shared__ __align__(16) float rt_ring[];                   // [RT_STAGES][ROWS][RT_PITCH]
    const int tid = threadIdx.x, te = tid & 15, tg = tid >> 4;
    const int t0 = blockIdx.x * TT;
    // a thread copies the same (row, 16-byte part) set of every tile: sources and ring offsets are computed once
    constexpr int NCP = (ROWS * RT_CPR + 32 * NW - 1) / (32 * NW);
    const float * src[NCP]; int dst[NCP]; bool live[NCP];
#pragma unroll
    for (int j = 0; j < NCP; ++j) {
        const int ch = tid + j * 32 * NW;
        const int row = ch / RT_CPR, part = (ch % RT_CPR) * 4;
        dst[j] = (ch < ROWS * RT_CPR) ? row * RT_PITCH + part : -1;
        if (row < TT) { const int tk = t0 + row; live[j] = tk < m; src[j] = H + (size_t) (tk < m ? tk : 0) * LKB_HIDDEN + part; }
        else          { live[j] = true; src[j] = Wr + (size_t) (row < ROWS ? row - TT : 0) * LKB_HIDDEN + part; }
    }
    auto issue = [&](int tile) {
        if (tile < NTILES) {
            float * st = rt_ring + (size_t) (tile % RT_STAGES) * ROWS * RT_PITCH;
            const int k0 = tile * RT_KT;
#pragma unroll
            for (int j = 0; j < NCP; ++j)
                if (dst[j] >= 0) rt_cp16(st + dst[j], src[j] + k0, live[j]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");      // (an empty group keeps the count uniform)
    };
    float acc[TPT][4];
#pragma unroll
    for (int i = 0; i < TPT; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = 0.0f;
#pragma unroll
    for (int s = 0; s < RT_STAGES - 1; ++s) issue(s);
    for (int tile = 0; tile < NTILES; ++tile) {
        asm volatile("cp.async.wait_group %0;" :: "n"(RT_STAGES - 2) : "memory");
        __syncthreads();                   // this tile has landed for everyone; the stage refilled below is no longer read
        issue(tile + RT_STAGES - 1);
        const float * st = rt_ring + (size_t) (tile % RT_STAGES) * ROWS * RT_PITCH;
        const float * sh = st + (tg * TPT) * RT_PITCH, * sw = st + (TT + te) * RT_PITCH;
#pragma unroll
        for (int c = 0; c < RT_KT; c += 4) {
            float4 w[4], h[TPT];
#pragma unroll
            for (int q = 0; q < 4; ++q) w[q] = *reinterpret_cast<const float4 *>(sw + 16 * q * RT_PITCH + c);
#pragma unroll
            for (int i = 0; i < TPT; ++i) h[i] = *reinterpret_cast<const float4 *>(sh + i * RT_PITCH + c);
            // k-major order: consecutive FMAs belong to different chains, so none waits for its predecessor
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(h[i].x, w[q].x, acc[i][q]);
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(h[i].y, w[q].y, acc[i][q]);
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(h[i].z, w[q].z, acc[i][q]);
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(h[i].w, w[q].w, acc[i][q]);
        }
    }
    // the ring is free after the last tile: the CTA's sel / sig rows pass through it to the selection warps
    float * s_sel = rt_ring, * s_sig = rt_ring + TT * LKB_N_EXPERTS;
    if (idx) __syncthreads();
#pragma unroll
    for (int i = 0; i < TPT; ++i) {
        const int tl = tg * TPT + i, tk = t0 + tl;
        if (tk >= m) continue;
        const float iv = inv[tk];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = te + 16 * q;
            const float l = __fmul_rn(acc[i][q], iv);
            const float gv = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-l)));
            const float sv = __fadd_rn(gv, bias[e]);
            sig[(size_t) tk * 64 + e] = gv;
            sel[(size_t) tk * 64 + e] = sv;
            if (idx) { s_sig[tl * LKB_N_EXPERTS + e] = gv; s_sel[tl * LKB_N_EXPERTS + e] = sv; }
        }
    }
    if (idx) {                                             // the selection in the same launch (lkb_pf_select's result)
        __syncthreads();
        const int warp = tid >> 5, lane = tid & 31;
        for (int tl = warp; tl < TT; tl += NW) {
            const int tk = t0 + tl;
            if (tk >= m) break;
            int ord[LKB_TOP_K]; float wv[LKB_TOP_K];
            lkb_router_select(s_sel + tl * LKB_N_EXPERTS, s_sig + tl * LKB_N_EXPERTS, lane, ord, wv);
            if (lane == 0) { idx[tk] = make_int4(ord[0], ord[1], ord[2], ord[3]); wout[tk] = make_float4(wv[0], wv[1], wv[2], wv[3]); }
        }
    }
}
template <int TPT, int NW, int KT, int STAGES>
static int rt_launch(const float * H, int m, const float * Wr, const float * bias, const float * inv, float * sel, float * sig,
                     int * idx, float * w, cudaStream_t st) {
    constexpr int TT = 2 * NW * TPT;
    constexpr size_t smem = (size_t) STAGES * (TT + LKB_N_EXPERTS) * (KT + 4) * sizeof(float);
    static int ready[LKB_STATIC_MAX_DEVICES] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < LKB_STATIC_MAX_DEVICES && !ready[dev]) {
        if (cudaFuncSetAttribute(k_pf_router_pipe<TPT, NW, KT, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem) != cudaSuccess) return -(int) cudaGetLastError();
        ready[dev] = 1;
    }
    LKB_PF_LAUNCH((k_pf_router_pipe<TPT, NW, KT, STAGES>), dim3((m + TT - 1) / TT), dim3(32 * NW), smem, st, H, m, Wr, bias, inv, sel, sig,
                  reinterpret_cast<int4 *>(idx), reinterpret_cast<float4 *>(w));
    return lkb_check_launch();
}

// Tiled form of longer chunks: the same chains, bound by
// shared memory's return path: a 128-bit load writes 512 bytes of registers, four cycles of the SM's, whatever it reads, so the eight loads
// of a thread's 4 tokens x 4 experts x 4 k-values cost the four warps 128 cycles and their 64 FMAs each 64.  CTA = NW warps of 4 TPT tokens x
// 32 experts (a thread: tokens l / 8, + 4, ..., experts l % 8, + 8, + 16, + 24), 4 * TPT independent chains a thread, and one warp that copies:
// k-tiles of the CTA's token rows and of all 64 router rows travel global -> shared by tensor copies, 128 bytes of every row at a time
// (swizzled: 128-bit loads of eight neighbouring rows are conflict-free), through a ring of RT_STAGES buffers handed over by mbarriers.
// us, calls back to back, at 1184 / 2048 / 4096 / 8192 tokens: 29.7 / 35.2 / 53.4 / 105 in the form above, 25.2 / 28.8 / 43.3 / 85 here (in an earlier run, where this took
// 26.9 / 30.5 / 44.6 / 86, 16 / 17 / 22 / 39 without the shared loads; with a bulk copy per row, 67 cycles each, 44 / 54 / 118 / 234).  At 509 tokens 21.2 there,
// 27.8 here with the same four-token CTAs.
// Waits are bounded; on expiry a status word is set and all roles leave, the copying warp after its copies have landed.
__device__ __forceinline__ float4 rt_lds(unsigned addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
template <int TPT, int NW, int RT_KT, int RT_STAGES> struct RtShape {
    static constexpr int TT = 2 * NW * TPT, H_BYTES = (TT * 128 + 1023) / 1024 * 1024, SUB = LKB_N_EXPERTS * 128 + H_BYTES;    // 32 k-values: router rows, token rows
    static constexpr int STAGE = RT_KT / 32 * SUB, NTILES = LKB_HIDDEN / RT_KT;
    static constexpr size_t SMEM = (size_t) RT_STAGES * STAGE + 1024;
};
template <int TPT, int NW, int RT_KT, int RT_STAGES>
__global__ void __launch_bounds__(32 * NW + 32) k_pf_router_tma(int m, const __grid_constant__ CUtensorMap map_h, const __grid_constant__ CUtensorMap map_w,
                                                        const float * __restrict__ bias, const float * __restrict__ inv,
                                                        float * __restrict__ sel, float * __restrict__ sig,
                                                        int4 * __restrict__ idx, float4 * __restrict__ wout) {
    using F = RtShape<TPT, NW, RT_KT, RT_STAGES>;
    constexpr int TT = F::TT, NTILES = F::NTILES;
    extern __shared__ unsigned char rt_raw[];
    unsigned char * const ring = rt_raw + ((1024u - (tc_smem_u32(rt_raw) & 1023u)) & 1023u);         // swizzled tiles start on 1024-byte boundaries
    __shared__ alignas(8) unsigned long long full[RT_STAGES], empty[RT_STAGES];
    __shared__ struct { int abort; } S;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, te = (warp & 1) * 32 + (lane & 7), tg = (warp >> 1) * (4 * TPT) + (lane >> 3);
    const int t0 = blockIdx.x * TT;
    if (tid == 0) {
        S.abort = 0;
        for (int i = 0; i < RT_STAGES; ++i) { tc_mbar_init(&full[i], 1); tc_mbar_init(&empty[i], NW); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    float acc[TPT][4];
#pragma unroll
    for (int i = 0; i < TPT; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = 0.0f;
    if (warp == NW) {
        int tile = 0;
        for (; tile < NTILES; ++tile) {
            const int stg = tile % RT_STAGES;
            if (!tc_wait<TC_HINT_PROD>(S, &empty[stg], ((unsigned) (tile / RT_STAGES) & 1u) ^ 1u, 41u)) break;
            if (lane == 0) tc_mbar_arrive_tx(&full[stg], (TT + LKB_N_EXPERTS) * RT_KT * 4);
            __syncwarp();
            unsigned char * const st = ring + stg * F::STAGE;
            if (lane < RT_KT / 32) {                                   // lane: 32 k-values (tokens past the chunk read as zero)
                tc_tma_tile(st + lane * F::SUB, &map_w, (tile * RT_KT + lane * 32) * 4, 0, &full[stg]);
                tc_tma_tile(st + lane * F::SUB + LKB_N_EXPERTS * 128, &map_h, (tile * RT_KT + lane * 32) * 4, t0, &full[stg]);
            }
        }
        tc_drain<RT_STAGES>(full, tile);
    } else for (int tile = 0; tile < NTILES; ++tile) {
        const int stg = tile % RT_STAGES;
        if (!tc_wait(S, &full[stg], (unsigned) (tile / RT_STAGES) & 1u, 42u)) break;
        const unsigned st = tc_smem_u32(ring) + stg * F::STAGE, sw = st + te * 128 + ((te & 7) << 4);
        float4 w[2][4], h[2][TPT];                          // four k-values in use, the next four on their way
        auto load = [&](int b, int c) {
            const unsigned at = (c >> 5) * F::SUB, part = ((c >> 2) & 7) << 4;
#pragma unroll
            for (int q = 0; q < 4; ++q) w[b][q] = rt_lds((sw ^ part) + at + q * (8 * 128));
#pragma unroll
            for (int i = 0; i < TPT; ++i) {
                const int row = tg + 4 * i;
                h[b][i] = rt_lds(((st + LKB_N_EXPERTS * 128 + row * 128 + ((row & 7) << 4)) ^ part) + at);
            }
        };
        load(0, 0);
#pragma unroll
        for (int c = 0; c < RT_KT; c += 4) {
            const int b = (c >> 2) & 1;
            if (c + 4 < RT_KT) load(b ^ 1, c + 4);
            // k-major order: consecutive FMAs belong to different chains, so none waits for its predecessor
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(h[b][i].x, w[b][q].x, acc[i][q]);
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(h[b][i].y, w[b][q].y, acc[i][q]);
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(h[b][i].z, w[b][q].z, acc[i][q]);
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(h[b][i].w, w[b][q].w, acc[i][q]);
        }
        __syncwarp();
        tc_mbar_arrive_if(&empty[stg], lane == 0);
    }
    // the ring is free after the last tile: the CTA's sel / sig rows pass through it to the selection warps
    float * s_sel = reinterpret_cast<float *>(ring), * s_sig = s_sel + TT * LKB_N_EXPERTS;
    if (idx) __syncthreads();
    if (warp < NW)
#pragma unroll
    for (int i = 0; i < TPT; ++i) {
        const int tl = tg + 4 * i, tk = t0 + tl;
        if (tk >= m) continue;
        const float iv = inv[tk];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = te + 8 * q;
            const float l = __fmul_rn(acc[i][q], iv);
            const float gv = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-l)));
            const float sv = __fadd_rn(gv, bias[e]);
            sig[(size_t) tk * 64 + e] = gv;
            sel[(size_t) tk * 64 + e] = sv;
            if (idx) { s_sig[tl * LKB_N_EXPERTS + e] = gv; s_sel[tl * LKB_N_EXPERTS + e] = sv; }
        }
    }
    if (idx) {                                             // the selection in the same launch (lkb_pf_select's result)
        __syncthreads();
        for (int tl = warp; tl < TT; tl += NW + 1) {
            const int tk = t0 + tl;
            if (tk >= m) break;
            int ord[LKB_TOP_K]; float wv[LKB_TOP_K];
            lkb_router_select(s_sel + tl * LKB_N_EXPERTS, s_sig + tl * LKB_N_EXPERTS, lane, ord, wv);
            if (lane == 0) { idx[tk] = make_int4(ord[0], ord[1], ord[2], ord[3]); wout[tk] = make_float4(wv[0], wv[1], wv[2], wv[3]); }
        }
    }
}
int lkb_tc_make_map(CUtensorMap * m, const void * base, unsigned row_bytes, unsigned long long pitch, unsigned long long rows,
                    unsigned box_bytes, unsigned box_rows, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2);           // lkb_gemm_tc.cu
template <int TPT, int NW, int KT, int STAGES>
static int rt_launch_tma(const float * H, int m, const float * Wr, const float * bias, const float * inv, float * sel, float * sig,
                     int * idx, float * w, cudaStream_t st) {
    using F = RtShape<TPT, NW, KT, STAGES>;
    static int ready[LKB_STATIC_MAX_DEVICES] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < LKB_STATIC_MAX_DEVICES && !ready[dev]) {
        if (cudaFuncSetAttribute(k_pf_router_tma<TPT, NW, KT, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) F::SMEM) != cudaSuccess) return -(int) cudaGetLastError();
        ready[dev] = 1;
    }
    if (((size_t) H | (size_t) Wr) & 15) return LKB_ERR_SHAPE;         // 16-byte copies of the rows
    CUtensorMap mh, mw;
    int r = lkb_tc_make_map(&mh, H, LKB_HIDDEN * 4, LKB_HIDDEN * 4, (unsigned long long) m, 128u, F::TT, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (r == LKB_OK) r = lkb_tc_make_map(&mw, Wr, LKB_HIDDEN * 4, LKB_HIDDEN * 4, LKB_N_EXPERTS, 128u, LKB_N_EXPERTS, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (r != LKB_OK) return r;
    LKB_PF_LAUNCH((k_pf_router_tma<TPT, NW, KT, STAGES>), dim3((m + F::TT - 1) / F::TT), dim3(32 * NW + 32), F::SMEM, st, m, mh, mw, bias, inv, sel, sig,
                  reinterpret_cast<int4 *>(idx), reinterpret_cast<float4 *>(w));
    return lkb_check_launch();
}

// Top-4 of 64 per token: warps stride over the tokens (any grid); the selection itself is the redux-based
// lkb_router_select shared with the decode router.  ref semantics: src/prefill.cu:1696-1708
__global__ void __launch_bounds__(256) k_pf_select(const float * __restrict__ sel, const float * __restrict__ sig, int m,
                                                   int4 * __restrict__ idx, float4 * __restrict__ w) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < m; t += nw) {
        int ord[LKB_TOP_K]; float wv[LKB_TOP_K];
        lkb_router_select(sel + (size_t) t * 64, sig + (size_t) t * 64, lane, ord, wv);
        if (lane == 0) {
            idx[t] = make_int4(ord[0], ord[1], ord[2], ord[3]);
            w[t] = make_float4(wv[0], wv[1], wv[2], wv[3]);
        }
    }
}

// ---------------------------------------------------------------------------
// count / plan / scatter.  ref: src/prefill.cu:1710-1756
// ---------------------------------------------------------------------------
// Per-CTA shared histogram, then 64 global atomics per CTA (integer: order-free).
__global__ void __launch_bounds__(256) k_pf_moe_count(const int * __restrict__ idx, int n, int * __restrict__ cnt) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    __shared__ int s_c[LKB_N_EXPERTS];
    if (threadIdx.x < LKB_N_EXPERTS) s_c[threadIdx.x] = 0;
    __syncthreads();
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) atomicAdd(&s_c[idx[s]], 1);
    __syncthreads();
    if (threadIdx.x < LKB_N_EXPERTS && s_c[threadIdx.x]) atomicAdd(&cnt[threadIdx.x], s_c[threadIdx.x]);
}

// One warp: exclusive scan over the 64 counts (lane: experts lane and lane + 32), then tiles in expert order.
__device__ __forceinline__ void pf_plan_warp(int lane, int c0, int c1, int * off, int4 * tiles, int * ntiles) {
    const int n0 = (c0 + LKB_MOE_BN - 1) / LKB_MOE_BN, n1 = (c1 + LKB_MOE_BN - 1) / LKB_MOE_BN;
    // inclusive scans over lanes for experts 0..31, then offset experts 32..63
    int so = c0, st = n0, so1 = c1, st1 = n1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(LKB_FULL, so, o), b = __shfl_up_sync(LKB_FULL, st, o);
        const int c = __shfl_up_sync(LKB_FULL, so1, o), d = __shfl_up_sync(LKB_FULL, st1, o);
        if (lane >= o) { so += a; st += b; so1 += c; st1 += d; }
    }
    const int tot_o = __shfl_sync(LKB_FULL, so, 31), tot_t = __shfl_sync(LKB_FULL, st, 31);
    const int off0 = so - c0, off1 = tot_o + so1 - c1;
    const int tb0 = st - n0, tb1 = tot_t + st1 - n1;
    off[lane] = off0; off[lane + 32] = off1;
    for (int i = 0; i < n0; ++i)
        tiles[tb0 + i] = make_int4(lane, off0 + i * LKB_MOE_BN, min(LKB_MOE_BN, c0 - i * LKB_MOE_BN), 0);
    for (int i = 0; i < n1; ++i)
        tiles[tb1 + i] = make_int4(lane + 32, off1 + i * LKB_MOE_BN, min(LKB_MOE_BN, c1 - i * LKB_MOE_BN), 0);
    if (lane == 31) *ntiles = tot_t + st1;
}
__global__ void __launch_bounds__(32) k_pf_moe_plan(const int * __restrict__ cnt, int * __restrict__ off,
                                                    int4 * __restrict__ tiles, int * __restrict__ ntiles) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    pf_plan_warp(threadIdx.x, cnt[threadIdx.x], cnt[threadIdx.x + 32], off, tiles, ntiles);
}

// Stable scatter.  CTA c owns slots [1024c, 1024c+1024): it histograms every
// earlier slot (L2-resident reads) to learn how many slots of each expert precede
// its chunk, ranks its own slots with match_any, and writes perm.  Result:
// expert-major, slot-ascending within an expert -- identical to the reference's
// per-expert compaction (ref: src/prefill.cu:1733-1756) without re-reading idx 64x.
__global__ void __launch_bounds__(1024) k_pf_moe_scatter(const int * __restrict__ idx, int n, const int * __restrict__ off,
                                                         int * __restrict__ perm) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    if ((int) blockIdx.x * 1024 >= n) return;              // CTA-uniform: nothing of this chunk is live
    __shared__ int s_prior[LKB_N_EXPERTS];
    __shared__ int s_wc[32][LKB_N_EXPERTS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.x * 1024;
    if (tid < LKB_N_EXPERTS) s_prior[tid] = off[tid];
    for (int i = tid; i < 32 * LKB_N_EXPERTS; i += 1024) (&s_wc[0][0])[i] = 0;
    __syncthreads();
    for (int s = tid; s < c0; s += 1024) atomicAdd(&s_prior[idx[s]], 1);
    const int s = c0 + tid;
    const bool live = s < n;
    const int e = live ? idx[s] : -1 - lane;               // dead lanes match nobody
    const unsigned same = __match_any_sync(LKB_FULL, e);
    const int rank_w = __popc(same & ((1u << lane) - 1u));
    if (live && rank_w == 0) s_wc[warp][e] = __popc(same);
    __syncthreads();
    // exclusive scan over warps, per expert (64 threads x 32 steps)
    if (tid < LKB_N_EXPERTS) {
        int run = s_prior[tid];
        for (int wv = 0; wv < 32; ++wv) { const int c = s_wc[wv][tid]; s_wc[wv][tid] = run; run += c; }
    }
    __syncthreads();
    if (live) perm[s_wc[warp][e] + rank_w] = s;
}

// Memset, count, plan and scatter in one launch of one CTA, for the few slots of a short chunk: each of the four cost its
// launch, not its work.  A round of 1024 slots costs 1 to 1.5 us here, so up to PF_ROUTE_MAX slots this is the shorter
// way (prefill of 37 tokens: 7.60 -> 7.42 ms, of 2 3.7 -> 3.5).  The same results, byte for byte.
#define PF_ROUTE_MAX 2048
__global__ void __launch_bounds__(1024) k_pf_moe_route(const int * __restrict__ idx, int n, int * __restrict__ cnt, int * __restrict__ off,
                                                       int4 * __restrict__ tiles, int * __restrict__ ntiles, int * __restrict__ perm) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    __shared__ int s_cnt[LKB_N_EXPERTS], s_prior[LKB_N_EXPERTS];
    __shared__ int s_wc[32][LKB_N_EXPERTS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < LKB_N_EXPERTS) s_cnt[tid] = 0;
    __syncthreads();
    for (int s = tid; s < n; s += 1024) atomicAdd(&s_cnt[idx[s]], 1);
    __syncthreads();
    if (warp == 0) {
        pf_plan_warp(lane, s_cnt[lane], s_cnt[lane + 32], s_prior, tiles, ntiles);
        __syncwarp();
        off[lane] = s_prior[lane]; off[lane + 32] = s_prior[lane + 32];
        cnt[lane] = s_cnt[lane]; cnt[lane + 32] = s_cnt[lane + 32];
    }
    for (int c0 = 0; c0 < n; c0 += 1024) {
        for (int i = tid; i < 32 * LKB_N_EXPERTS; i += 1024) (&s_wc[0][0])[i] = 0;
        __syncthreads();
        const int s = c0 + tid;
        const bool live = s < n;
        const int e = live ? idx[s] : -1 - lane;               // dead lanes match nobody
        const unsigned same = __match_any_sync(LKB_FULL, e);
        const int rank_w = __popc(same & ((1u << lane) - 1u));
        if (live && rank_w == 0) s_wc[warp][e] = __popc(same);
        __syncthreads();
        if (tid < LKB_N_EXPERTS) {
            int run = s_prior[tid];
            for (int wv = 0; wv < 32; ++wv) { const int c = s_wc[wv][tid]; s_wc[wv][tid] = run; run += c; }
            s_prior[tid] = run;
        }
        __syncthreads();
        if (live) perm[s_wc[warp][e] + rank_w] = s;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// combine: x[t] += sum over the token's four slots in rank order (one fused multiply-add chain from zero, then
// one add), four channels per thread.  The combine that feeds the next layer's norm is k_pf_token_norm<1>.
// ref semantics: src/prefill.cu:1804-1814 and 1764-1800
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_pf_moe_combine(float4 * __restrict__ X, const float4 * __restrict__ D,
                                                        const float * __restrict__ w, int m) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    const int i = blockIdx.x * blockDim.x + threadIdx.x;          // float4 index into X
    if (i >= m * (LKB_HIDDEN / 4)) return;
    const int t = i / (LKB_HIDDEN / 4), c = i - t * (LKB_HIDDEN / 4);
    const float4 wk = *reinterpret_cast<const float4 *>(w + t * 4);
    const float wv[4] = {wk.x, wk.y, wk.z, wk.w};
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < LKB_TOP_K; ++k) {
        const float4 dv = D[(size_t) (t * 4 + k) * (LKB_HIDDEN / 4) + c];
        a.x = fmaf(wv[k], dv.x, a.x); a.y = fmaf(wv[k], dv.y, a.y); a.z = fmaf(wv[k], dv.z, a.z); a.w = fmaf(wv[k], dv.w, a.w);
    }
    const float4 xv = X[i];
    X[i] = make_float4(__fadd_rn(xv.x, a.x), __fadd_rn(xv.y, a.y), __fadd_rn(xv.z, a.z), __fadd_rn(xv.w, a.w));
}

// planar row -> 36-byte blocks (exact: 8 sum is a power-of-two multiple).  Eight lanes per block, one word each.
// ref semantics: src/prefill.cu:1819-1828
__global__ void __launch_bounds__(512) k_pf_pack_q8_1(const int8_t * __restrict__ aqs, const float2 * __restrict__ asc, int t,
                                                      lkb_q8blk * __restrict__ y) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    const int b = threadIdx.x >> 3, wd = threadIdx.x & 7;
    reinterpret_cast<int *>(y[b].qs)[wd] = reinterpret_cast<const int *>(aqs + (size_t) t * LKB_HIDDEN + b * 32)[wd];
    if (wd == 0) {
        const float2 s = asc[(size_t) t * 64 + b];
        y[b].ds = __floats2half2_rn(s.x, __fmul_rn(s.y, 0.125f));
    }
}

// ---------------------------------------------------------------------------
// Expert-parallel dispatch helpers (no counterpart in the reference, which is single-GPU).
// A slot travels as ONE 2576-byte row: 2048 B of quants | 512 B of (d8, 8sum) pairs | 1/rms | expert id on the
// owner | 8 B pad, so that a layer's dispatch is a single all-to-all.
// ---------------------------------------------------------------------------
#define EP_ROW_BYTES (LKB_HIDDEN + (LKB_HIDDEN / 32) * 8 + 16)        // 2576, a multiple of 16

// Row p of `out` = the activation of slot send_order[p] (token = slot >> 2); pos[slot] = p.
__global__ void __launch_bounds__(192) k_ep_pack(const int8_t * __restrict__ aqs, const float2 * __restrict__ asc,
                                                 const float * __restrict__ inv, const int * __restrict__ idx,
                                                 const int * __restrict__ send_order, int experts_per_rank,
                                                 unsigned char * __restrict__ out, int * __restrict__ pos) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    const int p = blockIdx.x, i = threadIdx.x;
    const int slot = send_order[p], t = slot >> 2;
    uint4 * row = reinterpret_cast<uint4 *>(out + (size_t) p * EP_ROW_BYTES);
    if (i < 128) row[i] = reinterpret_cast<const uint4 *>(aqs + (size_t) t * LKB_HIDDEN)[i];
    else if (i < 160) row[i] = reinterpret_cast<const uint4 *>(asc + (size_t) t * (LKB_HIDDEN / 32))[i - 128];
    else if (i == 160) {
        const int e = idx[slot];
        row[160] = make_uint4(__float_as_uint(inv[t]), (unsigned) (e % experts_per_rank), 0u, 0u);
        pos[slot] = p;
    }
}

__global__ void __launch_bounds__(192) k_ep_unpack(const unsigned char * __restrict__ in, int8_t * __restrict__ qs,
                                                   float2 * __restrict__ sc, float * __restrict__ inv, int * __restrict__ le) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    const int p = blockIdx.x, i = threadIdx.x;
    const uint4 * row = reinterpret_cast<const uint4 *>(in + (size_t) p * EP_ROW_BYTES);
    if (i < 128) reinterpret_cast<uint4 *>(qs + (size_t) p * LKB_HIDDEN)[i] = row[i];
    else if (i < 160) reinterpret_cast<uint4 *>(sc + (size_t) p * (LKB_HIDDEN / 32))[i - 128] = row[i];
    else if (i == 160) { const uint4 v = row[160]; inv[p] = __uint_as_float(v.x); le[p] = (int) v.y; }
}


// ---------------------------------------------------------------------------
// CUDA-core form of the Q4_0 x Q8_1 GEMM (dense, grouped, SwiGLU epilogue).
// CTA = 64 weight rows (EPI 1: 32 gate + the same 32 up rows) x one 64-token
// tile; thread = rows (lane, lane+32) x 8 tokens, so a warp holds 32 consecutive
// rows of a token and the SwiGLU epilogue quantises with the standard warp
// quantiser: fused output == unfused output bit for bit.
// Per (row, token), b ascending: fold = 1: acc = fma(d4, fma(d8, F_b, -c), acc) with F_b = 12582912 + S_b and
// c = fma(d8, 12582912, 8sum) (the reference's shipped form, src/prefill.cu:131-139,341-342,381-384);
// fold = 0: acc = fma(d4, fma(d8, float(S_b), -8sum), acc) (src/prefill.cu:391-399); then * scale, then (+ out).
// ref: src/prefill.cu:172-491 (semantics)
// ---------------------------------------------------------------------------
#define SG_KB 8
#define SG_WP (SG_KB * 16 + 16)        // weight row pitch in smem (bytes), +16 against bank conflicts

template <int EPI>
__global__ void __launch_bounds__(256) k_pf_gemm_simple(const lkb_pf_gemm g, const int fold) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    __shared__ __align__(16) unsigned char s_w[64 * SG_WP];
    __shared__ __align__(16) __half        s_d[64 * SG_KB];
    __shared__ __align__(16) int8_t        s_a[64 * SG_KB * 32];
    __shared__ __align__(16) float2        s_s[64 * SG_KB];
    __shared__ int   s_arow[64];
    __shared__ int   s_orow[64];
    __shared__ float s_scl[64];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int rt, tstart, tcnt, expert = 0;
    if (g.perm) {
        if ((int) blockIdx.y >= *g.ntiles) return;
        const int4 tl = reinterpret_cast<const int4 *>(g.tiles)[blockIdx.y];
        expert = tl.x; tstart = tl.y; tcnt = tl.z; rt = blockIdx.x;
    } else {
        rt = blockIdx.x; tstart = blockIdx.y * 64;
        tcnt = g.ntok - tstart; if (tcnt > 64) tcnt = 64;
    }
    if (tid < 64) {
        int slot = -1;
        if (tid < tcnt) slot = g.perm ? g.perm[tstart + tid] : tstart + tid;
        const int ar = (slot >= 0) ? (slot >> g.a_shift) : -1;
        s_arow[tid] = ar; s_orow[tid] = slot;
        s_scl[tid] = (ar >= 0 && g.scale) ? g.scale[ar] : 1.0f;
    }
    // weight rows of this CTA: local row r in [0,64)
    const int row0 = EPI ? rt * 32 : rt * 64;
    const size_t eo = (size_t) expert * g.exp_stride;
    const uint4 * wq[2]; const __half * wd[2];
    if (EPI) {
        wq[0] = (const uint4 *) g.qs[0] + eo + (size_t) row0 * g.bpr; wd[0] = (const __half *) g.d[0] + eo + (size_t) row0 * g.bpr;
        wq[1] = (const uint4 *) g.qs[1] + eo + (size_t) row0 * g.bpr; wd[1] = (const __half *) g.d[1] + eo + (size_t) row0 * g.bpr;
    } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = row0 + 32 * h;
            const int seg = (r < g.seg_end[0]) ? 0 : (r < g.seg_end[1]) ? 1 : 2;
            const int sbase = seg ? g.seg_end[seg - 1] : 0;
            wq[h] = (const uint4 *) g.qs[seg] + eo + (size_t) (r - sbase) * g.bpr;
            wd[h] = (const __half *) g.d[seg] + eo + (size_t) (r - sbase) * g.bpr;
        }
    }
    __syncthreads();

    float acc[2][8];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[h][j] = 0.0f;

    for (int kb0 = 0; kb0 < g.bpr; kb0 += SG_KB) {
        // stage: 64 rows x 8 blocks of weights, 64 tokens x 8 blocks of activations
        for (int c = tid; c < 64 * SG_KB; c += 256) {
            const int r = c / SG_KB, kk = c % SG_KB;
            const int h = r >> 5, rr = r & 31;
            *reinterpret_cast<uint4 *>(s_w + r * SG_WP + kk * 16) = wq[h][(size_t) rr * g.bpr + kb0 + kk];
            s_d[r * SG_KB + kk] = wd[h][(size_t) rr * g.bpr + kb0 + kk];
            const int ar = s_arow[r];
            s_s[r * SG_KB + kk] = (ar >= 0) ? reinterpret_cast<const float2 *>(g.asc)[(size_t) ar * g.bpr + kb0 + kk]
                                            : make_float2(0.0f, 0.0f);
        }
        for (int c = tid; c < 64 * SG_KB * 2; c += 256) {
            const int r = c / (SG_KB * 2), kk = c % (SG_KB * 2);
            const int ar = s_arow[r];
            int4 v = make_int4(0, 0, 0, 0);
            if (ar >= 0) v = *reinterpret_cast<const int4 *>(g.aqs + (size_t) ar * g.bpr * 32 + (size_t) kb0 * 32 + kk * 16);
            *reinterpret_cast<int4 *>(s_a + r * SG_KB * 32 + kk * 16) = v;
        }
        __syncthreads();
#pragma unroll 2
        for (int kk = 0; kk < SG_KB; ++kk) {
            uint4 wv[2]; float d4[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                wv[h] = *reinterpret_cast<const uint4 *>(s_w + (lane + 32 * h) * SG_WP + kk * 16);
                d4[h] = __half2float(s_d[(lane + 32 * h) * SG_KB + kk]);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int tk = warp * 8 + j;
                const int4 a0 = *reinterpret_cast<const int4 *>(s_a + tk * SG_KB * 32 + kk * 32);
                const int4 a1 = *reinterpret_cast<const int4 *>(s_a + tk * SG_KB * 32 + kk * 32 + 16);
                const int xv[8] = { a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w };
                const float2 sc = s_s[tk * SG_KB + kk];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    {
                        const int si = lkb_sumi(wv[h], xv);
                        acc[h][j] = fold ? lkb_block_acc_pf(d4[h], sc.x, si, sc.y, acc[h][j]) : lkb_block_acc(d4[h], sc.x, si, sc.y, acc[h][j]);
                    }
            }
        }
        __syncthreads();
    }

#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int tk = warp * 8 + j;
        const int orow = s_orow[tk];            // warp-uniform
        if (orow < 0) continue;
        const float scl = s_scl[tk];
        if (EPI) {
            const float gt = __fmul_rn(acc[0][j], scl);
            const float up = __fmul_rn(acc[1][j], scl);
            const float v = __fmul_rn(lkb_silu(gt), up);
            // shipped arithmetic: the block sum in the reference's fused-epilogue order; exact mode: the quantiser's butterfly
            if (fold) lkb_quant_store_planar_fused_epilogue(v, g.oqs + (size_t) orow * (g.okb * 32) + row0,
                                                            reinterpret_cast<float2 *>(g.osc) + (size_t) orow * g.okb + row0 / 32, lane);
            else      lkb_quant_store_planar(v, g.oqs + (size_t) orow * (g.okb * 32) + row0,
                                             reinterpret_cast<float2 *>(g.osc) + (size_t) orow * g.okb + row0 / 32, lane);
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // the residual add is one fused multiply-add, as the reference's build contracts it (src/prefill.cu:484-486)
                float * p = g.out + (size_t) orow * g.out_ld + row0 + 32 * h + lane;
                *p = g.add ? fmaf(acc[h][j], scl, *p) : __fmul_rn(acc[h][j], scl);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
int lkb_gemm_tc_init();                                      // lkb_gemm_tc.cu
int lkb_gemm_tc_launch(const lkb_pf_gemm * g, int epi, int fold, int max_tiles, cudaStream_t st, float * const * out_rows, int a_pitch);   // LKB_ERR_UNSUPPORTED if shape not covered

int lkb_gemm_few_launch(const lkb_pf_gemm * g, int epi, int fold, int max_tiles, cudaStream_t st);       // lkb_gemm_few.cu: ... or where another form is faster

static int g_gemm_cfg = -1;        // -1: tensor-core form when it covers the shape; 0: CUDA-core form
static int g_gemm_fold = 1;        // 1: the reference's shipped per-block term (folded offset); 0: the exact term

int lkb_prefill_take_status() { return tc_take_status(); }
int lkb_prefill_init() {
    const char * v = getenv("LKB_PF_CFG");
    if (v) g_gemm_cfg = atoi(v);
    v = getenv("LKB_PF_ARITH");
    if (v) g_gemm_fold = atoi(v) ? 1 : 0;
    return lkb_gemm_tc_init();
}

static int gemm_check(const lkb_pf_gemm * g, int epi) {
    if (!g) return LKB_ERR_NULL;
    if (!g->qs[0] || !g->d[0] || !g->aqs || !g->asc) return LKB_ERR_NULL;
    if (epi) { if (!g->qs[1] || !g->d[1] || !g->oqs || !g->osc) return LKB_ERR_NULL; }
    else if (!g->out) return LKB_ERR_NULL;
    if (g->bpr <= 0 || g->bpr % 8) return LKB_ERR_SHAPE;
    if (epi ? (g->N % 64) : (g->N % 128)) return LKB_ERR_SHAPE;
    if (!epi && (g->seg_end[0] % 128 || g->seg_end[1] % 128)) return LKB_ERR_SHAPE;
    if (g->perm && (!g->tiles || !g->ntiles)) return LKB_ERR_NULL;
    // what either form loads or stores at a time (the tensor-core form asks for more and leaves such planes to the other)
    size_t by16 = (size_t) g->aqs | (size_t) g->tiles, by8 = (size_t) g->asc | (epi ? (size_t) g->osc : 0), by4 = epi ? 0 : (size_t) g->out, by2 = 0;
    const int nseg = epi ? 2 : (g->seg_end[0] >= g->N ? 1 : g->seg_end[1] >= g->N ? 2 : 3);
    for (int s = 0; s < nseg; ++s) { by16 |= (size_t) g->qs[s]; by2 |= (size_t) g->d[s]; }
    if ((by16 & 15) || (by8 & 7) || (by4 & 3) || (by2 & 1)) return LKB_ERR_SHAPE;
    return LKB_OK;
}

static int gemm_dispatch(const lkb_pf_gemm * g, int epi, int max_tiles, cudaStream_t st, float * const * out_rows = nullptr, int a_pitch = 0) {
    LKB_REQUIRE_INIT();
    const int r = gemm_check(g, epi);
    if (r != LKB_OK) return r;
    const int ty = g->perm ? max_tiles : (g->ntok + 63) / 64;
    if (ty <= 0) return g->perm ? LKB_ERR_SHAPE : LKB_OK;
    if (g_gemm_cfg < 0 && !out_rows && !a_pitch) {
        const int t = lkb_gemm_few_launch(g, epi, g_gemm_fold, max_tiles, st);
        if (t != LKB_ERR_UNSUPPORTED) return t;
    }
    if (g_gemm_cfg != 0) {
        const int t = lkb_gemm_tc_launch(g, epi, g_gemm_fold, max_tiles, st, out_rows, a_pitch);
        if (t != LKB_ERR_UNSUPPORTED) return t;
        if (g_gemm_cfg > 0) return t;
    }
    if (out_rows || a_pitch) return LKB_ERR_UNSUPPORTED;   // row targets and packed rows exist in the tensor-core form only
    if (epi) LKB_PF_LAUNCH((k_pf_gemm_simple<1>), dim3(dim3(g->N / 32, ty)), dim3(256), 0, st, *g, g_gemm_fold);
    else     LKB_PF_LAUNCH((k_pf_gemm_simple<0>), dim3(dim3(g->N / 64, ty)), dim3(256), 0, st, *g, g_gemm_fold);
    return lkb_check_launch();
}

extern "C" {

int lkb_pf_gemm_config(int cfg) { g_gemm_cfg = cfg; return LKB_OK; }
int lkb_pf_gemm_arith(int fold) { g_gemm_fold = fold ? 1 : 0; return LKB_OK; }

int lkb_pf_norm(const float * X, const float * w, int plain, lkb_pf_act a, float * inv_out, float * h32,
                int m, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!X || !w || !a.qs || !a.sc || !inv_out) return LKB_ERR_NULL;
    if (m <= 0) return m == 0 ? LKB_OK : LKB_ERR_SHAPE;
    if (plain) LKB_PF_LAUNCH(k_pf_token_norm_plain, dim3((m + PF_TOK_WARPS - 1) / PF_TOK_WARPS), dim3(PF_TOK_WARPS * 32), 0, (cudaStream_t) st, X, w, a.qs, reinterpret_cast<float2 *>(a.sc), inv_out, m);
    else       LKB_PF_LAUNCH((k_pf_token_norm<0>), dim3((m + PF_TOK_PER_CTA - 1) / PF_TOK_PER_CTA), dim3(PF_TOK_WARPS * 32), 0, (cudaStream_t) st, const_cast<float *>(X), nullptr, nullptr, nullptr, w, a.qs,
                                                                                  reinterpret_cast<float2 *>(a.sc), inv_out, h32, m);
    return lkb_check_launch();
}

int lkb_pf_quant_rows(const float * X, int ld, int kb, lkb_pf_act a, int rows, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!X || !a.qs || !a.sc) return LKB_ERR_NULL;
    if (rows <= 0 || kb <= 0) return (rows == 0) ? LKB_OK : LKB_ERR_SHAPE;
    if ((ld & 3) || (reinterpret_cast<uintptr_t>(X) & 15)) return LKB_ERR_SHAPE;      // 128-bit loads
    const long long warps = (long long) rows * ((kb + 3) / 4);
    LKB_PF_LAUNCH((k_pf_rows_q8<0>), dim3((unsigned) ((warps + 7) / 8)), dim3(256), 0, (cudaStream_t) st, X, ld, 0, kb, rows, a.qs, reinterpret_cast<float2 *>(a.sc));
    return lkb_check_launch();
}

int lkb_pf_swiglu(const float * Y, int ld, int up_off, int kb, lkb_pf_act a, int rows, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!Y || !a.qs || !a.sc) return LKB_ERR_NULL;
    if (rows <= 0 || kb <= 0) return (rows == 0) ? LKB_OK : LKB_ERR_SHAPE;
    if ((ld & 3) || (up_off & 3) || (reinterpret_cast<uintptr_t>(Y) & 15)) return LKB_ERR_SHAPE;
    const long long warps = (long long) rows * ((kb + 3) / 4);
    LKB_PF_LAUNCH((k_pf_rows_q8<1>), dim3((unsigned) ((warps + 7) / 8)), dim3(256), 0, (cudaStream_t) st, Y, ld, up_off, kb, rows, a.qs, reinterpret_cast<float2 *>(a.sc));
    return lkb_check_launch();
}

static int router_small(const float * H, int m, const float * Wr, const float * bias, const float * inv,
                        float * sel, float * sig, int * idx, float * w, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!H || !Wr || !bias || !inv || !sel || !sig) return LKB_ERR_NULL;
    if (m <= 0) return m == 0 ? LKB_OK : LKB_ERR_SHAPE;
    if (m > 65535) return LKB_ERR_SHAPE;
    // A cluster of CTAs a token while that is about a wave: a MoE layer at 2 / 9 / 37 / 64 / 100 tokens 47 / 63 / 114 / 152 / 155 -> 41 / 58 / 109 /
    // 146 / 150 us; at 180 equal, at 256 182 -> 186.
    if (m <= LKB_PF_NORM_ROUTER_TOKENS) {
        LKB_PF_LAUNCH(k_pf_router_cluster, dim3(m * RC_CTAS), dim3(256), 0, (cudaStream_t) st, H, Wr, bias, inv, sel, sig,
                      reinterpret_cast<int4 *>(idx), reinterpret_cast<float4 *>(w));
        return lkb_check_launch();
    }
    LKB_PF_LAUNCH(k_pf_router_token, dim3(m), dim3(256), 0, (cudaStream_t) st, H, Wr, bias, inv, sel, sig,
                  reinterpret_cast<int4 *>(idx), reinterpret_cast<float4 *>(w));
    return lkb_check_launch();
}

static int router_tiled(const float * H, int m, const float * Wr, const float * bias, const float * inv,
                        float * sel, float * sig, int * idx, float * w, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!H || !Wr || !bias || !inv || !sel || !sig) return LKB_ERR_NULL;
    if (m <= 0) return m == 0 ? LKB_OK : LKB_ERR_SHAPE;
    // The k loop of one CTA is the critical path and its length grows with the tokens per CTA, so a token range takes the smallest
    // CTA that still fits one wave.  Measured on B200, us, calls back to back, copies by every thread and by tensor copies:
    //   4-token CTAs (two warps)         up to 592 tokens   21.2   27.8
    //   8-token CTAs (two warps)         up to 1184         29.7   25.2
    //   16-token CTAs                    up to 2368         35.2   28.9
    //   32-token CTAs, 64 k-values a tile  at 4096          53.4   43.3
    // A rank's share of an expert-parallel chunk lands in the first three.  LKB_ROUTER_FORM = 4 / 8 / 16 / 32 forces a shape (tuning): 4 with copies by
    // every thread, the others with tensor copies.
    static const int form = [] { const char * e = getenv("LKB_ROUTER_FORM"); return e ? atoi(e) : 0; }();
    const int sms = lkb_context().sm_count;
    if (form == 4 || (form == 0 && m <= 4 * sms)) return rt_launch<1, 2, 128, 4>(H, m, Wr, bias, inv, sel, sig, idx, w, (cudaStream_t) st);
    if (form == 8 || (form == 0 && m <= 8 * sms)) return rt_launch_tma<2, 2, 128, 4>(H, m, Wr, bias, inv, sel, sig, idx, w, (cudaStream_t) st);
    if (form == 16 || (form == 0 && m <= 16 * sms)) return rt_launch_tma<2, 4, 128, 4>(H, m, Wr, bias, inv, sel, sig, idx, w, (cudaStream_t) st);
    return rt_launch_tma<4, 4, 64, 6>(H, m, Wr, bias, inv, sel, sig, idx, w, (cudaStream_t) st);
}

int lkb_pf_router_small(const float * H, int m, const float * Wr, const float * bias, const float * inv,
                        float * sel, float * sig, lkb_stream_t st) {
    return router_small(H, m, Wr, bias, inv, sel, sig, nullptr, nullptr, st);
}
int lkb_pf_router_tiled(const float * H, int m, const float * Wr, const float * bias, const float * inv,
                        float * sel, float * sig, lkb_stream_t st) {
    return router_tiled(H, m, Wr, bias, inv, sel, sig, nullptr, nullptr, st);
}
int lkb_pf_router(const float * H, int m, const float * Wr, const float * bias, const float * inv,
                  float * sel, float * sig, lkb_stream_t st) {
    if (m > 0 && m <= 256) return lkb_pf_router_small(H, m, Wr, bias, inv, sel, sig, st);
    return lkb_pf_router_tiled(H, m, Wr, bias, inv, sel, sig, st);
}
int lkb_pf_router_select(const float * H, int m, int small_form, const float * Wr, const float * bias, const float * inv,
                         float * sel, float * sig, int * idx, float * w, lkb_stream_t st) {
    if (!idx || !w) return LKB_ERR_NULL;
    return small_form ? router_small(H, m, Wr, bias, inv, sel, sig, idx, w, st) : router_tiled(H, m, Wr, bias, inv, sel, sig, idx, w, st);
}

int lkb_pf_norm_router_select(const float * X, const float * nw, lkb_pf_act a, float * inv, float * h32, int m, int small_form, const float * Wr,
                              const float * bias, float * sel, float * sig, int * idx, float * w, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!X || !nw || !a.qs || !a.sc || !inv || !h32 || !Wr || !bias || !sel || !sig || !idx || !w) return LKB_ERR_NULL;
    if (m <= 0) return m == 0 ? LKB_OK : LKB_ERR_SHAPE;
    if (small_form && m <= LKB_PF_NORM_ROUTER_TOKENS) {
        LKB_PF_LAUNCH(k_pf_norm_router_cluster, dim3(m * RC_CTAS), dim3(256), 0, (cudaStream_t) st, X, nw, a.qs, reinterpret_cast<float2 *>(a.sc), inv, Wr, bias, sel, sig,
                      reinterpret_cast<int4 *>(idx), reinterpret_cast<float4 *>(w));
        return lkb_check_launch();
    }
    const int r = lkb_pf_norm(X, nw, 0, a, inv, h32, m, st);
    return r != LKB_OK ? r : lkb_pf_router_select(h32, m, small_form, Wr, bias, inv, sel, sig, idx, w, st);
}

int lkb_pf_select(const float * sel, const float * sig, int m, int * idx, float * w, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!sel || !sig || !idx || !w) return LKB_ERR_NULL;
    if (m <= 0) return m == 0 ? LKB_OK : LKB_ERR_SHAPE;
    LKB_PF_LAUNCH(k_pf_select, dim3(min((m + 7) / 8, 148 * 8)), dim3(256), 0, (cudaStream_t) st, sel, sig, m, reinterpret_cast<int4 *>(idx), reinterpret_cast<float4 *>(w));
    return lkb_check_launch();
}

int lkb_pf_moe_count(const int * idx, int n, int * cnt, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!idx || !cnt) return LKB_ERR_NULL;
    if (n <= 0) return n == 0 ? LKB_OK : LKB_ERR_SHAPE;
    int grid = (n + 255) / 256; if (grid > 64) grid = 64;
    LKB_PF_LAUNCH(k_pf_moe_count, dim3(grid), dim3(256), 0, (cudaStream_t) st, idx, n, cnt);
    return lkb_check_launch();
}

int lkb_zero_i32(int * p, int n, lkb_stream_t st) {
    if (!p) return LKB_ERR_NULL;
    if (n < 0) return LKB_ERR_SHAPE;
    const cudaError_t e = cudaMemsetAsync(p, 0, (size_t) n * 4, (cudaStream_t) st);
    return e == cudaSuccess ? LKB_OK : -(int) e;
}

int lkb_pf_moe_plan(const int * cnt, int * off, int * tiles, int * ntiles, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!cnt || !off || !tiles || !ntiles) return LKB_ERR_NULL;
    LKB_PF_LAUNCH(k_pf_moe_plan, dim3(1), dim3(32), 0, (cudaStream_t) st, cnt, off, reinterpret_cast<int4 *>(tiles), ntiles);
    return lkb_check_launch();
}

int lkb_pf_moe_scatter(const int * idx, int n, const int * off, int * perm, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!idx || !off || !perm) return LKB_ERR_NULL;
    if (n <= 0) return n == 0 ? LKB_OK : LKB_ERR_SHAPE;
    LKB_PF_LAUNCH(k_pf_moe_scatter, dim3((n + 1023) / 1024), dim3(1024), 0, (cudaStream_t) st, idx, n, off, perm);
    return lkb_check_launch();
}

int lkb_pf_moe_route(const int * idx, int n, int * cnt, int * off, int * tiles, int * ntiles, int * perm, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!idx || !cnt || !off || !tiles || !ntiles || !perm) return LKB_ERR_NULL;
    if (n <= 0) return LKB_ERR_SHAPE;
    if (n <= PF_ROUTE_MAX) {
        LKB_PF_LAUNCH(k_pf_moe_route, dim3(1), dim3(1024), 0, (cudaStream_t) st, idx, n, cnt, off, reinterpret_cast<int4 *>(tiles), ntiles, perm);
        return lkb_check_launch();
    }
    int r = lkb_zero_i32(cnt, LKB_N_EXPERTS, st);
    if (r == LKB_OK) r = lkb_pf_moe_count(idx, n, cnt, st);
    if (r == LKB_OK) r = lkb_pf_moe_plan(cnt, off, tiles, ntiles, st);
    return r == LKB_OK ? lkb_pf_moe_scatter(idx, n, off, perm, st) : r;
}

int lkb_pf_gemm_dense(const lkb_pf_gemm * g, lkb_stream_t st) {
    if (g && g->perm) return LKB_ERR_SHAPE;
    return gemm_dispatch(g, 0, 0, (cudaStream_t) st);
}
int lkb_pf_gemm_moe(const lkb_pf_gemm * g, int max_tiles, lkb_stream_t st) {
    if (g && !g->perm) return LKB_ERR_NULL;
    return gemm_dispatch(g, 0, max_tiles, (cudaStream_t) st);
}
int lkb_pf_gemm_moe_rows(const lkb_pf_gemm * g, int max_tiles, float * const * out_rows, lkb_stream_t st) {
    if (!out_rows) return LKB_ERR_NULL;
    return gemm_dispatch(g, 0, max_tiles, (cudaStream_t) st, out_rows);
}
int lkb_pf_gemm_swiglu_packed(const lkb_pf_gemm * g, int max_tiles, int row_pitch, lkb_stream_t st) {
    if (row_pitch <= 0) return LKB_ERR_SHAPE;
    return gemm_dispatch(g, 1, max_tiles, (cudaStream_t) st, nullptr, row_pitch);
}
int lkb_pf_gemm_swiglu(const lkb_pf_gemm * g, int max_tiles, lkb_stream_t st) {
    return gemm_dispatch(g, 1, max_tiles, (cudaStream_t) st);
}

int lkb_pf_moe_combine(float * X, const float * D, const float * w, int m, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!X || !D || !w) return LKB_ERR_NULL;
    if (m <= 0) return m == 0 ? LKB_OK : LKB_ERR_SHAPE;
    LKB_PF_LAUNCH(k_pf_moe_combine, dim3(m * (LKB_HIDDEN / 4 / 256)), dim3(256), 0, (cudaStream_t) st, reinterpret_cast<float4 *>(X), reinterpret_cast<const float4 *>(D), w, m);
    return lkb_check_launch();
}

int lkb_pf_moe_combine_norm(float * X, const float * D, const float * w, const float * nw, lkb_pf_act a,
                            float * inv_out, int m, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!X || !D || !w || !nw || !a.qs || !a.sc || !inv_out) return LKB_ERR_NULL;
    if (m <= 0) return m == 0 ? LKB_OK : LKB_ERR_SHAPE;
    LKB_PF_LAUNCH((k_pf_token_norm<1>), dim3((m + PF_TOK_PER_CTA - 1) / PF_TOK_PER_CTA), dim3(PF_TOK_WARPS * 32), 0, (cudaStream_t) st, X, D, nullptr, w, nw, a.qs, reinterpret_cast<float2 *>(a.sc), inv_out, nullptr, m);
    return lkb_check_launch();
}

int lkb_ep_pack_rows(lkb_pf_act a, const float * inv, const int * idx, const int * send_order, int n,
                     int experts_per_rank, void * out, int * pos, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!a.qs || !a.sc || !inv || !idx || !send_order || !out || !pos) return LKB_ERR_NULL;
    if (n <= 0 || experts_per_rank <= 0) return n == 0 ? LKB_OK : LKB_ERR_SHAPE;
    LKB_PF_LAUNCH(k_ep_pack, dim3(n), dim3(192), 0, (cudaStream_t) st, a.qs, reinterpret_cast<const float2 *>(a.sc), inv, idx, send_order,
                                                experts_per_rank, static_cast<unsigned char *>(out), pos);
    return lkb_check_launch();
}

int lkb_ep_unpack_rows(const void * in, int n, lkb_pf_act a, float * inv, int * local_expert, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!in || !a.qs || !a.sc || !inv || !local_expert) return LKB_ERR_NULL;
    if (n <= 0) return n == 0 ? LKB_OK : LKB_ERR_SHAPE;
    LKB_PF_LAUNCH(k_ep_unpack, dim3(n), dim3(192), 0, (cudaStream_t) st, static_cast<const unsigned char *>(in), a.qs,
                                                  reinterpret_cast<float2 *>(a.sc), inv, local_expert);
    return lkb_check_launch();
}

int lkb_pf_moe_combine_norm_gather(float * X, const float * D, const int * pos, const float * w, const float * nw,
                                   lkb_pf_act a, float * inv_out, int m, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!X || !D || !pos || !w || !nw || !a.qs || !a.sc || !inv_out) return LKB_ERR_NULL;
    if (m <= 0) return m == 0 ? LKB_OK : LKB_ERR_SHAPE;
    LKB_PF_LAUNCH((k_pf_token_norm<2>), dim3((m + PF_TOK_PER_CTA - 1) / PF_TOK_PER_CTA), dim3(PF_TOK_WARPS * 32), 0, (cudaStream_t) st, X, D, pos, w, nw, a.qs, reinterpret_cast<float2 *>(a.sc), inv_out, nullptr, m);
    return lkb_check_launch();
}

int lkb_pf_pack_q8_1(lkb_pf_act a, int t, lkb_block_q8_1 * y, lkb_stream_t st) {
    LKB_REQUIRE_INIT();
    if (!a.qs || !a.sc || !y) return LKB_ERR_NULL;
    if (t < 0) return LKB_ERR_SHAPE;
    LKB_PF_LAUNCH(k_pf_pack_q8_1, dim3(1), dim3(512), 0, (cudaStream_t) st, a.qs, reinterpret_cast<const float2 *>(a.sc), t, reinterpret_cast<lkb_q8blk *>(y));
    return lkb_check_launch();
}

}  // extern "C"
