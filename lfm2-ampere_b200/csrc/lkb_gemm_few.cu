// lkb_gemm_few.cu - the Q4_0 x Q8_1 GEMM (dense and grouped) for a few tokens: weights streamed once, integer dots on the CUDA cores.
//
// The same sums as lkb_gemm_tc.cu, in the same order and rounding, so the same bits: per (row, token) one fp32 chain over the
// blocks, acc = fma(d4, fma(d8, 12582912 + S, -c), acc) (FOLD = 1) or fma(d4, fma(d8, float(S), -8sum), acc) (FOLD = 0).
//
// With the one to eight tokens a tile has in a short prompt, the tensor-core form is bound by what it does per block whatever
// the token count: expansion of the nibbles into TMEM, commits, arrivals and polls, 360 to 450 cycles a block of 256 rows, whose
// weights take 190 of HBM time.  Here a thread owns two weight rows and up to eight tokens: it expands a block's nibbles in
// registers once, and a token costs it eight dp4a and two FMAs a row.  One mbarrier a stage, nothing handed back but the stage.
//   * A producer warp fetches everything by tensor copies: nibbles and weight scales of 2 x 128 rows, and by row gathers (tile::gather4,
//     through perm or along a dense chunk) the quants and (d8, 8sum) pairs of the tokens.
//   * Two rows a thread because every load of the tokens' data has the same address in all lanes, and the load unit writes 512 bytes of
//     registers for it all the same: with one row the 20 loads of two tokens and a block would take as long as the weights.
//   * Three CTAs an SM, 53 KB of stages each: 150 KB of weights in flight per SM.
// Measured, a whole MoE layer of 64 experts at 2 / 9 / 20 / 37 / 64 tokens, us (router, norms and routing included):
//   tensor-core form   55 / 92 / 120 / 140 / 152 with balanced routing    54 / 88 / 112 / 127 / 147 with Zipf(1.1) routing
//   this form          47 / 63 /  87 / 113 / 145                          45 / 62 /  87 / 118 / 158
// What bounds it: whole waves of items.  gate|up, caches flushed before every call, CUDA events: 28 / 48 / 61 of 64 experts hit by 9 / 20 / 37 tokens
// are 99 / 170 / 216 MB in 32 / 50 / 62 us, 3.1 to 3.5 TB/s (tensor-core form 46 / 58 / 69 us), down 50 / 85 / 108 MB in 22 / 30 / 40 us.  At 20 tokens
// that is 576 gate|up items on 444 CTAs, 1.3 waves, and 0.9 of a wave of down items: a third of the CTA time is idle, and
// the dots wait for their stages (ncu: long scoreboard first, issue 40 %).  From 37 tokens on the dots, two cycles an instruction, count too.
// Tried: 128 bytes of a row per stage (37 tokens +15 %), tiles of 64 and 32 rows with more CTAs (+35 %), two stages and four
// CTAs (+4 %), one CTA of five stages (+29 %).
// No copy in this file is a multicast one; every tensor map covers memory of the GPU the kernel runs on.
// Every wait is bounded; on expiry a status word is set, the roles leave, the producer after its copies have landed.
#include "lkb_tc.cuh"

#define FW_ROWS   128                // rows of a tile; an item has two (SwiGLU form: gate and up rows)
#define FW_TOK    8                  // tokens of an item
#define FW_KB     4                  // blocks per stage
#define FW_NS     3                  // stages
#define FW_WS     4                  // pairs of stages of weight scales
#define FW_CTAS   3                  // per SM
#define FW_WARPS  4                  // dot warps; warp 4 fetches
// Where the forms cross.  Grouped: by the slots the caller states, spread over 64 experts: the crossing is near 45 tokens of four slots with
// skewed routing and near 75 with balanced.  A plan that cannot have a tile per expert is one of fewer experts, whose tiles may be
// full; it takes the other form, as does a call that does not state its slots.  Dense: a projection of 2048 rows is 8 items
// here and the chain of its 64 blocks shows, more from the second row gather on.  A whole layer (grouped part here both times) at
// 2 / 3 / 4 / 5 / 6 / 7 / 9 tokens: 71.2 / 71.6 / 73.2 / 82.4 / 85.1 / 93.6 / 98.9 us dense here, 73.8 / 76.7 / 79.4 / 82.7 / 85.4 / 89.0 / 94.1 there.
#define FW_MIN_TILES LKB_N_EXPERTS
#define FW_MAX_SLOTS (47 * LKB_TOP_K)
#define FW_MAX_DENSE 4
static_assert(2 * FW_WS >= FW_NS + 4, "weight scales stay until their stages have been read");

struct FwStage {
    alignas(1024) unsigned char q[2 * FW_ROWS * 64];        // nibbles: row r at r*64, 16-byte chunk c at c ^ ((r >> 1) & 3)
    alignas(128) signed char act[FW_TOK][FW_KB * 32];
    alignas(128) float2 asc[FW_TOK][FW_KB];                 // (d8, 8sum)
};
struct FwSmem {
    FwStage st[FW_NS];
    alignas(128) uint4 wsc[FW_WS][2 * FW_ROWS];             // eight fp16 scales per row (two stages)
    alignas(8) unsigned long long full[FW_NS], empty[FW_NS];
    int abort;
};

struct FwItem { int expert, tstart, cnt, rt; };             // cnt 0: nothing to do
// Items by chunk of eight tokens (slowest: the later chunks of a plan tile are mostly empty), tile and row tile.
__device__ __forceinline__ FwItem fw_item(const lkb_pf_gemm & g, int n_mt, int n_rt, int item) {
    FwItem I;
    const int c = item / (n_mt * n_rt), mt = item / n_rt - c * n_mt;
    I.rt = item % n_rt;
    if (g.perm) {
        const int4 tl = __ldg(reinterpret_cast<const int4 *>(g.tiles) + mt);
        I.expert = tl.x; I.tstart = tl.y + c * FW_TOK; I.cnt = max(0, min(FW_TOK, tl.z - c * FW_TOK));
    } else {
        I.expert = 0; I.tstart = mt * FW_TOK; I.cnt = min(FW_TOK, g.ntok - I.tstart);
    }
    return I;
}

// All stages of one item for NT tokens.  Returns false when a wait gave up.
template <int FOLD, int NT>
__device__ __forceinline__ bool fw_dots(FwSmem & S, unsigned & it, int nstage, int row, int lane, float (&acc)[2][FW_TOK]) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[r][t] = 0.0f;
#pragma unroll 1
    for (int ks = 0; ks < nstage; ++ks, ++it) {
        const unsigned stg = it % FW_NS;
        if (!tc_wait(S, &S.full[stg], (it / FW_NS) & 1u, 33u)) return false;
        const FwStage & T = S.st[stg];
        uint2 we[2];                                                     // the stage's four scales of both rows
#pragma unroll
        for (int r = 0; r < 2; ++r)
            we[r] = *(reinterpret_cast<const uint2 *>(&S.wsc[(it >> 1) % FW_WS][r * FW_ROWS + row]) + (it & 1u));
#pragma unroll
        for (int b = 0; b < FW_KB; ++b) {
            int w[2][8]; float d4[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint4 v = *reinterpret_cast<const uint4 *>(T.q + (r * FW_ROWS + row) * 64 + ((b ^ ((row >> 1) & 3)) << 4));
                const unsigned x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) { w[r][i] = (int) (x[i] & 0x0F0F0F0Fu); w[r][4 + i] = (int) ((x[i] >> 4) & 0x0F0F0F0Fu); }
                d4[r] = __half2float(__ushort_as_half((unsigned short) ((b & 2 ? we[r].y : we[r].x) >> (16 * (b & 1)))));
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int4 a0 = *reinterpret_cast<const int4 *>(&T.act[t][b * 32]), a1 = *reinterpret_cast<const int4 *>(&T.act[t][b * 32 + 16]);
                const int a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                const float2 sc = T.asc[t][b];
                const float c = FOLD ? fmaf(sc.x, 12582912.0f, sc.y) : sc.y;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    int s = FOLD ? 0x4B400000 : 0;                       // the bit pattern of 12582912.0f: the sum arrives as a float
#pragma unroll
                    for (int i = 0; i < 8; ++i) s = __dp4a(w[r][i], a[i], s);
                    acc[r][t] = fmaf(d4[r], fmaf(sc.x, FOLD ? __int_as_float(s) : (float) s, -c), acc[r][t]);
                }
            }
        }
        __syncwarp();
        tc_mbar_arrive_if(&S.empty[stg], lane == 0);
    }
    return true;
}

template <int EPI, int FOLD>
__global__ void __launch_bounds__((FW_WARPS + 1) * 32, FW_CTAS) k_pf_gemm_few(const lkb_pf_gemm g, const int max_tiles, const int rpe,
        const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_s,
        const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_w2,
        const __grid_constant__ CUtensorMap map_d0, const __grid_constant__ CUtensorMap map_d1, const __grid_constant__ CUtensorMap map_d2) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    extern __shared__ unsigned char fw_smem_raw[];
    FwSmem & S = *reinterpret_cast<FwSmem *>(fw_smem_raw + ((1024u - (tc_smem_u32(fw_smem_raw) & 1023u)) & 1023u));
    const int tid = threadIdx.x, warp = __shfl_sync(LKB_FULL, tid >> 5, 0), lane = tid & 31;
    const int n_mt = g.perm ? min(*g.ntiles, max_tiles) : (g.ntok + FW_TOK - 1) / FW_TOK;
    const int n_rt = EPI ? g.N / FW_ROWS : g.N / (2 * FW_ROWS), nstage = g.bpr / FW_KB;
    const int n_items = n_mt * n_rt * (g.perm ? 64 / FW_TOK : 1);
    if (tid == 0) {
        S.abort = 0;
        for (int i = 0; i < FW_NS; ++i) { tc_mbar_init(&S.full[i], 1); tc_mbar_init(&S.empty[i], FW_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    unsigned it = 0;
    if (warp == FW_WARPS) {
        // ============================ producer (one warp) ============================
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            const FwItem I = fw_item(g, n_mt, n_rt, item);
            if (I.cnt == 0) continue;
            int crd[4] = {0, 0, 0, 0};                                   // lane 0: tokens 0..3, lane 1: 4..7 (a dead one repeats the last)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int t = I.tstart + min(4 * (lane & 1) + q, I.cnt - 1);
                crd[q] = g.perm ? __ldg(g.perm + t) >> g.a_shift : t;
            }
            const int n_g = (I.cnt + 3) >> 2;
            const CUtensorMap * mw[2], * md[2];
            int wrow[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int row = EPI ? I.rt * FW_ROWS : (2 * I.rt + r) * FW_ROWS;
                const int seg = EPI ? r : (row < g.seg_end[0]) ? 0 : (row < g.seg_end[1]) ? 1 : 2;
                mw[r] = seg == 0 ? &map_w0 : seg == 1 ? &map_w1 : &map_w2;
                md[r] = seg == 0 ? &map_d0 : seg == 1 ? &map_d1 : &map_d2;
                wrow[r] = I.expert * rpe + row - (EPI || !seg ? 0 : g.seg_end[seg - 1]);
            }
            for (int ks = 0; ks < nstage; ++ks, ++it) {
                const unsigned stg = it % FW_NS;
                if (!tc_wait<TC_HINT_PROD>(S, &S.empty[stg], ((it / FW_NS) & 1u) ^ 1u, 11u)) { ok = false; break; }
                FwStage & T = S.st[stg];
                if (lane == 0) {
                    tc_mbar_arrive_tx(&S.full[stg], 2u * FW_ROWS * 64u + ((ks & 1) ? 0u : 2u * FW_ROWS * 16u) + (unsigned) n_g * (4u * 128u + 4u * 32u));
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        tc_tma_tile(T.q + r * (FW_ROWS * 64), mw[r], ks * (FW_KB * 16), wrow[r], &S.full[stg]);
                        if (!(ks & 1)) tc_tma_tile(&S.wsc[(it >> 1) % FW_WS][r * FW_ROWS], md[r], ks * (FW_KB * 2), wrow[r], &S.full[stg]);
                    }
                }
                __syncwarp();
                if (lane < n_g) {
                    tc_tma_gather4(&T.act[4 * lane][0], &map_a, ks * (FW_KB * 32), crd[0], crd[1], crd[2], crd[3], &S.full[stg]);
                    tc_tma_gather4(&T.asc[4 * lane][0], &map_s, ks * (FW_KB * 8), crd[0], crd[1], crd[2], crd[3], &S.full[stg]);
                }
            }
        }
        if (!ok)                                                         // copies in flight land before the block leaves (bounded)
            for (unsigned k = it < FW_NS ? 0u : it - FW_NS; k < it; ++k)
                for (unsigned i = 0; i < 4096u && !tc_mbar_try<TC_HINT_PROD>(&S.full[k % FW_NS], (k / FW_NS) & 1u); ++i) { }
    } else {
        // ============================ dots (four warps) ==============================
        const int e = warp * 32 + lane;                                  // this thread's row of both tiles
        float acc[2][FW_TOK];
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            const FwItem I = fw_item(g, n_mt, n_rt, item);
            switch (I.cnt) {
                case 0: continue;
                case 1: ok = fw_dots<FOLD, 1>(S, it, nstage, e, lane, acc); break;
                case 2: ok = fw_dots<FOLD, 2>(S, it, nstage, e, lane, acc); break;
                case 3: ok = fw_dots<FOLD, 3>(S, it, nstage, e, lane, acc); break;
                case 4: ok = fw_dots<FOLD, 4>(S, it, nstage, e, lane, acc); break;
                case 5: case 6: ok = fw_dots<FOLD, 6>(S, it, nstage, e, lane, acc); break;
                default: ok = fw_dots<FOLD, 8>(S, it, nstage, e, lane, acc); break;
            }
            if (!ok) break;
#pragma unroll
            for (int t = 0; t < FW_TOK; ++t) {
                if (t < I.cnt) {
                    const int slot = g.perm ? __ldg(g.perm + I.tstart + t) : I.tstart + t;
                    const float scl = g.scale ? __ldg(g.scale + (slot >> g.a_shift)) : 1.0f;
                    if constexpr (EPI) {
                        const int row0 = I.rt * FW_ROWS + warp * 32;
                        const float v = __fmul_rn(lkb_silu(__fmul_rn(acc[0][t], scl)), __fmul_rn(acc[1][t], scl));
                        int8_t * const qs = g.oqs + (size_t) slot * (g.okb * 32) + row0;
                        float2 * const sc = reinterpret_cast<float2 *>(g.osc) + (size_t) slot * g.okb + row0 / 32;
                        // shipped arithmetic: the block sum in the reference's fused-epilogue order; exact mode: the quantiser's butterfly
                        if (FOLD) lkb_quant_store_planar_fused_epilogue(v, qs, sc, lane);
                        else      lkb_quant_store_planar(v, qs, sc, lane);
                    } else {
                        float * const p = g.out + (size_t) slot * g.out_ld + I.rt * (2 * FW_ROWS) + e;
#pragma unroll
                        for (int r = 0; r < 2; ++r)                      // the residual add is one fused multiply-add (ref: src/prefill.cu:484-486)
                            p[r * FW_ROWS] = g.add ? fmaf(acc[r][t], scl, p[r * FW_ROWS]) : __fmul_rn(acc[r][t], scl);
                    }
                }
            }
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
int lkb_tc_make_map(CUtensorMap * m, const void * base, unsigned row_bytes, unsigned long long pitch, unsigned long long rows,
                    unsigned box_bytes, unsigned box_rows, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2);           // lkb_gemm_tc.cu

typedef void (*FwKernel)(lkb_pf_gemm, int, int, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap);
static FwKernel const FW_FORMS[4] = {k_pf_gemm_few<0, 0>, k_pf_gemm_few<0, 1>, k_pf_gemm_few<1, 0>, k_pf_gemm_few<1, 1>};      // 2 epi + fold

int lkb_gemm_few_init() {
    for (FwKernel k : FW_FORMS) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(FwSmem) + 1024);
        if (e != cudaSuccess) return -(int) e;
    }
    return LKB_OK;
}
int lkb_gemm_few_take_status() { return tc_take_status(); }

static bool fw_better(const lkb_pf_gemm * g, int max_tiles) {
    return g->perm ? max_tiles >= FW_MIN_TILES && g->ntok > 0 && g->ntok <= FW_MAX_SLOTS : g->ntok <= FW_MAX_DENSE;
}
// Test hook (not in the public header): whether a call of few tokens takes this form by itself, if its planes allow it.
extern "C" __attribute__((visibility("default"))) int lkb_debug_gemm_few_better(const lkb_pf_gemm * g, int max_tiles) { return fw_better(g, max_tiles); }

// LKB_ERR_UNSUPPORTED where another form is the better one or the planes do not have the alignment the copies ask for.
int lkb_gemm_few_launch(const lkb_pf_gemm * g, int epi, int fold, int max_tiles, cudaStream_t st) {
    if (!lkb_tensor_map_encoder()) return LKB_ERR_UNSUPPORTED;
    if (!fw_better(g, max_tiles)) return LKB_ERR_UNSUPPORTED;
    if (epi ? (g->N % FW_ROWS) : (g->N % (2 * FW_ROWS))) return LKB_ERR_UNSUPPORTED;
    if (g->bpr % 8 || (((size_t) g->aqs | (size_t) g->asc) & 15) || g->exp_stride % g->bpr) return LKB_ERR_UNSUPPORTED;
    const int nseg = epi ? 2 : (g->seg_end[0] >= g->N ? 1 : g->seg_end[1] >= g->N ? 2 : 3);
    for (int s = 0; s < nseg; ++s) if (((size_t) g->qs[s] | (size_t) g->d[s]) & 15) return LKB_ERR_UNSUPPORTED;
    // a stage takes 64 bytes of a row; fetched 256 at a time by L2 gate|up at 37 tokens took 12 us less
    const CUtensorMapL2promotion l2 = CU_TENSOR_MAP_L2_PROMOTION_L2_256B;
    const unsigned long long any = 1ull << 30;              // row bound of a plane whose extent the caller does not state: it only clips
    CUtensorMap ma, ms, mw[3], md[3];
    const unsigned long long rows = g->perm ? any : (unsigned long long) g->ntok;
    int r = lkb_tc_make_map(&ma, g->aqs, (unsigned) g->bpr * 32u, (unsigned) g->bpr * 32u, rows, FW_KB * 32u, 1u, CU_TENSOR_MAP_SWIZZLE_NONE, l2);
    if (r == LKB_OK) r = lkb_tc_make_map(&ms, g->asc, (unsigned) g->bpr * 8u, (unsigned) g->bpr * 8u, rows, FW_KB * 8u, 1u, CU_TENSOR_MAP_SWIZZLE_NONE, l2);
    for (int s = 0; s < 3 && r == LKB_OK; ++s) {
        const int src = s < nseg ? s : 0;
        r = lkb_tc_make_map(&mw[s], g->qs[src], (unsigned) g->bpr * 16u, (unsigned) g->bpr * 16u, any, 64u, FW_ROWS, CU_TENSOR_MAP_SWIZZLE_64B, l2);
        if (r == LKB_OK) r = lkb_tc_make_map(&md[s], g->d[src], (unsigned) g->bpr * 2u, (unsigned) g->bpr * 2u, any, 16u, FW_ROWS, CU_TENSOR_MAP_SWIZZLE_NONE, l2);
    }
    if (r != LKB_OK) return r;
    const dim3 grid(lkb_context().sm_count * FW_CTAS), block((FW_WARPS + 1) * 32);
    LKB_PF_LAUNCH(FW_FORMS[(epi ? 2 : 0) + (fold ? 1 : 0)], grid, block, sizeof(FwSmem) + 1024, st, *g, max_tiles, (int) (g->exp_stride / g->bpr), ma, ms,
                  mw[0], mw[1], mw[2], md[0], md[1], md[2]);
    return lkb_check_launch();
}
