// lkb_gemm_tc.cu - tensor-core form of the Q4_0 x Q8_1 GEMM (dense and grouped) for sm_100a.
//
//   out[slot][n] (+)= scale[arow] * sum_{b ascending} fma(d4[n][b], fma(d8[arow][b], F_b, -c[arow][b]), .)
//   S_b = sum_{i<32} nibble[n][b][i] * q8[arow][b][i]                     (int32, exact)
//   F_b = 12582912 + S_b (exact in fp32: |S_b| < 2^22),   c = fma(d8, 12582912, 8sum)
// This (FOLD = 1) is the arithmetic of the reference's shipped GEMM (its accumulator is seeded with the bit pattern of
// 1.5 * 2^23 and the offset is folded into a per-(token, block) constant), so fp32 results are bit-identical to that
// kernel's.  ref: src/prefill.cu:32-50,131-139,341-342,381-384.  FOLD = 0 evaluates the decode kernels' term
// fma(d4, fma(d8, float(S_b), -8sum), .) -- ref: src/quant.cuh:154-157, src/prefill.cu:391-399.
//
// One MMA per 32-element block (K = 32 int8 is one Q4_0 / Q8_1 block): the per-block scales forbid accumulating across
// blocks in the tensor core, so every block's int32 sums come back through TMEM and are folded into fp32 register
// accumulators, two FMAs per value.  That fold and the constants it reads bound the kernel: a packed fma.rn.f32x2 takes 2.1 cycles of a scheduler when
// it fetches two register pairs and 2.9 when it fetches three (measured, two warps a scheduler), and both FMAs of the fold
// have three operands that differ, so the 128 of a 16384-value block cost 370 cycles.  Integer instructions do not hide under
// them: one or two lop3 beside each make it 4.8 or 6.9 cycles.  And a 16-byte shared load costs the SM four cycles of return path,
// broadcasts too: the block's 128 loads of constants are 512 of its 600 or so cycles.
//
//   * TMEM lanes = weight rows, TMEM columns = tokens.  A work item is 256 weight rows (two 128-lane MMA tiles; the SwiGLU
//     form: 128 gate rows and the same 128 up rows) x the 1..64 tokens of one plan tile, and the MMA's N is the token count
//     rounded up to 16: no work for padding, which 128-token lane tiles paid in full (x1.25 with balanced routing, x1.5
//     with Zipf routing, x16 for a short prompt).  A thread folds two rows x up to 32 tokens: the row scales are its own
//     scalars and one 16-byte shared load {d8, d8', k, k'} serves two tokens of both rows.
//   * No integer-to-float step.  A small non-negative integer is, bit for bit, a denormal fp32 (S * 2^-149), and FMAs take
//     denormals at full rate.  A constant MMA ahead of each block's MMA seeds the accumulator with 65536, which makes every
//     block sum positive (|S_b| <= 60960); the powers of two cancel in the scales (d8 * 2^100, k * 2^-49, d4 * 2^49) and
//     k = (d8 * 12582912 - c) - 65536 * d8 is exact, so fma(d8, S, k) rounds once, to the value of fma(d8, F, -c).
//     (k: both differences are exact because c is within a factor of two of d8 * 12582912 whenever |8sum| is a Q8_1 sum, and
//     both terms are multiples of 2^10 units of d8's last place.)  Measured per block of the fold alone: 414 cycles, 548
//     with the integer add of F's bit pattern.
//   * The A operand (weights) lives in TMEM: four expansion warps turn staged nibbles into int8 with tcgen05.st, so the
//     expanded weights never touch shared memory, whose bandwidth the 16-byte fold loads need.
//   * A producer warp issues bulk tensor copies: nibble rows (64 B per row and stage), activation rows (dense: 16-row boxes;
//     grouped: row gathers through perm, four rows per copy) and weight scales (16 B per row and two stages; WCOPY below
//     has the other way and both times).  Only the activation scales travel by cp.async, six stages ahead.
//   * Persistent: one CTA per SM walks the items, expert by expert, so an expert's weights stay in L2.
// Measured, one layer's GEMMs, 64 experts, balanced routing, caches flushed before every call, us at 37 / 509 / 4096 tokens:
//   token lanes padded to 128 (before)       gate|up 284 / 312 / 740   down 152 / 159 / 388   in_proj 37 / 64 / 301
//   weight rows on lanes, one MMA issuer             82 / 126 / 632         55 /  66 / 285           25 / 53 / 256
//   ... weight scales in a ring of their own, expansion a stage at a time, no scale barriers, two issuers (this form)
//                                                    70 / 117 / 569         47 /  64 / 268           23 / 51 / 238
//   ... dense items cut to fill the waves (tc_dense_form)                                            20 / 45 / 236
//   ... SwiGLU stores two values at a time         gate|up at 4096 tokens 530; values of no token not asked 514
// (by itself the launcher takes this form above 1920 slots (480 tokens of four) grouped, and dense where that of lkb_gemm_few.cu would need the longer waves)
// With few tokens the hand-over of every block is the bound (300 to 440 cycles of polls, commits and arrivals).
// No copy in this file is a multicast one; every tensor map covers memory of the GPU the kernel runs on.
// Every wait is bounded; on expiry a status word is set and all roles drain and exit, freeing TMEM.
#include "lkb_tc.cuh"

#define TC_ROWS      128            // weight rows per MMA tile (TMEM lanes)
#define TC_TOK       64             // tokens per work item (TMEM columns of one tile's block sums)
#define TC_KB        4              // blocks per pipeline stage = 128 bytes of K per activation row
#define TC_NS        5              // stages
#define TC_DBUF      2              // block-sum buffers, 256 TMEM columns in all: block j of a stage lands in buffer j & 1
#define TC_AUNITS    2              // A buffers of one stage (2 tiles x 4 blocks x 8 TMEM columns)
#define TC_COL_A     256            // first TMEM column of the A buffers
#define TC_COL_SEED  384            // 8 columns of the constant A operand
#define TC_EPI_WARPS 8              // warps 0..7: lane quadrant = warp & 3, column half = warp >> 2
#define TC_EXP_W0    8              // expansion warps 8..11: quadrant = warp & 3
#define TC_EXP_WARPS 4
#define TC_MMA_WARP  12             // MMA issuers 12, 13
#define TC_PROD_WARP 14             // warp 15 only completes the warpgroup that setmaxnreg needs
#define TC_THREADS   512
#define TC_SC_AHEAD  6              // stages the activation scales are requested ahead
#define TC_SC_RING   8              // stages of activation scales in shared memory (read by the thread that requests them)
#define TC_WS_RING   16             // stages of weight scales: the epilogue reads them up to TC_NS stages behind the expansion
#define TC_MAGIC_I   0x4B400000
#define TC_MAGIC_F   12582912.0f
#define TC_SEED      65536.0f       // 32 products 64 * 32
#define TC_UP100     1.2676506002282294e30f     // 2^100
#define TC_UP49      562949953421312.0f         // 2^49
#define TC_DOWN49    1.7763568394002505e-15f    // 2^-49

struct TcStage {
    alignas(1024) unsigned char act[TC_TOK * 128];      // activations: row r at r*128, 16-byte chunk c at c ^ (r & 7)
    alignas(1024) unsigned char rawq[2 * TC_ROWS * 64]; // nibbles as in the pack: row r at r*64, chunk c at c ^ ((r >> 1) & 3)
};
static_assert(sizeof(TcStage) % 1024 == 0, "stages keep the 1024-byte alignment of the swizzled operands");
static_assert(TC_SC_RING > TC_NS, "constants stay until the epilogue has read them: see the expansion warps");
static_assert(TC_WS_RING >= 2 * TC_NS + 2 && TC_WS_RING >= TC_SC_AHEAD + TC_NS + 2 && !(TC_WS_RING & (TC_WS_RING - 1)), "weight scales stay until the epilogue has read them");

struct TcSmem {
    TcStage st[TC_NS];
    alignas(1024) unsigned seed_b[TC_TOK * 8];                              // constant B operand: 64 rows of 32 bytes
    alignas(16) float4 dk[TC_SC_RING][TC_KB][TC_TOK / 2];                   // per stage, block and token pair {d8, d8', k, k'}
    alignas(128) uint4 wsc[TC_WS_RING / 2][2 * TC_ROWS];                    // eight fp16 scales per row (two stages)
    alignas(16) float4 asc[TC_SC_RING][TC_EXP_WARPS * 32];                  // (d8, 8sum) of two blocks per expansion thread
    alignas(8) unsigned long long full[TC_NS], empty[TC_NS], afull[TC_AUNITS], aempty[TC_AUNITS], tfull[2][TC_DBUF], tempty[2][TC_DBUF];
    unsigned tmem_base;
    int      abort;
};

// The constant B operand: rows of 32 bytes, 32-byte swizzle (every byte is the same).
__device__ __forceinline__ unsigned long long tc_desc_seed(unsigned smem_addr) {
    return (unsigned long long) ((smem_addr >> 4) & 0x3FFFu) | (1ull << 16)
         | ((unsigned long long) (256u >> 4) << 32) | (1ull << 46) | (6ull << 61);
}
// s8 x s8 -> s32, M = 128, N from the item, B K-major
#define TC_IDESC(n) (0x20u | (1u << 7) | (1u << 10) | (((unsigned) (n) >> 3) << 17) | ((TC_ROWS >> 4) << 24))

// The dense form's items: tokens per item, and two 128-row tiles or one.  tc_dense_form (host) chooses.
struct TcDense { int tw, wide; };
// What every role derives from the launch arguments: the shape of the item grid.
struct TcPlan {
    int n_rt;            // row tiles per token tile
    int n_items;
    int wide;            // plain form: an item is two 128-row tiles (1) or one (0)
    int nstage;          // pipeline stages per item
    int tw;              // dense: tokens per item
};
struct TcItem { int expert, tstart, tcnt, rt; };
__device__ __forceinline__ TcItem tc_item(const lkb_pf_gemm & g, const TcPlan & P, int item) {
    TcItem I;
    const int mt = item / P.n_rt;
    I.rt = item - mt * P.n_rt;
    if (g.perm) {
        const int4 tl = __ldg(reinterpret_cast<const int4 *>(g.tiles) + mt);
        I.expert = tl.x; I.tstart = tl.y; I.tcnt = tl.z;
    } else {
        I.expert = 0; I.tstart = mt * P.tw; I.tcnt = min(P.tw, g.ntok - I.tstart);
    }
    return I;
}
__device__ __forceinline__ int tc_cols(int tcnt) { return (tcnt + 15) & ~15; }          // N of the item's MMAs
// First output row of tile r of the item (plain form), and whether the item has a second tile.
__device__ __forceinline__ int tc_tile_row(const TcPlan & P, int rt, int r) { return (P.wide ? 2 * rt + r : rt) * TC_ROWS; }
template <int EPI>
__device__ __forceinline__ bool tc_two(const lkb_pf_gemm & g, const TcPlan & P, int rt) {
    return EPI || (P.wide && tc_tile_row(P, rt, 1) < g.N);
}
__device__ __forceinline__ int tc_seg(const lkb_pf_gemm & g, int row) { return (row < g.seg_end[0]) ? 0 : (row < g.seg_end[1]) ? 1 : 2; }

// ---------------------------------------------------------------------------
// Epilogue state carried from item to item by every epilogue thread.
// ---------------------------------------------------------------------------
// Block-sum buffers and who fills them.  Free halves (SwiGLU form): each column half has two buffers and an MMA issuer of its
// own, so the four warps of a half never wait for the other four, which matters where the item ends in the long SwiGLU store
// (gate|up at 4096 tokens -4 %, at 509 -3 %, at 37 +2 %).  Plain form: one 64-column MMA per tile, common
// buffers, issuer h for buffer h; half the MMAs (down and in_proj at 37 tokens 4 % faster than with free halves, equal at 4096).
template <int EPI> struct TcSums {
    static constexpr int FREE = EPI, TILE = FREE ? TC_TOK / 2 : TC_TOK, BUF = 2 * TILE;      // columns between tiles, between buffers
    static constexpr int EPI_ARRIVE = FREE ? TC_EPI_WARPS / 2 : TC_EPI_WARPS;
};

struct TcEpi { unsigned it; };      // the number of the next stage

// Fold NL columns, from column C0 on, of one block into R rows' accumulators.
template <int FOLD, int R, int NC, int C0, int NL>
__device__ __forceinline__ void tc_fold(unsigned long long (&acc)[R][NC / 2], const unsigned (&sv)[R][NL], const float4 (&dk)[NL / 2],
                                        const unsigned long long (&ep)[2]) {
    const unsigned long long nmag = tc_pack(-TC_MAGIC_F, -TC_MAGIC_F);
#pragma unroll
    for (int i = 0; i < NL / 2; ++i) {
        const float4 q = dk[i];
        const unsigned long long d = tc_pack(q.x, q.y), k = tc_pack(q.z, q.w);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            unsigned long long f;
            if (FOLD) f = tc_pack_u(sv[r][2 * i], sv[r][2 * i + 1]);                 // the block sums as denormals
            else      f = tc_fadd2(tc_pack_u(sv[r][2 * i] + TC_MAGIC_I, sv[r][2 * i + 1] + TC_MAGIC_I), nmag);   // float(S), exact
            acc[r][C0 / 2 + i] = tc_ffma2(ep[r], tc_ffma2(d, f, k), acc[r][C0 / 2 + i]);
        }
    }
}

template <int FOLD> __device__ __forceinline__ float tc_row_scale(__half d4) {
    const float f = __half2float(d4);
    return FOLD ? __fmul_rn(f, TC_UP49) : f;
}

// All blocks of one item for this thread's R rows x NC tokens, as a software pipeline over column halves: while one half's
// sums are folded the TMEM load of the next half (of this block, or of the next one) is in flight.  (Whole-block double
// buffering needs 128 registers for the sums beside the 64 accumulators and leaves none to run the scale loads ahead.)
// Returns false when a wait gave up.
template <int EPI, int FOLD, int R, int NC>
__device__ __forceinline__ bool tc_fold_item(TcSmem & S, TcEpi & X, unsigned tbase, int half, int row, int lane, int nstage,
                                             unsigned long long (&acc)[R][NC / 2]) {
    constexpr int NA = NC == 24 ? 16 : NC == 8 ? 8 : NC / 2, NB = NC - NA;              // columns of the two halves (8: one piece)
    unsigned sva[R][NA], svb[R][NB ? NB : 8];
    using L = TcSums<EPI>;
    const unsigned tcol = tbase + half * (L::FREE ? 2 * L::BUF : NC);
    unsigned long long * const tfull = S.tfull[L::FREE ? half : 0], * const tempty = S.tempty[L::FREE ? half : 0];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < NC / 2; ++i) acc[r][i] = 0ull;
    if (!tc_wait(S, &tfull[0], 0u, 31u)) return false;
    tc_fence_after();
#pragma unroll
    for (int r = 0; r < R; ++r) tc_ld<NA>(tcol + r * L::TILE, sva[r]);
    for (int ks = 0; ks < nstage; ++ks) {
        __half we[2][TC_KB];                                                          // this thread's row scales of the stage
#pragma unroll
        for (int r = 0; r < R; ++r)
            *reinterpret_cast<uint2 *>(we[r]) = *(reinterpret_cast<const uint2 *>(&S.wsc[(X.it >> 1) & (TC_WS_RING / 2 - 1)][r * TC_ROWS + row]) + (X.it & 1u));
        // Two blocks per trip: buffers are then fixed (block j -> j & 1) and the phase parity is the trip number (a stage
        // uses each buffer twice), which keeps the synchronisation to a handful of instructions with fixed addresses.
#pragma unroll
        for (unsigned u = 0; u < 2; ++u) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 * dk = &S.dk[X.it & (TC_SC_RING - 1)][2 * u + h][(half * NC) / 2];
                const float e0 = tc_row_scale<FOLD>(we[0][2 * u + h]), e1 = R == 2 ? tc_row_scale<FOLD>(we[1][2 * u + h]) : 0.0f;
                const unsigned long long ep[2] = {tc_pack(e0, e0), tc_pack(e1, e1)};
                const bool more = h == 0 || u == 0 || ks < nstage - 1;
                float4 ka[NA / 2], kb[NB ? NB / 2 : 4];
#pragma unroll
                for (int i = 0; i < NA / 2; ++i) ka[i] = dk[i];
#pragma unroll
                for (int i = 0; i < NB / 2; ++i) kb[i] = dk[NA / 2 + i];
                tc_wait_ld();                                                         // the first half is in sva
                // (polled ahead of the fold and looked at behind it: the answer's latency is hidden)
                const bool ready = more && tc_mbar_try<0>(&tfull[h ^ 1], h == 0 ? u : u ^ 1u);
                if constexpr (NB > 0) {
#pragma unroll
                    for (int r = 0; r < R; ++r) tc_ld<NB ? NB : 8>(tcol + h * L::BUF + r * L::TILE + NA, svb[r]);
                    tc_fold<FOLD, R, NC, 0, NA>(acc, sva, ka, ep);
                    tc_wait_ld();
                } else tc_fold<FOLD, R, NC, 0, NA>(acc, sva, ka, ep);
                tc_fence_before();
                __syncwarp();
                tc_mbar_arrive_if(&tempty[h], lane == 0);                           // the buffer is free again
                if (more) {
                    if (!ready && !tc_wait(S, &tfull[h ^ 1], h == 0 ? u : u ^ 1u, 31u)) return false;
                    tc_fence_after();
#pragma unroll
                    for (int r = 0; r < R; ++r) tc_ld<NA>(tcol + (h ^ 1) * L::BUF + r * L::TILE, sva[r]);
                }
                if constexpr (NB > 0) tc_fold<FOLD, R, NC, NA, NB ? NB : 8>(acc, svb, kb, ep);
            }
        }
        ++X.it;
    }
    return true;
}

// Column c of this thread's accumulators.
template <int NC> __device__ __forceinline__ float tc_col(const unsigned long long (&acc)[NC / 2], int c) {
    float x, y;
    tc_unpack(acc[c >> 1], x, y);
    return (c & 1) ? y : x;
}

// What lane i knows of token half * NC + i: its slot and its row scale.  Asked for ahead of an item's fold: two loads, one after the other,
// that the item's store would wait for.
struct TcTok { int slot; float scl; bool live; };
template <int NC>
__device__ __forceinline__ TcTok tc_tok(const lkb_pf_gemm & g, const TcItem & I, int half, int lane) {
    TcTok K;
    const int tl = half * NC + lane;
    K.live = lane < NC && tl < I.tcnt;
    K.slot = K.live ? (g.perm ? __ldg(g.perm + I.tstart + tl) : I.tstart + tl) : 0;
    K.scl = (K.live && g.scale) ? __ldg(g.scale + (K.slot >> g.a_shift)) : 1.0f;
    return K;
}

// Plain output: lane = weight row, so a token's 32 rows of a warp are one 128-byte store.
template <int R, int NC>
__device__ __forceinline__ void tc_store_plain(const lkb_pf_gemm & g, const TcPlan & P, const TcItem & I, const TcTok & K, float * const * out_rows, int half,
                                               int row, int lane, const unsigned long long (&acc)[R][NC / 2]) {
    // out_rows: a row address of its own per slot (the expert-parallel form: the row goes straight into its home rank's buffer, a
    // peer's memory included -- plain stores)
    const bool live = K.live;
    const int slot = K.slot;
    const float scl = K.scl;
    const unsigned long long rp = !live ? 0ull : (unsigned long long) (out_rows ? out_rows[slot] : g.out + (size_t) slot * g.out_ld);
    const int o0 = tc_tile_row(P, I.rt, 0) + row;
    const int nlive = I.tcnt - half * NC;                                             // live tokens of this warp
#pragma unroll
    for (int c0 = 0; c0 < NC; c0 += 8) {
        if (c0 < nlive) {
            float * p[8]; float s[8], prev[8][R];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                p[c] = reinterpret_cast<float *>(__shfl_sync(LKB_FULL, rp, c0 + c)) + o0;
                s[c] = __shfl_sync(LKB_FULL, scl, c0 + c);
            }
            if (g.add) {
#pragma unroll
                for (int c = 0; c < 8; ++c)
#pragma unroll
                    for (int r = 0; r < R; ++r) prev[c][r] = c0 + c < nlive ? p[c][r * TC_ROWS] : 0.0f;
            }
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (c0 + c < nlive) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float a = tc_col<NC>(acc[r], c0 + c);
                        // the residual add is one fused multiply-add, as the reference's build contracts it
                        // (src/prefill.cu:484-486)
                        p[c][r * TC_ROWS] = g.add ? fmaf(a, s[c], prev[c][r]) : __fmul_rn(a, s[c]);
                    }
                }
        }
    }
}

// One level of the block-sum butterfly over lane bit B (xor 1 << B) on an array indexed by token: while the tokens still
// differ in bit B of their index a lane keeps the half whose bit equals its own and hands over the other (half the
// shuffles, and lane t ends with token t); tokens beyond that are summed in place.  Fp32 addition is commutative, so every
// partial sum has the operands of the plain butterfly.  K: the index bits already split off.
template <int N, int B, int K>
__device__ __forceinline__ void tc_sum_level(float (&t)[N], int lane) {
    if constexpr ((1 << B) < N) {
        const bool up = (lane >> B) & 1;
#pragma unroll
        for (int c = 0; c < N; ++c)
            if (!(c & (1 << B)) && !(c & K)) {
                const float keep = up ? t[c | (1 << B)] : t[c];
                const float give = up ? t[c] : t[c | (1 << B)];
                t[c] = __fadd_rn(keep, __shfl_xor_sync(LKB_FULL, give, 1 << B));
            }
    } else {
#pragma unroll
        for (int c = 0; c < N; ++c)
            if (!(c & K)) t[c] = __fadd_rn(t[c], __shfl_xor_sync(LKB_FULL, t[c], 1 << B));
    }
}

// SwiGLU + Q8_1 of NT tokens (columns c0.. of the accumulators): a warp holds one 32-row output block (lane = row).
template <int FOLD, int NC, int NT>
__device__ __forceinline__ void tc_store_swiglu(const lkb_pf_gemm & g, const TcItem & I, const TcTok & K, int half, int c0, int quad, int lane,
                                                const unsigned long long (&acc)[2][NC / 2]) {
    const int row0 = I.rt * TC_ROWS + quad * 32;                                      // first output row of this warp's block
    const int nlive = I.tcnt - (half * NC + c0);
    if (row0 >= g.N || nlive <= 0) return;
    const int slot = __shfl_sync(LKB_FULL, K.slot, c0 + lane);                        // lane t: token c0 + t
    const bool live = lane < NT && half * NC + c0 + lane < I.tcnt;
    float v[NT], t[NT];
    unsigned my_am = 0;
    bool sure = true;
#pragma unroll
    for (int c = 0; c < NT; c += 2) {                                                 // two tokens at a time
        const unsigned long long s = tc_pack(__shfl_sync(LKB_FULL, K.scl, c0 + c), __shfl_sync(LKB_FULL, K.scl, c0 + c + 1));
        bool ok = true;
        tc_unpack(tc_fmul2(tc_silu2(tc_fmul2(acc[0][(c0 + c) / 2], s), ok), tc_fmul2(acc[1][(c0 + c) / 2], s)), v[c], v[c + 1]);
        sure = sure && (ok || c + 1 >= nlive);
    }
    if ((nlive & 1) && nlive < NT) {                                                  // the last token, whose pair has another that is none
        float last = 0.0f;
#pragma unroll
        for (int c = 0; c < NT; c += 2) if (c + 1 == nlive) last = tc_col<NC>(acc[0], c0 + c);
        tc_silu2(tc_pack(__fmul_rn(last, __shfl_sync(LKB_FULL, K.scl, c0 + nlive - 1)), 1.0f), sure);
    }
    if (!__all_sync(LKB_FULL, sure)) {
#pragma unroll
        for (int c = 0; c < NT; ++c) {
            const float s = __shfl_sync(LKB_FULL, K.scl, c0 + c);
            v[c] = __fmul_rn(lkb_silu(__fmul_rn(tc_col<NC>(acc[0], c0 + c), s)), __fmul_rn(tc_col<NC>(acc[1], c0 + c), s));
        }
    }
#pragma unroll
    for (int c = 0; c < NT; ++c) {
        t[c] = v[c];
        const unsigned am = __reduce_max_sync(LKB_FULL, __float_as_uint(fabsf(v[c])));
        if (lane == c) my_am = am;
    }
    // lane t: block sum of token t.  Shipped arithmetic: the order of the reference's fused epilogue, where a lane adds rows
    // (g, g+8) + (g+16, g+24) and the eight lanes then pair over g ^ 1, 2, 4 (src/prefill.cu:424-448); exact mode: the
    // xor-butterfly order of the warp quantiser (16, 8, 4, 2, 1).
    if (FOLD) {
        tc_sum_level<NT, 3, 0>(t, lane); tc_sum_level<NT, 4, 8>(t, lane); tc_sum_level<NT, 0, 24>(t, lane);
        tc_sum_level<NT, 1, 25>(t, lane); tc_sum_level<NT, 2, 27>(t, lane);
    } else {
        tc_sum_level<NT, 4, 0>(t, lane); tc_sum_level<NT, 3, 16>(t, lane); tc_sum_level<NT, 2, 24>(t, lane);
        tc_sum_level<NT, 1, 28>(t, lane); tc_sum_level<NT, 0, 30>(t, lane);
    }
    const float d_l = __fdiv_rn(__uint_as_float(my_am), 127.0f);
    float rd_l;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rd_l) : "f"(d_l));
    if (live) {
        const __half2 ds = __floats2half2_rn(d_l, t[0]);
        reinterpret_cast<float2 *>(g.osc)[(size_t) slot * g.okb + row0 / 32] = make_float2(__low2float(ds), __fmul_rn(8.0f, __high2float(ds)));
    }
    int8_t * const oq = g.oqs + row0 + lane;
    const int pitch = g.okb * 32;
    // q = roundf(v / d) by the reciprocal, with the division for elements near a tie (see lkb_quad_quant_ds)
#pragma unroll
    for (int b = 0; b < NT; b += 8) {
        if (b < nlive) {
            float q[8];
            sure = true;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float rd = __shfl_sync(LKB_FULL, rd_l, b + c);
                q[c] = fmaf(v[b + c], rd, TC_MAGIC_F);
                const float diff = fmaf(v[b + c], rd, -__fadd_rn(q[c], -TC_MAGIC_F));
                sure = sure && (fabsf(diff) < 0.4999f || b + c >= nlive);
            }
            if (!__all_sync(LKB_FULL, sure)) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float d = __shfl_sync(LKB_FULL, d_l, b + c);
                    const unsigned am = __shfl_sync(LKB_FULL, my_am, b + c);
                    const float r = roundf(__fdiv_rn(v[b + c], d));
                    if (!sure) q[c] = (am != 0u && r == r) ? __fadd_rn(r, TC_MAGIC_F) : TC_MAGIC_F;   // (int) NaN is 0; an all-zero block is 0
                }
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int sl = __shfl_sync(LKB_FULL, slot, b + c);
                if (b + c < nlive) oq[(size_t) sl * pitch] = (int8_t) __float_as_uint(q[c]);
            }
        }
    }
}

template <int EPI, int FOLD, int R, int NC>
__device__ __forceinline__ bool tc_epilogue_item(TcSmem & S, TcEpi & X, const lkb_pf_gemm & g, const TcPlan & P, const TcItem & I, float * const * out_rows,
                                                 unsigned tbase, int half, int quad, int lane) {
    unsigned long long acc[R][NC / 2];
    const TcTok K = tc_tok<NC>(g, I, half, lane);
    if (!tc_fold_item<EPI, FOLD, R, NC>(S, X, tbase, half, quad * 32 + lane, lane, P.nstage, acc)) return false;
    if constexpr (EPI == 0) tc_store_plain<R, NC>(g, P, I, K, out_rows, half, quad * 32 + lane, lane, acc);
    else if constexpr (NC == 8) tc_store_swiglu<FOLD, NC, 8>(g, I, K, half, 0, quad, lane, acc);
    else {
        tc_store_swiglu<FOLD, NC, 16>(g, I, K, half, 0, quad, lane, acc);
        if constexpr (NC == 24) tc_store_swiglu<FOLD, NC, 8>(g, I, K, half, 16, quad, lane, acc);
        if constexpr (NC == 32) tc_store_swiglu<FOLD, NC, 16>(g, I, K, half, 16, quad, lane, acc);
    }
    return true;
}
template <int EPI, int FOLD, int R>
__device__ __forceinline__ bool tc_epilogue_cols(TcSmem & S, TcEpi & X, const lkb_pf_gemm & g, const TcPlan & P, const TcItem & I, float * const * out_rows,
                                                 unsigned tbase, int half, int quad, int lane) {
    switch (tc_cols(I.tcnt)) {                                  // columns split between the two warps of a quadrant
        case 16: return tc_epilogue_item<EPI, FOLD, R, 8>(S, X, g, P, I, out_rows, tbase, half, quad, lane);
        case 32: return tc_epilogue_item<EPI, FOLD, R, 16>(S, X, g, P, I, out_rows, tbase, half, quad, lane);
        case 48: return tc_epilogue_item<EPI, FOLD, R, 24>(S, X, g, P, I, out_rows, tbase, half, quad, lane);
        default: return tc_epilogue_item<EPI, FOLD, R, 32>(S, X, g, P, I, out_rows, tbase, half, quad, lane);
    }
}

// ---------------------------------------------------------------------------
// EPI 0: out (+)= scale * acc           (item: 256 rows, or 128, of one or two weight segments)
// EPI 1: SwiGLU + Q8_1                  (item: 128 gate rows and the same 128 up rows)
// rpe = weight rows per expert (exp_stride / bpr).  sc_plane / s_pitch: the (d8, 8sum) pairs of the activation rows.
// WCOPY 1: weight scales by tensor copy; 0: by the expansion warps' own 8-byte cp.async, for scale planes that start on an
// 8-byte boundary, where no tensor copy can (for the rest it is the slower one: see the copies above).
// ---------------------------------------------------------------------------
template <int EPI, int FOLD, int WCOPY>
__global__ void __launch_bounds__(TC_THREADS, 1) k_pf_gemm_tc(const lkb_pf_gemm g, const int max_tiles, const int rpe,
                                                              const char * __restrict__ sc_plane, const int s_pitch,
                                                              const __grid_constant__ CUtensorMap map_a,
                                                              const __grid_constant__ CUtensorMap map_w0,
                                                              const __grid_constant__ CUtensorMap map_w1,
                                                              const __grid_constant__ CUtensorMap map_w2,
                                                              const __grid_constant__ CUtensorMap map_d0,
                                                              const __grid_constant__ CUtensorMap map_d1,
                                                              const __grid_constant__ CUtensorMap map_d2,
                                                              float * const * __restrict__ out_rows, const TcDense dense) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    extern __shared__ unsigned char tc_smem_raw[];
    // the swizzle patterns are functions of the shared-memory address: stages start on 1024-byte boundaries
    TcSmem & S = *reinterpret_cast<TcSmem *>(tc_smem_raw + ((1024u - (tc_smem_u32(tc_smem_raw) & 1023u)) & 1023u));
    const int ptid = threadIdx.x, warp = __shfl_sync(LKB_FULL, ptid >> 5, 0), lane = ptid & 31;

    // ---- item grid: (token tile, row tile), row tiles fastest --------------------
    TcPlan P;
    P.tw = dense.tw;
    const int n_mt = g.perm ? min(*g.ntiles, max_tiles) : (g.ntok + P.tw - 1) / P.tw;
    P.wide = 1;
    P.n_rt = EPI ? (g.N + TC_ROWS - 1) / TC_ROWS : (g.N + 2 * TC_ROWS - 1) / (2 * TC_ROWS);
    // No more 128-row tiles than CTAs: one per item.  An item's time there is the latency of its chain of blocks, and twice the CTAs
    // share the weight stream.
    if (!EPI && (g.perm ? n_mt * (g.N / TC_ROWS) <= (int) gridDim.x : !dense.wide)) { P.wide = 0; P.n_rt = g.N / TC_ROWS; }
    P.n_items = n_mt * P.n_rt;
    P.nstage = g.bpr / TC_KB;
    if ((int) blockIdx.x >= P.n_items) return;

    // ---- set-up: barriers, TMEM, the constant operands ---------------------------
    if (ptid == 0) {
        S.abort = 0;
        for (int i = 0; i < TC_NS; ++i) {
            tc_mbar_init(&S.full[i], 1);                              // the lane that posts the bytes
            tc_mbar_init(&S.empty[i], 2);                       // both issuers' commits
        }
        for (int i = 0; i < TC_AUNITS; ++i) { tc_mbar_init(&S.afull[i], TC_EXP_WARPS); tc_mbar_init(&S.aempty[i], 2); }
        for (int i = 0; i < 2 * TC_DBUF; ++i) { tc_mbar_init(&S.tfull[0][i], 2); tc_mbar_init(&S.tempty[0][i], TcSums<EPI>::EPI_ARRIVE); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(tc_smem_u32(&S.tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (FOLD) {
        for (int i = ptid; i < TC_TOK * 8; i += TC_THREADS) S.seed_b[i] = 0x20202020u;
        tc_fence_async();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = S.tmem_base;
    if (FOLD && warp < 4) {
        const uint4 c = make_uint4(0x40404040u, 0x40404040u, 0x40404040u, 0x40404040u);
        tc_st8(tmem + ((unsigned) (warp * 32) << 16) + TC_COL_SEED, c, c);
        tc_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // Registers follow the work (setmaxnreg sits inside the branch it governs: after a join the compiler must assume the
    // smaller limit).  208 + 208 + 56 + 40 = the 4 x 128 the block was launched with.
    if (warp >= TC_MMA_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        // ============================ producer (one warp) ============================
        if (warp == TC_PROD_WARP) {
            constexpr int BR = EPI ? 64 : TC_ROWS, NB = 2 * TC_ROWS / BR;       // rows of a box; boxes of an item
            unsigned it = 0;
            bool ok = true;
            TcItem I = tc_item(g, P, blockIdx.x);
            for (int item = blockIdx.x; item < P.n_items && ok; item += gridDim.x) {
                // grouped: lane l fetches the activation rows of tokens 4l..4l+3 (a dead token repeats a live one: its
                // column is never stored)
                int crd[4] = {0, 0, 0, 0};
                if (g.perm) {
                    int last = 0;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int rr = 4 * lane + q;
                        if (rr < I.tcnt) last = __ldg(g.perm + I.tstart + rr) >> g.a_shift;
                        crd[q] = last;
                    }
                }
                const bool glive = g.perm && 4 * lane < I.tcnt;
                // weight rows: boxes of 64 rows (SwiGLU form, where half a tile may be missing) or of a whole tile
                const CUtensorMap * mw[2], * md[2];
                int wrow[2];
                unsigned boxes = 0;
                if (EPI) {
                    mw[0] = &map_w0; mw[1] = &map_w1; md[0] = &map_d0; md[1] = &map_d1;
                    wrow[0] = wrow[1] = I.expert * rpe + I.rt * TC_ROWS;
                    boxes = (g.N - I.rt * TC_ROWS >= TC_ROWS) ? 15u : 5u;              // N % 64 == 0: half a tile may be missing
                } else {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int row = tc_tile_row(P, I.rt, r);
                        if (r && !tc_two<EPI>(g, P, I.rt)) { mw[r] = &map_w0; md[r] = &map_d0; wrow[r] = 0; continue; }
                        const int seg = tc_seg(g, row);
                        mw[r] = seg == 0 ? &map_w0 : seg == 1 ? &map_w1 : &map_w2;
                        md[r] = seg == 0 ? &map_d0 : seg == 1 ? &map_d1 : &map_d2;
                        wrow[r] = I.expert * rpe + row - (seg ? g.seg_end[seg - 1] : 0);
                        boxes |= 1u << r;
                    }
                }
                const int abox = tc_cols(I.tcnt) / 16, tstart = I.tstart;
                const unsigned bytes = (unsigned) __popc(boxes) * (BR * 64u) + (g.perm ? 512u * (unsigned) ((I.tcnt + 3) >> 2) : 2048u * (unsigned) abox);
                if (item + (int) gridDim.x < P.n_items) I = tc_item(g, P, item + gridDim.x);
                for (int ks = 0; ks < P.nstage; ++ks, ++it) {
                    const unsigned stg = it % TC_NS;
                    if (!tc_wait<TC_HINT_PROD>(S, &S.empty[stg], ((it / TC_NS) & 1u) ^ 1u, 10u)) { ok = false; break; }
                    TcStage & T = S.st[stg];
                    if (lane == 0) {
                        tc_mbar_arrive_tx(&S.full[stg], bytes + (!WCOPY || (ks & 1) ? 0u : (unsigned) __popc(boxes) * (BR * 16u)));
#pragma unroll
                        for (int b = 0; b < NB; ++b) {
                            const int r = b / (NB / 2);
                            if ((boxes >> b) & 1u) tc_tma_tile(T.rawq + b * (BR * 64), mw[r], ks * (TC_KB * 16), wrow[r] + BR * b - TC_ROWS * r, &S.full[stg]);
                        }
                        if (WCOPY && !(ks & 1)) {                                      // the scales of two stages: 16 bytes a row
#pragma unroll
                            for (int b = 0; b < NB; ++b) {
                                const int r = b / (NB / 2);
                                if ((boxes >> b) & 1u) tc_tma_tile(&S.wsc[(it >> 1) % (TC_WS_RING / 2)][BR * b], md[r], ks * (TC_KB * 2), wrow[r] + BR * b - TC_ROWS * r, &S.full[stg]);
                            }
                        }
                        if (!g.perm)
                            for (int b = 0; b < abox; ++b) tc_tma_tile(T.act + b * 2048, &map_a, ks * 128, tstart + 16 * b, &S.full[stg]);
                    }
                    __syncwarp();
                    if (glive) tc_tma_gather4(T.act + lane * 512, &map_a, ks * 128, crd[0], crd[1], crd[2], crd[3], &S.full[stg]);
                }
            }
            tc_drain<TC_NS>(S.full, it);
        }
        // ============================ MMA issuers (two warps) ========================
        // Issuer q serves column half q (free halves) or block-sum buffer q, that is blocks q and q + 2 of every stage: polls,
        // issue and commits of a block take some 200 cycles, and one issuer for everything made that a serial part of the loop.
        // The whole warp runs the loop, so that descriptors and addresses stay in uniform registers; one elected lane issues.
        else if (warp < TC_MMA_WARP + 2) {
            using L = TcSums<EPI>;
            const unsigned q = warp - TC_MMA_WARP;
            unsigned stg = 0, par = 0, apar = 0, ab = 0;          // stage and its parity; A buffer and its
            bool ok = true;
            const unsigned long long dseed = tc_desc_seed(tc_smem_u32(S.seed_b));
            const unsigned d0 = tmem + (L::FREE ? q * (2 * L::BUF) : 0);
            unsigned long long * const tfull = S.tfull[L::FREE ? q : 0], * const tempty = S.tempty[L::FREE ? q : 0];
            const bool leader = tc_elect();
            TcItem I = tc_item(g, P, blockIdx.x);
            for (int item = blockIdx.x; item < P.n_items && ok; item += gridDim.x) {
                const unsigned nc = tc_cols(I.tcnt) / 2;          // columns of a half; the MMA's N is a multiple of 16 (rows past the half are dead)
                const unsigned idesc = TC_IDESC(L::FREE ? (nc + 15) & ~15u : 2 * nc);
                const bool two = tc_two<EPI>(g, P, I.rt);
                if (item + (int) gridDim.x < P.n_items) I = tc_item(g, P, item + gridDim.x);
                for (int ks = 0; ks < P.nstage && ok; ++ks) {
                    if (!tc_wait<TC_HINT_MMA>(S, &S.full[stg], par, 20u)) { ok = false; break; }
                    if (!tc_wait<TC_HINT_MMA>(S, &S.afull[ab], apar, 22u)) { ok = false; break; }
                    const unsigned long long b0 = tc_desc(tc_smem_u32(S.st[stg].act) + (L::FREE ? q * nc * 128 : 0));
                    const unsigned a0 = tmem + TC_COL_A + ab * 64;
#pragma unroll
                    for (unsigned i = 0; i < (L::FREE ? TC_KB : TC_KB / 2); ++i) {
                        const unsigned j = L::FREE ? i : 2 * i + q, h = L::FREE ? i & 1 : q;
                        // use k of a buffer waits for phase k: the epilogue releases every buffer once up front
                        if (!tc_wait<TC_HINT_MMA>(S, &tempty[h], L::FREE ? i >> 1 : i, 21u)) { ok = false; break; }
                        tc_fence_after();
                        if (leader) {
                            const unsigned d = d0 + h * L::BUF, a = a0 + j * 8;
                            const unsigned long long b = b0 + j * 2;               // a block is 32 bytes, in 16-byte units
                            if (FOLD) {
                                tc_mma_i8(d, tmem + TC_COL_SEED, dseed, idesc, 0u);
                                if (two) tc_mma_i8(d + L::TILE, tmem + TC_COL_SEED, dseed, idesc, 0u);
                            }
                            tc_mma_i8(d, a, b, idesc, FOLD);
                            if (two) tc_mma_i8(d + L::TILE, a + 32, b, idesc, FOLD);
                            tc_commit(&tfull[h]);                                  // this block's sums are ready
                            tc_mbar_arrive(&tfull[h]);                             // and this thread has acquired the stage's scales and constants
                            if (i + 1 == (L::FREE ? TC_KB : TC_KB / 2)) { tc_commit(&S.aempty[ab]); tc_commit(&S.empty[stg]); }    // the stage has been read
                        }
                        __syncwarp();
                    }
                    if (++stg == TC_NS) { stg = 0; par ^= 1u; }
                    ab ^= 1u;
                    if (ab == 0) apar ^= 1u;
                }
            }
        }
    }
    // ============================ expansion (four warps) ==========================
    // The epilogue waits for block sums only.  It reads weight scales (a tensor copy's writes, acquired here with full) and
    // constants (these warps' own stores) because afull releases them to the issuers, and an issuer's thread arrives on every
    // tfull itself, beside the commit of its MMAs: what a tcgen05.commit alone makes visible of other threads' writes is not
    // documented.  (The epilogue waiting for afull as well, once a stage and polled a block ahead, cost 2 to 4 %.)
    // Nothing is handed back: a stage comes round (empty) when the issuers have passed it, and a buffer they reused was
    // released behind every read of the stage before, so rings of more than TC_NS + 1 stages are never overwritten early.
    // Thread e serves weight rows e and 128 + e of the item and two blocks of token e / 2: it brings the token's block scales into
    // shared memory (its own cp.async, TC_SC_AHEAD stages ahead), forms the fold's constants, and turns its rows' nibbles
    // into int8 in TMEM (byte i of a block's 16: element i in the low nibble, element i + 16 in the high one).
    else if (warp >= TC_EXP_W0) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        const int e = ptid - TC_EXP_W0 * 32, tok = e >> 1;
        // ---- the scale requests run ahead of the consumption ----
        int p_item = blockIdx.x, p_ks = 0, n_slot = 0;
        unsigned p_it = 0;
        const char * p_sc = nullptr, * p_w[2] = {nullptr, nullptr};
        TcItem N = tc_item(g, P, p_item);
        if (g.perm && tok < N.tcnt) n_slot = __ldg(g.perm + N.tstart + tok);
        auto p_switch = [&]() {                          // N, n_slot describe item p_item: point at its scales, look one item further
            const int arow = g.perm ? n_slot >> g.a_shift : N.tstart + tok;
            p_sc = tok < N.tcnt ? sc_plane + (size_t) arow * s_pitch + (e & 1) * 16 : nullptr;
            if constexpr (!WCOPY) {                      // the scales of this thread's two weight rows
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int row = EPI ? N.rt * TC_ROWS : tc_tile_row(P, N.rt, r), seg = EPI ? r : tc_seg(g, row);
                    const bool there = EPI ? row + e < g.N : r == 0 || tc_two<EPI>(g, P, N.rt);
                    p_w[r] = there ? (const char *) g.d[seg] + ((size_t) N.expert * g.exp_stride
                                     + (size_t) (row - (EPI || !seg ? 0 : g.seg_end[seg - 1]) + e) * g.bpr) * 2 : nullptr;
                }
            }
            if (p_item + (int) gridDim.x < P.n_items) N = tc_item(g, P, p_item + gridDim.x);
        };
        p_switch();
        auto fetch = [&]() {
            if (p_item < P.n_items) {
                if (p_sc) tc_cp16(&S.asc[p_it % TC_SC_RING][e], p_sc + p_ks * (TC_KB * 8));
                if constexpr (!WCOPY) {
                    if (!(p_ks & 1)) {
#pragma unroll
                        for (int r = 0; r < 2; ++r)
                            if (p_w[r]) {
                                char * const w = (char *) &S.wsc[(p_it >> 1) % (TC_WS_RING / 2)][r * TC_ROWS + e];
                                tc_cp8(w, p_w[r] + p_ks * (TC_KB * 2));
                                tc_cp8(w + 8, p_w[r] + p_ks * (TC_KB * 2) + 8);
                            }
                    }
                }
                if (p_ks == 1 && g.perm && tok < N.tcnt) n_slot = __ldg(g.perm + N.tstart + tok);
                ++p_it;
                if (++p_ks == P.nstage) { p_ks = 0; p_item += gridDim.x; if (p_item < P.n_items) p_switch(); }
            }
            tc_cp_commit();
        };
        for (int i = 0; i < TC_SC_AHEAD; ++i) fetch();
        unsigned it = 0, stg = 0, par = 0;
        bool ok = true;
        const unsigned ta = tmem + ((unsigned) ((warp & 3) * 32) << 16) + TC_COL_A;
        TcItem I = tc_item(g, P, blockIdx.x);
        for (int item = blockIdx.x; item < P.n_items && ok; item += gridDim.x) {
            const bool two = tc_two<EPI>(g, P, I.rt), tlive = tok < I.tcnt;
            if (item + (int) gridDim.x < P.n_items) I = tc_item(g, P, item + gridDim.x);
            for (int ks = 0; ks < P.nstage && ok; ++ks, ++it) {
                tc_cp_wait<TC_SC_AHEAD - 1>();                                          // this stage's scales are here
                if (!tc_wait<TC_HINT_PROD>(S, &S.full[stg], par, 15u)) { ok = false; break; }
                TcStage & T = S.st[stg];
                // the fold's constants
                if (tlive) {
                    const float4 a = S.asc[it % TC_SC_RING][e];
                    const float dd[2] = {a.x, a.z}, ss[2] = {a.y, a.w};
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        float d = dd[b], k = -ss[b];
                        if (FOLD) {
                            const float c = fmaf(d, TC_MAGIC_F, ss[b]);
                            k = __fmul_rn(fmaf(-TC_SEED, d, fmaf(d, TC_MAGIC_F, -c)), TC_DOWN49);
                            d = __fmul_rn(d, TC_UP100);
                        }
                        float * const q = reinterpret_cast<float *>(&S.dk[it % TC_SC_RING][2 * (e & 1) + b][tok >> 1]) + (tok & 1);
                        q[0] = d; q[2] = k;
                    }
                }
                if (!tc_wait<TC_HINT_PROD>(S, &S.aempty[it & 1u], ((it >> 1) & 1u) ^ 1u, 16u)) { ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if (r && !two) continue;
                    const unsigned char * rq = T.rawq + (r * TC_ROWS + e) * 64;
                    uint4 w[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const uint4 *>(rq + ((j ^ ((e >> 1) & 3)) << 4));
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        tc_st8(ta + (it & 1u) * 64 + r * 32 + j * 8,
                               make_uint4(w[j].x & 0x0F0F0F0Fu, w[j].y & 0x0F0F0F0Fu, w[j].z & 0x0F0F0F0Fu, w[j].w & 0x0F0F0F0Fu),
                               make_uint4((w[j].x >> 4) & 0x0F0F0F0Fu, (w[j].y >> 4) & 0x0F0F0F0Fu, (w[j].z >> 4) & 0x0F0F0F0Fu, (w[j].w >> 4) & 0x0F0F0F0Fu));
                }
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                tc_mbar_arrive_if(&S.afull[it & 1u], lane == 0);
                fetch();
                if (++stg == TC_NS) { stg = 0; par ^= 1u; }
            }
        }
        tc_cp_wait<0>();
    }
    // ============================ epilogue (eight warps) ==========================
    else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int quad = warp & 3, half = warp >> 2;            // TMEM lane quadrant; which half of the item's columns
        const unsigned tbase = tmem + ((unsigned) (quad * 32) << 16);
        __syncwarp();
        if (lane == 0)                                          // all block-sum buffers start out free for the MMA issuer
            for (int i = 0; i < TC_DBUF; ++i) tc_mbar_arrive(&S.tempty[TcSums<EPI>::FREE ? half : 0][i]);
        TcEpi X;
        X.it = 0;
        bool ok = true;
        TcItem I = tc_item(g, P, blockIdx.x);
        for (int item = blockIdx.x; item < P.n_items && ok; item += gridDim.x) {
            const TcItem C = I;
            if (item + (int) gridDim.x < P.n_items) I = tc_item(g, P, item + gridDim.x);
            if constexpr (EPI == 1) ok = tc_epilogue_cols<EPI, FOLD, 2>(S, X, g, P, C, out_rows, tbase, half, quad, lane);
            else if (tc_two<EPI>(g, P, C.rt)) ok = tc_epilogue_cols<EPI, FOLD, 2>(S, X, g, P, C, out_rows, tbase, half, quad, lane);
            else ok = tc_epilogue_cols<EPI, FOLD, 1>(S, X, g, P, C, out_rows, tbase, half, quad, lane);
        }
        tc_wait_ld();                                           // nothing of this thread is left in flight
    }

    // ---- teardown: everyone meets, then the allocating warp frees TMEM ------------
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512) : "memory");
    }
}

// ---------------------------------------------------------------------------
static int g_tc_ready = 0;
static tc_encode_fn g_tc_encode = nullptr;
tc_encode_fn lkb_tensor_map_encoder() { return g_tc_encode; }
int lkb_pf_attn_init();                    // lkb_pfattn.cu
int lkb_pf_attn_take_status();
int lkb_gemm_few_init();                   // lkb_gemm_few.cu
int lkb_gemm_few_take_status();
int lkb_prefill_take_status();             // lkb_prefill.cu: the tiled router

typedef void (*TcKernel)(lkb_pf_gemm, int, int, const char *, int, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap,
                         CUtensorMap, float * const *, TcDense);
static TcKernel const TC_FORMS[8] = {               // 4 epi + 2 fold + weight scales by tensor copy
    k_pf_gemm_tc<0, 0, 0>, k_pf_gemm_tc<0, 0, 1>, k_pf_gemm_tc<0, 1, 0>, k_pf_gemm_tc<0, 1, 1>,
    k_pf_gemm_tc<1, 0, 0>, k_pf_gemm_tc<1, 0, 1>, k_pf_gemm_tc<1, 1, 0>, k_pf_gemm_tc<1, 1, 1>};

int lkb_gemm_tc_init() {
    cudaError_t e = cudaSuccess;
    const int sm = (int) sizeof(TcSmem) + 1024;
    for (int f = 0; f < 8; ++f)
        if (e == cudaSuccess) e = cudaFuncSetAttribute(TC_FORMS[f], cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return -(int) e;
    // the tensor-map encoder is a driver entry point; it is looked up through the runtime so that the
    // library carries no link-time dependency on the driver
    void * fn = nullptr;
    cudaDriverEntryPointQueryResult qr;
    e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr);
    if (e != cudaSuccess) return -(int) e;
    if (!fn || qr != cudaDriverEntryPointSuccess) return LKB_ERR_UNSUPPORTED;
    g_tc_encode = (tc_encode_fn) fn;
    g_tc_ready = 1;
    const int few = lkb_gemm_few_init();
    return few != LKB_OK ? few : lkb_pf_attn_init();
}

// A byte matrix [rows][row_bytes], rows `pitch` bytes apart, as a 2-D tensor; box = box_bytes x box_rows.  Rows past `rows`
// read as zero.
int lkb_tc_make_map(CUtensorMap * m, const void * base, unsigned row_bytes, unsigned long long pitch, unsigned long long rows,
                       unsigned box_bytes, unsigned box_rows, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2) {
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {pitch};
    const cuuint32_t box[2] = {box_bytes, box_rows};
    const cuuint32_t es[2] = {1, 1};
    const CUresult r = g_tc_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, es,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, sw, l2,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? LKB_OK : LKB_ERR_UNSUPPORTED;
}
#define TC_ANY_ROWS (1ull << 30)            // row bound of a plane whose extent the caller does not state: it only clips

// Items of a dense problem: the token width and height that need the least time, waves of items times an item's.  A block of an item
// takes about 330 + 6 N cycles with one tile and 350 + 6.2 N with two (measured at N = 16 .. 64 and 64 blocks a row; what an item takes besides its blocks is
// left out, and weighs more where a row has fewer), so a problem of less than a wave is
// cut into narrow items (each reads the weights again, from L2), and one that would leave most of its last wave empty is cut
// so that the waves fill.  us with 64-token items and with these, caches flushed: in_proj (6144 rows) at 37 / 130 / 509 tokens
// 22.5 / 26.6 / 51.2 -> 19.5 / 24.6 / 45.0, out_proj (2048 rows) 24.6 / 26.6 / 28.7 -> 18.4 / 20.5 / 26.6; at 4096 tokens the
// choice is 64 x 256 as before.  SwiGLU form: an item is 128 rows of either weight, two tiles always.
static TcDense tc_dense_form(int ntok, int N, int sms, int epi, long long * cost = nullptr) {
    TcDense best = {TC_TOK, 1};
    long long least = 0;
    for (int wide = 1; wide >= (epi ? 1 : 0); --wide)
        for (int tw = TC_TOK; tw >= 16; tw -= 16) {
            const int rows = wide && !epi ? 2 * TC_ROWS : TC_ROWS;
            const long long items = (long long) ((ntok + tw - 1) / tw) * ((N + rows - 1) / rows);
            const long long t = (items + sms - 1) / sms * (wide ? 3500 + 62 * tw : 3300 + 60 * tw);
            if (!least || t < least) { least = t; best = {tw, wide}; }
        }
    if (cost) *cost = least;
    return best;
}
// What a block of all its items' waves takes, in ns: the above at 1.87 GHz.
int lkb_gemm_tc_dense_ns(int ntok, int N, int sms, int epi) {
    long long c = 0;
    tc_dense_form(ntok, N, sms, epi, &c);
    return (int) (c * 100 / 1870 < (1 << 30) ? c * 100 / 1870 : 1 << 30);
}

// Test hook (not in the public header): the items a plain dense problem is cut into, tokens * 1000 + weight rows.
extern "C" __attribute__((visibility("default"))) int lkb_debug_gemm_dense_item(int ntok, int N) {
    const TcDense d = tc_dense_form(ntok, N, lkb_context().sm_count, 0);
    return d.tw * 1000 + (d.wide ? 2 : 1) * TC_ROWS;
}

// Shapes the tensor-core form covers; otherwise LKB_ERR_UNSUPPORTED (the caller falls back to the CUDA-core form): the
// planes must have the alignment the copies ask for.
int lkb_gemm_tc_launch(const lkb_pf_gemm * g, int epi, int fold, int max_tiles, cudaStream_t st, float * const * out_rows, int a_pitch) {
    if (a_pitch && (!g->perm || a_pitch % 16 || a_pitch < g->bpr * 40)) return LKB_ERR_SHAPE;     // packed rows: grouped form, 16-byte aligned
    if (out_rows && (epi || !g->perm || g->add)) return LKB_ERR_SHAPE;          // row targets: the plain grouped form, no residual add
    if (!g_tc_ready) return LKB_ERR_NOT_INIT;
    if (g->bpr % 8) return LKB_ERR_UNSUPPORTED;                                 // the scale copies take two stages of a row at a time
    if (epi ? (g->N % 64) : (g->N % TC_ROWS)) return LKB_ERR_UNSUPPORTED;
    if (((size_t) g->aqs & 15) || (!a_pitch && ((size_t) g->asc & 15))) return LKB_ERR_UNSUPPORTED;
    if (g->exp_stride % g->bpr) return LKB_ERR_UNSUPPORTED;
    const int nseg = epi ? 2 : (g->seg_end[0] >= g->N ? 1 : g->seg_end[1] >= g->N ? 2 : 3);
    const unsigned qrow = (unsigned) g->bpr * 32u, box_rows = epi ? 64u : TC_ROWS;
    CUtensorMap ma, mw[3], md[3];
    // dense: 16-token boxes of consecutive rows; grouped: rows gathered through perm, four per copy.  Packed rows
    // (a_pitch, as the expert-parallel dispatch delivers them): quants first, then the (d8, 8sum) pairs.
    int r = g->perm ? lkb_tc_make_map(&ma, g->aqs, qrow, a_pitch ? (unsigned) a_pitch : qrow, TC_ANY_ROWS, 128u, 1u, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B)
                    : lkb_tc_make_map(&ma, g->aqs, qrow, qrow, (unsigned long long) g->ntok, 128u, 16u, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    if (r != LKB_OK) return r;
    const char * sc_plane = a_pitch ? (const char *) g->aqs + qrow : (const char *) g->asc;
    const int s_pitch = a_pitch ? a_pitch : g->bpr * 8;
    int wcopy = 1;
    for (int s = 0; s < nseg; ++s) if ((size_t) g->d[s] & 15) wcopy = 0;
    for (int s = 0; s < 3; ++s) {
        const int src = s < nseg ? s : 0;
        if (((size_t) g->qs[src] & 15) || ((size_t) g->d[src] & 7)) return LKB_ERR_UNSUPPORTED;
        r = lkb_tc_make_map(&mw[s], g->qs[src], (unsigned) g->bpr * 16u, (unsigned) g->bpr * 16u, TC_ANY_ROWS, 64u, box_rows, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (r != LKB_OK) return r;
        md[s] = mw[s];                                                          // (not by tensor copy: never used)
        if (wcopy) r = lkb_tc_make_map(&md[s], g->d[src], (unsigned) g->bpr * 2u, (unsigned) g->bpr * 2u, TC_ANY_ROWS, 16u, box_rows, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (r != LKB_OK) return r;
    }
    const int rpe = (int) (g->exp_stride / g->bpr);
    const dim3 grid(lkb_context().sm_count), block(TC_THREADS);
    const size_t sm = sizeof(TcSmem) + 1024;
    LKB_PF_LAUNCH(TC_FORMS[(epi ? 4 : 0) + (fold ? 2 : 0) + wcopy], grid, block, sm, st, *g, max_tiles, rpe, sc_plane, s_pitch, ma, mw[0], mw[1], mw[2],
                  md[0], md[1], md[2], out_rows, g->perm ? TcDense{TC_TOK, 1} : tc_dense_form(g->ntok, g->N, lkb_context().sm_count, epi));
    return lkb_check_launch();
}

extern "C" {
int lkb_pf_gemm_workspace_bytes(int max_tiles, int k_max, size_t * bytes_out) {
    if (!bytes_out) return LKB_ERR_NULL;
    if (max_tiles <= 0 || k_max <= 0 || k_max % 32) return LKB_ERR_SHAPE;
    *bytes_out = (size_t) max_tiles * LKB_MOE_BN * ((size_t) k_max + (size_t) k_max / 4);      // quants + (d8, 8sum) per 32
    return LKB_OK;
}
// The GEMM gathers its activation rows itself and needs no workspace; a registered one is accepted and left alone.
int lkb_pf_gemm_set_workspace(void * ptr, size_t bytes) {
    (void) bytes;
    return ((size_t) ptr & 255) ? LKB_ERR_SHAPE : LKB_OK;
}
int lkb_pf_gemm_status(void) {
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    const int a = tc_take_status(), b = lkb_pf_attn_take_status(), c = lkb_gemm_few_take_status(), d = lkb_prefill_take_status();
    return a ? a : b ? b : c ? c : d;
}
}
