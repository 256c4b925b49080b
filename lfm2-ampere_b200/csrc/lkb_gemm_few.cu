// lkb_gemm_few.cu - the Q4_0 x Q8_1 GEMM (dense and grouped) for a few tokens a tile: weights streamed once, integer dots by warp-level MMAs.
//
// The same sums as lkb_gemm_tc.cu, in the same order and rounding, so the same bits: per (row, token) one fp32 chain over the
// blocks, acc = fma(d4, fma(d8, 12582912 + S, -c), acc) (FOLD = 1) or fma(d4, fma(d8, float(S), -8sum), acc) (FOLD = 0).
//
// The tensor-core form hands every block of 32 from the expansion warps to an MMA, through TMEM, to the epilogue warps and back: 330 to
// 450 cycles of a 256-row block whatever its tokens, where HBM brings the block in 190.  Here nothing is handed over.  A warp keeps 16 rows of
// both 128-row tiles: one ldmatrix brings the nibbles of a block as the fragments of two m16n8k32 u8 x s8 MMAs (byte 4q + i holds elements 4q + i
// and 16 + 4q + i, which is the A fragment after a mask and a shift), the sums start from the bit pattern of 12582912.0f and are folded
// from the registers they arrive in.  Measured without copies, ns a 256-row block at 8 / 16 / 32 / 64 tokens: 69 / 99 / 182 / 313 (35 for
// the rows, 4.3 a token, half of it MMA and half fold; they do not overlap), the other form 230 / 230 / 290 / 350.
//   * One CTA an SM: one item takes a whole SM for some 7 us, and few SMs idle behind the last wave.  Eight dot warps, three that
//     issue copies (one costs its thread 80 to 100 cycles: a single warp for all was the bound, one for all activations cost 5 % at 256 tokens), and
//     one that turns a stage's (d8, 8sum) into the constants of token pairs (in the dot warps, eight times over, that doubled a block's time).
//   * Stages of eight blocks: 128 bytes of a weight row, half the copies and waits of four (m = 128: gate|up 78 -> 66 us).
//   * 16 or 32 tokens an item; the part of a stage that activations leave goes into stages: five or four, 110 to 180 KB in flight.
// Measured in one run, 64 experts, balanced routing, caches flushed before every call, us at 9 / 20 / 37 / 64 / 128 / 256 / 384 / 480 tokens:
//   gate|up  dp4a form, three CTAs an SM (before, to 47 tokens)  32 / 48 / 63;  tensor-core form  80 / 81 / 92 / 96 / 114 from 64 on
//            this form                                           34 / 44 / 55 / 58 / 64 / 75 / 95 / 115
//   down     before  21 / 28 / 40;  51 / 53 / 57 / 58 / 62       this form  21 / 28 / 34 / 35 / 37 / 43 / 49 / 59
// What bounds it: to some 100 tokens whole waves of items (768 on 148 SMs: 5.2) of 4.5 TB/s each and 5 to 7 us of launch, fill and drain;
// then the MMAs and the fold.
// No copy in this file is a multicast one; every tensor map covers memory of the GPU the kernel runs on.
// Every wait is bounded; on expiry a status word is set, the roles leave, the producers after their copies have landed.
#include "lkb_tc.cuh"

#define FW_ROWS   128                // rows of a tile; an item has two (SwiGLU form: gate and up rows)
#define FW_KB     8                  // blocks per stage
#define FW_WARPS  8                  // dot warps: 16 rows of each tile
#define FW_W_WARP 8                  // fetches weights and their scales, and the activations' scales
#define FW_A_WARP 9                  // this one and the next fetch activations, four blocks of a stage each
#define FW_C_WARP 11                 // forms the token constants of a stage
#define FW_THREADS 384
#define FW_UNITS  2048               // parts of plan tiles that are listed

// The two sizes, by the most tokens of an item, and the stages that fit beside each.
template <int TOK> struct FwForm { static constexpr int NS = TOK == 16 ? 5 : 4; };

template <int TOK> struct FwStage {
    alignas(1024) unsigned char q[2 * FW_ROWS * 128];       // nibbles: row r at r*128, 16-byte chunk c at c ^ (r & 7)
    alignas(1024) signed char act[2][TOK * 128];            // activations of four blocks: token t at t*128, 16-byte chunk c at c ^ (t & 7)
    alignas(128) uint4 ws[2 * FW_ROWS];                     // eight fp16 scales per weight row
    alignas(128) float2 asc[TOK][FW_KB];                    // (d8, 8sum)
    alignas(128) float4 dc[FW_KB][TOK / 2];                 // per token pair {d8, d8', -c, -c'} (FOLD) or {.., -8sum, -8sum'}
};
template <int TOK> struct FwSmem {
    static constexpr int NS = FwForm<TOK>::NS;
    FwStage<TOK> st[NS];
    alignas(16) float2 swap[TOK / 8][FW_WARPS * 32];        // SwiGLU form: values that the two warps of an output block exchange
    int   slot[NS + 1][TOK];                                // an item's slots and row scales; a ring by item, of more than the items in NS stages
    float scl[NS + 1][TOK];
    unsigned short unit[FW_UNITS];                          // grouped: plan tile * (64 / TOK) + part of it
    alignas(8) unsigned long long full[NS], ready[NS], empty[NS], xfull[FW_WARPS / 2], xempty[FW_WARPS / 2];
    int abort, n_units, listed;
};

struct FwItem { int expert, tstart, cnt, rt, r0, rows; };   // cnt <= 0: nothing to do; rows r0 .. r0 + rows - 1 of both tiles
// The blocks' work: items, of which those from `whole` on -- a last wave that would leave half of the blocks or more without one -- are cut
// into 1 << cut parts of fewer rows, one a block, whose first warps have rows (an item's time is its weights' way into one SM).  us, whole -> cut in a run of its own, caches
// flushed: down at 2 / 20 tokens 15.3 -> 13.3, 29.7 -> 27.7; out_proj (2048 rows) at 2 to 64 tokens 13.3 -> 11.3, in_proj at 2 13.3 -> 11.3; a layer of 2 / 9 / 20 / 37 /
// 64 tokens 59.4 / 84.4 / 100.6 / 114.3 / 122.3 -> 55.6 / 79.2 / 96.3 / 111.3 / 119.8.  A choice of the width that counts a part as 0.6 of an item
// changed nothing (-1 % at 70 tokens, +0.5 % at 200).
struct FwWork { int whole, cut, n; };
__device__ __forceinline__ FwWork fw_work(int n_items, int cut, int blocks) {
    FwWork W;
    const int rem = n_items % blocks;
    W.cut = rem << cut <= blocks ? cut : 0;
    W.whole = n_items - rem;
    W.n = W.whole + (rem << W.cut);
    return W;
}
// Items by token unit (dense: tw tokens; grouped: a plan tile or a part of one) and row tile, row tiles fastest.
template <int TOK>
__device__ __forceinline__ FwItem fw_item(const FwSmem<TOK> & S, const lkb_pf_gemm & g, int tw, int n_rt, const FwWork & W, int n) {
    FwItem I;
    const int over = max(n - W.whole, 0), cut = n < W.whole ? 0 : W.cut, item = min(n, W.whole) + (over >> W.cut), u = item / n_rt;
    I.rt = item - u * n_rt;
    I.rows = FW_ROWS >> cut;
    I.r0 = (over & ((1 << cut) - 1)) * I.rows;
    if (g.perm) {
        const int t = S.listed ? S.unit[u] : u, t0 = (t % (64 / TOK)) * TOK;
        const int4 tl = __ldg(reinterpret_cast<const int4 *>(g.tiles) + t / (64 / TOK));
        I.expert = tl.x; I.tstart = tl.y + t0; I.cnt = min(TOK, tl.z - t0);
    } else {
        I.expert = 0; I.tstart = u * tw; I.cnt = min(tw, g.ntok - I.tstart);
    }
    return I;
}

// 8 x 16 bytes per matrix: lane l gives the address of row l & 7 of matrix l >> 3, and gets word l & 3 of row l >> 2 of each.
__device__ __forceinline__ void fw_ldm4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void fw_ldm2(unsigned (&r)[2], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}
// 16 rows x 8 tokens x 32: every sum starts from the bit pattern of 12582912.0f
__device__ __forceinline__ void fw_mma(unsigned (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(0x4B400000));
}

// All stages of one item for 8 NT tokens.  acc[r][n][k]: rows 128 r + 16 warp + 8 k + lane / 4, tokens 8 n + 2 (lane % 4) and the next.
// Returns false when a wait gave up.
template <int FOLD, int TOK, int NT>
__device__ __forceinline__ bool fw_dots(FwSmem<TOK> & S, unsigned & it, int nstage, int warp, int lane, unsigned long long (&acc)[2][NT][2]) {
    const int g = lane >> 2, q = lane & 3;
    const unsigned long long nmag = tc_pack(-12582912.0f, -12582912.0f);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[r][n][0] = acc[r][n][1] = 0ull;
    // ldmatrix rows of this lane: weight rows 16 warp + lane % 16 of tile lane / 16; tokens 8 (lane / 16) + lane % 8, low or high half of a block
    const int row = (lane >> 4) * FW_ROWS + 16 * warp + (lane & 15), tok = (lane >> 4) * 8 + (lane & 7), hi = (lane >> 3) & 1;
    const unsigned wrow = row * 128, wx = row & 7, arow = tok * 128, ax = tok & 7;
#pragma unroll 1
    for (int ks = 0; ks < nstage; ++ks, ++it) {
        const unsigned stg = it % S.NS, par = (it / S.NS) & 1u;
        // the copies' bytes are acquired here, the constants with ready
        if (!tc_wait(S, &S.ready[stg], par, 33u) || !tc_wait(S, &S.full[stg], par, 33u)) return false;
        const FwStage<TOK> & T = S.st[stg];
        const unsigned qb = tc_smem_u32(T.q) + wrow, ab = tc_smem_u32(T.act) + arow;
        uint4 we[2][2];                                                  // the stage's eight scales of this thread's four rows
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int k = 0; k < 2; ++k) we[r][k] = T.ws[r * FW_ROWS + 16 * warp + 8 * k + g];
#pragma unroll
        for (int b = 0; b < FW_KB; ++b) {
            unsigned bf[NT][2], w[4];
            const unsigned ab_b = ab + (b >> 2) * (TOK * 128);
            fw_ldm4(w, qb + ((b ^ wx) << 4));                            // rows g, g + 8 of the first tile and of the second
#pragma unroll
            for (int n = 0; n + 1 < NT; n += 2) {
                unsigned x[4];
                fw_ldm4(x, ab_b + n * 1024 + (((2 * (b & 3) + hi) ^ ax) << 4));
                bf[n][0] = x[0]; bf[n][1] = x[1]; bf[n + 1][0] = x[2]; bf[n + 1][1] = x[3];
            }
            if (NT & 1) fw_ldm2(bf[NT - 1], ab_b - (lane >> 4) * 1024 + (NT - 1) * 1024 + (((2 * (b & 3) + hi) ^ ax) << 4));
            unsigned a[2][4];
            unsigned long long e[2][2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                a[r][0] = w[2 * r] & 0x0F0F0F0Fu; a[r][1] = w[2 * r + 1] & 0x0F0F0F0Fu;
                a[r][2] = (w[2 * r] >> 4) & 0x0F0F0F0Fu; a[r][3] = (w[2 * r + 1] >> 4) & 0x0F0F0F0Fu;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const unsigned x = (b >> 1) == 0 ? we[r][k].x : (b >> 1) == 1 ? we[r][k].y : (b >> 1) == 2 ? we[r][k].z : we[r][k].w;
                    const float f = __half2float(__ushort_as_half((unsigned short) (x >> (16 * (b & 1)))));
                    e[r][k] = tc_pack(f, f);
                }
            }
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const float4 dc = T.dc[b][4 * n + q];
                const unsigned long long d = tc_pack(dc.x, dc.y), c = tc_pack(dc.z, dc.w);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    unsigned s[4];
                    fw_mma(s, a[r], bf[n]);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        unsigned long long f = tc_pack_u(s[2 * k], s[2 * k + 1]);              // 12582912 + the block sums, as floats
                        if (!FOLD) f = tc_fadd2(f, nmag);
                        acc[r][n][k] = tc_ffma2(e[r][k], tc_ffma2(d, f, c), acc[r][n][k]);
                    }
                }
            }
        }
        __syncwarp();
        tc_mbar_arrive_if(&S.empty[stg], lane == 0);
    }
    return true;
}

// out (+)= scale * acc: a store of a warp is 8 rows (a sector) of four tokens.
template <int NT>
__device__ __forceinline__ void fw_store_plain(const int * slots, const float * scls, const lkb_pf_gemm & g, const FwItem & I, int warp, int lane, const unsigned long long (&acc)[2][NT][2]) {
    const int o0 = I.rt * (2 * FW_ROWS) + I.r0 + 16 * warp + (lane >> 2);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int t = 8 * n + 2 * (lane & 3) + p;
            if (t >= I.cnt) continue;
            const float scl = scls[t];
            float * const out = g.out + (size_t) slots[t] * g.out_ld + o0;
            float prev[2][2] = {};
            if (g.add) {
#pragma unroll
                for (int i = 0; i < 4; ++i) prev[i >> 1][i & 1] = out[(i >> 1) * FW_ROWS + (i & 1) * 8];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float x[2];
                tc_unpack(acc[i >> 1][n][i & 1], x[0], x[1]);
                // the residual add is one fused multiply-add (ref: src/prefill.cu:484-486)
                out[(i >> 1) * FW_ROWS + (i & 1) * 8] = g.add ? fmaf(x[p], scl, prev[i >> 1][i & 1]) : __fmul_rn(x[p], scl);
            }
        }
}

// SwiGLU + Q8_1.  The 32 rows of an output block are two warps': the even one takes the first token of every pair and the odd one the
// second, and hands over its own two rows of the other.  Lane: rows lane / 4 + 0, 8, 16, 24 of the block.
template <int FOLD, int TOK, int NT>
__device__ __forceinline__ bool fw_store_swiglu(FwSmem<TOK> & S, const int * slots, const float * scls, unsigned xpar, const lkb_pf_gemm & g, const FwItem & I, int warp, int lane,
                                                const unsigned long long (&acc)[2][NT][2]) {
    const int row0 = I.rt * FW_ROWS + I.r0 + (warp >> 1) * 32, gr = lane >> 2, mine = warp & 1, q = lane & 3;
    float v[NT][2];                                                      // my token of pair n, my two rows
    if (!tc_wait(S, &S.xempty[warp >> 1], xpar ^ 1u, 34u)) return false; // what was handed over last has been read
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        float x[2][2];                                                   // [row][token]
        const float s0 = scls[8 * n + 2 * q], s1 = scls[8 * n + 2 * q + 1];
        const unsigned long long scl = tc_pack(s0, s1);
        const bool live0 = 8 * n + 2 * q < I.cnt, live1 = 8 * n + 2 * q + 1 < I.cnt;       // sums of no token are whatever the stages held
        bool sure = true;
#pragma unroll
        for (int k = 0; k < 2; ++k) tc_unpack(tc_fmul2(tc_silu2(tc_fmul2(acc[0][n][k], scl), sure, live0, live1), tc_fmul2(acc[1][n][k], scl)), x[k][0], x[k][1]);
        if (!sure) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                float gx[2], ux[2];
                tc_unpack(acc[0][n][k], gx[0], gx[1]);
                tc_unpack(acc[1][n][k], ux[0], ux[1]);
                x[k][0] = __fmul_rn(lkb_silu(__fmul_rn(gx[0], s0)), __fmul_rn(ux[0], s0));
                x[k][1] = __fmul_rn(lkb_silu(__fmul_rn(gx[1], s1)), __fmul_rn(ux[1], s1));
            }
        }
        v[n][0] = mine ? x[0][1] : x[0][0]; v[n][1] = mine ? x[1][1] : x[1][0];
        S.swap[n][(warp ^ 1) * 32 + lane] = mine ? make_float2(x[0][0], x[1][0]) : make_float2(x[0][1], x[1][1]);
    }
    __syncwarp();
    tc_mbar_arrive_if(&S.xfull[warp >> 1], lane == 0);
    if (!tc_wait(S, &S.xfull[warp >> 1], xpar, 35u)) return false;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        if (8 * n >= I.cnt) continue;                                    // (the whole warp)
        const float2 o2 = S.swap[n][warp * 32 + lane];
        const float u[4] = {mine ? o2.x : v[n][0], mine ? o2.y : v[n][1], mine ? v[n][0] : o2.x, mine ? v[n][1] : o2.y};
        const int t = 8 * n + 2 * q + mine;
        const bool live = t < I.cnt;
        const int slot = slots[t];
        unsigned am = max(max(__float_as_uint(fabsf(u[0])), __float_as_uint(fabsf(u[1]))), max(__float_as_uint(fabsf(u[2])), __float_as_uint(fabsf(u[3]))));
        // Shipped arithmetic: the reference's fused epilogue adds rows (g, g+8) + (g+16, g+24), then pairs over g ^ 1, 2, 4
        // (src/prefill.cu:424-448); exact mode: the quantiser's butterfly, rows 16, 8, 4, 2, 1 apart.
        float sum = FOLD ? __fadd_rn(__fadd_rn(u[0], u[1]), __fadd_rn(u[2], u[3])) : __fadd_rn(__fadd_rn(u[0], u[2]), __fadd_rn(u[1], u[3]));
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            const int x = FOLD ? 4 << o : 16 >> o;                       // lanes of rows 1, 2, 4 or 4, 2, 1 apart
            am = max(am, __shfl_xor_sync(LKB_FULL, am, x));
            sum = __fadd_rn(sum, __shfl_xor_sync(LKB_FULL, sum, x));
        }
        const float d = __fdiv_rn(__uint_as_float(am), 127.0f);
        const __half2 ds = __floats2half2_rn(d, sum);
        // q = roundf(u / d) by the reciprocal, with the division for elements near a tie (see lkb_quad_quant_ds)
        float rd, qf[4];
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rd) : "f"(d));
        bool sure = true;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            qf[j] = fmaf(u[j], rd, 12582912.0f);
            const float diff = fmaf(u[j], rd, -__fadd_rn(qf[j], -12582912.0f));
            sure = sure && fabsf(diff) < 0.4999f;
        }
        if (!sure) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float r = roundf(__fdiv_rn(u[j], d));
                qf[j] = (am != 0u && r == r) ? __fadd_rn(r, 12582912.0f) : 12582912.0f;       // (int) NaN is 0; an all-zero block is 0
            }
        }
        unsigned pk = __byte_perm(__byte_perm(__float_as_uint(qf[0]), __float_as_uint(qf[1]), 0x0040),       // rows lane / 4 + 8 j in byte j
                                  __byte_perm(__float_as_uint(qf[2]), __float_as_uint(qf[3]), 0x0040), 0x5410);
        // 4 x 4 bytes across the lanes of rows 4i .. 4i+3: byte j of lane i goes to byte i of lane j
        unsigned o = __shfl_xor_sync(LKB_FULL, pk, 8);                   // rows two apart: exchange pairs of bytes
        pk = (gr & 2) ? __byte_perm(pk, o, 0x3276) : __byte_perm(pk, o, 0x5410);
        o = __shfl_xor_sync(LKB_FULL, pk, 4);                            // rows one apart: exchange bytes
        pk = (gr & 1) ? __byte_perm(pk, o, 0x3715) : __byte_perm(pk, o, 0x6240);
        if (live) {
            reinterpret_cast<unsigned *>(g.oqs + (size_t) slot * (g.okb * 32) + row0)[2 * (gr & 3) + (gr >> 2)] = pk;
            if (gr == 0) reinterpret_cast<float2 *>(g.osc)[(size_t) slot * g.okb + row0 / 32] = make_float2(__low2float(ds), __fmul_rn(8.0f, __high2float(ds)));
        }
    }
    __syncwarp();
    tc_mbar_arrive_if(&S.xempty[warp >> 1], lane == 0);
    return true;
}

template <int EPI, int FOLD, int TOK, int NT>
__device__ __forceinline__ bool fw_do_item(FwSmem<TOK> & S, unsigned & it, unsigned n_item, const lkb_pf_gemm & g, const FwItem & I, int nstage, int warp, int lane) {
    unsigned long long acc[2][NT][2];
    if (!fw_dots<FOLD, TOK, NT>(S, it, nstage, warp, lane, acc)) return false;
    const int * const slots = S.slot[n_item % (S.NS + 1)];
    const float * const scls = S.scl[n_item % (S.NS + 1)];
    if constexpr (EPI) return fw_store_swiglu<FOLD, TOK, NT>(S, slots, scls, n_item & 1u, g, I, warp, lane, acc);
    fw_store_plain<NT>(slots, scls, g, I, warp, lane, acc);
    return true;
}

// Nibbles and scales of the three row segments, in boxes of 128 rows and of a part's.
struct FwMaps { CUtensorMap w[2][3], d[2][3]; };

template <int EPI, int FOLD, int TOK>
__global__ void __launch_bounds__(FW_THREADS, 1) k_pf_gemm_few(const lkb_pf_gemm g, const int max_tiles, const int rpe, const int tw, const int cut,
        const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_s,
        const __grid_constant__ FwMaps maps) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    extern __shared__ unsigned char fw_smem_raw[];
    FwSmem<TOK> & S = *reinterpret_cast<FwSmem<TOK> *>(fw_smem_raw + ((1024u - (tc_smem_u32(fw_smem_raw) & 1023u)) & 1023u));
    const int tid = threadIdx.x, warp = __shfl_sync(LKB_FULL, tid >> 5, 0), lane = tid & 31;
    const int n_rt = EPI ? g.N / FW_ROWS : g.N / (2 * FW_ROWS), nstage = g.bpr / FW_KB;
    if (tid == 0) {
        S.abort = 0;
        for (int i = 0; i < S.NS; ++i) { tc_mbar_init(&S.full[i], 3); tc_mbar_init(&S.ready[i], 1); tc_mbar_init(&S.empty[i], FW_WARPS); }
        for (int i = 0; i < FW_WARPS / 2; ++i) { tc_mbar_init(&S.xfull[i], 2); tc_mbar_init(&S.xempty[i], 2); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (g.perm && warp == 1) {                                           // the tiles' parts, in order
        const int n_mt = min(*g.ntiles, max_tiles);
        int n = 0;
        for (int t0 = 0; t0 < n_mt; t0 += 32) {
            const int t = t0 + lane, parts = t < n_mt ? (__ldg(reinterpret_cast<const int4 *>(g.tiles) + t).z + TOK - 1) / TOK : 0;
            int at = parts;                                              // inclusive sum over the lanes
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(LKB_FULL, at, o);
                if (lane >= o) at += x;
            }
            for (int p = 0; p < parts; ++p)
                if (n + at - parts + p < FW_UNITS) S.unit[n + at - parts + p] = (unsigned short) (t * (64 / TOK) + p);
            n += __shfl_sync(LKB_FULL, at, 31);
        }
        if (lane == 0) {                                                 // more than the list holds: every part of every tile, empty ones too
            S.listed = n <= FW_UNITS;
            S.n_units = n <= FW_UNITS ? n : n_mt * (64 / TOK);
        }
    }
    __syncthreads();
    const FwWork W = fw_work((g.perm ? S.n_units : (g.ntok + tw - 1) / tw) * n_rt, cut, gridDim.x);
    unsigned it = 0;
    if (warp >= FW_W_WARP && warp < FW_C_WARP) {
        // ============================ producers (three warps) ========================
        bool ok = true;
        for (int item = blockIdx.x; item < W.n && ok; item += gridDim.x) {
            const FwItem I = fw_item<TOK>(S, g, tw, n_rt, W, item);
            if (I.cnt <= 0) continue;
            int crd[4] = {0, 0, 0, 0};                                   // lane l: tokens 4l .. 4l+3 (a dead one repeats the last)
            const int n_g = (I.cnt + 3) >> 2;
            const CUtensorMap * mw[2], * md[2];
            int wrow[2];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int t = I.tstart + min(4 * (lane & (TOK / 4 - 1)) + q, I.cnt - 1);
                crd[q] = g.perm ? __ldg(g.perm + t) >> g.a_shift : t;
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int row = EPI ? I.rt * FW_ROWS : (2 * I.rt + r) * FW_ROWS;
                const int seg = EPI ? r : (row < g.seg_end[0]) ? 0 : (row < g.seg_end[1]) ? 1 : 2;
                mw[r] = &maps.w[I.rows < FW_ROWS][seg];
                md[r] = &maps.d[I.rows < FW_ROWS][seg];
                wrow[r] = I.expert * rpe + I.r0 + row - (EPI || !seg ? 0 : g.seg_end[seg - 1]);
            }
            for (int ks = 0; ks < nstage; ++ks, ++it) {
                const unsigned stg = it % S.NS;
                if (!tc_wait<TC_HINT_PROD>(S, &S.empty[stg], ((it / S.NS) & 1u) ^ 1u, 11u)) { ok = false; break; }
                FwStage<TOK> & T = S.st[stg];
                if (warp == FW_W_WARP) {
                    if (lane == 0) {
                        tc_mbar_arrive_tx(&S.full[stg], 2u * (unsigned) I.rows * (128u + 16u) + (unsigned) n_g * (4u * 64u));
#pragma unroll
                        for (int r = 0; r < 2; ++r) tc_tma_tile(T.q + r * (FW_ROWS * 128), mw[r], ks * (FW_KB * 16), wrow[r], &S.full[stg]);
#pragma unroll
                        for (int r = 0; r < 2; ++r) tc_tma_tile(&T.ws[r * FW_ROWS], md[r], ks * (FW_KB * 2), wrow[r], &S.full[stg]);
                    }
                    __syncwarp();
                    if (lane < n_g) tc_tma_gather4(&T.asc[4 * lane][0], &map_s, ks * (FW_KB * 8), crd[0], crd[1], crd[2], crd[3], &S.full[stg]);
                } else {
                    const int h = warp - FW_A_WARP;
                    if (lane == 0) tc_mbar_arrive_tx(&S.full[stg], (unsigned) n_g * (4u * 128u));
                    __syncwarp();
                    if (lane < n_g) tc_tma_gather4(T.act[h] + 512 * lane, &map_a, ks * (FW_KB * 32) + 128 * h, crd[0], crd[1], crd[2], crd[3], &S.full[stg]);
                }
                __syncwarp();
            }
        }
        tc_drain<S.NS>(S.full, it);
    } else if (warp == FW_C_WARP) {
        // ============================ token constants (one warp) =====================
        bool ok = true;
        unsigned n_item = 0;
        for (int item = blockIdx.x; item < W.n && ok; item += gridDim.x, ++n_item) {
            const FwItem I = fw_item<TOK>(S, g, tw, n_rt, W, item);
            if (I.cnt <= 0) { --n_item; continue; }                      // (only items with tokens count)
            if (lane < TOK) {                                            // (no later than the item's first constants)
                const int slot = lane < I.cnt ? (g.perm ? __ldg(g.perm + I.tstart + lane) : I.tstart + lane) : 0;
                const float scl = lane < I.cnt && g.scale ? __ldg(g.scale + (slot >> g.a_shift)) : 1.0f;
                // an item's first stage is full when every dot warp has left the one NS stages before, and so the item NS + 1 before
                if (n_item >= S.NS + 1 && !tc_wait<TC_HINT_MMA>(S, &S.full[it % S.NS], (it / S.NS) & 1u, 36u)) ok = false;
                S.slot[n_item % (S.NS + 1)][lane] = slot;
                S.scl[n_item % (S.NS + 1)][lane] = scl;
            }
            if (__any_sync(LKB_FULL, !ok)) break;
            for (int ks = 0; ks < nstage; ++ks, ++it) {
                const unsigned stg = it % S.NS;
                if (!tc_wait<TC_HINT_MMA>(S, &S.full[stg], (it / S.NS) & 1u, 36u)) { ok = false; break; }
                FwStage<TOK> & T = S.st[stg];
                if (2 * lane < I.cnt) {                                  // lane: token pair
#pragma unroll
                    for (int b = 0; b < FW_KB; b += 2) {                 // two blocks a load
                        const float4 s0 = *reinterpret_cast<const float4 *>(&T.asc[2 * lane][b]), s1 = *reinterpret_cast<const float4 *>(&T.asc[2 * lane + 1][b]);
                        T.dc[b][lane]     = FOLD ? make_float4(s0.x, s1.x, -fmaf(s0.x, 12582912.0f, s0.y), -fmaf(s1.x, 12582912.0f, s1.y)) : make_float4(s0.x, s1.x, -s0.y, -s1.y);
                        T.dc[b + 1][lane] = FOLD ? make_float4(s0.z, s1.z, -fmaf(s0.z, 12582912.0f, s0.w), -fmaf(s1.z, 12582912.0f, s1.w)) : make_float4(s0.z, s1.z, -s0.w, -s1.w);
                    }
                }
                __syncwarp();
                tc_mbar_arrive_if(&S.ready[stg], lane == 0);
            }
        }
    } else {
        // ============================ dots (eight warps) =============================
        bool ok = true;
        unsigned n_item = 0;
        for (int item = blockIdx.x; item < W.n && ok; item += gridDim.x, ++n_item) {
            const FwItem I = fw_item<TOK>(S, g, tw, n_rt, W, item);
            if (I.cnt <= 0) { --n_item; continue; }                      // (only items with tokens count)
            if (16 * warp >= I.rows) {                                   // not a row of this part (the block's last): its stages as they come
                for (int ks = 0; ks < nstage && ok; ++ks, ++it) {
                    ok = tc_wait(S, &S.full[it % S.NS], (it / S.NS) & 1u, 33u);
                    tc_mbar_arrive_if(&S.empty[it % S.NS], lane == 0 && ok);
                }
                continue;
            }
            const int nt = (I.cnt + 7) >> 3;
            if (nt == 1) ok = fw_do_item<EPI, FOLD, TOK, 1>(S, it, n_item, g, I, nstage, warp, lane);
            if (nt == 2) ok = fw_do_item<EPI, FOLD, TOK, 2>(S, it, n_item, g, I, nstage, warp, lane);
            if constexpr (TOK > 16) {
                if (nt == 3) ok = fw_do_item<EPI, FOLD, TOK, 3>(S, it, n_item, g, I, nstage, warp, lane);
                if (nt == 4) ok = fw_do_item<EPI, FOLD, TOK, 4>(S, it, n_item, g, I, nstage, warp, lane);
            }
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
int lkb_tc_make_map(CUtensorMap * m, const void * base, unsigned row_bytes, unsigned long long pitch, unsigned long long rows,
                    unsigned box_bytes, unsigned box_rows, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2);           // lkb_gemm_tc.cu

typedef void (*FwKernel)(lkb_pf_gemm, int, int, int, int, CUtensorMap, CUtensorMap, FwMaps);
template <int TOK> static FwKernel fw_form(int epi, int fold) {
    return epi ? (fold ? k_pf_gemm_few<1, 1, TOK> : k_pf_gemm_few<1, 0, TOK>) : (fold ? k_pf_gemm_few<0, 1, TOK> : k_pf_gemm_few<0, 0, TOK>);
}
template <int TOK> static size_t fw_smem() { return sizeof(FwSmem<TOK>) + 1024; }
template <int TOK> static cudaError_t fw_allow_smem() {
    static_assert(sizeof(FwSmem<TOK>) + 1024 <= 227 * 1024, "a block's shared memory");
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < 4 && e == cudaSuccess; ++i) e = cudaFuncSetAttribute(fw_form<TOK>(i >> 1, i & 1), cudaFuncAttributeMaxDynamicSharedMemorySize, (int) fw_smem<TOK>());
    return e;
}
int lkb_gemm_few_init() {
    cudaError_t e = fw_allow_smem<16>();
    if (e == cudaSuccess) e = fw_allow_smem<32>();
    return e != cudaSuccess ? -(int) e : LKB_OK;
}
int lkb_gemm_few_take_status() { return tc_take_status(); }

// Where the forms cross.  Grouped: by the slots the caller states, spread over 64 experts.  A MoE layer at 400 / 440 / 480 / 520 / 600 tokens of four slots
// takes 196 / 214 / 223 / 241 / 268 us here and 212 / 220 / 224 / 240 / 260 in the
// tensor-core form with balanced routing, 209 / 212 / 223 / 235 / 260 and 235 / 239 / 242 / 250 / 270 with Zipf(1.1): the line lies at 480.  Items of 16 tokens to 200 tokens (at
// 180 gate|up 64 us, 68 with 32; the fifth stage is worth 7 % of a layer at 37 tokens), of 32 beyond.  A plan that cannot have a tile per expert is one of fewer experts, whose tiles may be
// full; it takes the other form, as does a call that does not state its slots.
#define FW_MIN_TILES LKB_N_EXPERTS
#define FW_MAX_SLOTS (480 * LKB_TOP_K)
#define FW_16_SLOTS  (200 * LKB_TOP_K)
// Dense: up to FW_MAX_DENSE tokens always, beyond by the time of either form's waves of items (fw_dense_width).
#define FW_MAX_DENSE 4
static int fw_row_tiles(int N, int epi) { return N / (epi ? FW_ROWS : 2 * FW_ROWS); }       // of an item: two tiles, SwiGLU form: of 128 output rows
// The token width of a dense problem's items, or 0 where the tensor-core form is faster: waves x the time of an item's block, which is 95, 128 or
// 176 ns at 8, 16 or 24 tokens here (64 blocks a row: a wave more takes 6.1, 8.2 or 11.3 us; 225 ns at 32, never better) against tc_dense_ns there, and 5 us more
// an item for launch, fill and drain.  us in the tensor-core form and here, caches flushed: in_proj (6144 rows) at 37 / 64 / 96 / 128 / 144 / 432 tokens
// 19.5 / 24.6 / 24.6 / 23.6 / 24.6 / 46.1 -> 14.3 / 16.4 / 16.4 / 18.9 / 19.0 / 39.9 (at 256 28.7 there, 32.8 here), out_proj (2048 rows) at 37 / 128 / 256 / 300 / 432
// 18.4 / 20.5 / 24.6 / 23.5 / 24.0 -> 12.3 / 12.3 / 16.4 / 17.9 / 18.9.
int lkb_gemm_tc_dense_ns(int ntok, int N, int sms, int epi);      // lkb_gemm_tc.cu
static int fw_dense_width(int ntok, int N, int bpr, int sms, int epi, bool always) {
    static const int ns[3] = {95, 128, 176};
    int best = 0;
    long long least = always ? 1ll << 62 : lkb_gemm_tc_dense_ns(ntok, N, sms, epi) - 5000 / bpr;
    for (int i = 0; i < 3; ++i) {
        const int tw = 8 * (i + 1);
        const long long items = (long long) ((ntok + tw - 1) / tw) * fw_row_tiles(N, epi), t = (items + sms - 1) / sms * ns[i];
        if (t < least) { least = t; best = tw; }
    }
    return best;
}
static int fw_width(const lkb_pf_gemm * g, int epi, int max_tiles, int sms) {
    if (!g->perm) return fw_dense_width(g->ntok, g->N, g->bpr, sms, epi, g->ntok <= FW_MAX_DENSE);
    if (max_tiles < FW_MIN_TILES || g->ntok <= 0 || g->ntok > FW_MAX_SLOTS) return 0;
    return g->ntok <= FW_16_SLOTS ? 16 : 32;
}
// Test hook (not in the public header): the items' token width where a call (with planes for quants: of the SwiGLU form) takes this form, if its
// planes allow it; else 0.
extern "C" __attribute__((visibility("default"))) int lkb_debug_gemm_few_width(const lkb_pf_gemm * g, int max_tiles, int sms) { return fw_width(g, g->oqs != nullptr, max_tiles, sms); }
// Test hook (not in the public header): the same for a call that this form serves whatever the other's time, at the smallest sizes: up to four dense
// tokens, or 47 routed ones.
extern "C" __attribute__((visibility("default"))) int lkb_debug_gemm_few_better(const lkb_pf_gemm * g, int max_tiles) {
    return g->ntok <= (g->perm ? 47 * LKB_TOP_K : FW_MAX_DENSE) && fw_width(g, 0, max_tiles, 148) > 0;
}

// Test hook (not in the public header): over `count` float bit patterns from `first` on, in either half of a pair whose other is 1, or any value that
// does not count: counts[0] += halves where tc_silu2 is sure of another result than lkb_silu's, counts[1] += those it is not sure of.
__global__ void k_debug_silu(unsigned first, unsigned long long count, unsigned long long * __restrict__ counts) {
    unsigned long long wrong = 0, unsure = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long) blockDim.x + threadIdx.x; i < count; i += (unsigned long long) gridDim.x * blockDim.x) {
        const unsigned bits = first + (unsigned) i;
        const float v = __uint_as_float(bits), other = __uint_as_float(bits * 2654435761u);
        const unsigned want = __float_as_uint(lkb_silu(v));
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int counts2 = 0; counts2 < 2; ++counts2) {
                const float o = counts2 ? 1.0f : (i & 1) ? other : (i & 2) ? __int_as_float(0x7FC00000) : 0.0f;
                bool sure = true;
                float q[2];
                tc_unpack(tc_silu2(half ? tc_pack(o, v) : tc_pack(v, o), sure, half ? counts2 : true, half ? true : counts2), q[0], q[1]);
                unsure += !sure;
                wrong += sure && __float_as_uint(q[half]) != want;
            }
    }
    if (wrong) atomicAdd(counts, wrong);
    if (unsure) atomicAdd(counts + 1, unsure);
}
extern "C" __attribute__((visibility("default"))) int lkb_debug_silu(unsigned first, unsigned long long count, unsigned long long * counts, lkb_stream_t st) {
    k_debug_silu<<<1184, 256, 0, (cudaStream_t) st>>>(first, count, counts);
    return lkb_check_launch();
}

// Parts of an item in a last wave (fw_work), as a shift: halves, or quarters where they fit.  Grouped the host does not know the items: halves.
static int fw_cut(long long items, int sms) {
    const long long rem = items % sms;
    return 4 * rem <= sms ? 2 : 2 * rem <= sms ? 1 : 0;
}

// LKB_ERR_UNSUPPORTED where another form is the better one or the planes do not have the alignment the copies ask for.
int lkb_gemm_few_launch(const lkb_pf_gemm * g, int epi, int fold, int max_tiles, cudaStream_t st) {
    if (!lkb_tensor_map_encoder()) return LKB_ERR_UNSUPPORTED;
    const int tw = fw_width(g, epi, max_tiles, lkb_context().sm_count);
    if (!tw) return LKB_ERR_UNSUPPORTED;
    if (epi ? (g->N % FW_ROWS) : (g->N % (2 * FW_ROWS))) return LKB_ERR_UNSUPPORTED;
    if (g->bpr % 8 || (((size_t) g->aqs | (size_t) g->asc) & 15) || g->exp_stride % g->bpr) return LKB_ERR_UNSUPPORTED;
    if (epi && ((size_t) g->oqs & 3)) return LKB_ERR_UNSUPPORTED;            // quants leave four at a time
    const int nseg = epi ? 2 : (g->seg_end[0] >= g->N ? 1 : g->seg_end[1] >= g->N ? 2 : 3);
    for (int s = 0; s < nseg; ++s) if (((size_t) g->qs[s] | (size_t) g->d[s]) & 15) return LKB_ERR_UNSUPPORTED;
    // L2 fetches 256 bytes at a time (with 64-byte pieces of a row gate|up at 37 tokens took 12 us less so)
    const CUtensorMapL2promotion l2 = CU_TENSOR_MAP_L2_PROMOTION_L2_256B;
    const unsigned long long any = 1ull << 30;              // row bound of a plane whose extent the caller does not state: it only clips
    CUtensorMap ma, ms;
    FwMaps maps;
    const unsigned long long rows = g->perm ? any : (unsigned long long) g->ntok;
    int r = lkb_tc_make_map(&ma, g->aqs, (unsigned) g->bpr * 32u, (unsigned) g->bpr * 32u, rows, FW_KB * 16u, 1u, CU_TENSOR_MAP_SWIZZLE_128B, l2);
    if (r == LKB_OK) r = lkb_tc_make_map(&ms, g->asc, (unsigned) g->bpr * 8u, (unsigned) g->bpr * 8u, rows, FW_KB * 8u, 1u, CU_TENSOR_MAP_SWIZZLE_NONE, l2);
    const int sms = lkb_context().sm_count, cut = g->perm ? 1 : fw_cut((long long) ((g->ntok + tw - 1) / tw) * fw_row_tiles(g->N, epi), sms);
    for (int p = 0; p < 2; ++p)
        for (int s = 0; s < 3 && r == LKB_OK; ++s) {
            const unsigned box = p ? FW_ROWS >> cut : FW_ROWS;
            if (s >= nseg || (p && !cut)) { const int f = s < nseg ? s : 0; maps.w[p][s] = maps.w[0][f]; maps.d[p][s] = maps.d[0][f]; continue; }
            r = lkb_tc_make_map(&maps.w[p][s], g->qs[s], (unsigned) g->bpr * 16u, (unsigned) g->bpr * 16u, any, FW_KB * 16u, box, CU_TENSOR_MAP_SWIZZLE_128B, l2);
            if (r == LKB_OK) r = lkb_tc_make_map(&maps.d[p][s], g->d[s], (unsigned) g->bpr * 2u, (unsigned) g->bpr * 2u, any, 16u, box, CU_TENSOR_MAP_SWIZZLE_NONE, l2);
        }
    if (r != LKB_OK) return r;
    const int rpe = (int) (g->exp_stride / g->bpr);
    const dim3 grid(sms), block(FW_THREADS);
    if (tw <= 16) LKB_PF_LAUNCH(fw_form<16>(epi, fold), grid, block, fw_smem<16>(), st, *g, max_tiles, rpe, tw, cut, ma, ms, maps);
    else           LKB_PF_LAUNCH(fw_form<32>(epi, fold), grid, block, fw_smem<32>(), st, *g, max_tiles, rpe, tw, cut, ma, ms, maps);
    return lkb_check_launch();
}
