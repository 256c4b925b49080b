// lkb_pfattn.cu - causal GQA flash attention of a prefill chunk for sm_100a: tcgen05 MMAs, scores and outputs in TMEM,
// operands by bulk tensor copies.
//
// m queries at positions P .. P+m-1 over keys 0 .. P+m-1, 32 heads on 8 KV heads, 64 dims, fp16 in (Q carries the exact 1/8),
// fp32 scores, softmax and output; P is rounded to fp16 for P V (the reference's own choice and error bound,
// ref: src/prefill.cu:1018-1028).
//
// An MMA tile is 128 rows = 32 positions x the 4 query heads of a KV head, so K and V are fetched once for all four.
//   S (128 x 128, fp32) = Q K^T        four K = 16 MMAs, both operands in shared memory
//   O (128 x 64, fp32) += P V          four K = 16 MMAs per 64 keys, P (fp16) from TMEM, V [key][dim] as an MN-major operand
// One thread owns one row: it reads the 128 scores from TMEM, needs no exchange for the row maximum, and writes the
// probabilities back to TMEM as the A operand of the second product.  The next tile's S is computed while this one's softmax
// runs.
//
// The softmax is the online one over steps of 64 keys, in the order of the warp-level (mma.sync) kernel that this one
// replaced, and both MMA forms add in the same order, so the outputs are the same bits (through forty layers of requantised
// activations the last bit of an attention output decides which experts later tokens take): per step the scores times
// log2 e, the running maximum, l = fma(l, alpha, the step's sum) in four chains of two keys out of eight, O *= alpha -- which
// touches TMEM only when a row of the warp has a new maximum (alpha is exactly 1 otherwise).
//
// What bounds it: a row and key cost 128 multiply-accumulates (1/32 cycle of the tensor pipe) and one ex2 (1/16 cycle of the
// SM's special function units): 1024 cycles per 128 x 128 tile against 512.  The exponentials are the busiest unit but do not
// fill it: 8192 tokens behind 24576 positions take 2.83 ms a layer, 64 % of the special function units' cycles, tensor pipe
// 32 %, issue 42 % (ncu); the rest is the softmax warps' waits for scores and for the P V product.  Two tiles per block
// (NT = 2: 64 positions, eight softmax warps) overlap those waits and halve the K / V traffic from L2; a chunk too short to
// give every SM such a block takes one tile per block.
// Every wait is bounded; on expiry a status word is set and all roles drain and exit, freeing TMEM.
#include "lkb_attn.cuh"
#include "lkb_tc.cuh"

#define FA_ROWS  128                        // rows of a tile
#define FA_POS   (FA_ROWS / AT_GQA)         // query positions of a tile
#define FA_KEYS  128                        // keys of a tile
#define FA_TILE  (FA_KEYS * AT_D * 2)       // bytes of a Q, K or V tile
#define FA_STEP  64                         // keys of a softmax step

template <int NT> struct FaCfg {
    static constexpr int SLOTS = NT == 2 ? 6 : 5;               // K and V tiles in flight, K0 V0 K1 V1 ...
    static constexpr int MMA_WARP = 4 * NT, TMA_WARP = 4 * NT + 1, THREADS = (4 * NT + 2) * 32;
    static constexpr int CTAS = NT == 2 ? 1 : 2;                // per SM
    static constexpr unsigned TMEM = 256 * NT;                  // per tile: S 0..127, P 128..191, O 192..255
};
template <int NT> struct FaSmem {
    alignas(1024) unsigned char q[NT][FA_TILE];
    alignas(1024) unsigned char kv[FaCfg<NT>::SLOTS][FA_TILE];
    alignas(8) unsigned long long qfull, full[FaCfg<NT>::SLOTS], empty[FaCfg<NT>::SLOTS], sfull[NT], sfree[NT], pfull[NT][2], pvdone[NT][2];
    unsigned tmem_base;
    int      abort;
};
// fp16 x fp16 -> fp32, M = 128
#define FA_IDESC_S  ((1u << 4) | ((FA_KEYS >> 3) << 17) | ((FA_ROWS >> 4) << 24))
#define FA_IDESC_PV ((1u << 4) | (1u << 16) | ((AT_D >> 3) << 17) | ((FA_ROWS >> 4) << 24))     // B is MN-major

__device__ __forceinline__ float fa_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned fa_pack(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const unsigned *>(&h);
}

// One row of Q (this softmax thread's) into the swizzled tile, for a base that no tensor copy takes: 16-byte chunk c of row r
// at c ^ (r & 7).  Rows past the chunk are zero.
__device__ __forceinline__ void fa_load_q(unsigned char * tile, const __half * q, int row, bool live) {
    const unsigned * p = reinterpret_cast<const unsigned *>(q);
#pragma unroll
    for (int c = 0; c < AT_D / 8; ++c) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (live) v = make_uint4(p[4 * c], p[4 * c + 1], p[4 * c + 2], p[4 * c + 3]);
        *reinterpret_cast<uint4 *>(tile + row * (AT_D * 2) + ((c ^ (row & 7)) << 4)) = v;
    }
    tc_fence_async();                                           // the MMAs read it through the asynchronous proxy
}

// Softmax of one row (one thread) over all key tiles.  Returns false when a wait gave up.
template <int NT>
__device__ __forceinline__ bool fa_softmax(FaSmem<NT> & S, int i, unsigned tb, int lane, int pos, int first_pos, int nkt, float & l_out) {
    const float LOG2E = 1.4426950408889634f;
    const unsigned long long le2 = tc_pack(LOG2E, LOG2E);
    float mrow = -1e30f, l[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int k = 0; k < nkt; ++k) {
        unsigned su[FA_KEYS];
        if (!tc_wait(S, &S.sfull[i], k & 1, 60u)) return false;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < FA_KEYS; c += 32) tc_ld32(tb + c, su + c);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        tc_mbar_arrive_if(&S.sfree[i], lane == 0);              // the next S may be computed
        // log2 domain.  (The product is rounded here, before the maximum is subtracted from it: one fused operation would
        // give other bits.)
#pragma unroll
        for (int c = 0; c < FA_KEYS; c += 2) {
            float x, y;
            tc_unpack(tc_fmul2(tc_pack_u(su[c], su[c + 1]), le2), x, y);
            su[c] = __float_as_uint(x); su[c + 1] = __float_as_uint(y);
        }
        if (k * FA_KEYS + FA_KEYS - 1 > first_pos) {            // the tile reaches past the first row's position (or the cache's end)
            const int last = pos - k * FA_KEYS;                 // last key of the tile that this row may see
#pragma unroll
            for (int c = 0; c < FA_KEYS; ++c) if (c > last) su[c] = 0xFF800000u;      // -inf: weight 0 under any maximum
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c0 = FA_STEP * h;
            float mx[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) mx[e] = __uint_as_float(su[c0 + e]);
#pragma unroll
            for (int c = 4; c < FA_STEP; c += 4)
#pragma unroll
                for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], __uint_as_float(su[c0 + c + e]));
            const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            const float mn = fmaxf(mrow, mt);
            const float alpha = fa_ex2(mrow - mn);
            const bool grown = mt > mrow;
            mrow = mn;
            // this half of P has been read; a new maximum also needs the output complete up to the step before
            if (k > 0 && !tc_wait(S, &S.pvdone[i][h], (k - 1) & 1, 61u)) return false;
            tc_fence_after();                                   // the stores into P below stay behind the MMAs that read it
            if ((k > 0 || h > 0) && __any_sync(LKB_FULL, grown)) {
                if (!tc_wait(S, &S.pvdone[i][h ^ 1], h ? k & 1 : (k - 1) & 1, 63u)) return false;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < AT_D; c += 8) {
                    unsigned o[8];
                    tc_ld8(tb + 192 + c, o);
                    tc_wait_ld();
#pragma unroll
                    for (int e = 0; e < 8; ++e) o[e] = __float_as_uint(__fmul_rn(__uint_as_float(o[e]), alpha));
                    tc_st8(tb + 192 + c, make_uint4(o[0], o[1], o[2], o[3]), make_uint4(o[4], o[5], o[6], o[7]));
                }
            }
            const unsigned long long nm2 = tc_pack(-mn, -mn);
            float ls[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < FA_STEP; c += 16) {
                unsigned p[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float x, y;
                    tc_unpack(tc_fadd2(tc_pack_u(su[c0 + c + 2 * e], su[c0 + c + 2 * e + 1]), nm2), x, y);
                    x = fa_ex2(x); y = fa_ex2(y);               // (below 2^-126 a term vanishes in fp16 and beside the row's 1)
                    ls[e & 3] = __fadd_rn(__fadd_rn(ls[e & 3], x), y);
                    p[e] = fa_pack(x, y);
                }
                tc_st8(tb + 128 + 32 * h + c / 2, make_uint4(p[0], p[1], p[2], p[3]), make_uint4(p[4], p[5], p[6], p[7]));
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) l[e] = fmaf(l[e], alpha, ls[e]);
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            tc_mbar_arrive_if(&S.pfull[i][h], lane == 0);
        }
    }
    l_out = __fadd_rn(__fadd_rn(l[0], l[1]), __fadd_rn(l[2], l[3]));
    return true;
}

template <int NT>
__global__ void __launch_bounds__(FaCfg<NT>::THREADS, FaCfg<NT>::CTAS) k_pf_attn_tc(const __grid_constant__ CUtensorMap map_q,
                                                                                    const __grid_constant__ CUtensorMap map_k,
                                                                                    const __grid_constant__ CUtensorMap map_v,
                                                                                    int m, int P, const __half * __restrict__ q_rows,
                                                                                    float * __restrict__ o) {
    lkb_pdl_wait(); lkb_pdl_trigger();           // programmatic dependent launch: inputs complete from here on
    typedef FaCfg<NT> C;
    extern __shared__ unsigned char fa_raw[];
    FaSmem<NT> & S = *reinterpret_cast<FaSmem<NT> *>(fa_raw + ((1024u - (tc_smem_u32(fa_raw) & 1023u)) & 1023u));
    const int ptid = threadIdx.x, warp = __shfl_sync(LKB_FULL, ptid >> 5, 0), lane = ptid & 31;
    const int qt = gridDim.x - 1 - blockIdx.x, kvh = blockIdx.y;                    // longest rows first
    const int q0 = qt * FA_POS * NT;
    const int kend = P + min(q0 + FA_POS * NT, m);                                  // keys 0 .. kend-1 matter to this block
    const int nkt = (kend + FA_KEYS - 1) / FA_KEYS;
    if (ptid == 0) {
        S.abort = 0;
        tc_mbar_init(&S.qfull, q_rows ? 4 * NT : 1);                                // the softmax warps, or the copy's issuer
        for (int s = 0; s < C::SLOTS; ++s) { tc_mbar_init(&S.full[s], 1); tc_mbar_init(&S.empty[s], 1); }
        for (int i = 0; i < NT; ++i) {
            tc_mbar_init(&S.sfull[i], 1); tc_mbar_init(&S.sfree[i], 4);             // MMA commit; the tile's four softmax warps
            for (int h = 0; h < 2; ++h) { tc_mbar_init(&S.pfull[i][h], 4); tc_mbar_init(&S.pvdone[i][h], 1); }
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(tc_smem_u32(&S.tmem_base)), "r"(C::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = S.tmem_base;

    if (warp == C::TMA_WARP) {
        const bool leader = tc_elect();
        if (leader && !q_rows) {
            tc_mbar_arrive_tx(&S.qfull, NT * FA_TILE);
            for (int i = 0; i < NT; ++i) tc_tma_tile3(S.q[i], &map_q, 0, kvh * AT_GQA, q0 + FA_POS * i, &S.qfull);
        }
        __syncwarp();
        int slot = 0;
        unsigned par = 1;                                       // every slot starts out empty
        int t = 0;
        for (; t < 2 * nkt; ++t) {                              // K0 V0 K1 V1 ...
            if (!tc_wait<TC_HINT_PROD>(S, &S.empty[slot], par, 50u)) break;
            if (leader) {
                tc_mbar_arrive_tx(&S.full[slot], FA_TILE);
                tc_tma_tile3(S.kv[slot], (t & 1) ? &map_v : &map_k, 0, kvh, (t >> 1) * FA_KEYS, &S.full[slot]);
            }
            __syncwarp();
            if (++slot == C::SLOTS) { slot = 0; par ^= 1u; }
        }
        tc_drain<1>(&S.qfull, q_rows ? 0 : 1);
        tc_drain<C::SLOTS>(S.full, t);
    } else if (warp == C::MMA_WARP) {
        const bool leader = tc_elect();
        int slot = 0;
        unsigned par = 0;
        auto next = [&]() { if (++slot == C::SLOTS) { slot = 0; par ^= 1u; } };
        auto scores = [&](int i) {                              // S_i = Q_i K^T from the current slot
            if (leader) {
                const unsigned long long a = tc_desc(tc_smem_u32(S.q[i])), b = tc_desc(tc_smem_u32(S.kv[slot]));
#pragma unroll
                for (int kk = 0; kk < AT_D / 16; ++kk) tc_mma_f16_ss(tmem + 256 * i, a + 2 * kk, b + 2 * kk, FA_IDESC_S, kk > 0);
                tc_commit(&S.sfull[i]);
            }
            __syncwarp();
        };
        bool ok = tc_wait<TC_HINT_MMA>(S, &S.qfull, 0u, 51u) && tc_wait<TC_HINT_MMA>(S, &S.full[slot], par, 52u);
        if (ok) {
            tc_fence_after();
            for (int i = 0; i < NT; ++i) scores(i);
            if (leader) tc_commit(&S.empty[slot]);
            __syncwarp();
            next();
        }
        for (int k = 0; k < nkt && ok; ++k) {
            const int vslot = slot;
            const unsigned vpar = par;
            next();
            if (k + 1 < nkt) {
                // the next scores, as soon as this tile's have been read
                if (!tc_wait<TC_HINT_MMA>(S, &S.full[slot], par, 52u)) { ok = false; break; }
                for (int i = 0; i < NT && ok; ++i) {
                    ok = tc_wait<TC_HINT_MMA>(S, &S.sfree[i], k & 1, 53u);
                    if (ok) { tc_fence_after(); scores(i); }
                }
                if (!ok) break;
                if (leader) tc_commit(&S.empty[slot]);
                __syncwarp();
                next();
            }
            if (!tc_wait<TC_HINT_MMA>(S, &S.full[vslot], vpar, 54u)) { ok = false; break; }
            // V [key][64 dims]: rows of 128 bytes, MN-major with the 128-byte swizzle; 16 keys = 2048 bytes
            const unsigned long long b = tc_desc(tc_smem_u32(S.kv[vslot]));
            for (int h = 0; h < 2 && ok; ++h)
                for (int i = 0; i < NT && ok; ++i) {
                    ok = tc_wait<TC_HINT_MMA>(S, &S.pfull[i][h], k & 1, 55u);
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
                        // no further than the tile's last key: a key that no row sees has weight 0, but 0 x inf is NaN, and a
                        // later token's value must not reach rows ahead of its own tile
                        const int live = P + min(q0 + FA_POS * (i + 1), m) - k * FA_KEYS - FA_STEP * h;
#pragma unroll
                        for (int kk = 0; kk < FA_STEP / 16; ++kk)
                            if (16 * kk < live)
                                tc_mma_f16_ts(tmem + 256 * i + 192, tmem + 256 * i + 128 + 32 * h + 8 * kk, b + 128 * (4 * h + kk), FA_IDESC_PV,
                                              (unsigned) (k > 0 || h > 0 || kk > 0));
                        tc_commit(&S.pvdone[i][h]);
                    }
                    __syncwarp();
                }
            if (leader && ok) tc_commit(&S.empty[vslot]);
            __syncwarp();
        }
    } else {
        const int i = warp >> 2, row = (warp & 3) * 32 + lane;
        const unsigned tb = tmem + 256 * i + ((unsigned) ((warp & 3) * 32) << 16);
        const int q = q0 + FA_POS * i + (row >> 2), head = kvh * AT_GQA + (row & 3);
        if (q_rows) {
            fa_load_q(S.q[i], q_rows + (size_t) (q < m ? q : 0) * LKB_HIDDEN + head * AT_D, row, q < m);
            __syncwarp();
            tc_mbar_arrive_if(&S.qfull, lane == 0);
        }
        float l;
        if (fa_softmax<NT>(S, i, tb, lane, P + q, P + q0 + FA_POS * i, nkt, l) && tc_wait(S, &S.pvdone[i][1], (nkt - 1) & 1, 62u)) {
            tc_fence_after();
            const float inv = __fdiv_rn(1.0f, l);
            unsigned r[AT_D];
            tc_ld32(tb + 192, r);
            tc_ld32(tb + 224, r + 32);
            tc_wait_ld();
            if (q < m) {
                float * const dst = o + (size_t) q * LKB_HIDDEN + head * AT_D;
#pragma unroll
                for (int c = 0; c < AT_D; c += 4) {
                    const float4 v = make_float4(__fmul_rn(__uint_as_float(r[c]), inv), __fmul_rn(__uint_as_float(r[c + 1]), inv),
                                                 __fmul_rn(__uint_as_float(r[c + 2]), inv), __fmul_rn(__uint_as_float(r[c + 3]), inv));
                    if (((size_t) o & 15) == 0) *reinterpret_cast<float4 *>(dst + c) = v;
                    else { dst[c] = v.x; dst[c + 1] = v.y; dst[c + 2] = v.z; dst[c + 3] = v.w; }
                }
            }
        }
    }
    // ---- teardown: everyone meets, then the allocating warp frees TMEM ------------
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(C::TMEM) : "memory");
    }
}

int lkb_pf_attn_init() {
    cudaError_t e = cudaFuncSetAttribute(k_pf_attn_tc<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(FaSmem<1>) + 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_pf_attn_tc<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(FaSmem<2>) + 1024);
    return e == cudaSuccess ? LKB_OK : -(int) e;
}
int lkb_pf_attn_take_status() { return tc_take_status(); }

// [rows][heads][64] fp16 as a 3-D tensor, box = 64 dims x box_heads x box_rows.  Rows past `rows` read as zero.
static int fa_make_map(CUtensorMap * t, const void * base, int heads, int rows, int box_heads, int box_rows) {
    const cuuint64_t dims[3] = {AT_D, (cuuint64_t) heads, (cuuint64_t) rows};
    const cuuint64_t strides[2] = {AT_D * 2, (cuuint64_t) heads * AT_D * 2};
    const cuuint32_t box[3] = {AT_D, (cuuint32_t) box_heads, (cuuint32_t) box_rows};
    const cuuint32_t es[3] = {1, 1, 1};
    return lkb_tensor_map_encoder()(t, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides, box, es,
                                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? LKB_OK : LKB_ERR_UNSUPPORTED;
}

extern "C" int lkb_pf_attn(const void * qh, int m, int P, const void * kc, const void * vc, float * o, lkb_stream_t st) {
    if (!lkb_context().inited || !lkb_tensor_map_encoder()) return LKB_ERR_NOT_INIT;
    if (!qh || !kc || !vc || !o) return LKB_ERR_NULL;
    // The cache is read by tensor copies alone (16 bytes); Q by one, or from 4-byte words where its base does not allow it.
    if (m <= 0 || P < 0 || ((size_t) qh & 3) || (((size_t) kc | (size_t) vc) & 15) || ((size_t) o & 3)) return LKB_ERR_SHAPE;
    const __half * const q_rows = ((size_t) qh & 15) ? (const __half *) qh : nullptr;
    CUtensorMap mq, mk, mv;
    int r = fa_make_map(&mk, kc, AT_KVH, P + m, 1, FA_KEYS);
    if (r == LKB_OK) r = fa_make_map(&mv, vc, AT_KVH, P + m, 1, FA_KEYS);
    mq = mk;                                                    // (q_rows: never used)
    if (r == LKB_OK && !q_rows) r = fa_make_map(&mq, qh, AT_HEADS, m, AT_GQA, FA_POS);
    if (r != LKB_OK) return r;
    const int two = (m + 2 * FA_POS - 1) / (2 * FA_POS);
    if (two * AT_KVH >= lkb_context().sm_count)
        return lkb_launch_next(k_pf_attn_tc<2>, dim3(two, AT_KVH), dim3(FaCfg<2>::THREADS), sizeof(FaSmem<2>) + 1024, (cudaStream_t) st, mq, mk, mv, m, P, q_rows, o);
    return lkb_launch_next(k_pf_attn_tc<1>, dim3((m + FA_POS - 1) / FA_POS, AT_KVH), dim3(FaCfg<1>::THREADS), sizeof(FaSmem<1>) + 1024, (cudaStream_t) st,
                      mq, mk, mv, m, P, q_rows, o);
}
