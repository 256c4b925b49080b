// lkb_tc.cuh - sm_100a primitives of the tensor-core kernels: mbarriers, bulk tensor copies, tcgen05 loads, stores and MMAs.
// No copy here is a multicast one.
#pragma once
#include "lkb_device.cuh"
#include <cuda.h>

#define TC_SPIN      (1u << 24)

// 0, or the code of the first bounded wait of this translation unit that expired
static __device__ unsigned g_tc_status;
static inline int tc_take_status() {             // reads and clears it; the device must be idle
    unsigned v = 0, z = 0;
    if (cudaMemcpyFromSymbol(&v, g_tc_status, sizeof v) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_tc_status, &z, sizeof z);
    return (int) v;
}
typedef CUresult (*tc_encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
tc_encode_fn lkb_tensor_map_encoder();           // cuTensorMapEncodeTiled, or null before lkb_init (lkb_gemm_tc.cu)

__device__ __forceinline__ unsigned tc_smem_u32(const void * p) { return (unsigned) __cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_mbar_init(unsigned long long * b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(tc_smem_u32(b)), "r"(count));
}
__device__ __forceinline__ void tc_mbar_arrive(unsigned long long * b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(tc_smem_u32(b)) : "memory");
}
__device__ __forceinline__ void tc_mbar_arrive_if(unsigned long long * b, bool yes) {      // without a divergent branch
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %1, 0;\n @p mbarrier.arrive.shared::cta.b64 _, [%0];\n}"
                 :: "r"(tc_smem_u32(b)), "r"((unsigned) yes) : "memory");
}
__device__ __forceinline__ void tc_mbar_arrive_tx(unsigned long long * b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(tc_smem_u32(b)), "r"(bytes) : "memory");
}
// One poll of an mbarrier phase.  HINT_NS > 0: the thread may stay suspended in hardware until the phase completes or
// the hint runs out, instead of coming back at once to spin through the issue slots the epilogue warps need.
template <int HINT_NS>
__device__ __forceinline__ bool tc_mbar_try(unsigned long long * b, unsigned parity) {
    unsigned ok;
    if (HINT_NS > 0)
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(tc_smem_u32(b)), "r"(parity), "r"((unsigned) HINT_NS) : "memory");
    else
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(tc_smem_u32(b)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false when it expired or another role of the block already gave up (S.abort).  The roles with slack (producer,
// expansion, issuer) poll with a suspend hint; the epilogue warps, whose waits are almost always over already, spin.
template <int HINT_NS = 0, class SM>
__device__ __forceinline__ bool tc_wait(SM & S, unsigned long long * b, unsigned parity, unsigned code) {
    if (__builtin_expect(tc_mbar_try<0>(b, parity), 1)) return true;
#pragma unroll 1
    for (unsigned i = 0; i < (HINT_NS > 0 ? TC_SPIN >> 4 : TC_SPIN); ++i) {
        if (tc_mbar_try<HINT_NS>(b, parity)) return true;
        if ((i & (HINT_NS > 0 ? 15u : 255u)) == 0u && *(volatile int *) &S.abort) return false;
    }
    atomicCAS(&g_tc_status, 0u, code);
    *(volatile int *) &S.abort = 1;
    return false;
}
#define TC_HINT_PROD 2000           // ns
#define TC_HINT_MMA  500
// How a copying role leaves, whoever gave up: the copies of the last N stages before `it` land before the block ends (bounded).  On the
// ordinary path another role needs them all the same.
template <int N> __device__ __forceinline__ void tc_drain(unsigned long long * full, unsigned it) {
#pragma unroll 1
    for (unsigned k = it < N ? 0u : it - N; k < it; ++k)
        for (unsigned i = 0; i < 4096u && !tc_mbar_try<TC_HINT_PROD>(&full[k % N], (k / N) & 1u); ++i) { }
}
__device__ __forceinline__ bool tc_elect() {
    unsigned p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tc_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after()  { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(unsigned long long * b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(tc_smem_u32(b)) : "memory");
}
// D (+)= A*B: int8 with A in TMEM, fp16 with A in TMEM or in shared memory; B in shared memory
__device__ __forceinline__ void tc_mma_i8(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc, unsigned idesc, unsigned acc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tc_mma_f16_ts(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc, unsigned idesc, unsigned acc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tc_mma_f16_ss(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc, unsigned idesc, unsigned acc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
// K-major B operand, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart (stride byte offset); a K step of
// 32 bytes inside the swizzle span moves the start address.
__device__ __forceinline__ unsigned long long tc_desc(unsigned smem_addr) {
    return (unsigned long long) ((smem_addr >> 4) & 0x3FFFu) | (1ull << 16)
         | ((unsigned long long) (1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// N columns of this warp's 32 lanes -> registers r[0..N)
__device__ __forceinline__ void tc_ld8(unsigned taddr, unsigned * r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld16(unsigned taddr, unsigned * r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld32(unsigned taddr, unsigned * r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
template <int NC>
__device__ __forceinline__ void tc_ld(unsigned taddr, unsigned (&r)[NC]) {
    static_assert(NC == 8 || NC == 16, "what the epilogue's halves need");
    if constexpr (NC == 8) tc_ld8(taddr, r); else tc_ld16(taddr, r);
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_st8(unsigned taddr, const uint4 a, const uint4 b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Two independent IEEE fused multiply-adds in one instruction.
__device__ __forceinline__ unsigned long long tc_pack(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ unsigned long long tc_pack_u(unsigned x, unsigned y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(x), "r"(y));
    return r;
}
__device__ __forceinline__ unsigned long long tc_ffma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long tc_fmul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long tc_fadd2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ void tc_unpack(unsigned long long v, float & x, float & y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
// lkb_silu of two values without the divide's branches, so that many are in flight: a reciprocal refined once (Newton), the quotient
// corrected by its exact remainder (Markstein 1990), which rounds as the IEEE division does unless something under- or overflows on
// the way.  `sure` is cleared where that may be (results of 0 and up to 1e-17, infinities, NaN) and the value counts: the caller takes lkb_silu there.
// Equal to it for every other float (test_gpu_silu.py).  gate|up, whose SwiGLU stores it is for, at 384 / 509 / 1237 / 4096 tokens 105 / 121 / 242 / 570 us
// with lkb_silu, 96 / 115 / 223 / 530 with this (without any silu 512 at 4096), 95 / 114 / 208 / 514 since a value of no token does not count.
__device__ __forceinline__ unsigned long long tc_silu2(unsigned long long v, bool & sure, bool counts0 = true, bool counts1 = true) {
    float v0, v1, d0, d1, y0, y1;
    tc_unpack(v, v0, v1);
    const unsigned long long one = tc_pack(1.0f, 1.0f), d = tc_fadd2(one, tc_pack(__expf(-v0), __expf(-v1)));
    tc_unpack(d, d0, d1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(d0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(d1));
    const unsigned long long nd = tc_pack(-d0, -d1);
    unsigned long long y = tc_pack(y0, y1);
    y = tc_ffma2(tc_ffma2(nd, y, one), y, y);
    unsigned long long q = tc_fmul2(v, y);
    q = tc_ffma2(tc_ffma2(nd, q, v), y, q);
    float q0, q1;
    tc_unpack(q, q0, q1);
    sure = sure && (!counts0 || fabsf(q0) > 1e-17f) && (!counts1 || fabsf(q1) > 1e-17f);
    return q;
}
// one tile of a 2-D tensor: box at (x, y) -> shared memory, bytes counted on the mbarrier
__device__ __forceinline__ void tc_tma_tile(void * dst, const CUtensorMap * map, int x, int y, unsigned long long * bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 :: "r"(tc_smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(tc_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_tma_tile3(void * dst, const CUtensorMap * map, int x, int y, int z, unsigned long long * bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 :: "r"(tc_smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(tc_smem_u32(bar)) : "memory");
}
// four rows y0..y3 of a 2-D tensor, columns from x on, one box width each -> four consecutive rows in shared memory
__device__ __forceinline__ void tc_tma_gather4(void * dst, const CUtensorMap * map, int x, int y0, int y1, int y2, int y3,
                                               unsigned long long * bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
                 :: "r"(tc_smem_u32(dst)), "l"(map), "r"(x), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(tc_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_cp16(void * dst, const void * src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(tc_smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void tc_cp8(void * dst, const void * src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"(tc_smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void tc_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void tc_cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }
