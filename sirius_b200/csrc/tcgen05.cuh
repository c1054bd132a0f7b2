// tcgen05.cuh — PTX wrappers for the 5th-generation tensor cores (sm_100a):
// UMMA shared-memory and instruction descriptors, tcgen05.mma / commit /
// ld / st, mbarriers with waits bounded by the device clock, the 1-D bulk
// copy, and the BF16 packing and SiLU used by the surrogate's epilogues.
//
// Shared-memory operand layout used throughout: K-major, no swizzle, in 8 x
// 16-byte core matrices; element (row, k) of an operand with K columns sits
// at byte (row % 8) * 16 + (row / 8) * SBO + (k / 8) * 128 + (k % 8) * 2 with
// SBO = (K / 8) * 128, and the descriptor's LBO (next core matrix along K)
// is 128 bytes.
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

namespace sirius {
namespace tc {

// byte offset of element (row, k) in a K-major core-matrix image with K columns
__host__ __device__ inline int packed_offset(int row, int k, int K) {
    return (row % 8) * 16 + (row / 8) * (K / 8) * 128 + (k / 8) * 128 + (k % 8) * 2;
}

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory descriptor: no swizzle, K-major; LBO = 128 B (next core
// matrix along K), SBO = stride between 8-row groups; version 1 (sm_100).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t sbo_bytes) {
    return uint64_t((addr & 0x3FFFF) >> 4) | (uint64_t(128 >> 4) << 16) | (uint64_t(sbo_bytes >> 4) << 32) |
           (uint64_t(1) << 46);
}

// Instruction descriptor of kind::f16: D F32, A and B BF16, both K-major, M = 128.
__device__ __forceinline__ uint32_t instr_desc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t phase) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    return done != 0;
}

__device__ __forceinline__ unsigned long long dev_clock_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Wait for the mbarrier phase, at most limit_ns on the device clock.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase, unsigned long long limit_ns) {
    if (mbar_test(bar, phase)) return true;
    const unsigned long long t0 = dev_clock_ns();
    while (!mbar_test(bar, phase))
        if (dev_clock_ns() - t0 > limit_ns) return false;
    return true;
}

// 2-D tiled tensor copy (TMA) from global to this CTA's shared memory, no
// multicast; tmap is the address of a CUtensorMap in kernel-parameter or global
// memory, (x, y) the box's first element (x the innermost, in elements). The
// copy's bytes complete on bar, which must expect them.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(tmap), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// UMMA shared-memory descriptor, K-major with the 128-byte swizzle that a TMA box
// of 128-byte rows writes: rows of 128 B with their 16-byte pieces XOR-permuted by
// row % 8, 8-row groups 1024 B apart (SBO), LBO 16 B, layout type 2 (bits 61-63),
// version 1. The box starts 1024-byte aligned; a K step of 16 elements advances
// the start address by 32 B.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    return uint64_t((addr & 0x3FFFF) >> 4) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
           (uint64_t(2) << 61);
}

// The same swizzle for an MN-major operand: each TMA box holds 64 K rows of 64
// MN elements (128 B per K row, 8 KB per box), the operand's MN extent in boxes
// 8 KB apart (LBO), 8-row K groups 1024 B apart (SBO); a K step of 16 advances the
// start by two groups (2048 B).
__device__ __forceinline__ uint64_t smem_desc_sw128_mn(uint32_t addr) {
    return uint64_t((addr & 0x3FFFF) >> 4) | (uint64_t(8192 >> 4) << 16) | (uint64_t(1024 >> 4) << 32) |
           (uint64_t(1) << 46) | (uint64_t(2) << 61);
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive FP32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 consecutive FP32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// SiLU x (1 + tanh(x / 2)) / 2 of two values plus a bias each, packed FP32 arithmetic, one MUFU op each
__device__ __forceinline__ float2 silu_bias2(float2 v, float2 bias) {
    const float2 u = __fmul2_rn(__fadd2_rn(v, bias), make_float2(0.5f, 0.5f));
    float2 t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.x) : "f"(u.x));
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.y) : "f"(u.y));
    return __fmul2_rn(u, __fadd2_rn(t, make_float2(1.f, 1.f)));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}

// A network input row as two BF16 terms per feature: columns 0..4 hold
// hi_i = bf16(f_i), columns 5..9 lo_i = bf16(f_i - hi_i) (f_i - hi_i is exact in
// FP32), columns 10..15 zero. With the first layer's weights repeated in columns
// 0..4 and 5..9, the product W1 (hi + lo) carries 16 significant bits of each
// feature instead of 8 (one BF16 step of alpha / 20 near 0.5 is 0.04 M, more
// than a pixel of a 2048-wide frame). The two 8-column chunks of the row as uint4.
__device__ __forceinline__ void pack_input_row(const float* f, uint4& c0, uint4& c1) {
    float hi[5], lo[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        hi[i] = __bfloat162float(__float2bfloat16_rn(f[i]));
        lo[i] = f[i] - hi[i];
    }
    c0 = make_uint4(pack_bf16x2(hi[0], hi[1]), pack_bf16x2(hi[2], hi[3]), pack_bf16x2(hi[4], lo[0]),
                    pack_bf16x2(lo[1], lo[2]));
    c1 = make_uint4(pack_bf16x2(lo[3], lo[4]), 0u, 0u, 0u);
}

// ---- pairs of CTAs (cta_group::2): one MMA over both CTAs' rows, M = 256. Each CTA
// holds its 128 rows of A and of D, and its half of B's N rows, at the same
// addresses; the even CTA issues.
__device__ __forceinline__ uint32_t instr_desc_pair(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(256 >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n" ::"r"(
            tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0));
}

__device__ __forceinline__ void mma_bf16_ts_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n" ::"r"(
            tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0));
}

// arrives once on the barrier at this address of both CTAs when the MMAs issued so far are done
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"(uint16_t(3))
        : "memory");
}

// the same on this CTA's barrier alone
__device__ __forceinline__ void mma_commit_pair_own(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// the address of CTA `rank`'s copy of a shared-memory address
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// The same without the release of ordinary memory at cluster scope, whose fence costs
// more than the arrival: for work in tensor memory alone, which tcgen05.fence orders (a
// proxy fence does not: it orders one thread's accesses, and hands none over to another).
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

__device__ __forceinline__ void st_cluster_u64(uint32_t cluster_addr, unsigned long long v) {
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(cluster_addr), "l"(v) : "memory");
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// mbar_wait for a phase that the other CTA may complete (acquire at cluster scope)
__device__ __forceinline__ bool mbar_test_cluster(uint32_t bar, uint32_t phase) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t phase, unsigned long long limit_ns) {
    if (mbar_test_cluster(bar, phase)) return true;
    const unsigned long long t0 = dev_clock_ns();
    while (!mbar_test_cluster(bar, phase))
        if (dev_clock_ns() - t0 > limit_ns) return false;
    return true;
}

// 16 consecutive 32-bit columns of this thread's TMEM lane, without the wait; the
// registers may be read once tmem_wait_ld16 has passed them.
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t r[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// (the registers are operands, so no use of them moves above the wait)
__device__ __forceinline__ void tmem_wait_ld16(uint32_t r[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])::"memory");
}

// 8 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t r[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

#endif  // __CUDACC__

}  // namespace tc
}  // namespace sirius
