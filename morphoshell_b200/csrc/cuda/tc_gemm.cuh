// Tensor-core primitives (tcgen05, tensor memory, mbarriers) of the warm-start
// network's kernels (learned.cu).  BF16 operands in shared memory in the
// no-swizzle core-matrix layouts, FP32 accumulators in tensor memory.  Every
// mbarrier wait is bounded.
#pragma once

#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace msb {
namespace tc {

constexpr int kBM = 128;  // rows of an accumulator tile

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor: no swizzle (layout type 0), descriptor
// version 1, base offset 0.  Core matrices are 128 contiguous bytes.  K-major:
// 8 rows x 16 bytes of K, the next 16 bytes of K lbo away, the next 8 rows sbo
// away.  MN-major: 8 K x 16 bytes of rows, the next 8 K lbo away, the next 8
// rows sbo away.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, M =
// 128, N = n; both K-major, or both MN-major.
__host__ __device__ constexpr uint32_t instr_desc_bf16(int n, bool mn_major = false) {
    return (1u << 4)                                        // C format F32
           | (1u << 7)                                      // A format BF16
           | (1u << 10)                                     // B format BF16
           | (mn_major ? (1u << 15) | (1u << 16) : 0u)      // A, B transposed
           | ((uint32_t)(n >> 3) << 17)                     // N / 8
           | ((uint32_t)(kBM >> 4) << 24);                  // M / 16
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// CLUSTER: with the arrivals of other CTAs of the cluster ordered before it.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    if constexpr (CLUSTER)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
    return ok != 0;
}

// Waits for the phase with the given parity to complete, for at most about
// a second of SM clock; false on timeout.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait<CLUSTER>(bar, parity)) {
        if (clock64() - t0 > 2000000000LL) return false;
    }
    return true;
}

// One lane of a converged warp, the same one each time.
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}

// The same place in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// 16 bytes into a peer's shared memory, counted on a barrier there when they
// have landed.
__device__ __forceinline__ void store_async(uint32_t dst, const uint4& v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     dst),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}

// Arrives on the barrier at this offset in every CTA of the mask once this
// thread's earlier MMAs are done.
__device__ __forceinline__ void mma_commit_cluster(uint64_t* bar, uint16_t mask) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"(mask)
        : "memory");
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Arms the barrier for `bytes` and starts the copy.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
    bulk_copy(dst, src, bytes, bar);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// Issues the load only; tmem_wait() before the values are used.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
        "%23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Largest magnitude of three; NaN when one is.
__device__ __forceinline__ float max_abs(float a, float b, float c) {
    float m;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}

// q[j] = a[j] / (1 + exp(-z[j])), a[j] = z[j] or finite: the quotient by an
// approximate reciprocal, corrected once by its own residual (Markstein, IBM J.
// Res. Dev. 34, 1990); the division itself for a |z| of 34 and more or NaN:
// there two divisors' product may leave the range in which the reciprocal is
// normal, an infinite a has no residual, and a NaN would reach the other of its
// pair.  One test for all of them, and one reciprocal for two divisors: the
// epilogues are bound by the special-function units (16 operations per SM and
// clock) and their issue slots.  The exponential may flush a denormal result
// to zero: it is added to 1.
// Against the division, over all 2^32 pairs of BF16 z with finite z: z / (1 +
// exp(-z)) differs in the last bit of 1,205 pairs' quotients, of none once
// rounded to BF16, and -0 gives +0; 1 / (1 + exp(-z)) in 152,492 pairs, all but
// 44 of them with the divisor 2 - 2^-23 (z near 1e-7), whose reciprocal lies
// 2^-25 of a unit of its last place from the middle between two numbers.
template <int N>
__device__ __forceinline__ void over_one_plus_exp(const float (&a)[N], const float (&z)[N], float (&q)[N]) {
    static_assert(N % 2 == 0, "divisors are taken in pairs");
    float d[N], most = 0.0f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        float e;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z[j] * -1.4426950408889634f));
        d[j] = 1.0f + e;
    }
#pragma unroll
    for (int j = 0; j < N; j += 2) most = max_abs(most, z[j], z[j + 1]);
    // One reciprocal for two divisors: 1 / x = y / (x y).
#pragma unroll
    for (int j = 0; j < N; j += 2) {
        float rr;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rr) : "f"(d[j] * d[j + 1]));
        const float r0 = rr * d[j + 1], r1 = rr * d[j];
        const float t0 = a[j] * r0, t1 = a[j + 1] * r1;
        q[j] = fmaf(fmaf(-t0, d[j], a[j]), r0, t0);
        q[j + 1] = fmaf(fmaf(-t1, d[j + 1], a[j + 1]), r1, t1);
    }
    if (!(most < 34.0f)) {
#pragma unroll
        for (int j = 0; j < N; ++j) q[j] = a[j] / (1.0f + __expf(-z[j]));
    }
}

}  // namespace tc
}  // namespace msb
