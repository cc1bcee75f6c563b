// pi_common.cuh -- device helpers shared by the power-iteration kernels.
#pragma once
#include <stdint.h>

#include <type_traits>

namespace sgpb {

// The next raw iterate value r_i of row i from u_i = (x_i - mu) / nu and
// its row sum acc (plain: sum_j w_ij x_j; MX: sum_j w_ij (x_i - x_j)):
// shifted Laplacian r = (gb - d) u + A u = gb u - L u, or the lazy random
// walk r = u / 2 + (A u)_i / (2 d) of the normalized variant (r = u / 2 for
// an isolated vertex).  All in FP64.
template <bool MX>
__device__ __forceinline__ double next_value(int normlap, double gb, double mu, double inv_nu, double ui, double acc,
                                             double d) {
    if constexpr (MX) {
        const double lu = acc * inv_nu;   // (L u)_i; the mean cancels in the differences
        return normlap ? (d > 0 ? ui - 0.5 * lu / d : 0.5 * ui) : gb * ui - lu;
    } else {
        const double au = (acc - mu * d) * inv_nu;   // (A u)_i
        return normlap ? 0.5 * ui + (d > 0 ? 0.5 * au / d : 0.0) : (gb - d) * ui + au;
    }
}

// An iterate whose norm is this much smaller than the terms it is the sum of
// has lost as much of its precision, and the order of its sums shows: a start
// vector against its mean (|x - mean|^2 / (n mean^2)), r against the shift
// (|r|^2 / gb^2 with |u| = 1; two vertices joined by an edge have r = 0).
constexpr double kCancel = 1e-6;

// Sum of three values over a warp, packed: value k of the warp ends up in
// lanes with (lane & 3) == k (k < 3).  6 double shuffles instead of 15.
__device__ __forceinline__ double warp_sum3(double a, double b, double c) {
    const unsigned lane = threadIdx.x & 31;
    const bool o1 = lane & 1, o2 = lane & 2;
    // step 1: even lanes keep (a, c), odd lanes keep (b, 0)
    double k0 = o1 ? b : a, s0 = o1 ? a : b;
    double k1 = o1 ? 0.0 : c, s1 = o1 ? c : 0.0;
    k0 += __shfl_xor_sync(0xFFFFFFFFu, s0, 1);
    k1 += __shfl_xor_sync(0xFFFFFFFFu, s1, 1);
    // step 2: lanes without bit 1 keep k0, the others k1
    double v = o2 ? k1 : k0;
    const double s = o2 ? k0 : k1;
    v += __shfl_xor_sync(0xFFFFFFFFu, s, 2);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 4);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 8);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 16);
    return v;
}

// mbarriers and 1-D bulk copies into shared memory
constexpr uint32_t kMbarWaitLimit = 1u << 22;   // polls before giving up
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait for the phase of the given parity to complete
__device__ __forceinline__ bool mbar_wait(uint64_t *b, uint32_t parity) {
    for (uint32_t k = 0; k < kMbarWaitLimit; k++)
        if (mbar_test(b, parity)) return true;
    return false;
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}

// nanoseconds of the device-wide timer
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

}  // namespace sgpb
