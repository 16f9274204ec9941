// What the recurrence kernels on thread-block clusters share (lstm_cluster.cu, lstm_single.cu, lstm_wide.cu): activations, bounded waits on
// transaction barriers, sequence lengths.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"

namespace b2 {
namespace cluster {

constexpr unsigned SPIN_LIMIT = 1u << 21;

// fp32 values as two fp16 terms, x*S = hi + lo*2^-11; the scales of h (below 1) and of the gate deltas (clipped to [-1, 1])
constexpr float LO_SCALE = 2048.0f, LO_UNSCALE = 1.0f / 2048.0f, S_H = 16384.0f, S_D = 32768.0f;
__device__ __forceinline__ uint32_t split_pair(float x, float S) {   // fp16 hi in the low half, lo in the high half
    const float xs = x * S;
    const __half h = __float2half_rn(xs);
    const __half l = __float2half_rn((xs - __half2float(h)) * LO_SCALE);
    return (uint32_t)__half_as_ushort(h) | ((uint32_t)__half_as_ushort(l) << 16);
}

// 1 / d, 1 <= d < 2^126: the hardware approximation (relative error e <= 2^-23) and one Newton step (r + r (1 - d r), relative error
// e^2 before the last rounding): within 0.5001 ulp, without the division's branches
__device__ __forceinline__ float cl_rcp(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-d, r, 1.0f), r);
}
// The exponent limits take the place of the reference's cut-offs (activation_functions/Logistic.cuh): above the upper one the quotients
// are 0 (logistic) and -1 (tanh); the lower one is where a NaN goes, which ends as 1 like there.  tanh as (1 - e) / (1 + e),
// e = exp(-2x), loses less than 2 logistic(2x) - 1 does.
__device__ __forceinline__ float cl_exp(float x, float most) { return expf(fminf(fmaxf(x, -88.0f), most)); }
__device__ __forceinline__ float cl_logistic(float x) { return cl_rcp(1.0f + cl_exp(-x, 88.0f)); }
__device__ __forceinline__ float cl_tanh(float x) {
    const float e = cl_exp(-2.0f * x, 40.0f);
    return (1.0f - e) * cl_rcp(1.0f + e);
}

// waits for a phase of a barrier in this block's shared memory; default (cta-scope) acquire, as for any transaction barrier
__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_bounded(uint32_t bar, uint32_t parity, int *status) {
    for (unsigned it = 0; it < SPIN_LIMIT; ++it) {
        if (try_wait(bar, parity)) return true;
        if ((it & 1023u) == 1023u && ptx::ld_relaxed_s32(status) != 0) return false;
    }
    atomicCAS(status, 0, (int)B2_ERR_STEP_TIMEOUT);
    return false;
}

// length of sequence pg: padding frames trail a sequence, as the data set writes them; frames below Tmin are real for all
__device__ __forceinline__ int sequence_length(const LstmShape &sh, const char *pat, int pg) {
    if (pg >= sh.P) return 0;
    int lo = sh.Tmin, hi = sh.T;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (pat[(size_t)mid * sh.P + pg] == PAT_NONE) hi = mid; else lo = mid + 1;
    }
    return lo;
}
// makes the compiler finish values here, ahead of a wait, instead of behind it where they would lengthen the chain of a step
template <class... F>
__device__ __forceinline__ void settle(F &...v) { (void)(int[]){(([&] { asm volatile("" : "+f"(v)); })(), 0)...}; }
__device__ __forceinline__ float lds(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }

// A launch in clusters of `cluster` blocks (0: none), cooperative where blocks of different clusters wait for each other
struct Launch {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    Launch(int blocks, int threads, size_t smem, int cluster, bool cooperative, cudaStream_t st) {
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = attr;
        if (cooperative) {
            attr[cfg.numAttrs].id = cudaLaunchAttributeCooperative;
            attr[cfg.numAttrs++].val.cooperative = 1;
        }
        if (cluster) {
            attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
            attr[cfg.numAttrs].val.clusterDim.x = cluster;
            attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
            ++cfg.numAttrs;
        }
    }
    Launch(const Launch &) = delete;
    Launch &operator=(const Launch &) = delete;
};
// allows a kernel `smem` bytes of dynamic shared memory and, above 8, clusters of `cluster` blocks
inline bool allow(const void *kern, size_t smem, int cluster) {
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
                    (cluster <= 8 || cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
    if (!ok) cudaGetLastError();
    return ok;
}
// clusters of a launch that the current device holds at once
inline int resident(const void *kern, const Launch &l) {
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &l.cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
    return n;
}

}  // namespace cluster
}  // namespace b2
