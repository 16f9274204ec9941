// What the recurrence kernels on thread-block clusters share (lstm_cluster.cu, lstm_single.cu, lstm_wide.cu): activations, bounded waits on
// transaction barriers, sequence lengths.
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace b2 {
namespace cluster {

constexpr unsigned SPIN_LIMIT = 1u << 21;

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

}  // namespace cluster
}  // namespace b2
