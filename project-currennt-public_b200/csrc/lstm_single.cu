// Persistent LSTM recurrence for ONE sequence per thread-block cluster (up to 512 units per direction): fp32 FFMA with the
// recurrent weights of a direction resident in the cluster's registers and tensor memory, exchange through distributed shared memory.
//
// Replaces the reference's per-timestep loop of 4 cublasSgemm + 1 Thrust functor per direction
// (layers/LstmLayer.cu:1805-1858,1878-1927 forward with ComputeBlockOutputFn :57-185; :2115-2176,2195-2253 backward with
// ComputeBlockErrorsFn :237-405 of the reference) where a fraction holds one or a few sequences.
//
// What bounds a step.  A matrix-vector product has no use for an MMA's 8 columns, so this is FFMA: 512 units are 65536 weights per
// block of a cluster of 16, 512 cycles of the FFMA pipes; the rest of a step is the exchange (450 cycles for the first byte plus about
// one per 16 bytes received), reductions and cell math.  65536 fp32 weights fill the register file, so half of them live in TENSOR
// MEMORY, which nothing else uses here: each thread reads its 128 words back with tcgen05.ld while the register half is multiplied
// (512 bytes per cycle and SM: half the time of the FFMAs).  Through L2 with 32 blocks per direction (lstm_persistent.cu) a step of
// 512 units took 1.60 / 1.43 us forward / backward, here 1.01 / 0.95 (256 units: 1.36 / 1.03 there, 0.84 / 0.80 here).
//
//   forward : warp w of 8 owns U/8 units x 4 gates (rows) of the block; a lane takes KP/32 source units of every row, a transposing
//             butterfly of shuffles leaves one row sum per lane group; the gates' activations run in different lanes, shuffles bring
//             them together, and the warp sends its h values to all blocks (one st.async per peer).  No block barrier in a step.
//   backward: thread t owns source unit t (and t + 256) and multiplies the block's 4U deltas, broadcast from shared memory, with its
//             weights: nothing to reduce.  Its partial error goes to the block that owns the unit, where warp 0 adds the partials in
//             rank order and runs the cells (lane = unit: coalesced accesses).  One block barrier per step.
// Buffers, waits and clusters as in lstm_cluster.cu: two buffers per exchange, bounded waits, clusters independent of each other.
#include <mutex>

#include "cluster.cuh"
#include "common.cuh"
#include "ptx.cuh"

namespace b2 {
namespace {

using namespace cluster;
using namespace ptx;

constexpr int NTHR = 256;
constexpr uint32_t TM_COLS = 256;     // two warps a lane quarter, 128 columns each

struct SingleArgs {
    LstmShape sh;
    LstmBuffers bf;
    const float *w;
    float *y;          // forward: block outputs (written)
    const float *dy;   // backward: output errors (read)
    int *status;
    int n_items;       // D * P: one sequence of one direction each
    int nclusters;
};

__device__ __forceinline__ void st_async_v2(uint32_t raddr, float x, float y, uint32_t rbar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(raddr), "f"(x), "f"(y), "r"(rbar)
                 : "memory");
}
__device__ __forceinline__ void st_async_f32(uint32_t raddr, float x, uint32_t rbar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(raddr), "f"(x), "r"(rbar) : "memory");
}
__device__ __forceinline__ float4 lds4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void tmem_st16(uint32_t t, const float (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(t),
                 "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]),
                 "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
                 : "memory");
}
// waits for this thread's tensor-memory loads; the registers pass through so that no use of them moves up
__device__ __forceinline__ void tmem_wait16(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}

extern __shared__ __align__(128) unsigned char sg_smem[];

// ---- forward -----------------------------------------------------------------------------------------------------------
template <int C, int U, bool TM>
__global__ void __launch_bounds__(NTHR, 1) lstm_fwd_single_kernel(SingleArgs a) {
    constexpr int KP = C * U, KL = KP / 32, UW = U / 8, R = 4 * UW, LPR = 32 / R;   // lanes that end up with one row
    constexpr int RR = TM ? R / 2 : R;                                              // rows in registers, the others in tensor memory
    static_assert(UW >= 1 && KL % 4 == 0 && (!TM || KL == 16), "geometry");
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ uint32_t tmem_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = lane / (4 * LPR), gate = (lane / LPR) & 3, base = unit * 4 * LPR;
    const uint32_t rank = cluster_ctarank(), hbuf = smem_u32(sg_smem);
    const int P = a.sh.P, T = a.sh.T, ls = a.sh.ls, els = a.sh.els, D = a.sh.D;
    const LstmOffsets off = lstm_offsets(a.sh.pls, ls, els);
    const int j = (int)rank * U + warp * UW + unit;
    auto bar = [&](unsigned e) { return smem_u32(&bars[e & 1u]); };
    if (threadIdx.x == 0) {
        mbar_init(bar(0), 1);
        mbar_init(bar(1), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (TM) {
        if (warp == 0) tmem_alloc(smem_u32(&tmem_s), TM_COLS);
        tc_fence_before();
    }
    cluster_sync_all();   // a peer's shared memory may be touched only once the peer runs
    uint32_t tm = 0;
    if constexpr (TM) {
        tc_fence_after();
        tm = tmem_s + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * 128);
    }
    const uint32_t peer = map_to_rank(hbuf, (uint32_t)(lane & (C - 1)));     // lane r < C sends to block r

    float w[RR][KL];
    int cur_d = -1;
    unsigned ev = 0;      // steps published so far
    bool ok = true;
    for (int item = (int)(blockIdx.x / C); item < a.n_items && ok; item += a.nclusters) {
        const int d = item % D, pg = item / D;
        if (d != cur_d) {
            // row = 4 * unit + gate of the warp's units; k = 128 i + 4 lane + c
            auto weight = [&](int row, int q) {
                const int jw = (int)rank * U + warp * UW + (row >> 2), k = 128 * (q >> 2) + 4 * lane + (q & 3);
                return (jw < els && k < els) ? __ldg(a.w + off.rec + ((size_t)(row & 3) * ls + (size_t)d * els + jw) * els + k) : 0.0f;
            };
#pragma unroll
            for (int row = 0; row < RR; ++row)
#pragma unroll
                for (int q = 0; q < KL; ++q) w[row][q] = weight(row, q);
            if constexpr (TM) {
#pragma unroll 1
                for (int row = RR; row < R; ++row) {
                    float v[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) v[q] = weight(row, q);
                    tmem_st16(tm + 16u * (uint32_t)(row - RR), v);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            cur_d = d;
        }
        const bool real = j < els;
        const int u = d * els + (real ? j : 0);
        const float bias = a.sh.bias * __ldg(a.w + off.bias + (size_t)gate * ls + u), p_og = __ldg(a.w + off.peep + (size_t)2 * ls + u);
        const float peep = gate == 1 || gate == 2 ? __ldg(a.w + off.peep + (size_t)(gate - 1) * ls + u) : 0.0f;
        const int Tc = sequence_length(a.sh, a.bf.pat, pg);
        const size_t fa = (size_t)4 * P * ls, fy = (size_t)P * ls;      // floats from a frame to the next
        float *acts = a.bf.acts + (size_t)pg * 4 * ls + (size_t)gate * ls + u;
        float cp = 0.0f, pre = 0.0f;
        auto fetch = [&](int s) {     // a step ahead, before the step waits
            const int sc = s < Tc ? s : Tc - 1;
            pre = acts[(size_t)(d ? Tc - 1 - sc : sc) * fa];
        };
        auto step = [&](int s) {
            const int t = d ? Tc - 1 - s : s;
            const bool publish = s + 1 < Tc;
            if (publish && threadIdx.x == 0) mbar_expect_tx(bar(ev), KP * 4u);
            float x = pre + bias;
            fetch(s + 1);
            if (s > 0) {
                uint32_t ta[16], tb[16];
                if constexpr (TM) tmem_ld16(tm, ta);
                ok = __all_sync(0xffffffffu, wait_bounded(bar(ev - 1), ((ev - 1) >> 1) & 1u, a.status));
                if (!ok) return;
                const uint32_t hb = hbuf + ((ev - 1) & 1u) * (KP * 4u) + 16u * (uint32_t)lane;
                float h[KL], v[R];
#pragma unroll
                for (int i = 0; i < KL / 4; ++i) {
                    const float4 q = lds4(hb + 512u * (uint32_t)i);
                    h[4 * i] = q.x; h[4 * i + 1] = q.y; h[4 * i + 2] = q.z; h[4 * i + 3] = q.w;
                }
#pragma unroll
                for (int row = 0; row < R; ++row) v[row] = 0.0f;
#pragma unroll
                for (int q = 0; q < KL; ++q)
#pragma unroll
                    for (int row = 0; row < RR; ++row) v[row] = fmaf(w[row][q], h[q], v[row]);
                if constexpr (TM) {
#pragma unroll
                    for (int row = RR; row < R; ++row) {
                        const bool odd = (row - RR) & 1;
                        if (odd) tmem_wait16(tb); else tmem_wait16(ta);
                        if (row + 1 < R) { if (odd) tmem_ld16(tm + 16u * (row + 1 - RR), ta); else tmem_ld16(tm + 16u * (row + 1 - RR), tb); }
                        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
                        for (int q = 0; q < 16; q += 2) {
                            s0 = fmaf(__uint_as_float(odd ? tb[q] : ta[q]), h[q], s0);
                            s1 = fmaf(__uint_as_float(odd ? tb[q + 1] : ta[q + 1]), h[q + 1], s1);
                        }
                        v[row] = s0 + s1;
                    }
                }
                // transposing butterfly: after log2(R) levels a lane holds one row, the rest adds the lanes of that row
                int o = 16;
#pragma unroll
                for (int half = R / 2; half >= 1; half /= 2, o /= 2) {
                    const bool up = lane & o;
#pragma unroll
                    for (int i = 0; i < half; ++i) {
                        const float keep = up ? v[half + i] : v[i], send = up ? v[i] : v[half + i];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
#pragma unroll
                for (; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
                x += v[0];
            }
            // gate 0 tanh, gates 1 and 2 logistic, each in the lanes of its row; gate 3 waits for the new cell state
            const float xp = fmaf(cp, peep, x);
            const float e = cl_exp(gate == 0 ? -2.0f * xp : -xp, gate == 0 ? 40.0f : 88.0f), r = cl_rcp(1.0f + e);
            float act = gate == 0 ? (1.0f - e) * r : r;
            const float ni = __shfl_sync(0xffffffffu, act, base), ig = __shfl_sync(0xffffffffu, act, base + LPR);
            const float fg = __shfl_sync(0xffffffffu, act, base + 2 * LPR), xo = __shfl_sync(0xffffffffu, x, base + 3 * LPR);
            float c = ni * ig + cp * fg;
            const float og = cl_logistic(fmaf(c, p_og, xo));
            float hh = cl_tanh(c) * og;
            if (!real) c = hh = 0.0f;
            if (publish) {
                const uint32_t dst = peer + (ev & 1u) * (KP * 4u) + (rank * U + (uint32_t)(warp * UW)) * 4u, rb = peer + (bar(ev) - hbuf);
                if constexpr (UW == 4) {
                    const float h0 = __shfl_sync(0xffffffffu, hh, 0), h1 = __shfl_sync(0xffffffffu, hh, 8);
                    const float h2 = __shfl_sync(0xffffffffu, hh, 16), h3 = __shfl_sync(0xffffffffu, hh, 24);
                    if (lane < C) st_async_v4(dst, __float_as_uint(h0), __float_as_uint(h1), __float_as_uint(h2), __float_as_uint(h3), rb);
                } else if constexpr (UW == 2) {
                    const float h0 = __shfl_sync(0xffffffffu, hh, 0), h1 = __shfl_sync(0xffffffffu, hh, 16);
                    if (lane < C) st_async_v2(dst, h0, h1, rb);
                } else {
                    if (lane < C) st_async_f32(dst, hh, rb);
                }
                ++ev;
            }
            cp = c;
            if (real) {       // the layer's own state, after h is on its way
                if (lane % LPR == 0) acts[(size_t)t * fa] = gate == 3 ? og : act;
                else if (lane % LPR == 1 && gate < 2) (gate ? a.y : a.bf.cells)[(size_t)t * fy + (size_t)pg * ls + u] = gate ? hh : c;
            }
        };
        if (Tc > 0) fetch(0);
#pragma unroll 1
        for (int s = 0; s < Tc && ok; ++s) step(s);
        if (real && lane % LPR == 1 && gate < 2)
            for (int t = Tc; t < T; ++t) (gate ? a.y : a.bf.cells)[(size_t)t * fy + (size_t)pg * ls + u] = 0.0f;
    }
    cluster_sync_all();   // nobody leaves while a peer may still write into its shared memory
    if constexpr (TM) {
        tc_fence_after();
        if (warp == 0) tmem_dealloc(tmem_s, TM_COLS);
    }
}

// ---- backward ------------------------------------------------------------------------------------------------------------
template <int C, int U, bool TM>
__global__ void __launch_bounds__(NTHR, 1) lstm_bwd_single_kernel(SingleArgs a) {
    constexpr int KP = C * U, ROWS = 4 * U;
    constexpr int KS = KP < NTHR ? NTHR / KP : 1;        // threads that share a source unit, each with ROWS / KS rows
    constexpr int RPT = ROWS / KS, SRC = C * KS;         // rows per thread; partials per unit
    constexpr int PARTS = 32 / U;                        // lanes of warp 0 that share a unit when the partials are added
    static_assert(U == 16 || U == 32, "warp 0 runs the cells");
    static_assert(TM == (KP == 2 * NTHR) && RPT % 16 == 0 && RPT <= 128, "geometry");
    constexpr uint32_t EBUF = SRC * U * 4u, DBUF = ROWS * 4u;
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ uint32_t tmem_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank(), ebuf = smem_u32(sg_smem), dbuf = ebuf + 2u * EBUF;
    const int P = a.sh.P, T = a.sh.T, ls = a.sh.ls, els = a.sh.els, D = a.sh.D;
    const LstmOffsets off = lstm_offsets(a.sh.pls, ls, els);
    auto bar = [&](unsigned e) { return smem_u32(&bars[e & 1u]); };
    if (tid == 0) {
        mbar_init(bar(0), 1);
        mbar_init(bar(1), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (TM) {
        if (warp == 0) tmem_alloc(smem_u32(&tmem_s), TM_COLS);
        tc_fence_before();
    }
    cluster_sync_all();
    uint32_t tm = 0;
    if constexpr (TM) {
        tc_fence_after();
        tm = tmem_s + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * 128);
    }
    const int k = tid % KP, part = KS > 1 ? tid / KP : 0;      // source unit (TM: also k + 256), which share of the rows
    const uint32_t place = ((rank * KS + (uint32_t)part) * U + (uint32_t)(k % U)) * 4u;
    const uint32_t peer0 = map_to_rank(ebuf, (uint32_t)(k / U)), peer1 = TM ? map_to_rank(ebuf, (uint32_t)((k + NTHR) / U)) : peer0;
    const int ul = lane % U, j = (int)rank * U + ul;           // warp 0: the lane's unit

    float w[RPT];
    int cur_d = -1;
    unsigned ev = 0;
    bool ok = true;
    for (int item = (int)(blockIdx.x / C); item < a.n_items && ok; item += a.nclusters) {
        const int d = item % D, pg = item / D;
        if (d != cur_d) {
            auto weight = [&](int row, int kk) {      // row = gate * U + unit of the block
                const int jw = (int)rank * U + row % U;
                return (jw < els && kk < els) ? __ldg(a.w + off.rec + ((size_t)(row / U) * ls + (size_t)d * els + jw) * els + kk) : 0.0f;
            };
#pragma unroll
            for (int r = 0; r < RPT; ++r) w[r] = weight(part * RPT + r, k);
            if constexpr (TM) {
#pragma unroll 1
                for (int r = 0; r < RPT; r += 16) {
                    float v[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) v[q] = weight(r + q, k + NTHR);
                    tmem_st16(tm + (uint32_t)r, v);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            cur_d = d;
        }
        const bool real = j < els;
        const int u = d * els + (real ? j : 0), Tc = sequence_length(a.sh, a.bf.pat, pg);
        const size_t fa = (size_t)4 * P * ls, fy = (size_t)P * ls, oa = (size_t)pg * 4 * ls + u, oy = (size_t)pg * ls + u;
        float pw[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) pw[q] = __ldg(a.w + off.peep + (size_t)q * ls + u);
        float in_e = 0, in_ni = 0, in_ig = 0, in_fg = 0, in_og = 0, in_cp = 0;
        float cc = 0.0f, st_fg = 0.0f, st_ce = 0.0f, st_dig = 0.0f, st_dfg = 0.0f;   // this frame's cell state; values of the step before
        auto fetch = [&](int s) {      // a step ahead, before the wait
            const int sc = s < Tc ? s : Tc - 1, t = d ? sc : Tc - 1 - sc, prev = sc == Tc - 1 ? t : (d ? t + 1 : t - 1);
            in_e = a.dy[(size_t)t * fy + oy];
            const float *ap = a.bf.acts + (size_t)t * fa + oa;
            in_ni = ap[0]; in_ig = ap[ls]; in_fg = ap[2 * (size_t)ls]; in_og = ap[3 * (size_t)ls];
            in_cp = a.bf.cells[(size_t)prev * fy + oy];
        };
        if (Tc > 0) {
            cc = a.bf.cells[(size_t)(d ? 0 : Tc - 1) * fy + oy];
            fetch(0);
        }
#pragma unroll 1
        for (int s = 0; s < Tc; ++s) {
            const int t = d ? s : Tc - 1 - s;
            const bool first = (s == 0), last = (s == Tc - 1);
            const uint32_t db = dbuf + (ev & 1u) * DBUF;
            float dd[4] = {0, 0, 0, 0};
            float e = in_e, cp = 0, fg = 0, k_og = 0, k_ce = 0, carry = 0, k_ni = 0, k_ig = 0, k_fg = 0;
            if (warp == 0) {
                if (!last && lane == 0) mbar_expect_tx(bar(ev), EBUF);
                const float nig = in_ni, ig = in_ig, og = in_og;
                fg = in_fg;
                cp = last ? 0.0f : in_cp;       // no previous cell state at the last step
                // the part of ComputeBlockErrorsFn that does not wait for the partial errors (see lstm_cluster.cu)
                const float tc = cl_tanh(cc);
                k_og = d_logistic(og) * tc;
                k_ce = og * d_tanh(tc);
                carry = st_fg * st_ce + pw[0] * st_dig + pw[1] * st_dfg;
                k_ni = ig * d_tanh(nig);
                k_ig = d_logistic(ig) * nig;
                k_fg = d_logistic(fg) * cp;
                settle(k_og, k_ce, carry, k_ni, k_ig, k_fg);
            }
            fetch(s + 1);      // by all warps: loads behind the branch would have to arrive where it ends
            if (warp == 0) {
                if (!first) {
                    ok = wait_bounded(bar(ev - 1), ((ev - 1) >> 1) & 1u, a.status);
                    const float *pe = reinterpret_cast<const float *>(sg_smem + ((ev - 1) & 1u) * EBUF) + (lane / U) * (SRC / PARTS) * U + ul;
                    float s4[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int q = 0; q < SRC / PARTS; ++q) s4[q & 3] += pe[q * U];
                    float sum = (s4[0] + s4[1]) + (s4[2] + s4[3]);
                    if (PARTS > 1) sum += __shfl_xor_sync(0xffffffffu, sum, 16);
                    e += sum;
                }
                const float dog = k_og * e;
                float ce = k_ce * e + pw[2] * dog + carry;
                dd[0] = limited_error(k_ni * ce); dd[1] = limited_error(k_ig * ce); dd[2] = limited_error(k_fg * ce); dd[3] = limited_error(dog);
                if (!real) ce = dd[0] = dd[1] = dd[2] = dd[3] = 0.0f;
                if (!last && lane < U) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) sts(db + (uint32_t)(q * U + ul) * 4u, dd[q]);
                }
                cc = cp;
                st_fg = fg; st_ce = ce; st_dig = dd[1]; st_dfg = dd[2];
            }
            if (!last) {
                uint32_t ta[16], tb[16];
                if constexpr (TM) tmem_ld16(tm, ta);
                if (__syncthreads_or(!ok)) { ok = false; break; }
                float acc[4] = {0, 0, 0, 0}, ac2[4] = {0, 0, 0, 0};
                const uint32_t dr = db + (uint32_t)(part * RPT) * 4u;
#pragma unroll
                for (int r = 0; r < RPT; r += 16) {
                    float4 q[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) q[i] = lds4(dr + (uint32_t)(r + 4 * i) * 4u);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        acc[0] = fmaf(w[r + 4 * i], q[i].x, acc[0]);
                        acc[1] = fmaf(w[r + 4 * i + 1], q[i].y, acc[1]);
                        acc[2] = fmaf(w[r + 4 * i + 2], q[i].z, acc[2]);
                        acc[3] = fmaf(w[r + 4 * i + 3], q[i].w, acc[3]);
                    }
                    if constexpr (TM) {
                        const bool odd = (r / 16) & 1;
                        if (odd) tmem_wait16(tb); else tmem_wait16(ta);
                        if (r + 16 < RPT) { if (odd) tmem_ld16(tm + (uint32_t)(r + 16), ta); else tmem_ld16(tm + (uint32_t)(r + 16), tb); }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            ac2[0] = fmaf(__uint_as_float(odd ? tb[4 * i] : ta[4 * i]), q[i].x, ac2[0]);
                            ac2[1] = fmaf(__uint_as_float(odd ? tb[4 * i + 1] : ta[4 * i + 1]), q[i].y, ac2[1]);
                            ac2[2] = fmaf(__uint_as_float(odd ? tb[4 * i + 2] : ta[4 * i + 2]), q[i].z, ac2[2]);
                            ac2[3] = fmaf(__uint_as_float(odd ? tb[4 * i + 3] : ta[4 * i + 3]), q[i].w, ac2[3]);
                        }
                    }
                }
                const uint32_t o = (ev & 1u) * EBUF + place, rb = bar(ev) - ebuf;
                st_async_f32(peer0 + o, (acc[0] + acc[1]) + (acc[2] + acc[3]), peer0 + rb);
                if constexpr (TM) st_async_f32(peer1 + o, (ac2[0] + ac2[1]) + (ac2[2] + ac2[3]), peer1 + rb);
                ++ev;
            }
            // the deltas go to memory after the partial errors have been sent
            if (warp == 0 && real && lane < U) {
                float *dl = a.bf.deltas + (size_t)t * fa + oa;
                dl[0] = dd[0]; dl[ls] = dd[1]; dl[2 * (size_t)ls] = dd[2]; dl[3 * (size_t)ls] = dd[3];
            }
        }
        ok = !__syncthreads_or(!ok);
        if (warp == 0 && real && lane < U)
            for (int t = Tc; t < T; ++t) {
                float *dl = a.bf.deltas + (size_t)t * fa + oa;
                dl[0] = 0.0f; dl[ls] = 0.0f; dl[2 * (size_t)ls] = 0.0f; dl[3 * (size_t)ls] = 0.0f;
            }
    }
    cluster_sync_all();
    if constexpr (TM) {
        tc_fence_after();
        if (warp == 0) tmem_dealloc(tmem_s, TM_COLS);
    }
}

// ---- host side -------------------------------------------------------------------------------------------------------------
typedef void (*Kernel)(SingleArgs);
struct Variant { int C, U; Kernel fwd, bwd; size_t smem_f, smem_b; };
template <int C, int U, bool TM>
constexpr Variant variant() {
    return Variant{C, U, lstm_fwd_single_kernel<C, U, TM>, lstm_bwd_single_kernel<C, U, TM>, (size_t)2 * C * U * 4,
                   (size_t)2 * ((size_t)C * (C * U < NTHR ? NTHR / (C * U) : 1) * U * 4 + (size_t)4 * U * 4)};
}
const Variant VARIANTS[] = {variant<8, 16, false>(), variant<16, 16, false>(), variant<16, 32, true>()};
constexpr int NVARIANTS = (int)(sizeof(VARIANTS) / sizeof(VARIANTS[0]));

// clusters of a variant that the current device holds at once with one block per SM (asked once per kernel and device)
int resident_clusters(bool backward, int vi) {
    static std::mutex mu;
    static short known[MAX_DEVICES][NVARIANTS][2];    // 0 = not asked yet, else clusters + 1
    const int dev = current_device();
    if (dev < 0) return 0;
    std::lock_guard<std::mutex> lk(mu);
    short &k = known[dev][vi][backward];
    if (!k) {
        const Variant &v = VARIANTS[vi];
        const Kernel f = backward ? v.bwd : v.fwd;
        const size_t spread = 120 * 1024;      // keeps a second block off the SM
        k = (short)(1 + (allow((const void *)f, spread, v.C) ? resident((const void *)f, Launch(v.C, NTHR, spread, v.C, false, nullptr)) : 0));
    }
    return k - 1;
}
int pick_variant(int els) {
    for (int vi = 0; vi < NVARIANTS; ++vi)
        if (VARIANTS[vi].C * VARIANTS[vi].U >= els) return vi;
    return -1;
}

}  // namespace

// Every (direction, sequence) needs a cluster of its own with one block per SM (7 clusters of 16, 15 of 8 on a B200); blocks that
// share an SM lose to the 8-column tiles of lstm_cluster.cu (128 units, 16 pairs: 0.73 us per step against 0.69).  Forward from 33
// units on (below, one block without an exchange is faster; 128 units 0.57 us a step, 512 units 1.01 against 1.33 of lstm_cluster.cu; at 256
// units this side of the line is the slower one, 0.84 against 0.75), backward from 129 on (128 units: 0.79 us against 0.72 of
// lstm_cluster.cu; 256 units 0.80 against 0.91, 512 units 0.95 against 1.91).
bool lstm_single_supported(const LstmShape &s, bool backward) {
    const int vi = pick_variant(s.els);
    return vi >= 0 && s.els > (backward ? 128 : 32) && s.D * s.P <= resident_clusters(backward, vi);
}

int lstm_single_sweep(bool backward, const LstmShape &s, const LstmBuffers &b, const float *w, float *y, const float *dy, int *status,
                      cudaStream_t st) {
    if (!lstm_single_supported(s, backward)) return 1;
    const Variant &v = VARIANTS[pick_variant(s.els)];
    SingleArgs a;
    a.sh = s; a.bf = b; a.w = w; a.y = y; a.dy = dy; a.status = status;
    a.n_items = a.nclusters = s.D * s.P;
    const Launch l(a.nclusters * v.C, NTHR, backward ? v.smem_b : v.smem_f, v.C, false, st);
    B2_CUDA(cudaLaunchKernelEx(&l.cfg, backward ? v.bwd : v.fwd, a));
    count_launch();
    return B2_OK;
}

}  // namespace b2
