// Persistent LSTM recurrence for up to 320 units per direction and any number of sequences: ONE launch runs a whole
// forward (or BPTT) sweep, each thread-block cluster keeps the recurrent weights of one direction in REGISTERS as
// tensor-core fragments and runs 8, 16 or 32 sequences through all timesteps.
//
// Replaces the reference's per-timestep loop of 4 cublasSgemm + 1 Thrust functor per direction
// (layers/LstmLayer.cu:1805-1858,1878-1927 forward with ComputeBlockOutputFn :57-185; :2115-2176,2195-2253 backward with
// ComputeBlockErrorsFn :237-405 of the reference).
//
// What bounds a step.  It is a chain: exchange between the blocks of a cluster (about 500 cycles for the first byte, then
// about one cycle per 16 bytes received, measured with a probe), recurrent product, cell math.  So the product has to be
// short for FEW sequences.  tcgen05 with the weights in shared memory costs 40-85 cycles per instruction whatever N is
// (lstm_ptc.cu); here the weights sit in the registers of the warps that own them, and a warp-level MMA of 16 x 16 weights
// with 8 sequences takes 8 cycles of its tensor core: 768 cycles per step for 256 units and 8 sequences on 8 SMs, against
// 2048 cycles of FFMA for the same product.  FFMA wins again at one or two sequences (lstm_persistent.cu).
//
// Decomposition.  Block b of a cluster of C owns U = 4*WN hidden units with all four gates; its WN warps own 4 units (16 gate
// rows, one m-tile) each.  Unit counts that do not fill C*U are padded with zero weights; the padding units' outputs are 0.
//   forward : a warp multiplies its 16 rows with ALL of h[t-1] (contraction over the C*U units, nothing to reduce across warps);
//             the accumulator layout puts the four gates of a (unit, sequence) cell into two adjacent lane groups, one
//             exchange by shuffle gives every lane one whole cell.  The lane computes it, and the warp packs its 4 units x 8
//             sequences as fp16 hi / lo words and stores them into every block's h buffer with st.async (16 bytes each, counted on
//             a transaction barrier).  No block barrier inside a step.
//   backward: the block's own gate deltas (4U x sequences, shared memory) times its weight slice transposed give partial
//             output errors of every unit; each partial goes to the block that owns the unit, which adds the C partials in rank order.
//
// Numerics.  fp32 values enter the tensor cores as two fp16 terms x*S = hi + lo*2^-11 (S a power of two: 2^14 for h, 2^15 for
// the deltas, which are clipped to [-1, 1], and 2^13 <= max|w|*S < 2^14 per warp tile for the weights), three products, fp32
// accumulation, the cross terms (which carry 2^-11) apart: 22 significant bits of each operand, the scheme of the large
// GEMMs.  The main products run in two chains of at most 10 MMAs.  Activations: expf and a reciprocal refined by one Newton step.
//
// Buffers.  A step's h (partial errors) goes into one of two buffers; a warp that sends step t has received all of step t-1,
// which every warp sent after it had read step t-2, so two buffers need no further hand-shake.  (Backward: the block
// barrier between the deltas and their product ties the warps of a block together; the deltas have two buffers as well.)
// Every wait is bounded; on expiry the thread records B2_ERR_STEP_TIMEOUT and all roles leave.  Clusters never wait for each
// other, so any number of them may be in flight or queued.
#include <mutex>

#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"

namespace b2 {
namespace {

using namespace ptx;

constexpr unsigned SPIN_LIMIT = 1u << 21;
constexpr float LO_SCALE = 2048.0f, LO_UNSCALE = 1.0f / 2048.0f;
constexpr float S_H = 16384.0f, S_D = 32768.0f;

struct ClusterArgs {
    LstmShape sh;
    LstmBuffers bf;
    const float *w;
    float *y;          // forward: block outputs (written)
    const float *dy;   // backward: output errors (read)
    int *status;
    int n_items;       // D * ceil(P / (8 * NT))
    int nclusters;
};

// logistic function with the reference's cut-offs (activation_functions/Logistic.cuh); 1 / d by the hardware approximation and one
// Newton step (r + r (1 - d r)), which is as exact as the division and has no branches
__device__ __forceinline__ float cl_logistic(float x) {
    const float lim = 88.722839f;
    const float d = 1.0f + expf(fminf(-x, 88.0f));
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    r = fmaf(r, fmaf(-d, r, 1.0f), r);
    r = x > -lim ? r : 0.0f;
    return x < lim ? r : 1.0f;
}
__device__ __forceinline__ float cl_tanh(float x) { return 2.0f * cl_logistic(2.0f * x) - 1.0f; }

__device__ __forceinline__ uint32_t split_pair(float x, float S) {   // fp16 hi in the low half, lo in the high half
    const float xs = x * S;
    const __half h = __float2half_rn(xs);
    const __half l = __float2half_rn((xs - __half2float(h)) * LO_SCALE);
    return (uint32_t)__half_as_ushort(h) | ((uint32_t)__half_as_ushort(l) << 16);
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t a0, const uint32_t a1, const uint32_t a2, const uint32_t a3,
                                         const uint32_t b0, const uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
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
        if ((it & 1023u) == 1023u && ld_relaxed_s32(status) != 0) return false;
    }
    atomicCAS(status, 0, (int)B2_ERR_STEP_TIMEOUT);
    return false;
}

// length of sequence pg: padding frames trail a sequence, as the data set writes them; frames below Tmin are real for all
__device__ __forceinline__ int sequence_length(const ClusterArgs &a, int pg) {
    const int P = a.sh.P, T = a.sh.T;
    if (pg >= P) return 0;
    int lo = a.sh.Tmin, hi = T;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a.bf.pat[(size_t)mid * P + pg] == PAT_NONE) hi = mid; else lo = mid + 1;
    }
    return lo;
}
__device__ __forceinline__ int warp_max(int v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// One fragment slot: the 8 fp32 weights of a lane for one 16 x 16 tile, turned in place into 4 registers of fp16 hi pairs and 4
// of lo pairs.  Returns 1 / S of the warp's tile set.
template <int N>
__device__ __forceinline__ float split_fragments(uint32_t (&f)[N][8]) {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = fabsf(__uint_as_float(f[i][e]));
            if (v < __int_as_float(0x7f800000)) m = fmaxf(m, v);   // NaN / Inf do not set the scale
        }
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    int e2 = 0;
    if (m > 0.0f) {
        e2 = 13 - ((int)(__float_as_uint(m) >> 23) - 127);
        e2 = e2 < -100 ? -100 : (e2 > 100 ? 100 : e2);
    }
    const float S = __int_as_float((127 + e2) << 23), inv = __int_as_float((127 - e2) << 23);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t p0 = split_pair(__uint_as_float(f[i][2 * q]), S), p1 = split_pair(__uint_as_float(f[i][2 * q + 1]), S);
            hi[q] = (p0 & 0xffffu) | (p1 << 16);
            lo[q] = (p0 >> 16) | (p1 & 0xffff0000u);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) { f[i][q] = hi[q]; f[i][4 + q] = lo[q]; }
    }
    return inv;
}

extern __shared__ __align__(128) unsigned char cl_smem[];

// h and the gate deltas lie in shared memory as [contraction index k][hi of 8 sequences | lo of 8 sequences], 16 bytes each; the two
// halves change places every other group of 4 rows, so that ldmatrix finds 8 consecutive rows in 8 different bank groups
__device__ __forceinline__ uint32_t row_off(int k, int half) { return (uint32_t)k * 32u + (uint32_t)((half ^ ((k >> 2) & 1)) * 16); }

// ---- forward -----------------------------------------------------------------------------------------------------------
template <int C, int WN, int NT>
__global__ void __launch_bounds__(32 * WN, 1) lstm_fwd_cluster_kernel(ClusterArgs a) {
    constexpr int U = 4 * WN, KP = C * U, KS = KP / 16;
    constexpr uint32_t TILE = KP * 32u, BUF = NT * TILE;
    __shared__ __align__(8) unsigned long long bars[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int uu = lane >> 3, n = 2 * tig + (g & 1);     // the cell this lane computes: unit uu of the warp's four, sequence n
    const uint32_t rank = cluster_ctarank(), hbuf = smem_u32(cl_smem);
    const int P = a.sh.P, T = a.sh.T, ls = a.sh.ls, els = a.sh.els, D = a.sh.D;
    const LstmOffsets off = lstm_offsets(a.sh.pls, ls, els);
    const int j = (int)rank * U + warp * 4 + uu;         // hidden unit of this lane's cell
    auto bar = [&](unsigned e) { return smem_u32(&bars[e & 1u]); };
    if (threadIdx.x == 0) {
        mbar_init(bar(0), 1);
        mbar_init(bar(1), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster_sync_all();   // a peer's shared memory may be touched only once the peer runs

    uint32_t wf[KS][8];
    float inv = 1.0f;
    int cur_d = -1;
    unsigned ev = 0;      // steps published so far
    bool ok = true;
    for (int item = (int)(blockIdx.x / C); item < a.n_items && ok; item += a.nclusters) {
        const int d = item % D, p0 = (item / D) * 8 * NT;
        if (d != cur_d) {
            // row r of the tile: unit r/2 mod 4, gate (r mod 2) + 2 * (r / 8), so that rows g and g + 8 are two gates of one unit
            const int jw = (int)rank * U + warp * 4 + (g >> 1);
            const float *w0 = a.w + off.rec + ((size_t)(g & 1) * ls + (size_t)d * els + jw) * els;
            const float *w1 = w0 + (size_t)2 * ls * els;
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int k = ks * 16 + 2 * tig + (e & 1) + ((e & 4) ? 8 : 0);
                    wf[ks][e] = (jw < els && k < els) ? __float_as_uint(__ldg(((e & 2) ? w1 : w0) + k)) : 0u;
                }
            inv = split_fragments<KS>(wf) * (1.0f / S_H);
            cur_d = d;
        }
        const int u = d * els + j;
        float b4[4] = {0, 0, 0, 0}, pw[3] = {0, 0, 0};
        if (j < els) {
#pragma unroll
            for (int q = 0; q < 4; ++q) b4[q] = a.sh.bias * __ldg(a.w + off.bias + (size_t)q * ls + u);
#pragma unroll
            for (int q = 0; q < 3; ++q) pw[q] = __ldg(a.w + off.peep + (size_t)q * ls + u);
        }
        int len[NT], Tc = 0;
        float cprev[NT], pre_n[NT][4];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            len[i] = sequence_length(a, p0 + 8 * i + n);
            Tc = max(Tc, len[i]);
            cprev[i] = 0.0f;
        }
        Tc = warp_max(Tc);    // the cluster's longest sequence: beyond it all frames are padding
        // what a step reads from HBM is independent of the recurrence and is fetched one step ahead
        auto fetch = [&](int s) {
            const int t = d ? Tc - 1 - s : s;
#pragma unroll
            for (int i = 0; i < NT; ++i) {
#pragma unroll
                for (int q = 0; q < 4; ++q) pre_n[i][q] = 0.0f;
                if (t < len[i] && j < els) {
                    const float *ap = a.bf.acts + ((size_t)t * P + p0 + 8 * i + n) * 4 * ls + u;
#pragma unroll
                    for (int q = 0; q < 4; ++q) pre_n[i][q] = ap[(size_t)q * ls];
                }
            }
        };
        const uint32_t ldsm_lane = (uint32_t)(((lane >> 3) & 1) * 8 + (lane & 7)) * 32u + (uint32_t)(((lane >> 4) ^ ((lane >> 2) & 1)) * 16);
        if (Tc > 0) fetch(0);
        for (int s = 0; s < Tc; ++s) {
            const int t = d ? Tc - 1 - s : s;
            const bool publish = s + 1 < Tc;
            float x[NT][4];
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) x[i][q] = pre_n[i][q] + b4[q];
            if (s + 1 < Tc) fetch(s + 1);
            if (publish && threadIdx.x == 0) mbar_expect_tx(bar(ev), BUF);
            if (s > 0) {
                ok = __all_sync(0xffffffffu, wait_bounded(bar(ev - 1), ((ev - 1) >> 1) & 1u, a.status));
                if (!ok) break;
                const uint32_t hb = hbuf + ((ev - 1) & 1u) * BUF + ldsm_lane;
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    float m0[4] = {0, 0, 0, 0}, m1[4] = {0, 0, 0, 0}, xa[4] = {0, 0, 0, 0}, xb[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) {
                        uint32_t b[4];
                        ldsm_x4_t(b, hb + (uint32_t)i * TILE + (uint32_t)ks * 512u);
                        const uint32_t *f = wf[ks];
                        mma16816(xa, f[4], f[5], f[6], f[7], b[0], b[1]);
                        mma16816((ks & 1) ? m1 : m0, f[0], f[1], f[2], f[3], b[0], b[1]);
                        mma16816(xb, f[0], f[1], f[2], f[3], b[2], b[3]);
                    }
                    float z[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) z[e] = ((m0[e] + m1[e]) + (xa[e] + xb[e]) * LO_UNSCALE) * inv;
                    // lanes with even g hold gates 0 and 2 of columns 2 tig and 2 tig + 1, their partners (lane ^ 4) gates 1 and 3
                    const bool odd = g & 1;
                    const float r0 = __shfl_xor_sync(0xffffffffu, odd ? z[0] : z[1], 4);
                    const float r1 = __shfl_xor_sync(0xffffffffu, odd ? z[2] : z[3], 4);
                    x[i][0] += odd ? r0 : z[0];
                    x[i][1] += odd ? z[1] : r0;
                    x[i][2] += odd ? r1 : z[2];
                    x[i][3] += odd ? z[3] : r1;
                }
            }
            float ni[NT], ig[NT], fg[NT], og[NT], hh[NT];
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const float cp = cprev[i];
                ni[i] = cl_tanh(x[i][0]);
                ig[i] = cl_logistic(x[i][1] + cp * pw[0]);
                fg[i] = cl_logistic(x[i][2] + cp * pw[1]);
                float c = ni[i] * ig[i] + cp * fg[i];
                og[i] = cl_logistic(x[i][3] + c * pw[2]);
                hh[i] = cl_tanh(c) * og[i];
                if (!(t < len[i] && j < els)) { ni[i] = ig[i] = fg[i] = og[i] = hh[i] = c = 0.0f; }   // padding frame or unit
                cprev[i] = c;
            }
            if (publish) {
                const int ch = lane & 7;     // chunk of 16 bytes: unit ch / 2 of the warp, hi or lo
                const int kk = (int)rank * U + warp * 4 + (ch >> 1);
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const uint32_t v = split_pair(hh[i], S_H);
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, v, 4);
                    const uint32_t word = (g & 1) ? ((o >> 16) | (v & 0xffff0000u)) : ((v & 0xffffu) | (o << 16));
                    uint32_t q4[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) q4[q] = __shfl_sync(0xffffffffu, word, 4 * ch + q);
                    const uint32_t la = hbuf + (ev & 1u) * BUF + (uint32_t)i * TILE + row_off(kk, ch & 1);
#pragma unroll
                    for (int r4 = 0; r4 < C / 4; ++r4) {
                        const uint32_t r = (uint32_t)(lane >> 3) + 4u * r4;
                        st_async_v4(map_to_rank(la, r), q4[0], q4[1], q4[2], q4[3], map_to_rank(bar(ev), r));
                    }
                }
                ++ev;
            }
            // the peers are waiting for h: the layer's own state goes to memory after it is on its way
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int pg = p0 + 8 * i + n;
                if (pg < P && j < els) {
                    const size_t f = (size_t)t * P + pg;
                    float *ap = a.bf.acts + f * 4 * ls + u;
                    ap[0] = ni[i]; ap[ls] = ig[i]; ap[2 * (size_t)ls] = fg[i]; ap[3 * (size_t)ls] = og[i];
                    a.bf.cells[f * ls + u] = cprev[i];
                    a.y[f * ls + u] = hh[i];
                }
            }
        }
        // frames beyond the cluster's longest sequence
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int pg = p0 + 8 * i + n;
            if (pg < P && j < els)
                for (int t = Tc; t < T; ++t) {
                    const size_t f = ((size_t)t * P + pg) * ls + u;
                    a.y[f] = 0.0f;
                    a.bf.cells[f] = 0.0f;
                }
        }
    }
    cluster_sync_all();   // nobody leaves while a peer may still write into its shared memory
}

// ---- backward ------------------------------------------------------------------------------------------------------------
template <int C, int WN, int NT>
__global__ void __launch_bounds__(32 * WN, 1) lstm_bwd_cluster_kernel(ClusterArgs a) {
    constexpr int U = 4 * WN, KP = C * U, MT = C / 4;     // MT m-tiles of 16 source units per warp
    constexpr uint32_t BUF = KP * 32u * NT;               // partial errors received per step: [source block][unit][8 * NT floats]
    constexpr uint32_t DTILE = 4u * U * 32u;              // the block's own deltas of 8 sequences
    __shared__ __align__(8) unsigned long long bars[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int uu = lane >> 3, n = 2 * tig + (g & 1);
    const uint32_t rank = cluster_ctarank(), ebuf = smem_u32(cl_smem), dbuf = ebuf + 2u * BUF;
    const int P = a.sh.P, T = a.sh.T, ls = a.sh.ls, els = a.sh.els, D = a.sh.D;
    const LstmOffsets off = lstm_offsets(a.sh.pls, ls, els);
    const int j = (int)rank * U + warp * 4 + uu;
    auto bar = [&](unsigned e) { return smem_u32(&bars[e & 1u]); };
    if (threadIdx.x == 0) {
        mbar_init(bar(0), 1);
        mbar_init(bar(1), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster_sync_all();

    uint32_t wf[MT * WN][8];
    float inv = 1.0f;
    int cur_d = -1;
    unsigned ev = 0;
    bool ok = true;
    for (int item = (int)(blockIdx.x / C); item < a.n_items && ok; item += a.nclusters) {
        const int d = item % D, p0 = (item / D) * 8 * NT;
        if (d != cur_d) {
            // rows: source units; contraction index 16 ks + 4 gate + unit: the block's own gate rows
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int ks = 0; ks < WN; ++ks)
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int src = (warp * MT + mt) * 16 + g + ((e & 2) ? 8 : 0);
                        const int pos = 2 * tig + (e & 1) + ((e & 4) ? 8 : 0);
                        const int jw = (int)rank * U + ks * 4 + (pos & 3);
                        wf[mt * WN + ks][e] = (jw < els && src < els)
                            ? __float_as_uint(__ldg(a.w + off.rec + ((size_t)(pos >> 2) * ls + (size_t)d * els + jw) * els + src)) : 0u;
                    }
            inv = split_fragments<MT * WN>(wf) * (1.0f / S_D);
            cur_d = d;
        }
        const int u = d * els + j;
        float pw[3] = {0, 0, 0};
        if (j < els)
#pragma unroll
            for (int q = 0; q < 3; ++q) pw[q] = __ldg(a.w + off.peep + (size_t)q * ls + u);
        int len[NT], Tc = 0;
        float st_ce[NT], st_dig[NT], st_dfg[NT], st_fg[NT], cc[NT];   // values of the step before; the cell state of this one
        float e_n[NT], a4_n[NT][4], cp_n[NT];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            len[i] = sequence_length(a, p0 + 8 * i + n);
            Tc = max(Tc, len[i]);
            st_ce[i] = st_dig[i] = st_dfg[i] = st_fg[i] = cc[i] = 0.0f;
        }
        Tc = warp_max(Tc);
        auto fetch = [&](int s) {
            const int t = d ? s : Tc - 1 - s, prev = d ? t + 1 : t - 1;
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int pg = p0 + 8 * i + n;
                e_n[i] = cp_n[i] = 0.0f;
#pragma unroll
                for (int q = 0; q < 4; ++q) a4_n[i][q] = 0.0f;
                if (j < els && pg < P) {
                    const size_t f = (size_t)t * P + pg;
                    if (t < len[i]) {
                        e_n[i] = a.dy[f * ls + u];
                        const float *ap = a.bf.acts + f * 4 * ls + u;
#pragma unroll
                        for (int q = 0; q < 4; ++q) a4_n[i][q] = ap[(size_t)q * ls];
                        if (s == 0) cc[i] = a.bf.cells[f * ls + u];
                    }
                    if (s != Tc - 1) cp_n[i] = a.bf.cells[((size_t)prev * P + pg) * ls + u];
                }
            }
        };
        const uint32_t ldsm_lane = (uint32_t)(((lane >> 3) & 1) * 8 + (lane & 7)) * 32u + (uint32_t)(((lane >> 4) ^ ((lane >> 2) & 1)) * 16);
        if (Tc > 0) fetch(0);
        for (int s = 0; s < Tc; ++s) {
            const int t = d ? s : Tc - 1 - s;
            const bool first = (s == 0), last = (s == Tc - 1);
            float e[NT], a4[NT][4], cp[NT], dd[NT][4];
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                e[i] = e_n[i];
                cp[i] = cp_n[i];
#pragma unroll
                for (int q = 0; q < 4; ++q) a4[i][q] = a4_n[i][q];
            }
            if (!last) fetch(s + 1);
            if (!last && threadIdx.x == 0) mbar_expect_tx(bar(ev), BUF);
            if (!first) {
                ok = wait_bounded(bar(ev - 1), ((ev - 1) >> 1) & 1u, a.status);
                const float *pe = reinterpret_cast<const float *>(cl_smem + ((ev - 1) & 1u) * BUF) + (size_t)(warp * 4 + uu) * NT * 8 + n;
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    float sum = 0.0f;
#pragma unroll
                    for (int src = 0; src < C; ++src) sum += pe[(src * U * NT + i) * 8];
                    e[i] += sum;
                }
            }
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const float nig = a4[i][0], ig = a4[i][1], fg = a4[i][2], og = a4[i][3];
                const float tc = cl_tanh(cc[i]);
                float dog = d_logistic(og) * tc * e[i];
                float ce = og * d_tanh(tc) * e[i] + pw[2] * dog;
                ce += st_fg[i] * st_ce[i] + pw[0] * st_dig[i] + pw[1] * st_dfg[i];    // zeros at the first step
                float dni = limited_error(ig * d_tanh(nig) * ce);
                float dfg = limited_error(d_logistic(fg) * cp[i] * ce);               // no previous cell state at the last step: cp = 0
                float dig = limited_error(d_logistic(ig) * nig * ce);
                dog = limited_error(dog);
                const bool real = t < len[i] && j < els;
                st_fg[i] = real ? fg : 0.0f;
                st_ce[i] = real ? ce : 0.0f;
                dd[i][0] = real ? dni : 0.0f; dd[i][1] = st_dig[i] = real ? dig : 0.0f;
                dd[i][2] = st_dfg[i] = real ? dfg : 0.0f; dd[i][3] = real ? dog : 0.0f;
                cc[i] = cp[i];          // the previous step's cell state is the next one's own
            }
            if (!last) {
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t v = split_pair(dd[i][q], S_D);
                        const int k = warp * 16 + q * 4 + uu;
                        const uint32_t o = dbuf + ((ev & 1u) * NT + (uint32_t)i) * DTILE + 2u * (uint32_t)n;
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(o + row_off(k, 0)), "h"((unsigned short)(v & 0xffffu)) : "memory");
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(o + row_off(k, 1)), "h"((unsigned short)(v >> 16)) : "memory");
                    }
                ok = !__syncthreads_or(!ok);
                if (!ok) break;
#pragma unroll 1
                for (int i = 0; i < NT; ++i) {
                    float m0[MT][4], xa[MT][4];
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int q = 0; q < 4; ++q) m0[mt][q] = xa[mt][q] = 0.0f;
#pragma unroll
                    for (int ks = 0; ks < WN; ++ks) {
                        uint32_t b[4];
                        ldsm_x4_t(b, dbuf + ((ev & 1u) * NT + (uint32_t)i) * DTILE + ldsm_lane + (uint32_t)ks * 512u);
#pragma unroll
                        for (int mt = 0; mt < MT; ++mt) {
                            const uint32_t *f = wf[mt * WN + ks];
                            mma16816(xa[mt], f[4], f[5], f[6], f[7], b[0], b[1]);
                            mma16816(m0[mt], f[0], f[1], f[2], f[3], b[0], b[1]);
                            mma16816(xa[mt], f[0], f[1], f[2], f[3], b[2], b[3]);
                        }
                    }
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        float v[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = (m0[mt][q] + xa[mt][q] * LO_UNSCALE) * inv;
                        // even tig takes row g, columns 4 (tig / 2) .. + 3, odd tig row g + 8
                        const bool odd = tig & 1;
                        const float r0 = __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[2], 1);
                        const float r1 = __shfl_xor_sync(0xffffffffu, odd ? v[1] : v[3], 1);
                        const int src = (warp * MT + mt) * 16 + g + (odd ? 8 : 0);
                        const uint32_t owner = (uint32_t)(src / U), ul = (uint32_t)(src % U);
                        const uint32_t la = ebuf + (ev & 1u) * BUF + (((rank * U + ul) * NT + (uint32_t)i) * 8u + 4u * (uint32_t)(tig >> 1)) * 4u;
                        if (odd)
                            st_async_v4(map_to_rank(la, owner), __float_as_uint(r0), __float_as_uint(r1), __float_as_uint(v[2]),
                                        __float_as_uint(v[3]), map_to_rank(bar(ev), owner));
                        else
                            st_async_v4(map_to_rank(la, owner), __float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(r0),
                                        __float_as_uint(r1), map_to_rank(bar(ev), owner));
                    }
                }
                ++ev;
            }
            // the deltas go to memory after the partial errors the peers wait for have been sent
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int pg = p0 + 8 * i + n;
                if (pg < P && j < els) {
                    float *dl = a.bf.deltas + ((size_t)t * P + pg) * 4 * ls + u;
#pragma unroll
                    for (int q = 0; q < 4; ++q) dl[(size_t)q * ls] = dd[i][q];
                }
            }
        }
        ok = !__syncthreads_or(!ok);
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int pg = p0 + 8 * i + n;
            if (pg < P && j < els)
                for (int t = Tc; t < T; ++t) {
                    float *dl = a.bf.deltas + ((size_t)t * P + pg) * 4 * ls + u;
#pragma unroll
                    for (int q = 0; q < 4; ++q) dl[(size_t)q * ls] = 0.0f;
                }
        }
    }
    cluster_sync_all();
}

// ---- host side ---------------------------------------------------------------------------------------------------------------
typedef void (*Kernel)(ClusterArgs);
struct Variant { int C, WN, NT; Kernel fwd, bwd; };
template <int C, int WN, int NT>
constexpr Variant variant() { return Variant{C, WN, NT, lstm_fwd_cluster_kernel<C, WN, NT>, lstm_bwd_cluster_kernel<C, WN, NT>}; }
#define VARIANTS_OF(C, WN) variant<C, WN, 1>(), variant<C, WN, 2>(), variant<C, WN, 4>()
const Variant VARIANTS[] = {VARIANTS_OF(4, 2), VARIANTS_OF(4, 4), VARIANTS_OF(4, 6), VARIANTS_OF(4, 8), VARIANTS_OF(8, 4), VARIANTS_OF(8, 5),
                            VARIANTS_OF(8, 6), VARIANTS_OF(8, 7), VARIANTS_OF(8, 8), VARIANTS_OF(16, 2), VARIANTS_OF(16, 4),
                            variant<16, 5, 1>(), variant<16, 5, 2>()};
constexpr int NVARIANTS = (int)(sizeof(VARIANTS) / sizeof(VARIANTS[0]));

size_t smem_bytes(const Variant &v, bool backward) {
    const size_t buf = (size_t)v.C * 4 * v.WN * 32 * v.NT;
    return 2 * buf + (backward ? (size_t)2 * v.NT * 16 * v.WN * 32 : 0);
}

void launch_config(const Variant &v, bool backward, int clusters, cudaStream_t st, cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = v.C; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(clusters * v.C);
    cfg->blockDim = dim3(32 * v.WN);
    cfg->dynamicSmemBytes = smem_bytes(v, backward);
    cfg->stream = st;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

// clusters of a variant the current device holds at once (asked once per kernel and device)
int resident_clusters(int vi, bool backward) {
    static std::mutex mu;
    static int known[MAX_DEVICES][NVARIANTS][2];    // 0 = not asked yet, else clusters + 1
    const int dev = current_device();
    if (dev < 0) return 0;
    std::lock_guard<std::mutex> lk(mu);
    int &k = known[dev][vi][backward];
    if (!k) {
        const Variant &v = VARIANTS[vi];
        const Kernel f = backward ? v.bwd : v.fwd;
        int n = 0;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        launch_config(v, backward, 1, nullptr, &cfg, attr);
        if (cudaFuncSetAttribute((const void *)f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(v, backward)) != cudaSuccess ||
            (v.C > 8 && cudaFuncSetAttribute((const void *)f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
            cudaOccupancyMaxActiveClusters(&n, f, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        k = n + 1;
    }
    return k - 1;
}

// Cycles per step as measured with probes and sweeps: 900 for the chain (first byte of the exchange, gate math), 1 (cluster of
// 16: 1.2) per 16 bytes a block receives, 8 per MMA of an SM quarter; blocks that share an SM share its tensor cores and network port.
int pick_variant(const LstmShape &s, bool backward) {
    int best = -1;
    double best_t = 0.0;
    for (int vi = 0; vi < NVARIANTS; ++vi) {
        const Variant &v = VARIANTS[vi];
        const int KP = v.C * 4 * v.WN;
        if (KP < s.els) continue;
        const int res = resident_clusters(vi, backward);
        if (res < 1) continue;
        const int items = s.D * ((s.P + 8 * v.NT - 1) / (8 * v.NT));
        const int passes = (items + res - 1) / res, live = items < res ? items : res;
        const int share = (live * v.C + sm_count() - 1) / sm_count();
        const double step = 900.0 + 60.0 * v.NT + share * v.NT * ((v.C > 8 ? 1.2 : 1.0) * KP * 2 + (KP / 16) * 24.0 * ((v.WN + 3) / 4));
        const double t = passes * step * (1.0 + 1e-4 * live * v.C / sm_count());    // the smaller launch where two are equal
        if (best < 0 || t < best_t) { best = vi; best_t = t; }
    }
    return best;
}

}  // namespace

bool lstm_cluster_supported(const LstmShape &s) { return s.els <= 320 && pick_variant(s, false) >= 0 && pick_variant(s, true) >= 0; }

int lstm_cluster_sweep(bool backward, const LstmShape &s, const LstmBuffers &b, const float *w, float *y, const float *dy, int *status,
                       cudaStream_t st) {
    const int vi = pick_variant(s, backward);
    if (vi < 0) return 1;
    const Variant &v = VARIANTS[vi];
    ClusterArgs a;
    a.sh = s; a.bf = b; a.w = w; a.y = y; a.dy = dy; a.status = status;
    a.n_items = s.D * ((s.P + 8 * v.NT - 1) / (8 * v.NT));
    const int res = resident_clusters(vi, backward);
    a.nclusters = a.n_items < res ? a.n_items : res;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    launch_config(v, backward, a.nclusters, st, &cfg, attr);
    B2_CUDA(cudaLaunchKernelEx(&cfg, backward ? v.bwd : v.fwd, a));
    count_launch();
    return B2_OK;
}

}  // namespace b2
