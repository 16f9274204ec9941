// Persistent LSTM recurrence for up to 512 units per direction and any number of sequences: ONE launch runs a whole
// forward (or BPTT) sweep; each thread-block cluster keeps the recurrent weights of one direction in REGISTERS as
// tensor-core fragments (above 320 units the lo parts in TENSOR MEMORY) and runs tiles of 8 sequences through all timesteps.
//
// Replaces the reference's per-timestep loop of 4 cublasSgemm + 1 Thrust functor per direction
// (layers/LstmLayer.cu:1805-1858,1878-1927 forward with ComputeBlockOutputFn :57-185; :2115-2176,2195-2253 backward with
// ComputeBlockErrorsFn :237-405 of the reference).
//
// What bounds a step.  It is a chain: exchange between the blocks of a cluster (450 cycles for one 16-byte st.async to be seen by
// its receiver, then about a cycle per 16 bytes a block receives: measured with probes), recurrent product, cell math.  The
// product has to be short for FEW sequences.  tcgen05 with the weights in shared memory costs 40-85 cycles per instruction
// whatever N is (lstm_ptc.cu); here the weights sit in the registers of the warps that own them, and a warp-level MMA of 16 x 16
// weights with 8 sequences takes 8 cycles of its tensor core: 256 units, 8 sequences on 8 SMs are 768 cycles, against 2048 of FFMA.
// Measured (B200, us per step forward / backward, against the FFMA kernels of lstm_persistent.cu or, for unit counts those do not
// have, one launch per step): 256 units per direction, 32 sequences 1.17 / 1.18 (1.74 / 1.56), 4 sequences 0.75 / 0.91 (1.74 / 1.40),
// 128 sequences 3.6 / 3.6 (6.0 / 5.8); 128 units, 16 sequences 0.68 / 0.74; 160 units, 8 sequences 0.94 / 0.94 (20 / 57); a sweep
// takes 5 to 30 us besides (launch, weights).  ncu, 256 units, 32 sequences: tensor pipe 32 % of the cycles, DRAM 0.36 TB/s.
//
// Decomposition.  Block b of a cluster of C owns U = 4*WN hidden units with all four gates; its WN warps own 4 units (16 gate
// rows, one m-tile) each.  Unit counts that do not fill C*U are padded with zero weights; the padding units' outputs are 0.
//   forward : a warp multiplies its 16 rows with ALL of h[t-1] (contraction over the C*U units, nothing to reduce across warps);
//             the accumulator layout puts the four gates of a (unit, sequence) cell into two adjacent lane groups, one
//             exchange by shuffle gives every lane one whole cell.  The lane computes it, and the warp packs its 4 units x 8
//             sequences as fp16 hi / lo words and stores them into every block's h buffer with st.async (16 bytes each, counted on
//             a transaction barrier).  No block barrier inside a step.
//   backward: the block's own gate deltas (4U x 8, shared memory) times its weight slice transposed give partial output
//             errors of every unit; each partial goes to the block that owns the unit, which adds the C partials in a fixed order.
// Up to 32 units one block does it alone (C = 1): plain shared memory and block barriers take the place of the exchange.
//
// Above 320 units (TM): a block's 65536 weights are twice the register file.  The fp16 hi parts stay in registers, the lo parts in tensor
// memory, from where a warp reads the fragments of four k-steps while it multiplies those before.  Here the product (1536 cycles of
// the tensor cores a tile) is long enough for a second tile to hide the exchange: 512 units, 32 sequences 3.2 / 3.9 us (4.1 / 4.9 with
// lstm_ptc.cu), one direction of 50 sequences 2.0 / 2.0 (4.1 / 4.9), 384 units and 8 sequences 1.4 / 1.6 (38 / 125, a launch per step).
//
// Tried and dropped: several tiles per cluster in turn where all weights are in registers (the second tile costs as much as the first:
// a warp's own instruction stream, not the exchange, is what fills its time); inputs through a cp.async ring (0.13 us per step more than plain loads).
//
// Numerics.  fp32 values enter the tensor cores as two fp16 terms x*S = hi + lo*2^-11 (S a power of two: 2^14 for h, 2^15 for
// the deltas, which are clipped to [-1, 1], and 2^13 <= max|w|*S < 2^14 per warp for the weights), three products, fp32
// accumulation, the cross terms (which carry 2^-11) apart: 22 significant bits of each operand, the scheme of the large
// GEMMs.  The main products run in two chains of at most 10 MMAs.  Against float64 the outputs and gradients are as close as the
// FFMA kernels' (relative L2 2.5e-7 / 2.7e-7 against 4.8e-7 / 2.8e-7 at 256 units).
//
// Buffers.  A step's h (partial errors) goes into one of two buffers; a warp that sends step t has received all of step t-1,
// which every warp sent after it had read step t-2, so two buffers need no further hand-shake.  (Backward: the block
// barrier between the deltas and their product ties the warps of a block together; the deltas have two buffers as well.)
// Every wait is bounded; on expiry the thread records B2_ERR_STEP_TIMEOUT and all warps leave.  Clusters never wait for each
// other, so any number of them may be in flight or queued.
#include <mutex>

#include "cluster.cuh"
#include "common.cuh"
#include "ptx.cuh"

namespace b2 {
namespace {

using namespace cluster;
using namespace ptx;

constexpr int MAX_NT = 4;            // tiles a cluster runs in turn at most (kernels with weights in tensor memory)
constexpr uint32_t TM_COLS = 256;    // tensor-memory columns for the lo parts: two warps a lane quarter, 128 columns each

struct ClusterArgs {
    LstmShape sh;
    LstmBuffers bf;
    const float *w;
    float *y;          // forward: block outputs (written)
    const float *dy;   // backward: output errors (read)
    int *status;
    int tiles;         // ceil(P / 8)
    int nt;            // tiles per work item
    int n_items;       // D * ceil(tiles / nt): a work item is nt tiles of 8 sequences of one direction
    int nclusters;
};

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
__device__ __forceinline__ int warp_max(int v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The weight fragments of a warp: N slots of 16 x 16 weights, 8 per lane, of which weight(i, e) returns entry e of slot i.  Every
// slot becomes 4 registers of fp16 hi pairs and 4 of lo pairs; the lo parts stay in registers too, or (TM) go to tensor memory, which
// holds them as long as the kernel runs: 4 columns per slot from `tmem` on.  Returns 1 / S of the warp.
template <int N, bool TM, class Weight>
__device__ __forceinline__ float load_fragments(uint32_t (&hi)[N][4], uint32_t (&lo)[TM ? 1 : N][4], uint32_t tmem, Weight weight) {
    float m = 0.0f;
#pragma unroll 4
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = fabsf(weight(i, e));
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
        uint32_t l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t p0 = split_pair(weight(i, 2 * q), S), p1 = split_pair(weight(i, 2 * q + 1), S);
            hi[i][q] = (p0 & 0xffffu) | (p1 << 16);
            l[q] = (p0 >> 16) | (p1 & 0xffff0000u);
        }
        if constexpr (TM) {
            asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tmem + 4u * i), "r"(l[0]), "r"(l[1]), "r"(l[2]),
                         "r"(l[3])
                         : "memory");
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) lo[i][q] = l[q];
        }
    }
    if constexpr (TM) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    return inv;
}
// 4 slots of lo parts from tensor memory; they may be used after frag_wait on the same registers
__device__ __forceinline__ void frag_load(uint32_t (&r)[16], uint32_t tmem) { tmem_ld16(tmem, r); }
__device__ __forceinline__ void frag_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}
// 4 sequences: columns 0-3 of the 8 an MMA has carry the hi parts, columns 4-7 (lane ^ 2) the lo parts.  m and x are this lane's
// products with the weights' hi and lo parts; valid in the lanes of columns 0-3
__device__ __forceinline__ float join_half(float m, float x) {
    const float cross = __shfl_xor_sync(0xffffffffu, fmaf(x, LO_UNSCALE, m), 2);
    return fmaf(x + cross, LO_UNSCALE, m);
}

extern __shared__ __align__(128) unsigned char cl_smem[];

// h and the gate deltas lie in shared memory as [contraction index k][hi of 8 sequences | lo of 8 sequences], 16 bytes each; the two
// halves change places every other group of 4 rows, so that ldmatrix finds 8 consecutive rows in 8 different bank groups
__device__ __forceinline__ uint32_t row_off(int k, int half) { return (uint32_t)k * 32u + (uint32_t)((half ^ ((k >> 2) & 1)) * 16); }

// hi and lo of one value into rows of 8 sequences; addr: the tile, plus two bytes per sequence
__device__ __forceinline__ void st_shared_parts(uint32_t addr, int k, uint32_t parts) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr + row_off(k, 0)), "h"((unsigned short)(parts & 0xffffu)) : "memory");
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr + row_off(k, 1)), "h"((unsigned short)(parts >> 16)) : "memory");
}

// ---- forward -----------------------------------------------------------------------------------------------------------
// HALF: at most 4 sequences; columns 0-3 of the tile carry the hi parts, columns 4-7 the lo parts: two MMAs per 16 x 16
// weights instead of three and half the bytes to exchange
// TM: the lo parts of the weights live in tensor memory and a cluster runs a.nt tiles in turn, whose state is in shared memory
template <int C, int WN, bool HALF, bool TM>
constexpr size_t fwd_smem(int nt) { return (size_t)2 * nt * C * 4 * WN * (HALF ? 16 : 32) + (TM ? (size_t)nt * 2 * 32 * WN * 4 : 0); }
template <int C, int WN, bool HALF, bool TM>
__global__ void __launch_bounds__(32 * WN, 1) lstm_fwd_cluster_kernel(ClusterArgs a) {
    constexpr int U = 4 * WN, KP = C * U, KS = KP / 16;
    constexpr uint32_t TILE = KP * (HALF ? 16u : 32u);
    __shared__ __align__(8) unsigned long long bars[TM ? MAX_NT : 1][2];
    __shared__ uint32_t tmem_s;
    const int nt = TM ? a.nt : 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    // the cell this lane computes: unit uu of the warp's four, sequence n (HALF: the lanes with tig < 2)
    const int uu = lane >> 3, n = 2 * (HALF ? tig & 1 : tig) + (g & 1);
    const bool owner = !HALF || tig < 2;
    const uint32_t rank = cluster_ctarank(), hbuf = smem_u32(cl_smem), state = hbuf + 2u * nt * TILE + 4u * threadIdx.x;
    const int P = a.sh.P, T = a.sh.T, ls = a.sh.ls, els = a.sh.els, D = a.sh.D;
    const LstmOffsets off = lstm_offsets(a.sh.pls, ls, els);
    const int j = (int)rank * U + warp * 4 + uu;         // hidden unit of this lane's cell
    auto bar = [&](int i, unsigned e) { return smem_u32(&bars[i][e & 1u]); };
    if (threadIdx.x == 0) {
        for (int i = 0; i < nt; ++i) { mbar_init(bar(i, 0), 1); mbar_init(bar(i, 1), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (TM) {
        if (warp == 0) tmem_alloc(smem_u32(&tmem_s), TM_COLS);
        tc_fence_before();
    }
    if constexpr (C > 1) cluster_sync_all();   // a peer's shared memory may be touched only once the peer runs
    else __syncthreads();
    uint32_t tm = 0;                           // this warp's lo fragments: its lane quarter, the columns of its half of the warps
    if constexpr (TM) {
        tc_fence_after();
        tm = tmem_s + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * KS * 4);
    }

    // peers this lane sends to: C / PEERS of them (shared-memory addresses of a peer are linear)
    constexpr int PEERS = HALF ? 8 : 4, NP = C > 1 ? (C + PEERS - 1) / PEERS : 1;
    uint32_t peer[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) peer[q] = C > 1 ? map_to_rank(hbuf, (uint32_t)((HALF ? lane >> 2 : lane >> 3) + PEERS * q) & (C - 1)) : hbuf;

    uint32_t whi[KS][4], wlo[TM ? 1 : KS][4];
    float inv = 1.0f;
    int cur_d = -1;
    unsigned ev = 0;      // steps published so far
    bool ok = true;
    // ldmatrix rows of this lane: hi and lo of one k-step, or (HALF) two k-steps
    const uint32_t ldsm_lane = HALF ? (uint32_t)lane * 16u
        : (uint32_t)(((lane >> 3) & 1) * 8 + (lane & 7)) * 32u + (uint32_t)(((lane >> 4) ^ ((lane >> 2) & 1)) * 16);
    for (int item = (int)(blockIdx.x / C); item < a.n_items && ok; item += a.nclusters) {
        const int d = item % D, tile0 = (item / D) * nt, ntr = TM ? min(nt, a.tiles - tile0) : 1;
        if (d != cur_d) {
            // row r of the tile: unit r/2 mod 4, gate (r mod 2) + 2 * (r / 8), so that rows g and g + 8 are two gates of one unit
            const int jw = (int)rank * U + warp * 4 + (g >> 1);
            const float *w0 = a.w + off.rec + ((size_t)(g & 1) * ls + (size_t)d * els + jw) * els;
            const float *w1 = w0 + (size_t)2 * ls * els;
            inv = load_fragments<KS, TM>(whi, wlo, tm, [&](int ks, int e) {
                const int k = ks * 16 + 2 * tig + (e & 1) + ((e & 4) ? 8 : 0);
                return (jw < els && k < els) ? __ldg(((e & 2) ? w1 : w0) + k) : 0.0f;
            }) * (1.0f / S_H);
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
        const bool unit = j < els;
        // per tile: sequence length and cell state of this lane's cell
        int len = 0, Tc = 0;
        float cp = 0.0f, pre[4];
        for (int i = 0; i < ntr; ++i) {
            len = sequence_length(a.sh, a.bf.pat, (tile0 + i) * 8 + n);
            if (TM) { sts(state + (uint32_t)(2 * i) * (128u * WN), __int_as_float(len)); sts(state + (uint32_t)(2 * i + 1) * (128u * WN), 0.0f); }
            Tc = max(Tc, len);
        }
        Tc = warp_max(Tc);   // beyond the longest sequence all frames are padding
        // Frame t of this lane's cell: uniform base of the frame's row plus 32-bit offsets that stay the same.  Loads are
        // unconditional (a value behind a branch would have to arrive before the branches join): cells that do not exist read
        // the offsets of one that does.
        const uint32_t uc = (uint32_t)(d * els + (unit ? j : 0)), of_g = (uint32_t)ls * 4u;
        const uint32_t of_y = ((uint32_t)n * ls + uc) * 4u, of_a = ((uint32_t)n * 4u * ls + uc) * 4u, of_a0 = uc * 4u;
        // pre-activations are independent of the recurrence and fetched a tile-step ahead, BEFORE the step waits for its peers:
        // behind the step's stores the same loads cost 0.2 us per step
        auto fetch = [&](int s, int i) {
            const int sc = s < Tc ? s : Tc - 1, t = d ? Tc - 1 - sc : sc, row0 = (tile0 + i) * 8;
            const char *ap = reinterpret_cast<const char *>(a.bf.acts + ((size_t)t * P + row0) * 4 * ls);
            const uint32_t o = row0 + n < P ? of_a : of_a0;
#pragma unroll
            for (int q = 0; q < 4; ++q) pre[q] = *reinterpret_cast<const float *>(ap + (o + (uint32_t)q * of_g));
        };
        auto step = [&](int s, int i) {
                const int t = d ? Tc - 1 - s : s, row0 = (tile0 + i) * 8;
                const uint32_t st = state + (uint32_t)(2 * i) * (128u * WN);
                if (TM) { len = __float_as_int(lds(st)); cp = lds(st + 128u * WN); }
                const bool publish = s + 1 < Tc, real = t < len && unit, mine = unit && owner && row0 + n < P;
                if (C > 1 && publish && threadIdx.x == 0) mbar_expect_tx(bar(i, ev), TILE);
                float x[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) x[q] = pre[q] + b4[q];
                if (TM && i + 1 < ntr) fetch(s, i + 1); else fetch(s + 1, 0);
                uint32_t la[TM ? 16 : 1] = {}, lb[TM ? 16 : 1] = {};
                if (s > 0) {
                    if constexpr (TM) frag_load(la, tm);
                    if constexpr (C > 1) {
                        ok = __all_sync(0xffffffffu, wait_bounded(bar(i, ev - 1), ((ev - 1) >> 1) & 1u, a.status));
                        if (!ok) return;
                    } else {
                        __syncthreads();
                    }
                    const uint32_t hb = hbuf + (((ev - 1) & 1u) * nt + (uint32_t)i) * TILE + ldsm_lane;
                    float m0[4] = {0, 0, 0, 0}, m1[4] = {0, 0, 0, 0}, xa[4] = {0, 0, 0, 0}, xb[4] = {0, 0, 0, 0};
                    float z[4];
                    // lo parts of four k-steps are on their way from tensor memory while those before are in use
                    auto lo_of = [&](int ks, int q) { if constexpr (TM) return (ks & 4) ? lb[(ks & 3) * 4 + q] : la[(ks & 3) * 4 + q]; else return wlo[ks][q]; };
                    auto stage = [&](int ks) {
                        if constexpr (TM) {
                            if (ks & 4) { frag_wait(lb); if (ks + 4 < KS) frag_load(la, tm + 4u * (ks + 4)); }
                            else { frag_wait(la); if (ks + 4 < KS) frag_load(lb, tm + 4u * (ks + 4)); }
                        }
                    };
                    if constexpr (HALF) {
#pragma unroll
                        for (int ks = 0; ks < KS; ks += 2) {
                            if ((ks & 3) == 0) stage(ks);
                            uint32_t b[4];
                            ldsm_x4_t(b, hb + (uint32_t)ks * 256u);
                            mma16816(m0, whi[ks][0], whi[ks][1], whi[ks][2], whi[ks][3], b[0], b[1]);
                            mma16816(xa, lo_of(ks, 0), lo_of(ks, 1), lo_of(ks, 2), lo_of(ks, 3), b[0], b[1]);
                            mma16816(m1, whi[ks + 1][0], whi[ks + 1][1], whi[ks + 1][2], whi[ks + 1][3], b[2], b[3]);
                            mma16816(xb, lo_of(ks + 1, 0), lo_of(ks + 1, 1), lo_of(ks + 1, 2), lo_of(ks + 1, 3), b[2], b[3]);
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) z[e] = join_half(m0[e] + m1[e], xa[e] + xb[e]) * inv;
                    } else {
#pragma unroll
                        for (int ks = 0; ks < KS; ++ks) {
                            if ((ks & 3) == 0) stage(ks);
                            uint32_t b[4];
                            ldsm_x4_t(b, hb + (uint32_t)ks * 512u);
                            const uint32_t *f = whi[ks];
                            mma16816(xa, lo_of(ks, 0), lo_of(ks, 1), lo_of(ks, 2), lo_of(ks, 3), b[0], b[1]);
                            mma16816((ks & 1) ? m1 : m0, f[0], f[1], f[2], f[3], b[0], b[1]);
                            mma16816(xb, f[0], f[1], f[2], f[3], b[2], b[3]);
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) z[e] = ((m0[e] + m1[e]) + (xa[e] + xb[e]) * LO_UNSCALE) * inv;
                    }
                    // lanes with even g hold gates 0 and 2 of columns 2 tig and 2 tig + 1, their partners (lane ^ 4) gates 1 and 3
                    const bool odd = g & 1;
                    const float r0 = __shfl_xor_sync(0xffffffffu, odd ? z[0] : z[1], 4);
                    const float r1 = __shfl_xor_sync(0xffffffffu, odd ? z[2] : z[3], 4);
                    x[0] += odd ? r0 : z[0];
                    x[1] += odd ? z[1] : r0;
                    x[2] += odd ? r1 : z[2];
                    x[3] += odd ? z[3] : r1;
                }
                float ni = cl_tanh(x[0]), ig = cl_logistic(x[1] + cp * pw[0]), fg = cl_logistic(x[2] + cp * pw[1]);
                float c = ni * ig + cp * fg;
                float og = cl_logistic(x[3] + c * pw[2]);
                float hh = cl_tanh(c) * og;
                if (!real) { ni = ig = fg = og = hh = c = 0.0f; }   // padding frame or unit
                if (publish) {
                    const uint32_t v = split_pair(hh, S_H);
                    const uint32_t hd = hbuf + ((ev & 1u) * nt + (uint32_t)i) * TILE;
                    if constexpr (C > 1) {
                        // chunks of 16 bytes: hi or lo of 8 sequences of a unit (HALF: hi and lo of 4)
                        const int ch = HALF ? lane & 3 : lane & 7, kk = (int)rank * U + warp * 4 + (HALF ? ch : ch >> 1);
                        const uint32_t o = __shfl_xor_sync(0xffffffffu, v, 4);
                        const uint32_t word = (g & 1) ? ((o >> 16) | (v & 0xffff0000u)) : ((v & 0xffffu) | (o << 16));
                        uint32_t q4[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            q4[q] = __shfl_sync(0xffffffffu, word, HALF ? 8 * ch + (q & 1) + 4 * (q >> 1) : 4 * ch + q);
                        const uint32_t o2 = hd - hbuf + (HALF ? (uint32_t)kk * 16u : row_off(kk, ch & 1));
#pragma unroll
                        for (int q = 0; q < NP; ++q)
                            if (C % PEERS == 0 || (lane >> 2) < C) st_async_v4(peer[q] + o2, q4[0], q4[1], q4[2], q4[3], peer[q] + (bar(i, ev) - hbuf));
                    } else {
                        st_shared_parts(hd + 2u * (uint32_t)n, warp * 4 + uu, v);
                    }
                }
                if (publish && i == ntr - 1) ++ev;
                cp = c;
                if (TM) sts(st + 128u * WN, c);
                // the peers are waiting for h: the layer's own state goes to memory after it is on its way
                if (mine) {
                    char *ap = reinterpret_cast<char *>(a.bf.acts + ((size_t)t * P + row0) * 4 * ls);
                    *reinterpret_cast<float *>(ap + of_a) = ni;
                    *reinterpret_cast<float *>(ap + (of_a + of_g)) = ig;
                    *reinterpret_cast<float *>(ap + (of_a + 2u * of_g)) = fg;
                    *reinterpret_cast<float *>(ap + (of_a + 3u * of_g)) = og;
                    const size_t r = ((size_t)t * P + row0) * ls;
                    *reinterpret_cast<float *>(reinterpret_cast<char *>(a.bf.cells + r) + of_y) = c;
                    *reinterpret_cast<float *>(reinterpret_cast<char *>(a.y + r) + of_y) = hh;
                }
        };
        if (Tc > 0) fetch(0, 0);
#pragma unroll 1
        for (int s = 0; s < Tc && ok; ++s)
#pragma unroll 1
            for (int i = 0; i < ntr && ok; ++i) step(s, i);
        // frames beyond the longest sequence
        for (int i = 0; i < ntr; ++i) {
            const int pg = (tile0 + i) * 8 + n;
            if (unit && owner && pg < P)
                for (int t = Tc; t < T; ++t) {
                    const size_t f = ((size_t)t * P + pg) * ls + u;
                    a.y[f] = 0.0f;
                    a.bf.cells[f] = 0.0f;
                }
        }
        if (C == 1) __syncthreads();
    }
    if constexpr (C > 1) cluster_sync_all();   // nobody leaves while a peer may still write into its shared memory
    if constexpr (TM) {
        tc_fence_after();
        if (warp == 0) tmem_dealloc(tmem_s, TM_COLS);
    }
}

// ---- backward ------------------------------------------------------------------------------------------------------------
// a warp: MT m-tiles of 16 source units times the block's NK k-steps of gate rows.  One block alone: one m-tile per four warps,
// which take a quarter of the rows each and stand for the source blocks of a cluster of four
template <int C, int WN>
struct BwdGeo {
    static constexpr int U = 4 * WN, MT = C > 1 ? C / 4 : 1, NK = C > 1 ? WN : WN / 4, SRC = C > 1 ? C : 4;
    static constexpr uint32_t BUF = SRC * U * 32u;          // partial errors: [source][unit][8 floats]
    static constexpr uint32_t DTILE = 4u * U * 32u;         // the block's own deltas
    // TM: per tile also length, cell state, and what a cell hands to its next step
    static constexpr size_t smem(int nt, bool tm) { return (size_t)2 * nt * (BUF + DTILE) + (tm ? (size_t)nt * 6 * 32 * WN * 4 : 0); }
};
template <int C, int WN, bool TM>
__global__ void __launch_bounds__(32 * WN, 1) lstm_bwd_cluster_kernel(ClusterArgs a) {
    typedef BwdGeo<C, WN> G;
    constexpr int U = G::U, MT = G::MT, NK = G::NK, SRC = G::SRC;
    constexpr uint32_t BUF = G::BUF, DTILE = G::DTILE;
    __shared__ __align__(8) unsigned long long bars[TM ? MAX_NT : 1][2];
    __shared__ uint32_t tmem_s;
    const int nt = TM ? a.nt : 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int uu = lane >> 3, n = 2 * tig + (g & 1);
    const uint32_t rank = cluster_ctarank(), ebuf = smem_u32(cl_smem), dbuf = ebuf + 2u * nt * BUF;
    const uint32_t state = dbuf + 2u * nt * DTILE + 4u * threadIdx.x;
    const int P = a.sh.P, T = a.sh.T, ls = a.sh.ls, els = a.sh.els, D = a.sh.D;
    const LstmOffsets off = lstm_offsets(a.sh.pls, ls, els);
    const int j = (int)rank * U + warp * 4 + uu;
    auto bar = [&](int i, unsigned e) { return smem_u32(&bars[i][e & 1u]); };
    if (threadIdx.x == 0) {
        for (int i = 0; i < nt; ++i) { mbar_init(bar(i, 0), 1); mbar_init(bar(i, 1), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (TM) {
        if (warp == 0) tmem_alloc(smem_u32(&tmem_s), TM_COLS);
        tc_fence_before();
    }
    if constexpr (C > 1) cluster_sync_all();
    else __syncthreads();
    uint32_t tm = 0;
    if constexpr (TM) {
        tc_fence_after();
        tm = tmem_s + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * MT * NK * 4);
    }
    const int mtile0 = C > 1 ? warp * MT : warp >> 2, k0 = C > 1 ? 0 : (warp & 3) * NK;   // first m-tile and k-step of this warp
    const uint32_t ldsm_lane = (uint32_t)(((lane >> 3) & 1) * 8 + (lane & 7)) * 32u + (uint32_t)(((lane >> 4) ^ ((lane >> 2) & 1)) * 16) +
                               (uint32_t)k0 * 512u;

    // lane's source unit of m-tile mt (even tig row g, odd tig row g + 8): the block that owns it, its place there
    uint32_t peer[MT], place[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        const int src = (mtile0 + mt) * 16 + g + ((tig & 1) ? 8 : 0);
        peer[mt] = C > 1 ? map_to_rank(ebuf, (uint32_t)(src / U)) : ebuf;
        place[mt] = (((C > 1 ? rank : (uint32_t)(warp & 3)) * U + (uint32_t)(src % U)) * 8u + 4u * (uint32_t)(tig >> 1)) * 4u;
    }

    uint32_t whi[MT * NK][4], wlo[TM ? 1 : MT * NK][4];     // slot ks * MT + mt
    float inv = 1.0f;
    int cur_d = -1;
    unsigned ev = 0;
    bool ok = true;
    for (int item = (int)(blockIdx.x / C); item < a.n_items && ok; item += a.nclusters) {
        const int d = item % D, tile0 = (item / D) * nt, ntr = TM ? min(nt, a.tiles - tile0) : 1;
        if (d != cur_d) {
            // rows: source units; contraction index 16 ks + 4 gate + unit: the block's own gate rows
            inv = load_fragments<MT * NK, TM>(whi, wlo, tm, [&](int sl, int e) {
                const int src = (mtile0 + sl % MT) * 16 + g + ((e & 2) ? 8 : 0);
                const int pos = 2 * tig + (e & 1) + ((e & 4) ? 8 : 0);
                const int jw = (int)rank * U + (k0 + sl / MT) * 4 + (pos & 3);
                return (jw < els && src < els) ? __ldg(a.w + off.rec + ((size_t)(pos >> 2) * ls + (size_t)d * els + jw) * els + src) : 0.0f;
            }) * (1.0f / S_D);
            cur_d = d;
        }
        const int u = d * els + j;
        float pw[3] = {0, 0, 0};
        if (j < els)
#pragma unroll
            for (int q = 0; q < 3; ++q) pw[q] = __ldg(a.w + off.peep + (size_t)q * ls + u);
        const bool unit = j < els;
        const uint32_t uc = (uint32_t)(d * els + (unit ? j : 0)), of_g = (uint32_t)ls * 4u;      // addresses as in the forward kernel
        const uint32_t of_y = ((uint32_t)n * ls + uc) * 4u, of_a = ((uint32_t)n * 4u * ls + uc) * 4u;
        struct In { float e, ni, ig, fg, og, cp; };     // output error, activations, the previous frame's cell state
        In in = {0, 0, 0, 0, 0, 0};
        int len = 0, Tc = 0;
        float cc = 0.0f, st_fg = 0.0f, st_ce = 0.0f, st_dig = 0.0f, st_dfg = 0.0f;   // this frame's cell state; values of the step before
        auto at = [&](int i, int q) { return state + (uint32_t)(6 * i + q) * (128u * WN); };
        for (int i = 0; i < ntr; ++i) Tc = max(Tc, sequence_length(a.sh, a.bf.pat, (tile0 + i) * 8 + n));
        Tc = warp_max(Tc);
        for (int i = 0; i < ntr; ++i) {
            const int pg = (tile0 + i) * 8 + n, t = d ? 0 : Tc - 1;
            len = sequence_length(a.sh, a.bf.pat, pg);
            cc = unit && t >= 0 && t < len ? a.bf.cells[((size_t)t * P + pg) * ls + u] : 0.0f;     // the sweep's first frame
            if (TM) {
                sts(at(i, 0), __int_as_float(len));
                sts(at(i, 1), cc);
#pragma unroll
                for (int q = 2; q < 6; ++q) sts(at(i, q), 0.0f);
            }
        }
        auto fetch = [&](int s, int i) {      // a tile-step ahead, before the wait (see the forward kernel)
            const int sc = s < Tc ? s : Tc - 1, t = d ? sc : Tc - 1 - sc, prev = sc == Tc - 1 ? t : (d ? t + 1 : t - 1);
            const int row0 = (tile0 + i) * 8;
            const uint32_t oy = row0 + n < P ? of_y : uc * 4u, oa = row0 + n < P ? of_a : uc * 4u;
            in.e = *reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.dy + ((size_t)t * P + row0) * ls) + oy);
            const char *ap = reinterpret_cast<const char *>(a.bf.acts + ((size_t)t * P + row0) * 4 * ls);
            in.ni = *reinterpret_cast<const float *>(ap + oa);
            in.ig = *reinterpret_cast<const float *>(ap + (oa + of_g));
            in.fg = *reinterpret_cast<const float *>(ap + (oa + 2u * of_g));
            in.og = *reinterpret_cast<const float *>(ap + (oa + 3u * of_g));
            in.cp = *reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.bf.cells + ((size_t)prev * P + row0) * ls) + oy);
        };
        auto step = [&](int s, int i) {
                const int t = d ? s : Tc - 1 - s, row0 = (tile0 + i) * 8;
                if (TM) {
                    len = __float_as_int(lds(at(i, 0)));
                    cc = lds(at(i, 1)); st_fg = lds(at(i, 2)); st_ce = lds(at(i, 3)); st_dig = lds(at(i, 4)); st_dfg = lds(at(i, 5));
                }
                const bool first = (s == 0), last = (s == Tc - 1), real = t < len && unit, mine = unit && row0 + n < P;
                if (C > 1 && !last && threadIdx.x == 0) mbar_expect_tx(bar(i, ev), BUF);
                float e = in.e;
                const float nig = in.ni, ig = in.ig, fg = in.fg, og = in.og, cp = last || !mine ? 0.0f : in.cp;    // no previous cell state at the last step
                // ComputeBlockErrorsFn, the part that does not wait for the peers' partial errors: with e the output error,
                //   dog = k_og e, ce = k_ce e + p_og dog + carry, d{ni,ig,fg} = k_{ni,ig,fg} ce
                const float tc = cl_tanh(cc);
                float k_og = d_logistic(og) * tc, k_ce = og * d_tanh(tc);
                float carry = st_fg * st_ce + pw[0] * st_dig + pw[1] * st_dfg;      // zeros at the first step
                float k_ni = ig * d_tanh(nig), k_ig = d_logistic(ig) * nig, k_fg = d_logistic(fg) * cp;
                settle(k_og, k_ce, carry, k_ni, k_ig, k_fg);
                if (TM && i + 1 < ntr) fetch(s, i + 1); else fetch(s + 1, 0);
                if (!first) {
                    if constexpr (C > 1) ok = wait_bounded(bar(i, ev - 1), ((ev - 1) >> 1) & 1u, a.status);
                    else __syncthreads();
                    const float *pe = reinterpret_cast<const float *>(cl_smem + (((ev - 1) & 1u) * nt + (uint32_t)i) * BUF) + (warp * 4 + uu) * 8 + n;
                    // rank order; four chains where there are more than four sources
                    float sum = 0.0f;
                    if constexpr (SRC > 4) {
                        float s4[4] = {0, 0, 0, 0};
#pragma unroll
                        for (int src = 0; src < SRC; ++src) s4[src & 3] += pe[src * U * 8];
                        sum = (s4[0] + s4[1]) + (s4[2] + s4[3]);
                    } else {
#pragma unroll
                        for (int src = 0; src < SRC; ++src) sum += pe[src * U * 8];
                    }
                    e += sum;
                }
                const float dog_ = k_og * e;
                float ce = __fadd_rn(__fadd_rn(__fmul_rn(k_ce, e), __fmul_rn(pw[2], dog_)), carry);   // rounded term by term, as on the host
                float dd[4] = {limited_error(k_ni * ce), limited_error(k_ig * ce), limited_error(k_fg * ce), limited_error(dog_)};
                if (!real) ce = dd[0] = dd[1] = dd[2] = dd[3] = 0.0f;
                if (!last) {
                    const uint32_t db = dbuf + ((ev & 1u) * nt + (uint32_t)i) * DTILE;
                    uint32_t la[TM ? 16 : 1], lb[TM ? 16 : 1];     // lo parts of a k-step's m-tiles, on their way while those before are in use
#pragma unroll
                    for (int q = 0; q < 4; ++q) st_shared_parts(db + 2u * (uint32_t)n, warp * 16 + q * 4 + uu, split_pair(dd[q], S_D));
                    if (__syncthreads_or(!ok)) { ok = false; return; }
                    if constexpr (TM) { static_assert(MT == 4, "four m-tiles a k-step"); frag_load(la, tm); }
                    float m0[MT][4], xa[MT][4];
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int q = 0; q < 4; ++q) m0[mt][q] = xa[mt][q] = 0.0f;
#pragma unroll
                    for (int ks = 0; ks < NK; ++ks) {
                        uint32_t b[4];
                        ldsm_x4_t(b, db + ldsm_lane + (uint32_t)ks * 512u);
                        if constexpr (TM) {
                            if (ks & 1) { frag_wait(lb); if (ks + 1 < NK) frag_load(la, tm + 16u * (ks + 1)); }
                            else { frag_wait(la); if (ks + 1 < NK) frag_load(lb, tm + 16u * (ks + 1)); }
                        }
#pragma unroll
                        for (int mt = 0; mt < MT; ++mt) {
                            const uint32_t *f = whi[ks * MT + mt];
                            auto lo_of = [&](int q) { if constexpr (TM) return (ks & 1) ? lb[4 * mt + q] : la[4 * mt + q]; else return wlo[ks * MT + mt][q]; };
                            mma16816(xa[mt], lo_of(0), lo_of(1), lo_of(2), lo_of(3), b[0], b[1]);
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
                        const float4 f4 = make_float4(odd ? r0 : v[0], odd ? r1 : v[1], odd ? v[2] : r0, odd ? v[3] : r1);
                        const uint32_t o2 = ((ev & 1u) * nt + (uint32_t)i) * BUF + place[mt];
                        if constexpr (C > 1)
                            st_async_v4(peer[mt] + o2, __float_as_uint(f4.x), __float_as_uint(f4.y), __float_as_uint(f4.z), __float_as_uint(f4.w),
                                        peer[mt] + (bar(i, ev) - ebuf));
                        else
                            *reinterpret_cast<float4 *>(cl_smem + o2) = f4;
                    }
                }
                if (!last && i == ntr - 1) ++ev;
                cc = cp;                // the previous frame's cell state is the next step's own
                st_fg = real ? fg : 0.0f; st_ce = ce; st_dig = dd[1]; st_dfg = dd[2];
                if (TM) { sts(at(i, 1), cc); sts(at(i, 2), st_fg); sts(at(i, 3), st_ce); sts(at(i, 4), st_dig); sts(at(i, 5), st_dfg); }
                // the deltas go to memory after the partial errors the peers wait for have been sent
                if (mine) {
                    char *dl = reinterpret_cast<char *>(a.bf.deltas + ((size_t)t * P + row0) * 4 * ls);
#pragma unroll
                    for (int q = 0; q < 4; ++q) *reinterpret_cast<float *>(dl + (of_a + (uint32_t)q * of_g)) = dd[q];
                }
        };
        if (Tc > 0) fetch(0, 0);
#pragma unroll 1
        for (int s = 0; s < Tc && ok; ++s)
#pragma unroll 1
            for (int i = 0; i < ntr && ok; ++i) step(s, i);
        ok = !__syncthreads_or(!ok);
        for (int i = 0; i < ntr; ++i) {
            const int pg = (tile0 + i) * 8 + n;
            if (unit && pg < P)
                for (int t = Tc; t < T; ++t) {
                    float *dl = a.bf.deltas + ((size_t)t * P + pg) * 4 * ls + u;
#pragma unroll
                    for (int q = 0; q < 4; ++q) dl[(size_t)q * ls] = 0.0f;
                }
        }
    }
    if constexpr (C > 1) cluster_sync_all();
    if constexpr (TM) {
        tc_fence_after();
        if (warp == 0) tmem_dealloc(tmem_s, TM_COLS);
    }
}

// x(n) and behind it, for each entry, its logistic, its tanh and 1 / (1 + |x|) as the recurrence kernels compute them
__global__ void activations_selftest_kernel(float *v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = v[i];
    v[(size_t)n + i] = cl_logistic(x);
    v[(size_t)2 * n + i] = cl_tanh(x);
    v[(size_t)3 * n + i] = cl_rcp(1.0f + fabsf(x));
}

// ---- host side ---------------------------------------------------------------------------------------------------------------
typedef void (*Kernel)(ClusterArgs);
struct Variant {
    int C, WN;
    bool half, tm;
    Kernel kern;
    size_t smem1, smem2;    // shared memory for nt tiles: smem1 + nt * smem2
    size_t smem(int nt) const { return smem1 + nt * smem2; }
};
template <int C, int WN, bool HALF, bool TM>
constexpr Variant fwd_variant() {
    return Variant{C, WN, HALF, TM, lstm_fwd_cluster_kernel<C, WN, HALF, TM>, fwd_smem<C, WN, HALF, TM>(0),
                   fwd_smem<C, WN, HALF, TM>(1) - fwd_smem<C, WN, HALF, TM>(0)};
}
template <int C, int WN, bool TM>
constexpr Variant bwd_variant() {
    typedef BwdGeo<C, WN> G;
    return Variant{C, WN, false, TM, lstm_bwd_cluster_kernel<C, WN, TM>, G::smem(0, TM), G::smem(1, TM) - G::smem(0, TM)};
}
// geometries (blocks of a cluster, warps of a block): 16 to 320 units with all weights in registers, to 384 and 512 with the lo parts in
// tensor memory
#define SHAPES(X) X(1, 4) X(1, 8) X(4, 4) X(4, 6) X(4, 8) X(8, 4) X(8, 5) X(8, 6) X(8, 7) X(8, 8) X(16, 2) X(16, 4) X(16, 5)
#define SHAPES_HALF(X) X(4, 4) X(4, 6) X(4, 8) X(8, 4) X(8, 5) X(8, 6) X(8, 7) X(8, 8) X(16, 2) X(16, 4) X(16, 5)
#define SHAPES_TM(X) X(16, 6) X(16, 8)
#define FWD_FULL(C, WN) fwd_variant<C, WN, false, false>(),
#define FWD_HALF(C, WN) fwd_variant<C, WN, true, false>(),
#define FWD_TM(C, WN) fwd_variant<C, WN, false, true>(), fwd_variant<C, WN, true, true>(),
#define BWD_FULL(C, WN) bwd_variant<C, WN, false>(),
#define BWD_TM(C, WN) bwd_variant<C, WN, true>(),
const Variant FWD[] = {SHAPES(FWD_FULL) SHAPES_HALF(FWD_HALF) SHAPES_TM(FWD_TM)};
const Variant BWD[] = {SHAPES(BWD_FULL) SHAPES_TM(BWD_TM)};
constexpr int NFWD = (int)(sizeof(FWD) / sizeof(FWD[0])), NBWD = (int)(sizeof(BWD) / sizeof(BWD[0]));
constexpr int NMAX = NFWD > NBWD ? NFWD : NBWD;

// clusters of a variant that the current device holds at once (asked once per kernel and device; *alone: with one block per SM, which
// is also how many there are of the kernels that run several tiles)
int resident_clusters(bool backward, int vi, int *alone) {
    static std::mutex mu;
    static short known[MAX_DEVICES][2][NMAX][2];    // 0 = not asked yet, else clusters + 1
    const int dev = current_device();
    const Variant &v = backward ? BWD[vi] : FWD[vi];
    if (dev < 0) return 0;
    std::lock_guard<std::mutex> lk(mu);
    short *k = known[dev][backward][vi];
    if (!k[0]) {
        const int spread = v.tm ? (int)v.smem(MAX_NT) : 120 * 1024;     // shared memory that keeps a second block off the SM
        allow((const void *)v.kern, spread, v.C);
        for (int q = 0; q < 2; ++q)
            k[q] = (short)(1 + resident((const void *)v.kern, Launch(v.C, 32 * v.WN, q ? spread : v.smem(1), v.C, false, nullptr)));
    }
    *alone = k[1] - 1;
    return k[0] - 1;
}

// Cycles of a step, fitted to sweeps on a B200 at 1.95 GHz (forward / backward, us per step: 256 units on clusters of 16 x 4 warps
// 0.97 / 0.99, of 8 x 8 warps 1.28 / 1.29; 128 units, 8 x 4: 0.67 / 0.85; 64 units, 4 x 4: 0.60 / 0.75; 16 units, one block: 0.46 /
// 0.58).  A second warp on an SM quarter adds its own cell math; share = blocks of an SM.
double step_cycles(const Variant &v, int KP, int nt, double share, bool backward) {
    const int waves = (v.WN + 3) / 4;
    const double mma = (v.half ? 16.0 : 24.0) * (KP / 16) * waves;
    const double packets = v.C > 1 ? (v.C > 8 ? 0.7 : 0.4) * KP * (v.half ? 1.0 : 2.0) : 0.0;
    const double first = (backward ? 850.0 : 620.0) + (v.C > 1 ? 430.0 : 0.0) + 350.0 * (waves - 1) + share * (mma + packets);
    return first + (nt - 1) * ((mma > packets ? mma : packets) + 400.0);
}

struct Plan { int vi, nt, items, clusters; double cycles; };
Plan search_plan(const LstmShape &s, bool backward) {
    Plan best{-1, 0, 0, 0, 0.0};
    double best_t = 0.0;
    const int tiles = (s.P + 7) / 8;
    for (int vi = 0; vi < (backward ? NBWD : NFWD); ++vi) {
        const Variant &v = backward ? BWD[vi] : FWD[vi];
        const int KP = v.C * 4 * v.WN;
        if (KP < s.els || (v.half && s.P > 4)) continue;
        int alone = 0;
        const int res = resident_clusters(backward, vi, &alone);
        if (res < 1 || alone < 1) continue;
        for (int nt = 1; nt <= (v.tm ? MAX_NT : 1) && nt <= tiles; ++nt) {
            const int items = s.D * ((tiles + nt - 1) / nt), room = v.tm ? alone : res;
            const int live = items < room ? items : room, passes = (items + live - 1) / live;
            const double share = (double)((live + alone - 1) / alone);
            // where two come out equal, the one on fewer SMs: another net's kernels may want the rest
            const double t = passes * step_cycles(v, KP, nt, share, backward) * (1.0 + 0.05 * live * v.C / sm_count());
            if (best.vi < 0 || t < best_t) { best = Plan{vi, nt, items, live, passes * step_cycles(v, KP, nt, share, backward)}; best_t = t; }
        }
    }
    return best;
}

// a layer asks for its plan several times a pass (the search takes 5 us of host time): every thread keeps those of the last shapes it met
Plan make_plan(const LstmShape &s, bool backward) {
    struct Memo { int dev, els, D, P; Plan plan; };
    constexpr int N = 16;
    static thread_local Memo memo[2][N];
    static thread_local int used[2], next[2];
    const int dev = current_device();
    for (int i = 0; i < used[backward]; ++i) {
        const Memo &m = memo[backward][i];
        if (m.dev == dev && m.els == s.els && m.D == s.D && m.P == s.P) return m.plan;
    }
    const Memo m{dev, s.els, s.D, s.P, search_plan(s, backward)};
    memo[backward][next[backward]] = m;
    next[backward] = (next[backward] + 1) % N;
    if (used[backward] < N) ++used[backward];
    return m.plan;
}

}  // namespace

int lstm_selftest_activations(const float *x, int n, float *logistic, float *tanh, float *rcp) {
    float *dev = nullptr;
    const size_t bytes = (size_t)n * sizeof(float);
    B2_CUDA(cudaMalloc(&dev, 4 * bytes));
    cudaError_t e = cudaMemcpy(dev, x, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        activations_selftest_kernel<<<(n + 255) / 256, 256>>>(dev, n);
        count_launch();
        e = cudaGetLastError();
    }
    float *const out[3] = {logistic, tanh, rcp};
    for (int i = 0; i < 3 && e == cudaSuccess; ++i) e = cudaMemcpy(out[i], dev + (size_t)(i + 1) * n, bytes, cudaMemcpyDeviceToHost);
    cudaFree(dev);
    B2_CUDA(e);
    return B2_OK;
}

bool lstm_cluster_supported(const LstmShape &s) { return s.els <= 512 && make_plan(s, false).vi >= 0 && make_plan(s, true).vi >= 0; }

// The fit of step_cycles holds up to 256 units; beyond, several tiles in turn and 16 blocks a cluster, measured steps are 1.4 times as long
// (us per step, forward + backward, estimated and measured: 512 units, 64 sequences, bidirectional 7.8 and 11.5, 32 sequences 5.9 and
// 7.1; 400 units, 128 sequences 15.7 and 23.8; 300 units, 64 sequences 6.5 and 8.8).
double lstm_cluster_step_us(const LstmShape &s) {
    return (s.els > 256 ? 1.4 : 1.0) * (make_plan(s, false).cycles + make_plan(s, true).cycles) / 1950.0;
}

int lstm_cluster_sweep(bool backward, const LstmShape &s, const LstmBuffers &b, const float *w, float *y, const float *dy, int *status,
                       cudaStream_t st) {
    const Plan pl = make_plan(s, backward);
    if (pl.vi < 0) return 1;
    const Variant &v = backward ? BWD[pl.vi] : FWD[pl.vi];
    ClusterArgs a;
    a.sh = s; a.bf = b; a.w = w; a.y = y; a.dy = dy; a.status = status;
    a.tiles = (s.P + 7) / 8; a.nt = pl.nt; a.n_items = pl.items; a.nclusters = pl.clusters;
    const Launch l(pl.clusters * v.C, 32 * v.WN, v.smem(pl.nt), v.C, false, st);
    B2_CUDA(cudaLaunchKernelEx(&l.cfg, v.kern, a));
    count_launch();
    return B2_OK;
}

}  // namespace b2
