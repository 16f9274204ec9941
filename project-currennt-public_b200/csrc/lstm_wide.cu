// Persistent tensor-core recurrence for 257 to 1024 units per direction: ONE launch runs all timesteps of a sweep with the
// recurrent weights resident on chip, fp16 hi parts in shared memory, lo parts in TENSOR MEMORY.
//
// Replaces the reference's per-timestep loop of 4 cublasSgemm + 1 Thrust functor per direction
// (layers/LstmLayer.cu:1805-1858,1878-1927 forward with ComputeBlockOutputFn :57-185; :2115-2176,2195-2253 backward with
// ComputeBlockErrorsFn :237-405 of the reference), and the launch pair per timestep of lstm_step_tc.cu, which streams the weights
// of both directions (67 MB as tf32 parts) from L2 at every step.
//
// Decomposition.  A direction (or a share of the sequences of the only one) is a group of 64 blocks, two groups run side by side.  A
// block holds 128 rows x 512 contraction positions of the recurrent matrix (65536 weights): hi parts as a K-major SWIZZLE_128B operand in
// 128 KB of shared memory, lo parts in 256 tensor-memory columns (operand A of tcgen05.mma may come from there), which leaves 256 columns
// for accumulators.
//   forward : rows = 32 units x 4 gates, contraction = 512 of the 1024 source units; 32 row tiles x 2 slices, a cluster of 2 blocks
//             holds the slices of a row tile and exchanges partial sums through distributed shared memory.
//   backward: rows = 128 source units, contraction = 512 of the 4096 gate rows (128 units x 4 gates); 8 row tiles x 8 slices.  Clusters of
//             8 would not fit 16 times, so the slices of a row tile exchange partial sums through L2.
// The two sweeps are one kernel: gather an operand slice, multiply, exchange partial sums, run the cells of the 16 units a block
// finishes, publish what the next step gathers (h, resp. the gate deltas).  Fewer units are padded to 1024 with zero weights.
// Up to 512 units (padded to 512) a group has 16 blocks and eight groups run side by side, a chunk of sequences each: 16 row tiles with the
// whole contraction forward (no exchange), 4 row tiles x 4 slices backward; a block finishes 32 units.
//
// A step of a chunk of NC sequences (16, 32 or 64).  The operand lies in global memory (L2) as images of 64 contraction positions:
// 2 NC rows (hi of every sequence, then lo) of 128 bytes, swizzled.  The polling warp watches the step counters of the blocks that
// write the images of its slice and fetches each image with one bulk copy as soon as its writers are through; NI issuing warps, each
// with an accumulator of its own, multiply the images of their part of the slice: hi x [hi | lo] as ONE instruction with N = 2 NC (main
// products and one cross term side by side) and lo x hi with N = NC onto the cross columns.  Drain warps combine the accumulators and
// deliver each row to the block that finishes its unit; the cell warps add the partial sums in slice order (deterministic).
//
// What bounds a step (1024 units, 64 sequences, 15000 cycles): the chain publish 1300 - counters 1000 to 2500 - first image 700 - products
// 3500 (3072 at the rate of the tensor cores: 4096 MAC per cycle and SM) - drain and exchange 1800 - cells 2500.  What shortened it, in us
// per step forward / backward: one thread issuing all MMAs and a proxy fence before each bulk copy 12.7 / 16.8; several issuers (a
// tcgen05.mma with run-time descriptors costs its thread 118 cycles) and one fence on the publishing side 10.3 / 14.0; copies issued by 8
// lanes side by side and the layer's state stored only after the publication 8.4 / 11.8; the counters on lines of their own and
// partial sums read straight from L2 7.6 / 7.8 (at 1.95 GHz; four layers under the power cap at 1.6 GHz 8.9 / 10.2).  512 units, 256 sequences in eight groups: 8.2 / 9.4, of which the cells of 32 units x 64
// sequences take 2 (lstm_ptc.cu 11.1 / 13.5).  The launch pair per step of lstm_step_tc.cu takes 24.6 / 26.6; 16 sequences: 4.3 / 5.7
// and 23.0 / 23.8.
// Numerics as in lstm_ptc.cu: x*S = hi + lo*2^-11, S = 2^14 for h, 2^15 for the deltas, 2^13 <= max|w|*S < 2^14 per block; a chain holds at
// most 16 main products (tensor-memory accumulation truncates).
//
// Blocks of a group wait for each other, so the launch is cooperative.  Every wait is bounded as in lstm_ptc.cu.
#include <algorithm>
#include <mutex>

#include "cluster.cuh"
#include "common.cuh"
#include "ptx.cuh"

namespace b2 {
namespace {

using namespace ptx;
using cluster::cl_logistic;
using cluster::cl_tanh;
using cluster::settle;
using cluster::split_pair;
using cluster::LO_UNSCALE;
using cluster::S_D;
using cluster::S_H;

constexpr int KB = 8;                                     // operand images of a slice
// Step counters: a line of 128 bytes for each slice (fewer readers wait longer for a line that many SMs poll: one line for all slices,
// polled by 8 warps of a block, cost the backward step of 16 sequences 3 us), in several copies that the readers share; behind them a line
// for the partial sums of each row tile.
constexpr int LINE = 32, GROUP_FLAGS = (16 + 8) * LINE;
constexpr long long WAIT_CYCLES = 4000000000LL;
constexpr unsigned POLL_LIMIT = 1u << 22;
constexpr int W_POLL = 0, W_MMA = 1;
constexpr uint32_t A_BYTES = 131072;

struct WideArgs {
    LstmShape sh;
    LstmBuffers bf;
    const float *w;
    float *y;                // forward: block outputs
    const float *dy;         // backward: output errors
    unsigned char *img;      // per group: 2 step parities x operand images
    unsigned *flags;         // per group: step counters of its blocks, for the operand images and for partial sums
    int *status;
    unsigned tag_base;
    int nchunks;             // chunks of NC sequences
};

// E: the units of a direction are padded to E = 1024 or 512
template <int E, bool BWD, int NC>
struct Geo {
    static constexpr int GROUP = E * E / 16384, UPB = E / GROUP;       // blocks of a group; units a block finishes
    static constexpr int CS = BWD ? E / 128 : E / 512, ROWS = 128 / CS;   // slices of a row tile; rows of partial sums a block finishes
    static constexpr int CL = BWD ? 1 : CS;                            // blocks of a cluster
    // warps that issue MMAs, each on an accumulator of its own (columns NI x 2 NC <= 256); the other roles follow.  16 sequences side by
    // side in the cell warps.
    static constexpr int NI = NC == 64 ? 2 : 4, ACC = 256 / NI, NCW = UPB / 2;
    static constexpr int W_DRAIN = W_MMA + NI, W_CELL = W_DRAIN + 4, W_PUB = W_CELL + NCW, NTHR = 32 * (W_PUB + 1);
    static constexpr uint32_t IMG = 2 * NC * 128;                      // one operand image
    static constexpr int STAGES = NC == 64 ? 4 : 8;                    // images in flight: a whole slice where shared memory allows it
    static constexpr int NIMG = BWD ? E / 16 : E / 64;                 // images of a whole operand
    static constexpr uint32_t F_B = A_BYTES, F_Z = F_B + STAGES * IMG; // z: [source][NC / 4][ROWS][4]
    static constexpr uint32_t ZSRC = ROWS * NC * 4, F_END = F_Z + (BWD ? 0 : CS * ZSRC);
    static constexpr size_t smem() { return F_END + 1024; }
    static constexpr size_t IMG_BYTES = (size_t)2 * NIMG * IMG;                                  // two step parities
    static constexpr size_t GROUP_BYTES = IMG_BYTES + (BWD ? (size_t)2 * GROUP * CS * ZSRC : 0);   // + partial sums
};

__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, u64 bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// the end of a round of polling; every lane of the warp leaves in the same round
__device__ __forceinline__ bool stop(unsigned round, const int *status, volatile int *give_up) {
    return __any_sync(0xffffffffu, round >= POLL_LIMIT || *give_up || ((round & 255u) == 255u && ld_relaxed_s32(status) != 0));
}
__device__ __forceinline__ void load_l2(const float *p, float (&v)[1]) { asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v[0]) : "l"(p) : "memory"); }
__device__ __forceinline__ void load_l2(const float *p, float (&v)[2]) {
    asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p) : "memory");
}
__device__ __forceinline__ void load_l2(const float *p, float (&v)[4]) {
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p) : "memory");
}

template <int E, bool BWD, int NC>
__global__ void __launch_bounds__(Geo<E, BWD, NC>::NTHR, 1) lstm_wide_kernel(WideArgs a) {
    typedef Geo<E, BWD, NC> G;
    constexpr int GROUP = G::GROUP, UPB = G::UPB;
    constexpr int CS = G::CS, ROWS = G::ROWS, STAGES = G::STAGES, NI = G::NI, NTHR = G::NTHR;
    constexpr int W_DRAIN = G::W_DRAIN, W_CELL = G::W_CELL, W_PUB = G::W_PUB, CPT = NC / 16;        // CPT: cells per cell thread
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) u64 bars[2 * STAGES + 7 + NI];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int give_up_s, never_s;
    __shared__ int lens_s[NC], Tc_s;
    __shared__ unsigned wmax_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *gbase = smem_raw + (sbase - smem_u32(smem_raw));
    const uint32_t bar0 = smem_u32(bars);
    auto b_full = [&](int s) { return bar0 + 8u * (uint32_t)s; };                   // bulk copy -> MMA
    auto b_free = [&](int s) { return bar0 + 8u * (uint32_t)(STAGES + s); };        // MMA -> poll warp
    const uint32_t acc_full = bar0 + 8u * (2 * STAGES), acc_free = acc_full + 8u;   // MMA -> drain, drain -> MMA
    const uint32_t z_full = acc_full + 16u, z_free = acc_full + 24u;                // partial sums of the cluster -> cells, and back
    const uint32_t rel_full = acc_full + 32u, rel_free = acc_full + 40u;            // cells -> publisher, and back
    const uint32_t part_full = acc_full + 48u, quit = acc_full + 56u;               // drain -> publisher; (NI) last MMAs after a wait ran out

    const int P = a.sh.P, T = a.sh.T, ls = a.sh.ls, els = a.sh.els, D = a.sh.D;
    const int grp = blockIdx.x / GROUP, ngroups = gridDim.x / GROUP, bidx = blockIdx.x % GROUP, r = bidx / CS, q = bidx % CS;
    const LstmOffsets off = lstm_offsets(a.sh.pls, ls, els);
    unsigned char *img = a.img + (size_t)grp * G::GROUP_BYTES;
    unsigned *flags = a.flags + grp * GROUP_FLAGS, *pflags = flags + 16 * LINE;
    constexpr int NW = GROUP / CS, COPIES = 16 / CS;      // writers of a slice, copies of its line of counters
    // backward: partial sums of step parity b for the units of block `to`, from the block of slice `from` of its row tile
    auto zpart = [&](unsigned b, int to, int from) { return img + G::IMG_BYTES + (((size_t)(b & 1u) * GROUP + (size_t)to) * CS + (size_t)from) * G::ZSRC; };

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(b_full(s), 1); mbar_init(b_free(s), 1); }
        mbar_init(acc_full, NI); mbar_init(acc_free, 4);
        mbar_init(z_full, BWD ? 1 : 5);       // forward: 4 drain warps and the arrival that announces the peer's bytes; backward: poll warp
        mbar_init(z_free, G::NCW * G::CL);         // every cell warp of every block of the cluster
        mbar_init(rel_full, G::NCW); mbar_init(rel_free, 1);
        mbar_init(part_full, 4);
        for (int h = 0; h < NI; ++h) mbar_init(quit + 8u * (uint32_t)h, 1);
        give_up_s = 0; never_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(smem_u32(&tmem_base_s), 512);
    tc_fence_before();
    if constexpr (G::CL == 1) __syncthreads(); else cluster_sync_all();     // a peer's shared memory and barriers may be touched only once the peer runs
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;      // columns 0-255: accumulators [half][main NC | cross NC], 256-511: lo parts of the weights

    int n_b = 0, n_m = 0, n_d = 0, n_e = 0, n_p = 0;    // images fetched / multiplied; steps drained (multiplied), run (summed), published
    const int items = D * a.nchunks, wi_end = (grp + 1) * items / ngroups;
    unsigned ev = 0;                                     // published steps so far (parity of the operand images)
    int cur_d = -1, order = 0;
    float inv = 1.0f;
    for (int wi = grp * items / ngroups; wi < wi_end; ++wi, ++order) {
        const int d = wi / a.nchunks, p0 = (wi % a.nchunks) * NC;
        if (d != cur_d) {
            // weight(row, k): entry of this block's tile; forward row = gate * 32 + unit, backward k = unit * 4 + gate
            auto weight = [&](int row, int k) {
                const int gate = BWD ? k & 3 : row >> 5, j = BWD ? 128 * q + (k >> 2) : 32 * r + (row & 31), src = BWD ? 128 * r + row : 512 * q + k;
                return (j < els && src < els) ? __ldg(a.w + off.rec + ((size_t)gate * ls + (size_t)d * els + j) * els + src) : 0.0f;
            };
            if (tid == 0) wmax_s = 0u;
            __syncthreads();
            unsigned m = 0u;
#pragma unroll 8
            for (int i = tid; i < 128 * 512; i += NTHR) {      // coalesced along the contiguous index of the weight matrix
                const unsigned b = __float_as_uint(fabsf(BWD ? weight(i & 127, i >> 7) : weight(i >> 9, i & 511)));
                if (b < 0x7f800000u) m = max(m, b);            // NaN / Inf do not set the scale
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0) atomicMax(&wmax_s, m);
            __syncthreads();
            m = wmax_s;
            int e2 = m ? 13 - ((int)(m >> 23) - 127) : 0;
            e2 = e2 < -100 ? -100 : (e2 > 100 ? 100 : e2);
            const float S = __int_as_float((127 + e2) << 23);
            inv = __int_as_float((127 - e2) << 23) * (BWD ? 1.0f / S_D : 1.0f / S_H);
            if (warp >= W_DRAIN && warp < W_CELL) {
                // lane = row of this warp's lane quarter; 16 positions (one k-step) at a time
                const int row = 32 * (warp & 3) + lane;
                const uint32_t tl = tmem + 256u + ((uint32_t)(32 * (warp & 3)) << 16);
#pragma unroll 1
                for (int ks = 0; ks < 32; ++ks) {
                    uint32_t hi[8], lo[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const uint32_t x0 = split_pair(weight(row, 16 * ks + 2 * e), S), x1 = split_pair(weight(row, 16 * ks + 2 * e + 1), S);
                        hi[e] = (x0 & 0xffffu) | (x1 << 16);
                        lo[e] = (x0 >> 16) | (x1 & 0xffff0000u);
                    }
                    const uint32_t o = (uint32_t)(ks >> 2) * 16384u + (uint32_t)row * 128u;
                    const int c = 2 * (ks & 3);
                    *reinterpret_cast<uint4 *>(gbase + o + (uint32_t)((c ^ (row & 7)) * 16)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    *reinterpret_cast<uint4 *>(gbase + o + (uint32_t)(((c + 1) ^ (row & 7)) * 16)) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
                    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(tl + 8u * ks), "r"(lo[0]),
                                 "r"(lo[1]), "r"(lo[2]), "r"(lo[3]), "r"(lo[4]), "r"(lo[5]), "r"(lo[6]), "r"(lo[7])
                                 : "memory");
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                fence_async_smem();
                tc_fence_before();
            }
            cur_d = d;
        }
        // lengths of the chunk's sequences (padding frames trail a sequence), their maximum
        if (tid < NC) lens_s[tid] = cluster::sequence_length(a.sh, a.bf.pat, p0 + tid);
        __syncthreads();
        tc_fence_after();
        if (tid == 0) {
            int m = 0;
            for (int n = 0; n < NC; ++n) m = max(m, lens_s[n]);
            Tc_s = m;
        }
        __syncthreads();
        const int Tc = Tc_s;
        const unsigned tag0 = a.tag_base + (unsigned)order * (unsigned)(T + 1);

        if (warp == W_POLL) {
            // ---------------- watch the writers of this slice's images, fetch image by image ----------------
            const unsigned *line = flags + (q * COPIES + r % COPIES) * LINE + lane;
            unsigned late = 0u;                                  // images of an unfinished step that are on their way
            for (int s = 1; s < Tc; ++s) {
                if (__any_sync(0xffffffffu, give_up_s)) break;
                const unsigned want = tag0 + (unsigned)(s - 1);
                const unsigned char *src = img + ((size_t)((ev + (unsigned)(s - 1)) & 1u) * G::NIMG + (size_t)(KB * q)) * G::IMG;
                // lane = place of an image in the order of fetching: the parts of the slice in turn, an issuing warp takes each
                const int kb = (lane & 7) / NI + KB / NI * (lane % NI), nb = n_b + (lane & 7), st = nb % STAGES;
                // writers of this image: 64 units of h, or the gate deltas of 16 units
                const unsigned need = BWD ? 1u << (16 * kb / UPB) : ((1u << (64 / UPB)) - 1u) << (64 / UPB * kb);
                constexpr unsigned ALL = (1u << KB) - 1u;
                unsigned ready = 0u, sent = 0u;
                bool ok = true;
                for (unsigned round = 0; ok && sent != ALL; ++round) {
                    if (ready != (unsigned)((1ull << NW) - 1ull))
                        ready |= __ballot_sync(0xffffffffu, lane < NW && (int)(ld_acquire_u32(line) - want) >= 0);
                    const bool go = lane < KB && !(sent >> lane & 1u) && (ready & need) == need && (lane < STAGES || (sent >> (lane - STAGES) & 1u)) &&
                                    mbar_test(b_free(st), ((uint32_t)(nb / STAGES) & 1u) ^ 1u);
                    if (go) {
                        mbar_expect_tx(b_full(st), G::IMG);
                        bulk_g2s(sbase + G::F_B + (uint32_t)st * G::IMG, src + (size_t)kb * G::IMG, G::IMG, b_full(st));
                    }
                    sent |= __ballot_sync(0xffffffffu, go);
                    ok = !stop(round, a.status, &give_up_s);
                }
                n_b += ok ? KB : 0;
                if (!ok) late = sent;
                if constexpr (BWD) {
                    // the 8 blocks of this row tile hold partial sums for this block's units
                    ready = 0u;
                    for (unsigned round = 0; ok && ready != (1u << CS) - 1u; ++round) {
                        ready = __ballot_sync(0xffffffffu, lane < CS && (int)(ld_acquire_u32(pflags + r * LINE + lane) - want) >= 0);
                        ok = !stop(round, a.status, &give_up_s);
                    }
                    if (ok && lane == 0) mbar_arrive(z_full);
                }
                if (!ok) { give_up_s = 1; atomicCAS(a.status, 0, (int)B2_ERR_STEP_TIMEOUT); break; }
            }
            __syncwarp();
            if (give_up_s && lane == 0) {    // copies still in flight
                for (int k = n_b > STAGES ? n_b - STAGES : 0; k < n_b + KB; ++k)
                    if (k < n_b || (late >> (k - n_b) & 1u)) mbar_wait_bounded<false>(b_full(k % STAGES), (uint32_t)(k / STAGES) & 1u, &never_s, WAIT_CYCLES / 64);
            }
        } else if (warp < W_DRAIN) {
            // ---------------- MMA issue: a warp for each part of the slice, with an accumulator of its own ----------------
            if (lane == 0) {
                const int h = warp - W_MMA;
                const uint32_t id_main = idesc_f16(128, 2 * NC), id_cross = idesc_f16(128, NC);
                const uint32_t dm = tmem + (uint32_t)(G::ACC * h), dc = dm + NC;
                for (int s = 1; s < Tc; ++s) {
                    if (give_up_s) break;
                    bool ok = mbar_wait_bounded<false>(acc_free, ((uint32_t)n_d & 1u) ^ 1u, &give_up_s, WAIT_CYCLES);
                    ++n_d;
                    for (int i = KB / NI * h; i < KB / NI * (h + 1) && ok; ++i, n_m += NI) {
                        const int st = (n_m + h) % STAGES;
                        ok = mbar_wait_bounded<false>(b_full(st), (uint32_t)((n_m + h) / STAGES) & 1u, &give_up_s, WAIT_CYCLES);
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            const u64 bd = desc_kmajor_sw128(sbase + G::F_B + (uint32_t)st * G::IMG + 32u * ks, 1024);
                            const u64 ad = desc_kmajor_sw128(sbase + (uint32_t)i * 16384u + 32u * ks, 1024);
                            mma_f16(dm, ad, bd, id_main, (i % (KB / NI)) | ks ? 1u : 0u);
                            mma_f16_ts(dc, tmem + 256u + (uint32_t)(32 * i + 8 * ks), bd, id_cross, 1u);
                        }
                        mma_commit(b_free(st));
                    }
                    if (!ok) { give_up_s = 1; break; }
                    mma_commit(acc_full);
                }
                if (give_up_s) { mma_commit(quit + 8u * (uint32_t)h); mbar_wait_bounded<false>(quit + 8u * (uint32_t)h, 0u, &never_s, WAIT_CYCLES / 64); }
            }
            __syncwarp();
        } else if (warp < W_CELL) {
            // ---------------- drain tensor memory: every row to the block that finishes its unit ----------------
            const int row = 32 * (warp & 3) + lane;
            const int to = BWD ? row / ROWS : (row & 31) / UPB;                           // rank of that block
            const int rl = BWD ? row % ROWS : (row >> 5) * UPB + row % UPB;              // row among its ROWS
            const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
            const uint32_t zl = G::F_Z + (uint32_t)q * G::ZSRC + (uint32_t)rl * 16u;
            const uint32_t zr = G::CL == 1 ? 0u : map_to_rank(sbase + zl, (uint32_t)to), rbar = G::CL == 1 ? 0u : map_to_rank(z_full, (uint32_t)to);
            for (int s = 1; s < Tc; ++s, ++n_d) {
                if (__any_sync(0xffffffffu, give_up_s)) break;
                const uint32_t ph = (uint32_t)n_d & 1u;
                bool ok = true;
                if constexpr (!BWD) {
                    // the partial sums of the step before have been read, here and in the peer this warp writes to
                    ok = mbar_wait_bounded<false>(z_free, ph ^ 1u, &give_up_s, WAIT_CYCLES);
                    if (warp == W_DRAIN && lane == 0) mbar_expect_tx(z_full, (uint32_t)(CS - 1) * G::ZSRC);
                }
                unsigned char *zg = BWD ? zpart(ev + (unsigned)s, CS * r + to, q) + (uint32_t)rl * 16u : nullptr;
                ok = ok && mbar_wait_bounded<false>(acc_full, ph, &give_up_s, WAIT_CYCLES);
                if (!__all_sync(0xffffffffu, ok)) { give_up_s = 1; atomicCAS(a.status, 0, (int)B2_ERR_STEP_TIMEOUT); break; }
                tc_fence_after();
#pragma unroll
                for (int col = 0; col < NC; col += 16) {
                    float v[16];
#pragma unroll
                    for (int h = 0; h < NI; h += 2) {
                        uint32_t m0[16], m1[16], c0[16], c1[16];
                        const uint32_t th = tl + (uint32_t)(G::ACC * h + col);
                        tmem_ld16(th, m0);
                        tmem_ld16(th + G::ACC, m1);
                        tmem_ld16(th + NC, c0);
                        tmem_ld16(th + G::ACC + NC, c1);
                        tmem_ld_wait();
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const float x = (__uint_as_float(m0[c]) + __uint_as_float(m1[c])) + (__uint_as_float(c0[c]) + __uint_as_float(c1[c])) * LO_UNSCALE;
                            v[c] = h ? v[c] + x : x;
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 16; ++c) v[c] *= inv;
#pragma unroll
                    for (int g4 = 0; g4 < 4; ++g4) {
                        const uint32_t o = (uint32_t)((col >> 2) + g4) * (ROWS * 16u);
                        if constexpr (BWD)
                            *reinterpret_cast<float4 *>(zg + o) = make_float4(v[4 * g4], v[4 * g4 + 1], v[4 * g4 + 2], v[4 * g4 + 3]);
                        else if (G::CL == 1 || to == q)
                            *reinterpret_cast<float4 *>(gbase + zl + o) = make_float4(v[4 * g4], v[4 * g4 + 1], v[4 * g4 + 2], v[4 * g4 + 3]);
                        else
                            st_async_v4(zr + o, __float_as_uint(v[4 * g4]), __float_as_uint(v[4 * g4 + 1]), __float_as_uint(v[4 * g4 + 2]),
                                        __float_as_uint(v[4 * g4 + 3]), rbar);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(acc_free); mbar_arrive(BWD ? part_full : z_full); }
            }
        } else if (warp == W_PUB) {
            // ---------------- publisher: step counters follow the block's part of the operand and (backward) its partial sums ----------------
            for (int s = 0; s < Tc; ++s) {
                if (__any_sync(0xffffffffu, give_up_s)) break;
                bool ok = true;
                if (BWD && s > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait_bounded<false>(part_full, (uint32_t)n_d & 1u, &give_up_s, WAIT_CYCLES));
                    ++n_d;
                    if (ok && lane == 0) st_release_u32(pflags + r * LINE + q, tag0 + (unsigned)(s - 1));
                }
                if (s + 1 < Tc) {
                    ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded<false>(rel_full, (uint32_t)n_p & 1u, &give_up_s, WAIT_CYCLES));
                    ++n_p;
                    if (ok && lane < COPIES) {
                        fence_async_global();    // ordinary stores wrote what other blocks fetch with bulk copies (async proxy)
                        st_release_u32(flags + (bidx / NW * COPIES + lane) * LINE + bidx % NW, tag0 + (unsigned)s);
                    }
                    __syncwarp();
                    if (ok && lane == 0) mbar_arrive(rel_free);
                }
                __syncwarp();
                if (!ok) { give_up_s = 1; atomicCAS(a.status, 0, (int)B2_ERR_STEP_TIMEOUT); break; }
            }
        } else {
            // ---------------- cells: thread = unit (of UPB) of CPT sequences ----------------
            const int ct = tid - 32 * W_CELL, ul = ct % UPB, n0 = ct / UPB;
            const int j = (BWD ? 128 : 32) * r + UPB * q + ul;                 // unit inside the direction
            const bool unit = j < els;
            auto seq = [&](int i) { return BWD ? n0 * CPT + i : n0 + 16 * i; };     // sequence of this thread's i-th cell
            const int u = d * els + (unit ? j : 0);
            float b4[4], pw[3];
#pragma unroll
            for (int g = 0; g < 4; ++g) b4[g] = a.sh.bias * __ldg(a.w + off.bias + (size_t)g * ls + u);
#pragma unroll
            for (int g = 0; g < 3; ++g) pw[g] = __ldg(a.w + off.peep + (size_t)g * ls + u);
            int len[CPT];
            float in[CPT][BWD ? 6 : 4];                    // forward: pre-activations; backward: error, activations, previous cell state
            float st[CPT][BWD ? 5 : 1];                    // forward: cell state; backward: cell state, fg, cell error, two deltas of the step before
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
                len[i] = lens_s[seq(i)];
#pragma unroll
                for (int k = 0; k < (BWD ? 5 : 1); ++k) st[i][k] = 0.0f;
                if (BWD && Tc > 0) {
                    const int t = d ? 0 : Tc - 1, pg = p0 + seq(i);
                    if (t < len[i]) st[i][0] = a.bf.cells[((size_t)t * P + pg) * ls + u];
                }
            }
            // a step ahead, before the step waits; unconditional (see lstm_cluster.cu): slots without a sequence read that of the first
            auto fetch = [&](int s) {
                const int sc = s < Tc ? s : Tc - 1, t = (d != 0) != BWD ? Tc - 1 - sc : sc;
#pragma unroll
                for (int i = 0; i < CPT; ++i) {
                    const int pg = p0 + seq(i);
                    const size_t f = (size_t)t * P + (pg < P ? pg : p0);
                    const float *ap = a.bf.acts + f * 4 * ls + u;
#pragma unroll
                    for (int g = 0; g < 4; ++g) in[i][g] = ap[(size_t)g * ls];
                    if constexpr (BWD) {
                        const int prev = sc == Tc - 1 ? t : (d ? t + 1 : t - 1);
                        in[i][4] = a.dy[f * ls + u];
                        in[i][5] = a.bf.cells[((size_t)prev * P + (pg < P ? pg : p0)) * ls + u];
                    }
                }
            };
            if (Tc > 0) fetch(0);
            for (int s = 0; s < Tc; ++s) {
                if (__any_sync(0xffffffffu, give_up_s)) break;
                const int t = (d != 0) != BWD ? Tc - 1 - s : s;
                const bool first = (s == 0), last = (s == Tc - 1);
                float x[CPT][BWD ? 1 : 4], k_og[CPT], k_ce[CPT], carry[CPT], k_ni[CPT], k_ig[CPT], k_fg[CPT], fgk[CPT];
#pragma unroll
                for (int i = 0; i < CPT; ++i) {
                    if constexpr (!BWD) {
#pragma unroll
                        for (int g = 0; g < 4; ++g) x[i][g] = in[i][g] + b4[g];
                    } else {
                        // the part of ComputeBlockErrorsFn that does not wait for the partial errors (see lstm_cluster.cu)
                        x[i][0] = in[i][4];
                        const float ni = in[i][0], ig = in[i][1], og = in[i][3], tc = cl_tanh(st[i][0]);
                        const float cp = last || p0 + seq(i) >= P ? 0.0f : in[i][5];      // no previous cell state at the last step
                        fgk[i] = in[i][2];
                        k_og[i] = d_logistic(og) * tc;
                        k_ce[i] = og * d_tanh(tc);
                        carry[i] = st[i][1] * st[i][2] + pw[0] * st[i][3] + pw[1] * st[i][4];
                        k_ni[i] = ig * d_tanh(ni);
                        k_ig[i] = d_logistic(ig) * ni;
                        k_fg[i] = d_logistic(fgk[i]) * cp;
                        st[i][0] = cp;
                        settle(k_og[i], k_ce[i], carry[i], k_ni[i], k_ig[i], k_fg[i]);
                    }
                }
                fetch(s + 1);
                if (!first) {
                    const bool ok = mbar_wait_bounded<false>(z_full, (uint32_t)n_e & 1u, &give_up_s, WAIT_CYCLES);
                    ++n_e;
                    if (!__all_sync(0xffffffffu, ok)) { give_up_s = 1; atomicCAS(a.status, 0, (int)B2_ERR_STEP_TIMEOUT); break; }
                    if constexpr (BWD) {
                        const float *zp = reinterpret_cast<const float *>(zpart(ev + (unsigned)s, bidx, 0)) + ((seq(0) >> 2) * ROWS + ul) * 4 + (seq(0) & 3);
                        float v[CS][CPT], sum[CPT];
#pragma unroll
                        for (int src = 0; src < CS; ++src) load_l2(zp + (size_t)src * (G::ZSRC / 4), v[src]);
#pragma unroll
                        for (int i = 0; i < CPT; ++i) {
                            sum[i] = 0.0f;
#pragma unroll
                            for (int src = 0; src < CS; ++src) sum[i] += v[src][i];
                            x[i][0] += sum[i];
                        }
                    } else {
                        const float *z = reinterpret_cast<const float *>(gbase + G::F_Z);
#pragma unroll
                        for (int i = 0; i < CPT; ++i) {
                            const int n = seq(i);
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                const uint32_t o = (uint32_t)(((n >> 2) * ROWS + g * UPB + ul) * 4 + (n & 3));
                                float sum = 0.0f;
#pragma unroll
                                for (int src = 0; src < CS; ++src) sum += z[(size_t)src * (G::ZSRC / 4) + o];
                                x[i][BWD ? 0 : g] += sum;
                            }
                        }
                        __syncwarp();
                        if constexpr (G::CL == 1) {
                            if (lane == 0) mbar_arrive(z_free);
                        } else if (lane < CS) {
                            mbar_arrive_cluster_relaxed(map_to_rank(z_free, (uint32_t)lane));
                        }
                    }
                }
                unsigned char *dst = img + (size_t)((ev + (unsigned)s) & 1u) * G::NIMG * G::IMG;
                float o[CPT][6];
#pragma unroll
                for (int i = 0; i < CPT; ++i) {
                    const int n = seq(i);
                    const bool real = t < len[i] && unit;
                    if constexpr (!BWD) {
                        const float cp = st[i][0];
                        float ni = cl_tanh(x[i][0]), ig = cl_logistic(x[i][1] + cp * pw[0]), fg = cl_logistic(x[i][2] + cp * pw[1]);
                        float c = ni * ig + cp * fg;
                        float og = cl_logistic(x[i][3] + c * pw[2]), h = cl_tanh(c) * og;
                        if (!real) ni = ig = fg = og = c = h = 0.0f;
                        st[i][0] = c;
                        o[i][0] = ni; o[i][1] = ig; o[i][2] = fg; o[i][3] = og; o[i][4] = c; o[i][5] = h;
                        if (!last) {
                            // 8 units of sequence n sit in 8 adjacent lanes: their fp16 hi (lo) parts make one 16-byte chunk
                            const unsigned v = split_pair(h, S_H), y1 = __shfl_down_sync(0xffffffffu, v, 1);
                            const unsigned hp = (v & 0xffffu) | (y1 << 16), lp = (v >> 16) | (y1 & 0xffff0000u);
                            const unsigned h1 = __shfl_down_sync(0xffffffffu, hp, 2), h2 = __shfl_down_sync(0xffffffffu, hp, 4);
                            const unsigned h3 = __shfl_down_sync(0xffffffffu, hp, 6);
                            const unsigned l1 = __shfl_down_sync(0xffffffffu, lp, 2), l2 = __shfl_down_sync(0xffffffffu, lp, 4);
                            const unsigned l3 = __shfl_down_sync(0xffffffffu, lp, 6);
                            if ((ul & 7) == 0) {
                                const int unit0 = 32 * r + UPB * q + ul;        // first unit of the chunk
                                unsigned char *c16 = dst + (size_t)(unit0 >> 6) * G::IMG + (size_t)n * 128 + (size_t)((((unit0 & 63) >> 3) ^ (n & 7)) * 16);
                                *reinterpret_cast<uint4 *>(c16) = make_uint4(hp, h1, h2, h3);
                                *reinterpret_cast<uint4 *>(c16 + NC * 128) = make_uint4(lp, l1, l2, l3);
                            }
                        }
                    } else {
                        const float e = x[i][0], dog = k_og[i] * e;
                        float ce = k_ce[i] * e + pw[2] * dog + carry[i];
                        float dd[4] = {limited_error(k_ni[i] * ce), limited_error(k_ig[i] * ce), limited_error(k_fg[i] * ce), limited_error(dog)};
                        if (!real) ce = dd[0] = dd[1] = dd[2] = dd[3] = 0.0f;
                        st[i][1] = real ? fgk[i] : 0.0f; st[i][2] = ce; st[i][3] = dd[1]; st[i][4] = dd[2];
#pragma unroll
                        for (int g = 0; g < 4; ++g) o[i][g] = dd[g];
                        if (!last) {
                            // contraction position 4 * unit + gate: this thread's four gates are 8 bytes of each part
                            const unsigned v0 = split_pair(dd[0], S_D), v1 = split_pair(dd[1], S_D), v2 = split_pair(dd[2], S_D), v3 = split_pair(dd[3], S_D);
                            unsigned char *c8 = dst + (size_t)(j >> 4) * G::IMG + (size_t)n * 128 + (size_t)((((ul & 15) >> 1) ^ (n & 7)) * 16 + 8 * (ul & 1));
                            *reinterpret_cast<uint2 *>(c8) = make_uint2((v0 & 0xffffu) | (v1 << 16), (v2 & 0xffffu) | (v3 << 16));
                            *reinterpret_cast<uint2 *>(c8 + NC * 128) = make_uint2((v0 >> 16) | (v1 & 0xffff0000u), (v2 >> 16) | (v3 & 0xffff0000u));
                        }
                    }
                }
                if (!last) {
                    // this warp's part of the operand is on its way: hand it to the publisher.  The layer's own state is stored once the
                    // publisher is through, its fence and release would wait for these stores as well.
                    __syncwarp();
                    if (lane == 0) mbar_arrive(rel_full);
                    const bool ok = mbar_wait_bounded<false>(rel_free, (uint32_t)n_p & 1u, &give_up_s, WAIT_CYCLES);
                    ++n_p;
                    if (!__all_sync(0xffffffffu, ok)) { give_up_s = 1; atomicCAS(a.status, 0, (int)B2_ERR_STEP_TIMEOUT); break; }
                }
                if (unit)
#pragma unroll
                    for (int i = 0; i < CPT; ++i) {
                        const int pg = p0 + seq(i);
                        if (pg >= P) continue;
                        const size_t f = (size_t)t * P + pg;
                        float *ap = (BWD ? a.bf.deltas : a.bf.acts) + f * 4 * ls + u;
#pragma unroll
                        for (int g = 0; g < 4; ++g) ap[(size_t)g * ls] = o[i][g];
                        if constexpr (!BWD) {
                            a.bf.cells[f * ls + u] = o[i][4];
                            a.y[f * ls + u] = o[i][5];
                        }
                    }
            }
            // frames beyond the chunk's longest sequence
            if (unit)
                for (int i = 0; i < CPT; ++i) {
                    const int pg = p0 + seq(i);
                    if (pg >= P) continue;
                    for (int t = Tc; t < T; ++t) {
                        const size_t f = (size_t)t * P + pg;
                        if constexpr (BWD) {
#pragma unroll
                            for (int g = 0; g < 4; ++g) a.bf.deltas[f * 4 * ls + (size_t)g * ls + u] = 0.0f;
                        } else {
                            a.y[f * ls + u] = 0.0f;
                            a.bf.cells[f * ls + u] = 0.0f;
                        }
                    }
                }
        }
        if (Tc > 1) ev += (unsigned)(Tc - 1);
        __syncthreads();     // every role is through this work item
        if (give_up_s) break;
    }
    tc_fence_before();
    __syncthreads();
    if (give_up_s && tid == 0) atomicCAS(a.status, 0, (int)B2_ERR_STEP_TIMEOUT);
    if constexpr (G::CL > 1) cluster_sync_all();      // nobody leaves while a peer may still write into its shared memory
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

typedef void (*WideKernel)(WideArgs);
constexpr int NVARIANTS = 3, CHUNK[NVARIANTS] = {16, 32, 64};
struct Variant { WideKernel kern; int group, cluster, threads; size_t smem, xchg; };
template <int E, bool BWD, int NC>
constexpr Variant variant_of() {
    typedef Geo<E, BWD, NC> G;
    return Variant{lstm_wide_kernel<E, BWD, NC>, G::GROUP, G::CL, G::NTHR, G::smem(), G::GROUP_BYTES};
}
#define CHUNKS(E, BWD) {variant_of<E, BWD, 16>(), variant_of<E, BWD, 32>(), variant_of<E, BWD, 64>()}
const Variant VARIANTS[2][2][NVARIANTS] = {{CHUNKS(512, false), CHUNKS(512, true)}, {CHUNKS(1024, false), CHUNKS(1024, true)}};   // [wide][backward]

// groups that the current device holds at once, at most those the exchange buffers are made for
constexpr int MAX_GROUPS[2] = {8, 2};
int resident_groups(bool wide) {
    static std::mutex mu;
    static short known[MAX_DEVICES][2];      // 0 = not asked yet, else groups + 1
    const int dev = current_device();
    if (dev < 0) return 0;
    std::lock_guard<std::mutex> lk(mu);
    if (!known[dev][wide]) {
        int groups = std::min(MAX_GROUPS[wide], sm_count() / VARIANTS[wide][0][0].group);
        for (int i = 0; wide && i < NVARIANTS; ++i) {
            const Variant &v = VARIANTS[wide][0][i];
            const cluster::Launch l(v.group, v.threads, v.smem, v.cluster, true, nullptr);
            const int n = cluster::allow((const void *)v.kern, v.smem, v.cluster) ? cluster::resident((const void *)v.kern, l) : 0;
            groups = std::min(groups, v.cluster * n / v.group);
        }
        known[dev][wide] = (short)(groups + 1);
    }
    return known[dev][wide] - 1;
}
// The smallest chunk that leaves every group one work item (us per step on a B200, 1024 units, forward / backward: chunks of 16 4.5 / 6.0, of
// 32 5.4 / 7.0, of 64 7.6 / 7.7), else chunks of 64.
struct Plan { bool wide; int v, nchunks, groups; };
Plan make_plan(const LstmShape &s) {
    Plan p;
    p.wide = s.els > 512;
    const int room = resident_groups(p.wide), per_dir = room > s.D ? room / s.D : 1, share = (s.P + per_dir - 1) / per_dir;
    p.v = share <= 16 ? 0 : (share <= 32 ? 1 : 2);
    p.nchunks = (s.P + CHUNK[p.v] - 1) / CHUNK[p.v];
    p.groups = std::min(room, s.D * p.nchunks);
    return p;
}

}  // namespace

// measured on a B200: a step of the forward sweep and one of the backward sweep, for each work item of a group
double lstm_wide_step_us(const LstmShape &s) {
    static const double us[2][NVARIANTS] = {{10.5, 12.5, 17.3}, {10.5, 12.4, 15.3}};
    const Plan p = make_plan(s);
    return us[p.wide][p.v] * ((s.D * p.nchunks + p.groups - 1) / p.groups);
}

bool lstm_wide_supported(const LstmShape &s) { return s.els > 256 && s.els <= 1024 && s.P >= 1 && resident_groups(s.els > 512) >= 1; }

void lstm_wide_sizes(const LstmShape &s, size_t *exchange_bytes, size_t *flag_words) {
    const bool wide = s.els > 512;
    *exchange_bytes = 0;
    for (int b = 0; b < 2; ++b)
        for (int i = 0; i < NVARIANTS; ++i) *exchange_bytes = std::max(*exchange_bytes, MAX_GROUPS[wide] * VARIANTS[wide][b][i].xchg);
    *flag_words = (size_t)MAX_GROUPS[wide] * GROUP_FLAGS;
}

int lstm_wide_sweep(bool backward, const LstmShape &s, const LstmBuffers &b, const WideBuffers &wb, const float *w, float *y, const float *dy,
                    int *status, unsigned *tag_next, cudaStream_t st) {
    if (!lstm_wide_supported(s)) return 1;
    const Plan pl = make_plan(s);
    const Variant &v = VARIANTS[pl.wide][backward][pl.v];
    WideArgs a;
    a.sh = s; a.bf = b; a.w = w; a.y = y; a.dy = dy;
    a.img = wb.xchg; a.flags = wb.flags; a.status = status;
    a.tag_base = *tag_next;
    a.nchunks = pl.nchunks;
    B2_TRY(set_max_dynamic_smem((const void *)v.kern, (int)v.smem));
    const cluster::Launch l(pl.groups * v.group, v.threads, v.smem, v.cluster > 1 ? v.cluster : 0, true, st);
    B2_CUDA(cudaLaunchKernelEx(&l.cfg, v.kern, a));
    count_launch();
    *tag_next += (unsigned)(s.D * a.nchunks) * ((unsigned)s.T + 1u);
    return B2_OK;
}

}  // namespace b2
