// bpmax_strip.cuh -- R0 + R3 + R4 of a strip of outer cells, inner tables of width Np = 8*NB <= 64.
//
// The same triangular (max,+) product as r0_kernel (bpmax_r0.cuh: operands, cell images, warp
// programs, merge), for T neighbouring cells of one outer row at once: a job is the strip of cells
// (i1, i1+d+t), t = 0 .. T-1, of one pair and a range of offsets w = k1 - i1 in [w0, w1). For each
// k1 the T cells share the operand A = F(i1, k1), and their operands B_t = F(k1+1, i1+d+t) are
// neighbours in memory (row-major outer triangle), so one step of K values of k1 lands K images of A
// and K runs of T images of B with 2K bulk copies, (1+T)/(2T) of the bytes that T separate cells
// need. Cell t's offsets t <= w <= d-1 read only tables of diagonals < d (its B at offset w lies on diagonal
// d+t-1-w); the remaining ones, w < t and w >= d, are the first t of its offset pairs (w, d+t-1-w), and
// r0_kernel's, per diagonal.
//
// One CTA per SM: T groups of warps, group t computing cell t with the lane table and warp programs of
// the width class. A warp waits for a stage of the shared-memory ring, does its tasks and counts
// itself done with one mbarrier arrive; no warp waits for another within a job, except that one of
// them, the producing warp, also walks the jobs: it waits until every warp has left a stage, writes
// the stage's next record (valid k1, end of job, destination) and issues its copies. The warps of the
// T groups are placed so that every SM sub-partition gets about the same number of steps
// (c_strip_warp). (A producer warp of its own would cost the registers of four: 128 a thread, or the
// 160 / 32 split of setmaxnreg, which measured 1,116 cycles per item against 957.)
// Each group merges its cell's partial maxima in its own shared tile at the end of a job, as
// r0_kernel does; a group's warps meet on an mbarrier of their own. Every wait is bounded in time.
//
// Bound: the issue of packed adds and 3-input maxima, about 1.8 cycles per warp and term on one
// sub-partition with every operand in registers (the two share it: either alone issues every second
// cycle, and so do both together), 780 cycles per 64x64 item of 54,784 evaluated terms per SM; the
// tasks alone on resident stages take 835. Measured per item (M = 512, d = 244, 193,842 items): 957
// cycles, 943 with the copies left out; the refill's address arithmetic once took 105 of 1,092 (the
// whole ring waits for it), hence the cursor that only adds. r0_kernel took 1,240 with 20,160 bytes
// per item, against 13,440 here. Fill: 1024x64 766 -> 661 ms, the 512-pair batch 523 -> 460 ms;
// 661 -> 616 and 428 -> 424 since cell t takes every offset that meets final tables (before, only those that
// all T cells share); 601 -> 595.5 since lane 0 alone refills stages of one k1.
#pragma once
#include <cstddef>

#include "bpmax_r0.cuh"

namespace bpmax {

// one job: cells (i1, i1+d+t) of pair `pair`, offsets w in [w0, w1)
struct StripJob {
    int pair, i1, w0, w1;
};

// widths with a strip kernel (narrower ones keep r0_kernel alone)
constexpr int STRIP_MIN_NB = 2;
// cells per strip = consumer groups per CTA, R0_TAB_THREADS[NB] threads a group: 12 consumer warps
// (9 at NB = 2, whose two stages of 24 k1 leave no shared memory for a fourth cell)
__host__ __device__ constexpr int strip_cells(int nb) { return nb == 7 ? 4 : 3; }

// Strips are taken from this outer diagonal on: a job holds one strip's offsets, and with few of them
// most of a stage's K values of k1 stay empty (as in the T-1 stages of one k1 at its head), while the first offset
// pairs of the later cells are merged by r0_kernel besides. Fill ms with strips from diagonal 1 / 10 / 25 / 37 / 49 / 79 /
// never: 100 pairs 60x16 (K = 24) 5.78 / 5.78 / 5.12 / 4.75 / 4.55 / 4.54 / 4.55, 20 of 200x16 20.1 / 20.1 / 19.6 / 19.2 / 18.9 /
// 18.6 / 20.3; 30 of 90x24 (12) 5.87 / 5.87 / 5.58 / 5.50 / 5.49 / 5.71 / 5.72; 100 of 60x32 (6) 8.54 / 8.28 / 7.83 / 7.73 / 7.85 /
// 8.04 / 8.43; 30 of 90x48 (2) 12.0 / 11.9 / 11.8 / 11.9 / 12.1 / 12.3 / 12.3; 100 of 60x64 (1) 21.7 / 21.6 / 22.4 / 23.5 / 24.8 /
// 25.2 / 25.2.
__host__ __device__ constexpr int strip_min_d(int nb) { return nb >= 7 ? 9 : (nb >= 5 ? 25 : (nb == 4 ? 37 : (nb == 3 ? 49 : 79))); }

template <int NB>
struct StripCfg {
    static constexpr int GT = R0_TAB_THREADS[NB];  // threads per group
    static constexpr int GW = GT / 32;             // warps per group
    static constexpr int T = strip_cells(NB);      // groups = cells per strip
    static constexpr int CW = T * GW;              // consumer warps
    static constexpr int THREADS = 32 * CW;
    static constexpr int K = R0_TAB_ITEMS[NB];     // values of k1 per stage
    static constexpr int IMG = R0_TAB_COLBASE[NB][NB];
    // pitch of the A images and of the B runs of a stage (chunks): item slots of the lane table lie
    // 2*IMG+IPAD chunks apart, and the same distance modulo 8 keeps its bank groups
    static constexpr int ITEM = 2 * IMG + R0_TAB_IPAD[NB];
    static constexpr int PA = IMG + (ITEM - IMG % 8 + 8) % 8;
    static constexpr int PB = T * IMG + (ITEM - T * IMG % 8 + 8) % 8;
    static constexpr int OFF_B = K * PA;  // B runs of a stage (chunks)
    static constexpr int STAGE_BYTES = 16 * (K * PA + K * PB);
    static constexpr int NBLK = NB * (NB + 1) / 2;
    static constexpr int RED_WORDS = 65 * NBLK;  // merge tile of one group
    static constexpr int BUDGET = 227 * 1024 - 4 * T * RED_WORDS - 4 * NBLK - 512;
    static constexpr int STAGES = BUDGET / STAGE_BYTES < 6 ? BUDGET / STAGE_BYTES : 6;
    static constexpr int OFF_RED = STAGES * STAGE_BYTES;
    static constexpr int OFF_DST = OFF_RED + 4 * T * RED_WORDS;
    static constexpr int OFF_REC = (OFF_DST + 4 * NBLK + 15) / 16 * 16;  // stage records
    static constexpr int OFF_FULL = OFF_REC + 16 * STAGES;               // mbarriers: stage landed
    static constexpr int OFF_FREE = OFF_FULL + 8 * STAGES;               // stage read by every consumer warp
    static constexpr int OFF_GRP = OFF_FREE + 8 * STAGES;                // group merge
    static constexpr int OFF_ARM = OFF_GRP + 8 * T;                      // phases armed per stage
    static constexpr size_t SMEM = (size_t)OFF_ARM + 4 * STAGES;
    // the producing warp refills the stage it left LAG stages ago
    static constexpr int LAG = STAGES >= 4 ? 1 : 0;
    // the consumer warp that also produces: of the sub-partition with the fewest steps, a light program
    static constexpr int PW = GW == 3 ? CW - 1 : 10;
    static_assert(PA % 8 == ITEM % 8 && PB % 8 == ITEM % 8, "bank groups of the lane table");
    static_assert(STAGES >= 2 && SMEM <= 227 * 1024, "shared memory per CTA");
    static_assert(OFF_REC % 16 == 0 && OFF_FULL % 8 == 0, "shared-memory alignment");
};

// what a stage holds, written by the producing warp before it announces the stage's bytes
struct __align__(16) StripRec {
    int info;       // k1 values in the stage | cells of the strip that take them << 8; -1: no more stages
    int last;       // the job ends with this stage
    long long out;  // float offset of the table of cell t = 0 (the others follow it)
};

// the producing warp's position, in shared memory (the product tile leaves no registers for it)
struct __align__(16) StripCursor {
    unsigned long long a_src, b_src;  // next A image and next run of B images (byte addresses)
    int left, w;                      // k1 of the job still to be produced, offset of the next
    int b_step;                       // cells from one run of B images to the next (one less each time)
    int pair, job;                    // job >= njobs: no more; 0x7fffffff once the closing record is out
    long long out;                    // float offset of the table of cell t = 0
    int cells;                        // cells of the strip inside the table
    alignas(16) StripJob next;        // prefetched (16 bytes by cp.async): the job gridDim.x further on
    unsigned long long F_pair;        // byte address of the pair's tables
    int M;
};

static_assert(sizeof(StripJob) == 16 && offsetof(StripCursor, next) % 16 == 0, "cp.async of the next job");

// (group, table warp) of consumer warp c, whose SM sub-partition is c % 4: the warp programs' step
// counts (128, 92, 80, 49) summed per sub-partition come to at most 336 for programs 0 0 1 2 (mean
// 321), 269 for 0 1 2 3 (mean 262) and are equal for groups of three warps
__constant__ unsigned char c_strip_warp[4][12][2] = {
    // 4 warps a group, programs 0 0 1 2
    {{0, 0}, {0, 1}, {2, 0}, {2, 1}, {1, 1}, {1, 0}, {0, 2}, {1, 2}, {2, 3}, {0, 3}, {1, 3}, {2, 2}},
    // 4 warps a group, programs 0 1 2 3
    {{0, 0}, {1, 0}, {2, 0}, {2, 1}, {0, 1}, {1, 1}, {0, 2}, {1, 2}, {0, 3}, {1, 3}, {2, 3}, {2, 2}},
    // 3 warps a group, four groups
    {{0, 0}, {1, 0}, {2, 0}, {3, 0}, {0, 1}, {1, 1}, {2, 1}, {3, 1}, {0, 2}, {1, 2}, {2, 2}, {3, 2}},
    // 3 warps a group, three groups
    {{0, 0}, {1, 0}, {2, 0}, {0, 1}, {1, 1}, {2, 1}, {0, 2}, {1, 2}, {2, 2}}};

__device__ __forceinline__ void mbar_arrive(unsigned bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// mbar_wait with one outcome for the whole warp
__device__ __forceinline__ bool mbar_wait_warp(unsigned bar, unsigned parity, unsigned long long limit_ns)
{
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
    const unsigned long long t0 = globaltimer_ns();
    while (true) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
        if (__any_sync(0xffffffffu, globaltimer_ns() - t0 > limit_ns)) return false;
    }
}

template <int NB>
__global__ void __launch_bounds__(StripCfg<NB>::THREADS, 1)
r0_strip_kernel(const StripJob *__restrict__ jobs, int njobs, const PairDesc *__restrict__ pairs, float *__restrict__ F,
                int d, WaitCtl ctl)
{
    using C = StripCfg<NB>;
    constexpr int S = C::STAGES;
    constexpr long long CELL = 4LL * C::IMG;
    extern __shared__ __align__(128) float r0sm[];
    char *sm = reinterpret_cast<char *>(r0sm);
    int *red = reinterpret_cast<int *>(sm + C::OFF_RED);
    int *red_dst = reinterpret_cast<int *>(sm + C::OFF_DST);
    StripRec *rec = reinterpret_cast<StripRec *>(sm + C::OFF_REC);
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + C::OFF_FULL);
    int *armed = reinterpret_cast<int *>(sm + C::OFF_ARM);
    const unsigned full_u = smem_u32(full), free_u = smem_u32(sm + C::OFF_FREE), grp_u = smem_u32(sm + C::OFF_GRP);
    __shared__ StripCursor cur;  // the producer's position (shared memory: no registers beside the product tile)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(full_u + 8 * s, 1);
            mbar_init(free_u + 8 * s, C::CW);
            armed[s] = 0;
        }
        for (int g = 0; g < C::T; ++g) mbar_init(grp_u + 8 * g, C::GW);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int q = tid; q < C::T * C::RED_WORDS; q += C::THREADS) red[q] = 0;  // +0: below every partial maximum
    if (tid < C::NBLK) {
        int BI, BJ;
        blk_decode(NB, tid, BI, BJ);
        red_dst[tid] = 4 * (c_img_colbase[NB][BJ] + 17 * BI);
    }
    // cell_index in 32 bits: exact, since the triangle of M <= 65535 rows has fewer than 2^31 cells
    auto cell32 = [](unsigned M, unsigned i, unsigned j) { return i * M - i * (i - 1) / 2 + (j - i); };
    // the producing lane moves its cursor to job j, jb, and fetches the record of the one after it into
    // cur.next (jb is a copy: it may come from there)
    auto open_job = [&](int j, const StripJob jb) {
        cur.job = j;
        if (j >= njobs) return;
        if (j + (int)gridDim.x < njobs) cp_async16(&cur.next, jobs + j + gridDim.x);
        cp_async_commit();
        if (jb.pair != cur.pair) {
            cur.pair = jb.pair;
            cur.M = pairs[jb.pair].M;
            cur.F_pair = (unsigned long long)(F + pairs[jb.pair].F_off);
        }
        const int M = cur.M, j1 = jb.i1 + d, k1 = jb.i1 + jb.w0;
        cur.a_src = cur.F_pair + (unsigned long long)cell32(M, jb.i1, k1) * (4 * CELL);
        cur.b_src = cur.F_pair + (unsigned long long)cell32(M, k1 + 1, j1) * (4 * CELL);
        cur.b_step = M - k1 - 2;  // from row k1+1 to row k1+2
        cur.left = jb.w1 - jb.w0;
        cur.w = jb.w0;
        const float *out = reinterpret_cast<const float *>(cur.F_pair) + cell32(M, jb.i1, j1) * CELL;
        cur.out = out - F;
        cur.cells = min(C::T, M - j1);
    };
    // the producing warp fills a free stage with the next K k1 of its jobs; after the last, the closing
    // record that lets the warps leave. With one k1 a stage (K == 1) lane 0 alone does this and nothing else
    // touches the cursor; otherwise every lane issues copies, and lane 0 moves the cursor once all have read it.
    auto produce_lanes = [&](int stage) {
        const int job = cur.job, left = cur.left, b_step = cur.b_step, w = cur.w;
        const unsigned long long a_src = cur.a_src, b_src = cur.b_src;
        // offsets below a cell's place in the strip are not its: one k1 a stage there, for cells 0 .. w
        const int valid = C::K == 1 || w < C::T - 1 ? 1 : min(C::K, left), cells = min(cur.cells, w + 1);
        const long long out = cur.out;
        if constexpr (C::K > 1) __syncwarp();  // every lane has read the cursor
        if (job >= njobs) {
            if (lane == 0 && job != 0x7fffffff) {
                rec[stage].info = -1;
                mbar_arrive(full_u + 8 * stage);
                armed[stage] += 1;
                cur.job = 0x7fffffff;
            }
            return;
        }
        const unsigned bar = full_u + 8 * stage, dst = smem_u32(sm) + stage * C::STAGE_BYTES;
        if (lane == 0) {
            rec[stage] = StripRec{valid | cells << 8, left == valid, out};
            mbar_arrive_tx(bar, (unsigned)(valid * (1 + cells) * C::IMG * 16));
            armed[stage] += 1;
            cur.left = left - valid;
            cur.w = w + valid;
            cur.a_src = a_src + valid * 4 * CELL;
            // `valid` steps of b_step, b_step - 1, ... cells
            cur.b_src = b_src + (long long)(valid * b_step - valid * (valid - 1) / 2) * (4 * CELL);
            cur.b_step = b_step - valid;
        }
        if constexpr (C::K > 1) __syncwarp();  // the bytes are announced
        for (int kk = lane; kk < valid; kk += 32) {
            bulk_g2s(dst + 16 * (kk * C::PA), reinterpret_cast<const void *>(a_src + kk * 4 * CELL),
                     (unsigned)(C::IMG * 16), bar);
            bulk_g2s(dst + 16 * (C::OFF_B + kk * C::PB),
                     reinterpret_cast<const void *>(b_src + (long long)(kk * b_step - kk * (kk - 1) / 2) * (4 * CELL)),
                     (unsigned)(cells * C::IMG * 16), bar);
        }
        if (lane == 0 && left == valid) {
            cp_async_wait<0>();
            open_job(job + gridDim.x, cur.next);
        }
    };
    auto produce = [&](int stage) {
        if (C::K > 1 || lane == 0) produce_lanes(stage);
        __syncwarp();
    };
    if (warp == C::PW) {
        if (lane == 0) {
            cur.pair = -1;
            open_job(blockIdx.x, jobs[blockIdx.x]);
        }
        __syncwarp();
    }
    __syncthreads();
    chain_wait();
    if (warp == C::PW && !ctl.inject)
        for (int s = 0; s < S; ++s) produce(s);

    constexpr int MAP = C::GW == 3 ? (C::T == 4 ? 2 : 3) : (R0_TAB_ROLE[NB][1] == 0 ? 0 : 1);
    const int grp = c_strip_warp[MAP][warp][0], tw = c_strip_warp[MAP][warp][1];
    const int role = (int)(R0Cfg<NB>::ROLE_BITS >> (2 * tw)) & 3;
    const unsigned char *lt = c_r0_lane[NB - 1][32 * tw + lane];
    const bool has_task = lt[0] != 255;
    const int tg = has_task ? lt[0] : 0, bi = lt[1], bj = lt[2], kb = lt[3];
    int a_off = 0, b_off = 0, red_off = 0;
    if (has_task) {
        red_off = grp * C::RED_WORDS + 65 * (bi * NB - bi * (bi - 1) / 2 + (bj - bi));
        a_off = 4 * (tg * C::PA + c_img_colbase[NB][kb] + 17 * bi);
        b_off = 4 * (C::OFF_B + tg * C::PB + grp * C::IMG + c_img_colbase[NB][bj] + 17 * kb + 2);
    }
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = NEG_INF;
    int stage = 0;
    unsigned phase = 0;  // parity of the ring's current round
    bool refills = false;  // the producing warp has LAG stages behind it
    // a wait that runs out ends its warp's work; the waits of the others (for the stages or copies that
    // this warp no longer frees or issues, or for its group) then run out too
    bool bad = false;
#pragma unroll 1
    while (true) {
        if (!mbar_wait_warp(full_u + 8 * stage, phase, ctl.wait_ns)) {
            bad = true;
            break;
        }
        const int info = rec[stage].info;
        if (info < 0) break;
        const bool in = grp < info >> 8;
        if (has_task && in && (C::K == 1 || tg < (info & 0xff))) {
            const float *st = r0sm + stage * (C::STAGE_BYTES / 4);
            const float *As = st + a_off, *Bs = st + b_off;
            if (role == 0)
                r0_task<0>(As, Bs, acc);
            else if (role == 1)
                r0_task<1>(As, Bs, acc);
            else if (role == 2)
                r0_task<2>(As, Bs, acc);
            else
                r0_task<3>(As, Bs, acc);
            if (kb == bi) {  // k = 8bi-1 term of row 8bi: S1(i1,k1) + B[8bi][j2]
                const float s1a = st[4 * tg * C::PA + 8];  // A[1][0] = S1(i1,k1)
                const float4 r0 = *reinterpret_cast<const float4 *>(Bs - 8);
                const float4 r1 = *reinterpret_cast<const float4 *>(Bs - 4);
                const float rv[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[0][j] = fmaxf(acc[0][j], s1a + rv[j]);
            }
        }
        const bool last = rec[stage].last != 0;
        const long long out_off = rec[stage].out + grp * CELL;
        __syncwarp();
        if (lane == 0) mbar_arrive(free_u + 8 * stage);
        if (warp == C::PW) {  // refill the stage this warp left LAG stages ago, once every warp has
            const bool wrap = stage < C::LAG;
            const int s = wrap ? stage - C::LAG + S : stage - C::LAG;
            if (C::LAG == 0 || refills) {
                if (!mbar_wait_warp(free_u + 8 * s, phase ^ (wrap ? 1u : 0u), ctl.wait_ns)) {
                    bad = true;
                    break;
                }
                produce(s);
            }
            refills = true;
        }
        if (++stage == S) {
            stage = 0;
            phase ^= 1u;
        }
        if (last && in) {  // job done: merge the group's partial maxima into F(i1, i1+d+grp)
            // (entries past N or below the subdiagonal are -inf; one on the subdiagonal, S1 + S1, may
            // land in the table, where the finalize does not read it and stores S1)
            if (has_task) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int v = __float_as_int(acc[i][j]);
                        if (v > 0) atomicMax(red + red_off + 8 * i + j, v);
                        acc[i][j] = NEG_INF;
                    }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(grp_u + 8 * grp);
            if (!mbar_wait_warp(grp_u + 8 * grp, 0, ctl.wait_ns)) {
                bad = true;
                break;
            }
            int *out = reinterpret_cast<int *>(F + out_off), *rt = red + grp * C::RED_WORDS;
            for (int e = 32 * tw + lane; e < 64 * C::NBLK; e += C::GT) {
                const int q = e >> 6, x = e & 63;
                const int v = rt[65 * q + x];
                if (v > 0) {
                    atomicMax(out + red_dst[q] + x, v);
                    rt[65 * q + x] = 0;
                }
            }
            __syncwarp();  // the tile is clear before any warp of the group merges its next job
            if (lane == 0) mbar_arrive(grp_u + 8 * grp);
            if (!mbar_wait_warp(grp_u + 8 * grp, 1, ctl.wait_ns)) {
                bad = true;
                break;
            }
        }
    }
    // no copy may be in flight into the shared memory of a finished CTA: after a timeout, wait
    // (bounded) for the last armed phase of every stage; otherwise every stage has been waited for
    if (__syncthreads_or(bad) && tid == 0) {
        atomicExch(ctl.err, 1);
        mbar_drain(full, armed, S, ctl.wait_ns);
    }
}

}  // namespace bpmax
