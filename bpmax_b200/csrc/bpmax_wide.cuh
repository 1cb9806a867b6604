// bpmax_wide.cuh -- the R0 + R3 + R4 product kernel for inner tables stored as tile images
// (Np = 64 * NT > 64; layout in bpmax_kernels.cuh).
//
// The triangular (max,+) product of one item of the width-64 kernel (bpmax_r0.cuh),
//   max_{k in [i2-1, j2]} A[i2][k] + Bs[k][j2]      (R0, and R3 / R4 through S1 on the subdiagonals)
// splits over tiles: output tile (BI, BJ) takes the k tiles KB in [BI, BJ], item (k1, KB) being
// A = tile (BI, KB) of F(i1, k1) and B = tile (KB, BJ) of F(k1+1, j1) (every k outside [i2-1, j2] meets
// a -inf below a diagonal, and the k = 64 BI - 1 term of tile row BI's first row is the R3 step of
// the width-64 kernel: S1(i1, k1) + B[64 BI][j2], B's local row 0). Items are of four kinds:
//   DD  BI = BJ (= KB): both diagonal tiles, exactly an item of the width-64 kernel (its lane table
//       and warp programs);
//   DA  KB = BI < BJ: A diagonal, B dense;   F  BI < KB < BJ: both dense;   DB  BI < KB = BJ: B diagonal.
// A job is one output tile of one outer cell and a range of k1 offset pairs (w, d-1-w) as in the
// width-64 kernel; for each k1 it walks KB = BI .. BJ. Per item two bulk copies (cp.async.bulk, the
// whole A tile image and the whole B tile image) land in a stage of a shared-memory ring counted on
// the stage's mbarrier, with the width-64 kernel's refill scheme (the last warp done with a stage
// refills it; no CTA barrier per item) and bounded waits. In off-diagonal jobs each lane owns one
// 8x8 micro-tile of the output tile (two lanes per micro-tile) and takes, per item, part of its k
// blocks (wide_tables.inc). At the end of a job every lane merges its partial maxima into the
// output tile with global atomicMax on the bit patterns (exact: every value is >= +0; -inf and +0
// partials are skipped), so jobs of one tile commute.
#pragma once
#include "bpmax_r0.cuh"

namespace bpmax {

// float offset of the dense tile (I, J), I < J, among the S2 images of a pair
__host__ __device__ __forceinline__ long long s2_image_off(int NT, int I, int J)
{
    return ((long long)I * (NT - 1) - (long long)I * (I - 1) / 2 + (J - I - 1)) * (4LL * WIDE_DENSE_CHUNKS);
}

// R1 and R2 over finished tiles of the cell itself are items of the same form: S2 is the table of an
// empty strand-1 interval, so R1 is A = tile (BI, KB) of F(i1, j1), B = tile (KB, BJ) of S2, KB = BI .. BJ-1,
// and R2 is A = tile (BI, KB) of S2, B = tile (KB, BJ) of F(i1, j1), KB = BI+1 .. BJ (S2 as dense tile
// images with halo pieces; the one k between the two, 64(BI+1)-1 of R2, is left to tile_final_kernel).
//
// Output tiles of the last tile column hold only nbc = ceil((N - 64 BJ) / 8) block columns of the table: their
// jobs give every micro-tile of those columns wide_split(nbc) lanes instead of 2 and leave the rest of
// the tile out (it is -inf), in the copies too, so a strand 2 of 130 costs little more than one of 128
// (90x130: 16.6 -> 12.1 ms of products).
//
// one job: output tile (BI, BJ) (tile = nbc << 16 | BI << 8 | BJ) of cell (i1, i1+d) of pair `pair`, k1 offset
// pairs p in [p0, p1) (offsets w = p and d-1-p, as R0Job); with p0 < 0 the R1/R2 items n in [-1-p0, p1),
// the BJ-BI of R1 first
struct R0JobW {
    int pair, i1, d, tile, p0, p1;
};

// lanes per micro-tile in output tiles of nbc block columns (8 nbc micro-tiles on 128 lanes), and what an
// item of such a tile costs, in 1/16 of a full one (warps times steps of a lane)
__host__ __device__ constexpr int wide_split(int nbc)
{
    return nbc <= 2 ? 8 : (nbc == 3 ? 5 : (nbc == 4 ? 4 : (nbc == 5 ? 3 : 2)));
}
constexpr int wide_cost(int nbc)
{
    return (8 * nbc * wide_split(nbc) + 31) / 32 * ((8 + wide_split(nbc) - 1) / wide_split(nbc));
}

// Shape variants: STAGES = 2 keeps three CTAs per SM (168 registers), 3 two CTAs per SM.
template <int STAGES_>
struct WideCfg {
    static constexpr int THREADS = 128;
    static constexpr int STAGES = STAGES_;
    static constexpr int SLOT = WIDE_DENSE_CHUNKS;  // chunks of one operand slot (a dense image fits)
    static constexpr int STAGE_BYTES = 2 * SLOT * 16;
    static constexpr int OFF_BAR = STAGES * STAGE_BYTES;
    static constexpr int OFF_CNT = OFF_BAR + 8 * STAGES;
    static constexpr int OFF_ARM = OFF_CNT + 4 * STAGES;
    static constexpr size_t SMEM = (size_t)OFF_ARM + 4 * STAGES;
    static constexpr int MINB = STAGES <= 2 ? 3 : 2;  // CTAs per SM the shared memory allows
    static constexpr int WARPS = THREADS / 32;
    static_assert(STAGE_BYTES % 16 == 0 && OFF_BAR % 8 == 0, "shared-memory alignment");
    static_assert((SMEM + 1024) * MINB <= 228 * 1024, "shared memory per SM");
};

template <int STAGES>
__global__ void __launch_bounds__(128, WideCfg<STAGES>::MINB)
r0_wide_kernel(const R0JobW *__restrict__ jobs, int njobs, const PairDesc *__restrict__ pairs, float *__restrict__ F,
               const float *__restrict__ Sa, WaitCtl ctl)
{
    using C = WideCfg<STAGES>;
    constexpr int S = STAGES;
    extern __shared__ __align__(128) float wsm[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(reinterpret_cast<char *>(wsm) + C::OFF_BAR);
    int *done_cnt = reinterpret_cast<int *>(reinterpret_cast<char *>(wsm) + C::OFF_CNT);
    int *armed = reinterpret_cast<int *>(reinterpret_cast<char *>(wsm) + C::OFF_ARM);
    const int tid = threadIdx.x, lane = tid & 31;
    int jid = blockIdx.x;
    if (jid >= njobs) return;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(bars + s), 1);
            done_cnt[s] = 0;
            armed[s] = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    const unsigned smem_base = smem_u32(wsm);
    auto job_items = [&](const R0JobW &jb) {
        if (jb.p0 < 0) return jb.p1 + 1 + jb.p0;
        return r0_job_items(R0Job{jb.pair, jb.i1, jb.p0, jb.p1}, jb.d) * ((jb.tile & 0xff) - (jb.tile >> 8 & 0xff) + 1);
    };
    // the producer's current job, one copy per warp in shared memory, refreshed when the warp's producer
    // position moves to another job (as in r0_kernel: no dependent global loads per refill). A refill is
    // in the way of the whole ring, so its addresses take 32-bit arithmetic on these: a pair's triangle has
    // fewer than 2^31 cells and a table fewer than 2^31 chunks.
    struct PJob {
        unsigned long long F, S2;  // byte addresses of the pair's tables and of its S2 images
        unsigned cell;             // bytes of a table
        int M, NT, i1, d, p0, tile;
    };
    __shared__ PJob pjob_sh[C::WARPS];
    const int warp_id = tid >> 5;
    auto load_pjob = [&](int j_) {
        __syncwarp();  // every lane of the warp is done with the previous copy
        if (lane == 0) {
            const R0JobW jb = jobs[j_];
            const PairDesc *pd = pairs + jb.pair;
            const int NT = pd->Np >> 6;
            pjob_sh[warp_id] = PJob{(unsigned long long)(F + pd->F_off), (unsigned long long)(Sa + pd->S2x_off),
                                    (unsigned)(4 * wide_cell_floats(NT)), pd->M, NT, jb.i1, jb.d, jb.p0, jb.tile};
        }
        __syncwarp();
    };
    // arms stage s for the producer's item (k1 number pk of the job's, k tile pkb of it; R1/R2: pk) and
    // issues its two copies (one thread)
    auto fill_stage = [&](int s, int pk, int pkb) {
        constexpr unsigned SD = WIDE_DIAG_CHUNKS, SQ = WIDE_DENSE_CHUNKS;
        const PJob &jb = pjob_sh[warp_id];
        const int M = jb.M, NT = jb.NT, i1 = jb.i1, j1 = i1 + jb.d, p0 = jb.p0, tile = jb.tile;
        const int BI = tile >> 8 & 0xff, BJ = tile & 0xff, nbc = tile >> 16;
        auto cell = [&](unsigned i, unsigned j) { return i * M - i * (i - 1) / 2 + (j - i); };
        auto row = [&](unsigned I) { return I * (2 * NT - 1 - I) / 2; };  // dense tiles before tile row I
        auto chunk = [&](unsigned I, unsigned J) { return I * SD + row(I) * SQ + (J > I ? SD + (J - I - 1) * SQ : 0); };
        unsigned long long A, B;
        bool a_diag, b_diag;
        if (p0 >= 0) {
            const int p = p0 + (pk >> 1), k1 = i1 + (pk & 1 ? jb.d - 1 - p : p), KB = BI + pkb;
            A = jb.F + (unsigned long long)cell(i1, k1) * jb.cell + 16ull * chunk(BI, KB);
            B = jb.F + (unsigned long long)cell(k1 + 1, j1) * jb.cell + 16ull * chunk(KB, BJ);
            a_diag = pkb == 0;
            b_diag = KB == BJ;
        } else {
            const int m = pk - 1 - p0, t = BJ - BI;
            const unsigned long long Fc = jb.F + (unsigned long long)cell(i1, j1) * jb.cell;
            auto image = [&](unsigned I, unsigned J) { return jb.S2 + 16ull * SQ * (row(I) + J - I - 1); };
            A = m < t ? Fc + 16ull * chunk(BI, BI + m) : image(BI, BI + 1 + m - t);
            B = m < t ? image(BI + m, BJ) : Fc + 16ull * chunk(BI + 1 + m - t, BJ);
            a_diag = m == 0;
            b_diag = m == 2 * t - 1;
        }
        unsigned ab = a_diag ? SD : SQ, bb = b_diag ? SD : SQ;  // chunks to copy
        if (nbc < 8) {  // of a tile of the last column, its nbc block columns (a prefix of the image)
            bb = b_diag ? c_img_colbase[8][nbc] : c_wide_dense_colbase[nbc];
            if (b_diag) ab = a_diag ? c_img_colbase[8][nbc] : c_wide_dense_colbase[nbc];
        }
        const unsigned bar = smem_u32(bars + s);
        mbar_arrive_tx(bar, 16 * (ab + bb));
        armed[s] += 1;
        const unsigned dst = smem_base + (unsigned)(s * C::STAGE_BYTES);
        bulk_g2s(dst, reinterpret_cast<const void *>(A), 16 * ab, bar);
        bulk_g2s(dst + 16 * C::SLOT, reinterpret_cast<const void *>(B), 16 * bb, bar);
    };

    // consumer position (job jid, item it of items) and producer position S items ahead
    int items = job_items(jobs[jid]), it = 0;
    int pj = jid, pitems = items, pk = 0, pkb = 0;
    // the producer's advance (every warp the same way) also refreshes the warp's copy of its job
    auto advance_p = [&]() {
        --pitems;
        if (pjob_sh[warp_id].p0 < 0 || ++pkb > (pjob_sh[warp_id].tile & 0xff) - (pjob_sh[warp_id].tile >> 8 & 0xff)) {
            pkb = 0;
            ++pk;
        }
        if (pitems == 0) {
            pk = 0;
            pkb = 0;
            pj += gridDim.x;
            if (pj < njobs) {
                pitems = job_items(jobs[pj]);
                load_pjob(pj);
            }
        }
    };
    load_pjob(pj);
    chain_wait();
    for (int s = 0; s < S; ++s)
        if (pj < njobs) {
            if (tid == 0 && !ctl.inject) fill_stage(s, pk, pkb);
            advance_p();
        }

    // the lane's task: DD jobs use the width-64 kernel's lane table and warp programs (task (bi, bj,
    // kb) packed as bi | bj << 4 | kb << 8, or -1 for an idle lane); the other jobs the micro-tile
    // table of wide_tables.inc (bi | bj << 4 | h << 8)
    const int warp_role = (int)(R0Cfg<8>::ROLE_BITS >> (2 * (tid >> 5))) & 3;
    const int dd_task = c_r0_lane[7][tid][0] == 255
                            ? -1
                            : (c_r0_lane[7][tid][1] | c_r0_lane[7][tid][2] << 4 | c_r0_lane[7][tid][3] << 8);
    const int full_task = c_tile_lane[tid][0] | c_tile_lane[tid][1] << 4 | c_tile_lane[tid][2] << 8;
    // the lane's micro-tile and share of its k blocks in a job's output tile (-1: none)
    auto tile_task = [&](int tile) {
        const int nbc = tile >> 16;
        if (nbc == 8) return full_task;
        const int h = tid / (8 * nbc), m = tid - 8 * nbc * h;
        return h < wide_split(nbc) ? (m & 7) | (m >> 3) << 4 | h << 8 : -1;
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = NEG_INF;

    unsigned phase = 0;
    int stage = 0;
    bool bad = false;  // as in r0_kernel: a wait ran out; no more copies, leave at the next job end
    // the job's output tile; k tile of the item = BI + kbi; first R1/R2 item of the job (-1: R0 items)
    int tile = jobs[jid].tile, mt_task = tile_task(tile), slab = jobs[jid].p0 < 0 ? -1 - jobs[jid].p0 : -1, kbi = 0;
#pragma unroll 1
    while (true) {
        const int BI = tile >> 8 & 0xff, BJ = tile & 0xff;
        if (slab >= 0) kbi = slab + it < BJ - BI ? slab + it : slab + it - (BJ - BI) + 1;
        const int KB = BI + kbi;
        if (!bad && !mbar_wait(smem_u32(bars + stage), (phase >> stage) & 1u, ctl.wait_ns)) {
            atomicExch(ctl.err, 1);
            bad = true;
        }
        phase ^= 1u << stage;
        if (!bad) {
            const float *As = wsm + (size_t)stage * (C::STAGE_BYTES / 4);
            const float *Bs = As + 4 * C::SLOT;
            if (BI == BJ) {  // DD: one task of the width-64 table per lane
                if (dd_task >= 0) {
                    const int bi = dd_task & 15, bj = (dd_task >> 4) & 15, kb = dd_task >> 8;
                    const float *a = As + 4 * (c_img_colbase[8][kb] + 17 * bi);
                    const float *b = Bs + 4 * (c_img_colbase[8][bj] + 17 * kb + 2);
                    if (warp_role == 0)
                        r0_task<0>(a, b, acc);
                    else if (warp_role == 1)
                        r0_task<1>(a, b, acc);
                    else if (warp_role == 2)
                        r0_task<2>(a, b, acc);
                    else
                        r0_task<3>(a, b, acc);
                    if (kb == bi) {  // k = 8bi-1 term of row 8bi: S1(i1,k1) + B[8bi][j2]
                        const float s1a = As[8];
                        const float *r3 = Bs + 4 * (c_img_colbase[8][bj] + 17 * bi);
                        const float4 r0 = *reinterpret_cast<const float4 *>(r3);
                        const float4 r1 = *reinterpret_cast<const float4 *>(r3 + 4);
                        const float rv[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[0][j] = fmaxf(acc[0][j], s1a + rv[j]);
                    }
                }
            } else if (mt_task >= 0) {
                const int bi = mt_task & 15, bj = (mt_task >> 4) & 15, h = mt_task >> 8;
                const bool a_diag = KB == BI, b_diag = KB == BJ;
                int k0 = 4 * h, k1 = k0 + 4, dk = 1;  // k blocks of the lane
                if (tile >> 16 < 8) {
                    k0 = (a_diag ? bi : 0) + h;
                    k1 = b_diag ? bj + 1 : 8;
                    dk = wide_split(tile >> 16);
                } else if (a_diag || b_diag) {
                    const int lo = a_diag ? bi : 0, cnt = a_diag ? 8 - bi : bj + 1, half = (cnt + 1) >> 1;
                    k0 = h == 0 ? lo : lo + half;
                    k1 = h == 0 ? lo + half : lo + cnt;
                }
                const float *bcol = Bs + 4 * ((b_diag ? c_img_colbase[8][bj] : c_wide_dense_colbase[bj]) + 2);
#pragma unroll 1
                for (int kb = k0; kb < k1; kb += dk)
                    r0_task<0>(As + 4 * ((a_diag ? c_img_colbase[8][kb] : c_wide_dense_colbase[kb]) + 17 * bi),
                               bcol + 4 * 17 * kb, acc);
                if (a_diag && h == 0) {  // kb == bi is the first block of this lane: the k = 8bi-1 term
                    const float s1a = As[8];
                    const float *r3 = bcol + 4 * (17 * bi - 2);
                    const float4 r0 = *reinterpret_cast<const float4 *>(r3);
                    const float4 r1 = *reinterpret_cast<const float4 *>(r3 + 4);
                    const float rv[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[0][j] = fmaxf(acc[0][j], s1a + rv[j]);
                }
            }
        }
        // the last warp done with this stage refills it with the item S ahead (not after a timeout)
        __syncwarp();
        int last = 0;
        if (lane == 0) last = atomicAdd(done_cnt + stage, 1) == C::WARPS - 1;
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last) {
            const bool refill = pj < njobs && !__any_sync(0xffffffffu, bad);  // (test mode: every warp is bad)
            if (lane == 0) {
                done_cnt[stage] = 0;
                if (refill) fill_stage(stage, pk, pkb);
            }
        }
        if (pj < njobs) advance_p();
        if (++kbi > BJ - BI) kbi = 0;
        if (++it >= items) {  // job done: merge the partial maxima into the output tile
            const R0JobW job = jobs[jid];
            const PairDesc pd = pairs[job.pair];
            const int NT = pd.Np >> 6;
            float *out = F + pd.F_off + cell_index(pd.M, job.i1, job.i1 + job.d) * wide_cell_floats(NT) +
                         wide_tile_off(NT, BI, BJ);
            const int task = BI == BJ ? dd_task : mt_task;
            if (task >= 0) {
                const int bi = task & 15, bj = (task >> 4) & 15;
                int *o = reinterpret_cast<int *>(out) +
                         4 * ((BI == BJ ? c_img_colbase[8][bj] : c_wide_dense_colbase[bj]) + 17 * bi);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int i2 = 64 * BI + 8 * bi + i, j2 = 64 * BJ + 8 * bj + j;
                        const int v = __float_as_int(acc[i][j]);
                        if (i2 <= j2 && j2 < pd.N && v > 0) atomicMax(o + 8 * i + j, v);
                        acc[i][j] = NEG_INF;
                    }
            }
            if (__syncthreads_or(bad)) {  // no thread arms or issues from here on
                if (tid == 0) mbar_drain(bars, armed, S, ctl.wait_ns);
                return;
            }
            jid += gridDim.x;
            if (jid >= njobs) break;
            const R0JobW nx = jobs[jid];
            items = job_items(nx);
            tile = nx.tile;
            mt_task = tile_task(tile);
            slab = nx.p0 < 0 ? -1 - nx.p0 : -1;
            it = 0;
            kbi = 0;
        }
        stage = (stage + 1) % S;
    }
}

}  // namespace bpmax
