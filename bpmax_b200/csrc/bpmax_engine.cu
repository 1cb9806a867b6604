// bpmax_engine.cu -- host side of the B200 BPMax fill: device arenas, the outer-diagonal
// schedule, CUDA-graph capture, and the C ABI declared in include/bpmax_gpu.h.
//
// Schedule of one fill (any number of pairs of uneven lengths, batched on one stream):
//   clear F; single-strand tables S1, S2 of every pair;
//   for d = 0 .. max(M)-1:                     (outer wavefront over j1-i1, V3/bpmax.c:300-323)
//     R0+R3+R4 product kernel over the cells (i1, i1+d) of every pair with M > d: jobs of k1
//       offset pairs (w, d-1-w), ordered by offset pair so both uses of a table meet in L2; from a
//       certain size on, the strip kernel takes most offsets of several diagonals in one launch;
//     finalize kernel over the same cells (init, SW1, inner R1/R2/SW2 wavefront).
// A plan's first run launches the sequence as it is; when its shapes come again it is captured as a CUDA
// graph, which the later runs replay.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include <sys/mman.h>
#include <unistd.h>

#include "../../include/bpmax_gpu.h"
#include "bpmax_kernels.cuh"
#include "bpmax_r0.cuh"
#include "bpmax_adjoint.cuh"
#include "bpmax_r0only.cuh"
#include "bpmax_wide.cuh"
#include "bpmax_persist.cuh"
#include "bpmax_strip.cuh"
#include "bpmax_tile.cuh"

using namespace bpmax;

namespace {

// schedule tunables in key order: pairs per job, merge cost, class streams, product shape variant,
// tile-product stages, class shares, persistent fill
using Tuned = std::array<int, 7>;

constexpr int MAX_SMALL_NP = 64;
constexpr int MAX_CLASS_STREAMS = 8;  // side streams for the per-width-class chains of a batch
constexpr int MAX_NP = 4096;
// outer diagonals per event of the copy-out: an event is a node between the launches of the fill's graph
// (it also keeps them from starting early), 8 us of 42 a diagonal at 128x64; the copies it holds
// back are those of the next few diagonals, and the last diagonals have few cells
constexpr int COPYOUT_DIAGS = 8;

// inner table width of a strand-2 length: multiples of 8 up to 64, then multiples of 64
int padded_width(int N) { return N <= MAX_SMALL_NP ? std::max(8, (N + 7) / 8 * 8) : (N + 63) / 64 * 64; }

// Offset pairs per product job on a diagonal with `cells` cells of P2 offset pairs each, for
// `resident` CTAs that each take every resident-th job. The launch lasts about
// ceil(jobs / resident) job lengths, a job of q pairs being 2q items plus one merge
// (`merge_items` items' worth): pick the chunk count that minimises that.
long long r0_pairs_per_job(long long cells, long long P2, long long resident, long long qmin, long long qmax,
                           long long merge_items)
{
    long long best_q = std::max(qmin, std::min(qmax, P2)), best_cost = -1;
    for (long long nch = 1; nch <= std::min<long long>(P2, 64); ++nch) {
        const long long q = std::max(qmin, std::min(qmax, (P2 + nch - 1) / nch));
        const long long jobs = cells * ((P2 + q - 1) / q);
        const long long cost = (jobs + resident - 1) / resident * (2 * q + merge_items);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best_q = q;
        }
    }
    return best_q;
}

// Stages per strip job, the same way: jobs of q of the cells' `stages` stages and one merge each
// (`merge_items` items' worth, three items to a stage)
long long strip_stages_per_job(long long cells, long long stages, long long resident, long long qmax,
                               long long merge_items)
{
    long long best_q = std::min(qmax, stages), best_cost = -1;
    for (long long nch = 1; nch <= std::min<long long>(stages, 64); ++nch) {
        const long long q = std::min(qmax, (stages + nch - 1) / nch);
        const long long jobs = cells * ((stages + q - 1) / q);
        const long long cost = (jobs + resident - 1) / resident * (3 * q + merge_items);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best_q = q;
        }
    }
    return best_q;
}

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
};

struct Plan {
    std::vector<int> Ms, Ns;
    std::vector<PairDesc> pairs;
    long long F_floats = 0, S_floats = 0;
    int bases_bytes = 0;
    int maxM = 0;
    // per step and Np class: ranges in the job arrays. d = the step: the outer diagonal, for tile tables the
    // outer diagonal plus the tile diagonal. np = inner table width class; strip (product launches): strips
    // of diagonals d .. d+T-1
    // cap: at most this many CTAs (0: as many as are resident), from the class shares
    // r0_kernel launches of one pair: q offset pairs per job of `edge`, by arithmetic (0: jobs from the list)
    struct Launch {
        int d, np, first, count, s1_first = 0, s1_count = 0;
        bool strip = false;
        int cap = 0, cells = 0, q = 0, edge = 0;
        int tile_first = 0, tile_count = 0;  // finalize launches of tile tables: the tiles (count: cells)
    };
    std::vector<Launch> r0_launches, fin_launches;
    std::vector<R0Job> r0_jobs;
    std::vector<StripJob> strip_jobs;  // jobs of strip launches (first/count index this array)
    std::vector<R0JobW> r0w_jobs;  // jobs of launches with tile-image tables (first/count index this array)
    std::vector<TileJob> tile_jobs;
    int steps = 0;  // of the fill: outer diagonals, and the tile diagonals after the last
    std::vector<CellJob> cell_jobs;
    std::vector<int> classes;  // distinct inner widths, ascending
    std::vector<int> wide_pairs;  // indices of the pairs with tile tables
    int pairs_per_job = 0, merge_items = 0, class_streams = 1;  // tunables the plan was built with
    int r0_variant = 0, wide_stages = 2, class_share = 0, persist = 0;
    long strip_tasks = 0;
    bool r0_only = false;  // R0-only double max-plus (bpmax_gpu_r0_only) instead of the BPMax fill
    std::vector<cudaEvent_t> diag_ev;  // copy-out of one pair: outer diagonal d finalized (recorded by the graph)
    // persistent fill (one launch per width class walking the diagonals with dependency counters):
    // the work queues of all classes back to back, each class's range and CTA count
    bool persistent = false, copyout = false;
    RefOut ref{nullptr, 0, 0};  // finalize launches also write the reference layout (bpmax_gpu_fill)
    std::vector<PItem> pitems;
    struct PClass { int np, first, count, ctas; };
    std::vector<PClass> pclasses;
    std::vector<int> prod_need;  // per cell (PairDesc::cell_base + cell): product jobs
    int n_counters = 0;          // per-diagonal counters of all pairs
    cudaGraphExec_t graph = nullptr;
    bool ran = false;  // launched once without a graph
    long launches = 0;
};

}  // namespace

struct bpmax_ctx {
    int device = 0;
    int sms = 148;
    cudaStream_t stream = nullptr;
    cudaStream_t class_stream[8] = {};  // MAX_CLASS_STREAMS
    cudaStream_t aux_stream = nullptr;  // reference-layout conversion and copy-out, overlapped with the fill
    cudaEvent_t fork_ev = nullptr, join_ev[8] = {};
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    Weights W;
    std::string err;
    DevBuf F, S, bases, pairs, r0jobs, stripjobs, r0wjobs, tilejobs, celljobs, widepairs, scores, conv, tbstack, grads, tbstatus, errflag;
    DevBuf r0vals;         // R0-only mode: seq1 then seq2 of the pair, as floats
    DevBuf pq, pcnt, pneed;  // persistent fill: work queue; counters (class heads, diagonals, cells); jobs per cell
    bool copyout = false;    // the next fill copies the reference layout out per diagonal (graph path)
    RefOut want_ref{nullptr, 0, 0};  // the next fill's finalize also writes the reference layout there
    DevBuf refdev;                   // that reference layout, diagonal-major
    bool r0_only = false;  // mode of the next prepare()
    bool one_chain = false;  // the fill being enqueued runs as one chain of launches
    int r0_occ_v[2][9] = {};  // resident product CTAs per SM, per shape variant and width class NB
    int wide_occ[4] = {};     // resident tile-product CTAs per SM, per stage count
    // schedule tunables (bpmax_gpu_set_tuning / bpmax_gpu_autotune); a plan is built with the
    // values current at build time, or with the values an autotune run stored for its shapes
    int r0_pairs_per_job = 1 << 20;                 // upper bound of k1 offset pairs per product job
    int r0_merge_items = 2;                         // cost of one job merge, in items, for job sizing
    int class_streams = 1;                          // run the width classes of a batch on parallel streams
    int r0_variant = 0;                             // shape variant of the width-64 product kernel (0 or 1)
    int wide_stages = 2;                            // shared-memory stages of the tile-image product (2 or 3)
    int class_share = 0;                            // cap each width class's product CTAs by its share of the work
    int persist = 0;  // width classes <= 64 by the persistent kernel: 0 no, 1 side by side, 2 one after another
    long strip_tasks = 1200;                        // least product tasks per SM of a strip launch
    int persist_occ[9] = {};                        // resident persistent-fill CTAs per SM, per width class
    // bounded waits of the product kernels: time limit of one wait, and the one-shot test mode in
    // which the next fill's product kernels issue no copies (their first waits run out)
    unsigned long long wait_ns = 4000000000ULL;
    bool inject_wait_timeout = false;
    std::map<std::vector<int>, Tuned> tuned;  // shape signature (Ms then Ns) -> tunables
    float *host_stage[2] = {nullptr, nullptr};
    void *copy_stage = nullptr;  // pinned buffers of copy_out
    size_t fresh_bytes = 0;      // copied into fresh pageable memory so far
    size_t host_stage_bytes = 0;
    cudaEvent_t stage_ev[2] = {nullptr, nullptr};
    Plan plan;
    bool plan_valid = false;
    float last_ms = 0.f;
    long last_launches = 0;
};

namespace {

int fail(bpmax_ctx *ctx, int status, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (ctx) ctx->err = buf;
    return status;
}

#define CK(call)                                                                                        \
    do {                                                                                                \
        cudaError_t e_ = (call);                                                                        \
        if (e_ != cudaSuccess)                                                                          \
            return fail(ctx, e_ == cudaErrorMemoryAllocation ? BPMAX_ENOMEM : BPMAX_ECUDA, "%s: %s (%s:%d)", \
                        #call, cudaGetErrorString(e_), __FILE__, __LINE__);                              \
    } while (0)

int ensure(bpmax_ctx *ctx, DevBuf &b, size_t bytes)
{
    if (b.bytes >= bytes) return BPMAX_OK;
    if (b.p) CK(cudaFree(b.p));
    b.p = nullptr;
    b.bytes = 0;
    size_t want = std::max(bytes, (size_t)256);
    CK(cudaMalloc(&b.p, want));
    b.bytes = want;
    return BPMAX_OK;
}

WaitCtl wait_ctl(const bpmax_ctx *ctx)
{
    return WaitCtl{(int *)ctx->errflag.p, ctx->wait_ns, ctx->inject_wait_timeout ? 1 : 0};
}

int weights_ok(const float *w)
{
    for (int t = 0; t < 12; ++t)
        if (!std::isfinite(w[t]) || w[t] < 0.0f || std::signbit(w[t])) return 0;
    return 1;
}

long long align64(long long x) { return (x + 63) / 64 * 64; }

// Builds the device layout and the per-diagonal job lists for the given pair shapes.
std::vector<int> shape_key(const std::vector<int> &Ms, const std::vector<int> &Ns)
{
    std::vector<int> k(Ms);
    k.insert(k.end(), Ns.begin(), Ns.end());
    return k;
}

// Work queue of the persistent fill, per width class: for d = 1, 2, ... the finalize items of
// diagonal d-1, then the product jobs of diagonal d with offset pairs >= 1, then the jobs of d for
// offset pair 0 (the only ones reading diagonal d-1); the finalize items of the last diagonal close
// it. Every item depends only on items before it (bpmax_persist.cuh), and the finalize of d-1 runs
// beside the long product group of d. Jobs of one group are ordered by pair chunk, then cell, as in
// the graph path. CTA counts: one class takes every resident CTA. Several classes either run one
// after another, each with every resident CTA (mode 2), or side by side (mode 1), each with a number
// of SMs proportional to its estimated time, so that all of them are resident at once.
void build_queue(bpmax_ctx *ctx, Plan &P)
{
    const int n = (int)P.pairs.size();
    long long ncells = 0;
    for (const auto &pd : P.pairs) ncells += (long long)pd.M * (pd.M + 1) / 2;
    P.prod_need.assign(ncells, 0);
    P.pitems.clear();
    P.pclasses.clear();
    // estimated CTA-microseconds per class: product items (one C(Np)+2T(Np) block each) and
    // finalizes, at the per-CTA costs of each width measured with this kernel on a B200, per SM
    // (divided by the CTAs one SM holds)
    static const double ITEM_US[9] = {0, 0.19, 0.30, 0.42, 0.65, 0.93, 1.2, 2.1, 2.1};
    static const double FIN_US[9] = {0, 4.0, 6.0, 9.0, 14.0, 24.0, 36.0, 72.0, 80.0};
    auto C3 = [](double x) { return x * (x * x - 1) / 6; };
    auto T2 = [](double x) { return x * (x + 1) / 2; };
    std::map<int, double> sm_time;
    double sm_tot = 0;
    for (const auto &pd : P.pairs) {
        const int NB = pd.Np / 8;
        const double t = (C3(pd.M) * ITEM_US[NB] + T2(pd.M) * FIN_US[NB]) / std::max(1, ctx->persist_occ[NB]);
        sm_time[pd.Np] += t;
        sm_tot += t;
    }
    std::map<int, int> sms_of;
    const bool side = P.classes.size() > 1 && P.persist == 1;
    if (side) {  // SMs per class, all classes resident at once (a margin of 2 SMs for uneven packing)
        const int budget = std::max((int)P.classes.size(), ctx->sms - 2);
        int used = 0;
        for (int np : P.classes) {
            sms_of[np] = std::max(1, (int)std::lround(budget * sm_time[np] / sm_tot));
            used += sms_of[np];
        }
        while (used > budget) {  // take the excess from the largest shares
            int big = P.classes[0];
            for (int np : P.classes)
                if (sms_of[np] > sms_of[big]) big = np;
            if (sms_of[big] <= 1) break;
            --sms_of[big];
            --used;
        }
    }
    for (int np : P.classes) {
        const int NB = np / 8, G = R0_TAB_ITEMS[NB];
        const int occ = std::max(1, ctx->persist_occ[NB]);
        const int ctas = side ? sms_of[np] * occ : occ * ctx->sms;
        const int first = (int)P.pitems.size();
        int maxM = 0;
        for (const auto &pd : P.pairs)
            if (pd.Np == np) maxM = std::max(maxM, pd.M);
        auto fin_items = [&](int e) {
            for (int p = 0; p < n; ++p)
                if (P.pairs[p].Np == np && P.pairs[p].M > e)
                    for (int i1 = 0; i1 < P.pairs[p].M - e; ++i1) P.pitems.push_back(PItem{p, i1, e, 0, 0, 1});
        };
        const long long qmin = std::max(1, (G + 1) / 2);
        for (int d = 1; d <= maxM; ++d) {
            const long long P2 = (d + 1) / 2;
            long long cells = 0;
            for (const auto &pd : P.pairs)
                if (pd.Np == np && pd.M > d) cells += pd.M - d;
            fin_items(d - 1);
            if (cells > 0 && P2 > 1) {  // offset pairs >= 1
                const long long q = r0_pairs_per_job(cells, P2 - 1, ctas, qmin, std::max<long long>(P.pairs_per_job, qmin),
                                                     P.merge_items);
                for (long long c0 = 1; c0 < P2; c0 += q)
                    for (int p = 0; p < n; ++p)
                        if (P.pairs[p].Np == np && P.pairs[p].M > d)
                            for (int i1 = 0; i1 < P.pairs[p].M - d; ++i1) {
                                P.pitems.push_back(PItem{p, i1, d, (int)c0, (int)std::min(c0 + q, P2), 0});
                                P.prod_need[P.pairs[p].cell_base + cell_index(P.pairs[p].M, i1, i1 + d)] += 1;
                            }
            }
            if (cells > 0)  // offset pair 0 (offsets 0 and d-1)
                for (int p = 0; p < n; ++p)
                    if (P.pairs[p].Np == np && P.pairs[p].M > d)
                        for (int i1 = 0; i1 < P.pairs[p].M - d; ++i1) {
                            P.pitems.push_back(PItem{p, i1, d, 0, 1, 0});
                            P.prod_need[P.pairs[p].cell_base + cell_index(P.pairs[p].M, i1, i1 + d)] += 1;
                        }
        }
        P.pclasses.push_back(Plan::PClass{np, first, (int)P.pitems.size() - first, ctas});
    }
}

// Launches of one step of the tile tables of width np: tile diagonal t of outer diagonal d with d + t = step
// (the R0-only mode keeps to outer diagonals: step = d, every tile)
void build_tile_step(bpmax_ctx *ctx, Plan &P, int np, int step, long long resident, bool uncapped)
{
    const int NT = np / 64, n = (int)P.pairs.size();
    // jobs: one per output tile of a cell and chunk of k1 offset pairs, and per chunk of the 2t terms over
    // finished tiles, sized so that jobs cost about the same: cost per offset pair in warp task steps
    // of both of its items, DD 3.3, DA and DB 12, F 16 per item, in a narrow last tile column less, but
    // 5 at the least (the copies)
    auto nbc = [&](int p, int J) { return J == NT - 1 ? (P.pairs[p].N - 64 * J + 7) / 8 : 8; };
    auto item_cost = [&](int p, int J, double full) { return std::max(5.0, full * wide_cost(nbc(p, J)) / 16.0); };
    auto pair_cost = [&](int p, int t, int J) {
        return t == 0 ? 2 * 3.3 : 2 * (2 * item_cost(p, J, 12.0) + item_cost(p, J, 16.0) * (t - 1));
    };
    auto each = [&](auto &&f) {  // (pair, d, t) of the step
        for (int p = 0; p < n; ++p)
            if (P.pairs[p].Np == np)
                for (int t = ctx->r0_only ? 0 : std::max(0, step - P.pairs[p].M + 1); t < NT; ++t) {
                    const int d = ctx->r0_only ? step : step - t;
                    if (d >= 0 && d < P.pairs[p].M) f(p, d, t);
                }
    };
    double total = 0;
    Plan::Launch fl{step, np, (int)P.cell_jobs.size(), 0};
    fl.tile_first = (int)P.tile_jobs.size();
    each([&](int p, int d, int t) {
        for (int J = t; J < NT; ++J)
            total += (P.pairs[p].M - d) *
                     ((d + 1) / 2 * pair_cost(p, t, J) + (ctx->r0_only ? 0.0 : 2.0 * t * item_cost(p, J, 16.0)));
    });
    const double target = std::max(total / (3.0 * resident), 4.0 * 16.0);
    const size_t first = P.r0w_jobs.size();
    for (int T = NT - 1; T >= 0; --T)  // heavy tiles first
        each([&](int p, int d, int t) {
            if (t != T) return;
            const int P2 = (d + 1) / 2, cells = P.pairs[p].M - d;
            for (int I = 0; I + t < NT; ++I) {
                const int J = I + t, tile = nbc(p, J) << 16 | I << 8 | J;
                const int q = std::max(1, (int)std::min<long long>(P2, std::llround(target / pair_cost(p, t, J))));
                const int qs = std::max(1, (int)std::min<long long>(2 * t, std::llround(target / item_cost(p, J, 16.0))));
                if (!ctx->r0_only)
                    for (int n0 = 0; n0 < 2 * t; n0 += qs)
                        for (int i1 = 0; i1 < cells; ++i1)
                            P.r0w_jobs.push_back(R0JobW{p, i1, d, tile, -1 - n0, std::min(n0 + qs, 2 * t)});
                for (int c0 = 0; c0 < P2; c0 += q)
                    for (int i1 = 0; i1 < cells; ++i1)
                        P.r0w_jobs.push_back(R0JobW{p, i1, d, tile, c0, std::min(c0 + q, P2)});
                if (!ctx->r0_only)
                    for (int i1 = 0; i1 < cells; ++i1) P.tile_jobs.push_back(TileJob{p, i1, d, I << 8 | J});
            }
        });
    // jobs of the same offset pairs together (both uses of a table meet in L2), heavy tiles first
    std::stable_sort(P.r0w_jobs.begin() + first, P.r0w_jobs.end(),
                     [](const R0JobW &a, const R0JobW &b) { return std::max(a.p0, -1) < std::max(b.p0, -1); });
    Plan::Launch wl{step, np, (int)first, (int)(P.r0w_jobs.size() - first)};
    wl.cap = uncapped ? 0 : (int)resident;
    if (wl.count > 0) P.r0_launches.push_back(wl);
    for (int p = 0; p < n; ++p)  // the cells of outer diagonal `step` (S1; the finalize of the R0-only mode)
        if (P.pairs[p].Np == np && P.pairs[p].M > step)
            for (int i1 = 0; i1 < P.pairs[p].M - step; ++i1) P.cell_jobs.push_back(CellJob{p, i1});
    fl.count = (int)P.cell_jobs.size() - fl.first;
    fl.tile_count = (int)P.tile_jobs.size() - fl.tile_first;
    if (fl.count > 0 || fl.tile_count > 0) P.fin_launches.push_back(fl);
}

int build_plan(bpmax_ctx *ctx, const std::vector<int> &Ms, const std::vector<int> &Ns, Plan &P)
{
    P = Plan();
    P.Ms = Ms;
    P.Ns = Ns;
    P.pairs_per_job = ctx->r0_pairs_per_job;
    P.merge_items = ctx->r0_merge_items;
    P.class_streams = ctx->class_streams;
    P.r0_variant = ctx->r0_variant;
    P.wide_stages = ctx->wide_stages;
    P.class_share = ctx->class_share;
    P.persist = ctx->persist;
    P.strip_tasks = ctx->strip_tasks;
    const auto tu = ctx->tuned.find(shape_key(Ms, Ns));
    if (tu != ctx->tuned.end()) {
        P.pairs_per_job = tu->second[0];
        P.merge_items = tu->second[1];
        P.class_streams = tu->second[2];
        P.r0_variant = tu->second[3];
        P.wide_stages = tu->second[4];
        P.class_share = tu->second[5];
        P.persist = tu->second[6];
    }
    const int n = (int)Ms.size();
    long long f = 0, s = 0;
    int b = 0;
    for (int p = 0; p < n; ++p) {
        PairDesc pd{};
        pd.M = Ms[p];
        pd.N = Ns[p];
        pd.Np = padded_width(Ns[p]);
        if (pd.Np > MAX_NP) return fail(ctx, BPMAX_EINVAL, "strand-2 length %d > %d is not supported", Ns[p], MAX_NP);
        pd.F_off = f;
        f = align64(f + (long long)Ms[p] * (Ms[p] + 1) / 2 * cell_floats(pd.Np));
        pd.S1_off = s;
        s = align64(s + (long long)Ms[p] * Ms[p]);
        pd.S2_off = s;
        s = align64(s + (long long)pd.Np * pd.Np);
        if (pd.Np > MAX_SMALL_NP) {  // S2 as tile images
            pd.S2x_off = s;
            s = align64(s + (long long)pd.Np * pd.Np);
            P.wide_pairs.push_back(p);
        }
        pd.seq1_off = b;
        b += Ms[p];
        pd.seq2_off = b;
        b += Ns[p];
        pd.cnt_off = P.n_counters;
        P.n_counters += Ms[p];
        pd.cell_base = p == 0 ? 0 : P.pairs.back().cell_base + (long long)P.pairs.back().M * (P.pairs.back().M + 1) / 2;
        P.pairs.push_back(pd);
        P.maxM = std::max(P.maxM, Ms[p]);
    }
    P.F_floats = f;
    P.S_floats = s;
    P.bases_bytes = b;
    std::vector<int> classes;
    for (const auto &pd : P.pairs) classes.push_back(pd.Np);
    std::sort(classes.begin(), classes.end());
    classes.erase(std::unique(classes.begin(), classes.end()), classes.end());
    P.classes = classes;
    // class shares: with several width classes on parallel graph branches, a product launch of one
    // class may hold every SM until its last job ends, so the branches run one after another. With
    // class shares on, each class's product launches take at most its share of the resident CTAs
    // (its share of the padded product terms, at least 1/16), so every branch keeps progressing.
    std::map<int, double> share;
    if (P.class_share && classes.size() > 1 && P.class_streams) {
        auto C3 = [](double x) { return x * (x * x - 1) / 6; };
        auto T2 = [](double x) { return x * (x + 1) / 2; };
        double tot = 0;
        for (const auto &pd : P.pairs) {
            const double w = C3(pd.M) * (C3(pd.Np) + 2 * T2(pd.Np));
            share[pd.Np] += w;
            tot += w;
        }
        for (auto &kv : share) kv.second = std::max(kv.second / tot, 1.0 / 16);
    }
    auto capped = [&](int np, long long resident) {
        const auto it = share.find(np);
        return it == share.end() ? resident : std::max(1LL, (long long)std::llround(resident * it->second));
    };
    // jobs, grouped by diagonal then inner width class
    const int NTmax = classes.back() > MAX_SMALL_NP && !ctx->r0_only ? classes.back() / 64 : 1;
    P.steps = P.maxM + NTmax - 1;
    for (int d = 0; d < P.steps; ++d) {
        for (int np : classes) {
            if (np > MAX_SMALL_NP) {
                build_tile_step(ctx, P, np, d, capped(np, (long long)std::max(1, ctx->wide_occ[P.wide_stages]) * ctx->sms),
                                share.empty());
                continue;
            }
            long long cells = 0;
            for (int p = 0; p < n; ++p)
                if (P.pairs[p].Np == np && Ms[p] > d) cells += Ms[p] - d;
            if (cells == 0) continue;
            Plan::Launch fl{d, np, (int)P.cell_jobs.size(), 0};
            for (int p = 0; p < n; ++p)
                if (P.pairs[p].Np == np && Ms[p] > d)
                    for (int i1 = 0; i1 < Ms[p] - d; ++i1) P.cell_jobs.push_back(CellJob{p, i1});
            fl.count = (int)P.cell_jobs.size() - fl.first;
            P.fin_launches.push_back(fl);
            if (d == 0) continue;
            {
                // Strips of T cells (bpmax_strip.cuh), once per T diagonals d .. d+T-1 (d = 1 mod T): the
                // offsets [0, d-1], of which cell t of a strip takes those >= t. The first t offset pairs
                // of diagonal d+t, which meet diagonals >= d, are the jobs of r0_kernel. Diagonals
                // with few offsets (strip_min_d) or little work keep r0_kernel alone: a strip launch adds a
                // launch to the chain and clears T merge tiles per CTA (strip_tasks = 0: strips everywhere).
                // Fill ms, with strips from diagonal 1 on, everywhere / from 400 / 1,200 (10 width-64
                // items) / 3,400 tasks per SM / nowhere: 37x23 0.41 / 0.35 / 0.35 / 0.35 / 0.35, 100x64
                // 2.56 / 2.56 / 2.56 / 2.66 / 2.67, 128x64 3.86 / 3.86 / 3.86 / 4.10 / 4.10, 128x32 1.93 /
                // 1.88 / 1.81 / 1.82 / 1.81, 200x64 9.1 / 9.1 / 9.1 / 9.1 / 10.2, 256x64 15.5 / 15.5 / 15.5 /
                // 15.5 / 18.1.
                const int NB = np / 8, G = R0_TAB_ITEMS[NB];
                const long long P2 = (d + 1) / 2;  // offset pairs per cell
                long long edge = P2;               // offset pairs per cell of r0_kernel's jobs
                const int T = strip_cells(NB), d0 = d - (d - 1) % T;  // the strips' first diagonal
                long long cells0 = 0;
                for (int p = 0; p < n; ++p)
                    if (P.pairs[p].Np == np && Ms[p] > d0) cells0 += Ms[p] - d0;
                // tasks of an item: NB(NB+1)(NB+2)/6
                const bool enough = d0 >= strip_min_d(NB) &&
                                    cells0 * d0 * (NB * (NB + 1) * (NB + 2) / 6) >= P.strip_tasks * ctx->sms;
                if (NB >= STRIP_MIN_NB && (P.strip_tasks == 0 || enough)) {
                    edge = std::min<long long>(P2, d - d0);
                    if (d == d0) {
                        const long long stages = (d + G - 1) / G;  // of G offsets
                        const long long resident = capped(np, ctx->sms);
                        const long long q =
                            strip_stages_per_job(cells, stages, resident, std::max<long long>(1, 2LL * P.pairs_per_job / G),
                                                 P.merge_items);
                        Plan::Launch sl{d, np, (int)P.strip_jobs.size(), 0};
                        sl.strip = true;
                        sl.cap = (int)resident;
                        for (long long w0 = 0; w0 < d; w0 += q * G)
                            for (int p = 0; p < n; ++p)
                                if (P.pairs[p].Np == np && Ms[p] > d)
                                    for (int i1 = 0; i1 < Ms[p] - d; ++i1)
                                        P.strip_jobs.push_back(StripJob{p, i1, (int)w0, (int)std::min<long long>(w0 + q * G, d)});
                        sl.count = (int)P.strip_jobs.size() - sl.first;
                        P.r0_launches.push_back(sl);
                    }
                }
                if (edge == 0) continue;
                // jobs of q offset pairs, ordered by pair chunk, then pair, then cell: the two uses of a
                // table (A of cell (a, a+d) at offset w, B of cell (a+w-d, a+w) at offset d-1-w) fall in
                // the same pair chunk
                const long long resident =
                    capped(np, (long long)std::max(1, ctx->r0_occ_v[P.r0_variant][NB]) * ctx->sms);
                const long long qmin = std::max(1, (G + 1) / 2), qmax = std::max<long long>(P.pairs_per_job, qmin);
                const long long q = r0_pairs_per_job(cells, edge, resident, qmin, qmax, P.merge_items);
                Plan::Launch rl{d, np, (int)P.r0_jobs.size(), 0};
                rl.cap = share.empty() ? 0 : (int)resident;
                if (n == 1 && P.r0_variant == 0) {
                    rl.cells = (int)cells;
                    rl.q = (int)q;
                    rl.edge = (int)edge;
                    rl.count = (int)(cells * ((edge + q - 1) / q));
                } else {
                    for (long long c0 = 0; c0 < edge; c0 += q)
                        for (int p = 0; p < n; ++p)
                            if (P.pairs[p].Np == np && Ms[p] > d)
                                for (int i1 = 0; i1 < Ms[p] - d; ++i1)
                                    P.r0_jobs.push_back(R0Job{p, i1, (int)c0, (int)std::min(c0 + q, edge)});
                    rl.count = (int)P.r0_jobs.size() - rl.first;
                }
                P.r0_launches.push_back(rl);
                continue;
            }
        }
    }
    // S1 of diagonal d+1 is computed by the finalize launch of diagonal d (same class); it stays 0 up to a span of 3
    for (auto &fl : P.fin_launches)
        for (const auto &nx : P.fin_launches)
            if (nx.d > 3 && nx.d == fl.d + 1 && nx.np == fl.np) { fl.s1_first = nx.first; fl.s1_count = nx.count; }
    // the persistent fill: width classes <= 64 only, not the R0-only mode, not the reference-layout
    // fill with its per-diagonal copy-out (both keep the graph of per-diagonal launches)
    P.copyout = ctx->copyout;
    P.persistent = P.persist && !ctx->r0_only && !ctx->copyout && P.classes.back() <= MAX_SMALL_NP;
    if (P.persistent) build_queue(ctx, P);
    return BPMAX_OK;
}

// Launch of a kernel of a fill's chain. early: by programmatic dependent launch (chain_wait in the
// kernel), where the chain is the only one of its fill (the early CTAs of several chains would hold each
// other's room). That hides the launch and the first loads of a short kernel (37x23 0.53 -> 0.35 ms,
// 200x8 2.42 -> 1.52, 128x32 2.44 -> 1.97), but places its CTAs where room comes free first, several to
// an SM: kernels of a few hundred large CTAs start normally (early 512-thread finalizes 128x64 4.61 against
// 4.21 ms, early tile kernels 90x70 9.36 against 8.85, early tile products 256x256 737 against 709).
template <class... P, class... A>
void launch_chain(bool early, dim3 grid, int threads, size_t smem, cudaStream_t s, void (*kernel)(P...), A... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, P(args)...);
}

template <int STAGES>
void launch_r0_wide_t(bpmax_ctx *ctx, const Plan::Launch &L, cudaStream_t s)
{
    const int grid = std::min(L.count, L.cap > 0 ? L.cap : std::max(1, ctx->wide_occ[STAGES]) * ctx->sms);
    launch_chain(false, grid, WideCfg<STAGES>::THREADS, WideCfg<STAGES>::SMEM, s, r0_wide_kernel<STAGES>,
                 (const R0JobW *)ctx->r0wjobs.p + L.first, L.count, (const PairDesc *)ctx->pairs.p, (float *)ctx->F.p,
                 (const float *)ctx->S.p, wait_ctl(ctx));
}

void launch_r0_wide(bpmax_ctx *ctx, const Plan &P, const Plan::Launch &L, cudaStream_t s)
{
    if (P.wide_stages == 3)
        launch_r0_wide_t<3>(ctx, L, s);
    else
        launch_r0_wide_t<2>(ctx, L, s);
}

// the tiles of one step, and S1 of outer diagonal step+1
void launch_fin_tiles(bpmax_ctx *ctx, const Plan::Launch &L, cudaStream_t s)
{
    const int grid = L.tile_count + (L.s1_count + TILE_THREADS / 32 - 1) / (TILE_THREADS / 32);
    launch_chain(false, grid, TILE_THREADS, TILE_SMEM, s,
                 L.tile_count > 2 * ctx->sms ? tile_final_kernel<3> : tile_final_kernel<2>,
                 (const TileJob *)ctx->tilejobs.p + L.tile_first, L.tile_count,
                 (const CellJob *)ctx->celljobs.p + L.s1_first, L.s1_count, (const PairDesc *)ctx->pairs.p,
                 (float *)ctx->F.p, (float *)ctx->S.p, (const uint8_t *)ctx->bases.p, ctx->W, L.d);
}

template <int NB, int V>
void launch_r0_v(bpmax_ctx *ctx, const Plan::Launch &L, cudaStream_t s)
{
    using C = R0Cfg<NB, V>;
    // resident CTAs (or the class's share of them); each loops over jobs
    const int grid = std::min(L.count, L.cap > 0 ? L.cap : std::max(1, ctx->r0_occ_v[V][NB]) * ctx->sms);
    auto go = [&](auto kernel, auto jobs) {
        launch_chain(ctx->one_chain, grid, C::THREADS, C::SMEM, s, kernel, jobs, L.count, (const PairDesc *)ctx->pairs.p,
                     (float *)ctx->F.p, L.d, wait_ctl(ctx));
    };
    if constexpr (V == 0)
        if (L.q) return go(r0_kernel<NB, V, R0Jobs>, R0Jobs{L.cells, L.q, L.edge});
    go(r0_kernel<NB, V>, R0List{(const R0Job *)ctx->r0jobs.p + L.first});
}

template <int NB>
void launch_strip(bpmax_ctx *ctx, const Plan::Launch &L, cudaStream_t s)
{
    launch_chain(ctx->one_chain, std::min(L.count, L.cap), StripCfg<NB>::THREADS, StripCfg<NB>::SMEM, s,
                 r0_strip_kernel<NB>, (const StripJob *)ctx->stripjobs.p + L.first, L.count,
                 (const PairDesc *)ctx->pairs.p, (float *)ctx->F.p, L.d, wait_ctl(ctx));
}

template <int NB>
void launch_persist(bpmax_ctx *ctx, const PersistCtl &pc, int ctas, cudaStream_t s)
{
    fill_persistent_kernel<NB><<<ctas, R0Cfg<NB>::THREADS, R0Cfg<NB>::SMEM, s>>>(
        pc, (const PairDesc *)ctx->pairs.p, (float *)ctx->F.p, (float *)ctx->S.p, (const uint8_t *)ctx->bases.p, ctx->W,
        wait_ctl(ctx));
}

template <int NB>
void launch_r0(bpmax_ctx *ctx, const Plan &P, const Plan::Launch &L, cudaStream_t s)
{
    if constexpr (NB >= STRIP_MIN_NB)
        if (L.strip) return launch_strip<NB>(ctx, L, s);
    if (P.r0_variant == 1)
        launch_r0_v<NB, 1>(ctx, L, s);
    else
        launch_r0_v<NB, 0>(ctx, L, s);
}

template <int NB, int T>
void launch_fin_t(bpmax_ctx *ctx, const Plan::Launch &L, cudaStream_t s)
{
    using Sh = FinShape<8 * NB, T>;
    launch_chain(ctx->one_chain && T < 512, L.count + (L.s1_count + Sh::WARPS - 1) / Sh::WARPS, Sh::THREADS,
                 Sh::SMEM, s, finalize_small_kernel<8 * NB, T>, (const CellJob *)ctx->celljobs.p + L.first, L.count,
                 (const CellJob *)ctx->celljobs.p + L.s1_first, L.s1_count, (const PairDesc *)ctx->pairs.p,
                 (float *)ctx->F.p, (float *)ctx->S.p, (const uint8_t *)ctx->bases.p, ctx->W, L.d, ctx->plan.ref);
}

template <int NB>
void launch_fin(bpmax_ctx *ctx, const Plan::Launch &L, cudaStream_t s)
{
    if (L.count > fin_bulk_per_sm(8 * NB) * ctx->sms) return launch_fin_t<NB, fin_bulk_threads(8 * NB)>(ctx, L, s);
    if constexpr (fin_has_mid(8 * NB))
        if (L.count > ctx->sms) return launch_fin_t<NB, FIN_MID_THREADS>(ctx, L, s);
    launch_fin_t<NB, fin_threads(8 * NB)>(ctx, L, s);
}

void launch_r0only_fin(bpmax_ctx *ctx, const Plan::Launch &L, cudaStream_t s)
{
    const CellJob *jobs = (const CellJob *)ctx->celljobs.p + L.first;
    const PairDesc *pd = (const PairDesc *)ctx->pairs.p;
    const float *vals = (const float *)ctx->r0vals.p;
    auto go = [&](auto kernel) {
        launch_chain(ctx->one_chain, L.count, 128, 0, s, kernel, jobs, pd, (float *)ctx->F.p, vals, L.d);
    };
    switch (L.np > MAX_SMALL_NP ? 0 : L.np / 8) {
    case 0:
        launch_chain(ctx->one_chain, dim3(L.count, L.np / 64), 256, 0, s, r0only_finalize_tile_kernel, jobs, pd,
                     (float *)ctx->F.p, vals, L.d);
        break;
    case 1: go(r0only_finalize_small_kernel<8>); break;
    case 2: go(r0only_finalize_small_kernel<16>); break;
    case 3: go(r0only_finalize_small_kernel<24>); break;
    case 4: go(r0only_finalize_small_kernel<32>); break;
    case 5: go(r0only_finalize_small_kernel<40>); break;
    case 6: go(r0only_finalize_small_kernel<48>); break;
    case 7: go(r0only_finalize_small_kernel<56>); break;
    default: go(r0only_finalize_small_kernel<64>); break;
    }
}

// The product kernels, the small finalize and the persistent fill prefer the largest shared-memory
// carveout: an SM runs CTAs of different kernels side by side only when they use the same L1 /
// shared-memory split (parallel graph branches of a batch, the persistent launches of its width
// classes).
template <typename K>
int prefer_smem(bpmax_ctx *ctx, K kernel)
{
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    return BPMAX_OK;
}

template <int NB>
int set_smem_attr(bpmax_ctx *ctx)
{
    int st;
    if ((st = prefer_smem(ctx, r0_kernel<NB>)) || (st = prefer_smem(ctx, r0_kernel<NB, 0, R0Jobs>)) ||
        (st = prefer_smem(ctx, r0_kernel<NB, 1>)) ||
        (st = prefer_smem(ctx, finalize_small_kernel<8 * NB>)) || (st = prefer_smem(ctx, r0only_finalize_small_kernel<8 * NB>)))
        return st;
    if ((st = prefer_smem(ctx, finalize_small_kernel<8 * NB, fin_bulk_threads(8 * NB)>))) return st;
    if constexpr (fin_has_mid(8 * NB)) {
        if ((st = prefer_smem(ctx, finalize_small_kernel<8 * NB, FIN_MID_THREADS>))) return st;
        CK(cudaFuncSetAttribute(finalize_small_kernel<8 * NB, FIN_MID_THREADS>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)FinShape<8 * NB, FIN_MID_THREADS>::SMEM));
    }
    if constexpr (NB >= STRIP_MIN_NB) {
        if ((st = prefer_smem(ctx, r0_strip_kernel<NB>))) return st;
        CK(cudaFuncSetAttribute(r0_strip_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)StripCfg<NB>::SMEM));
    }
    if (NB == 8)
        if ((st = prefer_smem(ctx, r0_wide_kernel<2>)) || (st = prefer_smem(ctx, r0_wide_kernel<3>)) ||
            (st = prefer_smem(ctx, tile_final_kernel<2>)) || (st = prefer_smem(ctx, tile_final_kernel<3>)))
            return st;
    CK(cudaFuncSetAttribute(r0_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R0Cfg<NB>::SMEM));
    CK(cudaFuncSetAttribute(r0_kernel<NB, 0, R0Jobs>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R0Cfg<NB>::SMEM));
    CK(cudaFuncSetAttribute(r0_kernel<NB, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R0Cfg<NB, 1>::SMEM));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctx->r0_occ_v[1][NB], r0_kernel<NB, 1>, R0Cfg<NB, 1>::THREADS,
                                                     R0Cfg<NB, 1>::SMEM));
    CK(cudaFuncSetAttribute(finalize_small_kernel<8 * NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)FinShape<8 * NB>::SMEM));
    CK(cudaFuncSetAttribute(finalize_small_kernel<8 * NB, fin_bulk_threads(8 * NB)>,
                            cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)FinShape<8 * NB, fin_bulk_threads(8 * NB)>::SMEM));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctx->r0_occ_v[0][NB], r0_kernel<NB>, R0Cfg<NB>::THREADS,
                                                     R0Cfg<NB>::SMEM));
    CK(cudaFuncSetAttribute(fill_persistent_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R0Cfg<NB>::SMEM));
    CK(cudaFuncSetAttribute(fill_persistent_kernel<NB>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctx->persist_occ[NB], fill_persistent_kernel<NB>,
                                                     R0Cfg<NB>::THREADS, R0Cfg<NB>::SMEM));
    if (NB == 8) {
        CK(cudaFuncSetAttribute(r0_wide_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WideCfg<2>::SMEM));
        CK(cudaFuncSetAttribute(r0_wide_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WideCfg<3>::SMEM));
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctx->wide_occ[2], r0_wide_kernel<2>, 128, WideCfg<2>::SMEM));
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctx->wide_occ[3], r0_wide_kernel<3>, 128, WideCfg<3>::SMEM));
        CK(cudaFuncSetAttribute(tile_final_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_SMEM));
        CK(cudaFuncSetAttribute(tile_final_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_SMEM));
    }
    return BPMAX_OK;
}

struct KernelProfile {
    bool on = false;
    cudaEvent_t a = nullptr, b = nullptr;
    float ms[3] = {0, 0, 0};
    long launches[3] = {0, 0, 0};
};

// brackets one launch with events when profiling (eager runs only, never inside a capture)
struct ProfScope {
    bpmax_ctx *ctx;
    KernelProfile *kp;
    int kind;
    ProfScope(bpmax_ctx *c, KernelProfile *k, int kind_) : ctx(c), kp(k), kind(kind_)
    {
        if (kp && kp->on) cudaEventRecord(kp->a, ctx->stream);
    }
    ~ProfScope()
    {
        if (kp && kp->on) {
            cudaEventRecord(kp->b, ctx->stream);
            cudaEventSynchronize(kp->b);
            float t = 0.f;
            cudaEventElapsedTime(&t, kp->a, kp->b);
            kp->ms[kind] += t;
            kp->launches[kind] += 1;
        }
    }
};

int enqueue_fill(bpmax_ctx *ctx, Plan &P, KernelProfile *kp = nullptr)
{
    long launches = 0;
    ctx->one_chain = !(kp && kp->on) && !(P.classes.size() > 1 && P.class_streams);
    CK(cudaMemsetAsync(ctx->F.p, 0, (size_t)P.F_floats * sizeof(float), ctx->stream));
    CK(cudaMemsetAsync(ctx->S.p, 0, (size_t)P.S_floats * sizeof(float), ctx->stream));  // S1 starts at 0
    CK(cudaMemsetAsync(ctx->errflag.p, 0, sizeof(int), ctx->stream));
    if (!P.r0_only) {
        ProfScope ps(ctx, kp, 0);
        single_strand_kernel<<<(int)P.pairs.size(), 512, 0, ctx->stream>>>(
            (const PairDesc *)ctx->pairs.p, (const uint8_t *)ctx->bases.p, (float *)ctx->S.p, ctx->W);
        for (int p = 0; p < (int)P.pairs.size(); ++p)  // wider tables: one launch per diagonal of S2
            if (P.pairs[p].Np > S2_ONE_CTA_NP)
                for (int d = 4; d < P.pairs[p].N; ++d, ++launches)
                    launch_chain(
                        ctx->one_chain, (P.pairs[p].N - d + 7) / 8, 256, 0, ctx->stream, s2_diag_kernel,
                        (const PairDesc *)ctx->pairs.p, p, (const uint8_t *)ctx->bases.p, (float *)ctx->S.p, ctx->W, d);
        launches += 1;
        if (!P.wide_pairs.empty()) {
            launch_chain(ctx->one_chain, dim3((int)P.wide_pairs.size(), 64), 256, 0, ctx->stream, s2_aux_kernel,
                         (const int *)ctx->widepairs.p, (const PairDesc *)ctx->pairs.p, (float *)ctx->S.p);
            launches += 1;
        }
    }
    const bool prof = kp && kp->on;
    if (P.persistent) {  // one persistent launch per width class: side by side on the class streams, or in turn
        const int nclass = (int)P.pclasses.size();
        int *cnt = (int *)ctx->pcnt.p;
        int *diag_done = cnt + 64, *prod_done = diag_done + align64(P.n_counters);
        CK(cudaMemsetAsync(cnt, 0, ((size_t)64 + align64(P.n_counters) + P.prod_need.size()) * sizeof(int), ctx->stream));
        const bool pfork = !prof && nclass > 1 && P.persist == 1;
        if (pfork) {
            CK(cudaEventRecord(ctx->fork_ev, ctx->stream));
            for (int k = 0; k < std::min(nclass, MAX_CLASS_STREAMS); ++k)
                CK(cudaStreamWaitEvent(ctx->class_stream[k], ctx->fork_ev, 0));
        }
        for (int c = 0; c < nclass; ++c, ++launches) {
            const auto &pcl = P.pclasses[c];
            const cudaStream_t st = pfork ? ctx->class_stream[c % MAX_CLASS_STREAMS] : ctx->stream;
            const PersistCtl pctl{(const PItem *)ctx->pq.p + pcl.first, pcl.count, cnt + c, diag_done, prod_done,
                                  (const int *)ctx->pneed.p};
            ProfScope ps(ctx, kp, 1);
            switch (pcl.np / 8) {
            case 1: launch_persist<1>(ctx, pctl, pcl.ctas, st); break;
            case 2: launch_persist<2>(ctx, pctl, pcl.ctas, st); break;
            case 3: launch_persist<3>(ctx, pctl, pcl.ctas, st); break;
            case 4: launch_persist<4>(ctx, pctl, pcl.ctas, st); break;
            case 5: launch_persist<5>(ctx, pctl, pcl.ctas, st); break;
            case 6: launch_persist<6>(ctx, pctl, pcl.ctas, st); break;
            case 7: launch_persist<7>(ctx, pctl, pcl.ctas, st); break;
            default: launch_persist<8>(ctx, pctl, pcl.ctas, st); break;
            }
        }
        if (pfork)
            for (int k = 0; k < std::min(nclass, MAX_CLASS_STREAMS); ++k) {
                CK(cudaEventRecord(ctx->join_ev[k], ctx->class_stream[k]));
                CK(cudaStreamWaitEvent(ctx->stream, ctx->join_ev[k], 0));
            }
        CK(cudaGetLastError());
        P.launches = launches;
        return BPMAX_OK;
    }
    // pairs of different inner widths never interact: each width class runs its own chain of
    // diagonals on its own stream (parallel branches of the captured graph); profiling runs
    // serialise everything on the main stream so every launch can be timed
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(ctx->stream, &cap));
    const bool capturing = cap == cudaStreamCaptureStatusActive;
    const bool fork = !prof && P.classes.size() > 1 && P.class_streams;
    auto chain_of = [&](int np) {
        if (!fork) return 0;
        return (int)(std::find(P.classes.begin(), P.classes.end(), np) - P.classes.begin()) % MAX_CLASS_STREAMS;
    };
    auto stream_of = [&](int np) { return fork ? ctx->class_stream[chain_of(np)] : ctx->stream; };
    const int nstreams = fork ? std::min((int)P.classes.size(), MAX_CLASS_STREAMS) : 0;
    if (fork) {
        CK(cudaEventRecord(ctx->fork_ev, ctx->stream));
        for (int k = 0; k < nstreams; ++k) CK(cudaStreamWaitEvent(ctx->class_stream[k], ctx->fork_ev, 0));
    }
    size_t ri = 0, fi = 0;
    // outer diagonal final after step d (tile tables: with its last tile diagonal)
    const int lag = P.classes.back() > MAX_SMALL_NP && !P.r0_only ? P.classes.back() / 64 - 1 : 0;
    for (int d = 0; d < P.steps; ++d) {
        for (; ri < P.r0_launches.size() && P.r0_launches[ri].d == d; ++ri, ++launches) {
            const auto &L = P.r0_launches[ri];
            const cudaStream_t st = stream_of(L.np);
            {
                ProfScope ps(ctx, kp, 1);
                switch (L.np > MAX_SMALL_NP ? 0 : L.np / 8) {
                case 0: launch_r0_wide(ctx, P, L, st); break;
                case 1: launch_r0<1>(ctx, P, L, st); break;
                case 2: launch_r0<2>(ctx, P, L, st); break;
                case 3: launch_r0<3>(ctx, P, L, st); break;
                case 4: launch_r0<4>(ctx, P, L, st); break;
                case 5: launch_r0<5>(ctx, P, L, st); break;
                case 6: launch_r0<6>(ctx, P, L, st); break;
                case 7: launch_r0<7>(ctx, P, L, st); break;
                default: launch_r0<8>(ctx, P, L, st); break;
                }
            }
        }
        for (; fi < P.fin_launches.size() && P.fin_launches[fi].d == d; ++fi, ++launches) {
            const auto &L = P.fin_launches[fi];
            const cudaStream_t st = stream_of(L.np);
            {
                ProfScope ps(ctx, kp, 2);
                if (P.r0_only) {
                    launch_r0only_fin(ctx, L, st);
                } else {
                    switch (L.np > MAX_SMALL_NP ? 0 : L.np / 8) {
                    case 0: launch_fin_tiles(ctx, L, st); break;
                    case 1: launch_fin<1>(ctx, L, st); break;
                    case 2: launch_fin<2>(ctx, L, st); break;
                    case 3: launch_fin<3>(ctx, L, st); break;
                    case 4: launch_fin<4>(ctx, L, st); break;
                    case 5: launch_fin<5>(ctx, L, st); break;
                    case 6: launch_fin<6>(ctx, L, st); break;
                    case 7: launch_fin<7>(ctx, L, st); break;
                    default: launch_fin<8>(ctx, L, st); break;
                    }
                }
            }
        }
        // outer diagonal d is final: rows of the reference layout that end on it can be copied out
        // (in a captured graph the events are external nodes)
        if (!P.diag_ev.empty() && !prof && d >= lag && P.diag_ev[d - lag])
            CK(cudaEventRecordWithFlags(P.diag_ev[d - lag], ctx->stream, capturing ? cudaEventRecordExternal : cudaEventRecordDefault));
    }
    for (int k = 0; k < nstreams; ++k) {  // join the class chains back into the main stream
        CK(cudaEventRecord(ctx->join_ev[k], ctx->class_stream[k]));
        CK(cudaStreamWaitEvent(ctx->stream, ctx->join_ev[k], 0));
    }
    CK(cudaGetLastError());
    P.launches = launches;
    return BPMAX_OK;
}

// Makes the plan for these shapes current (reusing the cached one and its graph when the
// shapes repeat) and uploads the sequences. Sequences are validated by the caller.
int prepare(bpmax_ctx *ctx, const std::vector<int> &Ms, const std::vector<int> &Ns,
            const std::vector<const int *> &s1s, const std::vector<const int *> &s2s)
{
    int st;
    const auto tu = ctx->tuned.find(shape_key(Ms, Ns));
    const Tuned want = tu != ctx->tuned.end() ? tu->second
                                              : Tuned{ctx->r0_pairs_per_job, ctx->r0_merge_items, ctx->class_streams,
                                                      ctx->r0_variant, ctx->wide_stages, ctx->class_share, ctx->persist};
    const bool same_tuning = ctx->plan.pairs_per_job == want[0] && ctx->plan.merge_items == want[1] &&
                             ctx->plan.class_streams == want[2] && ctx->plan.r0_variant == want[3] &&
                             ctx->plan.wide_stages == want[4] && ctx->plan.class_share == want[5] &&
                             ctx->plan.persist == want[6] && ctx->plan.strip_tasks == ctx->strip_tasks &&
                             ctx->plan.copyout == ctx->copyout &&
                             ctx->plan.ref.out == ctx->want_ref.out && ctx->plan.ref.T == ctx->want_ref.T &&
                             ctx->plan.ref.Ns == ctx->want_ref.Ns;
    if (!(ctx->plan_valid && ctx->plan.Ms == Ms && ctx->plan.Ns == Ns && same_tuning && ctx->plan.r0_only == ctx->r0_only)) {
        if (ctx->plan.graph) cudaGraphExecDestroy(ctx->plan.graph);
        ctx->plan.graph = nullptr;
        for (cudaEvent_t e : ctx->plan.diag_ev)
            if (e) cudaEventDestroy(e);
        ctx->plan.diag_ev.clear();
        ctx->plan_valid = false;
        if ((st = build_plan(ctx, Ms, Ns, ctx->plan)) != BPMAX_OK) return st;
        Plan &P = ctx->plan;
        P.r0_only = ctx->r0_only;
        P.ref = ctx->want_ref;
        if (P.copyout) {  // an event per COPYOUT_DIAGS diagonals, and one after the last
            P.diag_ev.assign(P.maxM, nullptr);
            for (int d = 0; d < P.maxM; ++d)
                if (d % COPYOUT_DIAGS == COPYOUT_DIAGS - 1 || d == P.maxM - 1)
                    CK(cudaEventCreateWithFlags(&P.diag_ev[d], cudaEventDisableTiming));
        }
        if ((st = ensure(ctx, ctx->F, P.F_floats * sizeof(float))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->errflag, sizeof(int))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->S, P.S_floats * sizeof(float))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->bases, P.bases_bytes + 16)) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->pairs, P.pairs.size() * sizeof(PairDesc))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->r0jobs, P.r0_jobs.size() * sizeof(R0Job))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->stripjobs, P.strip_jobs.size() * sizeof(StripJob))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->r0wjobs, P.r0w_jobs.size() * sizeof(R0JobW))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->tilejobs, P.tile_jobs.size() * sizeof(TileJob))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->widepairs, P.wide_pairs.size() * sizeof(int))) != BPMAX_OK) return st;
        if (P.persistent) {
            if ((st = ensure(ctx, ctx->pq, P.pitems.size() * sizeof(PItem))) != BPMAX_OK) return st;
            if ((st = ensure(ctx, ctx->pneed, P.prod_need.size() * sizeof(int))) != BPMAX_OK) return st;
            if ((st = ensure(ctx, ctx->pcnt, (64 + align64(P.n_counters) + P.prod_need.size()) * sizeof(int))) != BPMAX_OK)
                return st;
            CK(cudaMemcpyAsync(ctx->pq.p, P.pitems.data(), P.pitems.size() * sizeof(PItem), cudaMemcpyHostToDevice,
                               ctx->stream));
            CK(cudaMemcpyAsync(ctx->pneed.p, P.prod_need.data(), P.prod_need.size() * sizeof(int),
                               cudaMemcpyHostToDevice, ctx->stream));
        }
        if ((st = ensure(ctx, ctx->celljobs, P.cell_jobs.size() * sizeof(CellJob))) != BPMAX_OK) return st;
        if ((st = ensure(ctx, ctx->scores, P.pairs.size() * sizeof(float))) != BPMAX_OK) return st;
        CK(cudaMemcpyAsync(ctx->pairs.p, P.pairs.data(), P.pairs.size() * sizeof(PairDesc), cudaMemcpyHostToDevice, ctx->stream));
        if (!P.r0_jobs.empty())
            CK(cudaMemcpyAsync(ctx->r0jobs.p, P.r0_jobs.data(), P.r0_jobs.size() * sizeof(R0Job), cudaMemcpyHostToDevice, ctx->stream));
        if (!P.strip_jobs.empty())
            CK(cudaMemcpyAsync(ctx->stripjobs.p, P.strip_jobs.data(), P.strip_jobs.size() * sizeof(StripJob),
                               cudaMemcpyHostToDevice, ctx->stream));
        if (!P.r0w_jobs.empty())
            CK(cudaMemcpyAsync(ctx->r0wjobs.p, P.r0w_jobs.data(), P.r0w_jobs.size() * sizeof(R0JobW), cudaMemcpyHostToDevice,
                               ctx->stream));
        if (!P.tile_jobs.empty())
            CK(cudaMemcpyAsync(ctx->tilejobs.p, P.tile_jobs.data(), P.tile_jobs.size() * sizeof(TileJob),
                               cudaMemcpyHostToDevice, ctx->stream));
        if (!P.wide_pairs.empty())
            CK(cudaMemcpyAsync(ctx->widepairs.p, P.wide_pairs.data(), P.wide_pairs.size() * sizeof(int),
                               cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaMemcpyAsync(ctx->celljobs.p, P.cell_jobs.data(), P.cell_jobs.size() * sizeof(CellJob), cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        ctx->plan_valid = true;
    }
    Plan &P = ctx->plan;
    if (P.r0_only) {  // the sequences are the base values themselves: seq1, then seq2 unreversed
        std::vector<float> hv;
        for (int i = 0; i < Ms[0]; ++i) hv.push_back((float)s1s[0][i]);
        for (int i = 0; i < Ns[0]; ++i) hv.push_back((float)s2s[0][i]);
        if ((st = ensure(ctx, ctx->r0vals, hv.size() * sizeof(float))) != BPMAX_OK) return st;
        CK(cudaMemcpyAsync(ctx->r0vals.p, hv.data(), hv.size() * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        return BPMAX_OK;
    }
    // sequences: seq1 as is, seq2 reversed (V3/transform_reverse_1D_to_2D.c:131-135)
    std::vector<uint8_t> hb(P.bases_bytes);
    for (size_t p = 0; p < P.pairs.size(); ++p) {
        const PairDesc &pd = P.pairs[p];
        for (int i = 0; i < pd.M; ++i) hb[pd.seq1_off + i] = (uint8_t)s1s[p][i];
        for (int i = 0; i < pd.N; ++i) hb[pd.seq2_off + i] = (uint8_t)s2s[p][pd.N - 1 - i];
    }
    CK(cudaMemcpyAsync(ctx->bases.p, hb.data(), hb.size(), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return BPMAX_OK;
}

// Launches the fill of the current plan on the context's stream.
int launch_fill(bpmax_ctx *ctx)
{
    Plan &P = ctx->plan;
    int st;
    // The first run of a plan is launched as it is, and so is the test of the timeout path; a graph is
    // captured when the shapes come a second time. Capturing and instantiating one takes about a
    // millisecond for a 200-long strand 1, which launches that run ahead of the GPU do not cost: 24 pairs
    // of different shapes one by one 101 -> 82 ms.
    if (ctx->inject_wait_timeout || (!P.graph && !P.ran)) {
        P.ran = !ctx->inject_wait_timeout;
        CK(cudaEventRecord(ctx->ev0, ctx->stream));
        if ((st = enqueue_fill(ctx, P)) != BPMAX_OK) return st;
        CK(cudaEventRecord(ctx->ev1, ctx->stream));
        gather_scores_kernel<<<((int)P.pairs.size() + 127) / 128, 128, 0, ctx->stream>>>(
            (const PairDesc *)ctx->pairs.p, (const float *)ctx->F.p, (int)P.pairs.size(), (float *)ctx->scores.p);
        CK(cudaGetLastError());
        return BPMAX_OK;
    }
    if (!P.graph) {
        cudaGraph_t g;
        CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        st = enqueue_fill(ctx, P);
        cudaGraph_t captured = nullptr;
        cudaError_t ce = cudaStreamEndCapture(ctx->stream, &captured);
        if (st != BPMAX_OK) {
            if (captured) cudaGraphDestroy(captured);
            return st;
        }
        if (ce != cudaSuccess) return fail(ctx, BPMAX_ECUDA, "graph capture: %s", cudaGetErrorString(ce));
        g = captured;
        CK(cudaGraphInstantiate(&P.graph, g, 0));
        cudaGraphDestroy(g);
    }
    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    CK(cudaGraphLaunch(P.graph, ctx->stream));
    CK(cudaEventRecord(ctx->ev1, ctx->stream));
    gather_scores_kernel<<<((int)P.pairs.size() + 127) / 128, 128, 0, ctx->stream>>>(
        (const PairDesc *)ctx->pairs.p, (const float *)ctx->F.p, (int)P.pairs.size(), (float *)ctx->scores.p);
    CK(cudaGetLastError());
    return BPMAX_OK;
}

// Waits for the fill launched by launch_fill, reads its error word and times it.
int finish_fill(bpmax_ctx *ctx)
{
    Plan &P = ctx->plan;
    int errv = 0;
    CK(cudaMemcpyAsync(&errv, ctx->errflag.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaEventSynchronize(ctx->ev1));
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaEventElapsedTime(&ctx->last_ms, ctx->ev0, ctx->ev1));
    ctx->last_launches = P.launches + 1;  // + the score gather
    const bool injected = ctx->inject_wait_timeout;
    ctx->inject_wait_timeout = false;  // one-shot
    if (errv)
        return fail(ctx, BPMAX_ETIMEOUT, "a product kernel gave up waiting for its operand copies%s",
                    injected ? " (test mode: no copies were issued)" : "");
    return BPMAX_OK;
}

int run_fill(bpmax_ctx *ctx)
{
    const int st = launch_fill(ctx);
    return st ? st : finish_fill(ctx);
}

int check_pair(bpmax_ctx *ctx, const int *s1, long M, const int *s2, long N)
{
    if (!s1 || !s2) return fail(ctx, BPMAX_EINVAL, "null sequence pointer");
    if (M < 1 || N < 1) return fail(ctx, BPMAX_EINVAL, "sequence lengths must be >= 1 (M=%ld, N=%ld)", M, N);
    if (M > 65535 || N > MAX_NP) return fail(ctx, BPMAX_EINVAL, "sequence length too large (M=%ld, N=%ld)", M, N);
    for (long i = 0; i < M; ++i)
        if (s1[i] < 0 || s1[i] > 4) return fail(ctx, BPMAX_EINVAL, "seq1[%ld]=%d is not a base code 0..4", i, s1[i]);
    for (long i = 0; i < N; ++i)
        if (s2[i] < 0 || s2[i] > 4) return fail(ctx, BPMAX_EINVAL, "seq2[%ld]=%d is not a base code 0..4", i, s2[i]);
    return BPMAX_OK;
}

int fill_pairs(bpmax_ctx *ctx, int num_pairs, const int *const *seq1s, const long *Ms, const int *const *seq2s,
               const long *Ns, bool async = false)
{
    if (!ctx) return BPMAX_EINVAL;
    if (num_pairs < 1 || !seq1s || !seq2s || !Ms || !Ns) return fail(ctx, BPMAX_EINVAL, "empty batch");
    std::vector<int> vm(num_pairs), vn(num_pairs);
    std::vector<const int *> a(num_pairs), b(num_pairs);
    for (int p = 0; p < num_pairs; ++p) {
        int st = check_pair(ctx, seq1s[p], Ms[p], seq2s[p], Ns[p]);
        if (st) return st;
        vm[p] = (int)Ms[p];
        vn[p] = (int)Ns[p];
        a[p] = seq1s[p];
        b[p] = seq2s[p];
    }
    CK(cudaSetDevice(ctx->device));
    int st = prepare(ctx, vm, vn, a, b);
    if (st) return st;
    return async ? launch_fill(ctx) : run_fill(ctx);
}

int ensure_host_stage(bpmax_ctx *ctx, size_t bytes)
{
    if (ctx->host_stage_bytes >= bytes) return BPMAX_OK;
    for (int i = 0; i < 2; ++i) {
        if (ctx->host_stage[i]) cudaFreeHost(ctx->host_stage[i]);
        ctx->host_stage[i] = nullptr;
    }
    ctx->host_stage_bytes = 0;
    for (int i = 0; i < 2; ++i) CK(cudaMallocHost(&ctx->host_stage[i], bytes));
    ctx->host_stage_bytes = bytes;
    return BPMAX_OK;
}

cudaMemoryType memory_type(const void *p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return cudaMemoryTypeUnregistered;
    }
    return at.type;
}

bool is_pinned(const void *p) { return memory_type(p) == cudaMemoryTypeHost; }

// Whether more than a sixteenth of the pages of [dst, dst + bytes) are missing, as in an array never written; not where
// the system cannot tell.
bool is_fresh(const void *dst, size_t bytes)
{
    constexpr size_t CHUNK = (size_t)2 << 20;
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    const uintptr_t lo = ((uintptr_t)dst + page - 1) / page * page, hi = ((uintptr_t)dst + bytes) / page * page;
    unsigned char here[CHUNK / 4096];
    size_t missing = 0;
    for (uintptr_t p = lo; p < hi; p += CHUNK) {
        const size_t n = std::min<uintptr_t>(CHUNK, hi - p), pages = n / page;
        if (mincore((void *)p, n, here) != 0) return false;
        missing += std::count_if(here, here + pages, [](unsigned char c) { return !(c & 1); });
    }
    return missing * page > bytes / 16;
}

// Copies `bytes` of device memory to dst, after the work queued on the context's stream, and waits. Into
// fresh pageable memory of COPY_SPLIT bytes or more: COPY_THREADS threads take chunks in turn, each through two
// pinned buffers of its own on a class stream, so one chunk crosses PCIe while another is copied to its
// place. The driver's own staged copy runs at 16 to 19 GB/s, but faults in a fresh array's pages one after another,
// at 2 GB/s (5 in 2 MB pages). ms per table, plain copy / threads: into an array in use 3.1 MB 0.25 / 0.30, 31 MB 2.0 / 2.4;
// into a fresh one 1.46 / 0.43 and 14.2 / 2.7. The pinned buffers take 1 to 3 ms to allocate: a context has them
// from its COPY_WORTH bytes into fresh memory on (first table of a context, plain / with that allocation: 6.2 MB
// 3.2 / 3.5, 9.4 MB 4.9 / 4.0). 128x32 table into a new array: 10.1 -> 4.9 ms a call (4.5 with chunks of 512 KB, whose
// 8 MB of pinned buffers cost a new context 5 ms).
constexpr size_t COPY_SPLIT = (size_t)2 << 20, COPY_CHUNK = (size_t)128 << 10, COPY_WORTH = (size_t)8 << 20;
constexpr int COPY_THREADS = MAX_CLASS_STREAMS;
int copy_out(bpmax_ctx *ctx, void *dst, const void *src, size_t bytes)
{
    const int threads = (int)std::min<size_t>(std::min<size_t>(COPY_THREADS, bytes / COPY_CHUNK),
                                              std::max(1u, std::thread::hardware_concurrency()));
    bool split = bytes >= COPY_SPLIT && threads >= 2 && memory_type(dst) == cudaMemoryTypeUnregistered && is_fresh(dst, bytes);
    if (split) {
        ctx->fresh_bytes += bytes;
        split = ctx->fresh_bytes >= COPY_WORTH;
    }
    if (split && !ctx->copy_stage &&
        cudaMallocHost(&ctx->copy_stage, 2 * COPY_THREADS * COPY_CHUNK) != cudaSuccess) {
        cudaGetLastError();  // no pinned memory left: the plain copy
        ctx->copy_stage = nullptr;
        split = false;
    }
    if (!split) {
        CK(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        return BPMAX_OK;
    }
    CK(cudaEventRecord(ctx->fork_ev, ctx->stream));
    cudaError_t errs[COPY_THREADS] = {};
    auto work = [&](int t) {
        cudaError_t &e = errs[t];
        if ((e = cudaSetDevice(ctx->device)) != cudaSuccess) return;
        const cudaStream_t st = ctx->class_stream[t];
        if ((e = cudaStreamWaitEvent(st, ctx->fork_ev, 0)) != cudaSuccess) return;
        char *buf = (char *)ctx->copy_stage + 2 * t * COPY_CHUNK;
        size_t at = t * COPY_CHUNK, prev = 0, prev_n = 0;
        for (int k = 0; at < bytes; ++k, at += (size_t)threads * COPY_CHUNK) {
            const size_t n = std::min(COPY_CHUNK, bytes - at);
            // the chunk before is in the other buffer: wait for it, then send for this one and move that one
            if (k > 0 && (e = cudaStreamSynchronize(st)) != cudaSuccess) return;
            e = cudaMemcpyAsync(buf + (k & 1) * COPY_CHUNK, (const char *)src + at, n, cudaMemcpyDeviceToHost, st);
            if (e != cudaSuccess) return;
            if (k > 0) memcpy((char *)dst + prev, buf + (~k & 1) * COPY_CHUNK, prev_n);
            prev = at;
            prev_n = n;
        }
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess || !prev_n) return;
        const size_t last = (prev / COPY_CHUNK / threads) & 1;
        memcpy((char *)dst + prev, buf + last * COPY_CHUNK, prev_n);
    };
    std::thread pool[COPY_THREADS];
    int started = 1;  // this thread is the first worker, and does the parts of any that could not start
    try {
        for (; started < threads; ++started) pool[started] = std::thread(work, started);
    } catch (...) {
    }
    work(0);
    for (int t = started; t < threads; ++t) work(t);
    for (int t = 1; t < started; ++t) pool[t].join();
    for (int t = 0; t < threads; ++t) CK(errs[t]);
    return BPMAX_OK;
}

}  // namespace

extern "C" {

const char *bpmax_gpu_status_string(int s)
{
    switch (s) {
    case BPMAX_OK: return "ok";
    case BPMAX_EINVAL: return "invalid argument";
    case BPMAX_ENOMEM: return "out of memory";
    case BPMAX_ECUDA: return "CUDA error";
    case BPMAX_ENODEV: return "no usable CUDA device";
    case BPMAX_ETIMEOUT: return "device wait timed out";
    default: return "unknown status";
    }
}

int bpmax_gpu_create(int device, bpmax_ctx **out)
{
    if (!out) return BPMAX_EINVAL;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
        cudaGetLastError();
        return BPMAX_ENODEV;
    }
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess || prop.major != 10) {
        cudaGetLastError();
        return BPMAX_ENODEV;  // the kernels are built for sm_100a only
    }
    bpmax_ctx *ctx = new bpmax_ctx();
    ctx->device = device;
    ctx->sms = prop.multiProcessorCount;
    const float ref_w[12] = {1.0f, 1.0f, 3.0f, 3.0f, 1.5f, 1.5f, 1.0f, 1.0f, 3.0f, 3.0f, 1.5f, 1.5f};
    memcpy(ctx->W.w, ref_w, sizeof ref_w);
    int st = BPMAX_OK;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&ctx->ev0) != cudaSuccess || cudaEventCreate(&ctx->ev1) != cudaSuccess ||
        cudaEventCreateWithFlags(&ctx->stage_ev[0], cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&ctx->stage_ev[1], cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&ctx->fork_ev, cudaEventDisableTiming) != cudaSuccess)
        st = BPMAX_ECUDA;
    if (st == BPMAX_OK && cudaStreamCreateWithFlags(&ctx->aux_stream, cudaStreamNonBlocking) != cudaSuccess) st = BPMAX_ECUDA;
    for (int k = 0; k < MAX_CLASS_STREAMS && st == BPMAX_OK; ++k)
        if (cudaStreamCreateWithFlags(&ctx->class_stream[k], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&ctx->join_ev[k], cudaEventDisableTiming) != cudaSuccess)
            st = BPMAX_ECUDA;
    if (st == BPMAX_OK) st = set_smem_attr<1>(ctx);
    if (st == BPMAX_OK) st = set_smem_attr<2>(ctx);
    if (st == BPMAX_OK) st = set_smem_attr<3>(ctx);
    if (st == BPMAX_OK) st = set_smem_attr<4>(ctx);
    if (st == BPMAX_OK) st = set_smem_attr<5>(ctx);
    if (st == BPMAX_OK) st = set_smem_attr<6>(ctx);
    if (st == BPMAX_OK) st = set_smem_attr<7>(ctx);
    if (st == BPMAX_OK) st = set_smem_attr<8>(ctx);
    if (st != BPMAX_OK) {
        cudaGetLastError();
        bpmax_gpu_destroy(ctx);
        return st;
    }
    *out = ctx;
    return BPMAX_OK;
}

void bpmax_gpu_destroy(bpmax_ctx *ctx)
{
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    if (ctx->plan.graph) cudaGraphExecDestroy(ctx->plan.graph);
    for (DevBuf *b : {&ctx->tbstack, &ctx->grads, &ctx->tbstatus, &ctx->F, &ctx->S, &ctx->bases, &ctx->pairs,
                      &ctx->r0jobs, &ctx->stripjobs, &ctx->r0wjobs, &ctx->tilejobs, &ctx->widepairs, &ctx->pq, &ctx->pcnt, &ctx->pneed, &ctx->celljobs,
                      &ctx->scores, &ctx->conv, &ctx->refdev, &ctx->errflag,
                      &ctx->r0vals})
        if (b->p) cudaFree(b->p);
    for (int i = 0; i < 2; ++i) {
        if (ctx->host_stage[i]) cudaFreeHost(ctx->host_stage[i]);
        if (ctx->stage_ev[i]) cudaEventDestroy(ctx->stage_ev[i]);
    }
    if (ctx->copy_stage) cudaFreeHost(ctx->copy_stage);
    if (ctx->ev0) cudaEventDestroy(ctx->ev0);
    if (ctx->ev1) cudaEventDestroy(ctx->ev1);
    if (ctx->fork_ev) cudaEventDestroy(ctx->fork_ev);
    for (cudaEvent_t e : ctx->plan.diag_ev)
        if (e) cudaEventDestroy(e);
    if (ctx->aux_stream) cudaStreamDestroy(ctx->aux_stream);
    for (int k = 0; k < MAX_CLASS_STREAMS; ++k) {
        if (ctx->class_stream[k]) cudaStreamDestroy(ctx->class_stream[k]);
        if (ctx->join_ev[k]) cudaEventDestroy(ctx->join_ev[k]);
    }
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}

const char *bpmax_gpu_last_error(const bpmax_ctx *ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int bpmax_gpu_set_weights(bpmax_ctx *ctx, const float *w)
{
    if (!ctx) return BPMAX_EINVAL;
    if (!w || !weights_ok(w)) return fail(ctx, BPMAX_EINVAL, "weights must be 12 finite values >= +0");
    memcpy(ctx->W.w, w, sizeof ctx->W.w);
    // weights are kernel arguments baked into the captured graph: recapture on next use
    if (ctx->plan.graph) {
        cudaGraphExecDestroy(ctx->plan.graph);
        ctx->plan.graph = nullptr;
    }
    ctx->plan.ran = false;
    return BPMAX_OK;
}

int bpmax_gpu_score(bpmax_ctx *ctx, const int *seq1, long M, const int *seq2, long N, float *score)
{
    if (!ctx) return BPMAX_EINVAL;
    int st = fill_pairs(ctx, 1, &seq1, &M, &seq2, &N);
    if (st) return st;
    if (score) CK(cudaMemcpy(score, ctx->scores.p, sizeof(float), cudaMemcpyDeviceToHost));
    return BPMAX_OK;
}

int bpmax_gpu_score_batch(bpmax_ctx *ctx, int num_pairs, const int *const *seq1s, const long *Ms,
                          const int *const *seq2s, const long *Ns, float *scores)
{
    if (!ctx) return BPMAX_EINVAL;
    int st = fill_pairs(ctx, num_pairs, seq1s, Ms, seq2s, Ns);
    if (st) return st;
    if (scores) CK(cudaMemcpy(scores, ctx->scores.p, num_pairs * sizeof(float), cudaMemcpyDeviceToHost));
    return BPMAX_OK;
}

int bpmax_gpu_score_each(bpmax_ctx *ctx, int num_pairs, const int *const *seq1s, const long *Ms,
                         const int *const *seq2s, const long *Ns, float *scores)
{
    if (!ctx) return BPMAX_EINVAL;
    if (num_pairs < 1) return fail(ctx, BPMAX_EINVAL, "empty batch");
    float total = 0.f;
    long launches = 0;
    for (int p = 0; p < num_pairs; ++p) {
        int st = fill_pairs(ctx, 1, seq1s + p, Ms + p, seq2s + p, Ns + p);
        if (st) return st;
        total += ctx->last_ms;
        launches += ctx->last_launches;
        if (scores) CK(cudaMemcpy(scores + p, ctx->scores.p, sizeof(float), cudaMemcpyDeviceToHost));
    }
    ctx->last_ms = total;
    ctx->last_launches = launches;
    return BPMAX_OK;
}

int bpmax_gpu_r0_only(bpmax_ctx *ctx, const int *seq1, long M, const int *seq2, long N, float *F_compact,
                      float *score)
{
    if (!ctx) return BPMAX_EINVAL;
    if (!seq1 || !seq2) return fail(ctx, BPMAX_EINVAL, "null sequence");
    // the reference's domain {M,N | M>=2 && N>=2} (IPDPSW/.../ospsq_float.ab:1)
    if (M < 2 || N < 2 || M > 65535) return fail(ctx, BPMAX_EINVAL, "The value of parameters are not valid.");
    if (padded_width((int)N) > MAX_NP) return fail(ctx, BPMAX_EINVAL, "strand-2 length %ld > %d is not supported", N, MAX_NP);
    for (long i = 0; i < M; ++i)
        if (seq1[i] < 0) return fail(ctx, BPMAX_EINVAL, "seq1[%ld] = %d < 0: values must be non-negative", i, seq1[i]);
    for (long i = 0; i < N; ++i)
        if (seq2[i] < 0) return fail(ctx, BPMAX_EINVAL, "seq2[%ld] = %d < 0: values must be non-negative", i, seq2[i]);
    CK(cudaSetDevice(ctx->device));
    ctx->r0_only = true;
    int st = prepare(ctx, {(int)M}, {(int)N}, {seq1}, {seq2});
    ctx->r0_only = false;
    if (st) return st;
    if ((st = run_fill(ctx)) != BPMAX_OK) return st;
    if (score) CK(cudaMemcpy(score, ctx->scores.p, sizeof(float), cudaMemcpyDeviceToHost));
    if (!F_compact) return BPMAX_OK;
    const long long n_out = M * (M + 1) / 2 * N * N;
    if ((st = ensure(ctx, ctx->conv, n_out * sizeof(float))) != BPMAX_OK) return st;
    to_compact_kernel<<<4 * ctx->sms, 256, 0, ctx->stream>>>((const PairDesc *)ctx->pairs.p, (const float *)ctx->F.p,
                                                             n_out, (float *)ctx->conv.p);
    CK(cudaGetLastError());
    return copy_out(ctx, F_compact, ctx->conv.p, n_out * sizeof(float));
}

int bpmax_gpu_fill_compact(bpmax_ctx *ctx, const int *seq1, long M, const int *seq2, long N, float *F_compact,
                           float *score)
{
    if (!ctx) return BPMAX_EINVAL;
    int st = fill_pairs(ctx, 1, &seq1, &M, &seq2, &N);
    if (st) return st;
    if (score) CK(cudaMemcpy(score, ctx->scores.p, sizeof(float), cudaMemcpyDeviceToHost));
    if (!F_compact) return BPMAX_OK;
    const long long n_out = M * (M + 1) / 2 * N * N;
    if ((st = ensure(ctx, ctx->conv, n_out * sizeof(float))) != BPMAX_OK) return st;
    to_compact_kernel<<<4 * ctx->sms, 256, 0, ctx->stream>>>((const PairDesc *)ctx->pairs.p, (const float *)ctx->F.p,
                                                             n_out, (float *)ctx->conv.p);
    CK(cudaGetLastError());
    return copy_out(ctx, F_compact, ctx->conv.p, n_out * sizeof(float));
}

int bpmax_gpu_fill(bpmax_ctx *ctx, const int *seq1, long M, const int *seq2, long N, long N_tile, float *F_lin,
                   float *score)
{
    if (!ctx) return BPMAX_EINVAL;
    // preconditions of V3/bpmax.c:131 (N_sec>=2 and 0<=R<N_tile follow from the layout)
    if (M < 1 || N < 8 || N_tile < 4) return fail(ctx, BPMAX_EINVAL, "The value of parameters are not valid.");
    const long Ns = (N + N_tile - 1) / N_tile;
    if (Ns < 2) return fail(ctx, BPMAX_EINVAL, "The value of parameters are not valid. (N_sec=%ld < 2)", Ns);
    if (!F_lin) {
        int st = fill_pairs(ctx, 1, &seq1, &M, &seq2, &N);
        if (st) return st;
        if (score) CK(cudaMemcpy(score, ctx->scores.p, sizeof(float), cudaMemcpyDeviceToHost));
        return BPMAX_OK;
    }
    const long long cell_f = (long long)Ns * Ns * (N_tile + 1) * N_tile;
    // The table is copied out while the fill still runs (aux stream, waiting on the per-diagonal
    // events the graph records). Into pinned memory: per outer diagonal, as soon as it is final --
    // its cells (i1, i1+d) lie (M+1) cells apart in the reference layout, so one strided copy
    // places a diagonal converted into a staging slot, and the copy-out ends one diagonal after the
    // fill. Into pageable memory (through a pinned staging buffer and a host copy): per outer row,
    // contiguous in the layout and final once outer diagonal M-1-i1 is, from the last one up.
    const long long row_max = (long long)M * cell_f;
    int st;
    if ((st = ensure(ctx, ctx->conv, 2 * row_max * sizeof(float))) != BPMAX_OK) return st;
    const bool pinned = is_pinned(F_lin);
    if (!pinned && (st = ensure_host_stage(ctx, row_max * sizeof(float))) != BPMAX_OK) return st;
    // Widths <= 64 into pinned memory: the finalize launches themselves write every cell they
    // complete in the reference layout (diagonal-major, on the device), so only copy engines work
    // beside the fill. Without room for that buffer, or wider, a conversion launch per diagonal does
    // it (those launches share the SMs with the fill's).
    const size_t fused_bytes = (size_t)(M * (M + 1) / 2) * cell_f * sizeof(float);
    bool fused = false;
    if (pinned && padded_width((int)N) <= MAX_SMALL_NP) {
        fused = ctx->refdev.bytes >= fused_bytes;
        if (!fused) {
            if (ctx->refdev.p) cudaFree(ctx->refdev.p);
            ctx->refdev = DevBuf{};
            void *p = nullptr;
            if (cudaMalloc(&p, fused_bytes) == cudaSuccess) {
                ctx->refdev = DevBuf{p, fused_bytes};
                fused = true;
            } else {
                cudaGetLastError();  // out of memory: not sticky, take the conversion launches
            }
        }
    }
    ctx->want_ref = fused ? RefOut{(float *)ctx->refdev.p, (int)N_tile, (int)Ns} : RefOut{nullptr, 0, 0};
    ctx->copyout = true;
    st = fill_pairs(ctx, 1, &seq1, &M, &seq2, &N, true);
    ctx->copyout = false;
    ctx->want_ref = RefOut{nullptr, 0, 0};
    if (st != BPMAX_OK) return st;
    // the event after which outer diagonal d is final
    auto dev = [&](long d) { return ctx->plan.diag_ev[std::min(M - 1, d | (COPYOUT_DIAGS - 1))]; };
    if (fused) {
        const size_t cell_b = (size_t)cell_f * sizeof(float);
        for (long d = 0; d < M; ++d) {
            const float *src = (const float *)ctx->refdev.p + (d * M - d * (d - 1) / 2) * cell_f;
            CK(cudaStreamWaitEvent(ctx->aux_stream, dev(d), 0));
            CK(cudaMemcpy2DAsync(F_lin + d * cell_f, (size_t)(M + 1) * cell_b, src, cell_b, cell_b, (size_t)(M - d),
                                 cudaMemcpyDeviceToHost, ctx->aux_stream));
        }
        CK(cudaStreamSynchronize(ctx->aux_stream));
        if ((st = finish_fill(ctx)) != BPMAX_OK) return st;
        if (score) CK(cudaMemcpy(score, ctx->scores.p, sizeof(float), cudaMemcpyDeviceToHost));
        return BPMAX_OK;
    }
    if (pinned) {
        const size_t cell_b = (size_t)cell_f * sizeof(float);
        for (long d = 0; d < M; ++d) {
            float *slot = (float *)ctx->conv.p + (d & 1) * row_max;
            const long long n_out = (M - d) * cell_f;
            CK(cudaStreamWaitEvent(ctx->aux_stream, dev(d), 0));
            to_reference_diag_kernel<<<(int)std::min<long long>(4 * ctx->sms, (n_out + 255) / 256), 256, 0,
                                       ctx->aux_stream>>>((const PairDesc *)ctx->pairs.p, (const float *)ctx->F.p,
                                                          (int)N_tile, (int)Ns, (int)d, n_out, slot);
            CK(cudaGetLastError());
            CK(cudaMemcpy2DAsync(F_lin + d * cell_f, (size_t)(M + 1) * cell_b, slot, cell_b, cell_b, (size_t)(M - d),
                                 cudaMemcpyDeviceToHost, ctx->aux_stream));
        }
        CK(cudaStreamSynchronize(ctx->aux_stream));
        if ((st = finish_fill(ctx)) != BPMAX_OK) return st;
        if (score) CK(cudaMemcpy(score, ctx->scores.p, sizeof(float), cudaMemcpyDeviceToHost));
        return BPMAX_OK;
    }
    std::vector<long long> pending_n(2, 0);
    std::vector<float *> pending_dst(2, nullptr);
    for (long i1 = M - 1; i1 >= 0; --i1) {
        const int slot = (int)(i1 & 1);
        float *dbuf = (float *)ctx->conv.p + slot * row_max;
        const long long n_out = (M - i1) * cell_f;
        float *dst = F_lin + (i1 * M + i1) * cell_f;
        if (pending_dst[slot]) {  // drain the staging buffer this slot used before
            CK(cudaEventSynchronize(ctx->stage_ev[slot]));
            memcpy(pending_dst[slot], ctx->host_stage[slot], pending_n[slot] * sizeof(float));
            pending_dst[slot] = nullptr;
        }
        CK(cudaStreamWaitEvent(ctx->aux_stream, dev(M - 1 - i1), 0));
        to_reference_row_kernel<<<4 * ctx->sms, 256, 0, ctx->aux_stream>>>(
            (const PairDesc *)ctx->pairs.p, (const float *)ctx->F.p, (int)N_tile, (int)Ns, (int)i1, n_out, dbuf);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(ctx->host_stage[slot], dbuf, n_out * sizeof(float), cudaMemcpyDeviceToHost, ctx->aux_stream));
        CK(cudaEventRecord(ctx->stage_ev[slot], ctx->aux_stream));
        pending_dst[slot] = dst;
        pending_n[slot] = n_out;
    }
    for (int slot = 0; slot < 2; ++slot)
        if (pending_dst[slot]) {
            CK(cudaEventSynchronize(ctx->stage_ev[slot]));
            memcpy(pending_dst[slot], ctx->host_stage[slot], pending_n[slot] * sizeof(float));
        }
    CK(cudaStreamSynchronize(ctx->aux_stream));
    if ((st = finish_fill(ctx)) != BPMAX_OK) return st;
    if (score) CK(cudaMemcpy(score, ctx->scores.p, sizeof(float), cudaMemcpyDeviceToHost));
    return BPMAX_OK;
}

int bpmax_gpu_grad_batch(bpmax_ctx *ctx, int num_pairs, const int *const *seq1s, const long *Ms,
                         const int *const *seq2s, const long *Ns, float *scores, float *grads)
{
    if (!ctx) return BPMAX_EINVAL;
    int st = fill_pairs(ctx, num_pairs, seq1s, Ms, seq2s, Ns);
    if (st) return st;
    long maxlen = 0;
    for (int p = 0; p < num_pairs; ++p) maxlen = std::max(maxlen, Ms[p] + Ns[p]);
    const int cap = (int)(2 * maxlen + 64);  // DFS depth of the argmax tree <= M + N + 1
    if ((st = ensure(ctx, ctx->tbstack, (size_t)num_pairs * cap * sizeof(TbNode))) != BPMAX_OK) return st;
    if ((st = ensure(ctx, ctx->grads, (size_t)num_pairs * 12 * sizeof(float))) != BPMAX_OK) return st;
    if ((st = ensure(ctx, ctx->tbstatus, (size_t)num_pairs * sizeof(int))) != BPMAX_OK) return st;
    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    traceback_kernel<<<num_pairs, TB_THREADS, 0, ctx->stream>>>(
        (const PairDesc *)ctx->pairs.p, (const float *)ctx->F.p, (const float *)ctx->S.p, (const uint8_t *)ctx->bases.p,
        ctx->W, (TbNode *)ctx->tbstack.p, cap, (float *)ctx->grads.p, (int *)ctx->tbstatus.p);
    CK(cudaGetLastError());
    CK(cudaEventRecord(ctx->ev1, ctx->stream));
    std::vector<int> stat(num_pairs);
    CK(cudaMemcpyAsync(stat.data(), ctx->tbstatus.p, num_pairs * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    if (scores) CK(cudaMemcpyAsync(scores, ctx->scores.p, num_pairs * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    if (grads) CK(cudaMemcpyAsync(grads, ctx->grads.p, num_pairs * 12 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    float tb_ms = 0.f;
    CK(cudaEventElapsedTime(&tb_ms, ctx->ev0, ctx->ev1));
    ctx->last_ms += tb_ms;
    ctx->last_launches += 1;
    for (int p = 0; p < num_pairs; ++p)
        if (stat[p]) return fail(ctx, BPMAX_ECUDA, "adjoint pass of pair %d stopped (status %d)", p, stat[p]);
    return BPMAX_OK;
}

int bpmax_gpu_profile_kernels(bpmax_ctx *ctx, float *ms, long *launches, double *terms)
{
    if (!ctx) return BPMAX_EINVAL;
    if (!ctx->plan_valid) return fail(ctx, BPMAX_EINVAL, "no fill has run on this context");
    CK(cudaSetDevice(ctx->device));
    KernelProfile kp;
    kp.on = true;
    CK(cudaEventCreate(&kp.a));
    CK(cudaEventCreate(&kp.b));
    int st = enqueue_fill(ctx, ctx->plan, &kp);
    cudaEventDestroy(kp.a);
    cudaEventDestroy(kp.b);
    if (st) return st;
    CK(cudaStreamSynchronize(ctx->stream));
    // algorithmic candidates per kind
    auto C = [](double n) { return n * (n * n - 1) / 6.0; };
    auto T = [](double n) { return n * (n + 1) / 2.0; };
    double t[3] = {0, 0, 0};
    for (const PairDesc &pd : ctx->plan.pairs) {
        if (ctx->plan.r0_only) {  // the double max-plus alone; the other kinds only place values
            t[1] += C(pd.M) * C(pd.N);
            continue;
        }
        t[0] += C(pd.M) + C(pd.N);
        t[1] += C(pd.M) * (C(pd.N) + 2 * T(pd.N));
        t[2] += 2 * T(pd.M) * C(pd.N);
    }
    for (int k = 0; k < 3; ++k) {
        if (ms) ms[k] = kp.ms[k];
        if (launches) launches[k] = kp.launches[k];
        if (terms) terms[k] = t[k];
    }
    return BPMAX_OK;
}

int bpmax_gpu_maxplus_peak(bpmax_ctx *ctx, double *terms_per_s)
{
    if (!ctx || !terms_per_s) return BPMAX_EINVAL;
    CK(cudaSetDevice(ctx->device));
    float *buf = nullptr;
    const int grid = ctx->sms * 8, block = 128, reps = 250;
    CK(cudaMalloc(&buf, (size_t)grid * block * sizeof(float) + 64 * sizeof(float)));
    std::vector<float> h(64);
    for (int i = 0; i < 64; ++i) h[i] = (float)(i % 17);
    cudaMemcpyAsync(buf, h.data(), 64 * sizeof(float), cudaMemcpyHostToDevice, ctx->stream);
    maxplus_peak_kernel<<<grid, block, 0, ctx->stream>>>(buf, buf + 64, reps);
    cudaEventRecord(ctx->ev0, ctx->stream);
    for (int i = 0; i < 3; ++i) maxplus_peak_kernel<<<grid, block, 0, ctx->stream>>>(buf, buf + 64, reps);
    cudaEventRecord(ctx->ev1, ctx->stream);
    cudaError_t e = cudaEventSynchronize(ctx->ev1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    cudaFree(buf);
    if (e != cudaSuccess) return fail(ctx, BPMAX_ECUDA, "peak probe: %s", cudaGetErrorString(e));
    *terms_per_s = 3.0 * grid * block * (double)reps * (8.0 * MAXPLUS_PEAK_CHAINS) / (ms * 1e-3);
    return BPMAX_OK;
}

int bpmax_gpu_set_tuning(bpmax_ctx *ctx, int key, long value)
{
    if (!ctx) return BPMAX_EINVAL;
    switch (key) {
    case BPMAX_TUNE_R0_PAIRS_PER_JOB:
        if (value < 1) return fail(ctx, BPMAX_EINVAL, "pairs per job must be >= 1");
        ctx->r0_pairs_per_job = (int)std::min<long>(value, 1 << 20);
        break;
    case BPMAX_TUNE_R0_MERGE_ITEMS:
        if (value < 0 || value > 1 << 20) return fail(ctx, BPMAX_EINVAL, "merge cost out of range");
        ctx->r0_merge_items = (int)value;
        break;
    case BPMAX_TUNE_CLASS_STREAMS:
        ctx->class_streams = value != 0;
        break;
    case BPMAX_TUNE_WAIT_LIMIT_US:
        if (value < 1 || value > 600000000L) return fail(ctx, BPMAX_EINVAL, "wait limit out of range (1 us .. 600 s)");
        ctx->wait_ns = (unsigned long long)value * 1000ULL;
        if (ctx->plan.graph) {  // a kernel argument baked into the captured graph: recapture on next use
            cudaGraphExecDestroy(ctx->plan.graph);
            ctx->plan.graph = nullptr;
        }
        break;
    case BPMAX_TUNE_INJECT_WAIT_TIMEOUT:
        ctx->inject_wait_timeout = value != 0;
        break;
    case BPMAX_TUNE_WIDE_STAGES:
        if (value != 2 && value != 3) return fail(ctx, BPMAX_EINVAL, "tile-product stages must be 2 or 3");
        ctx->wide_stages = (int)value;
        break;
    case BPMAX_TUNE_R0_VARIANT:
        if (value != 0 && value != 1) return fail(ctx, BPMAX_EINVAL, "product shape variant must be 0 or 1");
        ctx->r0_variant = (int)value;
        break;
    case BPMAX_TUNE_CLASS_SHARE:
        ctx->class_share = value != 0;
        break;
    case BPMAX_TUNE_STRIP_TASKS:
        if (value < 0) return fail(ctx, BPMAX_EINVAL, "strip tasks must be >= 0");
        ctx->strip_tasks = std::min<long>(value, 1L << 40);
        break;
    case BPMAX_TUNE_PERSISTENT:
        if (value < 0 || value > 2) return fail(ctx, BPMAX_EINVAL, "persistent mode must be 0, 1 or 2");
        ctx->persist = (int)value;
        break;
    default: return fail(ctx, BPMAX_EINVAL, "unknown tuning key %d", key);
    }
    return BPMAX_OK;
}

int bpmax_gpu_get_tuning(const bpmax_ctx *ctx, int key, long *value)
{
    if (!ctx || !value) return BPMAX_EINVAL;
    switch (key) {
    case BPMAX_TUNE_R0_PAIRS_PER_JOB: *value = ctx->r0_pairs_per_job; break;
    case BPMAX_TUNE_R0_MERGE_ITEMS: *value = ctx->r0_merge_items; break;
    case BPMAX_TUNE_CLASS_STREAMS: *value = ctx->class_streams; break;
    case BPMAX_TUNE_WAIT_LIMIT_US: *value = (long)(ctx->wait_ns / 1000ULL); break;
    case BPMAX_TUNE_INJECT_WAIT_TIMEOUT: *value = ctx->inject_wait_timeout ? 1 : 0; break;
    case BPMAX_TUNE_WIDE_STAGES: *value = ctx->wide_stages; break;
    case BPMAX_TUNE_R0_VARIANT: *value = ctx->r0_variant; break;
    case BPMAX_TUNE_CLASS_SHARE: *value = ctx->class_share; break;
    case BPMAX_TUNE_STRIP_TASKS: *value = ctx->strip_tasks; break;
    case BPMAX_TUNE_PERSISTENT: *value = ctx->persist; break;
    default: return BPMAX_EINVAL;
    }
    return BPMAX_OK;
}

int bpmax_gpu_autotune(bpmax_ctx *ctx, int num_pairs, const int *const *seq1s, const long *Ms, const int *const *seq2s,
                       const long *Ns, int trials, long *best, float *best_ms)
{
    if (!ctx) return BPMAX_EINVAL;
    if (num_pairs < 1 || !Ms || !Ns) return fail(ctx, BPMAX_EINVAL, "empty batch");
    std::vector<int> vm(num_pairs), vn(num_pairs);
    for (int p = 0; p < num_pairs; ++p) {
        vm[p] = (int)Ms[p];
        vn[p] = (int)Ns[p];
    }
    const std::vector<int> key = shape_key(vm, vn);
    ctx->tuned.erase(key);
    const Tuned saved{ctx->r0_pairs_per_job, ctx->r0_merge_items, ctx->class_streams, ctx->r0_variant,
                      ctx->wide_stages,      ctx->class_share,    ctx->persist};
    std::set<int> classes;
    bool small = false, tiled = false;
    for (int n : vn) {
        const int np = padded_width(n);
        classes.insert(np);
        small = small || np <= MAX_SMALL_NP;
        tiled = tiled || is_tiled(np);
    }
    float best_t = -1.f;
    Tuned best_cfg = saved;
    int st = BPMAX_OK;
    auto try_cfg = [&](const Tuned &c) {
        ctx->r0_pairs_per_job = c[0];
        ctx->r0_merge_items = c[1];
        ctx->class_streams = c[2];
        ctx->r0_variant = c[3];
        ctx->wide_stages = c[4];
        ctx->class_share = c[5];
        ctx->persist = c[6];
        float t = -1.f;
        // the first run has no graph, the second captures it and is its first launch (37x23: 0.38 and 0.45 ms
        // against 0.35 of a replay)
        for (int r = 0; r < 2 + std::max(1, trials) && st == BPMAX_OK; ++r) {
            st = fill_pairs(ctx, num_pairs, seq1s, Ms, seq2s, Ns);
            if (st == BPMAX_OK && r > 1 && (t < 0 || ctx->last_ms < t)) t = ctx->last_ms;
        }
        if (st == BPMAX_OK && (best_t < 0 || t < best_t)) {
            best_t = t;
            best_cfg = c;
        }
    };
    // the schedule knobs with the default kernel shapes, then the kernel shapes with the best schedule
    const int jobs_cand[] = {8, 32, 1 << 20}, merge_cand[] = {1, 4}, streams_cand[] = {1, 0};
    for (int sc : streams_cand) {
        if (sc == 0 && classes.size() < 2) continue;  // one class: the stream setting changes nothing
        for (int jc : jobs_cand)
            for (int mc : merge_cand)
                if (st == BPMAX_OK) try_cfg(Tuned{jc, mc, sc, 0, 2, 0, 0});
    }
    if (classes.size() > 1 && best_cfg[2] == 1 && st == BPMAX_OK)
        try_cfg(Tuned{best_cfg[0], best_cfg[1], 1, 0, 2, 1, 0});
    const Tuned sched = best_cfg;
    if (small && st == BPMAX_OK) try_cfg(Tuned{sched[0], sched[1], sched[2], 1, sched[4], sched[5], 0});
    if (tiled && st == BPMAX_OK) try_cfg(Tuned{sched[0], sched[1], sched[2], best_cfg[3], 3, sched[5], 0});
    // the persistent fill, merge cost as found; several width classes one after another (side by side,
    // mode 1, they do not stay on their SM shares and measured 4.5x slower on the 512-pair batch)
    if (!tiled && st == BPMAX_OK)
        for (int jc : jobs_cand)
            if (st == BPMAX_OK) try_cfg(Tuned{jc, sched[1], sched[2], 0, sched[4], 0, classes.size() > 1 ? 2 : 1});
    ctx->r0_pairs_per_job = saved[0];
    ctx->r0_merge_items = saved[1];
    ctx->class_streams = saved[2];
    ctx->r0_variant = saved[3];
    ctx->wide_stages = saved[4];
    ctx->class_share = saved[5];
    ctx->persist = saved[6];
    if (st != BPMAX_OK) return st;
    ctx->tuned[key] = best_cfg;
    if (best)
        for (int k = 0; k < 7; ++k) best[k] = best_cfg[k];
    if (best_ms) *best_ms = best_t;
    return BPMAX_OK;
}

int bpmax_gpu_read_cells(bpmax_ctx *ctx, int pair, long i1_lo, long i1_hi, long j1_lo, long j1_hi, float *out)
{
    if (!ctx) return BPMAX_EINVAL;
    if (!ctx->plan_valid) return fail(ctx, BPMAX_EINVAL, "no fill has run on this context");
    const Plan &P = ctx->plan;
    if (pair < 0 || pair >= (int)P.pairs.size()) return fail(ctx, BPMAX_EINVAL, "pair %d out of range", pair);
    const PairDesc &pd = P.pairs[pair];
    if (!out || i1_lo < 0 || j1_lo < 0 || i1_lo >= i1_hi || j1_lo >= j1_hi || i1_hi > pd.M || j1_hi > pd.M)
        return fail(ctx, BPMAX_EINVAL, "outer cell window [%ld,%ld) x [%ld,%ld) outside 0..%d", i1_lo, i1_hi, j1_lo,
                    j1_hi, pd.M);
    CK(cudaSetDevice(ctx->device));
    const long long n_out = (long long)(i1_hi - i1_lo) * (j1_hi - j1_lo) * pd.N * pd.N;
    int st;
    if ((st = ensure(ctx, ctx->conv, n_out * sizeof(float))) != BPMAX_OK) return st;
    read_cells_kernel<<<4 * ctx->sms, 256, 0, ctx->stream>>>((const PairDesc *)ctx->pairs.p + pair, (const float *)ctx->F.p,
                                                             (int)i1_lo, (int)j1_lo, (int)(j1_hi - j1_lo), n_out,
                                                             (float *)ctx->conv.p);
    CK(cudaGetLastError());
    return copy_out(ctx, out, ctx->conv.p, n_out * sizeof(float));
}

int bpmax_gpu_last_timing(const bpmax_ctx *ctx, float *fill_ms, long *launches)
{
    if (!ctx) return BPMAX_EINVAL;
    if (fill_ms) *fill_ms = ctx->last_ms;
    if (launches) *launches = ctx->last_launches;
    return BPMAX_OK;
}

}  // extern "C"

// =========================================================================================
// Allocation-free score entry point (bpmax_gpu_score_noalloc).
//
// Some callers cannot allocate device memory: code that runs inside another framework's
// memory pool or under a fixed device-memory budget (where a raw cudaMalloc is forbidden or
// would exceed the budget), and latency-sensitive callers that must not risk the implicit
// device synchronisation cudaMalloc/cudaFree can cause. For them the fill's scratch (the F
// tables, S1/S2, the sequences and the job lists) lives in one fixed file-scope device array
// instead of the context's arenas. Every GPU that loads this library holds that array until
// the process exits.
// =========================================================================================
namespace {

constexpr size_t NOALLOC_FLOATS = (size_t)16 << 20;  // 64 MiB of fp32 scratch
constexpr unsigned long long NOALLOC_WAIT_NS = 4000000000ULL;  // time limit of one bounded wait

static __device__ __align__(256) float g_noalloc_scratch[NOALLOC_FLOATS];

struct NoallocDevice {
    float *ptr = nullptr;  // device address of g_noalloc_scratch on this device
    int sms = 0;
    int occ[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};  // resident product CTAs per SM, per width class
};
std::mutex g_noalloc_mu;
constexpr int NOALLOC_MAX_DEVICES = 64;
NoallocDevice g_noalloc_dev[NOALLOC_MAX_DEVICES];

// sequences (int32, seq1 then seq2) -> base codes (seq1, then seq2 reversed); cell job list
__global__ void noalloc_prep_kernel(const int *__restrict__ seqs, int M, int N, uint8_t *__restrict__ bases,
                                    CellJob *__restrict__ cells)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M + N; i += gridDim.x * blockDim.x) {
        bases[i] = (uint8_t)(i < M ? seqs[i] : seqs[M + (N - 1 - (i - M))]);
        if (i < M) cells[i] = CellJob{0, i};
    }
}

template <int NB>
int noalloc_set_attr(int *occ)
{
    const auto kernel = r0_kernel<NB, 0, R0Jobs>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R0Cfg<NB>::SMEM) != cudaSuccess)
        return BPMAX_ECUDA;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[NB], kernel, R0Cfg<NB>::THREADS, R0Cfg<NB>::SMEM) != cudaSuccess)
        return BPMAX_ECUDA;
    return cudaFuncSetAttribute(finalize_small_kernel<8 * NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)FinShape<8 * NB>::SMEM) == cudaSuccess ? BPMAX_OK : BPMAX_ECUDA;
}

// Once per device, with that device current: the device address of the scratch array (a host
// reference to g_noalloc_scratch is only a host-side stand-in) and the kernels' attributes.
int noalloc_setup(int dev, NoallocDevice *out)
{
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    NoallocDevice &nd = g_noalloc_dev[dev];
    if (!nd.ptr) {
        float *p = nullptr;
        if (cudaGetSymbolAddress((void **)&p, g_noalloc_scratch) != cudaSuccess || !p) {
            cudaGetLastError();
            return BPMAX_ECUDA;
        }
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return BPMAX_ECUDA;
        int st = noalloc_set_attr<1>(nd.occ);
        if (!st) st = noalloc_set_attr<2>(nd.occ);
        if (!st) st = noalloc_set_attr<3>(nd.occ);
        if (!st) st = noalloc_set_attr<4>(nd.occ);
        if (!st) st = noalloc_set_attr<5>(nd.occ);
        if (!st) st = noalloc_set_attr<6>(nd.occ);
        if (!st) st = noalloc_set_attr<7>(nd.occ);
        if (!st) st = noalloc_set_attr<8>(nd.occ);
        if (st) return st;
        nd.sms = sms;
        nd.ptr = p;
    }
    *out = nd;
    return BPMAX_OK;
}

template <int NB>
void noalloc_launch_diag(cudaStream_t s, const NoallocDevice &nd, int d, const R0Jobs &rj, int n_r0, int n_cells,
                         const CellJob *cj, const PairDesc *pd, float *F, float *S, const uint8_t *bases, const Weights &W,
                         int *err)
{
    if (d > 0)
        launch_chain(true, std::min(n_r0, std::max(1, nd.occ[NB]) * nd.sms), R0Cfg<NB>::THREADS, R0Cfg<NB>::SMEM, s,
                     r0_kernel<NB, 0, R0Jobs>, rj, n_r0, pd, F, d, WaitCtl{err, NOALLOC_WAIT_NS, 0});
    const int n_s1 = n_cells - 1;  // S1 cells of diagonal d+1: the first n_cells-1 entries of cj
    using Sh = FinShape<8 * NB>;
    launch_chain(Sh::THREADS < 512, n_cells + (n_s1 + Sh::WARPS - 1) / Sh::WARPS, Sh::THREADS, Sh::SMEM, s,
                 finalize_small_kernel<8 * NB>, cj, n_cells, cj, n_s1, pd, F, S, bases, W, d, RefOut{nullptr, 0, 0});
}

}  // namespace

extern "C" int bpmax_gpu_score_noalloc(const int *seq1, long M, const int *seq2, long N, const float *weights12,
                                       float *score, void *stream)
{
    if (!seq1 || !seq2 || !weights12 || !score || M < 1 || N < 1 || M > 65535 || N > MAX_SMALL_NP)
        return BPMAX_EINVAL;
    for (long i = 0; i < M; ++i)
        if (seq1[i] < 0 || seq1[i] > 4) return BPMAX_EINVAL;
    for (long i = 0; i < N; ++i)
        if (seq2[i] < 0 || seq2[i] > 4) return BPMAX_EINVAL;
    if (!weights_ok(weights12)) return BPMAX_EINVAL;
    // an error left pending by the caller's own earlier work is not this call's to report or clear
    if (cudaPeekAtLastError() != cudaSuccess) return BPMAX_ECUDA;
    const int Np = std::max(8, (int)(N + 7) / 8 * 8);
    const int nb = Np / 8;
    // scratch layout (floats), every region 256-byte aligned
    const long long nF = (long long)M * (M + 1) / 2 * cell_floats(Np);
    const long long off_S = align64(nF);
    const long long S2_rel = align64((long long)M * M);
    // (S2 and as much again twice: the documented size limits count it)
    const long long off_seq = off_S + S2_rel + 3 * align64((long long)Np * Np);
    const long long off_bases = off_seq + align64(M + N);
    const long long off_pd = off_bases + align64((M + N + 3) / 4);
    const long long off_score = off_pd + align64((long long)(sizeof(PairDesc) + 3) / 4);  // score, error flag
    const long long off_cj = off_score + 64;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
        cudaGetLastError();
        return BPMAX_ENODEV;
    }
    NoallocDevice nd;
    int st = noalloc_setup(dev, &nd);
    if (st) return st;
    const long long resident = (long long)std::max(1, nd.occ[nb]) * nd.sms;
    const int qmin = std::max(1, (R0_TAB_ITEMS[nb] + 1) / 2);
    // (room for the longest job list of a diagonal, M * ceil(P2 / qmin): the documented size limits count
    // it, the jobs themselves are computed in the kernel)
    const long long off_rj = off_cj + align64(2LL * M);
    const long long max_jobs = (long long)M * (((M + 1) / 2 + qmin - 1) / qmin);
    const long long total = off_rj + 4LL * max_jobs;
    if ((size_t)total > NOALLOC_FLOATS) return BPMAX_EINVAL;  // pair too large for the fixed scratch

    cudaStream_t s = (cudaStream_t)stream;
    float *base = nd.ptr;
    float *F = base, *S = base + off_S;
    int *seqs = reinterpret_cast<int *>(base + off_seq);
    uint8_t *bases = reinterpret_cast<uint8_t *>(base + off_bases);
    PairDesc *pdp = reinterpret_cast<PairDesc *>(base + off_pd);
    float *dscore = base + off_score;
    int *derr = reinterpret_cast<int *>(base + off_score + 1);
    CellJob *cj = reinterpret_cast<CellJob *>(base + off_cj);
    PairDesc pd{};
    pd.M = (int)M;
    pd.N = (int)N;
    pd.Np = Np;
    pd.F_off = 0;
    pd.S1_off = 0;
    pd.S2_off = S2_rel;
    pd.seq1_off = 0;
    pd.seq2_off = (int)M;
    Weights W;
    memcpy(W.w, weights12, sizeof W.w);

    auto ok = [](cudaError_t e) { return e == cudaSuccess; };
    // pageable host sources: the copies are staged before cudaMemcpyAsync returns
    if (!ok(cudaMemcpyAsync(seqs, seq1, sizeof(int) * M, cudaMemcpyHostToDevice, s)) ||
        !ok(cudaMemcpyAsync(seqs + M, seq2, sizeof(int) * N, cudaMemcpyHostToDevice, s)) ||
        !ok(cudaMemcpyAsync(pdp, &pd, sizeof pd, cudaMemcpyHostToDevice, s)) ||
        !ok(cudaMemsetAsync(F, 0, sizeof(float) * nF, s)) ||        // F starts at +0 on every call
        !ok(cudaMemsetAsync(S, 0, sizeof(float) * S2_rel, s)) ||    // and S1 at 0
        !ok(cudaMemsetAsync(derr, 0, sizeof(int), s))) {
        cudaGetLastError();
        return BPMAX_ECUDA;
    }
    noalloc_prep_kernel<<<8, 256, 0, s>>>(seqs, (int)M, (int)N, bases, cj);
    single_strand_kernel<<<1, 512, 0, s>>>(pdp, bases, S, W);
    for (int d = 0; d < (int)M; ++d) {
        const int cells = (int)M - d;
        int n_r0 = 0;
        R0Jobs rj{cells, 1, (d + 1) / 2};
        if (d > 0) {
            rj.q = (int)r0_pairs_per_job(cells, rj.pairs, resident, qmin, 1 << 20, 2);
            n_r0 = cells * ((rj.pairs + rj.q - 1) / rj.q);
        }
        switch (nb) {
        case 1: noalloc_launch_diag<1>(s, nd, d, rj, n_r0, cells, cj, pdp, F, S, bases, W, derr); break;
        case 2: noalloc_launch_diag<2>(s, nd, d, rj, n_r0, cells, cj, pdp, F, S, bases, W, derr); break;
        case 3: noalloc_launch_diag<3>(s, nd, d, rj, n_r0, cells, cj, pdp, F, S, bases, W, derr); break;
        case 4: noalloc_launch_diag<4>(s, nd, d, rj, n_r0, cells, cj, pdp, F, S, bases, W, derr); break;
        case 5: noalloc_launch_diag<5>(s, nd, d, rj, n_r0, cells, cj, pdp, F, S, bases, W, derr); break;
        case 6: noalloc_launch_diag<6>(s, nd, d, rj, n_r0, cells, cj, pdp, F, S, bases, W, derr); break;
        case 7: noalloc_launch_diag<7>(s, nd, d, rj, n_r0, cells, cj, pdp, F, S, bases, W, derr); break;
        default: noalloc_launch_diag<8>(s, nd, d, rj, n_r0, cells, cj, pdp, F, S, bases, W, derr); break;
        }
    }
    gather_scores_kernel<<<1, 32, 0, s>>>(pdp, F, 1, dscore);
    float out[2] = {0.f, 0.f};  // score, error flag bits
    if (!ok(cudaGetLastError()) || !ok(cudaMemcpyAsync(out, dscore, 2 * sizeof(float), cudaMemcpyDeviceToHost, s)) ||
        !ok(cudaStreamSynchronize(s))) {
        cudaGetLastError();
        return BPMAX_ECUDA;
    }
    int errbits = 0;
    memcpy(&errbits, &out[1], sizeof errbits);
    if (errbits != 0) return BPMAX_ETIMEOUT;
    *score = out[0];
    return BPMAX_OK;
}
