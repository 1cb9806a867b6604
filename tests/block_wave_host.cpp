// block_wave of bpmax_kernels.cuh compiled for the host (its source text is in BLOCK_WAVE_SOURCE): one
// fiber per CUDA thread, every barrier and shuffle a rendezvous of the CTA's or the warp's fibers.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <ucontext.h>
#include <vector>

using std::max;
using std::min;
#define __device__
#define __forceinline__ inline
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
static float2 make_float2(float x, float y) { return {x, y}; }
static const float NEG_INF = -INFINITY;
static float fmax3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }

struct Rendezvous { int size = 0, count = 0, round = 0; };
static ucontext_t g_main;
static std::vector<ucontext_t> g_fiber;
static int g_self;
static std::vector<Rendezvous> g_warp;
static Rendezvous g_cta;
static std::vector<float> g_slot;
static struct { struct Index { operator int() const { return g_self; } } x; } threadIdx;

static void meet(Rendezvous &r)
{
    const int round = r.round;
    if (++r.count == r.size) {
        r.count = 0;
        ++r.round;
    }
    while (r.round == round) swapcontext(&g_fiber[g_self], &g_main);
}
static void __syncthreads() { meet(g_cta); }
static float shuffle(float v, int from)
{
    Rendezvous &w = g_warp[g_self >> 5];
    g_slot[g_self] = v;
    meet(w);
    const float r = g_slot[(g_self & ~31) + from];
    meet(w);
    return r;
}
static float __shfl_xor_sync(unsigned, float v, int m) { return shuffle(v, (g_self & 31) ^ m); }
static float __shfl_down_sync(unsigned, float v, int d, int width)
{
    const int lane = g_self & 31;
    return shuffle(v, (lane & (width - 1)) + d < width ? lane + d : lane);
}

#include BLOCK_WAVE_SOURCE

static struct { float *T; const float *SX, *SJ, *wt; const uint8_t *rb; int ld, warps, nb, ncol, e0; bool tri; } g_arg;
static int g_left;
static void run()
{
    const auto &a = g_arg;
    auto go = [&](auto f) { f(a.T, a.SX, a.SJ, a.wt, a.rb, a.tri, a.nb, a.ncol, a.e0); };
#define CASE(LD, WARPS) if (a.ld == LD && a.warps == WARPS) go(block_wave<LD, WARPS>)
    CASE(12, 1); CASE(20, 1); CASE(28, 4); CASE(36, 4); CASE(44, 4); CASE(52, 4); CASE(60, 4); CASE(68, 4); CASE(68, 8); CASE(68, 16);
    --g_left;
    while (true) swapcontext(&g_fiber[g_self], &g_main);
}

extern "C" void host_block_wave(float *T, const float *SX, const float *SJ, const float *wt, const uint8_t *rb, int ld,
                                int warps, int tri, int nb, int ncol, int e0)
{
    const int threads = 32 * warps;
    static std::vector<std::vector<char>> stacks;
    stacks.assign(threads, std::vector<char>(64 << 10));
    g_arg = {T, SX, SJ, wt, rb, ld, warps, nb, ncol, e0, tri != 0};
    g_warp.assign(warps, Rendezvous{32, 0, 0});
    g_cta = Rendezvous{threads, 0, 0};
    g_slot.assign(threads, 0.0f);
    g_fiber.assign(threads, ucontext_t{});
    g_left = threads;
    for (int t = 0; t < threads; ++t) {
        getcontext(&g_fiber[t]);
        g_fiber[t].uc_stack.ss_sp = stacks[t].data();
        g_fiber[t].uc_stack.ss_size = stacks[t].size();
        makecontext(&g_fiber[t], run, 0);
    }
    while (g_left > 0)
        for (int t = 0; t < threads && g_left > 0; ++t) {
            g_self = t;
            swapcontext(&g_main, &g_fiber[t]);
        }
}
