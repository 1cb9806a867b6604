// bpmax_kernels.cuh -- sm_100a kernels of the BPMax fill.
//
// Recurrence (reference spec V3cs/bpmax_verify.ab:16-71, executed by
// V3/bpmax_verify.c:533-721; V3 = TPDS/source/release/MPT_RT_V3/bpmax_complete_otf_ftable/src):
//   F(i1,j1,i2,j2) = inter(s1[i1],s2r[i2])                            if i1==j1 && i2==j2
//                  = max( SW1, SW2, S1(i1,j1)+S2(i2,j2), R0, R1, R2, R3, R4 ) otherwise,
// each candidate one fp32 add of two stored values (or a literal 0 where undefined).
// With weights >= +0 every value is >= +0, so (a) max is exact and order-free, (b) integer
// max on the float bit patterns equals the float max, which lets partial maxima from many
// CTAs merge with atomicMax on int, and (c) masked cells can hold -inf (never a winner).
//
// Device layout of one sequence pair (a "pair" below):
//   outer cell (i1,j1), i1<=j1<M, index c = i1*M - i1*(i1-1)/2 + (j1-i1) (row-major triangle)
//   F: one inner table per outer cell, i2 over the reversed strand 2, Np = N rounded up:
//     Np <= 64 (Np = 8*NB): a "cell image" of 16-byte chunks -- block columns BJ = 0..NB-1 in
//       turn, column BJ holding the 8x8 blocks (0..BJ, BJ) of the upper block triangle at a pitch
//       of 17 chunks (row r of a block = chunks 2r, 2r+1; the 17th chunk is spare), then the
//       column's 2-chunk S1 piece (-inf x7, S1 of the cell), then R0_TAB_COLPAD[NB][BJ] spare
//       chunks (the pads spread the product kernel's shared loads over the bank groups). Inside
//       diagonal blocks the entries below the diagonal are -inf except the subdiagonal, which
//       holds S1 of the cell; padding rows/columns (>= N) are -inf.
//     Np > 64 (a multiple of 64): tile images (below).
//   S1[M][M], S2[Np][Np] single-strand tables (S2 over the reversed strand 2)
#pragma once
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

namespace bpmax {

constexpr float NEG_INF = -__builtin_inff();

#include "r0_tables.inc"

// chunk offset of block column c of a cell image of width class nb (c = nb: the image size)
#ifdef __CUDA_ARCH__
#define IMG_COLBASE(nb, c) c_img_colbase[nb][c]
#else
#define IMG_COLBASE(nb, c) R0_TAB_COLBASE[nb][c]
#endif

struct Weights {
    float w[12];  // intra AU,UA,GC,CG,GU,UG ; inter AU,UA,GC,CG,GU,UG
};

struct PairDesc {
    int M, N, Np;
    int cnt_off;       // persistent fill: offset of the pair's per-diagonal counters (M ints)
    long long F_off;   // float offset of F[0]
    long long S1_off;  // float offset of S1 in the S arena
    long long S2_off;  // float offset of S2 in the S arena
    long long S2x_off; // Np > 64 only: dense tile images of S2 (bpmax_tile.cuh)
    int seq1_off;      // offset of seq1 in the base arena (uint8)
    int seq2_off;      // offset of the REVERSED seq2 in the base arena (uint8)
    long long cell_base;  // persistent fill: index of the pair's cell (0, 0) among all pairs' cells
};

// pair type of ordered bases (a,b): AU=0 UA=1 GC=2 CG=3 GU=4 UG=5, else -1
// (V3/external_functions.c:21-39, split by order for the 12-entry table)
__host__ __device__ __forceinline__ int pair_type(int a, int b)
{
    if ((a | b) & ~3) return -1;
    // nibble (a*4+b) -> type, F = none: idx3 -> 0 (AU), idx6 -> 3 (CG), idx9 -> 2 (GC),
    // idx11 -> 4 (GU), idx12 -> 1 (UA), idx14 -> 5 (UG)
    const uint64_t tab = 0xF5F14F2FF3FF0FFFull;
    int v = (int)((tab >> (4 * (a * 4 + b))) & 0xF);
    return v == 0xF ? -1 : v;
}

__host__ __device__ __forceinline__ float score_w(const float *w6, int a, int b)
{
    int t = pair_type(a, b);
    return t < 0 ? 0.0f : w6[t];
}

__host__ __device__ __forceinline__ long long cell_index(int M, int i1, int j1)
{
    return (long long)i1 * M - (long long)i1 * (i1 - 1) / 2 + (j1 - i1);
}

// Launches of one chain follow each other by programmatic dependent launch: a kernel's CTAs may start
// while the launch before it still runs, read what no kernel of the fill writes (job lists, pair
// records, sequences, weights), and wait here until that launch is complete and its writes are visible.
// Every thread of every kernel of a chain calls this before it touches S1, S2 or F, and only then lets
// the next launch start, so whatever starts early has only the launch before it still running.
__device__ __forceinline__ void chain_wait()
{
    asm volatile("griddepcontrol.wait;\n griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ float fmax3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }

// ------------------------------------------------------------------------------------------
// Tile images: inner tables of width Np = 64 * NT > 64 are stored per outer cell as the upper triangle of
// NT x NT tiles of 64 x 64 in row-major tile-triangle order. A diagonal tile is a width-64 cell image (above); an off-diagonal ("dense") tile holds all 64 of
// its 8x8 blocks in block columns at WIDE_DENSE_COLBASE (wide_tables.inc), each column closed by a
// halo piece: row 0 of block (0, bj) of the tile below, the row after the tile, so the row-shifted
// operand of any tile is one image. Rows and columns >= N are -inf.
// ------------------------------------------------------------------------------------------
#include "wide_tables.inc"

constexpr int S2_ONE_CTA_NP = 320;                        // widest S2 filled by single_strand_kernel
constexpr int WIDE_DIAG_CHUNKS = R0_TAB_COLBASE[8][8];    // diagonal tile image (width-64 cell image)
constexpr int WIDE_DENSE_CHUNKS = WIDE_DENSE_COLBASE[8];  // dense tile image

__host__ __device__ __forceinline__ bool is_tiled(int Np) { return Np > 64; }

// float offset of tile (I, J), I <= J, inside a cell's table of NT x NT tiles
__host__ __device__ __forceinline__ long long wide_tile_off(int NT, int I, int J)
{
    const long long SD = 4LL * WIDE_DIAG_CHUNKS, SQ = 4LL * WIDE_DENSE_CHUNKS;
    long long o = (long long)I * SD + SQ * ((long long)I * (NT - 1) - (long long)I * (I - 1) / 2);
    if (J > I) o += SD + (long long)(J - I - 1) * SQ;
    return o;
}
__host__ __device__ __forceinline__ long long wide_cell_floats(int NT)
{
    return (long long)NT * 4 * WIDE_DIAG_CHUNKS + (long long)NT * (NT - 1) / 2 * 4 * WIDE_DENSE_CHUNKS;
}

#ifdef __CUDA_ARCH__
#define WIDE_DENSE_CB(c) c_wide_dense_colbase[c]
#else
#define WIDE_DENSE_CB(c) WIDE_DENSE_COLBASE[c]
#endif

// float offset, inside a cell's table of NT x NT tiles, of the stored entry (r, c) with r <= c
__host__ __device__ __forceinline__ long long wide_pos(int NT, int r, int c)
{
    const int I = r >> 6, J = c >> 6, lr = r & 63, lc = c & 63, bi = lr >> 3, bj = lc >> 3;
    const int cb = I == J ? IMG_COLBASE(8, bj) : WIDE_DENSE_CB(bj);
    return wide_tile_off(NT, I, J) + 4 * (cb + 17 * bi) + 8 * (lr & 7) + (lc & 7);
}

// floats per stored cell table of a pair
__host__ __device__ __forceinline__ long long cell_floats(int Np)
{
    if (Np <= 64) return 4LL * IMG_COLBASE(Np >> 3, Np >> 3);
    return wide_cell_floats(Np >> 6);
}

// F(cell)[r][c] for any r, c < Np (entries below the diagonal as the tables define them)
__device__ __forceinline__ float f_value(const PairDesc &pd, const float *__restrict__ F, long long cell, int r, int c)
{
    const float *C = F + pd.F_off + cell * cell_floats(pd.Np);
    if (pd.Np > 64) {
        if (r > c) return r == c + 1 ? C[4 * 17 + 7] : NEG_INF;  // S1 piece of column 0 of tile (0, 0)
        return C[wide_pos(pd.Np >> 6, r, c)];
    }
    const int NB = pd.Np >> 3, BI = r >> 3, BJ = c >> 3;
    if (BI > BJ) return r == c + 1 ? C[4 * 17 + 7] : NEG_INF;  // S1 piece of column 0
    return C[4 * (c_img_colbase[NB][BJ] + 17 * BI) + 8 * (r & 7) + (c & 7)];
}

// ------------------------------------------------------------------------------------------
// Single-strand table S2 over the reversed strand 2 (V3/bpmax_verify.c:560-571):
// S(i,j) = 0 if j-i<=3, else max(S(i+1,j-1)+intra(s[i],s[j]), max_{i<=k<j} S(i,k)+S(k+1,j)).
// One CTA per pair; wavefront over the diagonal j-i. Cells outside the N x N upper triangle are
// left at 0 and never read. (S1 is built diagonal by diagonal inside the finalizes.) Pairs
// wider than S2_ONE_CTA_NP are left to s2_diag_kernel, one launch per diagonal.
// ------------------------------------------------------------------------------------------
__global__ void single_strand_kernel(const PairDesc *__restrict__ pairs, const uint8_t *__restrict__ bases,
                                     float *__restrict__ S, Weights W)
{
    const PairDesc pd = pairs[blockIdx.x];
    if (pd.Np > S2_ONE_CTA_NP) return;  // one launch per diagonal (s2_diag_kernel)
    const int L = pd.N, ld = pd.Np;
    const uint8_t *s = bases + pd.seq2_off;
    float *T = S + pd.S2_off;
    for (int idx = threadIdx.x; idx < ld * ld; idx += blockDim.x) T[idx] = 0.0f;
    __syncthreads();
    for (int d = 4; d < L; ++d) {
        const int cells = L - d;
        // groups of g threads per cell, g a power of two <= 32
        int g = 1;
        while (g < 32 && g * 2 * cells <= (int)blockDim.x) g *= 2;
        const int lane_g = threadIdx.x & (g - 1);
        const int slots = blockDim.x / g;
        for (int base = 0; base < cells; base += slots) {
            const int i = base + threadIdx.x / g;
            float red = NEG_INF;
            const bool act = i < cells;
            const int j = i + d;
            if (act)
                for (int k = i + lane_g; k < j; k += g) red = fmaxf(red, T[i * ld + k] + T[(k + 1) * ld + j]);
            for (int o = g >> 1; o > 0; o >>= 1) red = fmaxf(red, __shfl_xor_sync(0xffffffffu, red, o, g));
            if (act && lane_g == 0) {
                const float pr = T[(i + 1) * ld + (j - 1)] + score_w(W.w, s[i], s[j]);
                T[i * ld + j] = fmaxf(pr, red);
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// Finalize the outer cells of diagonal d (Np <= 64, cell images; one CTA per cell):
// adds the candidates that do not come from R0/R3/R4 and runs the inner wavefront of R1/R2/SW2.
//   base  i1==j1 && i2==j2: inter(s1[i1], s2r[i2])            (assignment, eval_FTable :576)
//   S1(i1,j1)+S2(i2,j2)
//   SW2 = F(i1,j1,i2+1,j2-1)+intra(s2r[i2],s2r[j2]) if j2-i2>=4
//   R1 (:614-640) max_{k2} F(i1,j1,i2,k2)+S2(k2+1,j2); R2 (:641-667) max_{k2} S2(i2,k2)+F(i1,j1,k2+1,j2)
//   SW1 = F(i1+1,j1-1,.)+intra(s1[i1],s1[j1]) if j1-i1>=4     (V3/bpmax_outer_south_west.c:115-160)
// F arrives holding max(R0,R3,R4) (or +0), merged there by products of any earlier launch since the
// table was cleared: SW1 is read here from the table of (i1+1, j1-1), so nothing but products
// writes a table before its own finalize, and those of diagonal d may run before the finalize of
// d-1 and d-2. Every literal-0 candidate is covered because every value is >= +0. Writes the cell's
// blocks (-inf outside the logical triangle, S1(i1,j1) on the subdiagonal) and its S1 pieces.
// The inner wavefront goes by 8x8 blocks of the table in shared memory (block_wave).
// Bound: latency of the wavefront where a launch has few cells (at width 64, 8 block diagonals of
// 600-1,230 cycles of products and 930 of the blocks' own wavefronts), instructions where it has many.
// Before, batches of five inner diagonals, the next batch's in the registers of one warp while the
// others pushed the last one's candidates to all later entries: 19,400 cycles at width 64. Fill ms
// by batches / by blocks: 64x64 1.52 / 1.39, 128x32 1.98 / 1.82, 128x64 4.26 / 4.09, 1024x64 614 / 601,
// the 512-pair batch 424 / 418. Tried: the blocks' start values loaded ahead of their wavefronts, 1,150
// cycles; their S2 values picked from registers per column, 3,240 (divergent branches).
// CTAs after the first njobs compute S1 on diagonal d+1 (V3/bpmax_verify.c:533-544), one warp
// per cell, from S1 diagonals <= d (S1 is cleared to 0 before the fill; j-i <= 3 stays 0).
// ------------------------------------------------------------------------------------------
struct CellJob {
    int pair, i1;
};

// threads per cell. Up to one cell per SM what counts is the latency of one cell: many threads for its
// loads and products. Launches of more cells run several CTAs per SM, which hide each other's latency,
// and four warps per cell then idle least at the barriers; in between, up to three cells per SM, eight
// warps for widths >= 48 (256x64 15.8 -> 15.6, 200x56 7.80 -> 7.64, 512x64 86.9 -> 86.0). Fill ms with the
// latency threads for up to 1,024 / 296 / 148 cells: 1024x64 622 / 602 / 601, 256x64 16.2 / 16.2 / 15.8;
// the 512-pair batch at 256 / 160 / 128 threads beyond: 428 / 419 / 418. Up to 148 cells 128x64 takes 4.44 with 256 threads
// and 4.09 with 512, 64x32 0.83 with 128, 0.73 with 256 and 0.71 with 384. The one to three blocks of widths 8
// and 16 are work for one warp: 32 threads, 32 CTAs per SM, from three cells per SM on (10,000 pairs 3x6 at 128 / 64 /
// 32 threads 0.499 / 0.435 / 0.400, 1,000 pairs 16x16 2.49 / 2.34 / 2.24; up to three cells per SM 5 pairs 60x16
// 0.616 / 0.624 / 0.657). Width 24 keeps 128 throughout: one warp gains 9% there at 1,000 pairs of 16 and loses 5% at 4
// of 300.
constexpr int fin_threads(int NP) { return NP >= 48 ? 512 : (NP >= 32 ? 384 : 128); }
constexpr int fin_bulk_threads(int NP) { return NP <= 16 ? 32 : 128; }
constexpr int FIN_MID_THREADS = 256;
// bulk launches: more cells per SM than this
constexpr int fin_bulk_per_sm(int NP) { return NP >= 48 || NP <= 16 ? 3 : 1; }
constexpr bool fin_has_mid(int NP) { return NP >= 48; }
// element (r, c) of tile (I2, J2) of an outer cell in the reference layout (tiles of T+1 rows, the
// last one the halo; R = padding rows/columns of the first tile row/column); val(i2, j2) gives the
// cell's inner value for 0 <= i2 <= j2 < N, the only entries read
template <class Val>
__device__ __forceinline__ float reference_tile_elem_v(const Val &val, int T, int R, int I2, int J2, int r, int c)
{
    const int Ri = I2 == 0 ? R : 0, Rj = (I2 == 0 && J2 == 0) ? R : 0;
    float v = __int_as_float(0x7fc00000);  // NaN: a cell the reference leaves unwritten
    if (I2 <= J2 && c >= Rj) {
        if (r < T) {
            if (r >= Ri) {
                const int i2 = I2 * T + r - R, j2 = J2 * T + c - R;
                v = i2 <= j2 ? val(i2, j2) : -3.402823466e+38f;
            }
        } else {
            v = I2 == J2 ? -3.402823466e+38f : val((I2 + 1) * T - R, J2 * T + c - R);
        }
    }
    return v;
}
__device__ __forceinline__ float reference_tile_elem(const PairDesc &pd, const float *__restrict__ F, long long cell,
                                                     int T, int R, int I2, int J2, int r, int c)
{
    return reference_tile_elem_v([&](int i2, int j2) { return f_value(pd, F, cell, i2, j2); }, T, R, I2, J2, r, c);
}

// element `rem` (in [0, Ns*Ns*(T+1)*T)) of outer cell (i1, j1) in the reference layout
__device__ __forceinline__ float reference_elem(const PairDesc &pd, const float *__restrict__ F, int T, int Ns, int R,
                                                int i1, int j1, long long rem)
{
    const long long tile_f = (long long)(T + 1) * T;
    const int I2 = (int)(rem / ((long long)Ns * tile_f));
    rem %= (long long)Ns * tile_f;
    const int J2 = (int)(rem / tile_f);
    rem %= tile_f;
    return reference_tile_elem(pd, F, cell_index(pd.M, i1, j1), T, R, I2, J2, (int)(rem / T), (int)(rem % T));
}

// Reference-layout copy of the cells a finalize launch completes (the copy-out of bpmax_gpu_fill):
// out == nullptr for none; else cell (i1, i1+d) of the (single) pair goes to
// out + (d*M - d(d-1)/2 + i1) * cell_f, diagonal after diagonal, in the reference's tile layout of
// N_tile = T (Ns tiles a side; see reference_elem)
struct RefOut {
    float *out;
    int T, Ns;
};

template <int NP, int T = fin_threads(NP)>
struct FinShape {
    static constexpr int THREADS = T;
    static constexpr int WARPS = THREADS / 32;
    static constexpr int LD = NP + 4;  // row pitch of the tables: an odd number of 16-byte chunks
    // table (4 words before it, one row after it), two copies of S2, bases
    static constexpr size_t SMEM = ((size_t)4 + (3 * NP + 1) * LD) * sizeof(float) + NP;
    // at most 80 registers (512 threads: 128, one CTA per SM; 32 threads: 64, every CTA slot of an SM)
    static constexpr int MINB = THREADS == 32 ? 32 : 768 / THREADS;
};

// (BI, BJ) of the q-th block of the upper block triangle (row-major triangle order)
__device__ __forceinline__ void blk_decode(int NB, int q, int &BI, int &BJ)
{
    BI = 0;
    while (q >= NB - BI) { q -= NB - BI; ++BI; }
    BJ = BI + q;
}

// ------------------------------------------------------------------------------------------
// The inner wavefront of R1, R2 and SW2 inside a table (tri: an upper triangle of nb block rows) or a
// 64x64 tile, by 8x8 blocks, block diagonal by block diagonal; all threads of the CTA. T[r][c] holds the
// start values (-inf below the diagonal, in columns >= ncol, in column -1 and in the row after the
// last) and receives the final ones; SJ[x][y] = S2(x, y) of the columns' strand piece, SX[x][y] = S2(x, y-1)
// of the rows'; wt[LD*b + c] = the SW2 weight of row base b and column c; SJ and wt are -inf in columns >= ncol,
// which keeps T -inf there; rb = the rows' bases; entry (r, c) spans j2-i2 = e0 + c - r.
//   1. one warp per block adds the terms over the finished blocks of its row and column,
//        R1  T[r][k] + S2(k+1, c),  R2  S2(r, k-1) + T[k][c],
//      as products, four lanes sharing the k of a 2x4 piece, and SW2 from outside the block;
//   2. one warp per four blocks runs the blocks' own wavefronts over their 15 diagonals in registers, a row
//      per lane. S2 is 0 on spans <= 3, so inside a block an entry needs its two neighbours of the
//      previous diagonal (never less than the candidates of two to four diagonals back, each of which is a
//      candidate of theirs plus 0), SW2, and what lies five to seven columns left or rows below.
// The candidates of neighbours outside the block are in the products.
// ------------------------------------------------------------------------------------------
template <int LD, int WARPS>
__device__ __forceinline__ void block_wave(float *T, const float *SX, const float *SJ, const float *wt, const uint8_t *rb,
                                           bool tri, int nb, int ncol, int e0)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nbc = (ncol + 7) >> 3;
    const int kp = lane & 3, st = lane >> 2, la = lane & 7;
    for (int D = tri ? 0 : 1 - nb; D < nbc; ++D) {
        const int first = max(0, -D), count = min(nb - first, nbc - max(0, D));  // blocks (first + m, first + m + D)
        __syncthreads();  // the blocks of earlier block diagonals are final
        if (!tri || D > 0) {
            for (int m = warp; m < count; m += WARPS) {
                const int bi = first + m, bj = bi + D;
                // rows r0, r0+1, columns c0 .. c0+3, k = 2kp, 2kp+1 of every k block; in the end row r,
                // columns c, c+1, whose words from outside the block are loaded first
                const int r0 = 8 * bi + 2 * (st >> 1), c0 = 8 * bj + 4 * (st & 1);
                const int r = r0 + (kp & 1), c = c0 + (kp & 2);
                float2 *o = reinterpret_cast<float2 *>(T + r * LD + c);
                const float2 x = *o, wr = *reinterpret_cast<const float2 *>(wt + LD * rb[r] + c);
                const float q0 = T[(r + 1) * LD + c - 1], q1 = T[(r + 1) * LD + c];
                float v[2][4];
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[i][j] = NEG_INF;
                auto step = [&](const float *A, const float *B) {  // A: row r0, k = 2kp; B: row 2kp, column c0
                    const float2 x0 = *reinterpret_cast<const float2 *>(A), x1 = *reinterpret_cast<const float2 *>(A + LD);
                    const float4 y0 = *reinterpret_cast<const float4 *>(B), y1 = *reinterpret_cast<const float4 *>(B + LD);
                    v[0][0] = fmax3(v[0][0], x0.x + y0.x, x0.y + y1.x);
                    v[0][1] = fmax3(v[0][1], x0.x + y0.y, x0.y + y1.y);
                    v[0][2] = fmax3(v[0][2], x0.x + y0.z, x0.y + y1.z);
                    v[0][3] = fmax3(v[0][3], x0.x + y0.w, x0.y + y1.w);
                    v[1][0] = fmax3(v[1][0], x1.x + y0.x, x1.y + y1.x);
                    v[1][1] = fmax3(v[1][1], x1.x + y0.y, x1.y + y1.y);
                    v[1][2] = fmax3(v[1][2], x1.x + y0.z, x1.y + y1.z);
                    v[1][3] = fmax3(v[1][3], x1.x + y0.w, x1.y + y1.w);
                };
                const float *A1 = T + r0 * LD + 2 * kp, *B1 = SJ + (2 * kp + 1) * LD + c0;  // R1: k blocks k1 .. bj-1
                const float *A2 = SX + r0 * LD + 2 * kp, *B2 = T + 2 * kp * LD + c0;        // R2: k blocks bi+1 .. k2
                const int k1 = tri ? bi : 0, n1 = bj - k1, n2 = (tri ? bj : nb - 1) - bi;
                int t = 0;
                for (; t < min(n1, n2); ++t) {
                    step(A1 + 8 * (k1 + t), B1 + 8 * LD * (k1 + t));
                    step(A2 + 8 * (bi + 1 + t), B2 + 8 * LD * (bi + 1 + t));
                }
                for (int u = t; u < n1; ++u) step(A1 + 8 * (k1 + u), B1 + 8 * LD * (k1 + u));
                for (int u = t; u < n2; ++u) step(A2 + 8 * (bi + 1 + u), B2 + 8 * LD * (bi + 1 + u));
                float h[4], g[2];  // lane kp keeps row kp & 1, then columns kp & 2 and the next
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float keep = kp & 1 ? v[1][j] : v[0][j], give = kp & 1 ? v[0][j] : v[1][j];
                    h[j] = fmaxf(keep, __shfl_xor_sync(0xffffffffu, give, 1));
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float keep = kp & 2 ? h[j + 2] : h[j], give = kp & 2 ? h[j] : h[j + 2];
                    g[j] = fmaxf(keep, __shfl_xor_sync(0xffffffffu, give, 2));
                }
                const bool last = (r & 7) == 7;  // SW2 of the block's last row and first column
                const float w0 = (last || (c & 7) == 0) && e0 + c - r >= 4 ? q0 + wr.x : NEG_INF;
                const float w1 = last && e0 + c + 1 - r >= 4 ? q1 + wr.y : NEG_INF;
                *o = make_float2(fmax3(x.x, g[0], w0), fmax3(x.y, g[1], w1));
            }
            __syncthreads();
        }
        for (int w = warp; 4 * w < count; w += WARPS) {
            const int m = 4 * w + (lane >> 3), bi = first + min(m, count - 1), bj = bi + D;
            const int row = 8 * bi + la, cols = m < count ? min(8, ncol - 8 * bj) : 0, e1 = e0 + 8 * D;
            // lane la has row 8bi+la; at step s it computes column 8bj + b, b = s - 7 + la
            float *Tr = T + row * LD + 8 * bj;
            const float *wr = wt + LD * rb[row] + 8 * bj, *Sb = SJ + 8 * bj * LD + 8 * bj;
            float cx[3];  // S2(r, r+4 ..): R2 from rows five to seven below, inside the block
#pragma unroll
            for (int x = 0; x < 3; ++x) cx[x] = la + x + 5 < 8 ? SX[row * LD + row + 5 + x] : NEG_INF;
            float n[15], under = NEG_INF, left = NEG_INF, diag = NEG_INF;  // (r+1, b), (r, b-1), (r+1, b-1)
#pragma unroll
            for (int s = 0; s < 15; ++s) {
                const int b = s - 7 + la, bc = min(max(b, 0), 7);
                float v = Tr[bc];
                const float w2 = e1 + s - 7 >= 4 ? wr[bc] : NEG_INF;
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    if (s >= 5 + x) {  // five to seven diagonals back: R1 in the lane, R2 from lane la + 5 + x
                        const float r1 = n[s - 5 - x] + Sb[max(bc - 4 - x, 0) * LD + bc];  // S2(c-5-x + 1, c)
                        const float r2 = __shfl_down_sync(0xffffffffu, n[s - 5 - x], 5 + x, 8) + cx[x];
                        v = fmax3(v, r1, r2);
                    }
                under = s > 0 ? __shfl_down_sync(0xffffffffu, n[s - 1], 1, 8) : NEG_INF;
                if (la == 7) under = NEG_INF;
                const float r = fmaxf(fmax3(v, left, under), diag + w2);
                n[s] = b >= 0 && b < cols ? r : NEG_INF;
                diag = under;
                left = n[s];
            }
#pragma unroll
            for (int s = 0; s < 15; ++s) {
                const int b = s - 7 + la;
                if (b >= 0 && b < cols) Tr[b] = n[s];
            }
        }
    }
    __syncthreads();
}

template <int NP, int T = fin_threads(NP)>
__global__ void __launch_bounds__(FinShape<NP, T>::THREADS, FinShape<NP, T>::MINB)
finalize_small_kernel(const CellJob *__restrict__ jobs, int njobs, const CellJob *__restrict__ s1jobs, int ns1,
                      const PairDesc *__restrict__ pairs, float *__restrict__ F, float *__restrict__ S,
                      const uint8_t *__restrict__ bases, Weights W, int d, RefOut ro)
{
    using Sh = FinShape<NP, T>;
    constexpr int NB = NP / 8, NBLK = NB * (NB + 1) / 2;
    constexpr long long CELL = 4LL * R0_TAB_COLBASE[NB][NB];
    extern __shared__ __align__(16) float fsm[];
    constexpr int LD = Sh::LD;
    float *D = fsm + 4, *SX = D + (NP + 1) * LD, *SJ = SX + NP * LD;  // the table; S2(r, c-1) and S2(r, c)
    uint8_t *sb = reinterpret_cast<uint8_t *>(SJ + NP * LD);
    __shared__ __align__(16) float wt[5 * LD];  // wt[LD*x + c]: intra-strand weight of base x and column c, -inf from N on
    __shared__ int cbs[NB];    // float offset of each block column in the cell image
    __shared__ float wsh[12];  // the weight table (indexed by pair type)
    __shared__ float w5[25];   // intra-strand weight of bases a, b at 5a + b
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 12) wsh[tid] = W.w[tid];
    for (int q = tid - (T >= 64 ? 32 : 0); q < 25; q += T)
        if (q >= 0) w5[q] = score_w(W.w, q / 5, q % 5);
    if (tid < NB) cbs[tid] = 4 * c_img_colbase[NB][tid];
    __syncthreads();
    if ((int)blockIdx.x >= njobs) {  // S1 cells (i, i+d+1), one per warp
        const int q = ((int)blockIdx.x - njobs) * Sh::WARPS + warp;
        if (q >= ns1) {
            chain_wait();
            return;
        }
        const CellJob job = s1jobs[q];
        const PairDesc pd = pairs[job.pair];
        const int M = pd.M, i = job.i1, j = i + d + 1;
        float *S1 = S + pd.S1_off;
        chain_wait();
        if (j - i <= 3) return;  // stays 0
        const uint8_t *s1 = bases + pd.seq1_off;
        float r0 = NEG_INF, r1 = NEG_INF;
        int k = i + lane;
        for (; k + 32 < j; k += 64) {
            r0 = fmaxf(r0, S1[i * M + k] + S1[(k + 1) * M + j]);
            r1 = fmaxf(r1, S1[i * M + k + 32] + S1[(k + 33) * M + j]);
        }
        if (k < j) r0 = fmaxf(r0, S1[i * M + k] + S1[(k + 1) * M + j]);
        float red = fmaxf(r0, r1);
        for (int o = 16; o > 0; o >>= 1) red = fmaxf(red, __shfl_xor_sync(0xffffffffu, red, o));
        if (lane == 0) S1[i * M + j] = fmaxf(S1[(i + 1) * M + (j - 1)] + score_w(wsh, s1[i], s1[j]), red);
        return;
    }
    const CellJob job = jobs[blockIdx.x];
    const PairDesc pd = pairs[job.pair];
    const int M = pd.M, N = pd.N, i1 = job.i1, j1 = i1 + d;
    float *Fc = F + pd.F_off + cell_index(M, i1, j1) * CELL;
    const float *S1 = S + pd.S1_off;
    const float *S2 = S + pd.S2_off;
    const uint8_t *s1 = bases + pd.seq1_off;
    const uint8_t *s2r = bases + pd.seq2_off;
    for (int q = tid; q < NP; q += Sh::THREADS) sb[q] = q < N ? s2r[q] : 4;
    for (int q = tid; q < 5 * LD; q += Sh::THREADS) {
        const int c = q % LD;
        wt[q] = c < N ? w5[5 * (q / LD) + s2r[c]] : NEG_INF;
    }
    const int x1 = s1[i1], y1 = s1[j1];
    chain_wait();
    const float s1v = S1[i1 * M + j1];
    // start values (accumulated products, S1+S2, SW1; the inter-strand base on the diagonal of the
    // diagonal cells; -inf elsewhere) and S2, 4 columns of one block row per step
    const bool sw1 = d >= 4;
    const float w1 = sw1 ? score_w(wsh, x1, y1) : 0.0f;
    const float *Fi = F + pd.F_off + (sw1 ? cell_index(M, i1 + 1, j1 - 1) * CELL : 0);
    if (tid < 4) D[tid - 4] = NEG_INF;
    for (int q = tid; q < 4 * NP; q += Sh::THREADS) D[(q >> 2) * LD + NP + (q & 3)] = NEG_INF;  // the pad columns
    for (int q4 = tid; q4 < NBLK * 16; q4 += Sh::THREADS) {
        int BI, BJ;
        blk_decode(NB, q4 >> 4, BI, BJ);
        const int r = 8 * BI + ((q4 & 15) >> 1), c0 = 8 * BJ + 4 * (q4 & 1), o = cbs[BJ] + 68 * BI + 4 * (q4 & 15);
        const float4 f4 = *reinterpret_cast<const float4 *>(Fc + o), s4 = *reinterpret_cast<const float4 *>(S2 + r * NP + c0);
        float4 p4 = make_float4(NEG_INF, NEG_INF, NEG_INF, NEG_INF);
        if (sw1) p4 = *reinterpret_cast<const float4 *>(Fi + o);
        const float fv[4] = {f4.x, f4.y, f4.z, f4.w}, pv[4] = {p4.x, p4.y, p4.z, p4.w};
        float sv[4] = {s4.x, s4.y, s4.z, s4.w}, v[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int c = c0 + t;
            SX[r * LD + c + 1] = sv[t];  // (column NP is pad)
            v[t] = r <= c && c < N ? (d == 0 && r == c ? score_w(wsh + 6, x1, s2r[r]) : fmax3(fv[t], s1v + sv[t], pv[t] + w1))
                                   : NEG_INF;
            if (c >= N) sv[t] = NEG_INF;
        }
        *reinterpret_cast<float4 *>(D + r * LD + c0) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4 *>(SJ + r * LD + c0) = make_float4(sv[0], sv[1], sv[2], sv[3]);
    }
    block_wave<LD, Sh::WARPS>(D, SX, SJ, wt, sb, true, NB, N, 0);  // (starts and ends with a barrier)
    // write-back, 4 columns of one block row per step
    for (int q4 = tid; q4 < NBLK * 16; q4 += Sh::THREADS) {
        int BI, BJ;
        blk_decode(NB, q4 >> 4, BI, BJ);
        const int r = 8 * BI + ((q4 & 15) >> 1), c0 = 8 * BJ + 4 * (q4 & 1);
        float v[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int c = c0 + t;
            v[t] = r <= c && c < N ? D[r * LD + c] : (r == c + 1 ? s1v : NEG_INF);  // S1 on the subdiagonal
        }
        // block (BI, BJ), row r & 7, half
        *reinterpret_cast<float4 *>(Fc + cbs[BJ] + 68 * BI + 4 * (q4 & 15)) = make_float4(v[0], v[1], v[2], v[3]);
    }
    if (tid < 2 * NB) {  // S1 piece of every block column: -inf x7, S1(i1,j1)
        const int BJ = tid >> 1, h = tid & 1;
        float4 p = make_float4(NEG_INF, NEG_INF, NEG_INF, NEG_INF);
        if (h == 1) p.w = s1v;
        *reinterpret_cast<float4 *>(Fc + cbs[BJ] + 68 * (BJ + 1) + 4 * h) = p;
    }
    if (ro.out) {  // this cell in the reference layout, from the final table in shared memory (the
                   // values the image holds), one warp per tile row of T floats
        const int TT = ro.T, R = (TT - N % TT) % TT, tile_rows = TT + 1, rows = ro.Ns * ro.Ns * tile_rows;
        float *dst = ro.out + ((long long)d * M - (long long)d * (d - 1) / 2 + i1) * ((long long)rows * TT);
        auto dval = [&](int i2, int j2) { return D[i2 * LD + j2]; };
        for (int rr = warp; rr < rows; rr += Sh::WARPS) {
            const int I2 = rr / (ro.Ns * tile_rows), rem = rr % (ro.Ns * tile_rows);
            const int J2 = rem / tile_rows, r = rem % tile_rows;
            for (int c = lane; c < TT; c += 32) dst[rr * TT + c] = reference_tile_elem_v(dval, TT, R, I2, J2, r, c);
        }
    }
}

// ------------------------------------------------------------------------------------------
// Layout conversion: compact device tables -> the reference's linear layout for outer row i1
// (cells (i1, j1) for j1 in [i1, M)): out[(j1-i1)][I2][J2][r][c] of N_tile x (N_tile+1) tiles
// (V3/bpmax-wrapper.c:44, :175-197). Written cells follow V3/bpmax_ftable_init.c:171-214
// (-FLT_MAX masks, halo of diagonal tiles) and V3/bpmax_inner_reductions_finalize.c:132 (halo of
// off-diagonal tiles = row 0 of the tile below); cells the reference never writes become NaN.
// ------------------------------------------------------------------------------------------
__global__ void to_reference_row_kernel(const PairDesc *__restrict__ pdp, const float *__restrict__ F, int T, int Ns,
                                        int i1, long long n_out, float *__restrict__ out)
{
    const PairDesc pd = *pdp;
    const int R = (T - pd.N % T) % T;
    const long long cell_f = (long long)Ns * Ns * (T + 1) * T;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n_out;
         q += (long long)gridDim.x * blockDim.x)
        out[q] = reference_elem(pd, F, T, Ns, R, i1, i1 + (int)(q / cell_f), q % cell_f);
}

// the same conversion for the cells of outer diagonal d (cells (i1, i1+d), i1 = 0 .. M-1-d), one
// after another in `out`: final all at once when the diagonal is, unlike a row
__global__ void to_reference_diag_kernel(const PairDesc *__restrict__ pdp, const float *__restrict__ F, int T, int Ns,
                                         int d, long long n_out, float *__restrict__ out)
{
    const PairDesc pd = *pdp;
    const int R = (T - pd.N % T) % T;
    const long long cell_f = (long long)Ns * Ns * (T + 1) * T;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n_out;
         q += (long long)gridDim.x * blockDim.x) {
        const int i1 = (int)(q / cell_f);
        out[q] = reference_elem(pd, F, T, Ns, R, i1, i1 + d, q % cell_f);
    }
}

// compact device tables -> dense compact host layout (stride N), -FLT_MAX below the diagonal
__global__ void to_compact_kernel(const PairDesc *__restrict__ pdp, const float *__restrict__ F, long long n_out,
                                  float *__restrict__ out)
{
    const PairDesc pd = *pdp;
    const int N = pd.N;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n_out;
         q += (long long)gridDim.x * blockDim.x) {
        const long long c = q / ((long long)N * N);
        const int r = (int)((q / N) % N), col = (int)(q % N);
        out[q] = r <= col ? f_value(pd, F, c, r, col) : -3.402823466e+38f;
    }
}

// inner tables of the outer cells (i1, j1), i1 in [i1_lo, i1_lo+nI), j1 in [j1_lo, j1_lo+nJ), of one
// pair -> out[i1-i1_lo][j1-j1_lo][N][N]; -FLT_MAX where i2 > j2, NaN for outer cells with i1 > j1
__global__ void read_cells_kernel(const PairDesc *__restrict__ pdp, const float *__restrict__ F, int i1_lo, int j1_lo,
                                  int nJ, long long n_out, float *__restrict__ out)
{
    const PairDesc pd = *pdp;
    const long long NN = (long long)pd.N * pd.N;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n_out;
         q += (long long)gridDim.x * blockDim.x) {
        const long long oc = q / NN;
        const int i1 = i1_lo + (int)(oc / nJ), j1 = j1_lo + (int)(oc % nJ);
        const int r = (int)((q % NN) / pd.N), c = (int)(q % pd.N);
        float v = __int_as_float(0x7fc00000);
        if (i1 <= j1) v = r <= c ? f_value(pd, F, cell_index(pd.M, i1, j1), r, c) : -3.402823466e+38f;
        out[q] = v;
    }
}

__global__ void gather_scores_kernel(const PairDesc *__restrict__ pairs, const float *__restrict__ F, int num_pairs,
                                     float *__restrict__ scores)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= num_pairs) return;
    const PairDesc pd = pairs[p];
    scores[p] = f_value(pd, F, cell_index(pd.M, 0, pd.M - 1), 0, pd.N - 1);
}

// ------------------------------------------------------------------------------------------
// Max-plus issue ceiling: the product kernel's instruction mix with nothing to share between
// candidates. Each step of a chain is one packed add (two candidate sums, the running operand
// plus a step) and one 3-input max that merges both sums into the chain's maximum; every sum is
// new (the running operand changes each step) and is consumed once, so the compiler can neither
// hoist nor reuse an add. MAXPLUS_PEAK_CHAINS independent chains per thread give the schedulers
// the same independent work as the product kernel's 8x8 tile. Each iteration is
// 4 * 2 * MAXPLUS_PEAK_CHAINS candidates per thread.
// ------------------------------------------------------------------------------------------
constexpr int MAXPLUS_PEAK_CHAINS = 16;
__global__ void __launch_bounds__(128) maxplus_peak_kernel(const float *__restrict__ in, float *__restrict__ out,
                                                           int reps)
{
    constexpr int CH = MAXPLUS_PEAK_CHAINS;
    float2 p[CH], q[CH];
    float m[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        p[i] = make_float2(in[(threadIdx.x + i) & 63], in[(threadIdx.x + 2 * i + 1) & 63]);
        q[i] = make_float2(in[(threadIdx.x + 3 * i + 2) & 63] * 1e-7f, in[(threadIdx.x + 5 * i + 3) & 63] * 1e-7f);
        m[i] = NEG_INF;
    }
    for (int r = 0; r < reps; ++r) {
#pragma unroll
        for (int s = 0; s < 4; ++s)
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                p[i] = __fadd2_rn(p[i], q[i]);
                m[i] = fmax3(m[i], p[i].x, p[i].y);
            }
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < CH; ++i) s += p[i].x + p[i].y + m[i];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace bpmax
