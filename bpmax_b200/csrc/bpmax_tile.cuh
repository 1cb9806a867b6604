// bpmax_tile.cuh -- finalize of inner tables stored as tile images (Np = 64 * NT > 64, layout in
// bpmax_kernels.cuh), by tiles over the whole GPU.
//
// Tile (I, J) of a cell's table F (rows 64I.., columns 64J..) needs, beside its start values,
//   R1  F[i2][k] + S2(k+1, j2), k in [i2, j2): k < 64J lies in the finished tiles (I, K), K < J;
//       k >= 64J in the tile itself
//   R2  S2(i2, k-1) + F[k][j2], k in (i2, j2]: k >= 64(I+1) lies in the finished tiles (K, J), K > I;
//       k < 64(I+1) in the tile itself
// and the product R0+R3+R4 of the tile needs only tiles of other cells that lie at most as many tile
// diagonals t = J - I up. So tile diagonal t of outer diagonal d runs in step d + t, beside the earlier tile
// diagonals of later outer diagonals: M + NT - 1 steps of two launches, r0_wide_kernel (the products of
// the step's tiles, and the terms over finished tiles as items of the same kind) and tile_final_kernel
// (one CTA per tile of the step: start values, SW1, the tile's own terms, the tile image).
// The tile's own terms go by 8x8 blocks (block_wave in bpmax_kernels.cuh); SW2 from outside the tile is
// read where it lies.
//
// Bound: latency of a tile's own terms (a tile of t >= 1 runs 15 block diagonals of products
// and of the blocks' wavefronts, about 1,000 cycles each, and 5 us of loads). Fill ms with one CTA per cell
// walking every inner diagonal (up to width 320; above, row-major tables with a barrier per tile
// diagonal) / with the tile diagonals of one outer diagonal after another, the terms over finished tiles
// in launches of their own / in steps as here: 90x130 32.0 / 24.1 / 19.1,
// 256x256 950 / 709 / 698, 16x750 47.6 / 16.9 / 9.9, 32x1024 238 / 110 / 83.
// Tried for the tile's own terms: batches of five tile diagonals pushed to all later entries, 61 us a
// tile (the pushes took 2,800 cycles a batch); 512 and 1,024 threads a tile, no faster.
#pragma once
#include "bpmax_wide.cuh"

namespace bpmax {

constexpr int TILE_THREADS = 256;
constexpr int TILE_LD = 68;  // row pitch of the tile and of the S2 blocks in shared memory: 17 16-byte chunks
// shared memory: the tile (64 rows, after 4 words and before one row of -inf; the pad columns of a row
// are -inf too, so column -1, the pad before the row, columns 64.. and row 64 may be read), the S2 blocks
constexpr int TILE_OFF_S2 = 4 * (65 * TILE_LD + 8);
constexpr size_t TILE_SMEM = TILE_OFF_S2 + 2 * 4 * 64 * TILE_LD;

// tile (I, J) (tile = I << 8 | J) of the table of cell (i1, i1+d) of pair `pair`
struct TileJob {
    int pair, i1, d, tile;
};

// ------------------------------------------------------------------------------------------
// The dense tile images (with halo pieces) of S2 of the pairs with Np > 64, S2 over the reversed strand
// 2 (V3/bpmax_verify.c:560-571); -inf in columns >= N. The pairs are on x: a batch may hold more of them than
// a grid's y extent (65,535). Only wide pairs have CTAs: with 64 for every pair, one wide pair among 20,000 narrow
// ones added 1.47 ms to the batch, now 0.13.
// ------------------------------------------------------------------------------------------
__global__ void s2_aux_kernel(const int *__restrict__ wide, const PairDesc *__restrict__ pairs, float *__restrict__ S)
{
    const PairDesc pd = pairs[wide[blockIdx.x]];
    const int Np = pd.Np, N = pd.N, NT = Np >> 6;
    chain_wait();
    const float *S2 = S + pd.S2_off;
    float *img = S + pd.S2x_off;
    for (long long q = blockIdx.y * (long long)blockDim.x + threadIdx.x; q < (long long)Np * Np;
         q += (long long)gridDim.y * blockDim.x) {
        const int r = (int)(q / Np), c = (int)(q % Np), I = r >> 6, J = c >> 6, o = 4 * c_wide_dense_colbase[(c & 63) >> 3];
        const float v = c < N ? S2[q] : NEG_INF;
        if (I < J) img[s2_image_off(NT, I, J) + o + 4 * 17 * ((r & 63) >> 3) + 8 * (r & 7) + (c & 7)] = v;
        if ((r & 63) == 0 && I > 0 && I <= J) img[s2_image_off(NT, I - 1, J) + o + 4 * 17 * 8 + (c & 7)] = v;
    }
}

// ------------------------------------------------------------------------------------------
// S2 of one pair with Np > S2_ONE_CTA_NP, one launch per diagonal d of its wavefront
// (single_strand_kernel's one CTA per pair took 2.2 s at N = 3000), one warp per cell. The column
// operand S2(k+1, j) is read from ST[j][k], which the same launches fill as cells become final (in the
// room of the images, which s2_aux_kernel writes afterwards); S starts at 0, so ST holds the 0
// of every cell with j-i <= 3.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
s2_diag_kernel(const PairDesc *__restrict__ pairs, int p, const uint8_t *__restrict__ bases, float *__restrict__ S,
               Weights W, int d)
{
    const PairDesc pd = pairs[p];
    const int L = pd.N, ld = pd.Np;
    const int i = (int)blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    chain_wait();
    if (i >= L - d) return;
    const int j = i + d;
    float *T = S + pd.S2_off, *TT = S + pd.S2x_off;
    const uint8_t *s = bases + pd.seq2_off;
    float r0 = NEG_INF, r1 = NEG_INF;
    int k = i + lane;
    for (; k + 32 < j; k += 64) {
        r0 = fmaxf(r0, T[(long long)i * ld + k] + TT[(long long)j * ld + k]);
        r1 = fmaxf(r1, T[(long long)i * ld + k + 32] + TT[(long long)j * ld + k + 32]);
    }
    if (k < j) r0 = fmaxf(r0, T[(long long)i * ld + k] + TT[(long long)j * ld + k]);
    float red = fmaxf(r0, r1);
    for (int o = 16; o > 0; o >>= 1) red = fmaxf(red, __shfl_xor_sync(0xffffffffu, red, o));
    if (lane == 0) {
        const float v = fmaxf(T[(long long)(i + 1) * ld + (j - 1)] + score_w(W.w, s[i], s[j]), red);
        T[(long long)i * ld + j] = v;
        if (i >= 1) TT[(long long)j * ld + i - 1] = v;
    }
}

// S1 cell (i, i+d+1) of a job by one warp (V3/bpmax_verify.c:533-544), from S1 diagonals <= d
__device__ __forceinline__ void s1_cell(const CellJob &job, const PairDesc *__restrict__ pairs, float *__restrict__ S,
                                        const uint8_t *__restrict__ bases, const float *w, int d, int lane)
{
    const PairDesc pd = pairs[job.pair];
    const int M = pd.M, i = job.i1, j = i + d + 1;
    float *S1 = S + pd.S1_off;
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
    if (lane == 0) S1[i * M + j] = fmaxf(S1[(i + 1) * M + (j - 1)] + score_w(w, s1[i], s1[j]), red);
}

// CTAs [0, njobs): one tile each; after them one warp per S1 cell (i, i+step+1). MINB: CTAs per SM, 2
// (128 registers) or, for steps of more tiles than two per SM, 3 (80). Fill ms at 2 / 3: 90x70 (at most 90
// tiles) 6.12 / 6.24, 90x130 14.5 / 14.7, 256x256 680 / 676, 32x1024 81.2 / 80.1.
template <int MINB>
__global__ void __launch_bounds__(TILE_THREADS, MINB)
tile_final_kernel(const TileJob *__restrict__ jobs, int njobs, const CellJob *__restrict__ s1jobs, int ns1,
                  const PairDesc *__restrict__ pairs, float *__restrict__ F, float *__restrict__ S,
                  const uint8_t *__restrict__ bases, Weights W, int step)
{
    constexpr int LD = TILE_LD;
    extern __shared__ __align__(16) float tsm[];
    float *T = tsm + 4;
    __shared__ float wsh[12], w5[25];
    __shared__ __align__(16) float wt[5 * LD];  // wt[LD*x + c]: weight of base x and column c of the tile, -inf from ncol on
    __shared__ uint8_t bI[64], bJ[64];
    __shared__ float below[64], s2r_end[64];  // F[64(I+1)][64J+c] and S2(64I+r, 64I+63)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 12) wsh[tid] = W.w[tid];
    if (tid >= 32 && tid < 57) w5[tid - 32] = score_w(W.w, (tid - 32) / 5, (tid - 32) % 5);
    if ((int)blockIdx.x >= njobs) {
        __syncthreads();
        const int q = ((int)blockIdx.x - njobs) * (TILE_THREADS / 32) + warp;
        chain_wait();
        if (q < ns1) s1_cell(s1jobs[q], pairs, S, bases, wsh, step, lane);
        return;
    }
    const TileJob job = jobs[blockIdx.x];
    const int I = job.tile >> 8, J = job.tile & 0xff, t = J - I, d = job.d;
    const PairDesc pd = pairs[job.pair];
    const int M = pd.M, N = pd.N, Np = pd.Np, NT = Np >> 6, i1 = job.i1, j1 = i1 + d;
    const int ncol = min(64, N - 64 * J);  // columns of the tile inside the table
    const long long CELL = wide_cell_floats(NT);
    float *Fc = F + pd.F_off + cell_index(M, i1, j1) * CELL;
    float *Ft = Fc + wide_tile_off(NT, I, J);
    const float *S2 = S + pd.S2_off;
    const uint8_t *s1 = bases + pd.seq1_off, *s2r = bases + pd.seq2_off;
    if (tid < 64)
        bI[tid] = 64 * I + tid < N ? s2r[64 * I + tid] : 4;
    else if (tid < 128)
        bJ[tid - 64] = 64 * J + tid - 64 < N ? s2r[64 * J + tid - 64] : 4;
    const int x1 = s1[i1], y1 = s1[j1];
    chain_wait();
    const float s1v = S[pd.S1_off + i1 * M + j1];
    // row 0 of the tile below: the halo pieces, and with the last column of S2's block I the one k of R2
    // between this tile and the finished ones, S2(i2, 64I+63) + F[64(I+1)][j2]
    const float *Fb = t > 0 ? Fc + wide_tile_off(NT, I + 1, J) : nullptr;
    if (t > 0 && tid < 64)
        below[tid] = Fb[4 * (t == 1 ? c_img_colbase[8][tid >> 3] : c_wide_dense_colbase[tid >> 3]) + (tid & 7)];
    else if (t > 0 && tid < 128)
        s2r_end[tid - 64] = S2[(long long)(64 * I + tid - 64) * Np + 64 * I + 63];
    __syncthreads();
    // start values: accumulated products, S1+S2, SW1 (F(i1+1,j1-1,.)+intra if j1-i1 >= 4); the
    // inter-strand base on the diagonal of the diagonal cells. Entries outside the table stay -inf.
    const bool sw1 = d >= 4;
    const float w1 = sw1 ? score_w(wsh, x1, y1) : 0.0f;
    const float *Fi = F + pd.F_off + (sw1 ? cell_index(M, i1 + 1, j1 - 1) * CELL : 0) + wide_tile_off(NT, I, J);
    const int nblk = t == 0 ? 36 : 64;
    for (int q = tid - 4; q < 65 * LD; q += TILE_THREADS)
        if (t == 0 || q < 0 || q % LD >= ncol || q >= 64 * LD) T[q] = NEG_INF;
    for (int q = tid; q < 5 * LD; q += TILE_THREADS) {
        const int c = q % LD;
        wt[q] = c < ncol ? w5[5 * (q / LD) + bJ[c]] : NEG_INF;
    }
    // four columns of one block row per step; every load of a thread is issued before the first is used
    constexpr int Q = 1024 / TILE_THREADS;
    float4 f4[Q], s4[Q], p4[Q];
    int rc[Q];  // row << 8 | first column, -1: none
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const int q4 = tid + TILE_THREADS * k;
        int bi = (q4 >> 4) & 7, bj = q4 >> 7;
        rc[k] = -1;
        if (t == 0 && q4 < 36 * 16) blk_decode(8, q4 >> 4, bi, bj);
        if (q4 < nblk * 16) {
            const int r = 8 * bi + ((q4 & 15) >> 1), c0 = 8 * bj + 4 * (q4 & 1);
            const int o = 4 * ((t == 0 ? c_img_colbase[8][bj] : c_wide_dense_colbase[bj]) + 17 * bi) + 4 * (q4 & 15);
            rc[k] = r << 8 | c0;
            f4[k] = *reinterpret_cast<const float4 *>(Ft + o);
            s4[k] = *reinterpret_cast<const float4 *>(S2 + (long long)(64 * I + r) * Np + 64 * J + c0);
            p4[k] = sw1 ? *reinterpret_cast<const float4 *>(Fi + o) : make_float4(NEG_INF, NEG_INF, NEG_INF, NEG_INF);
        }
    }
    if (t == 0) __syncthreads();
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        if (rc[k] < 0) continue;
        const int r = rc[k] >> 8, c0 = rc[k] & 255;
        const float fv[4] = {f4[k].x, f4[k].y, f4[k].z, f4[k].w}, sv[4] = {s4[k].x, s4[k].y, s4[k].z, s4[k].w};
        const float pv[4] = {p4[k].x, p4[k].y, p4[k].z, p4[k].w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = c0 + u;
            if (c < ncol && (t > 0 || r <= c)) {
                float v = fmax3(fv[u], s1v + sv[u], pv[u] + w1);
                if (t > 0) v = fmaxf(v, s2r_end[r] + below[c]);
                if (d == 0 && t == 0 && r == c) v = score_w(wsh + 6, x1, bI[r]);
                T[r * LD + c] = v;
            }
        }
    }
    __syncthreads();
    // SW2 of the first column and the last row, from the finished tiles left of and below the tile
    if (t > 0 && tid < 127) {
        const int a = tid < 64 ? tid : 63, b = tid < 64 ? 0 : tid - 63;
        if (b < ncol && 64 * t + b - a >= 4) {
            const float f = Fc[wide_pos(NT, 64 * I + a + 1, 64 * J + b - 1)];
            T[a * LD + b] = fmaxf(T[a * LD + b], f + w5[5 * bI[a] + bJ[b]]);
        }
    }
    // S2 inside the tile's row block and column block: SX[x][y] = S2(64I+x, 64I+y-1) (y > x),
    // SJ[x][y] = S2(64J+x, 64J+y), -inf in columns outside the table
    float *SX = tsm + TILE_OFF_S2 / 4, *SJ = SX + 64 * LD;
#pragma unroll
    for (int q = tid; q < 1024; q += TILE_THREADS) {
        const int x = q >> 4, y = 4 * (q & 15);
        const float4 u = *reinterpret_cast<const float4 *>(S2 + (long long)(64 * I + x) * Np + 64 * I + y);
        float4 v = *reinterpret_cast<const float4 *>(S2 + (long long)(64 * J + x) * Np + 64 * J + y);
        float *o = SX + x * LD + y + 1;
        o[0] = u.x;
        o[1] = u.y;
        o[2] = u.z;
        o[3] = u.w;  // (column 64 is pad)
        if (y >= ncol) v.x = NEG_INF;
        if (y + 1 >= ncol) v.y = NEG_INF;
        if (y + 2 >= ncol) v.z = NEG_INF;
        if (y + 3 >= ncol) v.w = NEG_INF;
        *reinterpret_cast<float4 *>(SJ + x * LD + y) = v;
    }
    block_wave<LD, TILE_THREADS / 32>(T, SX, SJ, wt, bI, t == 0, 8, ncol, 64 * t);  // (starts and ends with a barrier)
    // the tile image: S1(i1,j1) on the subdiagonal of a diagonal tile, -inf elsewhere outside the table;
    // then the closing pieces of the block columns: S1 pieces, or row 0 of the tile below (halo)
    for (int q4 = tid; q4 < nblk * 16 + 16; q4 += TILE_THREADS) {
        if (q4 >= nblk * 16) {
            const int bj = (q4 - nblk * 16) >> 1, h = q4 & 1;
            float4 v = make_float4(NEG_INF, NEG_INF, NEG_INF, NEG_INF);
            if (t == 0) {
                if (h == 1) v.w = s1v;
            } else {
                v = make_float4(below[8 * bj + 4 * h], below[8 * bj + 4 * h + 1], below[8 * bj + 4 * h + 2],
                                below[8 * bj + 4 * h + 3]);
            }
            *reinterpret_cast<float4 *>(Ft + 4 * ((t == 0 ? c_img_colbase[8][bj] + 17 * (bj + 1)
                                                          : c_wide_dense_colbase[bj] + 17 * 8) + h)) = v;
            continue;
        }
        int bi, bj;
        if (t == 0) {
            blk_decode(8, q4 >> 4, bi, bj);
        } else {
            bi = (q4 >> 4) & 7;
            bj = q4 >> 7;
        }
        const int r = 8 * bi + ((q4 & 15) >> 1), c0 = 8 * bj + 4 * (q4 & 1);
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = c0 + u;
            v[u] = t == 0 && r > c ? (r == c + 1 ? s1v : NEG_INF) : T[r * LD + c];
        }
        *reinterpret_cast<float4 *>(Ft + 4 * ((t == 0 ? c_img_colbase[8][bj] : c_wide_dense_colbase[bj]) + 17 * bi) +
                                    4 * (q4 & 15)) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

}  // namespace bpmax
