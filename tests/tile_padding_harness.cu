// Runs the tile finalize over the one cell of a pair with M = 1 and counts the entries of its table image
// in columns >= N that are not -inf.
#include <cstdio>
#include <vector>

#include "bpmax_tile.cuh"

using namespace bpmax;

extern "C" int tile_padding(const unsigned char *bases, int N, const float *weights)
{
    const int NT = (N + 63) / 64, Np = 64 * NT;
    Weights W;
    for (int k = 0; k < 12; ++k) W.w[k] = weights[k];
    PairDesc pd{};
    pd.M = 1;
    pd.N = N;
    pd.Np = Np;
    pd.S2_off = 64;
    pd.seq2_off = 1;
    PairDesc *dpd;
    float *F, *S;
    unsigned char *db;
    TileJob *dj;
    const size_t nF = (size_t)wide_cell_floats(NT), nS = 64 + (size_t)Np * Np;
    std::vector<float> img(nF);
    bool ok = N <= S2_ONE_CTA_NP && cudaMalloc(&dpd, sizeof pd) == cudaSuccess && cudaMalloc(&F, 4 * nF) == cudaSuccess &&
              cudaMalloc(&S, 4 * nS) == cudaSuccess && cudaMalloc(&db, N + 1) == cudaSuccess &&
              cudaMalloc(&dj, NT * sizeof(TileJob)) == cudaSuccess;
    if (!ok) return -1;
    cudaMemcpy(dpd, &pd, sizeof pd, cudaMemcpyHostToDevice);
    cudaMemcpy(db, bases, N + 1, cudaMemcpyHostToDevice);
    cudaMemset(F, 0, 4 * nF);
    cudaMemset(S, 0, 4 * nS);
    cudaFuncSetAttribute(tile_final_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_SMEM);
    single_strand_kernel<<<1, 512>>>(dpd, db, S, W);
    for (int t = 0; t < NT; ++t) {
        std::vector<TileJob> jobs;
        for (int I = 0; I + t < NT; ++I) jobs.push_back(TileJob{0, 0, 0, I << 8 | (I + t)});
        cudaMemcpy(dj, jobs.data(), jobs.size() * sizeof(TileJob), cudaMemcpyHostToDevice);
        tile_final_kernel<2><<<(int)jobs.size(), TILE_THREADS, TILE_SMEM>>>(dj, (int)jobs.size(), nullptr, 0, dpd, F, S, db,
                                                                          W, t);
    }
    ok = cudaMemcpy(img.data(), F, 4 * nF, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(dpd), cudaFree(F), cudaFree(S), cudaFree(db), cudaFree(dj);
    if (!ok) return -2;
    int bad = 0;
    for (int r = 0; r < Np; ++r)
        for (int c = r > N ? r : N; c < Np; ++c) bad += img[wide_pos(NT, r, c)] != NEG_INF;
    if (img[wide_pos(NT, 0, N - 1)] == NEG_INF) return -3;  // the table itself is there
    return bad;
}
