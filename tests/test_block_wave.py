"""The inner wavefront by 8x8 blocks (block_wave in bpmax_b200/csrc/bpmax_kernels.cuh) on the CPU: the function's own
source is compiled for the host, with a fiber for every CUDA thread, and run over the tables of every
width class and over the 64x64 tiles of wider ones, against the plain wavefront
(V3/bpmax_verify.c:614-667). What the kernels leave unset in shared memory is poisoned.

Also the order of the tile steps (bpmax_tile.cuh), the S2 tile images, and the lanes of a narrow last
tile column (wide_split in bpmax_wide.cuh)."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bpmax_b200", "csrc")
NEG, POISON = np.float32(-np.inf), np.float32(1e30)


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


@pytest.fixture(scope="module")
def wave(tmp_path_factory):
    d = tmp_path_factory.mktemp("wave")
    body = re.search(r"template <int LD, int WARPS>\n__device__ __forceinline__ void block_wave\(.*?\n}\n",
                     source("bpmax_kernels.cuh"), re.S).group(0)
    (d / "block_wave.inc").write_text(body)
    out = str(d / "wave.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wno-unknown-pragmas",
                    f'-DBLOCK_WAVE_SOURCE="{d / "block_wave.inc"}"', "-o", out,
                    os.path.join(ROOT, "tests", "block_wave_host.cpp")], check=True)
    lib = ctypes.CDLL(out)

    def run(T, SX, SJ, wt, rb, warps, tri, nb, ncol, e0):
        """T: (rows + 1) x LD after its 4 leading words, as in shared memory."""
        ld = wt.shape[1]
        lib.host_block_wave(ctypes.c_void_p(T.ctypes.data + 16), *(ctypes.c_void_p(a.ctypes.data) for a in (SX, SJ, wt, rb)),
                            ld, warps, tri, nb, ncol, e0)

    return run


def strand_table(n, rng):
    """A single-strand table: 0 up to a span of 3, a maximum over splits and pairs beyond."""
    S = np.zeros((n + 1, n + 1), np.float32)
    for d in range(4, n):
        for i in range(n - d):
            j = i + d
            S[i, j] = max(S[i + 1, j - 1] + np.float32(rng.integers(0, 4)), (S[i, i:j] + S[i + 1:j + 1, j]).max())
    return S


def problem(N, seed):
    rng = np.random.default_rng(seed)
    bases = rng.integers(0, 5, N).astype(np.uint8)
    w5 = rng.random((5, 5)).astype(np.float32)
    w5[4] = w5[:, 4] = 0
    F0 = np.full((N, N), NEG, np.float32)
    iu = np.triu_indices(N)
    F0[iu] = (rng.random(len(iu[0])) * 9).astype(np.float32)
    return F0, strand_table(N, rng), bases, w5


def plain(F0, S2, bases, w5):
    N = len(bases)
    F = F0.copy()
    for d in range(1, N):
        for i in range(N - d):
            j = i + d
            v = max(F[i, j], (F[i, i:j] + S2[i + 1:j + 1, j]).max(), (S2[i, i:j] + F[i + 1:j + 1, j]).max())
            if d >= 4:
                v = max(v, F[i + 1, j - 1] + w5[bases[i], bases[j]])
            F[i, j] = v
    return F


def buffer(rows, ld):
    T = np.full(4 + (rows + 1) * ld, NEG, np.float32)
    return T, T[4:].reshape(rows + 1, ld)


def weights(w5, bases, ncol, ld):
    wt = np.full((5, ld), NEG, np.float32)
    wt[:, :ncol] = w5[:, bases[:ncol]]
    return wt


@pytest.mark.parametrize("N", [1, 2, 3, 5, 7, 8, 9, 12, 13, 16, 17, 21, 24, 25, 31, 33, 40, 41, 47, 50, 56, 57, 60, 63, 64])
def test_triangle(wave, N):
    """finalize_small_kernel's tables: only the upper block triangle of S2 is loaded."""
    F0, S2, bases, w5 = problem(N, N)
    nb = (N + 7) // 8
    NP, ld = 8 * nb, 8 * nb + 4
    raw, T = buffer(NP, ld)
    T[:N, :N] = F0
    SX, SJ = np.full((NP, ld), POISON), np.full((NP, ld), POISON)
    S = np.zeros((NP, NP), np.float32)
    S[:N, :N] = S2[:N, :N]
    for r in range(NP):
        b = r // 8 * 8
        SX[r, b + 1:NP + 1] = S[r, b:]
        SJ[r, b:NP] = np.where(np.arange(b, NP) < N, S[r, b:], NEG)
    rb = np.full(NP, 4, np.uint8)
    rb[:N] = bases
    wave(raw, SX, SJ, weights(w5, bases, N, ld), rb, 1 if nb <= 2 else 4, 1, nb, N, 0)
    assert np.array_equal(T[:N, :N], plain(F0, S2, bases, w5))
    assert np.all(T[:, N:] == NEG) and np.all(T[N:] == NEG) and np.all(raw[:4] == NEG)


@pytest.mark.parametrize("N,warps", [(65, 8), (70, 8), (72, 8), (73, 16), (100, 8), (128, 8), (130, 4), (137, 8), (150, 8)])
def test_tiles(wave, N, warps):
    """Tile diagonal by tile diagonal, as the steps run them: the terms over finished tiles, the k of R2 between
    them and the tile, SW2 of its first column and last row, then the tile's own wavefront."""
    F0, S2, bases, w5 = problem(N, N)
    NT, ld = (N + 63) // 64, 68
    S = np.zeros((64 * NT, 64 * NT + 1), np.float32)
    S[:N, :N] = S2[:N, :N]
    b = np.full(64 * NT, 4, np.uint8)
    b[:N] = bases
    F = np.full((64 * NT + 1, 64 * NT), NEG, np.float32)
    for t in range(NT):
        for I in range(NT - t):
            J, r0 = I + t, 64 * I
            c0, ncol = 64 * J, min(64, N - 64 * J)
            raw, T = buffer(64, ld)
            for r in range(64):
                for c in range(ncol):
                    i, j = r0 + r, c0 + c
                    if i > j:
                        continue
                    v = F0[i, j]
                    if t > 0:
                        v = max(v, (F[i, i:c0] + S[i + 1:c0 + 1, j]).max(), (S[i, r0 + 63:j] + F[r0 + 64:j + 1, j]).max())
                        if (c == 0 or r == 63) and j - i >= 4:
                            v = max(v, F[i + 1, j - 1] + w5[b[i], b[j]])
                    T[r, c] = v
            SX, SJ = np.full((64, ld), POISON), np.full((64, ld), POISON)
            SX[:, 1:65] = S[r0:r0 + 64, r0:r0 + 64]
            SJ[:, :64] = np.where(np.arange(64) < ncol, S[c0:c0 + 64, c0:c0 + 64], NEG)
            wave(raw, SX, SJ, weights(w5, b[c0:], ncol, ld), b[r0:r0 + 64].copy(), warps, int(t == 0), 8, ncol, 64 * t)
            F[r0:r0 + 64, c0:c0 + 64] = T[:64, :64]
    assert np.array_equal(F[:N, :N], plain(F0, S2, bases, w5))
    assert np.all(F[:, N:] == NEG)


def test_steps_meet_only_finished_tiles():
    """Step of tile (I, J) of outer cell (i1, j1): j1 - i1 + J - I. Everything it reads is of an earlier step."""
    M, NT = 6, 4
    step = lambda i1, j1, I, J: j1 - i1 + J - I
    for i1 in range(M):
        for j1 in range(i1, M):
            for I in range(NT):
                for J in range(I, NT):
                    s = step(i1, j1, I, J)
                    for k1 in range(i1, j1):  # products: tiles (I, K) and (K, J) of two other cells, and the row after
                        for K in range(I, J + 1):
                            assert step(i1, k1, I, K) < s and step(k1 + 1, j1, K, J) < s
                    for K in range(I, J):  # R1, R2, the halo row and SW2 of the cell itself
                        assert step(i1, j1, I, K) < s and step(i1, j1, K + 1, J) < s
                    if j1 - i1 >= 2:  # SW1
                        assert step(i1 + 1, j1 - 1, I, J) < s


def test_s2_images_are_disjoint_and_fit():
    dense = 4 * int(re.search(r"WIDE_DENSE_COLBASE\[9\] = \{(.*?)\}", source("wide_tables.inc")).group(1).split(",")[8])
    off = lambda NT, I, J: (I * (NT - 1) - I * (I - 1) // 2 + (J - I - 1)) * dense  # s2_image_off
    for NT in (2, 3, 5, 16, 47, 64):
        at = sorted(off(NT, I, J) for I in range(NT) for J in range(I + 1, NT))
        assert at == [k * dense for k in range(NT * (NT - 1) // 2)]
        assert at[-1] + dense <= (64 * NT) ** 2  # the room the plan gives them


def test_lanes_of_a_narrow_tile_column():
    """Output tiles of nbc < 8 block columns: every micro-tile has its lanes, and they take each of its k blocks once,
    whatever the kinds of the operand tiles."""
    text = re.search(r"constexpr int wide_split\(int nbc\)\n{\n    return (.*?);", source("bpmax_wide.cuh")).group(1)
    split = {n: int(eval(re.sub(r"nbc == (\d) \? (\d) : ", r"\2 if nbc == \1 else ",
                                re.sub(r"nbc <= (\d) \? (\d) : ", r"\2 if nbc <= \1 else ", text)), {"nbc": n})) for n in range(1, 8)}
    for nbc in range(1, 8):
        s = split[nbc]
        assert 8 * nbc * s <= 128
        for a_diag, b_diag in ((0, 0), (1, 0), (0, 1)):
            seen = {}
            for tid in range(128):
                h, m = divmod(tid, 8 * nbc)
                if h >= s:
                    continue
                bi, bj = m & 7, m >> 3
                for kb in range((bi if a_diag else 0) + h, bj + 1 if b_diag else 8, s):
                    assert (bi, bj, kb) not in seen
                    seen[bi, bj, kb] = tid
            exp = {(bi, bj, kb) for bi in range(8) for bj in range(nbc) for kb in range(bi if a_diag else 0, bj + 1 if b_diag else 8)}
            assert set(seen) == exp
