"""Columns past the end of strand 2 in a table's tile images stay -inf, as the layout says."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from bpmax_b200 import build as B, workloads as W

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tiles") / "harness.so")
    subprocess.run([B.nvcc(), *B.NVCC_FLAGS, "-I", B.CSRC, "-o", out, os.path.join(HERE, "tile_padding_harness.cu")],
                   check=True, capture_output=True)
    lib = ctypes.CDLL(out)
    lib.tile_padding.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("N", [65, 66, 70, 71, 72, 73, 100, 127, 128, 130, 137, 190, 255, 320])
def test_padding_columns_stay_minus_inf(harness, N):
    rng = np.random.default_rng(N)
    bases = np.concatenate([W.random_sequence(1, rng), W.random_sequence(N, rng)]).astype(np.uint8)
    w = W.random_weights(N)
    assert harness.tile_padding(bases.ctypes.data, N, w.ctypes.data) == 0
