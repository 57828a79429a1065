"""The DWT's copy of the odd levels' details when levels differ in the accesses
their width admits: the rule on the CPU, the coefficients on the GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import bpc_synth
from conftest import ROOT


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("dwt")
    src, out = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write('#include "bpc_dwt_plan.h"\n'
                'extern "C" int vec_level(long a, long b, int X, int levels) '
                '{ return bpc::dwt_copy_vec_level((void *)a, (void *)b, X, levels); }\n'
                'extern "C" int columns() { return bpc::kDwtCopyColumns; }\n'
                'extern "C" int column(int wide, int t, int j) { return bpc::dwt_copy_column(wide, t, j); }\n')
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "cuda_bpc-paco_b200", "csrc"), src, "-o", out])
    L = ctypes.CDLL(out)
    L.vec_level.argtypes = [ctypes.c_long, ctypes.c_long, ctypes.c_int, ctypes.c_int]
    return L


@pytest.mark.parametrize("X,levels,want", [
    (8192, 5, 5), (8256, 5, 3), (8224, 5, 3), (1984, 5, 3), (8224, 4, 3), (8208, 4, 1), (8, 1, 1), (8, 2, 1),
    (12, 1, 0), (4, 1, 0), (264, 3, 1), (96, 1, 1), (32768, 14, 13)])
def test_each_level_has_its_own_accesses(plan, X, levels, want):
    assert plan.vec_level(1 << 20, 3 << 20, X, levels) == want
    for a, b in ((4, 0), (0, 8), (12, 12)):  # a raster off the 16-byte boundary: none
        assert plan.vec_level((1 << 20) + a, (3 << 20) + b, X, levels) == 0


@pytest.mark.parametrize("wide", [0, 1])
def test_copy_covers_each_column_once(plan, wide):
    for w in (2, 8, 128, 510, 512, 520, 1544, 5998):
        threads = -(-w // plan.columns()) * 128
        cols = sorted(plan.column(wide, t, j) for t in range(threads) for j in range(4))
        assert cols == list(range(threads * 4)) and threads * 4 >= w


@pytest.mark.gpu
@pytest.mark.parametrize("H,W,levels", [(96, 320, 5), (64, 1984, 5), (128, 8256, 5), (40, 264, 3), (32, 4112, 4),
                                        (64, 96, 5), (34, 1030, 1), (36, 1500, 2), (30, 514, 1)])
def test_mixed_accesses(bpc, H, W, levels):
    import torch
    rng = np.random.default_rng(W + levels)
    img = rng.integers(0, 256, size=(H, W)).astype(np.uint8)
    want = bpc_synth.dwt53(img, levels)
    d = torch.from_numpy(img.astype(np.int32) - 128).cuda()
    tmp = torch.full_like(d, 77)
    bpc.dwt53(d, levels, tmp=tmp)
    np.testing.assert_array_equal(d.cpu().numpy(), want)
    tmp.fill_(77)
    bpc.dwt53(d, levels, inverse=True, tmp=tmp)
    np.testing.assert_array_equal(d.cpu().numpy() + 128, img)
