"""Which decodes run one-warp CTAs: the rule on the CPU, at table depths whose
copies fill the shared memory of an SM sooner than its registers, and the
coefficients on the GPU on both sides of it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, lut_folder

SMS, SMEM = 148, 228 * 1024


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("forms")
    src, out = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write('#include <cstddef>\n#include "bpc_kernels.h"\nusing namespace bpc;\n'
                'extern "C" int one_warp(int passes, int cbs, int levels, int warps, int sms, int smem) {\n'
                '  const long long cta = lut_offsets(levels, passes, 1).tab_n + kSignTableBytes +\n'
                '    4 * (cbs == 64 ? Geo<64>::RING_WORDS : Geo<32>::RING_WORDS);\n'
                '  return one_warp_pays(passes, cbs, warps, (long long)sms * kMinCtasDec * kWarps,\n'
                '                       one_warp_resident(sms, smem, cta));\n}\n')
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", "/usr/local/cuda/include", "-I",
                           os.path.join(ROOT, "cuda_bpc-paco_b200", "csrc"), src, "-o", out])
    return ctypes.CDLL(out).one_warp


@pytest.mark.parametrize("passes,cb,levels,warps,want", [
    (3, 64, 5, 1, True), (3, 64, 5, 4096, True), (2, 64, 5, 4144, True), (3, 64, 5, 4145, False),
    (3, 64, 8, 3600, True), (3, 64, 8, 4096, False), (3, 64, 10, 3249, True), (3, 64, 10, 4096, False),
    (3, 64, 16, 2162, True), (3, 64, 16, 2916, False), (2, 64, 10, 4096, True), (2, 64, 16, 3600, True),
    (2, 64, 16, 4096, False), (2, 32, 5, 1036, True), (2, 32, 5, 1037, False), (2, 32, 4, 4050, False),
    (3, 32, 5, 512, True), (3, 32, 5, 2592, True), (3, 32, 5, 3200, False), (3, 32, 16, 1152, True),
    (3, 32, 16, 2048, False)])
def test_rule(rule, passes, cb, levels, warps, want):
    assert bool(rule(passes, cb, levels, warps, SMS, SMEM)) == want


def test_no_shared_memory_known(rule):
    """Device attributes that cannot be read leave the 4-warp form."""
    assert not rule(3, 64, 5, 1, 0, 0) and not rule(3, 64, 5, 1, SMS, 0)


def deep_table(base, passes, levels):
    """The 5-level table with level 5's groups repeated down to `levels`."""
    out, o = [], 0
    for n in (1, 9, 4) if passes == 2 else (1, 9, 4, 9, 4):
        s = base[o:o + 240 * n].reshape(240, n)
        o += 240 * n
        out += [s[45 * min(k, 4):45 * min(k, 4) + 45] for k in range(levels)] + [s[225:]]
    return np.concatenate([x.reshape(-1) for x in out]).astype(np.int32)


class Lut:
    def __init__(self, a, passes, levels):
        import torch
        self.t = torch.from_numpy(a).cuda()
        self.ptr, self.n, self.passes, self.levels = self.t.data_ptr(), a.size, passes, levels


@pytest.mark.gpu
@pytest.mark.parametrize("passes,cb,levels,X,Y", [
    (3, 64, 16, 3072, 3136), (3, 64, 16, 3136, 3136), (2, 64, 16, 4096, 3904), (3, 64, 5, 4096, 4160),
    (3, 32, 5, 2432, 2304), (3, 32, 5, 2432, 2432), (2, 32, 4, 608, 352), (2, 32, 5, 1472, 1440), (2, 32, 5, 1472, 1472)])
def test_both_sides_of_the_rule(bpc, luts, passes, cb, levels, X, Y):
    import torch
    import bpc_synth
    side = -(-max(X, Y) // 32) * 32
    img = bpc_synth.synthetic_coefficients_gpu(side, 5, 17, amp=30.0, nrect=60)[:Y, :X].contiguous()
    lut = Lut(deep_table(luts(passes), passes, levels), passes, levels)
    s = torch.empty(X * Y, dtype=torch.int32, device="cuda")
    st = torch.zeros(3, dtype=torch.int32, device="cuda")
    bpc.encode_device(img, s, lut, cb, st[0:1])
    a, b = (torch.full((Y, X), 0x7F7F7F7F, dtype=torch.int32, device="cuda") for _ in range(2))
    bpc.decode_device(s, a, lut, cb, st[1:2])
    bpc.decode_device(s, b, lut, cb, st[2:3], grid=1 << 20)  # 4-warp CTAs
    assert torch.equal(a, b) and st[1] == st[2]
    if st[0].item() == 0:
        assert torch.equal(a, img)
