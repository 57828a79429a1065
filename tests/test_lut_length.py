"""A probability table longer than its mode's: the entries past the ones the coder
indexes are range-checked and take no shared memory, so every launch form codes
with it as with the table alone."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, lut_folder

# longer than the shared memory of an SM leaves for a table beside a 4-warp
# decoder's own state
LONG = 215040


@pytest.fixture(scope="module")
def table_bytes(tmp_path_factory):
    d = tmp_path_factory.mktemp("lut")
    src, out = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write('#include <cstddef>\n#include "bpc_core.cuh"\n'
                'extern "C" int table_bytes(int levels, int passes, int n) '
                '{ return bpc::lut_offsets(levels, passes, n).tab_n; }\n')
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "cuda_bpc-paco_b200", "csrc"), src, "-o", out])
    return ctypes.CDLL(out).table_bytes


@pytest.mark.parametrize("passes", [2, 3])
@pytest.mark.parametrize("levels", [1, 5, 16])
def test_kept_table_does_not_grow(table_bytes, levels, passes, bpc):
    own = bpc.lib().bpc_lut_entries(passes, levels, 15)
    kept = table_bytes(levels, passes, own)
    assert own <= kept <= 20480 and kept % 16 == 0
    assert table_bytes(levels, passes, LONG) == kept
    assert table_bytes(levels, passes, 1) == kept


class LongLut:
    """The committed table with entries of 64 behind it, on the device; `at`: the
    first int's distance from a 16-byte boundary."""

    def __init__(self, host, passes, levels, n, at=0, last=64):
        import torch
        a = np.full(at + n, 64, np.int32)
        a[at:at + host.size] = host
        a[-1] = last
        self.t = torch.from_numpy(a).cuda()
        self.ptr, self.n, self.passes, self.levels = self.t.data_ptr() + 4 * at, n, passes, levels


# one-warp CTAs, 4-warp CTAs (more than a wave), the isolated decode, 32x32
# codeblocks; an odd length, and a table without 16-byte alignment
@pytest.mark.gpu
@pytest.mark.parametrize("side,passes,cb,sched,n,at", [
    (512, 3, 64, False, LONG, 0), (512, 2, 32, False, LONG - 3, 1), (4224, 3, 64, False, LONG, 0),
    (4096, 3, 64, True, LONG, 0), (4096, 2, 64, True, LONG - 1, 1)])
def test_long_table(bpc, luts, side, passes, cb, sched, n, at):
    import torch
    import bpc_synth
    img = bpc_synth.synthetic_coefficients_gpu(side, 5, 5, amp=40.0, nrect=60)
    own = bpc.DeviceLut(lut_folder(passes), passes, 5)
    long_ = LongLut(luts(passes), passes, 5, n, at)
    work = bpc.sched_buffer(side, side, cb) if sched else None
    got = []
    for lut in (own, long_):
        s = torch.full((side * side,), 0x7F7F7F7F, dtype=torch.int32, device="cuda")
        out = torch.full((side, side), 0x7F7F7F7F, dtype=torch.int32, device="cuda")
        st = torch.zeros(2, dtype=torch.int32, device="cuda")
        bpc.encode_device(img, s, lut, cb, st[0:1], sched=work)
        bpc.decode_device(s, out, lut, cb, st[1:2], sched=work)
        got.append((s, out, st))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert torch.equal(got[0][1], img) or got[0][2][0].item() != 0
    bad = LongLut(luts(passes), passes, 5, n, at, last=256)
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    bpc.decode_device(got[0][0], out, bad, cb, st, sched=work)
    assert st.item() & 8 and torch.equal(out, got[0][1])
