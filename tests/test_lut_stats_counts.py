"""LUT training counts where codeblocks lie in one subband (counts summed over
their lanes) and where they straddle several (per lane), mixed in a warp of two
codeblocks, an odd number of codeblocks, planes above the tables', all-zero
codeblocks: against the oracle, on the CPU emulator and the GPU; and what the
counting costs against coding."""
import numpy as np
import pytest

import bpc_synth
from test_emu import emu, run  # noqa: F401  (fixture)


def image(Y, X, levels, kind):
    rng = np.random.default_rng(X * Y + levels)
    if kind == "planes":  # up to plane 17, above the tables' 15
        img = rng.integers(-(1 << 17), 1 << 17, size=(Y, X))
    else:
        img = bpc_synth.laplacian_coefficients(256, levels, 4)[:Y, :X].copy()
        img[:64, X // 2:] = 0
    return np.ascontiguousarray(img, dtype=np.int32)


CASES = [(64, 64, 5, "planes"), (128, 192, 1, "lap"), (192, 128, 2, "lap"), (64, 192, 6, "lap")]


@pytest.mark.parametrize("Y,X,levels,kind", CASES)
@pytest.mark.parametrize("passes,cb", [(2, 64), (3, 64), (2, 32), (3, 32)])
def test_counts_emulated(emu, oracle_mod, Y, X, levels, kind, passes, cb):  # noqa: F811
    img = image(Y, X, levels, kind)
    lut = np.full(oracle_mod.lut_entries(passes, levels), 64, np.int32)
    st = np.zeros(2 * lut.size, np.uint64)
    run(emu, 1, img, img.shape, lut, passes, levels, cb, kind=1, stats=st)
    np.testing.assert_array_equal(st, oracle_mod.lut_stats(img, passes, levels, cb))


@pytest.mark.gpu
@pytest.mark.parametrize("Y,X,levels,kind", CASES + [(96, 32, 2, "lap"), (32, 160, 1, "planes")])
@pytest.mark.parametrize("passes,cb", [(2, 64), (3, 64), (2, 32), (3, 32)])
def test_counts(bpc, oracle_mod, Y, X, levels, kind, passes, cb):
    import torch
    if Y % cb or X % cb:
        pytest.skip("not a multiple of the codeblock")
    img = image(Y, X, levels, kind)
    got = bpc.lut_stats(torch.from_numpy(img).cuda(), passes, levels, cb).cpu().numpy()
    np.testing.assert_array_equal(got, oracle_mod.lut_stats(img, passes, levels, cb))


@pytest.mark.gpu
@pytest.mark.parametrize("passes,cb", [(2, 64), (3, 64), (2, 32), (3, 32)])
def test_counting_costs_less_than_two_encodes(bpc, passes, cb):
    """A count is the encoder without its coder and its output; with a set of
    atomics per word and lane it took 4 to 7 times an encode (0.3 to 0.6 with one
    per codeblock)."""
    import torch
    from conftest import lut_folder
    img = bpc_synth.synthetic_coefficients_gpu(4096, 5, 12, amp=40.0, nrect=60)
    lut = bpc.DeviceLut(lut_folder(passes), passes, 5)
    s = torch.empty(img.numel(), dtype=torch.int32, device="cuda")
    stats = bpc.lut_stats(img, passes, 5, cb)

    def best(f):
        ts = []
        for _ in range(5):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            f()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return min(ts)

    enc = best(lambda: bpc.encode_device(img, s, lut, cb))
    cnt = best(lambda: bpc.lut_stats(img, passes, 5, cb, stats=stats))
    assert cnt < 2 * enc, (cnt, enc)
