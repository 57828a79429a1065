"""Edges of the coder's fast paths, against the oracle: the decoder's
sign-context hash, its eight-symbol groups of a codeblock without significant
coefficients (broken off at any symbol by a damaged stream), probabilities
outside 1..127, and rasters that are only 4-byte aligned."""
import os
import re

import numpy as np
import pytest

import bpc_synth
from conftest import PKG, lut_folder
from test_emu import emu, run  # noqa: F401


def test_sign_hash_is_perfect():
    """The 256 combinations of the eight neighbour bits give 256 table indices."""
    src = open(os.path.join(PKG, "csrc", "bpc_core.cuh")).read()
    m = re.search(r"kSignBits = (0x[0-9A-Fa-f]+)u, kSignHash = (0x[0-9A-Fa-f]+)u", src)
    bits, mul = int(m.group(1), 16), int(m.group(2), 16)
    pos = [i for i in range(32) if bits >> i & 1]
    assert len(pos) == 8 and mul % 2 == 0
    idx = set()
    for k in range(256):
        v = sum(1 << pos[i] for i in range(8) if k >> i & 1)
        left, right = (v * mul) & 0xFFFFFFFF, ((v << 1) * (mul >> 1)) & 0xFFFFFFFF
        assert left == right
        idx.add(left >> 24)
    assert len(idx) == 256


@pytest.mark.parametrize("passes", [2, 3])
@pytest.mark.parametrize("cb", [64, 32])
def test_damaged_zero_codeblocks(emu, oracle_mod, passes, cb):  # noqa: F811
    """Codeblocks marked all-zero (MSB 32) whose codewords are noise of many
    sizes: runs of zero symbols end at every position of the eight-symbol
    groups, and coefficients become significant in the middle of a plane."""
    lut = oracle_mod.load_luts(lut_folder(passes), passes, 5)
    rng = np.random.default_rng(7 * passes + cb)
    Y, X = 2 * cb, 4 * cb
    slots = np.full((Y // cb * (X // cb), cb * cb), -1, np.int32)
    for k, s in enumerate(slots):
        s[0] = 32
        n = int(rng.integers(1, cb * cb - 1))
        hi = 1 << int(rng.integers(0, 17))  # small codewords keep the zeros going
        s[1:1 + n] = np.where(rng.random(n) < 0.9, rng.integers(0, max(1, hi), n), rng.integers(0, 65536, n))
    want, wst = oracle_mod.decode(slots.reshape(-1), (Y, X), lut, passes, 5, cb, with_status=True)
    for kind in (0, 2):
        got, st = run(emu, 0, slots, (Y, X), lut, passes, 5, cb, kind=kind)
        np.testing.assert_array_equal(got.reshape(Y, X), want)
        assert st == int(np.bitwise_or.reduce(wst))


@pytest.mark.parametrize("passes", [2, 3])
@pytest.mark.parametrize("cb", [64, 32])
def test_zero_codeblocks(emu, oracle_mod, passes, cb):  # noqa: F811
    """All-zero codeblocks, inside one subband (all lanes' codewords end at the
    same symbol) and straddling several; with random probabilities the ends
    fall on every symbol of the eight-symbol groups."""
    z = np.zeros((cb, 2 * cb), np.int32)
    rng = np.random.default_rng(passes + cb)
    for levels in (1, 5):
        lut0 = oracle_mod.load_luts(lut_folder(passes), passes, levels)
        for lut in (lut0, rng.integers(1, 128, size=lut0.size).astype(np.int32),
                    rng.integers(100, 128, size=lut0.size).astype(np.int32)):
            want, wst = oracle_mod.encode(z, lut, passes, levels, cb, with_status=True)
            got, st = run(emu, 1, z, z.shape, lut, passes, levels, cb)
            np.testing.assert_array_equal(got, want)
            assert st == int(np.bitwise_or.reduce(wst))
            wdec = oracle_mod.decode(want, z.shape, lut, passes, levels, cb)
            for kind in (0, 2):
                dec, _ = run(emu, 0, want, z.shape, lut, passes, levels, cb, kind=kind)
                np.testing.assert_array_equal(dec.reshape(z.shape), wdec)


@pytest.mark.parametrize("passes,cb", [(2, 64), (3, 32)])
@pytest.mark.parametrize("lo,hi", [(0, 3), (126, 131), (200, 256)])
def test_unusual_probabilities(emu, oracle_mod, passes, cb, lo, hi):  # noqa: F811
    """Table entries 0 (a codeword per symbol) and 128..255 (intervals that
    grow): accepted, and coded like the oracle."""
    rng = np.random.default_rng(hi)
    lut = rng.integers(lo, hi, size=oracle_mod.load_luts(lut_folder(passes), passes, 5).size).astype(np.int32)
    img = bpc_synth.synthetic_coefficients(128, 5, 9, amp=30)
    img[:, 64:] = 0
    want, wst = oracle_mod.encode(img, lut, passes, 5, cb, with_status=True)
    wdec = oracle_mod.decode(want, img.shape, lut, passes, 5, cb)
    for kind in (0, 2, 3):
        got, st = run(emu, 1, img, img.shape, lut, passes, 5, cb, kind=kind)
        np.testing.assert_array_equal(got, want)
        assert st == int(np.bitwise_or.reduce(wst))
        dec, _ = run(emu, 0, want, img.shape, lut, passes, 5, cb, kind=kind)
        np.testing.assert_array_equal(dec.reshape(img.shape), wdec)


@pytest.mark.parametrize("passes", [2, 3])
@pytest.mark.parametrize("cb", [64, 32])
def test_magnitudes_out_of_range(emu, oracle_mod, passes, cb):  # noqa: F811
    """|x| >= 2^28 (MSB 28..31) is flagged and its codeblock marked with that
    plane; the other codeblocks are coded as ever."""
    img = bpc_synth.synthetic_coefficients(128, 5, 9, amp=30)
    lut = oracle_mod.load_luts(lut_folder(passes), passes, 5)
    want = oracle_mod.encode(img, lut, passes, 5, cb).reshape(-1, cb * cb)
    bad = {}
    for y, x, v in ((3, 5, 1 << 28), (70, 3, -(1 << 30)), (90, 100, -(1 << 31))):
        img[y, x] = v
        bad[y // cb * (128 // cb) + x // cb] = abs(v).bit_length() - 1
    for kind in (0, 2, 3):
        got, st = run(emu, 1, img, img.shape, lut, passes, 5, cb, kind=kind)
        got = got.reshape(-1, cb * cb)
        assert st == 4
        assert {k: int(got[k, 0]) for k in bad} == bad
        rest = [k for k in range(len(got)) if k not in bad]
        np.testing.assert_array_equal(got[rest], want[rest])


@pytest.mark.gpu
@pytest.mark.parametrize("cb", [64, 32])
def test_decode_into_4_byte_aligned_raster(bpc, cb):
    import torch
    img = bpc_synth.synthetic_coefficients(256, 5, 9, amp=30)
    lut = bpc.DeviceLut(lut_folder(3), 3, 5)
    d = torch.from_numpy(img).cuda()
    s = torch.empty(img.size, dtype=torch.int32, device="cuda")
    bpc.encode_device(d, s, lut, cb)
    buf = torch.full((img.size + 2,), 777, dtype=torch.int32, device="cuda")
    out = buf[1:-1].view(img.shape)
    assert out.data_ptr() % 8 == 4
    bpc.decode_device(s, out, lut, cb)
    np.testing.assert_array_equal(out.cpu().numpy(), img)
    assert buf[0].item() == 777 and buf[-1].item() == 777
