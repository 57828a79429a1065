"""The work order's kernels: every unit exactly once whatever the unit count's
remainder, heaviest first, and the streams and coefficients of the raster order."""
import numpy as np
import pytest

from conftest import lut_folder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,Y,cb,enc", [(5120, 4800, 64, True), (8704, 8704, 64, True), (4128, 2976, 32, True),
                                        (6144, 5760, 64, False), (5120, 5152, 32, False), (4096, 3968, 64, False)])
def test_order_is_a_permutation(bpc, X, Y, cb, enc):
    import torch
    lut = bpc.DeviceLut(lut_folder(2), 2, 5)
    g = torch.Generator(device="cuda").manual_seed(X + cb)
    img = torch.randint(-3, 4, (Y, X), generator=g, device="cuda", dtype=torch.int32)
    # codeblocks of different weight: whole rows of codeblocks scaled, some zero
    scale = torch.randint(0, 9, (Y // cb, X // cb), generator=g, device="cuda", dtype=torch.int32)
    img *= scale.repeat_interleave(cb, 0).repeat_interleave(cb, 1)
    raster, ordered = (torch.empty(X * Y, dtype=torch.int32, device="cuda") for _ in range(2))
    sched = torch.full((bpc.sched_buffer(X, Y, cb).numel() + 1,), 123456789, dtype=torch.int32, device="cuda")
    bpc.encode_device(img, raster, lut, cb)
    src = ordered if enc else raster
    if enc:
        bpc.encode_device(img, ordered, lut, cb, sched=sched[:-1])
        assert torch.equal(raster, ordered)
    else:
        # (some all-zero codeblocks overflow their slot, so not the input itself)
        plain, out = torch.empty_like(img), torch.empty_like(img)
        bpc.decode_device(raster, plain, lut, cb)
        bpc.decode_device(raster, out, lut, cb, sched=sched[:-1])
        assert torch.equal(out, plain)
    assert sched[-1].item() == 123456789
    ng = 1 if cb == 64 else 2
    ncb = (X // cb) * (Y // cb)
    units = (ncb + ng - 1) // ng
    order = sched[:units].cpu().numpy()
    np.testing.assert_array_equal(np.sort(order), np.arange(units) * ng)
    # heaviest first: the mean MSB plane of the first eighth is above that of the last
    msb = src.view(ncb, cb * cb)[:, 0].cpu().numpy()
    msb = np.where(msb == 32, 40, msb)
    w = np.array([msb[o:o + ng].mean() for o in order])
    assert w[:units // 8].mean() > w[-(units // 8):].mean()
