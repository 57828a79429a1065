"""The DWT's strip kernels at their edges, against the numpy lifting: strips cut
off by the image's height, partial warps, rasters without 16-byte alignment, odd
and even level counts (details end in either buffer), every strip length."""
import numpy as np
import pytest

import bpc_synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,levels", [(70, 264, 1), (4, 256, 1), (62, 8, 1), (36, 500, 2), (96, 1928, 3),
                                        (1208, 2048, 3), (2416, 2080, 4), (5000, 8192, 2)])
@pytest.mark.parametrize("offset", [0, 1])
def test_strips(bpc, H, W, levels, offset):
    import torch
    if offset and H * W > 1 << 24:
        pytest.skip("alignment is covered by the small sizes")
    rng = np.random.default_rng(H * W + levels)
    img = rng.integers(0, 256, size=(H, W)).astype(np.uint8)
    want = bpc_synth.dwt53(img, levels)
    buf = torch.zeros(2, H * W + 2 * offset, dtype=torch.int32, device="cuda")
    d, tmp = (b[offset:offset + H * W].view(H, W) for b in buf)
    d.copy_(torch.from_numpy(img.astype(np.int32) - 128))
    bpc.dwt53(d, levels, tmp=tmp)
    np.testing.assert_array_equal(d.cpu().numpy(), want)
    tmp.fill_(77)
    bpc.dwt53(d, levels, inverse=True, tmp=tmp)
    np.testing.assert_array_equal(d.cpu().numpy() + 128, img)
    if offset:  # nothing written outside the rasters
        assert buf[:, 0].abs().max().item() == 0 and buf[:, -1].abs().max().item() == 0
