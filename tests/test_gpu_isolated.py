"""Isolated decodes over their range of sizes, both pass counts: every codeblock
coded once (outputs start from a sentinel), the plain call's coefficients and
status, and the work order really planned."""
import numpy as np
import pytest

import bpc_synth
from conftest import lut_folder

pytestmark = pytest.mark.gpu


# 3,782 (just above nine tenths of a wave) to 8,281 codeblocks (just below two)
@pytest.mark.parametrize("X,Y", [(3904, 3968), (4096, 4096), (4608, 4224), (5824, 5824)])
@pytest.mark.parametrize("passes", [2, 3])
def test_isolated(bpc, X, Y, passes):
    import torch
    lut = bpc.DeviceLut(lut_folder(passes), passes, 5)
    img = bpc_synth.synthetic_coefficients_gpu(-(-max(X, Y) // 32) * 32, 5, 31, amp=60.0, nrect=100)
    img = img[:Y, :X].contiguous()
    stream = torch.empty(X * Y, dtype=torch.int32, device="cuda")
    st = torch.zeros(3, dtype=torch.int32, device="cuda")
    bpc.encode_device(img, stream, lut, 64, st[0:1])
    plain, out = (torch.full_like(img, 0x7F7F7F7F) for _ in range(2))
    bpc.decode_device(stream, plain, lut, 64, st[1:2])
    ncb = (X // 64) * (Y // 64)
    sched = torch.full_like(bpc.sched_buffer(X, Y, 64), -7)
    counts = torch.full((ncb,), -7, dtype=torch.int32, device="cuda")
    bpc.decode_device(stream, out, lut, 64, st[2:3], counts, sched=sched)
    assert torch.equal(out, plain) and st[1] == st[2]
    if st[0].item() == 0:
        assert torch.equal(out, img)
        assert torch.equal(counts, ((stream.view(ncb, -1) != -1).sum(1) - 1).int())
    s = sched.cpu().numpy()
    np.testing.assert_array_equal(np.sort(s[:ncb]), np.arange(ncb))
    assert s[2 * ncb] >= 0  # the bulk launch's queue counter
