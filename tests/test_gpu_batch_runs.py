"""A batch large enough for work items of several codeblocks (smaller ones use
one codeblock per item whatever the schedule asks for)."""
import pytest

from conftest import lut_folder

pytestmark = pytest.mark.gpu


def test_large_batch_in_runs(bpc):
    import torch
    X = Y = 16384
    images = [(X, Y, 3, 2, 32)] * 3  # 786,432 codeblocks: runs of two pairs' worth
    g = torch.Generator(device="cuda").manual_seed(3)
    img = torch.randint(-2, 3, (Y, X), generator=g, device="cuda", dtype=torch.int32)
    b = bpc.Batch(images, {2: lut_folder(2), 3: lut_folder(3)})
    compact = torch.empty(b.words, dtype=torch.int32, device="cuda")
    offs = torch.zeros(b.codeblocks + 1, dtype=torch.int64, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    b.encode([img] * 3, compact, offs, st)
    n = b.codeblocks // 3
    words = int(offs[n])
    for k in (1, 2):  # three times the same image: three times the same container
        assert torch.equal(offs[k * n:(k + 1) * n + 1] - offs[k * n], offs[:n + 1])
        assert torch.equal(compact[k * words:(k + 1) * words], compact[:words])
    plain = torch.empty(X * Y, dtype=torch.int32, device="cuda")
    lut = bpc.DeviceLut(lut_folder(2), 2, 3)
    bpc.encode_device(img, plain, lut, 32)
    for cb in (0, 1, n // 2, n - 2, n - 1):  # against the one-image call's slots
        o0, o1 = int(offs[cb]), int(offs[cb + 1])
        assert torch.equal(compact[o0:o1], plain[cb * 1024:cb * 1024 + o1 - o0])
    out = [torch.empty_like(img) for _ in range(3)]
    b.decode(compact, offs, out, st)
    for o in out:
        assert torch.equal(o, img)
    assert st.item() == 0
    b.close()
