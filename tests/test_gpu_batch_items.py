"""Codeblocks per work item of the batched form: the caller's number is what the
queue holds (pairs for 32x32 codeblocks, a short last item per image), and the
container and coefficients do not depend on it."""
import numpy as np
import pytest

import bpc_synth
from conftest import lut_folder

pytestmark = pytest.mark.gpu

IMAGES = [  # X, Y, levels, passes, cb: 64, 15, 96, 15 and 77 codeblocks
    (512, 512, 5, 3, 64),
    (320, 192, 4, 2, 64),
    (256, 384, 3, 2, 32),
    (160, 96, 3, 3, 32),
    (704, 448, 4, 3, 64),
]


@pytest.fixture(scope="module")
def setup(bpc, oracle_mod):
    import torch
    imgs, words = [], []
    for k, (X, Y, lv, ps, cb) in enumerate(IMAGES):
        img = bpc_synth.synthetic_coefficients(max(X, Y), lv, 70 + k, amp=30) if X == Y else \
            bpc_synth.laplacian_coefficients(max(X, Y), lv, 70 + k)[:Y, :X]
        img = np.ascontiguousarray(img)
        lut = oracle_mod.load_luts(lut_folder(ps), ps, lv)
        words += bpc.slots_to_compact(oracle_mod.encode(img, lut, ps, lv, cb), cb)
        imgs.append(torch.from_numpy(img).cuda())
    return imgs, words


def count(per):
    n = 0
    for X, Y, _, _, cb in IMAGES:
        ncb = (X // cb) * (Y // cb)
        step = per if cb == 64 else (per + 1) // 2 * 2
        n += -(-ncb // step)
    return n


def test_default_is_one(bpc):
    b = bpc.Batch(IMAGES, {2: lut_folder(2), 3: lut_folder(3)})
    assert b.schedule()[2] == 1 and b.items() == count(1)
    b.close()


@pytest.mark.parametrize("per", [1, 2, 3, 4, 8, 64])
@pytest.mark.parametrize("warps,cost", [(4, False), (2, True)])
def test_items_of_the_callers_length(bpc, setup, per, warps, cost):
    import torch
    imgs, words = setup
    b = bpc.Batch(IMAGES, {2: lut_folder(2), 3: lut_folder(3)})
    b.set_tuning(warps, warps, cost, cost)
    b.set_schedule(2, 3, per)
    assert b.schedule() == (2, 3, per, True)
    assert b.items() == count(per)
    compact = torch.full((b.words,), 777, dtype=torch.int32, device="cuda")
    offs = torch.zeros(b.codeblocks + 1, dtype=torch.int64, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    b.encode(imgs, compact, offs, st)
    out = [torch.full_like(t, 0x7F7F7F7F) for t in imgs]
    b.decode(compact, offs, out, st)
    o, c = offs.cpu().numpy(), compact.cpu().numpy()
    assert len(words) == b.codeblocks and st.item() == 0
    for g, w in enumerate(words):
        np.testing.assert_array_equal(c[o[g]:o[g + 1]], w, err_msg=f"codeblock {g}")
    for t, i in zip(out, imgs):
        assert torch.equal(t, i)
    b.close()
