"""The hash insertion where lanes of a warp have slots of their own, share them in groups, or share one:
winner (the smallest stored index that is not clipped) and count of every slot against numpy, whole
numbers; table sizes and array offsets around the four slots a thread clears."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300 import native as N, renderer

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def build(pos, flux, pw, ph, slots, flags, offset):
    dev = "cuda"
    p, f = torch.from_numpy(pos).to(dev), torch.from_numpy(flux).to(dev)
    w = torch.full((slots + 8,), 77, dtype=torch.int32, device=dev)
    c = torch.full((slots + 8,), 77, dtype=torch.int32, device=dev)
    renderer.hash_build(p.data_ptr(), f.data_ptr(), pw, ph, slots, (0.0, 0.0, 0.0), 1.0, flags,
                        w[offset:].data_ptr(), c[offset:].data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for a in (w, c):  # nothing outside the arrays
        assert bool((a[:offset] == 77).all()) and bool((a[offset + slots:] == 77).all())
    return w[offset:offset + slots].cpu().numpy(), c[offset:offset + slots].cpu().numpy()


@pytest.mark.parametrize("cells", [1, 2, 7, 31, 100000])
@pytest.mark.parametrize("pw,ph,slots,offset", [(1, 1, 1, 0), (33, 3, 5, 1), (64, 64, 4097, 0), (129, 65, 4098, 2),
                                                (256, 128, 100003, 3)])
@pytest.mark.parametrize("flags", [0, N.FLAG_GL_DEPTH_CLIP])
def test_groups_of_any_size(cells, pw, ph, slots, offset, flags):
    n = pw * ph
    rng = np.random.default_rng(cells + slots)
    cell = rng.integers(0, cells, n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, 0], pos[:, 1] = cell % 317 + 0.5, cell // 317 + 0.5
    flux = np.ones((n, 4), np.float32)
    flux[rng.random(n) < 0.2] = -1.0
    winner, count = build(pos, flux, pw, ph, slots, flags, offset)
    stored = np.nonzero(flux[:, 0] >= 0)[0]
    clipped = (stored >= (ph - 1) * pw + (pw + 1) // 2) & bool(flags)
    # the slot of each cell, from a table that holds one photon of that cell alone
    slot_of = {}
    for c in np.unique(cell[stored])[:24]:
        i = stored[cell[stored] == c][0]
        _, one = build(pos[i:i + 1].copy(), flux[i:i + 1].copy(), 1, 1, slots, 0, 0)
        slot_of[int(c)] = int(np.nonzero(one)[0][0])
    assert count.sum() == len(stored)
    if len(slot_of) == len(np.unique(cell[stored])):  # every cell's slot is known: the whole table
        s = np.array([slot_of[int(c)] for c in cell[stored]], np.int64)
        want_c = np.bincount(s, minlength=slots) if len(s) else np.zeros(slots, np.int64)
        want_w = np.full(slots, 0xFFFFFFFF, np.uint32)
        np.minimum.at(want_w, s[~clipped], stored[~clipped].astype(np.uint32))
        np.testing.assert_array_equal(count, want_c)
        np.testing.assert_array_equal(winner.view(np.uint32), want_w)
