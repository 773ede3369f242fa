"""The clustering's last rounds in one block (from 4096 clusters) at the sizes around its limits, against the
same clustering in numpy: the tree's boxes, triangles, child orders and miss links, all exact."""
import numpy as np
import pytest

import glslppm_gb300 as g
from glslppm_gb300.renderer import MATERIAL_DTYPE

pytestmark = pytest.mark.gpu
F = np.float32
RADIUS = 16


def expand(v):
    v = v.astype(np.uint32)
    for m, k in ((0x00010001, 0xFF0000FF), (0x00000101, 0x0F00F00F), (0x00000011, 0xC30C30C3), (0x00000005, 0x49249249)):
        v = (v * np.uint32(m)) & np.uint32(k)
    return v


def clustering(pos):
    """left, right, box, size of every node; leaves are n-1+k in Morton order; the root; the order."""
    n = len(pos)
    mn, mx = pos.min(1), pos.max(1)
    cen = ((pos[:, 0] + pos[:, 1]) + pos[:, 2]) * (F(1) / F(3))
    lo, hi = mn.min(0), mx.max(0)
    inv = np.where(hi > lo, F(1) / np.where(hi > lo, hi - lo, F(1)), F(0)).astype(F)
    x = np.clip((cen - lo) * inv, F(0), F(1))
    c = np.minimum((x * F(1024)).astype(np.uint32), 1023)
    code = (expand(c[:, 0]) << 2) | (expand(c[:, 1]) << 1) | expand(c[:, 2])
    order = np.argsort(code, kind="stable")
    box = np.zeros((2 * n - 1, 6), F)
    size = np.ones(2 * n - 1, np.int64)
    kids = np.full((2 * n - 1, 2), -1, np.int64)
    box[n - 1:, :3], box[n - 1:, 3:] = mn[order], mx[order]
    clu, nxt = np.arange(n - 1, 2 * n - 1), 0
    while len(clu) > 1:
        b, m = box[clu], len(clu)
        best, near = np.full(m, np.inf, F), np.full(m, -1)
        for d in [*range(-RADIUS, 0), *range(1, RADIUS + 1)]:  # ascending positions
            i = np.arange(max(0, -d), min(m, m - d))
            if not len(i):
                continue
            j = i + d
            e = np.maximum(b[i, 3:], b[j, 3:]) - np.minimum(b[i, :3], b[j, :3])
            a = (e[:, 0] * e[:, 1] + e[:, 1] * e[:, 2]) + e[:, 2] * e[:, 0]
            take = (near[i] < 0) | (a < best[i])
            best[i[take]], near[i[take]] = a[take], j[take]
        mutual = near[near] == np.arange(m)
        first = mutual & (np.arange(m) < near)
        new = clu.copy()
        for i in np.flatnonzero(first):
            l, r = clu[i], clu[near[i]]
            kids[nxt] = l, r
            box[nxt, :3], box[nxt, 3:] = np.minimum(box[l, :3], box[r, :3]), np.maximum(box[l, 3:], box[r, 3:])
            size[nxt] = size[l] + size[r]
            new[i], nxt = nxt, nxt + 1
        clu = new[~mutual | first]
    return kids, box, size, int(clu[0]), order


@pytest.mark.parametrize("n", [1, 2, 3, 17, 33, 34, 1023, 1025, 4095, 4096, 4097, 6000])
def test_the_same_tree_as_the_clustering_in_numpy(n):
    rng = np.random.default_rng(n)
    pos = (rng.uniform(0, 1, (n, 1, 3)) + rng.uniform(-0.02, 0.02, (n, 3, 3))).astype(F)
    pos[n // 2:, :, 0] *= rng.choice([1, 0.1])
    mats = np.zeros(1, MATERIAL_DTYPE)
    a = g.Mesh.from_arrays(pos, np.zeros(n, np.int32), mats).build_bvh(gpu=True).arrays()
    kids, box, size, root, order = clustering(a.positions)
    # canonical preorder: the child with the smaller min.x first, the second where they are equal
    want_box, want_tri, want_miss = [], [], []
    stack = [root]
    while stack:
        x = stack.pop()
        q = len(want_box)
        want_box.append(box[x])
        leaf = x >= n - 1
        want_tri.append(order[x - (n - 1)] if leaf else -1)
        end = q + 2 * size[x] - 1
        want_miss.append(q + 1 if leaf else (end if end < 2 * n - 1 else -1))
        if not leaf:
            l, r = kids[x]
            f, s = (l, r) if box[l, 0] < box[r, 0] else (r, l)
            stack += [s, f]
    np.testing.assert_array_equal(a.node_triangle, want_tri)
    np.testing.assert_array_equal(a.node_bounds.view(np.uint32), np.array(want_box, F).view(np.uint32))
    np.testing.assert_array_equal(a.order_miss[0], want_miss)
