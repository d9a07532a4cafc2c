"""abd_ee_pairs_static on lists that its kernels take by different routes:
few and many partners per edge (lists in shared memory, more partners than a
list holds, more pairs than the pool of lists holds), one to a few cells per
query, edges that share vertices and non-finite vertices.  The oracle is every
pair of edges, with the segment distance in float32.  Pair lists are whole
numbers: they must match exactly."""
import ctypes as C

import numpy as np
import pytest

from colb_b200.engine import load_library

pytestmark = pytest.mark.gpu


def _brute(x, edges, cand):
    """All pairs i < j without a common vertex closer than cand; the inputs keep every distance away from cand."""
    p, q = x[edges[:, 0]].astype(np.float32), x[edges[:, 1]].astype(np.float32)
    out = []
    for i in range(len(edges) - 1):
        d1, d2, r = q[i] - p[i], q[i + 1:] - p[i + 1:], p[i] - p[i + 1:]
        a, e, f, c, b = d1 @ d1, (d2 * d2).sum(1), (d2 * r).sum(1), r @ d1, d2 @ d1
        den = a * e - b * b
        with np.errstate(all="ignore"):
            s = np.where(den != 0, np.clip((b * f - c * e) / den, 0, 1), 0)
            t = (b * s + f) / e
            s = np.where(t < 0, np.clip(-c / a, 0, 1), np.where(t > 1, np.clip((b - c) / a, 0, 1), s))
            t = np.clip(t, 0, 1)
            d = np.linalg.norm(r + s[:, None] * d1 - t[:, None] * d2, axis=1)
            ok = d < cand
        share = (edges[i + 1:, :, None] == edges[i][None, None, :]).any((1, 2))
        for j in np.flatnonzero(ok & ~share):
            out.append([*edges[i], *edges[i + 1 + j]])
    return np.array(out, dtype=np.int32).reshape(-1, 4)


def _run(x, edges, cand, cap):
    import torch
    L = load_library()
    xd, ed = torch.from_numpy(x).cuda(), torch.from_numpy(edges).cuda()
    out = torch.full((cap + 8, 4), -7, dtype=torch.int32, device="cuda")
    n = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    rc = L.abd_ee_pairs_static(p(xd), p(ed), len(x), len(edges), cand, p(out), cap, p(n), None)
    assert rc == 0, L.abd_last_error(None)
    return int(n.item()), out.cpu().numpy()


# parallel segments along z at integer places of a plane, in random order: distances are whole
# square roots, and cand lies between two of them
@pytest.mark.parametrize("ne,cand,vertical", [(2, 1.2, False), (31, 1.2, False), (33, 1.2, True), (257, 2.1, False),
                                              (700, 5.05, False), (700, 7.02, True), (2000, 1.2, False), (1700, 40.006, False)])
def test_static_pairs_equal_all_pairs(ne, cand, vertical):
    rng = np.random.default_rng(ne)
    side = int(np.ceil(np.sqrt(ne)))
    at = rng.permutation(side * side)[:ne]
    x = np.zeros((2 * ne, 3))
    x[0::2, 0], x[0::2, 1] = at // side - side // 2, at % side - side // 2
    x[1::2] = x[0::2]
    x[1::2, 2] += 0.5 if vertical else 1.0
    edges = np.arange(2 * ne, dtype=np.int32).reshape(ne, 2)
    if vertical:
        # polylines: edges that share a vertex are no pair
        edges[1::2, 0] = edges[0::2, 1][:len(edges[1::2])]
    want = _brute(x, edges, cand)
    cap = len(want) + 3
    n, rows = _run(x, edges, cand, cap)
    assert n == len(want)
    assert np.array_equal(rows[:n], want)
    assert np.all(rows[n:] == -7)


def test_static_pairs_more_pairs_than_the_lists_hold():
    """Enough edges with 40 to 90 partners each that their lists outgrow the pool: 30,000
    parallel segments on a line, 1/64 apart, closer than 0.68 to the 43 (+ 43) nearest."""
    ne, near = 30000, 43
    x = np.zeros((2 * ne, 3))
    x[0::2, 0] = x[1::2, 0] = np.arange(ne) / 64
    x[1::2, 2] = 1.0
    edges = np.arange(2 * ne, dtype=np.int32).reshape(ne, 2)
    i = np.repeat(np.arange(ne), near)
    j = i + np.tile(np.arange(1, near + 1), ne)
    i, j = i[j < ne], j[j < ne]
    want = np.concatenate([edges[i], edges[j]], axis=1)
    assert len(want) > 1 << 20
    n, rows = _run(x, edges, (near + 0.5) / 64, len(want))
    assert n == len(want)
    assert np.array_equal(rows[:n], want)


def test_static_pairs_ignore_non_finite_vertices():
    x = np.zeros((8, 3))
    x[0::2, 0] = x[1::2, 0] = np.arange(4)
    x[1::2, 2] = 1.0
    x[5, 1] = np.nan
    edges = np.arange(8, dtype=np.int32).reshape(4, 2)
    n, rows = _run(x, edges, 1.2, 8)
    assert n == 1 and rows[0].tolist() == [0, 1, 2, 3]
