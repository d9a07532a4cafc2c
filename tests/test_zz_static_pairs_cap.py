"""abd_ee_pairs_static with a capacity below the pair count: the rows are the
first ones of the complete list, the same on every call, also where the edge
that crosses the capacity has more partners than a list in shared memory holds
(needs a GPU)."""
import ctypes as C

import numpy as np
import pytest

from colb_b200._abi import ABD_ERR_CONTACT_OVERFLOW
from colb_b200.engine import load_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("near,caps", [(40, (1, 39, 41, 1000)), (300, (1, 7, 299, 300, 301, 450, 20000, 88000))])
def test_rows_below_the_capacity_are_the_first_of_the_list(near, caps):
    """Parallel segments on a line in random order, each closer than cand to its `near` neighbours on both sides."""
    import torch
    ne = 600
    rng = np.random.default_rng(near)
    place = rng.permutation(ne)
    x = np.zeros((2 * ne, 3))
    x[0::2, 0] = x[1::2, 0] = place / 64
    x[1::2, 2] = 1.0
    edges = np.arange(2 * ne, dtype=np.int32).reshape(ne, 2)
    i, j = np.triu_indices(ne, 1)
    ok = np.abs(place[i] - place[j]) <= near
    want = np.concatenate([edges[i[ok]], edges[j[ok]]], axis=1)
    L = load_library()
    xd, ed = torch.from_numpy(x).cuda(), torch.from_numpy(edges).cuda()
    p = lambda t: C.c_void_p(t.data_ptr())
    for cap in caps:
        assert cap < len(want)
        for _ in range(4):
            out = torch.full((cap + 8, 4), -7, dtype=torch.int32, device="cuda")
            n = torch.zeros(1, dtype=torch.int32, device="cuda")
            rc = L.abd_ee_pairs_static(p(xd), p(ed), len(x), ne, (near + 0.5) / 64, p(out), cap, p(n), None)
            assert rc == ABD_ERR_CONTACT_OVERFLOW and int(n.item()) == len(want)
            rows = out.cpu().numpy()
            assert np.array_equal(rows[:cap], want[:cap])
            assert (rows[cap:] == -7).all()
