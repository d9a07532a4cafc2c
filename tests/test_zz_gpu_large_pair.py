"""Two bodies whose primitives are numbered without order, so that every cluster
of one overlaps every cluster of the other: more cluster pairs than the body-pair
broad phase holds at once, from a single pair of bodies (needs a GPU)."""
import numpy as np
import pytest

from colb_b200 import params as P, scene as S
from colb_b200.engine import Engine

pytestmark = pytest.mark.gpu


def test_one_body_pair_with_more_cluster_pairs_than_the_list_holds():
    side, n = 72, 373000                       # 373,000 edges a body: 11,657 clusters, 1.36e8 pairs of them (2^27 held)
    assert (n // 32) ** 2 > 1 << 27
    rng = np.random.default_rng(1)
    cells = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(float)
    near = rng.permutation(n)[:40]             # edges of the second body 0.1 from one of the first; the others half a cell away
    xs, edges = [], []
    for body in range(2):
        at = cells[rng.permutation(len(cells))[:n]] if body == 0 else at0 + 0.5
        if body == 0:
            at0 = at
        else:
            at[near] = at0[near] + [0.0, 0.1, 0.0]
            order = rng.permutation(n)
            at = at[order]
        x = np.repeat(at, 2, axis=0)
        x[1::2, 0] += 0.1
        xs.append(x)
        edges.append(np.arange(2 * n).reshape(n, 2) + 2 * n * body)
    place = np.empty(n, dtype=np.int64)
    place[order] = np.arange(n)                # where edge k of the second body went
    i, j = near, n + place[near]
    ok = np.argsort(i)
    e = np.concatenate(edges).astype(np.int32)
    want = np.concatenate([e[i[ok]], e[j[ok]]], axis=1)
    sc = dict(xbar=np.concatenate(xs), vert_body=np.repeat(np.arange(2), 2 * n).astype(np.int32), edges=e,
              tris=np.zeros((0, 3), dtype=np.int32), mass=np.ones(2), inertia_J=np.ones(2),
              state=S.make_state(np.zeros((2, 3)), v=np.zeros((2, 3))), planes=np.zeros((0, 4)))
    eng = Engine(P.config_params(contact_pt=0, broadphase=2, cand_dist=0.2), sc)
    quads, kinds = eng.pairs(cap=4096)
    assert (kinds == 0).all()
    assert np.array_equal(quads, want)
