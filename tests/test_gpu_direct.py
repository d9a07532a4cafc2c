"""Routes of the direct solver (needs a GPU): the wide band kernel, projected
components beyond any band, and components whose band solution failed its
check and are solved again on the pivoted paths."""
import numpy as np
import pytest

from oracle import oracle as O
from colb_b200 import params as P, scene as S
from colb_b200._abi import ABD_INJECT_BAND_CHECK
from colb_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _net(n, seed=3):
    return S.config2_chain_net(n=n, pitch=1.5 - 5e-4, seed=seed)


def _check_solve(e, sc, p, precision):
    """du against one dense solve of the oracle's system: the backward error of a stable factorization
    and the forward error it implies."""
    eps = 2.2e-16 if precision == 0 else 1.2e-7
    du, it = e.solve()
    g, H = O.OracleWorld(p, sc).assemble()
    ref = np.linalg.solve(H, g)
    n = len(g)
    assert it == 1
    assert np.abs(H @ du - g).max() <= 10 * n * eps * (np.abs(H).max() * np.abs(du).max() + np.abs(g).max())
    ev = np.abs(np.linalg.eigvalsh(H))
    assert np.abs(du - ref).max() <= max(1e-8, 10 * n * ev.max() / ev.min() * eps) * np.abs(ref).max()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,band", [(9, True), (11, True), (13, False)])
def test_projected_nets_by_bandwidth(n, band, precision):
    """Tight n x n nets: one component of body bandwidth n, on the wide band kernel (9, 11) or in cuSOLVER (13)."""
    sc = _net(n)
    p = P.config_params(linear_solver=2, hess_mode=1, precision=precision)
    e = Engine(p, sc)
    _check_solve(e, sc, p, precision)
    if precision == 0:
        rc, st = e.step(1)
        assert rc == 0 and st.unconverged == 0
        assert (st.comp_large == 0) == band and (st.comp_band > 0) == band and st.comp_small == 0 and st.krylov_fallbacks == 0


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [4, 5])
def test_failed_band_solutions_take_the_pivoted_paths(n, precision):
    """With every band solution declared failed (test hook), solves and steps are those of the pivoted paths: the
    shared-memory factorization up to 12 bodies, cuSOLVER above; the counters name each component once."""
    sc = _net(n, seed=2)
    kw = dict(dt=1.0 / 240.0, linear_solver=2, hess_mode=1)
    p = P.config_params(precision=precision, test_inject=ABD_INJECT_BAND_CHECK, **kw)
    _check_solve(Engine(p, sc), sc, p, precision)
    if precision and n > 4:
        return                                  # (first steps of larger mixed nets need not converge)
    e, plain = Engine(p, sc), Engine(P.config_params(precision=precision, **kw), sc)
    ref = Engine(P.config_params(**kw), sc)
    for _ in range(2):
        rc, st = e.step(1)
        rp, sp = plain.step(1)
        ref.step(1)
        assert rc == 0 and rp == 0 and st.unconverged == 0 and st.du_guard_hits == 0
        assert st.comp_band == 0 and st.comp_small + st.comp_large > 0 and (st.comp_large == 0) == (n == 4)
        assert sp.comp_band > 0 and sp.comp_small == 0 and sp.comp_large == 0     # no solution fails by itself
        # FP64: residuals below 1e-5 over masses of at least 400 leave 2.5e-8 per step; mixed: its usual tolerance
        x, xr = e.vertices(), ref.vertices()
        assert np.abs(x - xr).max() <= (1e-4 if precision else 1e-7) * np.abs(xr).max()
    assert e.count_intersections() == 0


@pytest.mark.parametrize("extra", [30, 1500])
def test_second_solves_by_block_pattern(extra):
    """The second solve reads the block pattern back from the device, as rows (30 more bodies) or as sorted keys
    (1,500 more): the increment of the first solve up to the rounding of two stable factorizations."""
    net = _net(5)
    p = dict(linear_solver=2, hess_mode=1)
    _, H = Engine(P.config_params(**p), net).assemble()
    d = [Engine(P.config_params(test_inject=inject, **p), [S.config5_pile(n=extra, seed=1), net]).solve()[0]
         for inject in (0, ABD_INJECT_BAND_CHECK)]
    assert np.all(np.isfinite(d[1]))
    d0, d1 = (v[-12 * 25:] for v in d)
    s = 1.0 / np.sqrt(np.diag(H))
    kappa = np.linalg.cond(H * s[:, None] * s)
    assert np.linalg.norm((d0 - d1) / s) <= 50 * 2.2e-16 * kappa * np.linalg.norm(d0 / s)
