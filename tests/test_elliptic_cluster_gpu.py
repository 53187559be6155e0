"""The elliptic solver's cluster kernels and fused passes at the sizes where they
change path: coarsest levels held by one cluster (J3: two CTAs, J4: six, J5:
eight) and the first one that is not (J6), V-cycle schedules around the fused
first sweeps.  Solutions against the CPU oracle's FMG; bound 1e-8: both sides
stop at a relative residual of 1e-10 and the operators' condition numbers are
below 100."""
import numpy as np
import pytest

from oracle.elliptic import Hierarchy
from wavetrisk_hydrostatic_b200 import Grid
from wavetrisk_hydrostatic_b200.cases import bathymetry, elliptic_rhs
from wavetrisk_hydrostatic_b200.model import EllipticSolver, solver_opts

pytestmark = pytest.mark.gpu
CASES = {}


def _case(lo, hi):
    if (lo, hi) not in CASES:
        G = Grid(lo, hi, radius=6371e3)
        levels = [G.level(l) for l in range(lo, hi + 1)]
        topos = [bathymetry(g, seed=3, nterms=24) for g in levels]
        H = Hierarchy(levels, topos, fine_tol=1e-11, coarse_tol=1e-11, max_vcycle=50, coarse_iter=300,
                      domain_level=G.domain_level)
        off = np.cumsum([0] + [g.NN for g in levels])
        f = np.zeros(off[-1])
        f[off[-2]:] = elliptic_rhs(levels[-1], seed=6)
        f = H.restrict_all(f)
        u, _, _ = H.solve(np.zeros(off[-1]), f, "fmg")
        CASES[lo, hi] = (G, levels, topos, off, f, u)
    return CASES[lo, hi]


def _owned(g, a):
    n = g.n
    return a.reshape(10, g.P, g.P)[:, 2:n + 2, 2:n + 2]


@pytest.mark.parametrize("lo,hi", [(3, 5), (4, 6), (5, 6), (6, 7)])
@pytest.mark.parametrize("method,kw", [
    ("fmg", {}), ("srj", dict(max_srj_iter=4000)), ("mixed", dict(down_iter=1, up_iter=1, coarse_iter=12)),
    ("mixed", dict(down_iter=3, up_iter=2, coarse_iter=7)), ("mg64", dict(down_iter=2, up_iter=2, coarse_iter=6)),
    ("mixed", dict(down_iter=2, up_iter=0, coarse_iter=8)), ("fcg_mg", dict(down_iter=2, up_iter=2, coarse_iter=6))])
def test_solutions(lo, hi, method, kw):
    G, levels, topos, off, f, want = _case(lo, hi)
    S = EllipticSolver(levels, topos, domain_level=G.domain_level)
    S.upload(u=np.zeros(off[-1]), f=f)
    kw = {"max_vcycle": 50, "coarse_iter": 300, "ir_max": 400, **kw}
    rep = S.solve(solver_opts(method, 1e-10, **kw))
    u, _ = S.download()
    S.close()
    assert rep.status == 0 and rep.true_rel_residual <= 1.01e-10
    a, b = _owned(levels[-1], u[off[-2]:]), _owned(levels[-1], want[off[-2]:])
    assert np.abs(a - b).max() <= 1e-8 * np.abs(b).max()


def test_zero_right_hand_side():
    G, levels, topos, off, _, _ = _case(4, 6)
    S = EllipticSolver(levels, topos, domain_level=G.domain_level)
    for method in ("mixed", "mg64"):
        S.upload(u=np.zeros(off[-1]), f=np.zeros(off[-1]))
        rep = S.solve(solver_opts(method, 1e-10, down_iter=2, up_iter=2, coarse_iter=6))
        assert rep.status == 0 and rep.outer_iterations == 0
        assert np.abs(S.download()[0]).max() == 0.0
    S.close()
