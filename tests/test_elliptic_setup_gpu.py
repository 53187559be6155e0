"""The solver's set-up (wt_elliptic_setup) waits for its own work only: another
stream's kernel, a bounded spin of about a second, is still running when it
returns, and the solver set up beside it solves as one set up alone."""
import numpy as np
import pytest

from wavetrisk_hydrostatic_b200 import Grid
from wavetrisk_hydrostatic_b200.cases import bathymetry, elliptic_rhs
from wavetrisk_hydrostatic_b200.model import EllipticSolver, solver_opts

pytestmark = pytest.mark.gpu


def test_setup_does_not_wait_for_other_streams():
    import torch

    G = Grid(4, 5, radius=6371e3)
    levels = [G.level(4), G.level(5)]
    topos = [bathymetry(lv, seed=3) for lv in levels]

    def solve(S):
        f = S.field()
        S.level_view(f, 1)[:] = elliptic_rhs(levels[1], seed=3)
        S.upload(u=S.field(), f=f)
        S.solve(solver_opts("mixed", 1e-10, coarse_iter=6))
        return S.download()[0]

    S = EllipticSolver(levels, topos)       # loads the set-up's kernels
    want = solve(S)
    side = torch.cuda.Stream()
    for attempt in range(3):                # an allocation can take longer than the spin on a busy host
        done = torch.cuda.Event()
        with torch.cuda.stream(side):
            torch.cuda._sleep(2_000_000_000)  # clock cycles: 1.0 s at 1965 MHz
            done.record(side)
        T = EllipticSolver(levels, topos)
        running = not done.query()
        side.synchronize()
        if running:
            break
        T.close()
    assert running
    assert np.array_equal(solve(T), want)
    S.close()
    T.close()
