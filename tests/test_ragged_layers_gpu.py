"""Layer counts that leave a short last group in the kernels that take several layers
at a time: the scalar restriction (4), the flux restriction (8 rows a block, one flux
or two), the columns (8) and the velocity trend (groups of up to 8, over work lists
of 2 or 4), on hierarchies against the CPU oracle, bit for bit (FP64 without FMA
contraction, the oracle's operand order)."""
import numpy as np
import pytest
import test_restrict_gpu
import test_trend_multi_gpu

import oracle
from oracle.wavelet import Hierarchy
from wavetrisk_hydrostatic_b200 import Grid, OceanParams, jet_state
from wavetrisk_hydrostatic_b200.grid import halo_edges
from wavetrisk_hydrostatic_b200.model import WaveletHierarchy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [5, 9])
def test_restrictions(nz):
    test_restrict_gpu.test_restrictions_match_oracle(3, 5, nz, True)


@pytest.mark.parametrize("nz,masks", [(5, "random"), (9, "built"), (13, "tolrnz")])
def test_trend(nz, masks):
    test_trend_multi_gpu.test_trend_multi_matches_oracle(4, 6, nz, masks)


# J6's list (46240 slots) takes groups of 4 layers at 5 and 13 layers, J5's groups of 2 at 13
@pytest.mark.parametrize("nz,kept", [(5, "all"), (13, "all"), (13, "adapted")])
def test_rk4_over_work_lists(nz, kept):
    ph = OceanParams()
    lmin, lmax, dt = 4, 6, 300.0
    G = Grid(lmin, lmax, radius=6371e3)
    levels = [G.level(l) for l in range(lmin, lmax + 1)]
    top = jet_state(levels[-1], nz, seed=3, ph=ph)
    top["velo"] = top["velo"] + 0.05 * np.random.default_rng(4).standard_normal(top["velo"].shape)
    halo_edges(levels[-1], top["velo"])
    orc = Hierarchy(levels, nz)
    names = (("mass", "s_m"), ("temp", "s_t"), ("velo", "s_v"))
    for name, key in names:
        orc.set(lmax, key, top[name])
    orc.forward()
    if kept == "all":
        masks = [(np.full(g.NN, 16, np.int32), np.full(3 * g.NN, 16, np.int32)) for g in levels]
    else:
        thr = np.full((3, nz), 0.12)
        thr[0] = 5.0
        orc.mask_build(thr, 0, lmax + 1)
        masks = [(orc.field(g.level, "mask_n").copy(), orc.field(g.level, "mask_e").copy()) for g in levels]
    states = []
    for g in levels:
        st = jet_state(g, nz, seed=3, ph=ph)
        for name, key in names:
            st[name] = orc.field(g.level, key).copy()
        states.append(st)
    dev = WaveletHierarchy(levels, [st["topo"] for st in states], nz, ph)
    for g, st, (mn, me) in zip(levels, states, masks):
        for name in ("mass", "temp", "velo", "mean_m", "mean_t"):
            dev.upload(g.level, name, st[name])
        dev.upload(g.level, "mask_n", mn)
        dev.upload(g.level, "mask_e", me)
    ref = oracle.rk4_multi(levels, nz, ph, states, masks, dt, nsteps=1)
    dev.rk4_multi(dt, 1)
    for q, g in enumerate(levels):
        own = np.nonzero(g.owned)[0]
        e = np.concatenate([own, own + g.NN, own + 2 * g.NN])
        for name, o, k in (("mass", ref[q][0], own), ("temp", ref[q][1], own), ("velo", ref[q][2], e)):
            assert np.array_equal(dev.download(g.level, name)[:, k], o[:, k]), (g.level, name)
    assert dev.status() == 0
    dev.close()
