"""The pipelined single-level kernels (csrc/trisk_pipe.cuh) where their tiling can
go wrong: levels narrower than a tile (n = 16, 32, run with the TMA kernels
forced), levels whose last tile is ragged (n = 64), layer counts around the
layer groups.  FP64 against the CPU oracle bit for bit; the FP32-flux variant
bit for bit against the untiled FP32-flux kernels, whose arithmetic it keeps."""
import numpy as np
import pytest

import oracle
from wavetrisk_hydrostatic_b200 import Grid, OceanParams
from wavetrisk_hydrostatic_b200.cases import bump_state
from wavetrisk_hydrostatic_b200.model import TriskModel

pytestmark = pytest.mark.gpu


def _run(monkeypatch, variant, g, nz, st, bits, steps):
    monkeypatch.setenv("WAVETRISK_TREND_KERNEL", variant)
    m = TriskModel(g, nz, st["topo"], OceanParams())
    m.upload(st)
    if bits == 32:
        m.flux_precision(32)
    trend = m.trend_ml()
    m.upload(st)
    m.rk4(150.0, steps)
    out = m.download()
    assert m.status() == 0
    m.close()
    return trend, out


@pytest.mark.parametrize("level,nz", [(4, 1), (4, 5), (5, 3), (6, 1), (6, 17), (7, 3)])
def test_fp64_pipeline_matches_oracle(level, nz, monkeypatch):
    g = Grid(level, level, radius=6371e3).level(level)
    st = bump_state(g, nz, seed=level + nz)
    (dm, dt, dv), out = _run(monkeypatch, "tma", g, nz, st, 64, 2)
    om, ot, ov, _ = oracle.trend(g, nz, OceanParams(), st)
    assert np.array_equal(dm, om) and np.array_equal(dt, ot) and np.array_equal(dv, ov)
    m, t, v = oracle.rk4(g, nz, OceanParams(), st, 150.0, 2)
    for a, b in ((out["mass"], m), (out["temp"], t), (out["velo"], v)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("level,nz", [(4, 3), (5, 8), (6, 9), (7, 2)])
def test_fp32_flux_pipeline_matches_untiled_kernels(level, nz, monkeypatch):
    g = Grid(level, level, radius=6371e3).level(level)
    st = bump_state(g, nz, seed=3 * level + nz)
    a = _run(monkeypatch, "tma", g, nz, st, 32, 2)
    b = _run(monkeypatch, "plain", g, nz, st, 32, 2)
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)
    for k in ("mass", "temp", "velo"):
        assert np.array_equal(a[1][k], b[1][k])
