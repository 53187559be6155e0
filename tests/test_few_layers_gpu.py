"""The single-level stepper on both sides of its rule for few layers: below three
layers FP64 runs the one-layer tiles (k_step1_tma, k_trend_tma) instead of the
pipelined ones, and FP32 fluxes run the L1 kernels where the tiles would not fill
eight rounds.  FP64 against the CPU oracle bit for bit; FP32 fluxes against the
untiled FP32 kernels bit for bit; and the kernels that ran, by name."""
import numpy as np
import pytest

import oracle
from wavetrisk_hydrostatic_b200 import Grid, OceanParams
from wavetrisk_hydrostatic_b200.cases import bump_state
from wavetrisk_hydrostatic_b200.model import TriskModel

pytestmark = pytest.mark.gpu


def _state(level, nz):
    g = Grid(level, level, radius=6371e3).level(level)
    return g, bump_state(g, nz, seed=5 * level + nz)


def _run(g, nz, st, bits):
    m = TriskModel(g, nz, st["topo"], OceanParams())
    m.upload(st)
    m.flux_precision(bits)
    trend = m.trend_ml()
    m.upload(st)
    m.rk4(150.0, 2)
    out = m.download()
    assert m.status() == 0
    m.close()
    return trend, out


@pytest.mark.parametrize("level,nz", [(6, 1), (6, 2), (6, 3), (7, 1), (7, 2)])
def test_fp64_matches_oracle(level, nz):
    g, st = _state(level, nz)
    (dm, dt, dv), out = _run(g, nz, st, 64)
    om, ot, ov, _ = oracle.trend(g, nz, OceanParams(), st)
    assert np.array_equal(dm, om) and np.array_equal(dt, ot) and np.array_equal(dv, ov)
    for a, b in zip((out["mass"], out["temp"], out["velo"]), oracle.rk4(g, nz, OceanParams(), st, 150.0, 2)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("level,nz", [(6, 2), (6, 3), (7, 1), (7, 2)])
def test_fp32_fluxes_match_untiled_kernels(level, nz, monkeypatch):
    g, st = _state(level, nz)
    a = _run(g, nz, st, 32)
    monkeypatch.setenv("WAVETRISK_TREND_KERNEL", "plain")
    b = _run(g, nz, st, 32)
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)
    for k in ("mass", "temp", "velo"):
        assert np.array_equal(a[1][k], b[1][k])


@pytest.mark.parametrize("level,nz,bits,kernel", [
    (6, 1, 64, "k_trend_tma"), (7, 2, 64, "k_trend_tma"), (7, 3, 64, "k_trend_pipe"),
    (7, 1, 32, "k_trend_mixed"), (7, 2, 32, "k_trend_pipe"), (6, 2, 32, "k_trend_mixed"), (6, 3, 32, "k_trend_pipe")])
def test_kernels_that_run(level, nz, bits, kernel):
    import torch
    from torch.profiler import ProfilerActivity, profile

    g, st = _state(level, nz)
    m = TriskModel(g, nz, st["topo"], OceanParams())
    m.upload(st)
    m.flux_precision(bits)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        m.trend_ml()
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages()]
    m.close()
    if not any("k_column" in n for n in names):
        pytest.skip("no kernel records on this machine")
    assert any(kernel in n for n in names), names
    assert sum("k_trend" in n for n in names) == 1, names
