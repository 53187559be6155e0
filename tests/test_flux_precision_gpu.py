"""Switching the single-level stepper's fluxes to FP32 (WT_TUNE_FLUX_PRECISION) where
the switch itself can go wrong: at level 1, whose FP32 rows (6 values) no bulk tensor
copy can take, so that both kernel families run the untiled FP32 kernels there; and
where the device has no room for the FP32 arrays, after which the call must be
repeatable."""
import numpy as np
import pytest

from wavetrisk_hydrostatic_b200 import Grid, OceanParams, jet_state
from wavetrisk_hydrostatic_b200 import _native as N
from wavetrisk_hydrostatic_b200.model import TriskModel

pytestmark = pytest.mark.gpu


def _model(monkeypatch, variant, g, nz, seed=2):
    monkeypatch.setenv("WAVETRISK_TREND_KERNEL", variant)
    ph = OceanParams()
    st = jet_state(g, nz, seed=seed, ph=ph)
    m = TriskModel(g, nz, st["topo"], ph)
    m.upload(st)
    return m, st


def test_level_1_takes_fp32_fluxes_in_both_kernel_families(monkeypatch):
    g = Grid(2, 2, radius=6371e3, domain_level=0).level(1)
    assert g.P == 6
    m, st = _model(monkeypatch, "plain", g, 3)
    d64 = m.trend_ml()
    m.flux_precision(32)
    want = m.trend_ml()
    assert m.status() == 0
    m.close()
    # a flux is a product of three FP32 values and a mean of two: at most 8 roundings of 2^-24; six of them a node
    own = np.nonzero(g.owned)[0]
    flux = np.abs(st["velo"]).max() * g.pedlen.max() * np.abs(st["mass"] + st["mean_m"]).max()
    assert np.abs(want[0][:, own] - d64[0][:, own]).max() <= 48 * 2.0 ** -24 * flux * g.hex_inv[own].max()
    m, _ = _model(monkeypatch, "tma", g, 3)
    m.flux_precision(32)
    got = m.trend_ml()
    assert m.status() == 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    m.close()


def test_switch_that_finds_no_memory_can_be_repeated(monkeypatch):
    import torch

    level, nz, dt = 7, 16, 150.0
    g = Grid(level, level, radius=6371e3).level(level)
    m, st = _model(monkeypatch, "tma", g, nz)
    m.flux_precision(32)
    m.rk4(dt, 2)
    want = m.download()
    m.close()

    m, st = _model(monkeypatch, "tma", g, nz)
    m.rk4(dt, 1)
    assert m.status() == 0
    one = 3 * nz * g.NN * 4                      # bytes of an FP32 edge array; three of them and two of a third
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(free - 5 * one // 2, dtype=torch.uint8, device="cuda")  # two of the arrays fit
    with pytest.raises(N.WtError) as e:
        m.flux_precision(32)
    assert e.value.code == N.WT_ERR_ALLOC
    m.upload(st)
    m.rk4(dt, 1)                                 # still the FP64 stepper
    assert m.status() == 0
    del fill
    torch.cuda.empty_cache()
    m.flux_precision(32)
    m.upload(st)
    m.rk4(dt, 2)
    assert m.status() == 0
    got = m.download()
    for k in ("mass", "temp", "velo"):
        assert np.array_equal(got[k], want[k]), k
    m.close()
