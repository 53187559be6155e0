"""The wait-timeout path of the pipelined single-level kernels (csrc/trisk_pipe.cuh)
in both of their types, FP64 and FP32 fluxes: WT_TUNE_TEST_TMA_TIMEOUT has every
block declare more bytes than its first copies deliver, so its bounded waits give
up; the producer then retires the extra bytes, lets its copies land and returns.
The handle reports WT_ERR_TIMEOUT, stays usable, and after wt_clear_status the next
steps are bit-identical to clean ones."""
import numpy as np
import pytest

from wavetrisk_hydrostatic_b200 import Grid, OceanParams, jet_state
from wavetrisk_hydrostatic_b200.model import TriskModel

pytestmark = pytest.mark.gpu
WT_ERR_TIMEOUT = -6


@pytest.mark.parametrize("bits", [64, 32])
def test_timeout_is_reported_and_the_handle_recovers(bits):
    level, nz, dt = 6, 5, 300.0          # five layers: the pipelined kernels
    g = Grid(level, level, radius=6371e3).level(level)
    ph = OceanParams()
    st = jet_state(g, nz, seed=3, ph=ph)
    m = TriskModel(g, nz, st["topo"], ph)
    m.flux_precision(bits)
    m.upload(st)
    m.rk4(dt, 2)
    assert m.status() == 0
    clean = m.download()
    m.upload(st)
    m.test_tma_timeout(True)
    m.rk4(dt, 1)
    assert m.status() == WT_ERR_TIMEOUT
    m.test_tma_timeout(False)
    m.clear_status()
    m.upload(st)
    m.rk4(dt, 2)
    assert m.status() == 0
    again = m.download()
    for k in ("mass", "temp", "velo"):
        assert np.array_equal(again[k], clean[k]), k
    m.close()
