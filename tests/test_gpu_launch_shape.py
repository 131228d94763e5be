"""The per-direction FP64 kernels at the sizes where their launch shape
changes (tj_fp64.cuh launch_shape: 32- or 64-thread blocks, four blocks an SM,
the grid's cap) and where a block or a warp ends: the 1-D shock tube (fluid
instances) and the plastic copper plate (plastic instances) against the oracle
port, bit for bit."""
import numpy as np
import pytest

from oracle import port
from tenjin_gb300 import cases
from tenjin_gb300.host import FP64, TenjinGPU, carried_components

pytestmark = pytest.mark.gpu


def _same(c):
    ref = port.run_port(c)
    g = TenjinGPU(c, FP64)
    done, _ = g.run(c.max_steps, c.final_t)
    assert done == len(ref["dts"])
    idx = carried_components(c)
    assert np.array_equal(g.state(0)[idx], ref["states"][0][idx])
    g.close()


@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 65, 1000, 38911, 38912, 38913])
def test_shock_tube(n):
    _same(cases.sod_1d(ncells=n, max_grid_size=max(2, n), max_steps=3))


@pytest.mark.parametrize("n", [2, 3, 7, 11])
def test_copper_plate(n):
    _same(cases.copper_plate_3d(n=n, max_grid_size=8, max_steps=2))
