"""The FP64 path where values are next to the subnormal numbers, whose halves are
not exact: a shock tube whose fluid moves at multiples of the smallest subnormal
number (the tail that the scheme sends ahead of a wave decays to such values),
against the oracle port, bit for bit."""
import numpy as np
import pytest

from oracle import port
from tenjin_gb300 import cases
from tenjin_gb300.host import FP64, TenjinGPU, carried_components

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thinc", [0, 1])
@pytest.mark.parametrize("most", [3, 40, 10 ** 6])
def test_subnormal_velocities(most, thinc):
    c = cases.sod_1d(ncells=96, max_grid_size=32, max_steps=3)
    c.thinc = thinc
    rng = np.random.default_rng(most)
    for row in (4, 5, 6):
        c.domains[0].prim[row] = rng.integers(-most, most + 1, c.domains[0].prim[row].shape) * 5e-324
    ref = port.run_port(c)
    g = TenjinGPU(c, FP64)
    done, _ = g.run(c.max_steps, c.final_t)
    assert done == len(ref["dts"])
    idx = carried_components(c)
    got, want = g.state(0)[idx], ref["states"][0][idx]
    assert np.array_equal(got, want)
    tiny = np.abs(want)
    assert ((tiny > 0) & (tiny < 2.2250738585072014e-308)).any()
    g.close()
