"""Overlapped launches of the per-direction kernels (tj_path_inst.cu
path_launch: outside of captured graphs, grids of at most 608 blocks) around
that number of blocks and in a run that mixes captured and single steps: the
1-D shock tube against the oracle port, bit for bit."""
import numpy as np
import pytest

from oracle import port
from tenjin_gb300 import cases
from tenjin_gb300.host import FP64, TenjinGPU, carried_components

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps", [(19455, 2), (19456, 2), (19457, 2), (300, 25)])
def test_shock_tube(n, steps):
    c = cases.sod_1d(ncells=n, max_grid_size=n, max_steps=steps)
    ref = port.run_port(c)
    g = TenjinGPU(c, FP64)
    done, _ = g.run(c.max_steps, c.final_t)
    assert done == len(ref["dts"])
    idx = carried_components(c)
    assert np.array_equal(g.state(0)[idx], ref["states"][0][idx])
    g.close()
