"""A run after the EOS parameters of a context changed (tj_forward and tj_tangent take
them): groups of 20 steps are captured, and must not run with the parameters that
they were captured with. Against a context made with the new ones, bit for bit."""
import dataclasses

import numpy as np
import pytest

from tenjin_gb300 import cases
from tenjin_gb300.adjoint import AdjointRun
from tenjin_gb300.host import FP64, TenjinGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("by", ["forward", "tangent"])
def test_run_with_new_parameters(by):
    torch = pytest.importorskip("torch")
    c = cases.shock_bubble_2d(n=24, max_grid_size=24, thinc=0, max_steps=45)
    r = AdjointRun(c)
    r.sim.set_primitive(0, c.domains[0].prim)
    r.sim.run(40, 1e300)  # captured
    d = cases.shock_bubble_2d(n=24, max_grid_size=24, thinc=0, max_steps=45)
    d.materials = [dataclasses.replace(m, params=list(m.params)) for m in d.materials]
    d.materials[1].params[0] = 1.6
    eos = AdjointRun(d).eos_array()
    prim = torch.from_numpy(np.ascontiguousarray(c.domains[0].prim)).cuda()
    dts = np.full(2, 1e-8)
    if by == "forward":
        r.forward(prim, eos, dts, 1)
    else:
        r.tangent(prim, torch.zeros_like(prim), eos, None, dts)
    r.sim._check(r.sim.L.tj_set_time(r.sim.h, 0.0, 0))
    r.sim.set_primitive(0, c.domains[0].prim)
    r.sim.run(45, 1e300)
    g = TenjinGPU(d, FP64)
    g.run(45, 1e300)
    assert np.array_equal(r.sim.state(0), g.state(0))
    g.close()
