"""Captured steps of the 3-D kernel after its tiles are chosen anew: the boxes
change, a run captures the launches that go with them, and the next upload tunes
the tiles, which replaces the work lists. The graph of the run before must not be
launched again. Against a context that never held another plan, bit for bit."""
import numpy as np
import pytest

from tenjin_gb300 import cases
from tenjin_gb300.host import MIXED, TenjinGPU

pytestmark = pytest.mark.gpu


def _states(g, c):
    return [g.state(q) for q in range(len(c.domains))]


def test_run_after_boxes_and_upload():
    c = cases.uneven_boxes_3d(nbox=5, seed=11, lo=6, hi=36, max_steps=60)
    g = TenjinGPU(c, MIXED)
    g.run(20, 1e300)
    for q in range(len(c.domains)):
        g._check(g.L.tj_set_max_grid_size(g.h, q, 8))
    g.run(20, 1e300)  # the plan of the new boxes, captured
    for q, d in enumerate(c.domains):
        g.set_primitive(q, d.prim)
    g._check(g.L.tj_set_time(g.h, 0.0, 0))
    done, t = g.run(20, 1e300)  # tuned by the upload
    got = _states(g, c)
    g.close()
    f = TenjinGPU(c, MIXED)
    for q in range(len(c.domains)):
        f._check(f.L.tj_set_max_grid_size(f.h, q, 8))
    want_done, want_t = f.run(20, 1e300)
    want = _states(f, c)
    f.close()
    assert (done, t) == (want_done, want_t)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
