"""Overlapped launches of the per-direction kernels (grids of at most 608 blocks,
outside of graphs) against the same steps launched plainly (events around each
kernel switch the overlap off), bit for bit: 2-D and 3-D, binary64 and binary32,
at sizes on both sides of 608 blocks, where the cells', the faces' and the THINC
candidates' kernels of one stage fall on different sides."""
import numpy as np
import pytest

from tenjin_gb300 import cases
from tenjin_gb300.host import FP64, MIXED, TenjinGPU

pytestmark = pytest.mark.gpu


def _bubble(nx, ny, **kw):
    n = max(nx, ny)
    c = cases.shock_bubble_2d(n=n, max_grid_size=4096, background=1e-3, **kw)
    prim = np.ascontiguousarray(c.domains[0].prim[:, :, :ny, :nx])
    c.domains = [cases.Domain([nx, ny, 1], [nx / n, ny / n, 1.0], [[0, 0, 0, nx - 1, ny - 1, 0]], prim)]
    return c


def _two(c):
    d = cases.shock_bubble_2d(n=c.domains[0].n_cells[0], max_grid_size=4096, seed=3, background=1e-3)
    c.domains = c.domains + d.domains
    return c


CASES = {
    # 19456 = 608 x 32 cells, 38912 = 608 x 64, 77824 = 608 x 128
    "fp64_2d_139": (lambda: _bubble(139, 139), FP64),
    "fp64_2d_128x152": (lambda: _bubble(128, 152), FP64),
    "fp64_2d_140": (lambda: _bubble(140, 140, thinc=0), FP64),
    "fp64_2d_152x256": (lambda: _bubble(152, 256), FP64),
    "fp64_3d_26": (lambda: cases.fluid_boxes_3d(n=26, max_grid_size=13), FP64),
    "fp64_copper_26": (lambda: cases.copper_plate_3d(n=26, max_grid_size=13), FP64),
    "fp64_copper_27": (lambda: cases.copper_plate_3d(n=27, max_grid_size=27), FP64),
    "mixed_copper_12": (lambda: cases.copper_plate_3d(n=12, max_grid_size=6), MIXED),
    "mixed_copper_26": (lambda: cases.copper_plate_3d(n=26, max_grid_size=13), MIXED),
    "mixed_copper_27": (lambda: cases.copper_plate_3d(n=27, max_grid_size=27), MIXED),
    "mixed_copper_42": (lambda: cases.copper_plate_3d(n=42, max_grid_size=42), MIXED),
    "mixed_two_domains": (lambda: _two(_bubble(98, 98)), MIXED),
    "mixed_fused_64": (lambda: _bubble(64, 64), MIXED),
    "mixed_boxes": (lambda: cases.uneven_boxes_3d(nbox=7, seed=2, lo=6, hi=36), MIXED),
}


def _run(c, precision, plain):
    g = TenjinGPU(c, precision)
    if plain:
        g._check(g.L.tj_set_profiling(g.h, 1))
    done, t = g.run(7, 1e300)
    s = np.concatenate([g.state(q).ravel() for q in range(len(c.domains))])
    g.close()
    assert done == 7 and np.isfinite(s).all()
    return s, t


@pytest.mark.parametrize("name", sorted(CASES))
def test_overlapped_equals_plain(name):
    make, precision = CASES[name]
    c = make()
    a, ta = _run(c, precision, False)
    b, tb = _run(c, precision, True)
    assert ta == tb and np.array_equal(a, b)
