"""Every candidate tile shape of the 3-D kernel, pinned (TJ_TILE3D, the pair of CTAs
an SM by the suffix p), over boxes of all three size classes with ragged and
one-cell tiles, with and without walls: the name selects the kernel that the
configuration reports, and the final states are the same bits."""
import ctypes
import os

import numpy as np
import pytest

from tenjin_gb300 import cases
from tenjin_gb300.host import MIXED, TenjinGPU

pytestmark = pytest.mark.gpu
SHAPES = ["8x8x8", "8x8x4", "16x8x4", "16x4x4", "4x4x4", "8x8x4p", "16x4x4p"]


def _case(walls):
    c = cases.uneven_boxes_3d(nbox=9, seed=23, lo=5, hi=38, max_steps=5)
    for n in ((1, 5, 3), (17, 9, 5), (33, 2, 37), (38, 37, 36)):
        d = cases.uneven_boxes_3d(nbox=1, seed=sum(n), lo=38, hi=38).domains[0]
        prim = np.ascontiguousarray(d.prim[:, :n[2], :n[1], :n[0]])
        c.domains.append(cases.Domain(list(n), [k * 1e-3 for k in n], [[0, 0, 0, n[0] - 1, n[1] - 1, n[2] - 1]], prim))
    if walls:
        c.lo_bc, c.hi_bc = [1, 0, 1], [1, 1, 0]
    return c


def _run(c, shape):
    os.environ["TJ_TILE3D"] = shape
    try:
        g = TenjinGPU(c, MIXED)
        g.run(5, 1e300)
    finally:
        del os.environ["TJ_TILE3D"]
    buf = ctypes.create_string_buffer(2048)
    g.L.tj_kernel_config(g.h, buf, 2048)
    s = np.concatenate([g.state(q).ravel() for q in range(len(c.domains))])
    g.close()
    return s, buf.value.decode()


@pytest.mark.parametrize("walls", [0, 1])
def test_every_shape(walls):
    c = _case(walls)
    want = None
    for shape in SHAPES:
        s, cfg = _run(c, shape)
        assert cfg.count(f"tile {shape},") == 3, cfg  # small, medium and large boxes
        assert cfg.count("launch:") == 1 and f"{320 if shape.endswith('p') else 640} threads" in cfg, cfg
        want = s if want is None else want
        assert np.isfinite(s).all() and np.array_equal(s, want), shape
