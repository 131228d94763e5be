"""The fused binary32 kernels at the sizes where their launch changes: 2-D grids
whose tile count picks the CTA width (up to one tile an SM, up to two, more;
28-cell tiles), and 3-D boxes whose tiles are one cell thin, full or ragged
(the divisions of the tile lists are multiplications). Density against the
binary64 kernels on the same input: a few steps of about a hundred binary32
roundings of 6e-8 each, so at most 1e-5 in the relative L1 norm."""
import numpy as np
import pytest

from tenjin_gb300 import cases
from tenjin_gb300.host import FP64, FUSED64, MIXED, TenjinGPU

TOL = 1e-5


def test_div3_is_exact_over_the_tile_lists():
    t = np.arange(2048, dtype=np.uint32)
    for d in range(1, 241):
        f = np.uint32(((1 << 20) + d - 1) // d)
        assert np.array_equal((t * f) >> np.uint32(20), t // np.uint32(d)), d


def _rect(nx, ny, thinc, steps):
    """The shock-bubble problem cut to nx x ny cells."""
    n = max(nx, ny)
    c = cases.shock_bubble_2d(n=n, max_grid_size=64, max_steps=steps, thinc=thinc)
    nn = [nx, ny, 1]
    prim = np.ascontiguousarray(c.domains[0].prim[:, :, :ny, :nx])
    c.domains = [cases.Domain(nn, [nx / n, ny / n, 1.0], cases.max_size_boxes(nn, 2, 64), prim)]
    return c


def _density(c, precision):
    g = TenjinGPU(c, precision)
    g.run(c.max_steps, c.final_t)
    r = np.concatenate([g.density(q).ravel() for q in range(len(c.domains))])
    g.close()
    return r


def _close(c, precision):
    ref = _density(c, precision)
    got = _density(c, MIXED)
    assert np.isfinite(got).all()
    assert np.abs(got - ref).sum() <= TOL * np.abs(ref).sum()


@pytest.mark.gpu
@pytest.mark.parametrize("thinc", [0, 1])
@pytest.mark.parametrize("nx,ny", [(5, 27), (28, 29), (224, 532), (476, 252), (448, 532), (140, 1708), (141, 1709)])
def test_fused_2d_tile_counts(nx, ny, thinc):
    _close(_rect(nx, ny, thinc, 6), FUSED64)


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [0, 1])
@pytest.mark.parametrize("n", [(4, 4, 4), (1, 5, 3), (16, 8, 4), (17, 9, 5), (33, 3, 2), (15, 31, 7), (64, 2, 9)])
def test_fused_3d_box_edges(n, walls):
    c = cases.uneven_boxes_3d(nbox=1, lo=64, hi=64, max_steps=4)
    x0, y0, z0 = (32 - k // 2 for k in n)  # cut from the middle of the cube
    prim = np.ascontiguousarray(c.domains[0].prim[:, z0:z0 + n[2], y0:y0 + n[1], x0:x0 + n[0]])
    nn = list(n)
    c.domains = [cases.Domain(nn, [k * 1e-3 for k in nn], [[0, 0, 0, nn[0] - 1, nn[1] - 1, nn[2] - 1]], prim)]
    if walls:
        c.lo_bc, c.hi_bc = [1, 0, 1], [1, 1, 0]
    _close(c, FP64)
