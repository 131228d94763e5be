"""The per-direction kernels without room for every direction's fluxes: where the
device refuses that array (TJ_FAIL_ALLOC names the allocation, tj_alloc.h), or a
later allocation needs its space, the context holds one direction's and updates
direction by direction. Final states against those of the one update per stage,
bit for bit in binary64; in binary32, where the sums of one update and of three may
be contracted differently, within their roundings."""
import ctypes
import os

import numpy as np
import pytest

from tenjin_gb300 import cases
from tenjin_gb300.host import FP64, MIXED, TenjinGPU

pytestmark = pytest.mark.gpu


def _with(c, **kw):
    for k, v in kw.items():
        setattr(c, k, v)
    return c


def _elastic(c):
    for d in c.domains:
        d.prim = np.ascontiguousarray(d.prim[:len(d.prim) - c.M])
    return _with(c, plastic=0)


CASES = {
    "bubble_thinc": lambda: cases.shock_bubble_2d(n=30, max_grid_size=12, max_steps=23),
    "bubble_muscl_radial": lambda: _with(cases.shock_bubble_2d(n=30, max_grid_size=12, thinc=0, max_steps=5), radial=1),
    "two_domains": lambda: cases.uneven_boxes_3d(nbox=2, seed=1, lo=4, hi=9, max_steps=4),
    "copper": lambda: cases.copper_plate_3d(n=9, max_grid_size=4, max_steps=4),
    "elastic": lambda: _elastic(cases.copper_plate_3d(n=7, max_grid_size=4, max_steps=4)),
    "solid_gas": lambda: cases.solid_mixture_3d(n=6, max_steps=3),
    "reactive": lambda: cases.reactive_charge(2, 24, thinc=1, max_steps=4),
}


def _config(g):
    buf = ctypes.create_string_buffer(512)
    g.L.tj_kernel_config(g.h, buf, 512)
    return buf.value.decode()


def _run(c, precision, fail=None):
    if fail:
        os.environ["TJ_FAIL_ALLOC"] = fail
    try:
        g = TenjinGPU(c, precision)
    finally:
        os.environ.pop("TJ_FAIL_ALLOC", None)
    cfg = _config(g)
    g.run(c.max_steps, 1e300)
    s = [g.state(q) for q in range(len(c.domains))]
    if precision == FP64:  # the average alone, and the stages one by one
        g.advance(1e-9)
        g.advance_stage(0, 1e-9)
        g.advance_stage(1, 1e-9)
        s += [g.state(q) for q in range(len(c.domains))]
    g.close()
    return s, cfg


@pytest.mark.parametrize("precision,name", [(FP64, n) for n in sorted(CASES)] + [(MIXED, "copper"), (MIXED, "elastic")])
def test_updates_per_direction(precision, name):
    from tenjin_gb300._lib import TjError
    c = CASES[name]()
    want, cfg = _run(c, precision)
    assert "per direction" not in cfg.replace("per-direction", "")
    seen = 0
    for n in range(1, 40):
        try:
            got, cfg = _run(c, precision, str(n))
        except TjError:
            continue  # an array that there is no way without
        if "updates per direction" not in cfg:
            break  # n is past the set-up
        seen += 1
        for a, b in zip(got, want):
            if precision == FP64:
                assert np.array_equal(a, b, equal_nan=True)
            else:  # partial densities, momentum along x, energy: 4 steps of 2 x 3 sums, each a few roundings of 6e-8
                for q in [*range(c.M, 2 * c.M), 3 * c.M + 1, 3 * c.M + 7]:
                    assert np.abs(a[q] - b[q]).max() <= 1e-5 * np.abs(b[q]).max(), q
    assert seen >= 2  # the array itself, and at least one after it
