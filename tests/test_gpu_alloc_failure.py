"""Every allocation of a run failing, alone or with all after it (TJ_FAIL_ALLOC,
tj_alloc.h): each call either does its work or returns an error and leaves the context so that the same
call, made again, does it; nothing is computed from buffers that are not there.
Final states against a run without a failure, bit for bit."""
import ctypes
import os

import numpy as np
import pytest

from tenjin_gb300 import _lib, cases
from tenjin_gb300.adjoint import AdjointRun
from tenjin_gb300.host import FP64, FUSED64, MIXED, TenjinGPU, make_params

pytestmark = pytest.mark.gpu
TJ_ERR_STATE = -7

CASES = {
    "bubble_fp64": (lambda: cases.shock_bubble_2d(n=24, max_grid_size=8, max_steps=22), FP64),
    "copper_fp64": (lambda: cases.copper_plate_3d(n=8, max_grid_size=4, max_steps=3), FP64),
    "bubble_mixed": (lambda: cases.shock_bubble_2d(n=24, max_grid_size=8, max_steps=22), MIXED),
    "bubble_fused64": (lambda: cases.shock_bubble_2d(n=24, max_grid_size=8, max_steps=3), FUSED64),
    "boxes_mixed": (lambda: cases.uneven_boxes_3d(nbox=6, seed=4, lo=5, hi=36, max_steps=22), MIXED),
    "copper_mixed": (lambda: cases.copper_plate_3d(n=8, max_grid_size=4, max_steps=3), MIXED),
    "solid_gas_mixed": (lambda: cases.solid_mixture_2d(n=12, max_steps=3), MIXED),
}


def _run(c, precision, fail):
    """The case's steps with the failing allocations that TJ_FAIL_ALLOC names
    (None: none) until a call returns an error; the final states, and whether one did."""
    L = _lib.load()
    g = TenjinGPU.__new__(TenjinGPU)
    g.L, g.case, g.precision, g.h = L, c, precision, ctypes.c_void_p()
    p = make_params(c, precision)
    assert L.tj_create(ctypes.byref(p), ctypes.byref(g.h)) == 0
    g.ncomp = L.tj_ncomp(g.h)
    nd = len(c.domains)
    nn = (ctypes.c_int * (3 * nd))(*[v for d in c.domains for v in d.n_cells])
    dl = (ctypes.c_double * (3 * nd))(*[v for d in c.domains for v in d.dim_l])

    def boxes(q, d):
        flat = [v for b in d.boxes for v in b]
        return L.tj_set_boxes(g.h, q, len(d.boxes), (ctypes.c_int * len(flat))(*flat))

    def raising(f):
        def call():
            try:
                f()
            except _lib.TjError as e:
                return e.code
            return 0
        return call

    calls = [lambda: L.tj_set_domains(g.h, nd, nn, dl)]
    calls += [lambda q=q, d=d: boxes(q, d) for q, d in enumerate(c.domains)]
    calls += [raising(lambda q=q, d=d: g.set_primitive(q, d.prim)) for q, d in enumerate(c.domains)]
    calls += [raising(lambda: g.run(c.max_steps, 1e300))]
    out = [None] * nd

    def read(q):
        out[q] = g.state(q)
    calls += [raising(lambda q=q: read(q)) for q in range(nd)]
    failed = False
    if fail:
        os.environ["TJ_FAIL_ALLOC"] = fail
    try:
        for k, call in enumerate(calls):
            if call() != 0:
                assert fail and not failed, f"call {k} failed without a failing allocation"
                failed = True
                del os.environ["TJ_FAIL_ALLOC"]
                if k == 0:
                    assert L.tj_step(g.h, 1e300) == TJ_ERR_STATE
                assert call() == 0, f"call {k} made again"
    finally:
        os.environ.pop("TJ_FAIL_ALLOC", None)
        g.close()
    return out, failed


@pytest.mark.parametrize("later", ["", "+"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_run(name, later):
    make, precision = CASES[name]
    c = make()
    want, failed = _run(c, precision, None)
    assert not failed
    errors = 0
    for n in range(1, 41):
        got, failed = _run(c, precision, f"{n}{later}")
        errors += failed
        for a, b in zip(got, want):
            assert np.array_equal(a, b, equal_nan=True), n
    assert errors >= 5  # allocations of the set-up, at least


@pytest.mark.parametrize("name", ["bubble", "copper"])
def test_adjoint(name):
    torch = pytest.importorskip("torch")
    c = (cases.shock_bubble_2d(n=16, max_grid_size=16, background=1e-3) if name == "bubble"
         else cases.copper_plate_3d(n=4, max_grid_size=4))
    r = AdjointRun(c)
    dts, eos = r.dt_schedule(3), r.eos_array()
    prim = torch.from_numpy(np.ascontiguousarray(c.domains[0].prim)).cuda()
    grad = torch.ones(r.shape_state, dtype=torch.float64).cuda()

    def calls():
        r.forward(prim, eos, dts, 2)
        p, e = r.backward(grad)
        return p.cpu().numpy(), np.asarray(e)
    # every allocation of the first call in turn: a failed forward leaves nothing to reverse
    errors = 0
    for n in range(1, 25):
        r = AdjointRun(c)
        os.environ["TJ_FAIL_ALLOC"] = f"{n}+"
        try:
            got = calls()
        except _lib.TjError:
            errors += 1
            del os.environ["TJ_FAIL_ALLOC"]
            try:  # nothing to reverse, or all of it
                r.backward(grad)
            except RuntimeError:
                pass
            got = calls()
        finally:
            os.environ.pop("TJ_FAIL_ALLOC", None)
        if n == 1:
            want = calls()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), n
    assert errors >= 5
