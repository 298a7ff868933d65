"""dftgpu_run replays a captured step when it is called again with the same
arguments.  A public field that the caller sets between two such calls (target
norm, mass, propagator, a functional's parameters) takes effect in the second
one: its result is bit for bit that of the steps launched singly."""
import ctypes as C

import numpy as np
import pytest

from conftest import liquid_psi

pytestmark = pytest.mark.gpu


def set_byte(w, offset, value):
    C.cast(w.ptr, C.POINTER(C.c_ubyte))[offset] = value


CHANGES = {
    "none": lambda G, w, ot: None,
    "target norm": lambda G, w, ot: setattr(w, "norm_target", 1.25 * w.norm()),
    "mass": lambda G, w, ot: C.cast(w.ptr, C.POINTER(C.c_double)).__setitem__(1, 1.1 * G.HELIUM_MASS),
    "propagator": lambda G, w, ot: set_byte(w, 25, G.WF_2ND_ORDER_CN),   # after grid, mass, norm and the boundary byte
    "c3": lambda G, w, ot: setattr(ot.params, "c3", 1.1 * ot.params.c3),
    "backflow strength": lambda G, w, ot: setattr(ot.params, "c_bfpot", 0.5),
}


@pytest.mark.parametrize("change", CHANGES)
def test_fields_set_between_two_runs(gpu, monkeypatch, change):
    G, shape, step = gpu, (16, 18, 20), 0.8
    G.set_precision(G.FP64)
    out = {}
    for graph in (True, False):
        if graph:
            monkeypatch.delenv("DFTGPU_NO_GRAPH", raising=False)
        else:
            monkeypatch.setenv("DFTGPU_NO_GRAPH", "1")
        w, wp = G.Wf(shape, step), G.Wf(shape, step)
        ot = G.OT(G.DFT_OT_KC | G.DFT_OT_BACKFLOW, w)
        P = G.CGrid(shape, step)
        w.set(liquid_psi(shape, step, 3))
        w.norm_target = w.norm()
        mu0 = ot.bulk_chempot(0.0)
        ot.run(w, wp, P, None, mu0, 20.0 - 5.0j, 3, True)
        CHANGES[change](G, w, ot)
        ot.run(w, wp, P, None, mu0, 20.0 - 5.0j, 3, True)
        out[graph] = w.get()
        for o in (P, ot, wp, w):
            o.free()
    assert np.array_equal(out[True], out[False])
