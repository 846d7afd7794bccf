"""Calls at the ends of what the entry points take, and meshes that strain a
kernel's assumptions: results against the oracle, states and costs as for any
other call."""
import ctypes as C

import numpy as np
import pytest

import tioga_b200 as tb
from tests.compare import diff_runs
from tioga_b200 import cases
from tioga_b200.capi import TiogaLibrary, run_system

pytestmark = pytest.mark.gpu


def _connected(system, **registration):
    """The GPU library after a connectivity call on the system."""
    t = TiogaLibrary(tb.library_path())
    tb.extras(t.lib)
    t.init()
    t.register_system(system, **registration)
    t.preprocess_grids()
    t.performconnectivity()
    assert t.lib.tioga_b200_last_error() == 0
    return t


@pytest.mark.parametrize("side", ["host", "device"])
def test_update_of_no_fields(side, oracle_lib):
    """An update of zero fields changes nothing, one of a negative number is
    refused, and the next update is the oracle's."""
    import torch
    system = cases.small_config0(0)
    q0 = cases.fields(system, nvar=2, seed=4)
    ref = run_system(oracle_lib, system, q_blocks=q0, nvar=2)
    t = _connected(system)
    assert tb.stats(t.lib)["nrecords"] > 0
    q = [torch.from_numpy(a.copy()).to("cuda" if side == "device" else "cpu") for a in q0]
    for b, a in zip(system.blocks, q):
        tag = C.byref(C.c_int(b.tag))
        if side == "device":
            t.lib.tioga_b200_registersolution_device_(tag, C.c_void_p(a.data_ptr()))
        else:
            t.lib.tioga_registersolution_(tag, C.c_void_p(a.data_ptr()))
    for nvar in (0, -1):
        t.dataupdate_mb(nvar, "row")
        assert (t.lib.tioga_b200_last_error() != 0) == (nvar < 0)
        for a, b in zip(q, q0):
            assert np.array_equal(a.cpu().numpy(), b)
    t.dataupdate_mb(2, "row")
    assert t.lib.tioga_b200_last_error() == 0
    for b, a in zip(system.blocks, q):
        assert np.array_equal(a.cpu().numpy().view(np.int64), ref["q"][b.tag].view(np.int64))
    t.delete()


def test_phase_times_are_the_connectivity_calls():
    """Elements described after a connectivity call have every cell boxed
    again; the times read afterwards are still those of the call."""
    system, ho = cases.small_config4()
    t = _connected(system)
    tb.set_int(t.lib, "tioga_b200_set_coords_resident_", 1)
    t.performconnectivity()
    assert tb.stats(t.lib)["boxed_cells"] > 0
    for b, h in zip(system.blocks, ho):
        x = np.ascontiguousarray(h.xdof)
        t._keep.append(x)
        t.lib.tioga_b200_set_highorder_lagrange_(C.byref(C.c_int(b.tag)), C.byref(C.c_int(h.p)),
                                                 x.ctypes.data_as(C.c_void_p))
    t.lib.tioga_performconnectivity_highorder_()
    assert t.lib.tioga_b200_last_error() == 0
    ms = tb.timing(t.lib)
    t.delete()
    assert 0 < ms["holemap"] < ms["total"] and 0 < ms["cell_boxes"] < ms["cell_pass"] < ms["boxes_refit"], ms
