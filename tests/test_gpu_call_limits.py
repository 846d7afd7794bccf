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


DELTA = 10.0 / 2 ** 19  # the coincidence gate's distance in a block 10 wide


def _graded(inner, gap, twin=None):
    """A box 10 wide whose inner nodes per axis lie `gap` apart around the
    origin, under a shell; with `twin` another node there, moved from a node
    of the box by that much."""
    a = (np.arange(inner) - 0.5 * (inner - 1)) * gap
    far = np.geomspace(a[-1] + gap, 5.0, 6)
    ax = np.concatenate([-far[::-1], a, far])
    n = len(ax)
    x, cells = cases.hex_box(n, -5.0, 5.0)
    ijk = np.rint((x + 5.0) * (n - 1) / 10.0).astype(int)
    x = ax[ijk]
    if twin is not None:
        mid = np.flatnonzero((ijk == n // 2).all(1))[0]
        x = np.concatenate([x, x[mid:mid + 1] + np.array([[0.0, twin, 0.0]])])
    none = np.zeros(0, np.int32)
    xs, cs, wall, outer, _ = cases.sphere_shell(9, 9, 17, 0.5, 2.0, 1.1, np.array([1.0, 0.2, 0.1]), 0.0,
                                                np.random.default_rng(0))
    return cases.System([cases.Block(1, np.ascontiguousarray(x), cells, none, none),
                         cases.Block(2, xs, cs, wall, outer)])


def _preprocess_ms(t):
    import time
    best = 1e9
    for _ in range(4):
        t0 = time.perf_counter()
        t.preprocess_grids()
        best = min(best, 1e3 * (time.perf_counter() - t0))
    return best


@pytest.mark.parametrize("inner,gap", [(17, 1.03), (30, 2.1), (44, 7.0)])
def test_coincidence_gate_of_graded_blocks(inner, gap, oracle_lib):
    """Thousands of nodes in a cell of the coincidence gate, none closer than
    its distance: no merge runs and a preprocess costs what it costs on a mesh
    of as many nodes that is not graded.  With one node closer than that (and
    within TOL) the merge runs and merges it."""
    plain = cases.config0(3, nbg=inner + 12, nr=9, nt=9, nphi=17, perturb=0.0)
    t = _connected(plain)
    plain_launches, plain_ms = tb.stats(t.lib)["launches"], _preprocess_ms(t)
    t.delete()
    for twin in (None, 1e-12, -0.3 * DELTA):
        system = _graded(inner, gap * DELTA, twin)
        ref = run_system(oracle_lib, system)
        t = _connected(system)
        st = tb.stats(t.lib)
        assert (st["nmerged"] > 0) == (twin == 1e-12)
        assert (st["launches"] > plain_launches + 10) == (twin is not None), (st["launches"], plain_launches)
        for b in system.blocks:
            assert np.array_equal(ref["iblank"][b.tag], t.iblank(b.tag))
            for a, c in zip(ref["donors"][b.tag], t.getdonorinfo(b.tag)):
                assert np.array_equal(a, c)
        ms = _preprocess_ms(t)
        t.delete()
        assert ms < 6 * plain_ms, (ms, plain_ms)


@pytest.mark.parametrize("octaves", [40, 180, 400])
def test_merge_of_points_across_many_octaves(octaves, oracle_lib):
    """Query points at distances 1, 1/2, 1/4 ... from a plane and thirty
    coincident ones beyond the last: a split halves a box, so they are apart
    only after as many levels as there are octaves.  At most 33 are farther
    apart than TOL and each of the merge's 128 levels takes one away, so all
    but 162 are merged, also where there are more octaves than levels."""
    base = cases.config0(2, nbg=13, nr=9, nt=11, nphi=21, perturb=0.0)
    bg = base.blocks[0]
    d = np.concatenate([2.0 ** -np.arange(octaves), np.full(30, 2.0 ** -octaves)])
    extra = np.stack([d, np.full(len(d), 0.8), np.full(len(d), 0.3)], 1)
    system = cases.System([cases.Block(bg.tag, np.concatenate([bg.x, extra]), bg.cells, bg.wbc, bg.obc),
                           *base.blocks[1:]])
    ref = run_system(oracle_lib, system)
    t = _connected(system)
    assert tb.stats(t.lib)["nmerged"] >= max(29, len(d) - 162), tb.stats(t.lib)
    for b in system.blocks:
        assert np.array_equal(ref["iblank"][b.tag], t.iblank(b.tag))
    t.delete()


def test_fp64_walks_far_from_the_origin(oracle_lib):
    """The FP64 form on a mesh moved by 2^20 with cells of about 1/128 (every
    coordinate exact in both places): the oracle's result there, and walks as
    short as at the origin."""
    base = cases.config0(3, nbg=41, nr=13, nt=25, nphi=49, perturb=0.02)
    ms = {}
    for offset in (0.0, 2.0 ** 20):
        system = cases.System([cases.Block(b.tag, np.round(b.x / 26.0 * 2.0 ** 26) / 2.0 ** 26 + offset, b.cells,
                                           b.wbc, b.obc) for b in base.blocks])
        ref = run_system(oracle_lib, system)
        t = TiogaLibrary(tb.library_path())
        tb.extras(t.lib)
        t.init()
        t.register_system(system)
        tb.set_int(t.lib, "tioga_b200_set_precision_", 0)
        t.preprocess_grids()
        walk = []
        for _ in range(5):
            t.performconnectivity()
            assert t.lib.tioga_b200_last_error() == 0
            walk.append(tb.timing(t.lib)["search_traverse"])
        ms[offset] = min(walk)
        for b in system.blocks:
            assert np.array_equal(ref["iblank"][b.tag], t.iblank(b.tag))
            for a, c in zip(ref["donors"][b.tag], t.getdonorinfo(b.tag)):
                assert np.array_equal(a, c)
        t.delete()
    assert ms[2.0 ** 20] < 4 * ms[0.0], ms


@pytest.mark.parametrize("form", [0, 1])
def test_high_order_search_in_another_form_than_the_last_call(form):
    """The precision changed between the connectivity call and the high-order
    one: the same point donors as with one precision throughout."""
    system, ho = cases.small_config4()
    got = []
    for forms in ((form, form), (1 - form, form)):
        t = TiogaLibrary(tb.library_path())
        tb.extras(t.lib)
        t.init()
        t.register_system(system)
        for b, h in zip(system.blocks, ho):
            x = np.ascontiguousarray(h.xdof)
            t._keep.append(x)
            t.lib.tioga_b200_set_highorder_lagrange_(C.byref(C.c_int(b.tag)), C.byref(C.c_int(h.p)),
                                                     x.ctypes.data_as(C.c_void_p))
        t.preprocess_grids()
        tb.set_int(t.lib, "tioga_b200_set_precision_", forms[0])
        t.performconnectivity()
        tb.set_int(t.lib, "tioga_b200_set_precision_", forms[1])
        t.lib.tioga_performconnectivity_highorder_()
        assert t.lib.tioga_b200_last_error() == 0
        points = []
        for b in system.blocks:
            n = t.lib.tioga_b200_pointdonors_(C.byref(C.c_int(b.tag)), None, None)
            rec = np.zeros((max(n, 1), 4), np.int32)
            t.lib.tioga_b200_pointdonors_(C.byref(C.c_int(b.tag)), rec.ctypes.data_as(C.c_void_p), None)
            points.append(rec[:n])
        got.append(points)
        t.delete()
    assert sum(len(p) for p in got[0]) > 0
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("where", ["pinned", "mixed"])
def test_device_arrays_that_only_copies_reach(where, oracle_lib):
    """Page-locked host memory given as a device iblank array, for all blocks
    and for one beside a device array: written by copies, as another GPU's
    memory would be."""
    import torch
    system = cases.config1(4, nbg=17, nshell=2, nr=7, nt=7, nphi=13, split_layers=2)
    ref = run_system(oracle_lib, system)
    t = TiogaLibrary(tb.library_path())
    tb.extras(t.lib)
    t.init()
    t.register_system(system)
    ibl = []
    for i, b in enumerate(system.blocks):
        here = where == "mixed" and i != 1
        a = torch.full((b.nnodes,), -7, dtype=torch.int32, device="cuda" if here else "cpu", pin_memory=not here)
        ibl.append(a)
        t.lib.tioga_b200_registeriblank_device_(C.byref(C.c_int(b.tag)), C.c_void_p(a.data_ptr()))
    torch.cuda.synchronize()
    t.preprocess_grids()
    assert t.lib.tioga_b200_last_error() == 0
    for a in ibl:
        assert (a == 1).all()
    t.performconnectivity()
    assert t.lib.tioga_b200_last_error() == 0
    for b, a in zip(system.blocks, ibl):
        assert np.array_equal(ref["iblank"][b.tag], a.cpu().numpy())
    t.delete()


def test_high_order_fields_that_only_copies_reach():
    """Device solutions of the high-order update in page-locked host memory
    for one block: the same values as with both on the device."""
    import torch
    system, ho = cases.small_config4()
    q0 = [np.ascontiguousarray(q, dtype=np.float64).reshape(-1) for q in cases.dof_fields(ho, 2, seed=3)]
    got = []
    for pinned in (False, True):
        t = TiogaLibrary(tb.library_path())
        tb.extras(t.lib)
        t.init()
        t.register_system(system)
        for b, h in zip(system.blocks, ho):
            x = np.ascontiguousarray(h.xdof)
            t._keep.append(x)
            t.lib.tioga_b200_set_highorder_lagrange_(C.byref(C.c_int(b.tag)), C.byref(C.c_int(h.p)),
                                                     x.ctypes.data_as(C.c_void_p))
        t.preprocess_grids()
        t.performconnectivity()
        t.lib.tioga_performconnectivity_highorder_()
        q = [torch.from_numpy(a.copy()) for a in q0]
        q = [a.pin_memory() if pinned and i == 1 else a.cuda() for i, a in enumerate(q)]
        for b, a in zip(system.blocks, q):
            t.lib.tioga_b200_registersolution_device_(C.byref(C.c_int(b.tag)), C.c_void_p(a.data_ptr()))
        t.dataupdate_mb(2, "row")
        assert t.lib.tioga_b200_last_error() == 0
        got.append([a.cpu().numpy() for a in q])
        t.delete()
    assert any((a != b).any() for a, b in zip(got[0], q0))
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "split"])
def test_batch_past_the_four_lane_walk(precision, oracle_lib):
    """A batch that is shown to have the million queries from which a walk
    has one lane, against the oracle, system by system."""
    two = [cases.config0(s, nbg=49, nr=17, nt=25, nphi=49, perturb=0.05) for s in (1, 2)]
    refs = [run_system(oracle_lib, s) for s in two]
    copies = [cases.System([cases.Block(b.tag, b.x.copy(), b.cells, b.wbc, b.obc) for b in two[k % 2].blocks])
              for k in range(50)]
    t = TiogaLibrary(tb.library_path())
    tb.extras(t.lib)
    t.init()
    t.register_batch(copies)
    tb.set_int(t.lib, "tioga_b200_set_precision_", precision)
    t.preprocess_grids()
    t.performconnectivity()
    assert t.lib.tioga_b200_last_error() == 0
    assert tb.stats(t.lib)["nquery"] >= 1 << 20, tb.stats(t.lib)
    for k, system in enumerate(copies):
        t.select_system(k)
        got = {"iblank": {b.tag: t.blocks[(k, b.tag)]["iblank"].copy() for b in system.blocks},
               "donors": {b.tag: t.getdonorinfo(b.tag) for b in system.blocks}, "q": {}}
        problems = diff_runs(system, refs[k % 2], got)
        assert not problems, "\n".join(problems)
    t.delete()


@pytest.mark.parametrize("side", ["device", "host"])
def test_update_after_a_refused_connectivity_call(side, oracle_lib):
    """A connectivity call refused for a coordinate that is not finite leaves
    the interpolation of the one before: an update then is the oracle's, and
    so is the next call on good coordinates."""
    import torch
    system = cases.small_config1(2)
    q0 = cases.fields(system, nvar=3, seed=5)
    ref = run_system(oracle_lib, system, q_blocks=q0, nvar=3)
    t = _connected(system)
    for again in (False, True):
        x = t.blocks[system.blocks[1].tag]["x"]
        good = x[7]
        if not again:
            x[7] = np.nan
        t.performconnectivity()
        assert (t.lib.tioga_b200_last_error() != 0) == (not again)
        x[7] = good
        q = [torch.from_numpy(a.copy()).to("cuda" if side == "device" else "cpu") for a in q0]
        for b, a in zip(system.blocks, q):
            tag = C.byref(C.c_int(b.tag))
            if side == "device":
                t.lib.tioga_b200_registersolution_device_(tag, C.c_void_p(a.data_ptr()))
            else:
                t.lib.tioga_registersolution_(tag, C.c_void_p(a.data_ptr()))
        t.dataupdate_mb(3, "row")
        assert t.lib.tioga_b200_last_error() == 0
        for b, a in zip(system.blocks, q):
            assert np.array_equal(a.cpu().numpy().view(np.int64), ref["q"][b.tag].view(np.int64))
    t.delete()


@pytest.mark.parametrize("nvar", [40, 360])
def test_columns_of_page_locked_fields(nvar, oracle_lib):
    """Column-layout updates on either side of the line from which page-locked
    fields go up whole, page-locked throughout, in part and not at all: the
    same bits, and on the small side the oracle's."""
    import torch
    system = cases.config1(3, nbg=45, nshell=2, nr=7, nt=11, nphi=21, split_layers=2)
    n = sum(b.nnodes for b in system.blocks)
    assert n * 40 < 1 << 25 <= n * 360
    rng = np.random.default_rng(nvar)
    q0 = [rng.standard_normal(b.nnodes * nvar) for b in system.blocks]
    t = _connected(system)
    got = []
    for pinned in ((False, False, False), (True, True, True), (True, False, True)):
        q = [torch.from_numpy(a.copy()) for a in q0]
        q = [a.pin_memory() if p else a for a, p in zip(q, pinned)]
        for b, a in zip(system.blocks, q):
            t.lib.tioga_registersolution_(C.byref(C.c_int(b.tag)), C.c_void_p(a.data_ptr()))
        for _ in range(2):
            t.dataupdate_mb(nvar, "column")
            assert t.lib.tioga_b200_last_error() == 0
        got.append([a.numpy() for a in q])
    t.delete()
    for g in got[1:]:
        for a, b in zip(got[0], g):
            assert np.array_equal(a.view(np.int64), b.view(np.int64))
    if nvar == 40:
        ref = TiogaLibrary(oracle_lib)
        ref.init()
        ref.register_system(system)
        ref.preprocess_grids()
        ref.performconnectivity()
        q = [a.copy() for a in q0]
        for b, a in zip(system.blocks, q):
            ref.registersolution(b.tag, a)
        for _ in range(2):
            ref.dataupdate_mb(nvar, "column")
        ref.delete()
        for a, b in zip(got[1], q):
            assert np.array_equal(a.view(np.int64), b.view(np.int64))
