"""Host side of the library on a CUDA runtime without a device (tests/engine_fake.py): what it
allocates and reports, and which kernels a call enqueues."""
import ctypes

import numpy as np
import pytest

import engine_fake
from bskit_gb300 import _lib
from bskit_gb300 import bins as B

TWO_PI = 2 * np.pi


@pytest.fixture(scope="module")
def eng(tmp_path_factory):
    return engine_fake.Engine(engine_fake.link(str(tmp_path_factory.mktemp("fake"))))


@pytest.fixture(autouse=True)
def clean(eng):
    eng.lib.fake_set_limit(0)
    eng.lib.fake_set_capturing(0)
    eng.lib.fake_set_symbol(0, -1)
    eng.lib.fake_reset_counts()
    yield


def binning(box, kmax, dk, fields=1):
    kf = TWO_PI / box
    kw = dict(kmin=kf, kmax=kmax * kf, dk=dk * kf)
    return (np.asarray(B.generate_bin_edge_list(**kw)),
            np.asarray(B.generate_triangle_bin_list(num_fields=fields, return_indices=True, **kw)))


def test_everything_is_given_back(eng):
    """Plans, their levels, sets and what measurements kept of them."""
    before = eng.live()
    for n, kmax, grid in ((64, 16, _lib.GRID_REDUCED), (128, 32, _lib.GRID_REDUCED),
                          (96, 40, _lib.GRID_NATIVE), (70, 16, _lib.GRID_NATIVE)):
        edges, tri = binning(100.0, kmax, 2.0)
        p = eng.plan(n, 100.0, edges, grid=grid)
        ts = eng.triangles(p, tri)
        eng.paint(p)
        eng.paint(p, 1)
        for prec in (_lib.PREC_BF16X3, _lib.PREC_FP32):
            eng.measure(p, ts, (0, 0, 1), prec)
        eng.ok(eng.lib.bsk_gridinfo(p, ts, engine_fake.OUT, engine_fake.OUT, None))
        eng.close(p, ts)
    assert eng.live() == before


# the flag that an expired wait of a contraction sets: never, left by an earlier launch, set by
# the route's own launches (second and later reads)
@pytest.mark.parametrize("at", [-1, 0, 1])
def test_gridinfo_does_not_trust_a_contraction_that_gave_up(eng, at):
    edges, tri = binning(100.0, 60, 5.0)
    p = eng.plan(192, 100.0, edges, grid=_lib.GRID_REDUCED_SINGLE)
    assert eng.info(p, _lib.INFO_QMAX) >= 53
    ts = eng.triangles(p, tri)
    eng.lib.fake_reset_counts()
    eng.lib.fake_set_symbol(1, at)
    eng.ok(eng.lib.bsk_gridinfo(p, ts, engine_fake.OUT, engine_fake.OUT, None))
    # the enumeration gives the answer instead, and the flag stays for bsk_sync_check
    assert (eng.launches("enum_finish_kernel") > 0) == (at >= 0)
    assert (eng.launches("modular_finish_kernel") > 0) == (at != 0)
    assert eng.lib.bsk_sync_check(None) == (_lib.BSK_OK if at < 0 else _lib.BSK_ERR_TIMEOUT)
    eng.close(p, ts)


def test_a_paint_without_memory_keeps_nothing_it_loses(eng):
    before = eng.live()
    edges, _ = binning(100.0, 16, 2.0)
    p = eng.plan(64, 100.0, edges)
    # room for the transform's output (1.08 MB), not for the slot's spectrum (0.46 MB) as well
    eng.lib.fake_set_limit(eng.live() + (1200 << 10))
    for _ in range(3):
        assert eng.lib.bsk_paint(p, 0, engine_fake.MESH, None) == _lib.BSK_ERR_OOM
    eng.lib.fake_set_limit(0)
    eng.paint(p)
    eng.close(p)
    assert eng.live() == before


def _synth_bytes(ng, qmax, shells):
    nk, cp = min(2 * qmax + 1, ng), (qmax + 16) // 16 * 16
    return shells * ng * cp * 8 * (nk + ng) + ng * 8


def _split_bytes(shells, k):
    return 2 * 2 * shells * ((k + 127) // 128 * 128)


@pytest.mark.parametrize("n,kmax,dk,levels", [(64, 16, 1.0, False), (128, 32, 6.0, False),
                                              (256, 64, 2.0, True)])
def test_budgeted_plans_hold_what_they_report(eng, monkeypatch, n, kmax, dk, levels):
    """Under a memory budget the synthesis' tables cost nothing beyond the workspace, every byte
    taken is in the footprint, and the figure is enough as the next plan's budget."""
    if levels:
        monkeypatch.setenv("BSK_LEVEL_MIN_POINTS", "0.2")
    edges, tri = binning(100.0, kmax, dk)
    grid = _lib.GRID_REDUCED if levels else _lib.GRID_REDUCED_SINGLE
    budget, shells = 1 << 40, len(edges)
    for _ in range(2):
        p = eng.plan(n, 100.0, edges, budget=budget, grid=grid)
        ts = eng.triangles(p, tri)
        assert (len(eng.levels(ts)) > 1) == levels
        eng.paint(p)
        live, fp = eng.live(), eng.footprint(p)
        eng.measure(p, ts)
        assert eng.info(p, _lib.INFO_STREAM) == 0
        assert eng.live() - live == eng.footprint(p) - fp
        if not levels:
            ng, alloc, batch = eng.info(p, _lib.INFO_NGRID), -(-shells // 8) * 8, 8
            if shells < 8:
                alloc = batch = shells
            assert eng.footprint(p) - fp == (
                4 * alloc * ng ** 3 + _split_bytes(alloc, ng ** 3)
                + _synth_bytes(ng, eng.info(p, _lib.INFO_QMAX), batch))
        budget = eng.footprint(p)
        eng.close(p, ts)


def _short_grid(eng, n=128, kmax=32.0, part=None):
    edges, tri = binning(100.0, kmax, 2.0)
    p = eng.plan(n, 100.0, edges, grid=_lib.GRID_REDUCED_SINGLE)
    return p, eng.triangles(p, tri if part is None else tri[tri.max(1) < part]), tri


def test_captured_contraction_of_ready_fields_has_no_allocation_node(eng):
    """Such a graph may be replayed beside any other call, cloned and instantiated twice."""
    p, ts, _ = _short_grid(eng)
    eng.paint(p)
    eng.measure(p, ts)
    assert eng.launches("tail_sum_kernel") == 1
    eng.lib.fake_reset_counts()
    with eng.capture():
        eng.measure(p, ts)
    assert eng.lib.fake_pool_allocs() == 0
    assert eng.launches("contract_tc_kernel") == 1
    eng.close(p, ts)


def test_captured_passes_share_the_plans_scratch(eng):
    """A pass that synthesises uses the plan's workspace, and with it the plan's scratch."""
    p, ts, _ = _short_grid(eng)
    for _ in range(2):  # the second pass finds everything there
        eng.paint(p)
        eng.measure(p, ts)
    live = eng.live()
    eng.lib.fake_reset_counts()
    for _ in range(3):
        with eng.capture():
            eng.paint(p)
            eng.measure(p, ts)
    assert eng.lib.fake_pool_allocs() == 0 and eng.live() == live
    assert eng.launches("tail_sum_kernel") == 3
    eng.close(p, ts)


@pytest.mark.parametrize("captured", [False, True])
def test_without_room_a_pass_runs_without_scratch(eng, captured):
    p, ts, tri = _short_grid(eng)
    eng.paint(p)
    eng.measure(p, ts, precision=_lib.PREC_FP32)  # fields and workspace, no scratch
    small = eng.triangles(p, tri[:1])
    eng.measure(p, small)                         # and the split
    eng.paint(p)
    eng.lib.fake_set_limit(eng.live() + (8 << 20))
    eng.lib.fake_reset_counts()
    if captured:
        with eng.capture():
            eng.paint(p)
            eng.measure(p, ts)
    else:
        eng.measure(p, ts)
    assert eng.launches("contract_tc_kernel") == 1 and eng.launches("tail_sum_kernel") == 0
    eng.close(p, ts, small)


def test_scratch_that_a_graph_holds_is_kept(eng):
    before = eng.live()
    p, small, tri = _short_grid(eng, part=8)
    large = eng.triangles(p, tri)
    eng.paint(p)
    eng.measure(p, small)
    with eng.capture():
        eng.paint(p)
        eng.measure(p, small)
    live = eng.live()
    # the larger set's scratch comes beside the one in the graph, whether captured or not
    with eng.capture():
        eng.paint(p)
        eng.measure(p, large)
    grown = eng.live()
    assert grown > live
    eng.lib.fake_reset_counts()
    eng.paint(p)
    eng.measure(p, large)
    assert eng.live() == grown and eng.launches("tail_sum_kernel") == 1
    eng.close(p, small, large)
    assert eng.live() == before


@pytest.mark.parametrize("n,levels", [(128, False), (256, True), (70, False)])
def test_plans_report_every_byte_they_keep(eng, monkeypatch, n, levels):
    """Footprint and scratch together are what a plan has taken, after eager and captured
    passes, contractions of ready fields on several streams, and a larger set."""
    if levels:
        monkeypatch.setenv("BSK_LEVEL_MIN_POINTS", "0.01")
    edges, tri = binning(100.0, 32, 2.0)
    p = eng.plan(n, 100.0, edges, grid=_lib.GRID_REDUCED if levels else _lib.GRID_REDUCED_SINGLE)
    sets = [eng.triangles(p, tri[tri.max(1) < 8]), eng.triangles(p, tri)]

    def reported():
        return eng.footprint(p) + eng.lib.bsk_plan_scratch_bytes(p)

    live, rep = eng.live(), reported()
    assert eng.lib.bsk_plan_scratch_bytes(p) == 0
    for ts in sets:
        for slots in ((0, 0, 0), (0, 0, 1)):
            eng.paint(p, 0)
            eng.paint(p, 1)
            eng.measure(p, ts, slots)
            for stream in (1, 2):
                eng.measure(p, ts, slots, stream=ctypes.c_void_p(stream))
            with eng.capture():
                eng.paint(p, 0)
                eng.paint(p, 1)
                eng.measure(p, ts, slots)
            assert eng.live() - live == reported() - rep
    assert eng.lib.bsk_plan_scratch_bytes(p) > 0
    eng.close(p, *sets)
    assert eng.lib.bsk_plan_scratch_bytes(None) == -1


@pytest.mark.parametrize("precision", [_lib.PREC_BF16X3, _lib.PREC_FP32])
def test_sets_of_other_shells_do_not_undo_each_other(eng, monkeypatch, precision):
    """Sets that use different shells of one painted mesh on one level: each is synthesised once,
    and measured again without a synthesis, in any order; no shell twice for the split alone."""
    monkeypatch.setenv("BSK_LEVEL_MIN_POINTS", "0.9")  # one level: the plan's grid
    edges, tri = binning(500.0, 64, 2.0)
    p = eng.plan(256, 500.0, edges)
    parts = [tri[tri.max(1) < 9], tri[tri.min(1) >= 20], tri[(tri.max(1) < 20)], tri]
    sets = [eng.triangles(p, t) for t in parts]
    assert all(len(eng.levels(ts)) == 1 for ts in sets)
    for order in ((0, 1, 2, 3), (1, 0, 3, 2), (3, 0, 1, 2), (2, 1, 0, 3)):
        eng.paint(p, 0)
        eng.paint(p, 1)
        for k in order:
            for slots in ((0, 0, 0), (0, 0, 1), (1, 0, 1)):
                eng.measure(p, sets[k], slots, precision)
        eng.lib.fake_reset_counts()
        for k in order[::-1] + order:
            for slots in ((1, 0, 1), (0, 0, 0), (0, 0, 1)):
                eng.measure(p, sets[k], slots, precision)
        assert eng.launches("x_kernel") == 0, order
        assert eng.launches("contract") == 8 * 3
    # a set whose shells are there but for one batch: that batch alone
    eng.paint(p, 0)
    eng.measure(p, sets[2], precision=precision)
    eng.lib.fake_reset_counts()
    eng.measure(p, sets[3], precision=precision)
    assert eng.launches("x_kernel") == 2  # shells 16 .. 31: two batches of eight
    eng.close(p, *sets)


def test_graphs_of_ready_fields_lease_scratch(eng):
    """A captured contraction of ready fields has scratch of its own, owned by the plan and
    handed back when the last copy of its graph goes: no allocation node, a bounded number of
    them, and whole items where there is no room."""
    before = eng.live()
    p, ts, _ = _short_grid(eng)
    eng.paint(p)
    eng.measure(p, ts)
    live, scratch = eng.live(), eng.lib.bsk_plan_scratch_bytes(p)
    eng.lib.fake_reset_counts()
    sizes = []
    for k in range(8):
        with eng.capture():
            eng.measure(p, ts)
        sizes.append(eng.live() - live)
        assert eng.lib.bsk_plan_scratch_bytes(p) - scratch == sizes[-1]
    assert eng.lib.fake_pool_allocs() == 0
    # 113 MB each, up to 512 MB of them
    assert sizes[0] > 100 << 20 and sizes[3:] == [4 * sizes[0]] * 5
    assert eng.launches("tail_sum_kernel") == 4 and eng.launches("contract_tc_kernel") == 8
    # graphs that went make room; an eager call gives the memory back as well
    eng.lib.fake_destroy_graphs()
    with eng.capture():
        eng.measure(p, ts)
    assert eng.live() - live == sizes[0] and eng.launches("tail_sum_kernel") == 5
    eng.lib.fake_destroy_graphs()
    eng.measure(p, ts)
    assert eng.live() - live == sizes[0]  # the eager call's own
    eng.lib.fake_set_limit(eng.live() + (1 << 20))
    with eng.capture():
        eng.measure(p, ts)
    assert eng.launches("tail_sum_kernel") == 6 and eng.launches("contract_tc_kernel") == 11
    eng.lib.fake_set_limit(0)
    with eng.capture():
        eng.measure(p, ts)
    eng.close(p, ts)
    assert eng.live() == before
    eng.lib.fake_destroy_graphs()  # after its plan
    assert eng.live() == before


# residues from |q| = 53 on (up to 159); below, not for plans of few modes (the fake's have none)
@pytest.mark.parametrize("q,residues", [(39, False), (41, False), (52, False), (53, True),
                                        (159, True), (160, False)])
def test_route_of_the_grid_information(eng, q, residues):
    edges = np.array([[0.5 * q, 0.7 * q], [q - 1.0, q + 0.5]]) * TWO_PI / 100.0
    p = eng.plan(2 * (3 * q // 2 + 4), 100.0, edges, grid=_lib.GRID_REDUCED_SINGLE)
    assert eng.info(p, _lib.INFO_QMAX) == q
    ts = eng.triangles(p, [[1, 1, 0]])
    eng.lib.fake_reset_counts()
    eng.ok(eng.lib.bsk_gridinfo(p, ts, engine_fake.OUT, engine_fake.OUT, None))
    assert (eng.launches("modular_finish_kernel") > 0) == residues
    assert (eng.launches("enum_finish_kernel") > 0) != residues
    eng.close(p, ts)


@pytest.mark.parametrize("n,box,kmax,dk,levels", [
    (64, 100.0, 16, 2.0, None), (128, 100.0, 32, 2.0, None), (256, 500.0, 64, 2.0, None),
    (256, 500.0, 64, 2.0, "0.2"), (512, 1000.0, 128, 2.0, None), (512, 1000.0, 128, 2.0, "1"),
    (128, 100.0, 32, 2.0, "single")])
def test_launches_that_the_benchmark_states(eng, monkeypatch, n, box, kmax, dk, levels):
    import bench
    grid = _lib.GRID_REDUCED
    if levels == "single":
        grid = _lib.GRID_REDUCED_SINGLE
    elif levels:
        monkeypatch.setenv("BSK_LEVEL_MIN_POINTS", levels)
    edges, tri = binning(box, kmax, dk)
    p = eng.plan(n, box, edges, grid=grid)
    ts = eng.triangles(p, tri)

    class Shim(object):
        box_size, shell_edges, n_shells = box, edges, len(edges)
        ngrid, qmax = eng.info(p, _lib.INFO_NGRID), eng.info(p, _lib.INFO_QMAX)
        indices = tri

        @staticmethod
        def levels():
            out = (ctypes.c_int64 * 60)()
            k = eng.lib.bsk_triset_levels(ts, out, 10)
            return [dict(ngrid=int(out[6 * i]), shells=int(out[6 * i + 5])) for i in range(k)]

    for _ in range(2):  # the second step has no tables to make
        eng.lib.fake_reset_counts()
        eng.paint(p)
        eng.measure(p, ts)
        eng.ok(eng.lib.bsk_normalize(len(tri), engine_fake.OUT, engine_fake.OUT, engine_fake.OUT,
                                     None))
    assert (bench.kernel_launches_per_step(Shim, Shim)
            == eng.launches() - eng.launches("tail_sum_kernel"))
    eng.close(p, ts)


def test_a_captured_synthesis_depends_on_no_earlier_one(eng, monkeypatch):
    """A graph that synthesises makes every shell its set needs: it may be replayed after another
    paint, when what an eager call had made is of the mesh before."""
    monkeypatch.setenv("BSK_LEVEL_MIN_POINTS", "0.9")
    edges, tri = binning(500.0, 64, 2.0)
    p = eng.plan(256, 500.0, edges)
    low, every = eng.triangles(p, tri[tri.max(1) < 9]), eng.triangles(p, tri)
    eng.paint(p)
    eng.lib.fake_reset_counts()
    eng.measure(p, every)
    whole = eng.launches("x_kernel")
    eng.paint(p)
    eng.measure(p, low)
    eng.lib.fake_reset_counts()
    with eng.capture():
        eng.measure(p, every)
    assert eng.launches("x_kernel") == whole == 4
    eng.close(p, low, every)
