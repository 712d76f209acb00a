"""Contraction of short grids: items cut into parts with a scratch area, against whole items.

bsk_contract gives the triangle set's scratch to the tensor-core launch, which then spreads
the last wave of work items over all SMs; bsk_contract_noalloc has none and walks whole items.
Both add the same FP32 slice sums, in FP64 and in any order, so a bin may differ by at most
(slices) x 2^-52 of the sum of its slices' magnitudes, which sum |f1 f2 f3| bounds.
"""
import ctypes

import numpy as np
import pytest
import torch

from bskit_gb300 import _lib
from bskit_gb300 import bins as B
from bskit_gb300.engine import Plan

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plans(cuda):
    kf = 2 * np.pi / 100.0
    out = {}
    for fields in (1, 2):
        kw = dict(kmin=kf, kmax=32 * kf, dk=2 * kf)
        edges = B.generate_bin_edge_list(**kw)
        tri = np.ascontiguousarray(B.generate_triangle_bin_list(
            num_fields=fields, return_indices=True, **kw), dtype=np.int32)
        plan = Plan(128, 100.0, edges)  # 15 shells, 96^3 points
        out[fields] = plan, plan.triangles(tri), tri
    return out


# one partial stage; whole stages; one slice less / more than full; several slices with a short
# last one; the plan's grid
@pytest.mark.parametrize("k", [8, 128, 136, 16384 - 8, 16384 + 8, 5 * 16384 + 1000, 96 ** 3])
@pytest.mark.parametrize("fields,precision", [(1, "bf16x3"), (2, "bf16x3"), (1, "bf16")])
def test_parts_equal_whole_items(plans, k, fields, precision):
    plan, ts, tri = plans[fields]
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    f = [torch.randn((plan.n_shells, k), generator=g, device="cuda") for _ in range(fields)]
    fs = [f[0], f[0], f[-1]]
    got = plan.contract(ts, *fs, precision=precision)
    whole = torch.full((len(tri),), float("nan"), dtype=torch.float64, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.call("bsk_contract_noalloc", plan.n_shells, len(tri), tri.ctypes.data,
              *[ctypes.c_void_p(x.data_ptr()) for x in fs], k, _lib.PRECISIONS[precision],
              ctypes.c_void_p(whole.data_ptr()), stream)
    plan.sync_check()
    abs_sum = plan.contract(ts, *[x.abs() for x in fs], precision="fp64")
    slices = -(-k // 16384)
    assert torch.all((got - whole).abs() <= slices * 2.0 ** -52 * 1.01 * abs_sum)


def test_streams_and_graphs_share_no_scratch_unordered(plans):
    """Contractions of one plan on several streams, eager and captured, overlapping as they may:
    each gives what it gives alone (bins within the FP64 order bound above)."""
    plan, ts, tri = plans[1]
    k = 96 ** 3
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    f = [torch.randn((plan.n_shells, k), generator=g, device="cuda") for _ in range(4)]
    want = [plan.contract(ts, x, x, x) for x in f]
    bound = [-(-k // 16384) * 2.0 ** -52 * 1.01 * plan.contract(ts, *[x.abs()] * 3, precision="fp64")
             for x in f]
    streams = [torch.cuda.Stream() for _ in f]
    graphs, outs = [], []
    for x, s in zip(f[:2], streams[:2]):
        torch.cuda.synchronize()
        gr = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gr, stream=s):
            outs.append(plan.contract(ts, x, x, x))
        graphs.append(gr)
    torch.cuda.synchronize()
    for _ in range(5):
        for gr, s in zip(graphs, streams[:2]):
            with torch.cuda.stream(s):
                gr.replay()
        eager = []
        for x, s in zip(f[2:], streams[2:]):
            with torch.cuda.stream(s):
                eager.append(plan.contract(ts, x, x, x))
        torch.cuda.synchronize()
        for got, w, b in zip(outs + eager, want, bound):
            assert torch.all((got - w).abs() <= b)


def test_captured_passes_keep_their_scratch(cuda):
    """Graphs of whole passes (paint, synthesis, contraction in parts) replayed after another set
    has grown the plan's scratch, and graphs of contractions alone, which have none, beside an
    eager pass of another plan: each gives what its eager call gave."""
    kf = 2 * np.pi / 100.0
    kw = dict(kmin=kf, kmax=32 * kf, dk=2 * kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = np.asarray(B.generate_triangle_bin_list(return_indices=True, **kw))
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    mesh = torch.randn((128,) * 3, generator=g, device="cuda")
    plan, other = (Plan(128, 100.0, edges, grid="single") for _ in range(2))
    small, large = plan.triangles(tri[tri.max(1) < 8]), plan.triangles(tri)
    other.paint(0, mesh)

    def run(ts, paint):
        if paint:
            plan.paint(0, mesh)
        return plan.measure_b(ts)

    want, graphs = [], []
    for ts, paint in ((small, True), (large, True), (small, False), (large, False)):
        want.append(run(ts, paint).clone())
        torch.cuda.synchronize()
        gr = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gr):
            out = run(ts, paint)
        graphs.append((gr, out))
    side = torch.cuda.Stream()
    whole = other.measure_b(other.triangles(tri))
    for order in ((0, 1, 2, 3), (3, 2, 1, 0), (1, 0, 1, 0)):
        for k in order:
            gr, out = graphs[k]
            out.zero_()
            torch.cuda.synchronize()
            gr.replay()
            with torch.cuda.stream(side):
                other.paint(0, mesh)
                beside = other.measure_b(other.triangles(tri))
            torch.cuda.synchronize()
            # slices added in FP64 in any order: 54 of them, each below the largest bin
            for got, ref in ((out, want[k]), (beside, whole)):
                assert torch.all((got - ref).abs() <= 54 * 2.0 ** -52 * 54 * ref.abs().max())
    plan.sync_check()


def test_plans_report_the_memory_they_keep(cuda):
    """Footprint and scratch against the device's own count, after an eager pass, one on fields
    that were there, and a captured one.  64 MiB cover the schedules, the FFT library's tables and
    the granularity of a few dozen allocations; the scratch alone is above that."""
    kf = 2 * np.pi / 100.0
    kw = dict(kmin=kf, kmax=32 * kf, dk=2 * kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = B.generate_triangle_bin_list(return_indices=True, **kw)
    mesh = torch.randn((128,) * 3, device="cuda")
    out = torch.empty(len(tri), dtype=torch.float64, device="cuda")

    def passes():
        plan = Plan(128, 100.0, edges, grid="single")
        ts = plan.triangles(tri)
        plan.paint(0, mesh)
        for _ in range(2):
            plan.measure_b(ts, out=out)
        torch.cuda.synchronize()
        gr = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gr):
            plan.paint(0, mesh)
            plan.measure_b(ts, out=out)
        gr.replay()
        torch.cuda.synchronize()
        return plan, gr

    plan, gr = passes()  # loads the kernels
    del gr
    plan.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    plan, gr = passes()
    taken = free - torch.cuda.mem_get_info()[0]
    assert plan.scratch_bytes() > 64 << 20
    assert abs(taken - plan.footprint() - plan.scratch_bytes()) <= 64 << 20
    plan.close()


def test_graphs_of_ready_fields(cuda):
    """A graph of a contraction of ready fields: instantiated twice, replayed beside the eager
    call on another stream, and its scratch goes back to the plan with it."""
    import time
    kf = 2 * np.pi / 100.0
    kw = dict(kmin=kf, kmax=32 * kf, dk=2 * kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = np.asarray(B.generate_triangle_bin_list(return_indices=True, **kw))
    plan = Plan(128, 100.0, edges, grid="single")
    ts = plan.triangles(tri)
    plan.paint(0, torch.randn((128,) * 3, device="cuda"))
    for _ in range(2):  # the second finds the fields ready
        want = plan.measure_b(ts).clone()
    torch.cuda.synchronize()
    kept = plan.scratch_bytes()
    out = torch.zeros_like(want)
    gr = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(gr):
        plan.measure_b(ts, out=out)
    assert plan.scratch_bytes() > kept
    runtime = ctypes.CDLL("libcudart.so.13")
    execs = [ctypes.c_void_p() for _ in range(2)]
    for e in execs:
        assert runtime.cudaGraphInstantiate(ctypes.byref(e), ctypes.c_void_p(gr.raw_cuda_graph()),
                                            ctypes.c_ulonglong(0)) == 0
    side = torch.cuda.Stream()
    tol = 54 * 2.0 ** -52 * 54 * want.abs().max()  # as above
    for e in execs + execs:
        out.zero_()
        torch.cuda.synchronize()
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert runtime.cudaGraphLaunch(e, stream) == 0
        with torch.cuda.stream(side):
            beside = plan.measure_b(ts)
        torch.cuda.synchronize()
        for got in (out, beside):
            assert torch.all((got - want).abs() <= tol)
    for e in execs:
        assert runtime.cudaGraphExecDestroy(e) == 0
    assert plan.scratch_bytes() > kept  # the graph itself has it still
    del gr
    for _ in range(100):  # the runtime's own thread hands it back
        plan.measure_b(ts)
        if plan.scratch_bytes() == kept:
            break
        time.sleep(0.05)
    assert plan.scratch_bytes() == kept
    plan.sync_check()
    plan.close()
