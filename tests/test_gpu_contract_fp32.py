"""Plain-FP32 contraction: every tile width, ragged chunk and slice, short and long grids.

A bin's slice sum is a chain of FP32 multiply-adds in point order on FP32 pair products.  The
reference runs that chain for every bin at once, each step exact in FP64 and rounded to FP32 (the
double rounding differs from a fused multiply-add's with a chance of ~2^-29 a step, by one
place of the running sum), so a bin may be off by a few places of its largest running sum.
"""
import numpy as np
import pytest
import torch

from bskit_gb300 import bins as B
from bskit_gb300.engine import Plan

pytestmark = pytest.mark.gpu

SLICE = 8192


def _chain(f, tri):
    i, j, l = (torch.as_tensor(tri[:, c].copy(), device="cuda", dtype=torch.long) for c in range(3))
    k = f[0].shape[1]
    total = torch.zeros(len(tri), dtype=torch.float64, device="cuda")
    top = torch.zeros_like(total)
    for x0 in range(0, k, SLICE):
        x1 = min(k, x0 + SLICE)
        cols = [v[:, x0:x1].T.contiguous() for v in f]
        acc = torch.zeros(len(tri), device="cuda")
        for x in range(x1 - x0):
            p = cols[0][x][i] * cols[1][x][j]
            acc = (acc.double() + p.double() * cols[2][x][l].double()).float()
            top = torch.maximum(top, acc.double().abs())
        total += acc.double()
    return total, top


# shells (tile widths 8, 16, 8 .. 64 in mixed tiles); points: one ragged chunk, a whole one, one
# slice less / more than full; and enough slices for the long-grid tiles (points repeated, so
# that one slice's chain stands for all)
@pytest.mark.parametrize("shells,fields", [(5, 1), (15, 1), (15, 2), (40, 1), (63, 1)])
@pytest.mark.parametrize("k", [8, 16, 40, SLICE - 8, SLICE + 24, "long"])
def test_chain(cuda, shells, fields, k):
    kf = 2 * np.pi / 100.0
    kw = dict(kmin=kf, kmax=(shells + 1.5) * kf, dk=kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = B.generate_triangle_bin_list(num_fields=fields, return_indices=True, **kw)
    n = len(edges)
    plan = Plan(max(32, 4 * ((shells + 2) // 2 * 2)), 100.0, edges, grid="native")
    g = torch.Generator(device="cuda")
    g.manual_seed(shells * 100 + fields)
    points = SLICE if k == "long" else k
    f = [torch.randn((n, points), generator=g, device="cuda") for _ in range(fields)]
    f = [f[0], f[0], f[-1]]
    want, top = _chain(f, tri)
    repeat = 1
    if k == "long":
        repeat = 700
        f = [v.repeat(1, repeat) for v in (f[0], f[2])]
        f = [f[0], f[0], f[1] if fields == 2 else f[0]]
    got = plan.contract(plan.triangles(tri), *f, precision="fp32")
    tol = 4 * 2.0 ** -24 * top + repeat * 2.0 ** -52 * top
    assert torch.all((got - repeat * want).abs() <= repeat * tol)


@pytest.mark.parametrize("cut", [1, 4099, 8190, 50001])
def test_shards_off_16_bytes(cuda, cut):
    # two point ranges that meet off a 16-byte boundary: 4-byte copies; the shards' sums are the
    # whole's up to where the slices are cut, within FP32 rounding of a slice's 8192 terms
    n, box = 64, 100.0
    kf = 2 * np.pi / box
    kw = dict(kmin=kf, kmax=16 * kf, dk=2 * kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = B.generate_triangle_bin_list(return_indices=True, **kw)
    plan = Plan(n, box, edges, grid="single")
    plan.paint(0, torch.randn((n, n, n), generator=torch.Generator(device="cuda").manual_seed(cut),
                              device="cuda"))
    ts = plan.triangles(tri)
    f = torch.stack([plan.field(0, s).reshape(-1) for s in range(len(edges))]).abs()
    top = plan.contract(ts, f, f, f, precision="fp64") * box ** 6 / plan.ngrid ** 3
    k = plan.ngrid ** 3
    parts = sum(plan.measure_b_range(ts, a, b, precision="fp32") for a, b in ((0, cut), (cut, k)))
    whole = plan.measure_b(ts, precision="fp64")
    assert torch.all((parts - whole).abs() <= (SLICE + 2) * 2.0 ** -24 * top)


# three different source arrays; more than 64 shells, where a tile's two factor ranges start at
# different shells even of one array
@pytest.mark.parametrize("shells,distinct", [(5, 3), (15, 3), (24, 2), (80, 3), (80, 1)])
@pytest.mark.parametrize("k", [8, 40, SLICE + 24, "long"])
def test_chain_of_two_sources(cuda, shells, distinct, k):
    kf = 2 * np.pi / 100.0
    edges = np.array([[q, q + 1.0] for q in range(1, shells + 1)]) * kf
    rng = np.random.default_rng(shells + distinct)
    tri = np.unique(rng.integers(0, shells, (700, 3)), axis=0)
    plan = Plan(2 * (shells + 4), 100.0, edges, grid="native")
    g = torch.Generator(device="cuda")
    g.manual_seed(shells * 10 + distinct)
    points = SLICE if k == "long" else k
    f = [torch.randn((shells, points), generator=g, device="cuda") for _ in range(distinct)]
    f = {1: [0, 0, 0], 2: [0, 1, 0], 3: [0, 1, 2]}[distinct], f
    f = [f[1][i] for i in f[0]]
    want, top = _chain(f, tri)
    # enough slices for the tiles of long grids (four items an SM), points repeated
    repeat = 700 if k == "long" else 1
    if repeat > 1:
        wide = {id(v): v.repeat(1, repeat) for v in f}
        f = [wide[id(v)] for v in f]
    got = plan.contract(plan.triangles(tri), *f, precision="fp32")
    tol = 4 * 2.0 ** -24 * top + repeat * 2.0 ** -52 * top
    assert torch.all((got - repeat * want).abs() <= repeat * tol)
    plan.close()


@pytest.mark.parametrize("cut", [1, 4099, 50001])
@pytest.mark.parametrize("n,kmax", [(64, 16), (256, 64)])
def test_shards_of_three_fields_off_16_bytes(cuda, cut, n, kmax):
    """As above for <ABC>, on a short grid and on one of whole-tile items."""
    box = 100.0
    kf = 2 * np.pi / box
    kw = dict(kmin=kf, kmax=kmax * kf, dk=kmax * kf / 8)
    edges = B.generate_bin_edge_list(**kw)
    tri = B.generate_triangle_bin_list(num_fields=3, return_indices=True, **kw)
    plan = Plan(n, box, edges, grid="single")
    g = torch.Generator(device="cuda").manual_seed(cut + n)
    for s in range(3):
        plan.paint(s, torch.randn((n, n, n), generator=g, device="cuda"))
    ts, k = plan.triangles(tri), plan.ngrid ** 3
    f = [torch.stack([plan.field(s, i).reshape(-1) for i in range(len(edges))]).abs()
         for s in range(3)]
    top = plan.contract(ts, *f, precision="fp64") * box ** 6 / k
    parts = sum(plan.measure_b_range(ts, a, b, slots=(0, 1, 2), precision="fp32")
                for a, b in ((0, cut), (cut, k)))
    whole = plan.measure_b(ts, slots=(0, 1, 2), precision="fp64")
    assert torch.all((parts - whole).abs() <= (SLICE + 2) * 2.0 ** -24 * top)
    plan.close()


# sparse sets, whose items of a short grid partly hold no bin: the diagonal, one far corner, a band
@pytest.mark.parametrize("shells", [9, 24, 40, 64, 90])
@pytest.mark.parametrize("kind", ["diagonal", "corner", "band"])
@pytest.mark.parametrize("k", [40, SLICE + 24])
def test_chain_of_sparse_sets(cuda, shells, kind, k):
    kf = 2 * np.pi / 100.0
    edges = np.array([[q, q + 1.0] for q in range(1, shells + 1)]) * kf
    s = np.arange(shells)
    tri = {"diagonal": np.stack([s, s, s], 1),
           "corner": np.array([[0, 0, 0], [shells - 1, shells - 2, shells - 1]]),
           "band": np.stack([s, s // 2, np.maximum(s - 3, 0)], 1)}[kind]
    plan = Plan(2 * (shells + 4), 100.0, edges, grid="native")
    g = torch.Generator(device="cuda")
    g.manual_seed(shells + k)
    f = [torch.randn((shells, k), generator=g, device="cuda")] * 3
    want, top = _chain(f, tri)
    got = plan.contract(plan.triangles(tri), *f, precision="fp32")
    assert torch.all((got - want).abs() <= 4 * 2.0 ** -24 * top + 2.0 ** -52 * top)
    plan.close()


# the same on long grids, where dense sets take whole tiles and sparse ones their parts
@pytest.mark.parametrize("shells,distinct", [(40, 1), (64, 2)])
def test_chain_of_sparse_sets_on_long_grids(cuda, shells, distinct):
    kf = 2 * np.pi / 100.0
    edges = np.array([[q, q + 1.0] for q in range(1, shells + 1)]) * kf
    s = np.arange(shells)
    tri = np.stack([s, s // 2, s], 1)
    plan = Plan(2 * (shells + 4), 100.0, edges, grid="native")
    g = torch.Generator(device="cuda")
    g.manual_seed(shells)
    f = [torch.randn((shells, SLICE), generator=g, device="cuda") for _ in range(distinct)]
    want, top = _chain([f[0], f[-1], f[0]], tri)
    repeat = 800
    wide = [v.repeat(1, repeat) for v in f]
    got = plan.contract(plan.triangles(tri), wide[0], wide[-1], wide[0], precision="fp32")
    tol = 4 * 2.0 ** -24 * top + repeat * 2.0 ** -52 * top
    assert torch.all((got - repeat * want).abs() <= repeat * tol)
    plan.close()
