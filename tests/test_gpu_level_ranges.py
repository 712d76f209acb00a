"""Grid levels synthesise only the shells their bins use: sets that use different shells of one
painted mesh, measured in any order on one plan, give what each gives on a plan of its own.

The contractions are the same ones on the same fields, so only the FP64 order of the slices'
sums may differ: relative to the largest bin, a few thousand slices x 2^-53.
"""
import itertools

import numpy as np
import pytest
import torch

from bskit_gb300 import bins as B
from bskit_gb300.engine import Plan
from bskit_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
def test_sets_of_different_shells(cuda, monkeypatch, precision):
    monkeypatch.setenv("BSK_LEVEL_MIN_POINTS", "0.2")  # at least two levels on 256^3
    n, box = 256, 500.0
    kf = 2 * np.pi / box
    kw = dict(kmin=kf, kmax=64 * kf, dk=2 * kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = B.generate_triangle_bin_list(return_indices=True, **kw)
    high = tri[tri[:, 2] >= 18]                       # no small shell at all
    equal = B.generate_equilateral_triangle_bin_list(return_indices=True, **kw)
    d = synthetic.lognormal_mesh_torch(n, box, seed=3, device=cuda).contiguous()
    e = (1.5 * d + 0.3 * torch.randn_like(d)).contiguous()
    sets = {"all": (tri, (0, 0, 0)), "high": (high, (0, 0, 0)), "equal": (equal, (0, 0, 1)),
            "cross": (high, (1, 0, 1))}

    def paint(p):
        p.paint(0, d)
        p.paint(1, e)

    want = {}
    for k, (t, slots) in sets.items():
        p = Plan(n, box, edges)
        paint(p)
        want[k] = p.measure_b(p.triangles(t), slots=slots, precision=precision)
        p.close()
    p = Plan(n, box, edges)
    made = {k: p.triangles(t) for k, (t, _) in sets.items()}
    assert len(made["all"].levels()) >= 2
    for order in itertools.permutations(sets):
        paint(p)
        for k in order + order[:1]:
            got = p.measure_b(made[k], slots=sets[k][1], precision=precision)
            assert torch.all((got - want[k]).abs() <= 4096 * 2.0 ** -53 * want[k].abs().max()), \
                (order, k)
    p.sync_check()


@pytest.mark.parametrize("low", [11, 21, 29])
def test_column_slot_without_fields(cuda, monkeypatch, low):
    """A slot that is only a third shell has no FP32 fields, and its level stops inside a batch
    of the level plan, which holds every shell that fits the side: none of the batch's further
    shells is written.  Same contraction as on a plan whose slot has them."""
    monkeypatch.setenv("BSK_LEVEL_MIN_POINTS", "0.01")
    n, box = 256, 500.0
    kf = 2 * np.pi / box
    kw = dict(kmin=kf, kmax=64 * kf, dk=2 * kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = B.generate_triangle_bin_list(return_indices=True, **kw)
    tri = tri[tri.max(1) < low]
    d = synthetic.lognormal_mesh_torch(n, box, seed=4, device=cuda).contiguous()
    e = (1.5 * d + 0.3 * torch.randn_like(d)).contiguous()
    got = []
    for first in ((), ((1, 1, 0),)):
        p = Plan(n, box, edges)
        p.paint(0, d)
        p.paint(1, e)
        t = p.triangles(tri)
        assert max(lv["shells"] for lv in t.levels()) == low
        for slots in first:
            p.measure_b(t, slots=slots, precision="bf16x3")
        got.append(p.measure_b(t, slots=(0, 0, 1), precision="bf16x3"))
        p.sync_check()
        p.close()
    assert torch.all((got[0] - got[1]).abs() <= 4096 * 2.0 ** -53 * got[1].abs().max())


@pytest.mark.parametrize("precision", ["bf16x3", "fp32"])
def test_ranges_that_grow_over_a_gap(cuda, monkeypatch, precision):
    """Low and high shells of one level, as pair factors, columns or both, in turn: the slot's
    ranges grow to hulls, whose middle is synthesised with the second set."""
    monkeypatch.setenv("BSK_LEVEL_MIN_POINTS", "0.9")  # one level
    n, box = 256, 500.0
    kf = 2 * np.pi / box
    kw = dict(kmin=kf, kmax=64 * kf, dk=2 * kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = B.generate_triangle_bin_list(return_indices=True, **kw)
    sets = [tri[tri.max(1) < 9], tri[tri.min(1) >= 20],
            tri[(tri.max(1) < 20) & (tri.min(1) >= 9)]]
    d = synthetic.lognormal_mesh_torch(n, box, seed=5, device=cuda).contiguous()
    e = (1.5 * d + 0.3 * torch.randn_like(d)).contiguous()
    slots = ((0, 0, 1), (0, 0, 0), (1, 0, 1))

    def plan():
        p = Plan(n, box, edges)
        p.paint(0, d)
        p.paint(1, e)
        return p, [p.triangles(t) for t in sets]

    want = {}
    for k in range(3):
        for sl in slots:
            p, made = plan()
            want[k, sl] = p.measure_b(made[k], slots=sl, precision=precision)
            p.close()
    for order in itertools.permutations(range(3)):
        p, made = plan()
        for k in order + order:
            for sl in slots:
                got = p.measure_b(made[k], slots=sl, precision=precision)
                assert torch.all((got - want[k, sl]).abs() <=
                                 4096 * 2.0 ** -53 * want[k, sl].abs().max()), (order, k, sl)
        p.sync_check()
        p.close()
