"""Shell fields of plans under a memory budget, whose synthesis launches take fewer shells where
the masks at the workspace's end are in the way: the same bits as without a budget, as a
shell's fields do not depend on the shells it is launched with."""
import math

import numpy as np
import pytest
import torch

from bskit_gb300.engine import Plan

pytestmark = pytest.mark.gpu


# one shell (the workspace holds one shell and the masks); fewer than a batch; a batch and one;
# several batches; a length of the run-time passes
@pytest.mark.parametrize("n,shells,kmax", [(64, 1, 15.0), (64, 5, 15.0), (64, 9, 15.0),
                                           (128, 30, 31.0), (330, 3, 107.0)])
def test_fields(cuda, n, shells, kmax):
    box = 100.0
    q = np.linspace(1.0, kmax, shells + 1)
    edges = np.stack([q[:-1], q[1:]], axis=1) * 2 * math.pi / box
    g = torch.Generator(device="cuda")
    g.manual_seed(n + shells)
    mesh = torch.randn((n, n, n), generator=g, device="cuda")
    plans = [Plan(n, box, edges, grid="single", mem_budget=b) for b in (0, 1 << 37)]
    for p in plans:
        p.paint(0, mesh)
    for s in range(shells):
        free, tight = (p.field(0, s) for p in plans)
        assert torch.equal(free, tight), s
        assert free.abs().max() > 0
    for p in plans:
        p.close()
