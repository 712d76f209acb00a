"""Grid information from residues modulo small primes, against the lattice enumeration.

Both evaluate the same integers (triangle counts, and |q| 2^44 summed over triangles), so the
counts are equal; the enumeration adds its |q| sums per batch of modes in FP64, fewer than 4096
batches here, the residues give the exact integer, rounded once: k_mean agrees to 4096 x 2^-52.
A memory budget with no room for the residues' scratch keeps a plan on the enumeration.
"""
import numpy as np
import pytest
import torch

from bskit_gb300 import bins as B
from bskit_gb300.engine import Plan

pytestmark = pytest.mark.gpu


# the smallest |q| range of the route (40); edges on and off multiples of k_f; one shell; three
# fields (unsorted triples); wide shells to a large radius; more than 32 shells; the last value
# of |q| below the route's range, where both plans enumerate
@pytest.mark.parametrize("n,box,kmax,dk,fields", [
    (192, 300.0, 41.0, 3.0, 1), (192, 1000.0, 60.9, 4.7, 2), (128, 100.0, 42.5, 40.0, 1),
    (256, 500.0, 63.9, 7.1, 3), (360, 720.0, 108.0, 9.0, 1), (200, 410.0, 46.0, 1.0, 1),
    (192, 300.0, 40.0, 3.0, 1)])
def test_residues_equal_enumeration(cuda, n, box, kmax, dk, fields):
    kf = 2 * np.pi / box
    kw = dict(kmin=kf, kmax=kmax * kf, dk=dk * kf)
    edges = B.generate_bin_edge_list(**kw)
    tri = B.generate_triangle_bin_list(num_fields=fields, return_indices=True, **kw)
    tri = np.concatenate([tri, tri[:1]])  # a repeated bin
    free = Plan(n, box, edges, grid="single")
    tight = Plan(n, box, edges, grid="single", mem_budget=free.footprint() + (1 << 20))
    (nt, km), (nt0, km0) = (p.gridinfo(p.triangles(tri)) for p in (free, tight))
    assert torch.equal(nt, nt0)
    ok = nt0 > 0
    assert torch.all(torch.isnan(km[~ok])) and torch.any(ok)
    assert torch.all((km[ok] - km0[ok]).abs() <= 4096 * 2.0 ** -52 * km0[ok])


# the upper half of the route's range: the headline's 127, sides of more than 192 points along
# z (135), blocks of 64 pairs (150, 159), and the first value past it (both plans enumerate).
# Thin shells keep the enumeration short: fewer than 4096 batches, as above.
@pytest.mark.parametrize("q", [127, 135, 150, 159, 160])
def test_large_q_equal_enumeration(cuda, q):
    n, box = 512, 900.0
    edges = np.array([[1.0, 3.0], [0.6 * q, 0.6 * q + 2.2], [q - 4.1, q + 0.4]])
    edges *= 2 * np.pi / box
    tri = np.array([(a, b, c) for a in range(3) for b in range(a + 1) for c in range(b + 1)])
    free = Plan(n, box, edges, grid="single")
    assert free.qmax == q
    tight = Plan(n, box, edges, grid="single", mem_budget=free.footprint() + (1 << 20))
    (nt, km), (nt0, km0) = (p.gridinfo(p.triangles(tri)) for p in (free, tight))
    free.sync_check()
    assert torch.equal(nt, nt0) and torch.any(nt0 > 0) and torch.any(nt0 == 0)
    ok = nt0 > 0
    assert torch.all(torch.isnan(km[~ok]))
    assert torch.all((km[ok] - km0[ok]).abs() <= 4096 * 2.0 ** -52 * km0[ok])
    free.close()
    tight.close()
