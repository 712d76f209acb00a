"""Shell fields at every compiled length of the field synthesis, and at run-time ones, against
an FP64 inverse transform of the same masked spectrum.

Lengths differ in their radices, lines per warp, ragged rounds and row pitch; shells of small,
middle and largest radius and one covering most modes differ in which inputs are zero.  Two
FP32 transforms (the mesh's and the synthesis) each err by at most about 2^-24 log2(points) of
the field's norm: 2^-24 (3 log2 Nmesh + 3 log2 Ng).
"""
import math

import numpy as np
import pytest
import torch

from bskit_gb300.engine import Plan

pytestmark = pytest.mark.gpu

COMPILED = [20, 32, 36, 40, 48, 60, 64, 72, 80, 96, 100, 108, 120, 128, 144, 160, 180, 192, 200,
            216, 240, 256, 288, 300, 320, 360, 384, 400, 480, 512]


@pytest.mark.parametrize("ng", COMPILED + [16, 24, 324])
@pytest.mark.parametrize("native", [False, True])
def test_fields(cuda, ng, native):
    if native and ng > 256:
        pytest.skip("the reduced case covers the length; native adds |q| up to N / 2")
    box = 100.0
    kf = 2 * math.pi / box
    qmax = ng // 2 if native else (ng - 1) // 3
    n = ng if native else ng + 6 + ng % 4
    e = np.array([[0.9, 1.1], [0.3 * qmax, 0.45 * qmax], [0.45 * qmax, 0.9 * qmax],
                  [0.95 * qmax, 0.9999 * qmax + 1e-3]]) * kf
    plan = Plan(n, box, e, grid="native" if native else "single")
    if plan.ngrid != ng:
        pytest.skip("the grid rule takes a smaller side")
    g = torch.Generator(device="cuda")
    g.manual_seed(ng)
    mesh = torch.randn((n, n, n), generator=g, device="cuda")
    plan.paint(0, mesh)
    fine = torch.fft.rfftn(mesh.double(), norm="forward")
    q = torch.fft.fftfreq(ng, 1.0 / ng, device="cuda", dtype=torch.float64)
    i = q.round().long() % n
    h = ng // 2 + 1
    spec = fine[i][:, i][:, :, :h]
    k = q * kf
    z = torch.arange(h, device="cuda", dtype=torch.float64) * kf
    kk = (k[:, None, None] ** 2 + k[None, :, None] ** 2 + z[None, None, :] ** 2).sqrt()
    bound = 2.0 ** -24 * 3 * (math.log2(n) + math.log2(ng))
    for s, (lo, hi) in enumerate(e):
        want = torch.fft.irfftn(torch.where((kk >= lo) & (kk <= hi), spec, 0.0), s=(ng,) * 3,
                                norm="forward")
        got = plan.field(0, s).double()
        assert torch.linalg.norm(got - want) <= bound * torch.linalg.norm(want), (ng, native, s)
    plan.close()


# The largest |q| itself: N / 2 on the mesh's own grid (every frequency kept, the Nyquist planes
# among them), (N - 1) // 3 on a reduced one, which reaches the sides that the last shell above
# stays below.
@pytest.mark.parametrize("ng", COMPILED + [16, 24, 324])
@pytest.mark.parametrize("native", [False, True])
def test_fields_at_the_largest_q(cuda, ng, native):
    box = 100.0
    kf = 2 * math.pi / box
    qmax = ng // 2 if native else (ng - 1) // 3
    n = ng if native else ng + 6 + ng % 4
    e = np.array([[0.4 * qmax, 0.6 * qmax], [0.8 * qmax, qmax + 1e-3]]) * kf
    plan = Plan(n, box, e, grid="native" if native else "single")
    if plan.ngrid != ng:
        plan.close()
        pytest.skip("the grid rule takes a smaller side")
    assert plan.qmax == qmax
    g = torch.Generator(device="cuda")
    g.manual_seed(ng)
    mesh = torch.randn((n, n, n), generator=g, device="cuda")
    plan.paint(0, mesh)
    fine = torch.fft.rfftn(mesh.double(), norm="forward")
    q = torch.fft.fftfreq(ng, 1.0 / ng, device="cuda", dtype=torch.float64)
    i = q.round().long() % n
    h = ng // 2 + 1
    spec = fine[i][:, i][:, :, :h]
    del fine
    k = q * kf
    z = torch.arange(h, device="cuda", dtype=torch.float64) * kf
    kk = (k[:, None, None] ** 2 + k[None, :, None] ** 2 + z[None, None, :] ** 2).sqrt()
    bound = 2.0 ** -24 * 3 * (math.log2(n) + math.log2(ng))
    for s, (lo, hi) in enumerate(e):
        want = torch.fft.irfftn(torch.where((kk >= lo) & (kk <= hi), spec, 0.0), s=(ng,) * 3,
                                norm="forward")
        got = plan.field(0, s).double()
        assert torch.linalg.norm(got - want) <= bound * torch.linalg.norm(want), (ng, native, s)
    plan.close()
