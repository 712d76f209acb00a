"""The work that users of this framework have it do, as cases that can be timed and checked.

A case is one measurement on a prepared plan, the way a measurement script or the serving
loop runs it for every new mesh: transform the mesh(es) (``Plan.paint``, ``paint_subbox``),
then the unnormalised bispectrum of every bin of a triangle set (``Plan.measure_b``).  The
plan and the triangle set are kept between meshes.  The grid information (exact triangle
counts and mean |k| per bin, ``Plan.gridinfo``) is measured once per binning and is a case
of its own.

Keys of a case:
  kind      "b" (paint + bispectrum), "subbox" (every sub-box of a mesh), "gridinfo"
  n         mesh points per side            box    box side in Mpc/h
  kmax, dk  largest wavenumber and bin width in units of the fundamental k_f; bins start at
            k_f
  bins      "all", "equilateral", "squeezed" (k1 in the first bin) or "isosceles" (k_L = k_S / 2)
  fields    1 <AAA>, 2 <AAB>, 3 <ABC>       precision of the contraction
  cic       the meshes carry a CIC assignment window that is deconvolved
  nsub      sub-boxes per side ("subbox")
"""
import math

import numpy as np
import torch

from bskit_gb300 import Plan

SLOTS = {1: (0, 0, 0), 2: (0, 0, 1), 3: (0, 1, 2)}


def _b(name, n, box, kmax, dk, bins="all", fields=1, precision="bf16x3", cic=False):
    return dict(name=name, kind="b", n=n, box=box, kmax=kmax, dk=dk, bins=bins, fields=fields,
                precision=precision, cic=cic)


def listed():
    return [
        # the serving loop's most frequent and smallest request: latency and launches count
        _b("auto64_equilateral", 64, 100.0, 16.0, 2.0, bins="equilateral"),
        # the same mesh with every triangle bin
        _b("auto64_all", 64, 100.0, 16.0, 2.0),
        # serving's <AAB> request at 128^3, with CIC-assigned meshes
        _b("cross128_all_cic", 128, 100.0, 32.0, 2.0, fields=2, cic=True),
        # the 256^3 configuration (31 shells, 3321 bins): an ordinary snapshot
        _b("auto256_all", 256, 500.0, 64.0, 2.0),
        # the same in plain FP32, the arithmetic users compare bf16x3 with
        _b("auto256_all_fp32", 256, 500.0, 64.0, 2.0, precision="fp32"),
        # error bars from the eight sub-boxes of a 256^3 mesh
        dict(name="subbox256_nsub2", kind="subbox", n=256, box=500.0, kmax=32.0, dk=2.0,
             bins="all", fields=1, precision="bf16x3", cic=False, nsub=2),
        # a mesh side and a bin width that are no powers of two (contraction grid 216)
        _b("auto300_ragged", 300, 730.0, 70.5, 3.3),
        # the 512^3 cross precision study's squeezed bins: many fields, few bins
        _b("cross512_squeezed", 512, 1000.0, 128.0, 2.0, bins="squeezed", fields=2),
        # the headline: 512^3, 63 shells, 24305 bins
        _b("auto512_all", 512, 1000.0, 128.0, 2.0),
        # the largest grid: 1024^3 up to 0.3 k_Nyq, 38 shells, 5833 bins
        _b("auto1024_all", 1024, 2000.0, 0.3 * 512, 4.0),
        # the grid information that goes with the 256^3 and the 512^3 binnings
        dict(name="gridinfo256_all", kind="gridinfo", n=256, box=500.0, kmax=64.0, dk=2.0,
             bins="all", fields=1),
        dict(name="gridinfo512_all", kind="gridinfo", n=512, box=1000.0, kmax=128.0, dk=2.0,
             bins="all", fields=1),
    ]


def draw(rng):
    """One more case: mesh sides 48 ... 768, k up to 0.2 ... 0.5 k_Nyq, 4 ... 60 shells of any
    width, every bin set, one to three fields, with grid information for a fifth."""
    kind = rng.choice(["b", "b", "b", "b", "gridinfo"])
    n = 2 * int(round(math.exp(rng.uniform(math.log(24), math.log(384)))))
    kmax = min(round(rng.uniform(0.2, 0.5) * n / 2, 2), 128.0 if kind == "b" else 100.0)
    shells = int(round(math.exp(rng.uniform(math.log(4), math.log(60)))))
    dk = max(1.0, round((kmax - 1.0) / (shells + 0.5), 2))
    c = dict(kind=kind, n=n, box=float(rng.randrange(80, 2000)), kmax=kmax, dk=dk,
             bins=rng.choice(["all", "all", "all", "equilateral", "squeezed", "isosceles"]),
             fields=rng.choice([1, 1, 2, 3]) if kind == "b" else 1)
    if kind == "gridinfo":
        return c
    if c["fields"] == 3 and c["bins"] == "all" and dk < kmax / 30:
        c["fields"] = 2  # every ordered triple of very many shells costs more than the headline
    c["precision"] = rng.choice(["bf16x3", "bf16x3", "bf16x3", "fp32", "bf16"])
    c["cic"] = rng.random() < 0.3
    return c


# ------------------------------------------------------------------ inputs
def _box(case, seed):
    """The box side: the stated one for a mesh; for grid information, which has no mesh, the
    boxes of different snapshots differ a little."""
    return case["box"] * (1.0 + (seed % 89) * 1e-3) if case["kind"] == "gridinfo" else case["box"]


def _plan_size(case, box):
    """Mesh and box side of the plan (a sub-box's for "subbox")."""
    s = case.get("nsub", 1)
    return case["n"] // s, box / s


def _binning(case, box):
    """(shell edges [n][2], triangle bins [T][3]), as bskit's bin-list generators give them."""
    kf = 2.0 * np.pi / _plan_size(case, box)[1]
    kmax, dk = case["kmax"] * kf, case["dk"] * kf
    lower = np.arange(kf, kmax - dk, dk)
    edges = np.stack([lower, lower + dk], axis=1)
    n = len(edges)
    if case["bins"] == "all":
        a, b, c = (v.ravel() for v in np.meshgrid(*[np.arange(n)] * 3, indexing="ij"))
        sel = {1: (a >= b) & (b >= c), 2: a >= b, 3: a >= 0}[case["fields"]]
        a, b, c = a[sel], b[sel], c[sel]
        lo, hi = edges[:, 0], edges[:, 1]
        ok = (hi[a] + hi[b] >= lo[c]) & (hi[a] + hi[c] >= lo[b]) & (hi[b] + hi[c] >= lo[a])
        tri = np.stack([a, b, c], axis=1)[ok]
    elif case["bins"] == "equilateral":
        tri = np.repeat(np.arange(n)[:, None], 3, axis=1)
    elif case["bins"] == "squeezed":
        s = np.arange(1, n)
        tri = np.stack([np.zeros_like(s), s, s], axis=1)
    else:  # isosceles, k_L = k_S / 2: the shell whose mean |k| is nearest, within 10%
        mean = 0.75 * (edges[:, 1] ** 4 - edges[:, 0] ** 4) / (edges[:, 1] ** 3 - edges[:, 0] ** 3)
        dist = np.abs(mean[None, :] - mean[:, None] / 2.0)
        s = np.arange(n)[dist.min(axis=1) / (mean / 2.0) < 0.1]
        tri = np.stack([dist.argmin(axis=1)[s], s, s], axis=1) if len(s) else np.zeros((1, 3), int)
    return edges, np.ascontiguousarray(tri, dtype=np.int32)


def _mesh(n, box, seed):
    """Lognormal density contrast with P(k) = 1e3 (k / 0.1)^-1.5 exp(-(k / 2)^2)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    w = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device="cuda"))
    kf = 2.0 * math.pi / box
    q2 = (torch.fft.fftfreq(n, 1.0 / n, device="cuda") * kf) ** 2
    z2 = (torch.arange(n // 2 + 1, device="cuda") * kf) ** 2
    kk = (q2[:, None, None] + q2[None, :, None] + z2[None, None, :]).sqrt_()
    amp = (kk * 10.0).pow_(-0.75) * torch.exp(-kk * kk / 8.0) * math.sqrt(1e3 * n ** 3 / box ** 3)
    amp[0, 0, 0] = 0.0
    del kk
    w *= amp
    del amp
    w = torch.fft.irfftn(w, s=(n, n, n))
    return torch.exp_(w - 0.5 * w.var()).sub_(1.0).contiguous()


def _meshes(case, seed):
    out = [_mesh(case["n"], case["box"], seed)]
    for k in range(1, case["fields"]):  # a biased, noisy tracer of the first field
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed) + 7919 * k)
        noise = torch.randn(out[0].shape, generator=g, device="cuda")
        out.append(1.5 * out[0] + noise * (0.1 * out[0].var()).sqrt())
    return out


def prepare(case, seed):
    box = _box(case, seed)
    n, l = _plan_size(case, box)
    edges, tri = _binning(case, box)
    plan = Plan(n, l, edges)
    state = {"case": case, "plan": plan, "bins": plan.triangles(tri)}
    if case["kind"] != "gridinfo":
        state["meshes"] = _meshes(case, seed)
    return state


def run(state):
    case, plan, bins = state["case"], state["plan"], state["bins"]
    if case["kind"] == "gridinfo":
        ntri, kmean = plan.gridinfo(bins)
        return {"ntri": ntri, "kmean": kmean}
    if case["kind"] == "subbox":
        s, out = case["nsub"], []
        for box in range(s ** 3):
            plan.paint_subbox(0, state["meshes"][0], (box // (s * s), box // s % s, box % s))
            out.append(plan.measure_b(bins, precision=case["precision"]))
        return out
    for slot, mesh in enumerate(state["meshes"]):
        plan.paint(slot, mesh, cic_nmesh=case["n"] if case["cic"] else None)
    return plan.measure_b(bins, slots=SLOTS[case["fields"]], precision=case["precision"])


# ------------------------------------------------------------------ what a pass needs
def _grid(edges, box, n):
    """The smallest even FFT-friendly side above 3 qmax (no triple of modes wraps around), qmax
    the largest wavevector component of a shell mode."""
    qmax = int(math.floor(edges[-1, 1] / (2.0 * math.pi / box) * (1.0 + 1e-9)))
    for m in range(3 * qmax + 1, n):
        k = m
        for p in (2, 3, 5, 7):
            while k % p == 0:
                k //= p
        if k == 1 and m % 2 == 0:
            return m
    return n


def work(case):
    n, box = _plan_size(case, case["box"])
    edges, tri = _binning(case, case["box"])
    m = float(_grid(edges, box, n)) ** 3
    fft = 2.5 * m * math.log2(m)
    if case["kind"] == "gridinfo":  # count and |k| fields of every shell, four sums per bin
        return {"bytes": 16 * len(edges) + 32 * len(tri),
                "flops": 2 * len(edges) * fft + 8.0 * len(tri) * m}
    times = case.get("nsub", 1) ** 3
    fwd = 2.5 * n ** 3 * math.log2(n ** 3)
    return {"bytes": times * (4.0 * case["fields"] * n ** 3 + 8.0 * len(tri)),
            "flops": times * (case["fields"] * (fwd + len(edges) * fft) + 2.0 * len(tri) * m)}


# ------------------------------------------------------------------ the same in 64 bits
def _shell_masks(edges, box, g, h):
    """|k| on the half grid of side g (last axis 0 .. h - 1), components as FFT frequencies."""
    kf = 2.0 * math.pi / box
    q = torch.fft.fftfreq(g, 1.0 / g, device="cuda", dtype=torch.float64) * kf
    z = torch.arange(h, device="cuda", dtype=torch.float64) * kf
    k2 = q[:, None, None] * q[:, None, None] + q[None, :, None] * q[None, :, None]
    return (k2 + z[None, None, :] * z[None, None, :]).sqrt()


def _triple_sums(pairs, col, rows, cols, tri, k, chunk=1 << 17):
    """sum over k points of f_i f_j f_l per bin; pairs(x0, x1, i or j), col likewise."""
    ij, inv = np.unique(tri[:, :2], axis=0, return_inverse=True)
    i, j = (torch.as_tensor(v.copy(), device="cuda", dtype=torch.long) for v in ij.T)
    acc = torch.zeros((len(ij), cols), dtype=torch.float64, device="cuda")
    for x0 in range(0, k, chunk):
        s = slice(x0, min(k, x0 + chunk))
        p = pairs(0, s).index_select(0, i).mul_(pairs(1, s).index_select(0, j))
        acc += p @ col(s).T
    t = torch.as_tensor(tri[:, 2].copy(), device="cuda", dtype=torch.long)
    return acc[torch.as_tensor(np.asarray(inv).reshape(-1), device="cuda"), t]


def _fields(spec, kk, edges, g):
    out = torch.empty((len(edges), g ** 3), dtype=torch.float64, device="cuda")
    for s, (lo, hi) in enumerate(edges):
        masked = torch.where((kk >= lo) & (kk <= hi), spec, torch.zeros((), dtype=spec.dtype,
                                                                        device="cuda"))
        out[s] = torch.fft.irfftn(masked, s=(g, g, g), norm="forward").reshape(-1)
    return out


def _exact_b(case, meshes, n, box, edges, tri):
    g = _grid(edges, box, n)
    h = g // 2 + 1
    kk = _shell_masks(edges, box, g, h)
    q = torch.fft.fftfreq(g, 1.0 / g, device="cuda").round().long()
    fields = []
    for mesh in meshes:
        fine = torch.fft.rfftn(mesh.double(), norm="forward")
        if case["cic"]:
            s = torch.sin(math.pi * torch.fft.fftfreq(n, 1.0, device="cuda", dtype=torch.float64))
            w = 1.0 / (1.0 - 2.0 / 3.0 * s * s).sqrt()
            fine *= w[:, None, None] * w[None, :, None] * w[None, None, : n // 2 + 1]
        spec = fine if g == n else fine[q % n][:, q % n][:, :, :h].contiguous()
        del fine
        fields.append(_fields(spec, kk, edges, g))
        del spec
    fa, fb, fc = (fields[s] for s in SLOTS[case["fields"]])
    out = _triple_sums(lambda r, s: (fa, fb)[r][:, s], lambda s: fc[:, s], len(edges), len(edges),
                       tri, g ** 3)
    return out * (box ** 6 / float(g) ** 3)


def _exact_gridinfo(case, box, edges, tri):
    """The count and |k| fields are even in every coordinate: one octant of the grid, weighted."""
    g = _grid(edges, box, case["n"])
    h = g // 2 + 1
    kk = _shell_masks(edges, box, g, h)
    w = torch.full((h,), 2.0, dtype=torch.float64, device="cuda")
    w[0] = w[h - 1] = 1.0
    w = (w[:, None, None] * w[None, :, None] * w[None, None, :]).reshape(-1)
    nf = torch.empty((len(edges), h ** 3), dtype=torch.float64, device="cuda")
    kf = torch.empty_like(nf)
    for s, (lo, hi) in enumerate(edges):
        ind = ((kk >= lo) & (kk <= hi)).double()
        for dst, v in ((nf, ind), (kf, ind * kk)):
            f = torch.fft.irfftn(v.to(torch.complex128), s=(g, g, g), norm="forward")
            dst[s] = f[:h, :h, :h].reshape(-1)

    def sums(a, b, c):
        return _triple_sums(lambda r, s: (a, b)[r][:, s], lambda s: c[:, s] * w[s], len(edges),
                            len(edges), tri, h ** 3) / float(g) ** 3
    cnt = torch.round(sums(nf, nf, nf))
    km = torch.stack([sums(kf, nf, nf), sums(nf, kf, nf), sums(nf, nf, kf)], dim=1)
    nan = torch.full((), math.nan, dtype=torch.float64, device="cuda")
    return {"ntri": cnt, "kmean": torch.where(cnt[:, None] > 0, km / cnt[:, None], nan)}


def exact(case, seed):
    box = _box(case, seed)
    n, l = _plan_size(case, box)
    edges, tri = _binning(case, box)
    pairs, g = len(np.unique(tri[:, :2], axis=0)), _grid(edges, l, n)
    flops = 2.0 * pairs * len(edges) * float(g) ** 3 * case.get("nsub", 1) ** 3
    if (0.5 * flops if case["kind"] == "gridinfo" else flops) > 1e13:
        return None  # over about 20 s in FP64
    if case["kind"] == "gridinfo":
        return _exact_gridinfo(case, box, edges, tri)
    meshes = _meshes(case, seed)
    if case["kind"] == "subbox":
        s, out = case["nsub"], []
        for b in range(s ** 3):
            at = [v * n for v in (b // (s * s), b // s % s, b % s)]
            part = meshes[0][at[0]:at[0] + n, at[1]:at[1] + n, at[2]:at[2] + n].contiguous()
            out.append(_exact_b(case, [part], n, l, edges, tri))
        return out
    return _exact_b(case, meshes, n, l, edges, tri)
