"""The fast kernel's chunk pipeline and step-by-step walk at their edges, against the FP64
oracle: trace counts around a chunk and its buffers (three, two and one of them), runs whose
last steps lie past the image or past the trace end, column counts around a CTA's, every
weight, and chunk caps.  Images do not depend on the chunk, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _case(seed, ntr, nt, nx, nz, dz, spread=900.0):
    rng = np.random.default_rng(seed)
    g = oracle.grid(nx, 30.0, -30.0 * nx / 2), oracle.grid(1, 25.0, 0.0), oracle.grid(nz, dz, 0.0)
    c = [rng.uniform(-spread, spread, ntr).astype(np.float32) for _ in range(2)]
    zero = np.zeros(ntr, np.float32)
    j = np.arange(nt)
    tr = sum(rng.standard_normal((ntr, 1)) * np.cos(w * j + rng.uniform(0, 6, (ntr, 1)))
             for w in (0.2, 0.33, 0.5)).astype(np.float32)
    vel = np.linspace(1500.0, 3000.0, nz).astype(np.float32)
    return g, c[0], zero, c[1], zero, tr, vel


def _run(dev, case, weight="prefold", fmt="f32", **kw):
    import torch

    import ktm
    g, mx, my, ox, oy, tr, vel = case
    t = [torch.as_tensor(a).to(dev) for a in (mx, my, ox, oy, vel, tr)]
    packed = ktm.prepare(t[5], 0.004, fmt=fmt, rho=0, prefold=weight == "prefold")
    return ktm.migrate(imageX=g[0], imageY=g[1], imageZ=g[2], dt=0.004, midX=t[0], midY=t[1],
                       offX=t[2], offY=t[3], velocity=t[4], traces=packed, weight=weight,
                       **kw).cpu().numpy()


# u = t / dt carries about 2^-22 relative error from the approximate square roots: at 700
# samples 1.7e-4 of a sample, times a slope of at most 0.5 per sample and amplitude
REL = 2e-4


@pytest.mark.parametrize("weight", ["prefold", "table", "sqrt"])
@pytest.mark.parametrize("ntr,nt,nx,nz,dz", [(1, 700, 1, 512, 0.002), (33, 700, 25, 513, 0.002),
                                             (97, 300, 24, 1000, 0.002), (200, 120, 5, 385, 0.001),
                                             (64, 701, 23, 65, 0.02), (70, 5000, 3, 300, 0.002)])
def test_edges(cuda, ktm_lib, ntr, nt, nx, nz, dz, weight):
    case = _case(ntr + nz, ntr, nt, nx, nz, dz)
    g, mx, my, ox, oy, tr, vel = case
    want = oracle.migrate_f64(*g, 0.004, mx, my, ox, oy, tr, vel, pick=1,
                              prefold={"prefold": 1, "table": 0, "sqrt": 0}[weight], aperture=700.0)
    base = _run(cuda, case, weight, aperture=700.0)
    rel = np.linalg.norm(base - want) / max(np.linalg.norm(want), 1e-30)
    assert rel <= REL * max(1.0, nt / 700.0), rel
    for kw in ({"tile_chunk": 1}, {"tile_chunk": 5}, {"tile_run": 512}, {"tile_run": 384}, {"tile_run": 256}):
        got = _run(cuda, case, weight, aperture=700.0, **kw)
        if "tile_chunk" in kw:
            assert np.array_equal(got.view(np.uint32), base.view(np.uint32)), kw
        # the trace slices, and so the order of the sums, follow the run
        assert np.linalg.norm(got - base) <= 3e-6 * np.linalg.norm(base), kw
    again = _run(cuda, case, weight, aperture=700.0)
    assert np.array_equal(again.view(np.uint32), base.view(np.uint32))


def test_one_buffer(cuda, ktm_lib):
    """The longest traces leave room for a single row buffer beside the tables; a sample
    more and the call is refused as before."""
    import ktm
    longest = max(n for n in range(14000, 15000)
                  if 2 * 4 * ktm.packed_pitch(n, "f32") + 48 + 8 * (n + 1) <= 227 * 1024)
    case = _case(3, 9, longest, 2, 130, 0.05)
    g, mx, my, ox, oy, tr, vel = case
    want = oracle.migrate_f64(*g, 0.004, mx, my, ox, oy, tr, vel, pick=1, prefold=0, aperture=0.0)
    got = _run(cuda, case, "table")
    assert np.linalg.norm(got - want) <= REL * longest / 700.0 * np.linalg.norm(want)
    with pytest.raises(ktm.KtmError):
        _run(cuda, _case(3, 2, longest + 4, 2, 30, 0.05), "table")


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("fmt,weight,lo,hi", [("f32", "prefold", 28774, 28818), ("f32", "sqrt", 28774, 28818),
                                              ("f32", "table", 14386, 14410), ("f16", "table", 19182, 19212),
                                              ("bf16", "table", 19182, 19212)])
def test_every_length_around_the_last_two_buffers(cuda, ktm_lib, fmt, weight, lo, hi, batch):
    """From two buffers beside the warps' tables to one, every trace length on the way."""
    import torch

    import ktm
    rel = {"f32": 0.0, "f16": 6e-4, "bf16": 4e-3}[fmt]             # storage: half an ulp of the largest sample
    for nt in range(lo, hi, 1 if not batch else 2):
        case = _case(nt, 3, nt, 2, 40, 0.3)
        g, mx, my, ox, oy, tr, vel = case
        want = oracle.migrate_f64(*g, 0.004, mx, my, ox, oy, tr, vel, pick=1,
                                  prefold={"prefold": 1, "table": 0, "sqrt": 0}[weight], aperture=0.0)
        if batch:
            t = [torch.as_tensor(a).to(cuda) for a in (mx, my, ox, oy, vel, tr)]
            packed = ktm.prepare(t[5], 0.004, fmt=fmt, rho=0, prefold=weight == "prefold")
            job = dict(imageX=g[0], imageY=g[1], imageZ=g[2], dt=0.004, midX=t[0], midY=t[1], offX=t[2], offY=t[3],
                       velocity=t[4], traces=packed, weight=weight, image=torch.empty(want.shape, device=cuda))
            got = ktm.migrate_batch([job])[0].cpu().numpy()
        else:
            got = _run(cuda, case, weight, fmt)
        assert np.linalg.norm(got - want) <= (REL * nt / 700.0 + rel) * np.linalg.norm(want), nt


@pytest.mark.parametrize("weight,pick", [("prefold", "linear"), ("table", "linear"), ("sqrt", "truncate")])
@pytest.mark.parametrize("run", [256, 384, 512])
@pytest.mark.parametrize("ntr,nt,nx,nz,aperture", [(50, 300, 7, 700, 0.0), (333, 260, 30, 515, 400.0), (1, 90, 1, 64, 0.0)])
def test_counts_the_pairs_it_evaluates(cuda, ktm_lib, ntr, nt, nx, nz, aperture, run, weight, pick):
    """Prefolded samples: each kept trace up to the last 64-sample step that starts before its end;
    the other weights: the whole run.  The kernel's bound lies 1e-4 and a sample past the end."""
    import torch
    g, mx, my, ox, oy, tr, vel = _case(ntr + nz, ntr, nt, nx, nz, 0.002)
    vel[:] = 2000.0
    counter = torch.zeros(1, dtype=torch.int64, device=cuda)
    _run(cuda, (g, mx, my, ox, oy, tr, vel), weight, "f32", pick=pick, aperture=aperture, tile_run=run, pairs_counter=counter)
    x = np.float64(g[0].imageStart) + np.float64(g[0].imageStep) * np.arange(nx)
    tau = np.float64(np.float32(0.002)) * np.arange(nz)
    bounds = []
    for sign in (-1.0, 1.0):
        total = 0
        for c in range(nx):
            d = mx.astype(np.float64) - x[c]
            ok = np.abs(d) <= aperture * (1.0 + sign * 1e-6) if aperture else np.full(ntr, True)
            u = sum(np.sqrt(tau ** 2 + ((d + s * ox)[:, None] / 2000.0) ** 2) for s in (-1.0, 1.0)) / np.float64(np.float32(0.004))
            early = u < (nt * 1.0001 + 1.0) * (1.0 + sign * 1e-5)
            for r0 in range(0, nz, run):
                valid = min(run, nz - r0)
                steps = early[:, r0:r0 + run:64].sum(1)
                per = np.minimum(64 * steps, valid) if weight == "prefold" else np.where(steps > 0, valid, 0)
                total += int(per[ok].sum())
        bounds.append(total)
    assert bounds[0] <= int(counter[0]) <= bounds[1], (bounds, int(counter[0]))
    assert bounds[1] - bounds[0] <= 0.02 * bounds[1] + 512
