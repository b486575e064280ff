"""Demigration with a row per warp against the rows shared by a CTA (the same velocity given
as a cube takes those): both evaluate every pair with the same code, so they differ by the
order of FP32 sums alone.  Sizes around a run of 256 samples, a CTA's traces and column blocks;
every weight; regular lines, whose zero-offset traces step by exactly one sample; coarse and
fine tau steps; velocities that turn, jump, vanish or are not numbers; accumulation."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(dev, c, cube, start=None, weight="prefold"):
    import torch

    import ktm
    from ktm._lib import check, lib
    gx, gz, nt, mx, my, ox, oy, vel, img, ap = c
    t = [torch.as_tensor(a).to(dev) for a in (mx, my, ox, oy)]
    v = torch.as_tensor(vel).to(dev)
    if cube:
        v = v.expand(gx[0], 1, gz[0]).contiguous()
    pitch = ktm.packed_pitch(nt, "f32") + 4
    data = torch.full((len(mx), pitch), 3.0, device=dev) if start is None else torch.as_tensor(start).to(dev)
    traces = ktm.PackedTraces(data, torch.ones(len(mx), device=dev), nt, "f32", False, 0)
    job = ktm.Job(imageX=gx, imageY=(1, 1.0, 0.0), imageZ=gz, dt=0.004, midX=t[0], midY=t[1], offX=t[2],
                  offY=t[3], velocity=v, traces=traces, image=torch.as_tensor(img).to(dev), weight=weight,
                  aperture=ap, accumulate=start is not None)
    check(lib().ktmDemigrate(C.byref(job.job), data.data_ptr(), pitch))
    return data.cpu().numpy()


def _case(seed, nx, ntr, nt, nz, dz, ap=0.0, line=False, vel=None):
    rng = np.random.default_rng(seed)
    gx, gz = (nx, 12.5, 0.0), (nz, dz, 0.0)
    zero = np.zeros(ntr, np.float32)
    if line:
        mx = (12.5 * (np.arange(ntr) % nx)).astype(np.float32)
        ox = (25.0 * (np.arange(ntr) // nx)).astype(np.float32)
    else:
        mx = rng.uniform(0, 12.5 * nx, ntr).astype(np.float32)
        ox = rng.uniform(-600, 600, ntr).astype(np.float32)
    if vel is None:
        vel = np.linspace(1500.0, 3200.0, nz)
    img = rng.standard_normal((nx, 1, nz)) * (rng.uniform(size=(nx, 1, nz)) < 0.5)
    img[nx // 2] = 0.0
    return gx, gz, nt, mx, zero, ox, zero.copy(), vel.astype(np.float32), img.astype(np.float32), ap


def _same(a, b):
    # at most some hundred summands a sample, FP32 rounding 6e-8 each, in another order
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    f = np.isfinite(b)
    assert np.linalg.norm(a[f] - b[f]) <= 2e-6 * np.linalg.norm(b[f])


@pytest.mark.parametrize("weight", ["prefold", "table", "sqrt"])
@pytest.mark.parametrize("nx,ntr,nt,nz,dz,ap,line", [
    (1, 1, 2, 1, 0.002, 0.0, False), (3, 7, 300, 255, 0.002, 0.0, False), (33, 17, 301, 256, 0.002, 150.0, False),
    (70, 9, 500, 257, 0.002, 0.0, True), (40, 120, 260, 600, 0.001, 0.0, True), (65, 33, 400, 300, 0.004, 300.0, True),
    (20, 50, 900, 200, 0.009, 0.0, False), (12, 40, 2300, 700, 0.002, 0.0, True)])
def test_rows_against_shared_rows(cuda, ktm_lib, nx, ntr, nt, nz, dz, ap, line, weight):
    c = _case(nx + ntr, nx, ntr, nt, nz, dz, ap, line)
    a, b = _run(cuda, c, False, weight=weight), _run(cuda, c, True, weight=weight)
    _same(a, b)
    assert np.all(a[:, 0] == 0) and np.all(a[:, nt:] == 0)


@pytest.mark.parametrize("kind", ["falling", "steps", "noise", "odd"])
def test_velocities(cuda, ktm_lib, kind):
    """Traveltimes that go back, jump by samples, or are not numbers."""
    rng = np.random.default_rng(5)
    nz = 520
    vel = np.linspace(1500.0, 3000.0, nz)
    if kind == "falling":
        vel = vel[::-1].copy()
    elif kind == "steps":
        vel[100:] *= 0.5
        vel[300:] *= 3.0
    elif kind == "noise":
        vel *= rng.uniform(0.7, 1.4, nz)
    else:
        vel[40], vel[200], vel[333], vel[400], vel[500] = 0.0, np.nan, np.inf, -1800.0, 1e30
    c = _case(8, 37, 90, 400, nz, 0.002, vel=vel)
    _same(_run(cuda, c, False), _run(cuda, c, True))


@pytest.mark.parametrize("ntr", [5, 3000])
def test_accumulates(cuda, ktm_lib, ntr):
    """Onto given data, with several column blocks (few traces) and with one."""
    c = _case(9, 70, ntr, 300, 280, 0.002)
    plain = _run(cuda, c, False)
    start = np.random.default_rng(1).standard_normal(plain.shape).astype(np.float32)
    _same(_run(cuda, c, False, start=start.copy()), start + plain)


@pytest.mark.parametrize("weight", ["prefold", "table"])
@pytest.mark.parametrize("nx,ntr,nz,dz", [(40, 9, 300, 0.002), (40, 10, 300, 0.002), (256, 10, 70, 0.002), (257, 63, 70, 0.002),
                                          (257, 64, 70, 0.002), (30, 40, 33, 0.004)])
def test_either_side_of_the_rules(cuda, ktm_lib, nx, ntr, nz, dz, weight):
    """Few traces, few samples: whichever kernel takes the call, the sums are the same."""
    c = _case(nx + ntr, nx, ntr, 300, nz, dz)
    _same(_run(cuda, c, False, weight=weight), _run(cuda, c, True, weight=weight))


def test_the_limit_is_every_calls(cuda, ktm_lib):
    """Rows longer than shared memory are refused whatever kernel would take the call."""
    import torch

    import ktm
    from ktm._lib import lib
    c = _case(3, 20, 40, 300, 100, 0.002)
    gx, gz, nt, mx, my, ox, oy, vel, img, ap = c
    t = [torch.as_tensor(a).to(cuda) for a in (mx, my, ox, oy, vel, img)]
    for pitch, ok in ((46000, True), (47000, False)):
        data = torch.zeros((40, pitch), device=cuda)
        job = ktm.Job(imageX=gx, imageY=(1, 1.0, 0.0), imageZ=gz, dt=0.004, midX=t[0], midY=t[1], offX=t[2], offY=t[3],
                      velocity=t[4], traces=ktm.PackedTraces(data, torch.ones(40, device=cuda), nt, "f32", False, 0),
                      image=t[5], weight="prefold")
        rc = lib().ktmDemigrate(C.byref(job.job), data.data_ptr(), pitch)
        assert rc == (0 if ok else ktm._lib.KTM_ERR_LIMIT)
