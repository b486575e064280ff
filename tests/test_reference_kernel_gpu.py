"""The reference-mode kernel at the edges of its work split, bit-identical to the oracle
restatement of psktmCPU.c: runs of 32 R tau samples for each R, column counts around a CTA's,
odd and single traces, chunk remainders, traces of 1 to 3 samples, rows that are longer than
their samples and start at every 4-byte offset, and operands on both sides of the ranges its
packed square roots and quotients take."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import same_with_nans

pytestmark = pytest.mark.gpu


def _case(seed, ntr, nt, nx, ny, nz, dt=0.004, spread=300.0, z0=0.0, v0=1500.0, stride=None):
    rng = np.random.default_rng(seed)
    gx, gy = oracle.grid(nx, 30.0, -60.0), oracle.grid(ny, 25.0, -20.0)
    gz = oracle.grid(nz, dt / 2.0, z0)
    c = [rng.uniform(-spread, spread, ntr).astype(np.float32) for _ in range(4)]
    tr = rng.standard_normal((ntr, stride or nt)).astype(np.float32)
    return gx, gy, gz, dt, c, tr, np.linspace(v0, 2.0 * v0, nz).astype(np.float32)


def _run(dev, case, nt=None, shift=0, run=0, start=None):
    import torch

    import ktm
    gx, gy, gz, dt, c, tr, vel = case
    ntr, stride = tr.shape
    buf = torch.zeros(ntr * stride + 4, device=dev)
    rows = buf[shift:shift + ntr * stride].view(ntr, stride)
    rows.copy_(torch.as_tensor(tr))
    up = [torch.as_tensor(a).to(dev) for a in c]
    img = None if start is None else torch.as_tensor(start).to(dev)
    job = ktm.Job(imageX=gx, imageY=gy, imageZ=gz, dt=dt, midX=up[0], midY=up[1], offX=up[2],
                  offY=up[3], traces=rows, velocity=torch.as_tensor(vel).to(dev), image=img,
                  mode="reference", pick="truncate", tile_run=run, accumulate=start is not None)
    if nt is not None:
        job.job.config.tracePts, job.job.traceStride = nt, stride
    return job.run().cpu().numpy()


def _oracle(case, nt=None):
    gx, gy, gz, dt, c, tr, vel = case
    return oracle.migrate_ref32(gx, gy, gz, dt, *c, np.ascontiguousarray(tr[:, :nt]), vel)


@pytest.mark.parametrize("run", [0, 32, 64, 128, 256, 512])
@pytest.mark.parametrize("ntr,nt,nx,ny,nz", [(1, 130, 1, 1, 1), (2, 1, 3, 1, 33), (33, 2, 5, 3, 32),
                                             (65, 131, 17, 1, 129), (70, 401, 11, 3, 127),
                                             (31, 3, 33, 2, 64), (37, 2003, 9, 2, 300)])
def test_sizes(cuda, ktm_lib, run, ntr, nt, nx, ny, nz):
    case = _case(ntr + nz, ntr, nt, nx, ny, nz, z0=0.001 if nz < 32 else 0.0)
    assert same_with_nans(_run(cuda, case, run=run), _oracle(case))


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("nt,stride", [(141, 141), (140, 140), (140, 141), (139, 160), (28924, 28924)])
def test_row_layouts(cuda, ktm_lib, shift, nt, stride):
    case = _case(shift + nt, 21 if nt < 1000 else 3, nt, 5, 3, 101, stride=stride)
    assert same_with_nans(_run(cuda, case, nt=nt, shift=shift), _oracle(case, nt))


def test_limit_kept(cuda, ktm_lib):
    import ktm
    with pytest.raises(ktm.KtmError):
        _run(cuda, _case(3, 2, 28925, 2, 1, 5))


@pytest.mark.parametrize("dt", [1e-6, 3e-5, 0.00199, 0.01, 1.7, 1023.0, 1.1e3, 5e-7])
def test_sample_intervals(cuda, ktm_lib, dt):
    # velocities scaled so that the traveltimes stay within the traces
    case = _case(7, 45, 150, 7, 2, 70, dt=dt, v0=max(30.0, min(1e6, 6.0 / dt)))
    assert same_with_nans(_run(cuda, case), _oracle(case))


@pytest.mark.parametrize("spread", [0.0, 1e-5, 1e-3, 3e6, 1e9])
def test_distances(cuda, ktm_lib, spread):
    """Zero, tiny and huge distances, inside and outside the packed ranges, some traces
    among ordinary ones."""
    case = _case(9, 67, 150, 4, 2, 140)
    c = case[4]
    rng = np.random.default_rng(3)
    far = rng.uniform(size=67) < 0.2
    for i in range(4):
        c[i][far] = rng.uniform(-spread, spread, int(far.sum())) if spread else 0.0
    c[0][5], c[1][5], c[2][5], c[3][5] = -60.0, -20.0, 0.0, 0.0     # on an image column
    assert same_with_nans(_run(cuda, case), _oracle(case))


def test_special_samples_at_zero_tau_and_accumulation(cuda, ktm_lib):
    """Infinite and NaN samples where tau = 0 (0 * inf) and finite ones elsewhere; a second
    image added to a first one, negative zeros in it included."""
    case = _case(11, 40, 160, 5, 3, 96)
    case[5][7, 20:] = np.inf
    case[5][9, 90:] = np.nan
    ref = _oracle(case)
    assert np.isnan(ref[:, :, 0]).any()
    assert same_with_nans(_run(cuda, case), ref)
    start = np.random.default_rng(1).standard_normal(ref.shape).astype(np.float32)
    start[0, 0, :3] = -0.0
    with np.errstate(invalid="ignore"):
        assert same_with_nans(_run(cuda, case, start=start.copy()), start + ref)


@pytest.mark.parametrize("run", [0, 32, 64])
@pytest.mark.parametrize("nt,nx,ny,nz", [(28856, 40, 1, 40), (28900, 80, 50, 64), (28924, 74, 64, 64), (28924, 60, 50, 1),
                                         (28900, 25, 1, 129), (28880, 500, 2, 33)])
def test_longest_traces_of_wide_images(cuda, ktm_lib, nt, nx, ny, nz, run):
    """The longest accepted traces leave room for fewer warps' tables than an SM has warps."""
    case = _case(nt + nx, 2, nt, nx, ny, nz, dt=0.001)
    assert same_with_nans(_run(cuda, case, run=run), _oracle(case))
