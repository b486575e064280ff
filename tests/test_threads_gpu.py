"""Host threads whose calls use the same kernels at different sizes, each on a stream of its own:
every call runs and gives what it gives alone."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _calls(dev, kind, nt):
    import torch

    import ktm
    from ktm import inverse
    rng = np.random.default_rng(nt)
    ntr, nx, nz = 3, 40, 64
    c = [torch.as_tensor(rng.uniform(0, 300, ntr).astype(np.float32)).to(dev) for _ in range(2)]
    zero = torch.zeros(ntr, device=dev)
    kw = dict(imageX=(nx, 10.0, 0.0), imageY=(1, 1.0, 0.0), imageZ=(nz, 0.002, 0.0), dt=0.004, midX=c[0], midY=zero,
              offX=c[1], offY=zero, velocity=torch.full((nz,), 2000.0, device=dev))
    traces = torch.as_tensor(rng.standard_normal((ntr, nt)).astype(np.float32)).to(dev)
    stream = torch.cuda.Stream(dev)
    if kind == "demigrate":
        image = torch.ones((nx, 1, nz), device=dev)
        op = inverse.MigrationOperator(**kw, nt=nt, stream=stream, aperture=0.0, weight="table")
        out = torch.empty((ntr, op.pitch), device=dev)
        return stream, (lambda: op.demigrate(image, out)), out
    image = torch.empty((nx, 1, nz), device=dev)
    if kind == "reference":
        job = ktm.Job(**kw, traces=traces, image=image, mode="reference", pick="truncate", stream=stream)
    else:
        job = ktm.Job(**kw, traces=ktm.prepare(traces, 0.004, rho=0), image=image, weight="table", stream=stream)
    return stream, job.run, image


@pytest.mark.parametrize("kind,sizes", [("fast", (9000, 5000, 2000)), ("reference", (20000, 9000, 3000)),
                                        ("demigrate", (9000, 3000, 1000))])
def test_threads_of_different_sizes(cuda, ktm_lib, kind, sizes):
    import torch
    calls = [_calls(cuda, kind, nt) for nt in sizes for _ in range(2)]
    alone = []
    for stream, run, out in calls:
        torch.cuda.synchronize()
        run()
        torch.cuda.synchronize()
        alone.append(out.clone())
    failed = []

    def work(run):
        try:
            for _ in range(400):
                run()
        except Exception as e:                      # reported below
            failed.append(e)

    threads = [threading.Thread(target=work, args=(run,)) for _, run, _ in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed[0]
    for (_, _, out), want in zip(calls, alone):
        # column blocks of a demigration are added in any order
        assert torch.equal(out, want) if kind != "demigrate" else torch.allclose(out, want, rtol=1e-4, atol=1e-4)
