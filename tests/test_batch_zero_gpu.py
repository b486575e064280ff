"""The batched launch overwrites every image: sizes from one sample to more than its zeroing
kernel covers at once, jobs with and without traces, images of NaNs."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(1, 1, 1)], [(3, 5, 41), (1, 1, 1), (64, 64, 300)], [(300, 200, 101)] + [(2, 2, 64)] * 40,
                                   [(200, 200, 401)]])
def test_images_are_overwritten(cuda, ktm_lib, sizes):
    import torch

    import ktm
    g = torch.Generator(device=cuda)
    g.manual_seed(len(sizes))
    packed = ktm.prepare(torch.randn((5, 100), device=cuda, generator=g), 0.004, rho=0)
    c = [torch.rand(5, device=cuda, generator=g) * 100.0 for _ in range(4)]
    jobs = []
    for i, (nx, ny, nz) in enumerate(sizes):
        n = 5 if i % 2 == 0 else 1
        traces = ktm.PackedTraces(packed.data[:n], packed.scale[:n], packed.nt, packed.fmt, packed.prefolded, packed.rho)
        jobs.append(dict(imageX=(nx, 25.0, 0.0), imageY=(ny, 25.0, 0.0), imageZ=(nz, 0.002, 0.0), dt=0.004,
                         midX=c[0][:n], midY=c[1][:n], offX=c[2][:n], offY=c[3][:n], traces=traces,
                         velocity=torch.full((nz,), 2000.0, device=cuda), pick="linear",
                         image=torch.full((nx, ny, nz), float("nan"), device=cuda)))
    got = ktm.migrate_batch(jobs)
    for job, image in zip(jobs, got):
        want = ktm.migrate(**dict(job, image=torch.empty_like(image)))
        # at most five terms a sample, one slice each: the same sums
        assert torch.allclose(image, want, rtol=1e-6, atol=1e-7 * float(want.abs().max()) + 1e-30)
