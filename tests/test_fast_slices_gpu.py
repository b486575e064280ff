"""Trace slices of the fast migration: their partial images stay within 256 MiB whatever
the image, and a call for which they do not fit into the device's memory runs without them."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _job(dev, nx, ny, nz, ntr, nt):
    import torch

    import ktm
    g = torch.Generator(device=dev)
    g.manual_seed(nx + ntr)
    c = [torch.rand(ntr, device=dev, generator=g) * 2000.0 for _ in range(4)]
    packed = ktm.prepare(torch.randn((ntr, nt), device=dev, generator=g), 0.004, fmt="f16", rho=0)
    return ktm.Job(imageX=(nx, 25.0, 0.0), imageY=(ny, 25.0, 0.0), imageZ=(nz, 0.002, 0.0), dt=0.004, midX=c[0],
                   midY=c[1], offX=c[2], offY=c[3], velocity=torch.full((nz,), 2500.0, device=dev), traces=packed,
                   image=torch.empty((nx, ny, nz), device=dev), pick="linear")


def _reserved():
    from ktm._lib import memory_stats
    return memory_stats()["reserved"]


@pytest.mark.parametrize("nx,ny,nz,ntr,nt", [(200, 200, 1501, 2500, 90), (100, 150, 1501, 10000, 100), (700, 1, 300, 50000, 60),
                                             (200, 100, 1000, 30000, 40)])
def test_partial_images_are_bounded(cuda, ktm_lib, nx, ny, nz, ntr, nt):
    import torch

    from ktm._lib import check
    job = _job(cuda, nx, ny, nz, ntr, nt)
    torch.cuda.synchronize()
    check(ktm_lib.ktmReleaseMemory())
    before = _reserved()
    job.run()
    torch.cuda.synchronize()
    # the pool maps its memory in pieces of 32 MiB
    assert _reserved() - before <= 256 * MB + 32 * MB


def test_without_room_for_partial_images(cuda, ktm_lib):
    """The device's memory taken but for a few MiB: the image comes from one slice."""
    import torch

    from ktm._lib import check, memory_stats
    job = _job(cuda, 100, 100, 1001, 4000, 300)
    want = job.run().clone()
    torch.cuda.synchronize()
    assert memory_stats()["allocations"] > 0
    check(ktm_lib.ktmReleaseMemory())
    torch.cuda.empty_cache()
    taken, size = [], 1 << 34
    try:
        while size >= 2 * MB:
            try:
                taken.append(torch.empty(size, dtype=torch.uint8, device=cuda))
            except torch.cuda.OutOfMemoryError:
                size //= 2
        assert torch.cuda.mem_get_info()[0] < 64 * MB          # less than two partial images
        job.run()
        torch.cuda.synchronize()
    finally:
        taken.clear()
        torch.cuda.empty_cache()
    got, want = job.image.double(), want.double()
    # the same products, 4000 of them a sample at most summed in another order: 2^-24 sqrt(4000)
    assert float((got - want).norm() / want.norm()) <= 3.8e-6
