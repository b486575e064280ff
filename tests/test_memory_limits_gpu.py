"""Calls that find little room on the device: least squares without the demigration's copy of the
model, and a failed allocation that leaves the next call alone."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("graph", [True, False])
def test_without_room_for_the_model_copy(cuda, ktm_lib, graph):
    import torch

    from ktm import inverse
    from ktm._lib import check
    # a shallow image: the copy pads its 33 samples to 256 (25 MiB -> 195 MiB)
    nx, nz, ntr, nt = 200000, 33, 160, 200
    g = torch.Generator(device=cuda)
    g.manual_seed(1)
    c = [torch.rand(ntr, device=cuda, generator=g) * 0.5 * nx for _ in range(2)]
    zero = torch.zeros(ntr, device=cuda)
    op = inverse.MigrationOperator(imageX=(nx, 0.5, 0.0), imageY=(1, 1.0, 0.0), imageZ=(nz, 0.002, 0.0), dt=0.004, nt=nt,
                                   midX=c[0], midY=zero, offX=c[1] * 1e-3, offY=zero,
                                   velocity=torch.full((nz,), 2500.0, device=cuda), aperture=400.0, weight="prefold")
    data = op.pack(torch.randn((ntr, nt), device=cuda, generator=g))
    want, residuals, gradients = op.least_squares(data, 2, use_graph=graph)
    check(ktm_lib.ktmReleaseMemory())
    model = torch.zeros_like(want)
    torch.cuda.empty_cache()
    # the workspace without the copy: 10 partial images and two model vectors, about 305 MiB
    room, taken, size = 400 * MB, [], 1 << 34
    try:
        while torch.cuda.mem_get_info()[0] > room and size >= 16 * MB:
            if torch.cuda.mem_get_info()[0] - size < room:
                size //= 2
                continue
            taken.append(torch.empty(size, dtype=torch.uint8, device=cuda))
        assert torch.cuda.mem_get_info()[0] < room + 32 * MB
        _, r, q = op.least_squares(data, 2, model=model, use_graph=graph)
    finally:
        taken.clear()
        check(ktm_lib.ktmReleaseMemory())
        torch.cuda.empty_cache()
    # two iterations of FP32 operators whose sums run in another order
    np.testing.assert_allclose(r, residuals, rtol=1e-5)
    np.testing.assert_allclose(q, gradients, rtol=1e-4)
    assert float((model.double() - want.double()).norm() / want.double().norm()) <= 1e-4


def test_a_failed_allocation_stays_in_its_call(cuda, ktm_lib):
    """A call that finds no memory reports it; the next one runs."""
    import torch

    import ktm
    from ktm import inverse
    nx, nz, ntr, nt = 300000, 64, 40, 100
    zero = torch.zeros(ntr, device=cuda)
    wide, narrow = (inverse.MigrationOperator(imageX=(n, 0.5, 0.0), imageY=(1, 1.0, 0.0), imageZ=(nz, 0.002, 0.0), dt=0.004,
                                              nt=nt, midX=zero, midY=zero, offX=zero, offY=zero, aperture=100.0,
                                              velocity=torch.full((nz,), 2000.0, device=cuda), weight="prefold")
                    for n in (nx, 50))
    model, image = torch.zeros((nx, 1, nz), device=cuda), torch.ones((50, 1, nz), device=cuda)
    data = wide.pack(torch.ones((ntr, nt), device=cuda))
    out = torch.empty_like(data)
    want = narrow.demigrate(image).clone()
    torch.cuda.synchronize()
    ktm._lib.check(ktm_lib.ktmReleaseMemory())
    torch.cuda.empty_cache()
    taken, size = [], 1 << 34
    try:
        while size >= 32 * MB:
            try:
                taken.append(torch.empty(size, dtype=torch.uint8, device=cuda))
            except torch.cuda.OutOfMemoryError:
                size //= 2
        with pytest.raises(ktm.KtmError):
            wide.least_squares(data, 1, model=model)       # some 400 MB
    finally:
        taken.clear()
        torch.cuda.empty_cache()
    narrow.demigrate(image, out)
    # two column blocks added in either order
    assert torch.allclose(out, want, rtol=1e-5, atol=1e-5 * float(want.abs().max()))
