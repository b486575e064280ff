"""Trace preparation at the edges of its transform sizes: every power of two from 1 to 16384
and its neighbours, all filters, storage formats and input kinds, odd trace counts, longer rows
and pitches, against the FP64 filter; without a filter against the plain FP32 arithmetic."""
from __future__ import annotations

import numpy as np
import pytest

import rho as oracle_rho

pytestmark = pytest.mark.gpu

# FP32 transforms: each of the 2 log2(M) <= 28 butterfly levels and the filter round relative
# to the trace's largest spectral amplitude, an L2 error of at most about 2^-24 * sqrt(2 * 28 + 6)
# = 4.7e-7 of the spectrum's L2 norm; twiddles add as much again.
REL = 1.5e-6


def _prepare(x, dt, opt, prefold=False, fmt="f32", **kw):
    import ktm
    return ktm.prepare(x, dt, fmt=fmt, rho=opt, prefold=prefold, **kw)


def _want(x, dt, opt, prefold):
    y = oracle_rho.rho_filter_traces(x, float(np.float32(dt)) * 1e6, opt) if opt else x.astype(np.float64)
    if prefold:
        y = y * np.sqrt(np.arange(x.shape[1]) * float(np.float32(dt)))
    y[:, 0] = 0.0
    return y


@pytest.mark.parametrize("opt", [1, 2, 3])
@pytest.mark.parametrize("log2m", range(15))
def test_transform_sizes(cuda, ktm_lib, log2m, opt):
    import torch
    for nt in sorted({1 << log2m, max(1, (1 << log2m) - 1), (1 << log2m) // 2 + 1}):
        rng = np.random.default_rng(nt)
        x = rng.standard_normal((5, nt)).astype(np.float32)
        p = _prepare(torch.as_tensor(x).to(cuda), 0.002, opt, prefold=opt == 2)
        got, want = p.unpacked().double().cpu().numpy(), _want(x, 0.002, opt, opt == 2)
        assert np.all(p.data[:, nt:].cpu().numpy() == 0) and np.all(got[:, 0] == 0)
        # relative to the whole filtered trace: the window keeps only its first nt samples
        full = np.linalg.norm(_want(np.pad(x, ((0, 0), (0, (1 << max(0, (nt - 1).bit_length())) - nt))),
                                    0.002, opt, opt == 2))
        assert np.linalg.norm(got - want) <= REL * max(full, 1e-300), (nt, opt)


@pytest.mark.parametrize("fmt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("opt", [0, 2])
@pytest.mark.parametrize("ntr,nt,stride,extra", [(1, 2, 2, 0), (2, 129, 131, 16), (7, 1001, 1001, 0),
                                                 (130, 100, 100, 8), (3, 2049, 2060, 32)])
def test_formats_strides_and_words(cuda, ktm_lib, ntr, nt, stride, extra, opt, fmt):
    """IBM words give exactly what their decoded floats give; guards are zero whatever the
    pitch; the scale and the quantised samples follow from the FP32 result."""
    import torch

    import ktm
    from ktm import synth
    rng = np.random.default_rng(ntr * nt)
    words = synth.encode_ibm32(rng.standard_normal((ntr, stride)).astype(np.float32))
    words[0, 1] = 0x7fffffff                            # 16^63: outside the FP32 range
    if opt:
        words[0, 1] = words[0, 0]
    raw = torch.as_tensor(words.view(np.int32)).to(cuda)
    flt = torch.empty((ntr, stride), device=cuda)
    ktm_lib.ktmIBM32toIEEEDevice(raw.data_ptr(), flt.data_ptr(), raw.numel(), None)
    pitch = ktm.packed_pitch(nt, fmt) + extra
    dtype = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[fmt]
    out = [torch.full((ntr, pitch), 7.0, device=cuda, dtype=dtype) for _ in range(2)]
    p = [_prepare(x, 0.004, opt, True, fmt, nt=nt, out=o) for x, o in zip((raw, flt), out)]
    assert torch.equal(p[0].data.view(torch.uint8), p[1].data.view(torch.uint8))
    assert torch.equal(p[0].scale.view(torch.int32), p[1].scale.view(torch.int32))
    assert np.all(p[1].data[:, nt:].float().cpu().numpy() == 0) and np.all(p[1].data[:, 0].float().cpu().numpy() == 0)
    if opt == 0:
        x = flt[:, :nt].cpu().numpy()
        w = np.sqrt(np.arange(nt, dtype=np.float32) * np.float32(0.004))
        v = x * w
        v[:, 0] = 0.0
        top = np.abs(v).max(axis=1)
        s = np.ones(ntr, np.float32) if fmt == "f32" else np.where(
            top > 0, top / np.float32(32768.0 if fmt == "f16" else 1.0), np.float32(1.0)).astype(np.float32)
        with np.errstate(over="ignore", invalid="ignore"):
            q = v * (np.float32(1.0) / s)[:, None]
        want = torch.as_tensor(q).to(dtype)
        assert np.array_equal(p[1].scale.cpu().numpy(), s)
        assert torch.equal(torch.nan_to_num(p[1].data[:, :nt].cpu().float()), torch.nan_to_num(want.float()))


def test_long_traces_without_a_filter(cuda, ktm_lib):
    """Beyond the largest transform, up to the limit, and past it."""
    import torch

    import ktm
    for nt in (16385, 29056):
        x = torch.randn((3, nt), device=cuda)
        p = _prepare(x, 0.001, 0, fmt="bf16")
        top = x[:, 1:].abs().amax(1)
        assert torch.equal(p.scale, top)
        q = (x * (1.0 / top)[:, None]).to(torch.bfloat16)
        q[:, 0] = 0
        assert torch.equal(p.data[:, :nt], q)
    with pytest.raises(ktm.KtmError):
        _prepare(torch.zeros((1, 29057), device=cuda), 0.001, 0)
    with pytest.raises(ktm.KtmError):
        _prepare(torch.zeros((1, 16385), device=cuda), 0.001, 2)


def test_script_order_of_odd_counts(cuda, ktm_lib):
    import torch
    x = torch.randn((5, 300), device=cuda)
    for opt in (0, 3):
        a, b = (_prepare(x, 0.002, opt, script_order=o).data for o in (False, True))
        assert torch.equal(torch.roll(a, -1, 0), b)


@pytest.mark.parametrize("fmt", ["f16", "bf16"])
@pytest.mark.parametrize("ntr,nt", [(24001, 601), (16001, 1001), (12001, 1501), (6001, 4096),
                                    (3001, 6001), (2001, 16384)])
def test_many_rounds_without_a_filter(cuda, ktm_lib, ntr, nt, fmt):
    """Counts that give every CTA several rounds, neighbouring traces whose maxima differ by
    orders of magnitude: each trace keeps its own scale, every sample is quantised by it."""
    import torch
    gen = torch.Generator(device=cuda)
    gen.manual_seed(nt)
    x = torch.randn((ntr, nt), device=cuda, generator=gen)
    x *= torch.pow(2.0, torch.randint(-20, 21, (ntr, 1), device=cuda, generator=gen).float())
    x[:, 0] = 0
    top = x.abs().amax(1) / (32768.0 if fmt == "f16" else 1.0)
    want = (x * (1.0 / top)[:, None]).to(torch.float16 if fmt == "f16" else torch.bfloat16)
    for _ in range(5):
        p = _prepare(x, 0.002, 0, fmt=fmt)
        assert torch.equal(p.scale, top)
        assert torch.equal(p.data[:, :nt], want) and not p.data[:, nt:].any()


@pytest.mark.parametrize("opt", [1, 2, 3])
@pytest.mark.parametrize("nt", [2, 4, 8])
def test_the_filter_is_rounded_once(cuda, ktm_lib, nt, opt):
    """One line of the spectrum, whose transform is exact: the result is the filter's own value,
    |w|, sqrt(|w| / 2) or w at a quarter of the sampling rate (at half of it for two samples), in
    64 bits rounded to FP32."""
    import torch
    rng = np.random.default_rng(nt)
    for dt in np.exp(rng.uniform(np.log(2e-4), np.log(2e-2), 200)).astype(np.float32):
        n = np.arange(nt)
        x = np.where(n % 2 == 0, 1.0, -1.0) if nt == 2 else np.rint(np.cos(np.pi * n / 2))
        got = _prepare(torch.as_tensor(x[None].astype(np.float32)).to(cuda), float(dt), opt).unpacked()[0].cpu().numpy()
        w = 2.0 * np.pi * (nt // 4 if nt > 2 else 1) / np.float64(dt)
        size = np.float32([0, w, np.sqrt(w / 2.0), w][opt])
        if nt == 2:                                     # Nyquist: the real part alone
            want = [0.0, 0.0 if opt == 3 else -size]
        else:
            c, s = np.rint(np.cos(np.pi * n / 2)), np.rint(np.sin(np.pi * n / 2))
            want = size * [0, c, c - s, -s][opt]
            want[0] = 0.0
        assert np.array_equal(got, np.float32(want)), (dt, got, want)


@pytest.mark.parametrize("fmt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("words,prefold", [(False, False), (False, True), (True, False)])
@pytest.mark.parametrize("ntr,nt,extra", [(1, 8193, 0), (3, 16384, 8), (2, 17408, 0), (5, 17409, 16), (301, 16385, 0),
                                          (2, 28673, 64), (3, 29056, 1024)])
def test_long_traces_equal_the_plain_arithmetic(cuda, ktm_lib, ntr, nt, extra, words, prefold, fmt):
    """A CTA per trace, around multiples of its threads, with guards past its registers."""
    import torch

    import ktm
    from ktm import synth
    rng = np.random.default_rng(nt)
    x = (rng.standard_normal((ntr, nt + 3)) * 2.0 ** rng.integers(-9, 9, (ntr, 1))).astype(np.float32)
    if words:
        w = synth.encode_ibm32(x)
        w[0, 5] = 0x7fffffff                            # 16^63: outside the FP32 range
        src = torch.as_tensor(w.view(np.int32)).to(cuda)
        flt = torch.empty((ntr, nt + 3), device=cuda)
        ktm_lib.ktmIBM32toIEEEDevice(src.data_ptr(), flt.data_ptr(), src.numel(), None)
        x = flt.cpu().numpy()
    else:
        src = torch.as_tensor(x).to(cuda)
    dtype = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[fmt]
    out = torch.full((ntr, ktm.packed_pitch(nt, fmt) + extra), 7.0, device=cuda, dtype=dtype)
    p = _prepare(src, 0.002, 0, prefold, fmt, nt=nt, out=out)
    v = x[:, :nt].copy()
    if prefold:
        v *= np.sqrt(np.arange(nt, dtype=np.float32) * np.float32(0.002))
    v[:, 0] = 0.0
    top = np.abs(v).max(axis=1)
    s = np.ones(ntr, np.float32) if fmt == "f32" else (top / np.float32(32768.0 if fmt == "f16" else 1.0))
    with np.errstate(over="ignore", invalid="ignore"):
        want = torch.as_tensor(v * (np.float32(1.0) / s)[:, None]).to(dtype)
    assert np.array_equal(p.scale.cpu().numpy(), s)
    assert torch.equal(torch.nan_to_num(p.data[:, :nt].cpu().float()), torch.nan_to_num(want.float()))
    assert not p.data[:, nt:].any()
