"""Kernels of the runtime-length block FFT (kfr_gb300/csrc/rp_kernels.cu) at the edges of their ranges, against
numpy's double-precision FFT at the unmultiplied bounds of the complex DFT tests."""
import numpy as np
import pytest

import kfr_gb300 as k
from oracle.oracle import c32_tolerance, c64_tolerance, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def check(n, batch, sfx, offset=0):
    rng = np.random.default_rng(n * 31 + batch)
    cdt = np.complex64 if sfx == "f32" else np.complex128
    tol = c32_tolerance(max(n, 2)) if sfx == "f32" else c64_tolerance(max(n, 2))
    x = (rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))).astype(cdt)
    buf = torch.zeros(batch * n + offset + 1, dtype=torch.complex64 if sfx == "f32" else torch.complex128, device="cuda")
    xd = buf[offset:offset + batch * n]
    xd.copy_(torch.from_numpy(x.reshape(-1)))
    yd = torch.full_like(buf, 7)
    plan = k.dft_plan(n, sfx)
    for inverse in (False, True):
        ref = np.fft.fft(x.astype(np.complex128)) if not inverse else np.fft.ifft(x.astype(np.complex128)) * n
        plan.execute_batch(yd[offset:offset + batch * n], xd, batch, inverse=inverse)
        got = yd.cpu().numpy()
        assert rel_rms(got[offset:offset + batch * n].reshape(batch, n), ref) <= tol
        # nothing outside the output is written
        assert np.all(got[:offset] == 7) and np.all(got[offset + batch * n:] == 7)
    # in place
    plan.execute_batch(xd, xd, batch)
    assert rel_rms(xd.cpu().numpy().reshape(batch, n), np.fft.fft(x.astype(np.complex128))) <= tol


# one codelet; two, three and four passes; every radix; the longest one-CTA lengths; batches of one signal, of
# part of a tile and of many tiles; pointers aligned to one element only
@pytest.mark.parametrize("n,batch,offset", [(2, 1, 1), (13, 1000, 1), (15, 77, 0), (18, 4001, 1), (49, 1, 0), (143, 333, 1),
                                            (200, 1, 1), (360, 3001, 0), (847, 19, 1), (1080, 700, 1), (2401, 3, 0),
                                            (3600, 611, 1), (5005, 5, 0), (6561, 2, 1), (14336, 3, 1), (15625, 2, 0),
                                            # primes of 17 to 127 as passes; 32 values per thread
                                            (17, 300, 1), (1088, 70, 1), (17 * 19 * 23, 3, 0), (12827, 2, 1),
                                            (18000, 3, 1), (25000, 2, 0)])
def test_signals_f32(n, batch, offset):
    check(n, batch, "f32", offset)


@pytest.mark.parametrize("n,batch", [(2, 3), (16, 65), (143, 33), (512, 1), (1000, 700), (2197, 3), (4096, 5), (7200, 2),
                                     (6561, 3), (8000, 2), (17 * 64, 9)])
def test_signals_f64(n, batch):
    check(n, batch, "f64")


# four-step splits with balanced and lopsided factors, narrow tiles, columns that do not fill a tile
@pytest.mark.parametrize("n,batch,sfx", [(20480, 3, "f32"), (21 * 1001, 5, "f32"), (65520, 7, "f32"), (1 << 17, 3, "f32"),
                                         (390625, 2, "f32"), (2939328, 1, "f32"), (1 << 21, 1, "f32"), (15625, 2, "f64"),
                                         (65536, 3, "f64"), (1 << 18, 1, "f64"), (1000000, 1, "f64")])
def test_fourstep(n, batch, sfx):
    check(n, batch, sfx, 1 if sfx == "f32" else 0)


# axes: fewer columns than a tile, an odd number of them, one column, every array of a batch
@pytest.mark.parametrize("shape,batch", [((1080, 30), 3), ((7, 1001), 2), ((600, 3), 5), ((64, 1), 2), ((16, 9, 22), 3),
                                         ((2048, 33), 1), ((15, 4096), 2)])
@pytest.mark.parametrize("sfx", ["f32", "f64"])
def test_axes(shape, batch, sfx):
    rng = np.random.default_rng(sum(shape))
    cdt = np.complex64 if sfx == "f32" else np.complex128
    total = int(np.prod(shape))
    tol = (c32_tolerance if sfx == "f32" else c64_tolerance)(total)
    x = (rng.uniform(-1, 1, (batch,) + shape) + 1j * rng.uniform(-1, 1, (batch,) + shape)).astype(cdt)
    axes = tuple(range(1, len(shape) + 1))
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    plan = k.dft_plan_md(shape, sfx)
    plan.execute_batch(yd, xd, batch)
    assert rel_rms(yd.cpu().numpy(), np.fft.fftn(x.astype(np.complex128), axes=axes)) <= tol
    plan.execute_batch(yd, xd, batch, inverse=True)
    assert rel_rms(yd.cpu().numpy(), np.fft.ifftn(x.astype(np.complex128), axes=axes) * total) <= tol


# the in-place kernels of the real DFT and the DCT: a tail of a tile, one signal, 32 values per thread, primes
@pytest.mark.parametrize("n,batch", [(2 * 30, 1001), (1000, 301), (2 * 1155, 70), (2 * 6561, 3), (2 * 18000, 2), (2 * 17 * 64, 5),
                                     # four-step half lengths: the merge in the column pass
                                     (44100, 3), (100000, 3), (131072, 2)])
@pytest.mark.parametrize("sfx", ["f32", "f64"])
def test_real(n, batch, sfx):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((batch, n)).astype(np.float32 if sfx == "f32" else np.float64)
    tol = (c32_tolerance if sfx == "f32" else c64_tolerance)(n)
    plan = k.dft_plan_real(n, dtype=sfx)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty((batch, n // 2 + 1), dtype=torch.complex64 if sfx == "f32" else torch.complex128, device="cuda")
    plan.execute_batch(yd, xd, batch)
    assert rel_rms(yd.cpu().numpy(), np.fft.rfft(x.astype(np.float64))) <= tol
    plan.execute_batch(xd, yd, batch, inverse=True)
    assert rel_rms(xd.cpu().numpy() / n, x.astype(np.float64)) <= 2 * tol


@pytest.mark.parametrize("n,batch", [(30, 1001), (1000, 301), (6561, 3), (18000, 2)])
def test_dct(n, batch):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (batch, n)).astype(np.float32)
    x64 = x.astype(np.float64)
    j, m = np.arange(n), min(n, 400)
    ks = np.unique(rng.integers(0, n, m))
    ref = x64 @ np.cos(np.pi * np.outer(2 * j + 1, ks) / (2 * n))
    plan = k.dct_plan(n)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    plan.execute_batch(yd, xd, batch)
    assert rel_rms(yd.cpu().numpy()[:, ks], ref) <= c32_tolerance(n)
    w = x64.copy()
    w[:, 0] *= 0.5
    plan.execute_batch(yd, xd, batch, inverse=True)
    assert rel_rms(yd.cpu().numpy()[:, ks], w @ np.cos(np.pi * np.outer(j, 2 * ks + 1) / (2 * n))) <= c32_tolerance(n)
