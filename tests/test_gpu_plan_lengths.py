"""Real DFTs and DCTs of the longest one-CTA lengths, whose radices (7, 9, 11, 13 and the like) leave a thread few
butterflies to hold, against numpy in double precision."""
import numpy as np
import pytest

import kfr_gb300 as k
from oracle.oracle import c32_tolerance, c64_tolerance, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# dot products for small primes, the cheapest radices that fit near the longest one-CTA lengths
@pytest.mark.parametrize("n,batch,sfx", [(58, 1000, "f32"), (946, 70, "f32"), (8177, 3, "f32"), (12312, 5, "f32"),
                                         (14880, 2, "f32"), (13851, 3, "f32"), (12433, 3, "f32"), (19, 1000, "f64"),
                                         (31, 300, "f64"), (6384, 3, "f64"), (7200, 3, "f64"), (7039, 2, "f64")])
def test_complex(n, batch, sfx):
    rng = np.random.default_rng(n)
    cdt = np.complex64 if sfx == "f32" else np.complex128
    x = (rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))).astype(cdt)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    k.dft_plan(n, sfx).execute_batch(yd, xd, batch)
    assert rel_rms(yd.cpu().numpy(), np.fft.fft(x.astype(np.complex128))) <= (c32_tolerance if sfx == "f32" else c64_tolerance)(n)


@pytest.mark.parametrize("n,sfx", [(23100, "f32"), (24648, "f32"), (28160, "f32"), (32766, "f32"), (11880, "f64"),
                                   (12384, "f64"), (14700, "f64")])
def test_real(n, sfx):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((3, n)).astype(np.float32 if sfx == "f32" else np.float64)
    tol = (c32_tolerance if sfx == "f32" else c64_tolerance)(n)
    plan = k.dft_plan_real(n, dtype=sfx)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty((3, n // 2 + 1), dtype=torch.complex64 if sfx == "f32" else torch.complex128, device="cuda")
    plan.execute_batch(yd, xd, 3)
    assert rel_rms(yd.cpu().numpy(), np.fft.rfft(x.astype(np.float64))) <= tol
    plan.execute_batch(xd, yd, 3, inverse=True)
    assert rel_rms(xd.cpu().numpy() / n, x.astype(np.float64)) <= 2 * tol


# primes as in-place passes: alone, at either end, in the rows of a four-step transform
@pytest.mark.parametrize("n,batch,sfx", [(2 * 17, 300, "f32"), (2 * 61, 1000, "f32"), (374, 301, "f32"), (442, 1, "f32"),
                                         (2 * 17 * 19, 70, "f32"), (31310, 3, "f32"), (30264, 2, "f32"),
                                         (2 * 127, 33, "f64"), (374, 65, "f64"), (16206, 2, "f64"), (31450, 3, "f64")])
def test_primes(n, batch, sfx):
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


def cosines(phase, n):
    """cos(pi phase / 2n) for whole numbers, reduced to one turn first."""
    return np.cos(np.pi * (phase % (4 * n)) / (2 * n))


@pytest.mark.parametrize("n,sfx", [(11880, "f32"), (12324, "f32"), (12375, "f32"), (16128, "f32"), (5676, "f64"),
                                   (6192, "f64"), (8181, "f64")])
def test_dct(n, sfx):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (3, n)).astype(np.float32 if sfx == "f32" else np.float64)
    x64 = x.astype(np.float64)
    tol = (c32_tolerance if sfx == "f32" else c64_tolerance)(n)
    j, ks = np.arange(n), np.unique(rng.integers(0, n, 300))
    plan = k.dct_plan(n, sfx)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    plan.execute_batch(yd, xd, 3)
    assert rel_rms(yd.cpu().numpy()[:, ks], x64 @ cosines(np.outer(2 * j + 1, ks), n)) <= tol
    w = x64.copy()
    w[:, 0] *= 0.5
    plan.execute_batch(yd, xd, 3, inverse=True)
    assert rel_rms(yd.cpu().numpy()[:, ks], w @ cosines(np.outer(j, 2 * ks + 1), n)) <= tol


# transforms of one pass, a thread per signal: the distance between signals is odd
@pytest.mark.parametrize("n", [4, 8, 13, 16])
@pytest.mark.parametrize("sfx", ["f32", "f64"])
def test_one_pass(n, sfx):
    rng = np.random.default_rng(n)
    dt = np.float32 if sfx == "f32" else np.float64
    tol = (c32_tolerance if sfx == "f32" else c64_tolerance)
    x = rng.uniform(-1, 1, (1001, 2 * n)).astype(dt)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty((1001, n + 1), dtype=torch.complex64 if sfx == "f32" else torch.complex128, device="cuda")
    k.dft_plan_real(2 * n, dtype=sfx).execute_batch(yd, xd, 1001)
    assert rel_rms(yd.cpu().numpy(), np.fft.rfft(x.astype(np.float64))) <= tol(2 * n)
    d = torch.from_numpy(x[:, :n].copy()).cuda()
    e = torch.empty_like(d)
    k.dct_plan(n, sfx).execute_batch(e, d, 1001)
    ref = x[:, :n].astype(np.float64) @ cosines(np.outer(2 * np.arange(n) + 1, np.arange(n)), n)
    assert rel_rms(e.cpu().numpy(), ref) <= tol(n)
