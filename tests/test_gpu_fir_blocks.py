"""Block kernels of the convolution filter and its gradients (kfr_gb300/csrc/conv.cu) at the edges of their blocks,
against sums in double precision.  One output block is a forward transform, a product and an inverse one: three
times the DFT bound at the block's FFT length F; a taps gradient has two forward transforms: four times."""
import numpy as np
import pytest

import kfr_gb300 as k
from oracle.oracle import c32_tolerance, c64_tolerance, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def fft_size(m, sfx):
    if sfx == "f32" and m <= 2049:
        return 4096  # paired blocks
    f = 2048
    while f < 8 * (m - 1):
        f *= 2
    return min(f, 32768 if sfx == "f32" else 16384)


def fir(h, x):
    return np.stack([np.convolve(r, h)[:x.shape[1]] for r in x])


# one tap, odd and even tap counts, signals shorter than the taps, of exactly one block, of one sample more, odd
# lengths (the second channel is then aligned to one sample only), every FFT length of the kernels
CASES = [(1, 1, 1), (2, 5000, 2), (16, 2033, 3), (1023, 7169, 2), (1024, 3, 1), (1023, 14340, 2), (255, 1794, 1),
         (256, 1793, 3), (700, 40001, 2), (2000, 20011, 2), (4000, 70000, 1), (2049, 6145, 2), (2050, 6145, 1)]


@pytest.mark.parametrize("sfx", ["f32", "f64"])
@pytest.mark.parametrize("m,n,channels", CASES)
def test_filter_and_gradients(m, n, channels, sfx):
    rng = np.random.default_rng(m + n)
    dt = np.float32 if sfx == "f32" else np.float64
    h, x, g = (rng.standard_normal(s).astype(dt) for s in ((m,), (channels, n), (channels, n)))
    hd, xd, gd = (torch.from_numpy(v).cuda() for v in (h, x, g))
    tol = (c32_tolerance if sfx == "f32" else c64_tolerance)(fft_size(m, sfx))
    h64, x64, g64 = h.astype(np.float64), x.astype(np.float64), g.astype(np.float64)
    ref = fir(h64, x64)
    # in two calls: the second starts from the first one's history
    y = torch.empty_like(xd)
    flt = k.convolve_filter(hd, 1024, dtype=sfx, channels=channels)
    cut = n // 3
    if cut:
        part = [torch.empty((channels, s), dtype=xd.dtype, device="cuda") for s in (cut, n - cut)]
        flt.apply(part[0], xd[:, :cut].contiguous())
        flt.apply(part[1], xd[:, cut:].contiguous())
        y.copy_(torch.cat(part, 1))
    else:
        flt.apply(y, xd)
    assert rel_rms(y.cpu().numpy(), ref) <= 3 * tol
    gx_ref = fir(h64, g64[:, ::-1])[:, ::-1]
    gh_ref = np.zeros(m)
    for c in range(channels):
        full = np.correlate(g64[c], x64[c], "full")[n - 1:][:m]
        gh_ref[:len(full)] += full
    gx, gh = torch.empty_like(xd), torch.empty_like(hd)
    k.fir_backward(hd, xd, gd, gx, gh, channels=channels)
    assert rel_rms(gx.cpu().numpy(), gx_ref) <= 3 * tol
    assert np.linalg.norm(gh.cpu().numpy() - gh_ref) <= 4 * tol * np.linalg.norm(g64) * np.linalg.norm(x64)
    # each gradient alone gives the same values
    gx2, gh2 = torch.empty_like(gx), torch.empty_like(gh)
    k.fir_backward(hd, xd, gd, gx2, None, channels=channels)
    k.fir_backward(hd, xd, gd, None, gh2, channels=channels)
    assert torch.equal(gx, gx2) and torch.equal(gh, gh2)
    # the signal gradient in place of the output gradient
    g2 = gd.clone()
    k.fir_backward(hd, xd, g2, g2, None, channels=channels)
    assert torch.equal(g2, gx)
