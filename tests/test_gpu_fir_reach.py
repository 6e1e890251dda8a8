"""How far one sample reaches in the FFT convolution filter and its gradients: a sample that is infinite spoils the
outputs of the block it lies in, at most F - (M - 1) of them and the M - 1 after the last, F = max(8 (M - 1), twice the
caller's block) samples rounded up to a power of two; short taps never wait for a longer block than that."""
import numpy as np
import pytest

import kfr_gb300 as k
from oracle.oracle import c32_tolerance, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def block(m, size):
    f = 64
    while f < max(8 * (m - 1), 2 * size):
        f *= 2
    return f


# blocks of 64 (the caller's), 2048, 4096 and 8192 samples (pairs of 4096 through one transform)
@pytest.mark.parametrize("m,size", [(5, 16), (33, 1024), (257, 1024), (400, 1024), (600, 1024), (1024, 1024), (33, 4096)])
def test_filter(m, size):
    n = 40000
    rng = np.random.default_rng(m)
    h = rng.standard_normal(m).astype(np.float32)
    x = rng.standard_normal((2, n)).astype(np.float32)
    flt = k.convolve_filter(torch.from_numpy(h).cuda(), size, dtype="f32", channels=2)
    y = torch.empty((2, n), dtype=torch.float32, device="cuda")
    flt.apply(y, torch.from_numpy(x).cuda())
    ref = np.stack([np.convolve(r.astype(np.float64), h.astype(np.float64))[:n] for r in x])
    assert rel_rms(y.cpu().numpy(), ref) <= 3 * c32_tolerance(block(m, size))
    x[0, 21000] = np.inf
    flt.reset()
    flt.apply(y, torch.from_numpy(x).cuda())
    bad = ~np.isfinite(y.cpu().numpy())
    assert m <= bad[0].sum() <= block(m, size) and not bad[1].any()


@pytest.mark.parametrize("m", [33, 400, 1024])
def test_signal_gradient(m):
    n = 40000
    rng = np.random.default_rng(m)
    h, x, g = (torch.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda() for s in ((m,), (1, n), (1, n)))
    g[0, 21000] = float("inf")
    gx = torch.empty_like(x)
    k.fir_backward(h, x, g, gx, None, channels=1)
    assert m <= int((~torch.isfinite(gx)).sum()) <= block(m, 1024)
