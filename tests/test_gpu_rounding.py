"""Rounding of single-precision transforms against pocketfft's (scipy.fft in single precision: correctly rounded twiddles), on
the same input.  Long transforms: at most a tenth more relative RMS error (twiddles formed as powers of two table values
give 21 and 29% more at these sizes)."""
import numpy as np
import pytest

import kfr_gb300 as k
from oracle.oracle import rel_rms

torch = pytest.importorskip("torch")
scipy_fft = pytest.importorskip("scipy.fft")
pytestmark = pytest.mark.gpu


# an axis of radix-16 passes; a four-step transform of two of them
@pytest.mark.parametrize("shape,batch", [((4096, 2), 64), ((1 << 23,), 1)])
def test_rounding(shape, batch):
    rng = np.random.default_rng(shape[0])
    x = (rng.standard_normal((batch,) + shape) + 1j * rng.standard_normal((batch,) + shape)).astype(np.complex64)
    axes = tuple(range(1, len(shape) + 1))
    ref = np.fft.fftn(x.astype(np.complex128), axes=axes)
    plan = k.dft_plan(shape[0], "f32") if len(shape) == 1 else k.dft_plan_md(shape, "f32")
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    plan.execute_batch(yd, xd, batch)
    assert rel_rms(yd.cpu().numpy(), ref) <= 1.1 * rel_rms(scipy_fft.fftn(x, axes=axes), ref)


# the taps' gradient of one short signal, whose blocks correlate with less zero padding than a whole-signal transform: at
# most a fifth more than pocketfft's over the whole signal, over 40 signals
@pytest.mark.parametrize("taps", [16, 300])
def test_taps_gradient_rounding(taps):
    err = ref_err = 0.0
    h = torch.randn(taps, device="cuda")
    for seed in range(40):
        n = 4096 + seed
        rng = np.random.default_rng(seed)
        x, g = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
        size = 1 << (n + taps - 1).bit_length()

        def correlate(fft, a, b):
            return fft.irfft(fft.rfft(a, size) * np.conj(fft.rfft(b, size)), size)[:taps]

        exact = correlate(np.fft, g.astype(np.float64), x.astype(np.float64))
        got = torch.empty(taps, device="cuda")
        k.fir_backward(h, torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda(), None, got, channels=1)
        err += np.sum((got.cpu().numpy() - exact) ** 2)
        ref_err += np.sum((correlate(scipy_fft, g, x) - exact) ** 2)
    assert err <= 1.2**2 * ref_err
