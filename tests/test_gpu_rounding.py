"""Rounding of long single-precision transforms against pocketfft's (scipy.fft on complex64: correctly rounded twiddles):
at most a tenth more relative RMS error, on the same input.  Twiddles formed as powers of two table values give 21 and
29% more at these sizes."""
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
