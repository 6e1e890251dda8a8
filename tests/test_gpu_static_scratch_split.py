"""kfr_dft_execute_static_scratch_f32 for lengths that one CTA could transform without scratch but that run with it: any
batch is taken, in parts that fit the static scratch."""
import numpy as np
import pytest

import kfr_gb300 as k
from oracle.oracle import c32_tolerance, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(12433, 63), (12433, 200), (15277, 129)])
def test_any_batch(n, batch):
    plan = k.dft_plan(n, "f32")
    x = torch.randn(batch, n, dtype=torch.complex64, device="cuda")
    y = torch.empty_like(x)
    lib = k.lib()
    for inverse in (False, True):
        lib.kfr_dft_execute_static_scratch_f32(plan.handle, batch, y.data_ptr(), x.data_ptr(), inverse, None)
        assert lib.kfr_last_error() == b""
        x64 = x.cpu().numpy().astype(np.complex128)
        ref = np.fft.ifft(x64) * n if inverse else np.fft.fft(x64)
        assert rel_rms(y.cpu().numpy(), ref) <= c32_tolerance(n)
