"""Uneven batches on CTAs of 256 and of 512 threads, each signal one item or some of several stages, built in either order,
against numpy in double precision."""
import numpy as np
import pytest

import kfr_gb300 as k
from oracle.oracle import c32_tolerance, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LENGTHS = [
    [64, 1000, 2048, 1021, 17],  # convolutions of 2048 points: 256 threads
    [4093, 4096, 1000, 64, 2011, 1],  # convolutions of 8192 points, one item each: 512 threads
    [8192, 5000, 64, 360],  # whole signals that only 512 threads hold
    [8192, 4099, 1000, 64, 20000],  # several stages
]


@pytest.mark.parametrize("order", [1, -1])
def test_shapes(order):
    rng = np.random.default_rng(7)
    for lengths in LENGTHS[::order]:
        lengths = lengths * 3
        x = (rng.uniform(-1, 1, sum(lengths)) + 1j * rng.uniform(-1, 1, sum(lengths))).astype(np.complex64)
        xd = torch.from_numpy(x).cuda()
        yd = torch.empty_like(xd)
        plan = k.dft_plan_uneven(lengths)
        for inverse in (False, True):
            plan.execute(yd, xd, inverse=inverse)
            y, at = yd.cpu().numpy(), 0
            for n in lengths:
                s = x[at:at + n].astype(np.complex128)
                ref = np.fft.ifft(s) * n if inverse else np.fft.fft(s)
                assert rel_rms(y[at:at + n], ref) <= c32_tolerance(max(n, 2)), (n, inverse)
                at += n
