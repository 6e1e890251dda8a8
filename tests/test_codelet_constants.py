"""The cosines and sines of the odd codelets (fft_device.cuh) are the doubles nearest to their values."""
import os
import re
from decimal import Decimal, getcontext

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _series(x, first):
    """cos (first = 0) or sin (first = 1) of x by its power series, to 50 digits."""
    term, total, k = x if first else Decimal(1), Decimal(0), first
    while abs(term) > Decimal(10) ** -55:
        total += term
        term *= -x * x / ((k + 1) * (k + 2))
        k += 2
    return total


def test_odd_codelet_constants():
    getcontext().prec = 60
    pi = Decimal("3.14159265358979323846264338327950288419716939937510582097494459")
    with open(os.path.join(ROOT, "kfr_gb300", "csrc", "fft_device.cuh")) as f:
        text = f.read()
    seen = 0
    for name, first in (("odd_cos", 0), ("odd_sin", 1)):
        body = text[text.index("constexpr double " + name):]
        body = body[:body.index("default:")]
        for r, k, v in re.findall(r"case (\d+) \* 32 \+ (\d+): return (-?[\d.]+);", body):
            assert float(v) == float(_series(2 * pi * int(k) / int(r), first)), (name, r, k)
            seen += 1
    assert seen == 42
