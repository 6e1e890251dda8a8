"""The calls whose time matters to a user of the library, each through the Python plan objects.

listed() names twelve of them, draw() gives more of the same ranges:

  dft     batched complex DFTs (complex64 and complex128, forward and inverse) of any length: powers of two,
          products of small primes, primes, any integer; 1 signal to a gigabyte of them
  real    batched real DFTs in both packings, forward and inverse
  dct     batched DCT-II (forward) and DCT-III (inverse)
  fir     a block of samples through an FIR convolution filter of many channels, alone or with the gradients
          with respect to the samples and the taps
  uneven  many complex signals of different lengths in one call
  md      two- and three-dimensional complex and real DFTs

Buffers are on the GPU, as in a program that keeps its data there.  Calls that take a stream get one of their
own ("stream" cases); the "sync" case is the plain execute() of the C API, which returns when the result is
there; the filter's calls have no stream argument.
"""
import math

import torch

import kfr_gb300 as kfr
from kfr_gb300.workloads import uneven_lengths

_STREAMS = {}


def _stream():
    """The stream this program's transforms run on."""
    d = torch.cuda.current_device()
    if d not in _STREAMS:
        _STREAMS[d] = torch.cuda.Stream()
    return _STREAMS[d]


def listed():
    return [
        # a single short spectrum, waited for: the latency of one call
        {"name": "one call 1024", "kind": "dft", "n": 1024, "batch": 1, "dtype": "f32", "inverse": False, "call": "sync"},
        # the plain configuration: 1024 signals of 4096 points
        {"name": "4096 x 1024", "kind": "dft", "n": 4096, "batch": 1024, "dtype": "f32", "inverse": False, "call": "stream"},
        # an everyday length that is a product of small primes
        {"name": "3600 x 4096", "kind": "dft", "n": 3600, "batch": 4096, "dtype": "f32", "inverse": False, "call": "stream"},
        # a prime length of the mixed-radix and prime configuration, 256 MiB
        {"name": "prime 8191 x 4096", "kind": "dft", "n": 8191, "batch": 4096, "dtype": "f32", "inverse": False, "call": "stream"},
        # long signals back to the time domain, 1 GiB
        {"name": "inverse 2^20 x 128", "kind": "dft", "n": 1 << 20, "batch": 128, "dtype": "f32", "inverse": True, "call": "stream"},
        # one long double-precision transform
        {"name": "c64 2^20", "kind": "dft", "n": 1 << 20, "batch": 1, "dtype": "f64", "inverse": False, "call": "stream"},
        # one-second audio frames at 48 kHz, 256 MiB of samples
        {"name": "real 48000 x 1398", "kind": "real", "n": 48000, "batch": 1398, "fmt": "CCs", "inverse": False},
        # and back to samples at 44.1 kHz
        {"name": "real inverse 44100 x 1521", "kind": "real", "n": 44100, "batch": 1521, "fmt": "CCs", "inverse": True},
        # block transform coding
        {"name": "dct 512 x 4096", "kind": "dct", "n": 512, "batch": 4096, "inverse": False},
        # 64 channels through a 1023-tap filter and the gradients of a training step
        {"name": "fir 64 x 2^20 with gradients", "kind": "fir", "channels": 64, "n": 1 << 20, "taps": 1023, "grad": True},
        # signals of many lengths in one call, a tenth of them prime
        {"name": "uneven 1024", "kind": "uneven", "count": 1024, "lo": 64, "hi": 65536, "lengths_seed": 20261206},
        # the two-dimensional spectra of eight full-HD frames
        {"name": "2-D 1080 x 1920 x 8", "kind": "md", "shape": "1080x1920", "batch": 8, "real": False, "inverse": False},
    ]


# ------------------------------------------------------------------------------------------------------
# draw
# ------------------------------------------------------------------------------------------------------


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _smooth_near(v):
    """The 2^a 3^b 5^c 7^d nearest to v."""
    best = 1
    p7 = 1
    while p7 <= 2 * v:
        p5 = p7
        while p5 <= 2 * v:
            p3 = p5
            while p3 <= 2 * v:
                p2 = p3
                while p2 <= 2 * v:
                    if abs(p2 - v) < abs(best - v):
                        best = p2
                    p2 *= 2
                p3 *= 3
            p5 *= 5
        p7 *= 7
    return best


def _prime_near(v):
    v = max(3, v | 1)
    while any(v % p == 0 for p in range(3, int(v**0.5) + 1, 2)):
        v += 2
    return v


def _length(rng, lo, hi_smooth, hi_any):
    """A transform length and the most elements of one call of it."""
    style = rng.choice(["smooth", "smooth", "smooth", "pow2", "any", "prime"])
    if style == "smooth":
        n = max(lo, _smooth_near(_log_int(rng, lo, hi_smooth)))
        return n, 1 << 25
    if style == "pow2":
        n = 1 << rng.randint(max(1, lo.bit_length() - 1), hi_smooth.bit_length() - 1)
        return n, 1 << 25
    n = _log_int(rng, lo, hi_any)
    n = n if style == "any" else _prime_near(n)
    return n, 1 << 22


def _batch(rng, n, most):
    """From one signal to `most` elements in all."""
    return _log_int(rng, 1, max(1, most // n))


def draw(rng):
    kind = rng.choice(["dft"] * 8 + ["real"] * 3 + ["dct", "fir", "fir", "uneven", "md", "md"])
    if kind == "dft":
        dtype = rng.choice(["f32", "f32", "f32", "f64"])
        n, most = _length(rng, 32, 1 << 23 if dtype == "f32" else 1 << 20, 1 << 17 if dtype == "f32" else 1 << 14)
        batch = _batch(rng, n, most if dtype == "f32" else 1 << 21)
        call = "sync" if batch == 1 and rng.random() < 0.5 else "stream"
        return {"kind": kind, "n": n, "batch": batch, "dtype": dtype, "inverse": rng.random() < 0.4, "call": call}
    if kind == "real":
        n, most = _length(rng, 64, 1 << 18, 1 << 15)
        n += n % 2
        return {"kind": kind, "n": n, "batch": _batch(rng, n, most), "fmt": rng.choice(["CCs", "CCs", "Perm"]),
                "inverse": rng.random() < 0.5}
    if kind == "dct":
        n, most = _length(rng, 8, 1 << 14, 1 << 12)
        return {"kind": kind, "n": n, "batch": _batch(rng, n, most // 2), "inverse": rng.random() < 0.5}
    if kind == "fir":
        channels = _log_int(rng, 1, 64)
        return {"kind": kind, "channels": channels, "n": _log_int(rng, 4096, (1 << 26) // channels // 2 if channels > 32 else 1 << 20),
                "taps": _log_int(rng, 16, 4096), "grad": rng.random() < 0.5}
    if kind == "uneven":
        return {"kind": kind, "count": _log_int(rng, 32, 1024), "lo": 64, "hi": 1 << rng.randint(11, 16),
                "lengths_seed": rng.randrange(1 << 30)}
    dims = rng.choice([2, 2, 3])
    most = 1 << 22
    shape = []
    for d in range(dims):
        v = _smooth_near(_log_int(rng, 24 if dims == 3 else 60, 200 if dims == 3 else 2000))
        shape.append(v + (v % 2 if d == dims - 1 else 0))
    return {"kind": kind, "shape": "x".join(str(v) for v in shape), "batch": _batch(rng, math.prod(shape), most),
            "real": rng.random() < 0.4, "inverse": rng.random() < 0.4}


# ------------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _normal(shape, dtype, seed):
    return torch.randn(shape, dtype=dtype, device="cuda", generator=_gen(seed))


def _spectrum(batch, n, fmt, seed):
    """Spectra of real signals: random bins, the first and last of them real."""
    c = n // 2 + 1
    s = _normal((batch, c), torch.complex64, seed)
    s[:, 0].imag.zero_()
    s[:, -1].imag.zero_()
    if fmt == "CCs":
        return s
    p = s[:, :-1].clone()
    p[:, 0] = torch.complex(s[:, 0].real.clone(), s[:, -1].real.clone())
    return p


def _taps(m, seed):
    """A Kaiser-windowed lowpass with a little noise."""
    t = torch.arange(m, dtype=torch.float64) - (m - 1) / 2
    h = torch.sinc(t / 4) / 4 * torch.kaiser_window(m, periodic=False, beta=8.0, dtype=torch.float64)
    return h.to(torch.float32).cuda() + 1e-2 / math.sqrt(m) * _normal((m,), torch.float32, seed)


def _shape(case):
    return tuple(int(v) for v in case["shape"].split("x"))


def _inputs(case, seed):
    """The input tensors of a case, from the seed alone."""
    kind = case["kind"]
    if kind == "dft":
        return {"x": _normal((case["batch"], case["n"]), torch.complex64 if case["dtype"] == "f32" else torch.complex128, seed)}
    if kind == "real":
        if case["inverse"]:
            return {"x": _spectrum(case["batch"], case["n"], case["fmt"], seed)}
        return {"x": _normal((case["batch"], case["n"]), torch.float32, seed)}
    if kind == "dct":
        return {"x": torch.rand((case["batch"], case["n"]), device="cuda", generator=_gen(seed)) * 2 - 1}
    if kind == "fir":
        shape = (case["channels"], case["n"])
        got = {"x": _normal(shape, torch.float32, seed), "taps": _taps(case["taps"], seed + 1)}
        if case["grad"]:
            got["gy"] = _normal(shape, torch.float32, seed + 2)
        return got
    if kind == "uneven":
        total = sum(_lengths(case))
        return {"x": torch.view_as_complex(torch.rand((total, 2), device="cuda", generator=_gen(seed)) * 2 - 1)}
    shape = (case["batch"],) + _shape(case)
    if not case["real"]:
        return {"x": _normal(shape, torch.complex64, seed)}
    x = _normal(shape, torch.float32, seed)
    if not case["inverse"]:
        return {"x": x}
    return {"x": torch.fft.rfftn(x, dim=tuple(range(1, len(shape))))}


def _lengths(case):
    return [int(v) for v in uneven_lengths(case["count"], case["lo"], case["hi"], 0.1, case["lengths_seed"])]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, **_inputs(case, seed)}
    x = s["x"]
    if kind == "dft":
        s["plan"] = kfr.dft_plan(case["n"], case["dtype"])
        s["y"] = torch.empty_like(x)
    elif kind == "real":
        s["plan"] = kfr.dft_plan_real(case["n"], case["fmt"])
        if case["inverse"]:
            s["y"] = torch.empty((case["batch"], case["n"]), dtype=torch.float32, device="cuda")
        else:
            s["y"] = torch.empty((case["batch"], s["plan"].complex_size), dtype=torch.complex64, device="cuda")
    elif kind == "dct":
        s["plan"] = kfr.dct_plan(case["n"])
        s["y"] = torch.empty_like(x)
    elif kind == "fir":
        s["plan"] = kfr.convolve_filter(s["taps"], 1024, dtype="f32", channels=case["channels"])
        s["y"] = torch.empty_like(x)
        if case["grad"]:
            s["gx"] = torch.empty_like(x)
            s["gtaps"] = torch.empty_like(s["taps"])
    elif kind == "uneven":
        s["plan"] = kfr.dft_plan_uneven(_lengths(case))
        s["y"] = torch.empty_like(x)
    else:
        shape = _shape(case)
        if case["real"]:
            s["plan"] = kfr.dft_plan_md_real(shape)
            if case["inverse"]:
                s["y"] = torch.empty((case["batch"],) + shape, dtype=torch.float32, device="cuda")
            else:
                s["y"] = torch.empty((case["batch"],) + s["plan"].complex_shape, dtype=torch.complex64, device="cuda")
        else:
            s["plan"] = kfr.dft_plan_md(shape)
            s["y"] = torch.empty_like(x)
    return s


def run(s):
    case, plan, x, y = s["case"], s["plan"], s["x"], s["y"]
    kind = case["kind"]
    if kind == "fir":
        plan.reset()
        plan.apply(y, x)
        if not case["grad"]:
            return y
        kfr.fir_backward(s["taps"], x, s["gy"], s["gx"], s["gtaps"], channels=case["channels"])
        return [y, s["gx"], s["gtaps"]]
    if kind == "uneven":
        plan.execute(y, x, stream=_stream())
        return y
    if case.get("call") == "sync":
        plan.execute(y, x, inverse=case["inverse"])
        return y
    plan.execute_batch(y, x, case["batch"], inverse=case["inverse"], stream=_stream())
    return y


# ------------------------------------------------------------------------------------------------------
# work and exact
# ------------------------------------------------------------------------------------------------------


def _fft_flops(n):
    return 5.0 * n * math.log2(n) if n > 1 else 0.0


def work(case):
    kind = case["kind"]
    if kind == "dft":
        n, b = case["n"], case["batch"]
        return {"bytes": (16 if case["dtype"] == "f32" else 32) * n * b, "flops": b * _fft_flops(n)}
    if kind == "real":
        n, b = case["n"], case["batch"]
        bins = n // 2 + (1 if case["fmt"] == "CCs" else 0)
        return {"bytes": b * (4 * n + 8 * bins), "flops": b * _fft_flops(n) / 2}
    if kind == "dct":
        n, b = case["n"], case["batch"]
        return {"bytes": 8 * n * b, "flops": b * _fft_flops(n) / 2}
    if kind == "fir":
        total, m = case["channels"] * case["n"], case["taps"]
        f = 8 * m  # overlap-save through real transforms of about eight times the taps
        per = (2 * _fft_flops(f) / 2 + 3 * f) / (f - m)
        # forward: x in, y out; with gradients also gy in, gx out, and x, gy once more shared with those reads
        return {"bytes": (16 if case["grad"] else 8) * total + 4 * m * (3 if case["grad"] else 1),
                "flops": total * per * (3.0 if case["grad"] else 1.0)}
    if kind == "uneven":
        lengths = _lengths(case)
        return {"bytes": 16 * sum(lengths), "flops": sum(_fft_flops(n) for n in lengths)}
    shape, b = _shape(case), case["batch"]
    n = math.prod(shape)
    if not case["real"]:
        return {"bytes": 16 * n * b, "flops": b * _fft_flops(n)}
    return {"bytes": b * (4 * n + 8 * (n // shape[-1]) * (shape[-1] // 2 + 1)), "flops": b * _fft_flops(n) / 2}


def _exact_dct(x, inverse):
    n = x.shape[-1]
    k = torch.arange(n, dtype=torch.float64, device=x.device)
    rot = torch.exp(torch.complex(torch.zeros_like(k), -math.pi * k / (2 * n)))
    evens, odds = (n + 1) // 2, n // 2
    if not inverse:
        # the even samples, then the odd ones backwards
        v = torch.cat([x[:, 0::2], x[:, 1::2].flip(-1)], dim=-1).to(torch.float64)
        return (torch.fft.fft(v) * rot).real
    w = x.to(torch.float64) * rot
    w[:, 0] *= 0.5
    v = torch.fft.fft(w).real
    y = torch.empty_like(v)
    y[:, 0::2] = v[:, :evens]
    y[:, 1::2] = v[:, evens:].flip(-1)[:, :odds]
    return y


def _exact_fir(s, case):
    n, m = case["n"], case["taps"]
    size = 1 << (n + m - 1).bit_length()
    h = torch.fft.rfft(s["taps"].to(torch.float64), size)
    y, gx = torch.empty_like(s["x"], dtype=torch.float64), None
    gt = torch.zeros(m, dtype=torch.float64, device="cuda")
    if case["grad"]:
        gx = torch.empty_like(y)
    for c in range(case["channels"]):
        xs = torch.fft.rfft(s["x"][c].to(torch.float64), size)
        y[c] = torch.fft.irfft(xs * h, size)[:n]
        if case["grad"]:
            gs = torch.fft.rfft(s["gy"][c].to(torch.float64), size)
            gx[c] = torch.fft.irfft(gs * h.conj(), size)[:n]
            gt += torch.fft.irfft(gs * xs.conj(), size)[:m]
    return [y, gx, gt] if case["grad"] else y


def exact(case, seed):
    kind = case["kind"]
    s = _inputs(case, seed)
    x = s["x"]
    if kind == "dft":
        x = x.to(torch.complex128)
        return torch.fft.ifft(x, norm="forward") if case["inverse"] else torch.fft.fft(x)
    if kind == "real":
        if not case["inverse"]:
            y = torch.fft.rfft(x.to(torch.float64))
            if case["fmt"] == "CCs":
                return y
            p = y[:, :-1].clone()
            p[:, 0] = torch.complex(y[:, 0].real.clone(), y[:, -1].real.clone())
            return p
        x = x.to(torch.complex128)
        if case["fmt"] != "CCs":
            zero = torch.zeros_like(x[:, 0].real)
            last = torch.complex(x[:, 0].imag.clone(), zero)
            x = torch.cat([x, last[:, None]], dim=-1)
            x[:, 0] = torch.complex(x[:, 0].real.clone(), zero)
        return torch.fft.irfft(x, case["n"], norm="forward")
    if kind == "dct":
        return _exact_dct(x, case["inverse"])
    if kind == "fir":
        return _exact_fir(s, case)
    if kind == "uneven":
        y = torch.empty(x.shape, dtype=torch.complex128, device="cuda")
        at = 0
        for n in _lengths(case):
            y[at:at + n] = torch.fft.fft(x[at:at + n].to(torch.complex128))
            at += n
        return y
    shape = _shape(case)
    dims = tuple(range(1, len(shape) + 1))
    if not case["real"]:
        x = x.to(torch.complex128)
        return torch.fft.ifftn(x, dim=dims, norm="forward") if case["inverse"] else torch.fft.fftn(x, dim=dims)
    if not case["inverse"]:
        return torch.fft.rfftn(x.to(torch.float64), dim=dims)
    return torch.fft.irfftn(x.to(torch.complex128), s=shape, dim=dims, norm="forward")
