"""Kernels launched behind one another without a full stop between them (launch_kernel): a chain of calls that read
and overwrite one another's buffers gives, bit for bit, what the same calls give one at a time, on a stream of their
own, on the default stream and in a captured graph, with foreign kernels and copies in between."""
import pytest
import torch

import kfr_gb300 as k

pytestmark = pytest.mark.gpu


def _calls(kind, n, batch):
    """two buffers and a launch forward into the second and back into the first"""
    g = torch.Generator().manual_seed(n)
    p = {"c2c": k.dft_plan, "real": k.dft_plan_real, "dct": k.dct_plan}[kind](n)
    x = torch.randn(batch, n, dtype=torch.complex64 if kind == "c2c" else torch.float32, generator=g).cuda()
    y = torch.zeros(batch, p.complex_size, dtype=torch.complex64, device="cuda") if kind == "real" else torch.zeros_like(x)
    size = k._call(p._fn("get_temp_size_batch"), p.handle, batch)
    tmp = torch.empty(max(1, size), dtype=torch.uint8, device="cuda")

    def step(st):
        p.execute_batch(y, x, batch, temp=tmp, stream=st)
        p.execute_batch(x, y, batch, temp=tmp, inverse=True, stream=st)
    return x, y, step, 1.0 / n


def _chain(x, y, step, scale, st, wait):
    seen = []
    for i in range(6):
        step(st)
        wait()
        x.mul_(scale)         # a foreign kernel between two calls
        wait()
        seen.append(y.clone())
        wait()
    return seen + [x.clone()]


@pytest.mark.parametrize("where", ["stream", "default", "graph"])
@pytest.mark.parametrize("kind,n,batch", [
    ("c2c", 64, 3), ("c2c", 4096, 300), ("c2c", 3600, 200), ("c2c", 8191, 40), ("c2c", 1 << 16, 8), ("c2c", 1 << 20, 2),
    ("c2c", 250000, 3), ("real", 600, 451), ("real", 1200, 451), ("real", 48000, 30), ("real", 44100, 30),
    ("dct", 512, 600), ("dct", 1000, 300)])
def test_chain(kind, n, batch, where):
    st = torch.cuda.current_stream() if where == "default" else torch.cuda.Stream()
    x, y, step, scale = _calls(kind, n, batch)
    x0 = x.clone()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        want = _chain(x, y, step, scale, st, torch.cuda.synchronize)
        torch.cuda.synchronize()
        x.copy_(x0)
        torch.cuda.synchronize()
        if where == "graph":
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=st):
                got = _chain(x, y, step, scale, st, lambda: None)
            graph.replay()
        else:
            got = _chain(x, y, step, scale, st, lambda: None)
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got))
