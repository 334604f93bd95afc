"""b200fft_c2c_noalloc calls on several streams: the table of a precision is
filled once, and calls on other streams (lengths, layouts and directions mixed)
need no ordering among themselves."""
import numpy as np
import pytest

from helpers import cdtype, to_dev, to_host, tol
from oracle import oracle as O
from parafaft_b200 import native as nv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [nv.F32, nv.F64])
def test_streams_and_lengths_interleave(prec):
    import torch
    streams = [torch.cuda.Stream() for _ in range(4)]
    work = []
    torch.cuda.synchronize()
    for i, length in enumerate([2, 4096, 8, 128, 512, 16, 1024, 64, 2048, 256, 4, 32]):
        for col in (True, False):
            batch = 33 + i
            stride, dist = (batch, 1) if col else (1, length)
            x = O.normal_complex(length * batch, i).astype(cdtype(prec))
            d = to_dev(x)
            out = torch.empty_like(d)
            torch.cuda.synchronize()
            direction = (nv.FORWARD, nv.BACKWARD)[i % 2]
            nv.c2c_noalloc(prec, direction, length, batch, stride, dist, d, out,
                           streams[(2 * i + col) % 4].cuda_stream)
            work.append((x, out, length, batch, stride, dist, direction))
    torch.cuda.synchronize()
    for x, out, length, batch, stride, dist, direction in work:
        ref = O.c2c_batch(x.astype(np.complex128), length, batch, stride, dist,
                          -1 if direction == nv.FORWARD else 1)
        assert O.rel_l2(to_host(out), ref) < tol(prec), (length, batch, stride)


def test_captured_calls_replay():
    """A captured forward and backward replays on new inputs."""
    import torch
    n, b = 256, 77
    x = to_dev(O.normal_complex(n * b, 3).astype(np.complex64))
    y, z = torch.empty_like(x), torch.empty_like(x)
    nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, x, y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s = torch.cuda.current_stream().cuda_stream
        nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, x, y, s)
        nv.c2c_noalloc(nv.F32, nv.BACKWARD, n, b, b, 1, y, z, s)
    for seed in (5, 6):
        h = O.normal_complex(n * b, seed).astype(np.complex64)
        x.copy_(to_dev(h))
        g.replay()
        assert O.rel_l2(to_host(y), O.c2c_batch(h.astype(np.complex128), n, b, b, 1, -1)) < 2e-6
        assert O.rel_l2(to_host(z) / n, h) < 2e-6
