"""Passes launched as programmatic dependent launches read what the work in front
of them wrote: chains of dependent passes without host waits, mixed with copies
and other kernels on the same and on other streams, repeated from the same start
must give the same bits as waiting after every call."""
import numpy as np
import pytest

from helpers import cdtype, to_dev, to_host
from oracle import oracle as O
from parafaft_b200 import native as nv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [nv.F32, nv.F64])
@pytest.mark.parametrize("shape", [(8, 16), (64, 64), (100, 36), (512, 128), (50, 2048)])
def test_chains_equal_synchronised_calls(prec, shape):
    import torch
    n0, n1 = shape
    x = O.normal_complex(n0 * n1, 1).astype(cdtype(prec))
    h = nv.Handle(prec, 2)
    h.plan_c2c(0, n0, n1, n1, 1)
    h.plan_c2c(1, n1, n0, 1, n1)
    a, b = to_dev(x), to_dev(np.zeros_like(x))
    nbytes = x.nbytes

    def chain(wait):
        step = h.sync if wait else (lambda: None)
        a.copy_(to_dev(x))
        torch.cuda.synchronize()
        for i in range(6):
            h.memcpy(b, a, nbytes)
            h.exec_c2c(1, nv.FORWARD, b); step()
            h.exec_c2c(0, nv.FORWARD, b); step()
            h.memcpy(a, b, nbytes)
            h.exec_c2c(0, nv.BACKWARD, a); step()
            h.exec_c2c(1, nv.BACKWARD, a); step()
            if i % 2:
                h.flush()
                a.mul_(1.0 / (n0 * n1))  # a kernel of another library in between
            else:
                h.flush()
                b.copy_(a)
                a.copy_(b.div_(n0 * n1))
        h.sync()
        return to_host(a), to_host(b)

    want = chain(True)
    for _ in range(3):
        got = chain(False)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert O.rel_l2(want[0], x) < (1e-4 if prec == nv.F32 else 1e-12)


def test_captured_by_the_caller_with_fork_and_join():
    """A caller's capture with two streams: passes of two handles forked and
    joined by events replay correctly."""
    import torch
    n, b = 64, 300
    xs = [O.normal_complex(n * b, k).astype(np.complex64) for k in (1, 2)]
    ds = [to_dev(x) for x in xs]
    side = torch.cuda.Stream()
    hs = []
    for _ in range(2):
        h = nv.Handle(nv.F32, 2)
        h.plan_c2c(0, n, b, b, 1)
        h.plan_c2c(1, b, n, 1, b)
        hs.append(h)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        for h, d, s in zip(hs, ds, (main, side)):
            h.set_stream(s.cuda_stream)
            h.exec_c2c(1, nv.FORWARD, d)
            h.exec_c2c(0, nv.FORWARD, d)
        main.wait_stream(side)
        hs[0].exec_c2c(0, nv.BACKWARD, ds[1])
        hs[0].exec_c2c(1, nv.BACKWARD, ds[1])
    for _ in range(2):
        for d, x in zip(ds, xs):
            d.copy_(to_dev(x))
        g.replay()
        torch.cuda.synchronize()
        assert O.rel_l2(to_host(ds[0]).reshape(n, b), np.fft.fft2(xs[0].reshape(n, b))) < 2e-6
        assert O.rel_l2(to_host(ds[1]) / (n * b), xs[1]) < 2e-6
    for h in hs:
        h.set_stream(None)


@pytest.mark.parametrize("captured", [False, True])
def test_single_grid_groups_chain(captured):
    """The levels of one grid's group follow one another, replayed back to back."""
    n0, n1, n2 = 36, 50, 64
    nc = n2 // 2 + 1
    x = O.normal_real((n0, n1, n2), 4).astype(np.float64)
    src, dst = to_dev(O.pad_real(x, np.float64)), to_dev(np.zeros(n0 * n1 * 2 * nc))
    h = nv.Handle(nv.F64, 2)
    h.plan_c2c(0, n0, n1 * nc, n1 * nc, 1)
    h.plan_c2c(1, n1, nc, nc, 1)
    h.plan_r2c(n2, n0 * n1, 1, 2 * nc)
    g = nv.Group([h])
    g.begin()
    h.memcpy(dst, src, n0 * n1 * 2 * nc * 8)
    h.exec_r2c(dst)
    for i in range(n0):
        h.exec_c2c(1, nv.FORWARD, dst.data_ptr() + i * n1 * nc * 16)
    h.exec_c2c(0, nv.FORWARD, dst)
    g.end()
    g.sync()
    if captured:
        g.capture()
    for _ in range(20):
        g.replay()
    g.sync()
    X = to_host(dst).view(np.complex128).reshape(n0, n1, nc)
    assert O.rel_l2(X, O.r2c_nd(x)) < 1e-12
