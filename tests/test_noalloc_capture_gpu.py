"""b200fft_c2c_noalloc around its table's one fill, each case in a process of its
own (the first call of a precision fills): captures after one warm-up call, calls
while the fill is still in flight, calls beside another stream's capture."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

PRELUDE = r"""
import ctypes as C, sys
import numpy as np, torch
sys.path[:0] = [%r, %r]
from helpers import cdtype, to_dev, to_host, tol
from oracle import oracle as O
from parafaft_b200 import native as nv
cu = C.CDLL("libcuda.so.1")

def begin(stream, mode=0):
    assert cu.cuStreamBeginCapture_v2(C.c_void_p(stream.cuda_stream), mode) == 0

def end(stream):
    g = C.c_void_p()
    assert cu.cuStreamEndCapture(C.c_void_p(stream.cuda_stream), C.byref(g)) == 0
    return g

def node_types(g):
    n = C.c_size_t(0)
    assert cu.cuGraphGetNodes(g, None, C.byref(n)) == 0
    if n.value == 0:
        return []
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(g, nodes, C.byref(n)) == 0
    out = []
    for x in nodes:
        t = C.c_int()
        assert cu.cuGraphNodeGetType(C.c_void_p(x), C.byref(t)) == 0
        out.append(t.value)
    return sorted(out)  # 0 kernel, 6 event wait

def launch(g, stream):
    e = C.c_void_p()
    assert cu.cuGraphInstantiateWithFlags(C.byref(e), g, C.c_ulonglong(0)) == 0
    assert cu.cuGraphLaunch(e, C.c_void_p(stream.cuda_stream)) == 0

def data(prec, n, b, seed):
    x = O.normal_complex(n * b, seed).astype(cdtype(prec))
    d = to_dev(x)
    return x, d, torch.empty_like(d)

def right(prec, x, out, n, b, direction=nv.FORWARD, stride=None, dist=1):
    ref = O.c2c_batch(x.astype(np.complex128), n, b, stride or b, dist,
                      -1 if direction == nv.FORWARD else 1)
    return O.rel_l2(to_host(out), ref) < tol(prec)

def load(prec, n, b, stride, dist):
    # the first launch of a kernel may wait for the device while it loads: a
    # handle's plan of the same shape launches the same kernels, and a call of
    # the other precision the library's own part, without filling this table
    h = nv.Handle(prec, 1)
    h.plan_c2c(0, n, b, stride, dist)
    d = torch.zeros(2 * n * b, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    h.exec_c2c(0, nv.FORWARD, d)
    h.exec_c2c(0, nv.BACKWARD, d)
    h.sync()
    nv.c2c_noalloc(1 - prec, nv.FORWARD, 2, 1, 1, 2, d, d)
    torch.cuda.synchronize()

def long_work(stream):
    # ordinary products, about a quarter of a second
    with torch.cuda.stream(stream):
        a = torch.ones(8192, 8192, device="cuda", dtype=torch.bfloat16)
        for _ in range(300):
            a @ a
    return a
""" % (str(ROOT), str(ROOT / "tests"))


def _run(body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + body], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_captured_calls_are_one_kernel_each():
    """One warm-up call and a wait, then a capture: no fill in the graph."""
    _run(r"""
n, b = 256, 77
for prec in (nv.F32, nv.F64):
    x, d, y = data(prec, n, b, 3)
    z = torch.empty_like(d)
    s = torch.cuda.Stream()
    nv.c2c_noalloc(prec, nv.FORWARD, n, b, b, 1, d, y)
    torch.cuda.synchronize()
    begin(s)
    nv.c2c_noalloc(prec, nv.FORWARD, n, b, b, 1, d, y, s.cuda_stream)
    nv.c2c_noalloc(prec, nv.BACKWARD, n, b, b, 1, y, z, s.cuda_stream)
    g = end(s)
    assert node_types(g) == [0, 0], node_types(g)
    y.zero_()
    torch.cuda.synchronize()
    launch(g, s)
    assert right(prec, x, y, n, b)
    assert O.rel_l2(to_host(z) / n, x) < tol(prec)
""")


def test_capture_while_the_fill_is_in_flight():
    """The fill waits behind other work of its stream: the captured call waits
    for it and does not fill again."""
    _run(r"""
n, b = 128, 50
load(nv.F32, n, b, b, 1)
x, d, y = data(nv.F32, n, b, 4)
y2 = torch.empty_like(d)
first, s = torch.cuda.Stream(), torch.cuda.Stream()
torch.cuda.synchronize()
keep = long_work(first)
nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, d, y, first.cuda_stream)
begin(s)
nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, d, y2, s.cuda_stream)
g = end(s)
assert not first.query()  # the fill was in flight all along
assert node_types(g) == [0, 6], node_types(g)
launch(g, s)
torch.cuda.synchronize()
nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, d, y)
launch(g, s)  # the event the graph waits for is still there
assert right(nv.F32, x, y, n, b) and right(nv.F32, x, y2, n, b)
""")


@pytest.mark.parametrize("prec", [0, 1])
def test_calls_on_other_streams_wait_for_the_fill(prec):
    """Calls of many lengths on four streams, nothing waited for in between, all
    issued while the first call's fill is behind other work."""
    _run(f"prec = {prec}" + r"""
streams = [torch.cuda.Stream() for _ in range(4)]
work = []
for i, n in enumerate([256, 4096, 8, 128, 512, 16, 1024, 64, 2048, 2, 4, 32]):
    for col in (True, False):
        b = 33 + i
        stride, dist = (b, 1) if col else (1, n)
        load(prec, n, b, stride, dist)
        x, d, out = data(prec, n, b, i)
        work.append((n, b, stride, dist, (nv.FORWARD, nv.BACKWARD)[i % 2], x, d, out))
torch.cuda.synchronize()
keep = long_work(streams[0])
for i, (n, b, stride, dist, direction, x, d, out) in enumerate(work):
    nv.c2c_noalloc(prec, direction, n, b, stride, dist, d, out, streams[i % 4].cuda_stream)
assert not streams[0].query()  # every call came before the fill
torch.cuda.synchronize()
for n, b, stride, dist, direction, x, d, out in work:
    assert right(prec, x, out, n, b, direction, stride, dist), (prec, n, stride)
""")


def test_calls_beside_another_streams_capture():
    """A call on a stream that captures nothing leaves a capture in global mode
    on another stream valid, also the one that first sees the fill finished."""
    _run(r"""
n, b = 64, 40
x, d, y = data(nv.F32, n, b, 5)
a, s = torch.cuda.Stream(), torch.cuda.Stream()
nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, d, y, s.cuda_stream)
torch.cuda.synchronize()
begin(a)
nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, d, y, s.cuda_stream)
g = end(a)
assert node_types(g) == []
assert right(nv.F32, x, y, n, b)
""")
