"""What a caller's own kernel may rely on behind the library's chained passes: one
launched with the programmatic attribute that reads before its wait finds what a
kernel two places in front of it wrote."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from helpers import to_dev, to_host
from oracle import oracle as O
from parafaft_b200 import native as nv

pytestmark = pytest.mark.gpu

SOURCE = r"""
extern "C" __global__ void early_read(const float *a, float *out, long long n) {
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * 256;
  if (i < n)
    out[i / 256] = __ldcg(a + i);
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
"""


class Attr(C.Structure):  # CUlaunchAttribute: id, padding, 64-byte value
    _fields_ = [("id", C.c_int), ("pad", C.c_int), ("value", C.c_int * 16)]


class Config(C.Structure):  # CUlaunchConfig
    _fields_ = [("dims", C.c_uint * 6), ("smem", C.c_uint), ("stream", C.c_void_p),
                ("attrs", C.POINTER(Attr)), ("count", C.c_uint)]


def test_early_reads_behind_chained_passes(tmp_path):
    import torch
    src, cubin = tmp_path / "k.cu", tmp_path / "k.cubin"
    src.write_text(SOURCE)
    subprocess.run(["nvcc", "-cubin", "-gencode", "arch=compute_100a,code=sm_100a", "-o",
                    str(cubin), str(src)], check=True)
    n, b, small = 512, 12000, 64  # 98 MB of traffic in the first pass
    x = O.normal_complex(n * b, 1).astype(np.complex64)
    a, c = to_dev(x), to_dev(np.zeros(64 * small, np.complex64))
    out = torch.zeros(2 * n * b // 256, device="cuda")
    s = torch.cuda.Stream()
    h = nv.Handle(nv.F32, 3)
    h.plan_c2c(0, n, b, 1, n)
    h.plan_c2c(1, 64, small, 1, 64)
    h.set_stream(s.cuda_stream)
    torch.cuda.synchronize()
    cu = C.CDLL("libcuda.so.1")
    mod, fn = C.c_void_p(), C.c_void_p()
    assert cu.cuModuleLoad(C.byref(mod), str(cubin).encode()) == 0
    assert cu.cuModuleGetFunction(C.byref(fn), mod, b"early_read") == 0
    attr = Attr(id=6)  # programmatic stream serialization
    attr.value[0] = 1
    total = C.c_longlong(2 * n * b)
    pa, po = C.c_void_p(a.data_ptr()), C.c_void_p(out.data_ptr())
    args = (C.c_void_p * 3)(C.addressof(pa), C.addressof(po), C.addressof(total))
    blocks = (2 * n * b // 256 + 255) // 256
    cfg = Config(dims=(blocks, 1, 1, 256, 1, 1), stream=s.cuda_stream, attrs=C.pointer(attr),
                 count=1)
    for i in range(20):
        direction = (nv.FORWARD, nv.BACKWARD)[i % 2]
        h.exec_c2c(0, direction, a)
        h.exec_c2c(1, direction, c)
        assert cu.cuLaunchKernelEx(C.byref(cfg), fn, args, None) == 0
        s.synchronize()
        want = to_host(a).view(np.float32)[::256]
        assert np.array_equal(to_host(out), want), i
    h.set_stream(None)
    cu.cuModuleUnload(mod)


LAUNCH_ERROR = r"""
import ctypes as C, sys
sys.path[:0] = [%r, %r]
import numpy as np, torch
from helpers import to_dev, to_host
from oracle import oracle as O
from parafaft_b200 import native as nv
cu = C.CDLL("libcuda.so.1")
n, b = 64, 40
x = O.normal_complex(n * b, 1).astype(np.complex64)
d = to_dev(x)
out = torch.empty_like(d)
for _ in range(2):
    nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, d, out)
    torch.cuda.synchronize()
s = C.c_void_p()  # a stream that the default stream would have to wait for
assert cu.cuStreamCreate(C.byref(s), 0) == 0
assert cu.cuStreamBeginCapture_v2(s, 2) == 0
try:
    nv.c2c_noalloc(nv.F32, nv.FORWARD, n, b, b, 1, d, out)
    raise SystemExit("the launch was accepted")
except nv.B200FFTError as e:
    assert "transform kernel" in str(e), e
g = C.c_void_p()
cu.cuStreamEndCapture(s, C.byref(g))
h = nv.Handle(nv.F32, 1)
h.plan_c2c(0, 17, 8, 1, 17)  # a table and a launch that ask for the last error
y = O.normal_complex(17 * 8, 2).astype(np.complex64)
e = to_dev(y)
h.exec_c2c(0, nv.FORWARD, e)
h.sync()
assert O.rel_l2(to_host(e), O.c2c_batch(y.astype(np.complex128), 17, 8, 1, 17, -1)) < 2e-6
"""


def test_a_refused_launch_leaves_no_error_behind():
    """A call on the default stream while a stream it synchronises with captures is
    refused; the next call does not report that error again."""
    root = Path(__file__).resolve().parents[1]
    r = subprocess.run([sys.executable, "-c", LAUNCH_ERROR % (str(root), str(root / "tests"))],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("prec", [nv.F32, nv.F64])
def test_default_stream_chains_wait_for_blocking_streams(prec):
    """Chained calls on the default stream with passes of a handle's own (blocking)
    stream in between: the same bits as waiting after every call."""
    import torch
    n, b = 512, 6000
    x = O.normal_complex(n * b, 3).astype(np.complex64 if prec == nv.F32 else np.complex128)
    a = to_dev(x)
    y, z = torch.empty_like(a), torch.empty_like(a)
    h = nv.Handle(prec, 1)
    h.plan_c2c(0, n, b, b, 1)

    def run(wait):
        step = torch.cuda.synchronize if wait else (lambda: None)
        for _ in range(4):
            nv.c2c_noalloc(prec, nv.FORWARD, n, b, 1, n, a, y); step()
            h.exec_c2c(0, nv.FORWARD, y); step()
            nv.c2c_noalloc(prec, nv.BACKWARD, n, b, 1, n, y, z); step()
        torch.cuda.synchronize()
        return to_host(z)

    torch.cuda.synchronize()
    want = run(True)
    for _ in range(3):
        z.zero_()
        torch.cuda.synchronize()
        assert np.array_equal(run(False), want)
