"""What a caller's own kernel may rely on behind the library's chained passes: one
launched with the programmatic attribute that reads before its wait finds what a
kernel two places in front of it wrote."""
import ctypes as C
import subprocess

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
