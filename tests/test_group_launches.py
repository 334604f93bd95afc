"""Groups of many small grids share their launches whatever the axis lengths
(record-only launch counts), large passes launch alone, and the shared launches
of compiled plans give the oracle's values."""
import math

import numpy as np
import pytest

from helpers import cdtype, rdtype, to_dev, to_host, tol
from oracle import oracle as O
from parafaft_b200 import native as nv


def _handle(shape, real, prec, flags=0):
    h = nv.Handle(prec, len(shape), flags=flags)
    w = shape[-1] // 2 + 1 if real else shape[-1]
    dims = shape[:-1] + (w,)
    for ax in range(len(shape) - 1):
        trail = math.prod(dims[ax + 1:])
        h.plan_c2c(ax, shape[ax], trail, trail, 1)
    rows = math.prod(shape[:-1])
    if real:
        h.plan_r2c(shape[-1], rows, 1, 2 * w)
        h.plan_c2r(shape[-1], rows, 1, 2 * w)
    else:
        h.plan_c2c(len(shape) - 1, shape[-1], rows, 1, shape[-1])
    return h, dims


def _forward(h, dims, real, ptr, csize):
    if real:
        h.exec_r2c(ptr)
    else:
        h.exec_c2c(len(dims) - 1, nv.FORWARD, ptr)
    for ax in range(len(dims) - 2, -1, -1):
        slab = math.prod(dims[ax:]) * csize
        for i in range(math.prod(dims[:ax])):
            h.exec_c2c(ax, nv.FORWARD, ptr + i * slab)


def _launches(shape, real, prec, count, flags=0):
    hs = [_handle(shape, real, prec, flags | nv.FLAG_RECORD_ONLY) for _ in range(count)]
    g = nv.Group([h for h, _ in hs])
    g.begin()
    cs = 16 if prec == nv.F64 else 8
    for i, (h, dims) in enumerate(hs):
        _forward(h, dims, real, (i + 1) << 34, cs)
    g.end()
    n = g.stats()["kernel_launches"]
    g.close()
    return n


@pytest.mark.parametrize("shape,real,prec", [
    ((256, 256), False, nv.F32), ((384, 384), True, nv.F32), ((64, 512), True, nv.F64),
    ((64, 1024), True, nv.F32), ((200, 200), False, nv.F32), ((30, 4096), False, nv.F32),
    ((300, 75), True, nv.F64), ((2025, 40), False, nv.F64)])
def test_many_small_grids_share_launches(monkeypatch, shape, real, prec):
    """64 grids run as three chains of one launch per axis."""
    monkeypatch.setenv("B200FFT_RECORD_ONLY", "1")
    assert _launches(shape, real, prec, 64) == 6


def test_large_compiled_passes_launch_alone(monkeypatch):
    """300x300x300 C2C FP32: 432 MB per pass; three grids of three axes. Two
    split-precision grids of 64x256x512 (128 MB per pass) share every launch."""
    monkeypatch.setenv("B200FFT_RECORD_ONLY", "1")
    assert _launches((300, 300, 300), False, nv.F32, 3) == 9
    assert _launches((64, 256, 512), False, nv.F32, 2, nv.FLAG_SPLIT_TC) == 3


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [nv.F32, nv.F64])
@pytest.mark.parametrize("shapes,real", [
    ([(20, 75), (9, 75)], True), ([(12, 15, 45), (36, 7, 45)], True),
    ([(256, 256), (64, 256)], False), ([(33, 512), (300, 512)], False),
    ([(24, 2048), (5, 2048)], False), ([(225, 384), (10, 384)], True),
    ([(40, 1024), (64, 1024)], True), ([(360, 200), (200, 200)], False)])
def test_shared_launches_match_the_oracle(prec, shapes, real):
    cs = 16 if prec == nv.F64 else 8
    hs, ds, xs = [], [], []
    for i, shape in enumerate(shapes * 2):
        h, dims = _handle(shape, real, prec)
        if real:
            x = O.normal_real(shape, i).astype(rdtype(prec))
            d = to_dev(O.pad_real(x, rdtype(prec)))
        else:
            x = O.normal_complex(math.prod(shape), i).reshape(shape).astype(cdtype(prec))
            d = to_dev(x)
        hs.append((h, dims))
        ds.append(d)
        xs.append(x)
    g = nv.Group([h for h, _ in hs])
    g.begin()
    for (h, dims), d in zip(hs, ds):
        _forward(h, dims, real, d.data_ptr(), cs)
    g.end()
    g.sync()
    assert g.stats()["kernel_launches"] < g.stats()["passes_per_run"]
    for (h, dims), d, x in zip(hs, ds, xs):
        X = to_host(d)
        X = X.view(cdtype(prec)).reshape(dims)
        ref = (O.r2c_nd(x.astype(np.float64)) if real
               else np.fft.fftn(x.astype(np.complex128)))
        assert O.rel_l2(X, ref) < tol(prec), (dims, real)
    g.close()
