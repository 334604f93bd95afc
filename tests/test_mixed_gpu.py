"""The compiled mixed-length kernels (lengths of factors 2, 3, 5, 7 and one 11 or
13 up to 2048) against the FP64 oracle: every length, both layouts, both
directions and precisions, at batches around the tile, and the calls that reach
them (slices, copies, pads, strided rows, groups)."""
import re

import numpy as np
import pytest

from helpers import cdtype, rdtype, to_dev, to_host, tol
from oracle import oracle as O
from parafaft_b200 import native as nv

pytestmark = pytest.mark.gpu

PRECS = [nv.F32, nv.F64]


def _lengths(lo, hi):
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m in (1, 11, 13) and n & (n - 1):
            out.append(n)
    return out


LENGTHS = _lengths(3, 2048)


def _c2c(prec, length, batch, stride, dist, direction, flags=0):
    span = (length - 1) * stride + (batch - 1) * dist + 1
    x = O.normal_complex(span, length + batch).astype(cdtype(prec))
    h = nv.Handle(prec, 1, flags=flags)
    h.plan_c2c(0, length, batch, stride, dist)
    d = to_dev(x)
    h.exec_c2c(0, direction, d)
    h.sync()
    ref = O.c2c_batch(x.astype(np.complex128), length, batch, stride, dist,
                      -1 if direction == nv.FORWARD else +1)
    return to_host(d), ref, h.plan_describe(nv.KIND_C2C, 0)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("part", range(4))
def test_every_length_rows_and_columns(prec, part):
    """One whole tile and one more transform of every length, both layouts."""
    for n in LENGTHS[part::4]:
        for col in (True, False):
            batch = 17 if n < 600 else 5
            stride, dist = (batch, 1) if col else (1, n)
            y, ref, desc = _c2c(prec, n, batch, stride, dist, n % 2)
            assert O.rel_l2(y, ref) < tol(prec), (n, col, desc)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("length", [3, 13, 30, 36, 105, 175, 264, 300, 350, 640, 1000, 1225, 2016])
def test_batches_around_the_tile(prec, length):
    for col in (True, False):
        if not col and length in (3, 13):
            continue
        d = nv.describe(prec, nv.KIND_C2C, length, 4, 4 if col else 1, 1 if col else length)
        tb = int(re.search(r"on \d+x(\d+) threads", d).group(1))
        for batch in {1, max(1, tb - 1), tb, tb + 1, 2 * tb + 1}:
            for direction in (nv.FORWARD, nv.BACKWARD):
                stride, dist = (batch, 1) if col else (1, length)
                y, ref, _ = _c2c(prec, length, batch, stride, dist, direction)
                assert O.rel_l2(y, ref) < tol(prec), (length, col, batch)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("length", [36, 100, 225, 1000])
def test_strides_and_gaps_match_the_generic_kernel(prec, length):
    """Point strides and distances with gaps: what the pass does not own keeps
    its values, and the results are the generic kernel's to rounding."""
    for batch, stride, dist in ((9, 3, 3 * length + 1), (9, 21, 2), (5, 1, length + 3), (4, 7, 1)):
        y, ref, _ = _c2c(prec, length, batch, stride, dist, nv.BACKWARD)
        g, _, gd = _c2c(prec, length, batch, stride, dist, nv.BACKWARD, nv.FLAG_GENERIC_ONLY)
        assert "compiled" not in gd
        assert O.rel_l2(y, ref) < tol(prec), (length, batch, stride, dist)
        assert O.rel_l2(y, g) < 2 * tol(prec)
        own = np.zeros(y.size, bool)
        for b in range(batch):
            own[b * dist + stride * np.arange(length)] = True
        assert np.array_equal(y[~own], g[~own])


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("n", [9, 12, 15, 18, 45, 72, 105, 126, 200, 225, 350, 500, 675, 1000,
                               1125, 1250, 2000, 2025, 3000, 4032])
def test_r2c_c2r_rows(prec, n):
    nc = n // 2 + 1
    for batch in (1, 3, 25):
        for dist in (2 * nc, 2 * nc + 4):
            x = O.normal_real((batch, n), n).astype(rdtype(prec))
            buf = np.full((batch, dist), 7.0, dtype=rdtype(prec))
            buf[:, :n] = x
            h = nv.Handle(prec, 0)
            h.plan_r2c(n, batch, 1, dist)
            h.plan_c2r(n, batch, 1, dist)
            d = to_dev(buf.reshape(-1))
            h.exec_r2c(d)
            h.sync()
            got = to_host(d).reshape(batch, dist)
            X = np.ascontiguousarray(got[:, :2 * nc]).view(cdtype(prec))
            ref = np.stack([O.r2c_nd(r) for r in x.astype(np.float64)])
            assert O.rel_l2(X, ref) < tol(prec), (n, batch, dist)
            assert np.all(got[:, 2 * nc:] == 7.0)
            # C2R ignores the imaginary parts of DC and (even n) Nyquist
            Y = X.copy()
            Y[:, 0] += 3j
            if n % 2 == 0:
                Y[:, -1] -= 2j
            got[:, :2 * nc] = Y.view(rdtype(prec))
            d = to_dev(got.reshape(-1))
            h.exec_c2r(d)
            h.sync()
            back = to_host(d).reshape(batch, dist)
            assert O.rel_l2(back[:, :n] / n, x) < tol(prec), (n, batch, dist)
            assert np.all(back[:, 2 * nc:] == 7.0)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("n", [75, 100])
def test_slices_copy_and_pad_fuse(prec, n):
    """A 3-D R2C forward on mixed sides: pad, copy and slice loop fold into
    three launches, equal to the unfused calls bit for bit."""
    n0, n1, nc = 21, 45, n // 2 + 1
    x = O.normal_real((n0, n1, n), 5).astype(rdtype(prec))
    es, outs = x.itemsize, {}
    for flags in (0, nv.FLAG_NO_DEFER):
        h = nv.Handle(prec, 2, flags=flags)
        h.plan_c2c(0, n0, n1 * nc, n1 * nc, 1)
        h.plan_c2c(1, n1, nc, nc, 1)
        h.plan_r2c(n, n0 * n1, 1, 2 * nc)
        src = to_dev(x.reshape(-1))
        a = to_dev(np.zeros(n0 * n1 * 2 * nc, rdtype(prec)))
        b = to_dev(np.zeros(n0 * n1 * 2 * nc, rdtype(prec)))
        h.memcpy2d(a, 2 * nc * es, src, n * es, n * es, n0 * n1)
        h.exec_r2c(a)
        h.memcpy(b, a, n0 * n1 * 2 * nc * es)
        for i in range(n0):
            h.exec_c2c(1, nv.FORWARD, b.data_ptr() + i * n1 * nc * 2 * es)
        h.exec_c2c(0, nv.FORWARD, b)
        h.sync()
        if flags == 0:
            st = h.stats()
            assert st["kernel_launches"] == 3 and st["copies_issued"] == 0, st
        outs[flags] = to_host(b).view(cdtype(prec)).reshape(n0, n1, nc)
    assert np.array_equal(outs[0], outs[nv.FLAG_NO_DEFER])
    assert O.rel_l2(outs[0], O.r2c_nd(x.astype(np.float64))) < tol(prec)


@pytest.mark.parametrize("count", [2, 24])
def test_groups_of_mixed_lengths(count):
    """Groups whose passes launch alone and (many small grids) share a launch."""
    sides = [(20, 36, 50), (100, 90, 84)]
    hs, ds, xs = [], [], []
    for i in range(count):
        s = sides[i % 2] if i < 4 else sides[0]
        nc = s[2] // 2 + 1
        x = O.normal_real(s, i).astype(np.float32)
        h = nv.Handle(nv.F32, 2)
        h.plan_c2c(0, s[0], s[1] * nc, s[1] * nc, 1)
        h.plan_c2c(1, s[1], nc, nc, 1)
        h.plan_r2c(s[2], s[0] * s[1], 1, 2 * nc)
        hs.append(h)
        ds.append(to_dev(O.pad_real(x, np.float32)))
        xs.append(x)
    g = nv.Group(hs)
    g.begin()
    for h, d, x in zip(hs, ds, xs):
        nc = x.shape[2] // 2 + 1
        h.exec_r2c(d)
        for k in range(x.shape[0]):
            h.exec_c2c(1, nv.FORWARD, d.data_ptr() + k * x.shape[1] * nc * 8)
        h.exec_c2c(0, nv.FORWARD, d)
    g.end()
    g.sync()
    assert g.stats()["passes_per_run"] == 3 * count
    for d, x in zip(ds, xs):
        nc = x.shape[2] // 2 + 1
        X = to_host(d).view(np.complex64).reshape(x.shape[0], x.shape[1], nc)
        assert O.rel_l2(X, O.r2c_nd(x.astype(np.float64))) < tol(nv.F32)
    g.close()


def test_measured_plans_keep_the_compiled_kernel():
    """Measure and Patient planning (and a plan cache entry of the runtime
    schedule) keep the compiled kernel of a mixed length."""
    nv.forget_wisdom()
    work = to_dev(np.zeros(100 * 64 * 2, np.float32))
    for flag in (nv.PLAN_MEASURE, nv.PLAN_PATIENT, nv.PLAN_MEASURE):
        h = nv.Handle(nv.F32, 1, plan_flag=flag)
        h.set_work_buffer(work, 100 * 64 * 8)
        h.plan_c2c(0, 100, 64, 64, 1)
        assert h.plan_describe(nv.KIND_C2C, 0).count("compiled=") == 1
    nv.forget_wisdom()


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("length", [8, 16, 32, 64, 128, 256, 512, 2048, 4096])
def test_compiled_power_of_two_rows(prec, length):
    """Rows of powers of two on compiled plans: batches around the tile, both
    directions, and R2C/C2R of twice the length."""
    d = nv.describe(prec, nv.KIND_C2C, length)
    tb = re.search(r"on \d+x(\d+) threads", d)
    tb = int(tb.group(1)) if tb else 4
    for batch in {1, max(1, tb - 1), tb, tb + 1, 3 * tb + 1}:
        for direction in (nv.FORWARD, nv.BACKWARD):
            y, ref, _ = _c2c(prec, length, batch, 1, length, direction)
            assert O.rel_l2(y, ref) < tol(prec), (length, batch, d)
        if length > 2048:
            continue
        n, nc = 2 * length, length + 1
        x = O.normal_real((batch, n), batch).astype(rdtype(prec))
        h = nv.Handle(prec, 0)
        h.plan_r2c(n, batch, 1, 2 * nc)
        h.plan_c2r(n, batch, 1, 2 * nc)
        buf = to_dev(O.pad_real(x, rdtype(prec)))
        h.exec_r2c(buf)
        h.sync()
        X = to_host(buf).view(cdtype(prec)).reshape(batch, nc)
        assert O.rel_l2(X, np.stack([O.r2c_nd(r) for r in x.astype(np.float64)])) < tol(prec)
        h.exec_c2r(buf)
        h.sync()
        back = to_host(buf).reshape(batch, 2 * nc)[:, :n]
        assert O.rel_l2(back / n, x) < tol(prec), (n, batch)


def test_grouped_split_precision_rows_keep_their_kernel():
    """A group's pass that launches alone runs its plan's own kernel: 512-point
    split-precision rows give the bits they give outside a group."""
    n, b = 512, 33
    x = O.normal_complex(n * b, 7).astype(np.complex64)
    outs = []
    for grouped in (False, True):
        h = nv.Handle(nv.F32, 1, flags=nv.FLAG_SPLIT_TC)
        h.plan_c2c(0, n, b, 1, n)
        assert h.plan_describe(nv.KIND_C2C, 0).startswith("split-tc")
        d = to_dev(x)
        if grouped:
            g = nv.Group([h])
            g.begin()
            h.exec_c2c(0, nv.FORWARD, d)
            g.end()
            g.sync()
        else:
            h.exec_c2c(0, nv.FORWARD, d)
            h.sync()
        outs.append(to_host(d))
    assert np.array_equal(outs[0], outs[1])
