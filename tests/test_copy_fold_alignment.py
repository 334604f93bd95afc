"""A held copy folds into the pass behind it only where its source is aligned to
what the pass loads at once: a legal source aligned to one real is copied first."""
import numpy as np
import pytest

from helpers import cdtype, rdtype, to_dev, to_host, tol
from oracle import oracle as O
from parafaft_b200 import native as nv

PRECS = [nv.F32, nv.F64]
BASE_SRC, BASE_DST = 1 << 20, 1 << 24  # record-only handles touch no memory


def _plan(h, kind, n, batch):
    """Plans the pass and returns (exec call, bytes of its region)."""
    es = 8 if h.precision == nv.F64 else 4
    if kind == "c2c":
        h.plan_c2c(0, n, batch, 1, n)
        return lambda p: h.exec_c2c(0, nv.FORWARD, p), 2 * es * n * batch
    pitch = 2 * (n // 2 + 1)
    if kind == "r2c":
        h.plan_r2c(n, batch, 1, pitch)
        return h.exec_r2c, es * pitch * batch
    h.plan_c2r(n, batch, 1, pitch)
    return h.exec_c2r, es * pitch * batch


def _handle(prec, flags=0, plan_flag=0):
    h = nv.Handle(prec, 1, flags=flags, plan_flag=plan_flag)
    h.precision = prec
    return h


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("kind,n,folds", [
    ("r2c", 100, False), ("r2c", 128, False), ("r2c", 120, False), ("r2c", 34, True),
    ("r2c", 75, True), ("r2c", 63, True), ("c2r", 100, False), ("c2r", 75, False),
    ("c2c", 100, False), ("c2c", 128, False), ("c2c", 17, False)])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_fold_needs_the_load_alignment(prec, kind, n, folds, offset):
    """`folds`: whether the pass loads single reals (34 = 2 x 17 points run the
    runtime-generic kernel). An offset of two reals is whole complex points."""
    es = 8 if prec == nv.F64 else 4
    h = _handle(prec, nv.FLAG_RECORD_ONLY)
    run, nbytes = _plan(h, kind, n, 3)
    h.memcpy(BASE_DST, BASE_SRC + offset * es, nbytes)
    run(BASE_DST)
    h.flush()
    st = h.stats()
    want = 1 if folds or offset != 1 else 0
    assert (st["fused_copies"], st["copies_issued"]) == (want, 1 - want), st


def test_generic_only_r2c_rows_fold_single_reals():
    h = _handle(nv.F32, nv.FLAG_RECORD_ONLY | nv.FLAG_GENERIC_ONLY)
    run, nbytes = _plan(h, "r2c", 100, 3)
    h.memcpy(BASE_DST, BASE_SRC + 4, nbytes)
    run(BASE_DST)
    h.flush()
    assert h.stats()["fused_copies"] == 1


def test_group_copies_a_misaligned_source(monkeypatch):
    """A group chooses the kernel of a recorded pass again: the copy stays an
    operation of its own."""
    monkeypatch.setenv("B200FFT_RECORD_ONLY", "1")
    hs = [_handle(nv.F32, nv.FLAG_RECORD_ONLY) for _ in range(2)]
    runs = [_plan(h, "r2c", 100, 3) for h in hs]
    g = nv.Group(hs)
    g.begin()
    for i, (h, (run, nbytes)) in enumerate(zip(hs, runs)):
        dst = BASE_DST + i * (1 << 16)
        h.memcpy(dst, BASE_SRC + i * (1 << 16) + 4 * i, nbytes)
        run(dst)
    g.end()
    assert g.stats()["copies_issued"] == 1
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("n", [100, 120, 128, 75, 34])
@pytest.mark.parametrize("offset", [0, 1])
def test_misaligned_sources_give_the_oracle_values(prec, n, offset):
    batch, nc = 21, n // 2 + 1
    x = O.normal_real((batch, n), n).astype(rdtype(prec))
    buf = np.zeros(offset + batch * 2 * nc, rdtype(prec))
    buf[offset:] = O.pad_real(x, rdtype(prec)).reshape(-1)
    src, dst = to_dev(buf), to_dev(np.zeros(batch * 2 * nc, rdtype(prec)))
    h = _handle(prec)
    run, nbytes = _plan(h, "r2c", n, batch)
    h.memcpy(dst, src.data_ptr() + offset * x.itemsize, nbytes)
    run(dst)
    h.sync()
    X = to_host(dst).view(cdtype(prec)).reshape(batch, nc)
    ref = np.stack([O.r2c_nd(r) for r in x.astype(np.float64)])
    assert O.rel_l2(X, ref) < tol(prec)
    z = O.normal_complex(n * batch, n).astype(cdtype(prec))
    buf = np.concatenate([np.zeros(offset, rdtype(prec)), z.view(rdtype(prec))])
    src, dst = to_dev(buf), to_dev(np.zeros_like(z))
    run, nbytes = _plan(h, "c2c", n, batch)
    h.memcpy(dst, src.data_ptr() + offset * x.itemsize, nbytes)
    run(dst)
    h.sync()
    ref = O.c2c_batch(z.astype(np.complex128), n, batch, 1, n, -1)
    assert O.rel_l2(to_host(dst), ref) < tol(prec)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("n,offset,extra,folds", [
    (100, 0, 0, True), (100, 1, 0, True), (100, 0, 1, True), (100, 0, 2, True),
    (350, 1, 1, True), (75, 1, 1, True), (120, 0, 1, False), (128, 1, 0, False),
    (128, 0, 2, True)])
def test_pads_fold_real_aligned_sources(prec, n, offset, extra, folds):
    """A pad whose source is aligned to or pitched by single reals folds into the
    R2C pass of every length without a specialised kernel."""
    es, pitch = (8 if prec == nv.F64 else 4), 2 * (n // 2 + 1)
    h = _handle(prec, nv.FLAG_RECORD_ONLY)
    run, _ = _plan(h, "r2c", n, 5)
    h.memcpy2d(BASE_DST, pitch * es, BASE_SRC + offset * es, (n + extra) * es, n * es, 5)
    run(BASE_DST)
    h.flush()
    st = h.stats()
    assert (st["fused_copies"], st["copies_issued"]) == (int(folds), int(not folds)), st


@pytest.mark.gpu
@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("n", [36, 100, 350, 1000, 75, 120])
@pytest.mark.parametrize("offset,extra", [(0, 0), (1, 0), (0, 1), (1, 3)])
def test_pads_give_the_oracle_values(prec, n, offset, extra):
    batch, nc = 21, n // 2 + 1
    rows = O.normal_real((batch, n + extra), n).astype(rdtype(prec))
    src = to_dev(np.concatenate([np.zeros(offset, rdtype(prec)), rows.reshape(-1)]))
    dst = to_dev(np.zeros(batch * 2 * nc, rdtype(prec)))
    h = _handle(prec)
    run, _ = _plan(h, "r2c", n, batch)
    es = rows.itemsize
    for _ in range(2):  # the plan keeps its kernel for aligned rows
        h.memcpy2d(dst, 2 * nc * es, src.data_ptr() + offset * es, (n + extra) * es, n * es,
                   batch)
        run(dst)
        h.sync()
        X = to_host(dst).view(cdtype(prec)).reshape(batch, nc)
        ref = np.stack([O.r2c_nd(r) for r in rows[:, :n].astype(np.float64)])
        assert O.rel_l2(X, ref) < tol(prec)
