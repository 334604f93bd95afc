"""NaN and infinity stay in their own transform: kernels whose spare lanes repeat
others' points, or whose idle butterflies compute along, write none of it to a
neighbour."""
import numpy as np
import pytest

from helpers import cdtype, rdtype, to_dev, to_host
from oracle import oracle as O
from parafaft_b200 import native as nv

pytestmark = pytest.mark.gpu


def _run(prec, kind, n, data, batch):
    h = nv.Handle(prec, 1)
    d = to_dev(data)
    if kind in ("row", "col"):
        h.plan_c2c(0, n, batch, *((1, n) if kind == "row" else (batch, 1)))
        h.exec_c2c(0, nv.FORWARD, d)
    elif kind == "r2c":
        h.plan_r2c(n, batch, 1, 2 * (n // 2 + 1))
        h.exec_r2c(d)
    else:
        h.plan_c2r(n, batch, 1, 2 * (n // 2 + 1))
        h.exec_c2r(d)
    h.sync()
    return to_host(d)


@pytest.mark.parametrize("prec", [nv.F32, nv.F64])
@pytest.mark.parametrize("n", [8, 12, 30, 45, 60, 105, 210, 300, 500, 1225, 2016])
@pytest.mark.parametrize("kind", ["row", "col", "r2c", "c2r"])
def test_other_transforms_keep_their_bits(prec, n, kind):
    batch = 37
    if kind in ("row", "col"):
        shape = (batch, n) if kind == "row" else (n, batch)
        x = O.normal_complex(n * batch, n).astype(cdtype(prec)).reshape(shape)
    else:
        x = O.normal_real((batch, 2 * (n // 2 + 1)), n).astype(rdtype(prec))
    want = _run(prec, kind, n, x, batch)
    bad = x.copy()
    for b, v in ((0, np.nan), (17, np.inf), (36, -np.inf)):
        if kind == "col":
            bad[n // 2, b] = v
        else:
            bad[b, n // 2] = v
    got = _run(prec, kind, n, bad, batch)
    keep = [b for b in range(batch) if b not in (0, 17, 36)]
    own = (lambda a: a[:, keep]) if kind == "col" else (lambda a: a[keep])
    assert np.array_equal(own(got), own(want))
    assert not np.isfinite(got[:, 0] if kind == "col" else got[0]).any() or kind in ("r2c", "c2r")
