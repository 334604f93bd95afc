"""Which power-of-two rows take a compiled plan: each kind by its own measurements
(FP32 R2C rows of 2 x 1024 and 2 x 2048 points are faster on their row tile)."""
import pytest

from parafaft_b200 import native as nv


def _compiled(prec, kind, n):
    dist = n if kind == nv.KIND_C2C else 2 * (n // 2 + 1)
    return "compiled=" in nv.describe(prec, kind, n, 100, 1, dist)


@pytest.mark.parametrize("prec,kind,lengths", [
    (nv.F32, nv.KIND_C2C, {8, 16, 32, 64, 128, 256, 512, 2048, 4096}),
    (nv.F64, nv.KIND_C2C, {8, 16, 128, 256, 2048}),
    (nv.F32, nv.KIND_R2C, {16, 32, 64, 128, 256, 1024}),
    (nv.F32, nv.KIND_C2R, {16, 32, 64, 128, 256, 1024, 2048, 4096}),
    (nv.F64, nv.KIND_R2C, {16, 32, 64, 128, 256, 512, 2048, 4096}),
    (nv.F64, nv.KIND_C2R, {16, 32, 64, 128, 256, 512, 2048, 4096})])
def test_rows_on_compiled_plans(prec, kind, lengths):
    assert {n for n in (1 << k for k in range(2, 13)) if _compiled(prec, kind, n)} == lengths
