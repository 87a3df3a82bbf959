"""Scaled forms whose combined row and column scale 2^s is no normal float
(results among the subnormals, or at the top of the range): the epilogue's
wide path, beside blocks that take the common one. Small integers times
powers of two, so every product and sum is exact and the only rounding is the
final one. Bar: equal to the FP64 product rounded to FP32 (infinities where it
overflows).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,tile", [
    ("bf16x6_scaled", t) for t in (10, 11, 12, 16, 18, 20, 22, 24, 26)] + [
    ("bf16x3_scaled", t) for t in (13, 14, 15, 17, 19, 21, 23, 25, 27)])
@pytest.mark.parametrize("ea,eb", [(-100, -45), (75, 48), (-20, 30), (-126, -15)])
def test_scale_beyond_normal_floats(variant, tile, ea, eb):
    import torch

    import hb_hammerbench_b200 as hb
    m, n, k = 130, 140, 16
    rng = np.random.Generator(np.random.PCG64(tile))
    A = rng.integers(0, 7, (m, k)) * 2.0 ** ea
    B = rng.integers(0, 3, (k, n)) * 2.0 ** eb
    A[64:96] *= 2.0 ** -ea  # one block of rows with ordinary scales
    with np.errstate(over="ignore"):
        want = (A @ B).astype(np.float32)
    a = torch.from_numpy(A.astype(np.float32)).cuda()
    b = torch.from_numpy(B.astype(np.float32)).cuda()
    out = hb.gemm(a, b, variant=variant, config={"tile": tile}).cpu().numpy()
    assert np.array_equal(out, want)
