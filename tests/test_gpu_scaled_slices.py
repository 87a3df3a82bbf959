"""Scaled forms sliced along K where one slice's product leaves the FP32 range
and the whole sum does not: slices beyond the largest float that cancel, and
slices among the subnormals. Integers times powers of two whose second half of
K cancels the first but for its last columns, so every sum of normalised values
is exact and the only rounding is the final one. Bar: equal to the FP64 product
rounded to FP32, as an unsliced tile gives it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 2^(ea + eb) in the product: a slice of 128 k sums to about 2^9 of it and the
# whole to under 2^6
EXPONENTS = [(61, 61), (-75, -76), (3, -5)]


def _inputs(m, n, k, ea, eb, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    half = k // 2
    A = np.zeros((m, k))
    B = np.zeros((k, n))
    A[:, :half] = A[:, half:2 * half] = rng.integers(1, 4, (m, half))
    B[:half] = rng.integers(1, 4, (half, n))
    B[half:2 * half] = -B[:half]
    B[2 * half - 3:2 * half] += rng.integers(-2, 3, (3, n))
    return A * 2.0 ** ea, B * 2.0 ** eb


def _want(A, B):
    # the halves cancel exactly: only the last three k differ
    import torch
    p = torch.from_numpy(A).cuda() @ torch.from_numpy(B).cuda()
    return p.cpu().numpy().astype(np.float32)


@pytest.mark.parametrize("variant,tile", [
    ("bf16x6_scaled", t) for t in (10, 11, 12, 16, 18, 20, 22, 24, 26)] + [
    ("bf16x3_scaled", t) for t in (13, 14, 15, 17, 19, 21, 23, 25, 27)])
@pytest.mark.parametrize("ea,eb", EXPONENTS)
@pytest.mark.parametrize("n,splits", [(140, 2), (137, 8)])
def test_whole_grid_in_slices(variant, tile, ea, eb, n, splits):
    import torch

    import hb_hammerbench_b200 as hb
    m, k = 130, 1024
    A, B = _inputs(m, n, k, ea, eb, tile + n)
    a = torch.from_numpy(A.astype(np.float32)).cuda()
    b = torch.zeros((k, 140), device="cuda")
    b[:, :n] = torch.from_numpy(B.astype(np.float32)).cuda()
    out = hb.gemm(a, b[:, :n], variant=variant, config={"tile": tile, "split_k": splits})
    assert np.array_equal(out.cpu().numpy(), _want(A, B))


@pytest.mark.parametrize("variant", ["bf16x3_scaled", "bf16x6_scaled"])
@pytest.mark.parametrize("ea,eb", EXPONENTS)
@pytest.mark.parametrize("m,n,k", [(2100, 2500, 3000), (1537, 3333, 4096)])
def test_last_round_in_slices(variant, ea, eb, m, n, k):
    import torch

    import hb_hammerbench_b200 as hb
    from hb_hammerbench_b200 import _lib
    L, v = _lib.lib(), _lib.VARIANTS[variant]
    # partials of a part of the output: the last round alone is sliced
    extra = (L.hbsg_gemm_workspace_size_ex(0, 1, m, n, k, v, None)
             - hb.split_layout(m, n, k, variant)["total_bytes"])
    assert 0 < extra < 8 * m * n
    A, B = _inputs(m, n, k, ea, eb, m)
    a = torch.from_numpy(A.astype(np.float32)).cuda()
    b = torch.from_numpy(np.ascontiguousarray(B.T).astype(np.float32)).cuda()
    out = hb.gemm(a, b, variant=variant, trans_b=True)
    assert np.array_equal(out.cpu().numpy(), _want(A, B))
