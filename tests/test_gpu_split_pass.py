"""Split pass at the edges of its launch shapes: rows longer than one CTA's
chunk (maxima reduced in chunks), single rows and columns, both layouts of
both operands, exponents whose scale 2^-e is no normal float (rows with a
subnormal maximum, rows near the FP32 maximum), zero and non-finite rows.
Bar: parts and maxima bit-exact against the oracle's split.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["bf16x3_scaled", "bf16x6_scaled", "bf16x6"])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(3, 2, 16384), (2, 3, 16385), (5, 1, 33000), (1, 65, 7),
                                   (130, 257, 65)])
def test_parts_and_maxima_bit_exact(oracle_mod, variant, ta, tb, m, n, k):
    import torch

    import hb_hammerbench_b200 as hb
    rng = np.random.Generator(np.random.PCG64(m + 10 * n + k))
    A = (rng.uniform(-1, 1, (m, k)) * np.exp2(rng.uniform(-20, 20, (m, k)))).astype(np.float32)
    B = (rng.uniform(-1, 1, (k, n)) * np.exp2(rng.uniform(-20, 20, (k, n)))).astype(np.float32)
    scaled = "scaled" in variant
    if scaled:  # one row / column each at the ends of the exponent range, one of zeros
        A[0] *= np.float32(2.0 ** -126)
        B[:, 0] = np.sign(B[:, 0]) * np.float32(3.0e38)
        if m > 2:
            A[1] = 0.0
            A[2, 0], A[2, -1] = np.inf, np.nan  # ignored by the maximum
    lay = hb.split_layout(m, n, k, variant)
    ws = torch.full((lay["total_bytes"],), 255, dtype=torch.uint8, device="cuda")
    a = torch.from_numpy(np.array(A.T, order="C", copy=True) if ta else A).cuda()
    b = torch.from_numpy(np.array(B.T, order="C", copy=True) if tb else B).cuda()
    hb.gemm(a, b, variant=variant, trans_a=bool(ta), trans_b=bool(tb), workspace=ws,
            config={"tile": 10 if lay["parts"] == 3 else 13, "split_k": 1})
    w = ws.cpu().numpy()
    P, kp = lay["parts"], lay["kp"]
    for off, mx_off, X in ((lay["a_offset"], lay["rowmax_offset"], A),
                           (lay["b_offset"], lay["colmax_offset"], np.ascontiguousarray(B.T))):
        rows = X.shape[0]
        parts = w[off:off + P * rows * kp * 2].view(np.uint16).reshape(P, rows, kp)
        for i in range(rows):
            if not np.isfinite(X[i]).all():
                continue
            want = oracle_mod.split_bf16(X[i], oracle_mod.pow2_exponent(X[i]) if scaled else 0, P)
            for p in range(P):
                assert np.array_equal(parts[p, i, :k], want[p]), (i, p)
        assert not parts[:, :, k:].any()
        if scaled:
            mx = w[mx_off:mx_off + 4 * rows].view(np.float32)
            finite = np.where(np.isfinite(X), np.abs(X), 0)
            assert np.array_equal(mx, finite.max(axis=1))
