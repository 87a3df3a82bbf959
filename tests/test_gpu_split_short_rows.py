"""Scaled split pass on many short rows (4096 and more, K up to 2048): K around
the sizes where a row takes 4 to 64 lanes and one to four units a lane, just
outside both limits, ragged row counts, aligned and unaligned row starts, zero,
subnormal and non-finite rows.
Bar: parts and maxima bit-exact against the oracle's split. A tall operand of
short rows may cost the scaled forms no more than twice the unscaled call on the
same split-pass tile: they read each operand at most once more, and the unscaled
pass already reads it and writes as many bytes of parts.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(4097, 3, k) for k in (
    1, 31, 32, 33, 64, 65, 128, 129, 256, 257, 500, 512, 513, 1000, 1024, 1025, 1500, 2047, 2048)] + [
    (3, 4099, 300), (4100, 4096, 40), (4098, 4097, 1100),  # the other operand, both
    (4095, 3, 100), (4097, 3, 2049)]  # the CTA-per-row form


def _operand(rng, rows, k):
    X = (rng.uniform(-1, 1, (rows, k)) * np.exp2(rng.uniform(-20, 20, (rows, k)))).astype(np.float32)
    X[0] *= np.float32(2.0 ** -126)
    if rows > 2:
        X[1] = 0.0
        X[2, 0], X[2, -1] = np.inf, np.nan  # ignored by the maximum
        X[-1] = np.sign(X[-1]) * np.float32(3.0e38)
    return X


def _padded(X, pad):
    import torch
    buf = torch.full((X.shape[0], X.shape[1] + pad), 1e30, device="cuda")
    buf[:, :X.shape[1]] = torch.from_numpy(X).cuda()
    return buf[:, :X.shape[1]]


@pytest.mark.parametrize("variant", ["bf16x3_scaled", "bf16x6_scaled"])
@pytest.mark.parametrize("pad", [0, 3, 4])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_parts_and_maxima_bit_exact(oracle_mod, variant, m, n, k, pad):
    import torch

    import hb_hammerbench_b200 as hb
    rng = np.random.Generator(np.random.PCG64(m + 10 * n + k))
    A, Bt = _operand(rng, m, k), _operand(rng, n, k)
    lay = hb.split_layout(m, n, k, variant)
    ws = torch.full((lay["total_bytes"],), 255, dtype=torch.uint8, device="cuda")
    hb.gemm(_padded(A, pad), _padded(Bt, pad), variant=variant, trans_b=True, workspace=ws,
            config={"tile": 10 if lay["parts"] == 3 else 13, "split_k": 1})
    w = ws.cpu().numpy()
    P, kp = lay["parts"], lay["kp"]
    for off, mx_off, X in ((lay["a_offset"], lay["rowmax_offset"], A),
                           (lay["b_offset"], lay["colmax_offset"], Bt)):
        rows = X.shape[0]
        parts = w[off:off + P * rows * kp * 2].view(np.uint16).reshape(P, rows, kp)
        for i in range(0, rows, 1 + rows // 100):
            if not np.isfinite(X[i]).all():
                continue
            want = oracle_mod.split_bf16(X[i], oracle_mod.pow2_exponent(X[i]), P)
            for p in range(P):
                assert np.array_equal(parts[p, i, :k], want[p]), (i, p)
        assert not parts[:, :, k:].any()
        mx = w[mx_off:mx_off + 4 * rows].view(np.float32)
        assert np.array_equal(mx, np.where(np.isfinite(X), np.abs(X), 0).max(axis=1))


@pytest.mark.parametrize("tile", [20, 24])  # fused tiles: A's maxima alone, at the workspace's start
@pytest.mark.parametrize("m,k", [(4097, 32), (4103, 96), (4099, 512), (4101, 1024), (4098, 1536), (4098, 1540), (65, 32)])
def test_maxima_alone(tile, m, k):
    import torch

    import hb_hammerbench_b200 as hb
    rng = np.random.Generator(np.random.PCG64(m + k))
    A = _operand(rng, m, k)
    b = torch.ones((k, 64), device="cuda")
    cfg = {"tile": tile, "split_k": 1}
    ws = torch.full((hb.gemm_workspace_size(m, 64, k, "bf16x6_scaled", cfg),), 255,
                    dtype=torch.uint8, device="cuda")
    hb.gemm(torch.from_numpy(A).cuda(), b, variant="bf16x6_scaled", config=cfg, workspace=ws)
    mx = ws[:4 * m].cpu().numpy().view(np.float32)
    assert np.array_equal(mx, np.where(np.isfinite(A), np.abs(A), 0).max(axis=1))


@pytest.mark.parametrize("products", ["bf16x3", "bf16x6"])
@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("k", [32, 128])
def test_tall_operand_of_short_rows_keeps_its_speed(products, trans_b, k):
    import torch

    import hb_hammerbench_b200 as hb
    m, n = 65536, 64
    a = torch.rand((m, k), device="cuda") * 2 - 1
    b = torch.rand((n, k) if trans_b else (k, n), device="cuda") * 2 - 1
    c = torch.empty((m, n), device="cuda")

    cfg = {"tile": 12 if products == "bf16x6" else 15, "split_k": 1}  # 128 x 64, split pass

    def us(variant):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        times = []
        for _ in range(7):
            e0.record()
            for _ in range(20):
                hb.gemm(a, b, c, variant=variant, trans_b=trans_b, config=cfg)
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1) * 50.0)
        return sorted(times)[3]

    assert us(products + "_scaled") < 2.0 * us(products)
