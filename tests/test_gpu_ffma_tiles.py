"""FFMA tile loads at the sizes where they can go wrong: partial k tiles, edge
rows and columns, every pairing of operand layouts, aligned and unaligned
rows, tiles picked by the library and by id. Bar: bit-exact against the
device kernel's own arithmetic (one fmaf per k, ascending, oracle
host_mm_fma), and nothing written outside the m x n result.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _strided(x, pad):
    """x on the device with `pad` NaN columns after each row."""
    import torch
    buf = torch.full((x.shape[0], x.shape[1] + pad), float("nan"), device="cuda")
    buf[:, :x.shape[1]] = torch.from_numpy(x).cuda()
    return buf[:, :x.shape[1]]


@pytest.mark.parametrize("trans", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("tile", [0, 1, 3])
@pytest.mark.parametrize("m,n,k,pad", [
    (64, 64, 16, 0), (128, 128, 64, 0),      # whole tiles
    (65, 127, 15, 0), (129, 63, 17, 4),      # one past / one short of a tile, ragged k
    (100, 68, 100, 4), (36, 260, 36, 0),     # aligned rows, partial k tile
    (31, 33, 97, 1), (130, 66, 113, 3),      # unaligned rows
    (1, 4, 4, 0), (4, 1, 1, 0), (3, 2, 161, 2),
])
def test_layouts_and_edges_bit_exact(oracle_mod, m, n, k, pad, tile, trans):
    import torch

    import hb_hammerbench_b200 as hb
    ta, tb = trans
    A, B = oracle_mod.uniform_inputs((m, k), (k, n), seed=m * 7 + n * 3 + k)
    a = _strided(np.ascontiguousarray(A.T if ta else A), pad)
    b = _strided(np.ascontiguousarray(B.T if tb else B), pad)
    out = torch.full((m + 2, n + 5), -7.0, device="cuda")
    hb.gemm(a, b, out[:m, :n], trans_a=ta, trans_b=tb, config={"tile": tile} if tile else None)
    out = out.cpu().numpy()
    assert np.array_equal(out[:m, :n], oracle_mod.host_mm_fma(A, B))
    assert (out[m:] == -7.0).all() and (out[:, n:] == -7.0).all()


@pytest.mark.parametrize("tile", range(1, 10))
@pytest.mark.parametrize("k", [16, 47, 96, 131])
def test_every_tile_partial_k_bit_exact(oracle_mod, tile, k):
    import torch

    import hb_hammerbench_b200 as hb
    A, B = oracle_mod.uniform_inputs((259, k), (k, 262), seed=k)
    out = hb.gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(),
                  config={"tile": tile}).cpu().numpy()
    assert np.array_equal(out, oracle_mod.host_mm_fma(A, B))
