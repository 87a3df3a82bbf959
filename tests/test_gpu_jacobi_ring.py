"""Jacobi step on grids around the ring form's tiles (128 z, 8 x, slabs of 12
y) and around the rule that picks it (17 planes, three-quarter-filled z tiles,
output alignment). Bar: bit-exact against the oracle's host_jacobi, nothing written
outside the grid.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [
    (8, 24, 128), (8, 17, 128), (8, 16, 128),    # whole tiles; each side of the rule
    (1, 25, 132), (9, 36, 124), (7, 13, 260),    # edge tiles in every direction
    (17, 37, 96), (3, 40, 92), (10, 18, 516),    # three-quarter-filled z tiles, one quad short
    (5, 100, 4), (2, 19, 254), (40, 12, 1280),   # narrow z, unaligned rows, many CTAs
])
@pytest.mark.parametrize("offset", [0, 4, 1])
def test_grids_bit_exact(oracle_mod, nx, ny, nz, offset):
    import torch

    import hb_hammerbench_b200 as hb
    n = nx * ny * nz
    rng = np.random.Generator(np.random.PCG64(n + offset))
    a = (rng.uniform(-1, 1, n) * np.exp2(rng.uniform(-30, 30, n))).astype(np.float32)
    src = torch.zeros(n + 8, device="cuda")
    src[:] = 99.0  # never read: neighbours outside the grid count as 0
    src[offset:offset + n] = torch.from_numpy(a).cuda()
    dst = torch.full((n + 8,), -7.0, device="cuda")
    hb.jacobi(src[offset:offset + n], nx, ny, nz, 3, 5, out=dst[offset:offset + n])
    out = dst.cpu().numpy()
    assert np.array_equal(out[offset:offset + n], oracle_mod.host_jacobi(a, nx, ny, nz, 3, 5))
    assert (out[:offset] == -7.0).all() and (out[offset + n:] == -7.0).all()
