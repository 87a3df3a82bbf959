"""Jacobi grids of at most 16 planes on each side of the second way into the
ring form, a CTA (128 z x 8 x x 12 y) for every SM: one plane, a few, two slabs.
Bar: bit-exact against the oracle's host_jacobi, nothing written outside the
grid.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [
    (1176, 1, 128), (1184, 1, 128), (1177, 1, 128), (1200, 2, 124),  # 147, 148, 148, 150 CTAs
    (128, 12, 1280), (113, 12, 1280), (112, 12, 1280),               # 160, 150, 140
    (592, 13, 128), (588, 16, 100), (75, 5, 2000),                   # 148, 148, 160
])
@pytest.mark.parametrize("offset", [0, 1])
def test_grids_bit_exact(oracle_mod, nx, ny, nz, offset):
    import torch

    import hb_hammerbench_b200 as hb
    n = nx * ny * nz
    rng = np.random.Generator(np.random.PCG64(n + offset))
    a = (rng.uniform(-1, 1, n) * np.exp2(rng.uniform(-30, 30, n))).astype(np.float32)
    src = torch.full((n + 8,), 99.0, device="cuda")  # neighbours outside the grid count as 0
    src[offset:offset + n] = torch.from_numpy(a).cuda()
    dst = torch.full((n + 8,), -7.0, device="cuda")
    hb.jacobi(src[offset:offset + n], nx, ny, nz, 3, 5, out=dst[offset:offset + n])
    out = dst.cpu().numpy()
    assert np.array_equal(out[offset:offset + n], oracle_mod.host_jacobi(a, nx, ny, nz, 3, 5))
    assert (out[:offset] == -7.0).all() and (out[offset + n:] == -7.0).all()
