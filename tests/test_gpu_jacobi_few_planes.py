"""Jacobi grids on each side of the rules that pick the ring form: 3 and 4 planes
where the grid exceeds what L2 holds of it, 12, 13, 16 and 17 planes below that,
one and several z tiles, and CTAs (128 z x 8 x x 12 y) around whole rounds of the
SMs in either form.
Bar: bit-exact against the oracle's host_jacobi, nothing written outside the
grid.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [
    (1184, 1, 128), (1200, 2, 124), (150, 12, 512),     # one slab
    (150, 13, 512), (64, 13, 512), (64, 17, 260),       # second slab; under a CTA an SM
    (296, 13, 256), (295, 16, 228), (280, 16, 256),     # 148, 148 and 140 CTAs
    (592, 17, 128), (1184, 17, 124), (170, 170, 128),   # one z tile: 148, 296 and 330 CTAs,
    (150, 250, 128), (160, 280, 100),                   # 399 and 480 (vector form: 304 and 360)
    (148, 16, 4096), (1200, 18, 512),                   # several CTAs an SM
])
@pytest.mark.parametrize("offset", [0, 1])
def test_grids_bit_exact(oracle_mod, nx, ny, nz, offset):
    _check(oracle_mod, nx, ny, nz, offset)


# 11 000 000 points and one plane's row more
@pytest.mark.parametrize("nx,ny,nz", [(3520, 3, 1024), (3584, 3, 1024), (2688, 4, 1024),
                                      (21484, 4, 128), (21488, 4, 128), (300, 300, 124)])
def test_grids_around_the_l2_line(oracle_mod, nx, ny, nz):
    _check(oracle_mod, nx, ny, nz, 0)


def _check(oracle_mod, nx, ny, nz, offset):
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
