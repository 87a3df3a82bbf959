"""Split-BF16 grids whose last, unfilled round of tiles is sliced along K:
sizes just past one to four full rounds, ragged edges, columns and output rows
that rule out 16-byte stores, each operand order, in exactly the workspace the
size query reports. Small integers make every product and partial sum exact,
so the result has to equal the FP64 product whatever the slicing.
"""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(3001, 2503, 3607), (2100, 2500, 3000), (4100, 4200, 1027), (128 * 149, 250, 1024),
          (2304, 2176, 512), (2433, 4096, 2048), (1537, 3333, 4096), (3000, 1300, 700)]


def _inputs(m, n, k, trans_b):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n * 3 + k)
    A = torch.randint(-3, 4, (m, k), device="cuda", generator=g).float()
    B = torch.randint(-3, 4, (k, n), device="cuda", generator=g).float()
    return A, B, (B.t().contiguous() if trans_b else B)


@pytest.mark.parametrize("variant", ["bf16x3", "bf16x6", "bf16x3_scaled", "bf16x6_scaled"])
@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("trans_b,pad", [(False, 0), (True, 5)])
def test_exact_in_the_reported_workspace(variant, m, n, k, trans_b, pad):
    import torch

    from hb_hammerbench_b200 import _lib
    L, v = _lib.lib(), _lib.VARIANTS[variant]
    A, B, b = _inputs(m, n, k, trans_b)
    need = L.hbsg_gemm_workspace_size_for(0, int(trans_b), m, n, k, A.data_ptr(), k, b.data_ptr(),
                                          b.stride(0), v, None)
    ws = torch.full((need + 256,), 7, dtype=torch.uint8, device="cuda")
    C = torch.full((m, n + pad), -1.0, device="cuda")
    st = L.hbsg_gemm_ex(0, int(trans_b), m, n, k, A.data_ptr(), k, b.data_ptr(), b.stride(0),
                        C.data_ptr(), n + pad, v, None, ws.data_ptr(), need,
                        torch.cuda.current_stream().cuda_stream)
    assert st == _lib.OK
    torch.cuda.synchronize()
    assert torch.equal(C[:, :n].double(), A.double() @ B.double())
    assert (C[:, n:] == -1.0).all()
    assert (ws[need:] == 7).all()


def test_some_of_these_sizes_slice_their_last_round():
    # partials of a part of the output only: more than the operands' parts,
    # less than two slices of the whole output
    from hb_hammerbench_b200 import _lib
    import hb_hammerbench_b200 as hb
    L, v = _lib.lib(), _lib.VARIANTS["bf16x3_scaled"]
    taken = 0
    for m, n, k in SHAPES:
        extra = (L.hbsg_gemm_workspace_size_ex(0, 1, m, n, k, v, None)
                 - hb.split_layout(m, n, k, "bf16x3_scaled")["total_bytes"])
        taken += 0 < extra < 8 * m * n
    assert taken >= 2
