"""Allocation-free products whose automatic schedule fits the scratch and whose
compact one does not (it keeps parts of both operands where the automatic one
splits A inside a fused tile): taken, bit-identical to the workspace entry point
with as many bytes and within the FP64 error bound. The same sizes with A transposed, whose
parts alone exceed the scratch, are still refused before anything is launched.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,variant", [(448, 1928, 1856, "bf16x3"),
                                           (768, 432, 2368, "bf16x6_scaled"),
                                           (512, 1280, 5472, "bf16x6_scaled")])
def test_automatic_schedule_that_fits_is_taken(m, n, k, variant):
    import torch

    import hb_hammerbench_b200 as hb
    from hb_hammerbench_b200 import _lib
    L, v = _lib.lib(), _lib.VARIANTS[variant]
    g = torch.Generator(device="cuda").manual_seed(k)
    A = torch.rand((m, k), device="cuda", generator=g) * 2 - 1
    B = torch.rand((k, n), device="cuda", generator=g) * 2 - 1
    st = torch.cuda.current_stream().cuda_stream
    scratch = _lib.NOALLOC_SCRATCH_BYTES
    assert hb.split_layout(m, n, k, variant)["total_bytes"] > scratch
    assert L.hbsg_gemm_workspace_size_for(0, 0, m, n, k, A.data_ptr(), k, B.data_ptr(), n, v,
                                          None) <= scratch
    C = torch.full((m, n), float("nan"), device="cuda")
    assert L.hbsg_gemm_noalloc(0, 0, m, n, k, A.data_ptr(), k, B.data_ptr(), n, C.data_ptr(), n, v,
                               st) == _lib.OK
    ws = torch.empty(scratch, dtype=torch.uint8, device="cuda")
    D = torch.full((m, n), float("nan"), device="cuda")
    assert L.hbsg_gemm_ex(0, 0, m, n, k, A.data_ptr(), k, B.data_ptr(), n, D.data_ptr(), n, v,
                          None, ws.data_ptr(), scratch, st) == _lib.OK
    assert torch.equal(C, D)
    ref = A.double() @ B.double()
    rel = (torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref)).item()
    assert rel < (2.0 ** -16 if "x3" in variant else 2e-6)

    at = A.t().contiguous()
    C.fill_(7.0)
    assert L.hbsg_gemm_noalloc(1, 0, m, n, k, at.data_ptr(), m, B.data_ptr(), n, C.data_ptr(), n, v,
                               st) == _lib.ERR_WORKSPACE
    torch.cuda.synchronize()
    assert bool((C == 7.0).all())
