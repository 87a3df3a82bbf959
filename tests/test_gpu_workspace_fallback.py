"""A call without a config in a buffer smaller than the automatic schedule's, down
to the compact schedule's: run within the buffer, right within the FP64 error
bound, and refused one step below it; the allocation-free entry point takes
exactly the products one of the two sizes of which fits its scratch.
"""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1248, 64, 4064), (224, 160, 3136), (64, 64, 65536), (100, 90, 4099), (33, 257, 2048),
          (2100, 2500, 3000), (512, 512, 512), (64, 64, 30000), (1100, 1100, 1152)]


@pytest.mark.parametrize("variant", ["bf16x3", "bf16x6", "bf16x3_scaled", "bf16x6_scaled"])
@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("trans", [False, True])
def test_down_to_the_compact_schedule(variant, m, n, k, trans):
    import torch

    from hb_hammerbench_b200 import _lib
    L, v = _lib.lib(), _lib.VARIANTS[variant]
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.rand((m, k), device="cuda", generator=g) * 2 - 1
    B = torch.rand((k, n), device="cuda", generator=g) * 2 - 1
    a = A.t().contiguous() if trans else A
    args = (int(trans), 0, m, n, k, a.data_ptr(), a.stride(0), B.data_ptr(), n)
    stream = torch.cuda.current_stream().cuda_stream
    need = L.hbsg_gemm_workspace_size_for(*args, v, None)
    ws = torch.full((need + 256,), 7, dtype=torch.uint8, device="cuda")

    def call(size):
        C = torch.full((m, n), float("nan"), device="cuda")
        st = L.hbsg_gemm_ex(*args, C.data_ptr(), n, v, None, ws.data_ptr(), size, stream)
        return st, C

    lo, hi = -1, (need + 255) // 256  # least accepted size, in steps of 256 bytes
    while hi - lo > 1:
        mid = (lo + hi) // 2
        st, _ = call(256 * mid)
        assert st in (_lib.OK, _lib.ERR_WORKSPACE)
        lo, hi = (mid, hi) if st == _lib.ERR_WORKSPACE else (lo, mid)
    least = 256 * hi
    if (m, n, k, variant, trans) == (1248, 64, 4064, "bf16x3", False):
        assert least == 2 * 64 * 4064 * 2 < need // 4  # B's parts alone
    ref = A.double() @ B.double()
    torch.cuda.synchronize()
    ws.fill_(7)
    st, C = call(least)
    assert st == _lib.OK
    assert (ws[least:] == 7).all()
    rel = (torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref)).item()
    assert rel < (2.0 ** -16 if "x3" in variant else 2e-6)
    if least:
        st, C = call(least - 256)
        assert st == _lib.ERR_WORKSPACE and bool(C.isnan().all())

    C = torch.full((m, n), float("nan"), device="cuda")
    fits = min(least, need) <= _lib.NOALLOC_SCRATCH_BYTES
    assert L.hbsg_gemm_noalloc(*args, C.data_ptr(), n, v, stream) == (
        _lib.OK if fits else _lib.ERR_WORKSPACE)
    assert bool(C.isnan().any()) == (not fits)
