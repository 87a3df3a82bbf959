"""Automatic split-BF16 schedules over the range of shapes: the call without a
config runs in the workspace the size queries report, in the compact
schedule's smaller one, and is within the FP64 error bound either way; the
allocation-free entry point takes shapes whose K-slice partials do not fit
its scratch and still refuses those whose parts alone do not.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(224, 160, 3136), (64, 64, 65536), (480, 256, 1920), (100, 90, 4099), (33, 257, 2048),
          (130, 700, 257), (2000, 72, 1500), (512, 512, 512), (1, 1, 20000), (1280, 1000, 640)]


@pytest.mark.parametrize("variant", ["bf16x3", "bf16x6", "bf16x3_scaled", "bf16x6_scaled"])
@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("trans", [False, True])
def test_automatic_and_compact_schedules(variant, m, n, k, trans):
    import torch

    import hb_hammerbench_b200 as hb
    from hb_hammerbench_b200 import _lib
    L, v = _lib.lib(), _lib.VARIANTS[variant]
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.rand((m, k), device="cuda", generator=g) * 2 - 1
    B = torch.rand((k, n), device="cuda", generator=g) * 2 - 1
    a = A.t().contiguous() if trans else A
    ref = A.double() @ B.double()
    bound = 2.0 ** -16 if "x3" in variant else 2e-6

    def call(entry, *tail):
        C = torch.full((m, n), float("nan"), device="cuda")
        st = entry(int(trans), 0, m, n, k, a.data_ptr(), a.stride(0), B.data_ptr(), n,
                   C.data_ptr(), n, v, *tail, torch.cuda.current_stream().cuda_stream)
        if st == _lib.OK:
            torch.cuda.synchronize()
            rel = torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref)
            assert rel.item() < bound
        return st

    need = L.hbsg_gemm_workspace_size_for(int(trans), 0, m, n, k, a.data_ptr(), a.stride(0),
                                          B.data_ptr(), n, v, None)
    covers = L.hbsg_gemm_workspace_size_ex(int(trans), 0, m, n, k, v, None)
    assert need <= covers
    ws = torch.empty(max(need, 256) + 256, dtype=torch.uint8, device="cuda")
    ws[need:] = 7
    assert call(L.hbsg_gemm_ex, None, ws.data_ptr(), need) == _lib.OK
    assert (ws[need:] == 7).all()
    # a buffer of the operand parts alone holds the schedule without slices
    parts = hb.split_layout(m, n, k, variant)["total_bytes"]
    one = L.hbsg_gemm_workspace_size_ex(int(trans), 0, m, n, k, v,
                                        ctypes.pointer(_lib.Config(split_k=1)))
    small = torch.empty(max(parts, one, 256), dtype=torch.uint8, device="cuda")
    assert call(L.hbsg_gemm_ex, ctypes.pointer(_lib.Config(split_k=1)), small.data_ptr(),
                max(parts, one)) == _lib.OK
    st = call(L.hbsg_gemm_noalloc)
    assert st in (_lib.OK, _lib.ERR_WORKSPACE)
    if parts <= _lib.NOALLOC_SCRATCH_BYTES // 4:
        assert st == _lib.OK
