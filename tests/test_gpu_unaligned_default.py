"""Calls without a schedule whose shape class names a fused-split tile, on operands
that tile cannot read (K or N no multiple of 4, views that start off a 16-byte
boundary): run on the library's own choice, within the FP64 error bound; the
aligned call of the class still runs the table's schedule, bit for bit.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def table(tmp_path, monkeypatch):
    from hb_hammerbench_b200 import autotune
    monkeypatch.setenv("HBSG_AUTOTUNE_CACHE", str(tmp_path / "t.json"))
    monkeypatch.setenv("HBSG_AUTOTUNE", "1")
    autotune.clear_memory_cache()
    yield autotune
    autotune.clear_memory_cache()


def _rand(rows, cols, seed, offset=0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand(rows * cols + offset, device="cuda", generator=g) * 2 - 1)[offset:].view(
        rows, cols)


def _rel(C, A, B):
    import torch
    ref = A.double() @ B.double()
    return (torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref)).item()


def _fused(hb, cfg):
    return cfg is not None and next(t for t in hb.tiles() if t["tile"] == cfg["tile"])["fused"]


# m10:n10:k10, m16:n6:k12 and m8:n8:k20
@pytest.mark.parametrize("variant", ["bf16x3", "bf16x6"])
@pytest.mark.parametrize("m,n,k,offset", [(1000, 1000, 1001, 0), (1000, 999, 1000, 0),
                                          (1000, 1000, 1000, 1), (40000, 50, 4001, 0),
                                          (40000, 52, 4000, 2), (200, 131, 600001, 0)])
def test_unaligned_operands(table, variant, m, n, k, offset):
    import hb_hammerbench_b200 as hb
    assert _fused(hb, table.lookup(m, n, k, variant))
    A, B = _rand(m, k, 1, offset), _rand(k, n, 2)
    assert _rel(hb.gemm(A, B, variant=variant), A, B) < (2.0 ** -16 if variant == "bf16x3" else 2e-6)


@pytest.mark.parametrize("variant", ["bf16x3", "bf16x6"])
def test_aligned_operands_keep_the_table(table, variant):
    import torch

    import hb_hammerbench_b200 as hb
    m, n, k = 1000, 1000, 1000
    cfg = table.lookup(m, n, k, variant)
    A, B = _rand(m, k, 1), _rand(k, n, 2)
    C = hb.gemm(A, B, variant=variant)
    assert torch.equal(C, hb.gemm(A, B, variant=variant, config=cfg))
    # a schedule the caller names is not replaced
    with pytest.raises(hb.HbsgError):
        hb.gemm(_rand(m, 1001, 1), _rand(1001, n, 2), variant=variant, config=cfg)


@pytest.mark.parametrize("offset", [0, 1])
def test_grouped_plans(table, offset):
    import torch

    import hb_hammerbench_b200 as hb
    dims = [(130, 96, 64), (64, 200, 101), (300, 64, 33)] if offset else [(130, 96, 64),
                                                                          (64, 200, 100)]
    fused = next(t["tile"] for t in hb.tiles() if t["fused"] and t["parts"] == 3 and t["bm"] == 256)
    table._store(table.grouped_key(dims, "bf16x6"), {"config": {"tile": fused}, "ms": 1.0})
    As = [_rand(m, k, i) for i, (m, n, k) in enumerate(dims)]
    Bs = [_rand(k, n, 50 + i) for i, (m, n, k) in enumerate(dims)]
    plan = hb.GroupedPlan(As, Bs, variant="bf16x6")
    assert (plan.config is None) == bool(offset)
    Cs = plan.run()
    torch.cuda.synchronize()
    for a, b, c in zip(As, Bs, Cs):
        assert _rel(c, a, b) < 2e-6
