"""Calls whose product kernel is launched as a programmatic dependent of the
split pass: back-to-back calls that reuse one workspace and rewrite their
inputs in between, the same calls captured in a CUDA graph and replayed, and
calls on several streams. Bar: bit-identical to isolated, synchronised calls.
"""
import pytest

pytestmark = pytest.mark.gpu

CASES = [("bf16x6", 300, 260, 700, None), ("bf16x6", 512, 64, 1024, {"tile": 24}),
         ("bf16x3_scaled", 300, 260, 700, None), ("bf16x3_scaled", 512, 64, 1024, {"tile": 25}),
         ("bf16x6_scaled", 256, 256, 20000, {"tile": 20, "split_k": 3}),
         ("bf16x6", 130, 120, 4096, {"tile": 12, "split_k": 4})]


def _inputs(m, n, k, count, scaled):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    out = []
    for _ in range(count):
        a = torch.rand((m, k), device="cuda", generator=g) * 2 - 1
        b = torch.rand((k, n), device="cuda", generator=g) * 2 - 1
        if scaled:
            a *= torch.exp2(torch.rand((m, 1), device="cuda", generator=g) * 40 - 20)
        out.append((a, b))
    return out


@pytest.mark.parametrize("variant,m,n,k,cfg", CASES)
def test_back_to_back_and_captured(variant, m, n, k, cfg):
    import torch

    import hb_hammerbench_b200 as hb
    ins = _inputs(m, n, k, 4, "scaled" in variant)
    want = []
    for a, b in ins:
        want.append(hb.gemm(a, b, variant=variant, config=cfg).clone())
        torch.cuda.synchronize()
    ws = torch.empty(hb.gemm_workspace_size(m, n, k, variant, cfg) + 256, dtype=torch.uint8,
                     device="cuda")
    a, b = torch.empty_like(ins[0][0]), torch.empty_like(ins[0][1])
    c = torch.empty((m, n), device="cuda")
    outs = [torch.empty((m, n), device="cuda") for _ in range(32)]
    for i in range(32):  # inputs and workspace rewritten right after each call
        a.copy_(ins[i % 4][0])
        b.copy_(ins[i % 4][1])
        hb.gemm(a, b, c, variant=variant, config=cfg, workspace=ws)
        outs[i].copy_(c)
    torch.cuda.synchronize()
    for i in range(32):
        assert torch.equal(outs[i], want[i % 4]), i

    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        hb.gemm(a, b, c, variant=variant, config=cfg, workspace=ws)
        hb.gemm(a, b, outs[0], variant=variant, config=cfg, workspace=ws)
    for i in range(8):
        a.copy_(ins[i % 4][0])
        b.copy_(ins[i % 4][1])
        c.zero_()
        outs[0].zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(c, want[i % 4]) and torch.equal(outs[0], want[i % 4]), i


def test_two_streams():
    import torch

    import hb_hammerbench_b200 as hb
    m, n, k, variant = 512, 320, 900, "bf16x6_scaled"
    ins = _inputs(m, n, k, 2, True)
    want = [hb.gemm(a, b, variant=variant) for a, b in ins]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    need = hb.gemm_workspace_size(m, n, k, variant) + 256
    ws = [torch.empty(need, dtype=torch.uint8, device="cuda") for _ in range(2)]
    outs = [[torch.empty((m, n), device="cuda") for _ in range(16)] for _ in range(2)]
    torch.cuda.synchronize()
    for i in range(16):
        for j in range(2):
            with torch.cuda.stream(streams[j]):
                hb.gemm(*ins[j], outs[j][i], variant=variant, workspace=ws[j])
    torch.cuda.synchronize()
    for j in range(2):
        for o in outs[j]:
            assert torch.equal(o, want[j])
