"""The per-stream workspace of both bindings against captured CUDA graphs, which keep its address."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _binding(name):
    import ascend_kernel_b200 as ak
    from ascend_kernel_b200 import cinfer_ascendc

    return ak if name == "mirror" else cinfer_ascendc


@pytest.mark.parametrize("name", ["mirror", "drop-in"])
def test_graph_replays_after_the_workspace_grew(name):
    """A GEMM is captured, then GEMVs on the same stream need more workspace (the split one 4.9 MB; the fp4 one of 640 rows
    14 MB with its f16 rows): replays still give the eager bits, leave tensors allocated since alone, and report what they find."""
    m = _binding(name)
    gen = torch.Generator().manual_seed(29)
    G, K, N = 4, 192, 512
    counts = torch.tensor([40, 0, 33, 7], dtype=torch.int64)
    M = int(counts.sum())
    x = torch.randn(M, K, generator=gen).to(torch.bfloat16).cuda()
    w = torch.randint(-128, 128, (G, K, N), generator=gen, dtype=torch.int8).cuda()
    scale = (torch.rand(G, N, generator=gen) * 0.009 + 0.001).to(torch.bfloat16).cuda()
    offset = (torch.rand(G, N, generator=gen) * 8 - 4).to(torch.bfloat16).cuda()
    gl = counts.cuda()
    rows, Kv = 640, 7168
    xv = torch.randn(rows, Kv, generator=gen).to(torch.bfloat16).cuda()
    wv = torch.randint(0, 256, (1, Kv, 128), generator=gen, dtype=torch.uint8).cuda()
    sv = torch.full((1, Kv // 16, 256), 0.5, dtype=torch.bfloat16, device="cuda")
    glv = torch.tensor([rows], device="cuda")
    yv = torch.empty(rows, 256, dtype=torch.bfloat16, device="cuda")
    ys = torch.empty(1, 256, dtype=torch.bfloat16, device="cuda")
    out = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    want = torch.zeros_like(out)
    torch.cuda.synchronize()

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        m.grouped_gemm(x, w, scale, offset, gl, "int8", want, group_list_type=1)  # the stream's workspace exists now
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        m.grouped_gemm(x, w, scale, offset, gl, "int8", out, group_list_type=1)
    with torch.cuda.stream(side):
        m.grouped_soft_gemv(xv[:1], wv[:, :, :128], sv, torch.ones(1, dtype=torch.int64, device="cuda"), "fp4", ys,
                            group_list_type=1, weight_layout="canonical")
        m.grouped_soft_gemv(xv, wv, sv, glv, "fp4", yv, group_list_type=1, weight_layout="canonical")
        fillers = [torch.full((n,), 0x5A, dtype=torch.uint8, device="cuda") for n in [1 << 20] * 8 + [5 << 20] * 2 + [8 << 20] * 2]
    torch.cuda.synchronize()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert all(bool((f == 0x5A).all()) for f in fillers)
    assert tuple(m.last_status()) == (0, 0)
    gl[2] = 1 << 20                       # a replay's finding reaches the status calls
    graph.replay()
    torch.cuda.synchronize()
    assert tuple(m.last_status(clear=True)) == (1, 2)
    assert tuple(m.last_status()) == (0, 0)
