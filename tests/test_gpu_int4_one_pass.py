"""int4 GEMM in one pass (calls without offsets: x and the weights as scaled f16) against the oracle and the two-pass kernel: ragged
row counts, rows and scales that f16 does not hold; and calls with offsets, which take the two-pass kernel."""
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_gemm import SENTINEL, run_gemm
from tests.util import assert_close_to_golden

pytestmark = pytest.mark.gpu


def _case(counts, K, N, offsets, seed):
    gen = torch.Generator().manual_seed(seed)
    G, M = len(counts), sum(counts)
    x = torch.randn(M + 3, K, generator=gen).to(torch.bfloat16)  # three rows of no expert
    w = torch.randint(0, 256, (G, K, N // 2), generator=gen, dtype=torch.uint8).view(torch.int8)
    s = (torch.rand(G, K // 128, N, generator=gen) * 0.045 + 0.005).to(torch.bfloat16)
    o = (torch.rand(G, K // 128, N, generator=gen) * 4 - 2).to(torch.bfloat16) if offsets else None
    return x, w, s, o, torch.tensor(counts, dtype=torch.int64)


def _one_pass(x, K, N, G, offsets):
    from ascend_kernel_b200 import _abi

    return _abi.lib.b200moe_grouped_gemm_scratch_bytes(x.shape[0], K, N, G, _abi.CT["int4"], int(offsets)) > 0


@pytest.mark.parametrize("counts,K,N,offsets", [
    ([1, 0, 127, 128, 129, 300, 1200], 2176, 4096, False),
    ([1, 0, 127, 128, 129, 300, 1200], 2176, 4096, True),
    ([700, 1, 33, 1000], 2048, 4096, False),
    ([1] * 950 + [300, 129, 256, 64], 128, 1536, False),    # one scale group: two stages a tile
    ([2] * 200 + [900], 896, 1024, False),
    ([2] * 200 + [900], 896, 1024, True),
])
def test_matches_oracle(counts, K, N, offsets):
    x, w, s, o, cnt = _case(counts, K, N, offsets, 5)
    assert _one_pass(x, K, N, len(counts), offsets) == (not offsets)
    x[3] *= 2.0 ** 60      # rows of any magnitude keep their accuracy
    x[5] *= 2.0 ** -70
    x[7] = 0
    gold = O.golden_f32(x, w, s, o, cnt, "int4", O.GROUP_LIST_COUNTS)
    out, st = run_gemm(x, w, s, o, cnt, "int4", gl_type=1)
    assert st == (0, 0)
    unit = torch.ones(x.shape[0])
    unit[3], unit[5] = 2.0 ** -60, 2.0 ** 70
    assert_close_to_golden((out.cpu().float() * unit[:, None]).to(torch.bfloat16), gold * unit[:, None])
    assert (out[sum(counts):].float() == SENTINEL).all()


@pytest.mark.parametrize("kind", ["few_rows", "most_rows", "scales"])
def test_what_f16_does_not_hold_goes_through_the_two_pass_kernel(kind):
    """Bit for bit the two-pass result in the tiles concerned, close to the oracle everywhere."""
    import ascend_kernel_b200 as ak
    from ascend_kernel_b200 import _abi

    K, N, counts = 2048, 4096, [1300, 0, 257, 1100]
    x, w, s, o, cnt = _case(counts, K, N, False, 6)
    assert _one_pass(x, K, N, len(counts), False)
    redone = torch.zeros(x.shape[0], N, dtype=torch.bool)
    if kind == "few_rows":
        x[300, 5] = 2.0 ** -60           # rows 256 .. 511 of expert 0
        x[1299] = 0
        x[1299, 1:3] = torch.tensor([2.0 ** -50, 1.0])
        w[0, 2] = 0                      # with the weights of the large element zero
        redone[256:512] = redone[1280:1300] = True
    elif kind == "most_rows":
        x[::2, 7] = 2.0 ** -80
        redone[:sum(counts)] = True
    else:
        s[2, 3, 300] = 2.0 ** -30        # expert 2, columns 256 .. 511
        s[3, 1, 0] = 2.0 ** 10           # expert 3, columns 0 .. 255
        redone[1300:1557, 256:512] = redone[1557:2657, 0:256] = True
    gold = O.golden_f32(x, w, s, o, cnt, "int4", O.GROUP_LIST_COUNTS)
    out, st = run_gemm(x, w, s, o, cnt, "int4", gl_type=1)
    assert st == (0, 0)
    d = [t.cuda() for t in (x, w, s, cnt)]
    two = torch.full((x.shape[0], N), SENTINEL, dtype=torch.bfloat16, device="cuda")
    need = _abi.lib.b200moe_grouped_gemm_workspace_bytes(x.shape[0], K, N, 4, _abi.CT["int4"], 0)
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    rc = _abi.lib.b200moe_grouped_gemm(*[t.data_ptr() for t in d[:3]], None, d[3].data_ptr(), two.data_ptr(), x.shape[0], K, N, 4, _abi.CT["int4"], 1, 0,
                                       ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0 and ak.read_status(ws) == (0, 0)
    assert torch.equal(out.cpu()[redone].view(torch.int16), two.cpu()[redone].view(torch.int16))
    if kind == "few_rows":
        assert float(out[1299].abs().max()) < 1e-12  # made of its small element alone
        inv = torch.ones(x.shape[0], 1)
        inv[1299] = 2.0 ** 50
        assert_close_to_golden((out.cpu().float() * inv).to(torch.bfloat16), gold * inv)
    else:
        assert_close_to_golden(out, gold)


def test_captured_graph_replays_on_new_inputs():
    """Scratch of a captured call comes from the graph's pool; the list of tiles to do again is made anew by each replay."""
    import ascend_kernel_b200 as ak

    K, N, counts = 2048, 2048, [1500, 0, 3100, 400]
    x, w, s, cnt = (t.cuda() for t in _case(counts, K, N, False, 8) if t is not None)
    assert _one_pass(x, K, N, 4, False)
    out = torch.zeros(x.shape[0], N, dtype=torch.bfloat16, device="cuda")
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        ak.grouped_gemm(x, w, s, None, cnt, "int4", out, group_list_type=1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        ak.grouped_gemm(x, w, s, None, cnt, "int4", out, group_list_type=1)
    for step in range(3):
        x.copy_(x.flip(0))
        if step == 1:
            x[700, 3] = 2.0 ** -70
        graph.replay()
        torch.cuda.synchronize()
        want = torch.zeros_like(out)
        ak.grouped_gemm(x, w, s, None, cnt, "int4", want, group_list_type=1)
        torch.cuda.synchronize()
        assert torch.equal(out[:5000].view(torch.int16), want[:5000].view(torch.int16))
    assert ak.last_status() == (0, 0)


@pytest.mark.parametrize("positive", [False, True])
def test_offsets_that_cancel_the_codes(positive):
    """Codes 5 .. 7 under offsets about -6: the result is a small part of the codes' and of the offsets' own sums, so it holds only
    where (w + o) * s is formed before the sum.  Rounding to bf16 leaves 2^-9 of each value at most, the fp32 sum about 1e-4 of it."""
    import ascend_kernel_b200 as ak

    gen = torch.Generator().manual_seed(9)
    G, rows, K, N = 16, 40, 7168, 2048
    x = torch.randn(G * rows, K, generator=gen)
    x = (x.abs() if positive else x).to(torch.bfloat16).cuda()
    w = torch.randint(5, 8, (G, K, N), generator=gen, dtype=torch.int8).cuda()
    s = (torch.rand(G, K // 128, N, generator=gen) * 0.045 + 0.005).to(torch.bfloat16).cuda()
    o = (torch.rand(G, K // 128, N, generator=gen) * 0.2 - 6.1).to(torch.bfloat16).cuda()
    packed = (w[:, :, 0::2] | (w[:, :, 1::2] << 4)).contiguous()
    counts = torch.full((G,), rows, dtype=torch.int64, device="cuda")
    y = torch.empty(G * rows, N, dtype=torch.bfloat16, device="cuda")
    ak.grouped_gemm(x, packed, s, o, counts, "int4", y, group_list_type=1)
    err = ref = 0.0
    for g in range(G):
        v = (w[g].double() + o[g].double().repeat_interleave(128, 0)) * s[g].double().repeat_interleave(128, 0)
        want = x[g * rows:(g + 1) * rows].double() @ v
        err += float((y[g * rows:(g + 1) * rows].double() - want).square().sum())
        ref += float(want.square().sum())
    assert (err / ref) ** 0.5 < 2.0 ** -9 + 1e-4


def _control_words(x, w, s, cnt, y):
    """One call on scratch of the test's own: tiles listed for the two-pass kernel, and rows of x that f16 does not hold."""
    from ascend_kernel_b200 import _abi

    (M, K), N, G, ct = x.shape, y.shape[1], cnt.numel(), _abi.CT["int4"]
    need = _abi.lib.b200moe_grouped_gemm_workspace_bytes(M, K, N, G, ct, 0)
    scratch = torch.zeros(_abi.lib.b200moe_grouped_gemm_scratch_bytes(M, K, N, G, ct, 0), dtype=torch.uint8, device="cuda")
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    rc = _abi.lib.b200moe_grouped_gemm_scratch(x.data_ptr(), w.data_ptr(), s.data_ptr(), None, cnt.data_ptr(), y.data_ptr(), M, K, N, G, ct, 1, 0,
                                               ws.data_ptr(), need, scratch.data_ptr(), scratch.numel(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0
    words = scratch[:12].view(torch.int32).tolist()
    return words[0], words[2]


def test_the_one_pass_kernel_runs_and_lists_what_it_leaves():
    """No tile is listed for clean input, and exactly the tiles of an inexact row or an outsized scale otherwise; both bindings give the
    one-pass result, which is not the two-pass one bit for bit."""
    import ascend_kernel_b200 as ak
    from ascend_kernel_b200 import _abi, cinfer_ascendc

    K, N, counts = 2048, 4096, [1300, 0, 257, 1100]
    x, w, s, cnt = (t.cuda() for t in _case(counts, K, N, False, 6) if t is not None)
    y = torch.zeros(x.shape[0], N, dtype=torch.bfloat16, device="cuda")
    assert _control_words(x, w, s, cnt, y) == (0, 0)
    rows = sum(counts)
    two, need = torch.zeros_like(y), _abi.lib.b200moe_grouped_gemm_workspace_bytes(x.shape[0], K, N, 4, _abi.CT["int4"], 0)
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    assert _abi.lib.b200moe_grouped_gemm(x.data_ptr(), w.data_ptr(), s.data_ptr(), None, cnt.data_ptr(), two.data_ptr(), x.shape[0], K, N, 4,
                                         _abi.CT["int4"], 1, 0, ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert not torch.equal(y[:rows].view(torch.int16), two[:rows].view(torch.int16))
    for call in (lambda o: ak.grouped_gemm(x, w, s, None, cnt, "int4", o, group_list_type=1),
                 lambda o: cinfer_ascendc.grouped_gemm(x, w, s, torch.empty(0, dtype=torch.bfloat16, device="cuda"), cnt, "int4", o, group_list_type=1)):
        out = torch.zeros_like(y)
        call(out)
        torch.cuda.synchronize()
        assert torch.equal(out[:rows].view(torch.int16), y[:rows].view(torch.int16))
    x[300, 5] = 2.0 ** -60  # rows 256 .. 511 of expert 0: 16 tiles
    s[2, 3, 300] = 2.0 ** -30  # expert 2, columns 256 .. 511: two tiles of rows
    assert _control_words(x, w, s, cnt, y) == (18, 1)
