"""The GEMV kernel that streams its operands through shared memory: row counts around its eight rows a unit, k ranges that end in
the middle of a stage, a last slab of 128 columns, more stages than the ring holds."""
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_gemv import SENTINEL, _fp4_case, _int8_case, run_gemv
from tests.util import assert_close_to_golden

pytestmark = pytest.mark.gpu
COUNTS = [8, 0, 9, 16, 17, 1, 7]


@pytest.mark.parametrize("ct,K,N", [
    ("int8", 64, 256), ("int8", 192, 512), ("int8", 1408, 768),
    ("fp8", 128, 128), ("fp8", 1408, 384),
    ("fp4", 64, 256), ("fp4", 320, 512), ("fp4", 2176, 256),
])
def test_matches_oracle(ct, K, N):
    import ascend_kernel_b200 as ak

    gen = torch.Generator().manual_seed(K + N)
    G, cnt, offset = len(COUNTS), torch.tensor(COUNTS, dtype=torch.int64), None
    if ct == "int8":
        x, w, scale, offset, cnt = _int8_case(COUNTS, K, N, K + N, True)
    elif ct == "fp8":
        x = torch.randn(sum(COUNTS), K, generator=gen).to(torch.bfloat16)
        w = torch.randint(0, 256, (G, K, N), generator=gen, dtype=torch.uint8)
        scale = torch.randn(G, K // 128, N // 128, generator=gen)
    else:
        x, w, scale, cnt = _fp4_case(COUNTS, K, N, K + N)
        x[3, 5] = 2.0 ** -100   # a row for the fp32 kernel, in a unit whose second four rows are not done again
        x[8:17, 1] = 2.0 ** -90  # and units that it does as a whole
    x = torch.cat([x, torch.full((2, K), float("nan"), dtype=torch.bfloat16)])  # rows of no expert, beside the last unit's
    gold = O.golden_f32(x, w, scale, offset, cnt, ct, O.GROUP_LIST_COUNTS, weight_layout="canonical", gemv=True)
    for lay in ("canonical", "ascend") if ct == "fp4" else ("canonical",):
        wd = ak.fp4_layout(w.cuda(), to_ascend=True).cpu() if lay == "ascend" else w
        out, st = run_gemv(x, wd, scale, cnt, ct, offset, gl_type=1, layout=lay)
        assert st == (0, 0)
        assert (out[sum(COUNTS):].float() == SENTINEL).all()
        assert_close_to_golden(out, gold, ulps=1.0 if ct == "int8" else 2.0)


def _call(x, w, scale, cnt, ct, y, layout=0):
    """The C entry on a workspace of the test's own, which comes back: status words, operands, counters and sums of the parts."""
    from ascend_kernel_b200 import _abi

    (M, K), N, G = x.shape, y.shape[1], cnt.numel()
    need = _abi.lib.b200moe_grouped_gemv_split_workspace_bytes(M, K, N, G, _abi.CT[ct], layout)
    ws = torch.full((need,), 0xFF, dtype=torch.uint8, device="cuda")
    ws[:256] = 0
    rc = _abi.lib.b200moe_grouped_gemv(x.data_ptr(), w.data_ptr(), scale.data_ptr(), None, cnt.data_ptr(), y.data_ptr(), M, K, N, G,
                                       _abi.CT[ct], 1, layout, ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0
    return ws


@pytest.mark.parametrize("ct,G,N,rows", [
    ("int8", 20, 4096, 1),   # 320 units in two parts of 1024 k: 640 slots of four rows
    ("fp8", 20, 4096, 4),
    ("fp4", 20, 2048, 1),    # 160 units in three parts
    ("int8", 20, 2048, 8),   # slots of eight rows
    ("fp4", 20, 1024, 7),
])
def test_parts_of_the_k_range(ct, G, N, rows):
    """Calls of one or two waves are cut along k as far as there is room for the parts' sums: the sums were written, and what comes
    out is what the oracle gives.  fp4 has rows in every third place that the fp32 kernel does, in parts too."""
    import ascend_kernel_b200 as ak

    K, counts = 2048, [rows] * G
    if ct == "int8":
        x, w, scale, _, cnt = _int8_case(counts, K, N, 3, False)
    elif ct == "fp8":
        gen = torch.Generator().manual_seed(4)
        x, cnt = torch.randn(rows * G, K, generator=gen).to(torch.bfloat16), torch.tensor(counts)
        w = torch.randint(0, 256, (G, K, N), generator=gen, dtype=torch.uint8)
        scale = torch.randn(G, K // 128, N // 128, generator=gen)
    else:
        x, w, scale, cnt = _fp4_case(counts, K, N, 5)
        x[::3, 5] = 2.0 ** -100
    gold = O.golden_f32(x, w, scale, None, cnt, ct, O.GROUP_LIST_COUNTS, weight_layout="canonical", gemv=True)
    x, w, scale, cnt = (t.cuda() for t in (x, w, scale, cnt))
    y = torch.full((rows * G, N), SENTINEL, dtype=torch.bfloat16, device="cuda")
    ws = _call(x, w, scale, cnt, ct, y)
    assert ak.read_status(ws) == (0, 0)
    assert_close_to_golden(y, gold, ulps=1.0 if ct == "int8" else 2.0)
    slots = ws[ws.numel() - 1184 * 1040 * 4:]  # behind the counters
    assert (slots != 0xFF).any(), "the k range was not cut"


def test_one_row_int8_is_as_close_as_fp32_multiply_adds():
    """Every product has its negative at another place of k, so the exact sum is zero and what comes out is the rounding of the
    partial sums alone: fp32 additions in a row and in two levels leave about 1e-7 of half the sum, chained tensor instructions twice that."""
    gen = torch.Generator().manual_seed(6)
    G, K, N = 8, 7168, 4096
    half = torch.randn(G, K // 2, generator=gen).to(torch.bfloat16)
    w = torch.randint(-128, 128, (G, K // 2, N), generator=gen, dtype=torch.int8)
    at = torch.randperm(K // 2, generator=gen)
    x = torch.cat([half, -half[:, at]], 1).cuda()
    scale = torch.ones(G, N, dtype=torch.bfloat16).cuda()
    y = torch.empty(G, N, dtype=torch.bfloat16, device="cuda")
    _call(x, torch.cat([w, w[:, at]], 1).cuda(), scale, torch.ones(G, dtype=torch.int64).cuda(), "int8", y)
    part = torch.einsum("gk,gkn->gn", half.cuda().double(), w.cuda().double())
    assert float(y.double().square().mean().sqrt() / part.square().mean().sqrt()) < 1.35e-7
