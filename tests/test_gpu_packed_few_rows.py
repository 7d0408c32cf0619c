"""The packed GEMM's path for at most 16 rows an expert: row counts around 8 and 16, k ranges that end in the middle of a
stage, plain, gate/up and scattered results."""
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_gemm import SENTINEL, _int8_case
from tests.test_gpu_gemm_packed import run_packed
from tests.util import assert_close_to_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,K,N,with_offset", [
    ([1], 64, 256, False),                             # half a stage
    ([8, 9, 0, 16, 1, 15] + [0] * 4, 192, 512, True),  # one and two instructions' rows; a stage and a half
    ([16, 7, 3] * 5 + [0] * 5, 1088, 1024, True),      # more stages than the ring, more tiles than it has slots
    ([2] * 170, 128, 256, False),                      # more tiles than multiprocessors, one stage each
    ([16, 17, 2, 1] + [0] * 4, 192, 512, True),        # one row too many on one expert: the other path
])
def test_matches_oracle(counts, K, N, with_offset):
    x, w, scale, offset, cnt = _int8_case(counts, K, N, 31, with_offset, extra_rows=2)
    assert x.shape[0] <= 8 * len(counts)
    x[-2:] = float("nan")  # rows of no expert, beside the last tile's
    gold = O.golden_f32(x, w, scale, offset, cnt, "int8", O.GROUP_LIST_COUNTS)
    out, st = run_packed(x, w, scale, offset, cnt)
    assert st == (0, 0)
    assert (out[-2:].float() == SENTINEL).all()
    assert_close_to_golden(out, gold)
    again, _ = run_packed(x, w, scale, offset, torch.cumsum(cnt, 0), gl_type=0)
    assert torch.equal(out.view(torch.int16), again.view(torch.int16))
    act, st = run_packed(x, w, scale, offset, cnt, gate_up=True)
    assert st == (0, 0)
    h = gold[:-2].to(torch.bfloat16).float()
    want = (torch.nn.functional.silu(h[:, :N // 2]) * h[:, N // 2:]).to(torch.bfloat16).float()
    assert O.rel_l2(act[:-2].float().cpu(), want) < 4e-3


def test_scattered_rows_are_the_plain_ones():
    """Rows go where their codes say, into two destination tensors; a code that names no destination, or a row past its end, is skipped
    and nothing else is touched.  Experts of at most 16 rows: results of one and of two instructions' rows."""
    from ascend_kernel_b200 import ops

    x, w, scale, offset, cnt = _int8_case([16, 0, 7, 9, 1, 3] + [0] * 4, 192, 512, 37, True)
    M, N = x.shape[0], w.shape[2]
    assert M <= 8 * cnt.numel()
    want, st = run_packed(x, w, scale, offset, cnt)
    assert st == (0, 0)
    at = torch.randperm(M, generator=torch.Generator().manual_seed(8))
    base = (torch.arange(M) % 2).to(torch.int64)
    code = (base << 32) | at.to(torch.int64)
    code[4], code[20] = (7 << 32) | 0, (1 << 32) | (M + 10)
    dst = [torch.full((M, N), SENTINEL, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    ops.grouped_gemm_packed_scatter(x.cuda(), ops.pack_weight_int8(w.cuda()), scale.cuda(), offset.cuda(), cnt.cuda(), code.cuda(),
                                    [d.data_ptr() for d in dst], M, group_list_type=1)
    torch.cuda.synchronize()
    expected = torch.full((2, M, N), SENTINEL, dtype=torch.bfloat16)
    for r in range(M):
        if r not in (4, 20):
            expected[base[r], at[r]] = want[r].cpu()
    assert torch.equal(torch.stack(dst).cpu().view(torch.int16), expected.view(torch.int16))
