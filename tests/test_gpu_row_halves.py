"""Row halves of the generic GEMM's tiles: 64 and 65 rows (M = 64 and M = 128), one and two boxes of 32 rows, in tiles of one half and of
two, in every format."""
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_gemm import SENTINEL, run_gemm
from tests.util import assert_close_to_golden, same_bits

pytestmark = pytest.mark.gpu
ONE_HALF = [128, 64, 65, 1, 32, 33, 0]
TWO_HALVES = [129, 192, 193, 64 + 256, 256, 160, 5]


@pytest.mark.parametrize("ct", ["int8", "int4", "fp8", "fp4", "bf16"])
def test_matches_oracle_and_does_not_depend_on_the_other_experts(ct):
    gen = torch.Generator().manual_seed(41)
    G, K, N = 7, 640, 512  # ten stages
    rows = max(sum(ONE_HALF), sum(TWO_HALVES))
    x = torch.randn(rows + 2, K, generator=gen).to(torch.bfloat16)
    scale = offset = None
    if ct == "int8":
        w = torch.randint(-128, 128, (G, K, N), generator=gen, dtype=torch.int8)
        scale = (torch.rand(G, N, generator=gen) * 0.009 + 0.001).to(torch.bfloat16)
        offset = (torch.rand(G, N, generator=gen) * 8 - 4).to(torch.bfloat16)
    elif ct == "int4":
        w = torch.randint(0, 256, (G, K, N // 2), generator=gen, dtype=torch.uint8).view(torch.int8)
        scale = (torch.rand(G, K // 128, N, generator=gen) * 0.045 + 0.005).to(torch.bfloat16)
        offset = (torch.rand(G, K // 128, N, generator=gen) * 4 - 2).to(torch.bfloat16)
    elif ct == "fp8":
        w = torch.randint(0, 256, (G, K, N), generator=gen, dtype=torch.uint8)
        scale = torch.randn(G, K // 128, N // 128, generator=gen) * 0.05
    elif ct == "fp4":
        w = torch.randint(0, 256, (G, K, N // 2), generator=gen, dtype=torch.uint8).view(torch.int8)
        scale = (torch.rand(G, K // 16, N, generator=gen) * 0.09 + 0.01).to(torch.bfloat16)
    else:
        w, scale = (torch.randn(G, K, N, generator=gen) * K ** -0.5).to(torch.bfloat16), torch.empty(0)
    for layout in ("canonical", "ascend") if ct == "fp4" else ("canonical",):
        wl = O.ascend_shuffle(w) if layout == "ascend" else w
        first = {}
        for counts in (ONE_HALF, TWO_HALVES):
            cnt = torch.tensor(counts, dtype=torch.int64)
            gold = O.golden_f32(x, w, scale, offset, cnt, ct, O.GROUP_LIST_COUNTS, weight_layout="canonical")
            out, st = run_gemm(x, wl, scale, offset, cnt, ct, gl_type=1, layout=layout)
            assert st == (0, 0)
            assert (out[sum(counts):].float() == SENTINEL).all()
            assert_close_to_golden(out, gold)
            first[len(first)] = out[:64]
        assert same_bits(first[0], first[1])  # the first expert's rows, in a tile of one half and of two
