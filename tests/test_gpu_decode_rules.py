"""The decode rules of the GEMM kernels at the scales where they change over, bit for bit: an identity x reads the dequantised
weights back."""
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_gemm import run_gemm

pytestmark = pytest.mark.gpu


def _readback(w, s, ct, layout, G, K, N):
    eye = torch.eye(K, dtype=torch.bfloat16).repeat(G, 1)
    out, st = run_gemm(eye, w, s, None, torch.full((G,), K, dtype=torch.int64), ct, gl_type=1, layout=layout)
    assert st == (0, 0)
    return out.cpu().float().reshape(G, K, N)


@pytest.mark.parametrize("layout", ["canonical", "ascend"])
def test_fp4_weights_for_scales_on_both_sides_of_four(layout):
    """Scales that hold the decode's 2^126 and scales that do not, in one matrix and in one warp."""
    gen = torch.Generator().manual_seed(12)
    G, K, N = 3, 128, 512
    w = torch.randint(0, 256, (G, K, N // 2), generator=gen, dtype=torch.uint8)
    s = (torch.rand(G, K // 16, N, generator=gen) * 3 + 0.5).to(torch.bfloat16)
    s[0, 1] = torch.tensor([3.984375, 4.0, -4.0, 448.0]).repeat(N // 4).to(torch.bfloat16)
    s[1, :, 100] = 2.0 ** 100
    s[1, 3] = torch.tensor([2.0 ** -120, 2.0 ** -125, 0.0, -2.0 ** -60]).repeat(N // 4).to(torch.bfloat16)
    s[2] *= -1
    got = _readback(O.ascend_shuffle(w) if layout == "ascend" else w, s, "fp4", layout, G, K, N)
    assert torch.equal(got, O.dequant_fp4(w, s, round_bf16=True))
