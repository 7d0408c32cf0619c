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


def test_fp8_weights_for_scales_of_every_kind():
    """Two-term bf16 products where the scale allows it, fp32 products elsewhere (large, tiny and tie-prone scales), every code."""
    gen = torch.Generator().manual_seed(11)
    G, K, N = 24, 256, 384
    w = torch.arange(256, dtype=torch.uint8).repeat(G * K * N // 256).reshape(G, K, N)
    w = w[:, torch.randperm(K, generator=gen)][:, :, torch.randperm(N, generator=gen)].contiguous()
    s = torch.randn(G, K // 128, N // 128, generator=gen)
    flat = s.view(-1)
    # exact middles of two bf16 numbers for some significand, and one fp32 step to either side of them
    tie = (257.0 / 256.0) / (1 + torch.arange(8, dtype=torch.float64) / 8)
    special = torch.cat([torch.tensor([0.0, 127.9, -128.0, 300.0, 2.0 ** -90, 2.0 ** -91, 2.0 ** -100, 1.0, 1.00390625, -0.75]),
                         tie.float(), torch.nextafter(tie.float(), torch.tensor(2.0)), torch.nextafter(tie.float(), torch.tensor(0.0)),
                         torch.exp2(torch.rand(40, generator=gen) * 96 - 90)])
    flat[:special.numel()] = special
    got = _readback(w, s, "fp8", "canonical", G, K, N)
    assert torch.equal(got, O.dequant_fp8(w, s, round_bf16=True))
