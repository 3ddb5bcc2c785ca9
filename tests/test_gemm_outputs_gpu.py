"""The forms of a product (bf16, fp32, bf16 values held in fp32, with max|D|, quantized) hold the same values, whichever
kernel and however many CTAs per tile the rule picks."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# one shape for each way the rule shares a tile: 64, 128 and 256 columns by 2, 4 and 8 CTAs; then tiles that are not shared
SHAPES = [(768, 768, 8192), (256, 1024, 8192), (104, 352, 9248), (99, 6064, 7136), (64, 4096, 14336), (64, 1104, 14336),
          (8, 14336, 4096), (768, 768, 16384), (2, 2144, 11296), (300, 528, 544), (1000, 2592, 2080)]


@pytest.fixture(scope="module")
def Q():
    import nvfp4_sm120_b200 as pkg
    return pkg


def _operands(Q, m, n, k):
    """Blocks whose scales spread over 2^12: the sums of the products are not exact in fp32, so their order shows."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)

    def make(rows):
        scale = torch.exp2(torch.randint(-6, 7, (rows, k // 16, 1), device="cuda", generator=g).float())
        return Q.quant_nvfp4((torch.randn(rows, k // 16, 16, device="cuda", generator=g) * scale).reshape(rows, k).bfloat16())

    return make(m), make(n).t()


@pytest.mark.parametrize("mnk", SHAPES)
def test_quantized_output_and_maximum_are_those_of_the_plain_product(Q, mnk):
    a, b = _operands(Q, *mnk)
    y = Q.nvfp4_mm(a, b, torch.bfloat16)
    word = torch.full((1,), 9.0, device="cuda")
    for dtype in (torch.bfloat16, torch.float32):
        d = Q.nvfp4_mm(a, b, dtype, amax_out=word)
        assert torch.equal(d, Q.nvfp4_mm(a, b, dtype))
        assert float(word) == float(d.abs().max())
    for factor in (1.0, 0.25):
        amax = y.abs().max().float().reshape(1) * factor
        got, want = Q.nvfp4_mm_fp4out(a, b, amax), Q.quant_nvfp4(y, amax=amax)
        assert torch.equal(got.qdata, want.qdata) and torch.equal(got.per_tensor_scale, want.per_tensor_scale)
        assert torch.equal(got.scale.view(torch.uint8), want.scale.view(torch.uint8))
    assert Q.gemm_status() == 0


@pytest.mark.parametrize("mnk", SHAPES + [(300, 523, 544), (1000, 2585, 2080), (8, 3001, 4096)])
def test_bf16_values_held_in_fp32(Q, mnk):
    """FP4Linear's products for fp32 activations; rows that the TMA store takes and rows (odd N) that it does not."""
    from nvfp4_sm120_b200.gemm import mm_as
    a, b = _operands(Q, *mnk)
    got = mm_as(a, b, torch.float32)
    assert got.dtype == torch.float32 and torch.equal(got, Q.nvfp4_mm(a, b, torch.bfloat16).float())
