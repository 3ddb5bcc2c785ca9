"""fp32 operands: the kernel that rounds to bf16 and finds the maxima on the way gives the bytes of a cast followed by
the quantization of the copy."""
import pytest
import torch

from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def Q():
    import nvfp4_sm120_b200 as pkg
    return pkg


def _same(a, b):
    return (torch.equal(a.qdata, b.qdata) and torch.equal(a.scale.view(torch.uint8), b.scale.view(torch.uint8))
            and torch.equal(a.per_tensor_scale, b.per_tensor_scale))


@pytest.mark.parametrize("shape,pad", [((16, 16), 0), ((48, 528), 0), ((80, 1040), 4), ((2064, 2048), 0), ((64, 48), 3)])
def test_fp32_operands_quantize_like_their_bf16_copy(Q, shape, pad):
    rows, cols = shape
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols + pad, device="cuda", generator=g)[:, :cols]
    x[rows // 2, cols - 1] = -77.3                              # the maximum is the last column's
    b = x.to(torch.bfloat16)
    signs = O.signs_from_seed(4).cuda()
    assert _same(Q.quant_nvfp4(x), Q.quant_nvfp4(b))
    assert _same(Q.quant_nvfp4(x, transpose=True), Q.quant_nvfp4(b, transpose=True))
    assert _same(Q.quant_nvfp4(x, True, seed=3, transpose=True), Q.quant_nvfp4(b, True, seed=3, transpose=True))
    for u, v in zip(Q.quant_weight_nvfp4(x), Q.quant_weight_nvfp4(b)):
        assert _same(u, v)
    for u, v in zip(Q.quant_dual_nvfp4(x, signs, None, None, True, True, 5, 6),
                    Q.quant_dual_nvfp4(b, signs, None, None, True, True, 5, 6)):
        assert _same(u, v)
    assert Q.quant_nvfp4(x).orig_dtype == torch.float32


def test_values_that_are_not_finite(Q):
    x = torch.randn(32, 64, device="cuda")
    x[3, 5], x[7, 9] = float("inf"), float("nan")
    a, b = Q.quant_weight_nvfp4(x), Q.quant_weight_nvfp4(x.to(torch.bfloat16))
    for u, v in zip(a, b):
        assert torch.equal(u.qdata, v.qdata) and torch.equal(u.scale.view(torch.uint8), v.scale.view(torch.uint8))


@pytest.mark.parametrize("offset", [1, 2, 3, 4])
def test_starts_that_are_not_aligned(Q, offset):
    """A view into a flat fp32 buffer at any element, as a parameter of a flattened module is."""
    flat = torch.randn(64 * 96 + 8, device="cuda")
    x = flat[offset:offset + 64 * 96].view(64, 96)
    b = x.to(torch.bfloat16)
    signs = O.signs_from_seed(4).cuda()
    for u, v in zip(Q.quant_weight_nvfp4(x), Q.quant_weight_nvfp4(b)):
        assert _same(u, v)
    for u, v in zip(Q.quant_dual_nvfp4(x, signs), Q.quant_dual_nvfp4(b, signs)):
        assert _same(u, v)
    assert _same(Q.quant_nvfp4(x, transpose=True), Q.quant_nvfp4(b, transpose=True))
    big = torch.randn(2048 * 2048 + 8, device="cuda")[offset:offset + 2048 * 2048].view(2048, 2048)
    assert _same(Q.quant_nvfp4(big), Q.quant_nvfp4(big.to(torch.bfloat16)))


def test_a_negated_view(Q):
    x = torch.randn(64, 96, device="cuda")
    for u, v in zip(Q.quant_weight_nvfp4(torch._neg_view(x)), Q.quant_weight_nvfp4(-x)):
        assert _same(u, v)
