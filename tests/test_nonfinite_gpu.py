"""NaN and infinities in the operands.  The per-tensor maximum counts every element that is a number (an infinity too) and
no NaN, whichever kernel finds it, so that the entry points agree on the bytes and one NaN does not rescale a tensor."""
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


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("shape", [(32, 64), (48, 528), (2064, 2048), (8192, 4096)])
def test_one_maximum_for_every_entry_point(Q, shape, bad):
    """The largest number sits in the 16-byte word of the value that is not finite."""
    from nvfp4_sm120_b200 import quant
    rows, cols = shape
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x32 = torch.randn(rows, cols, device="cuda", generator=g).bfloat16().float()
    x32[3, 6], x32[3, 5], x32[rows - 1, cols - 2] = -77.0, bad, bad
    signs = O.signs_from_seed(4).cuda()
    first = None
    for x in (x32.bfloat16(), x32):
        dual = Q.quant_dual_nvfp4(x, signs, None, None, True, True, 5, 6)
        single = Q.quant_nvfp4(x, True, seed=5), Q.quant_nvfp4(x, True, True, signs=signs, seed=6, transpose=True)
        assert _same(dual[0], single[0]) and _same(dual[1], single[1])
        assert _same(Q.quant_nvfp4(x), Q.quant_nvfp4(x, fused=False))
        assert _same(Q.quant_nvfp4(x, rht=True, signs=signs), Q.quant_nvfp4(x, rht=True, signs=signs, fused=False))
        want = 77.0 if bad != bad else bad
        both = quant.tensor_amax_both(x, signs)
        assert float(quant.tensor_amax(x)) == float(both[0]) == want
        assert float(quant.tensor_amax(x, True, signs, transpose=True)) == float(both[1])
        weight = Q.quant_weight_nvfp4(x)
        for u in (*weight, Q.quant_nvfp4(x, transpose=True), dual[0]):
            assert torch.equal(u.per_tensor_scale, weight[0].per_tensor_scale)
        assert _same(Q.quant_nvfp4(x), weight[0]) and _same(Q.quant_nvfp4(x, transpose=True), weight[1])
        if first is None:
            first = dual
        assert _same(dual[0], first[0]) and _same(dual[1], first[1])
    # pitched rows take the strided loads
    wide = torch.zeros(rows, cols + 8, device="cuda", dtype=torch.bfloat16)
    wide[:, :cols] = x32
    assert _same(Q.quant_nvfp4(wide[:, :cols]), Q.quant_nvfp4(x32.bfloat16()))
    assert float(quant.tensor_amax(wide[:, :cols])) == want


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_row_with_a_nan_leaves_the_other_rows_of_a_layer(Q, dtype):
    lin = Q.FP4Linear(256, 128)
    x = torch.randn(64, 256, device="cuda", dtype=dtype)
    spoiled = x.clone()
    spoiled[5, 7] = float("nan")
    y, z = (lin(t.requires_grad_(True)) for t in (x, spoiled))
    keep = torch.arange(64, device="cuda") != 5
    assert torch.equal(y[keep], z[keep]) and float(y.abs().max()) > 0


def test_products_that_are_not_numbers_do_not_count(Q):
    qa = Q.quant_nvfp4(torch.cat([torch.zeros(64, 64), torch.ones(64, 64)]).cuda().bfloat16())
    qb = Q.quant_nvfp4(torch.ones(48, 64, device="cuda", dtype=torch.bfloat16))
    qa.per_tensor_scale.fill_(float("inf"))              # 0 * inf in the first half of the rows
    word = torch.zeros(1, device="cuda")
    d = Q.nvfp4_mm(qa, qb.t(), torch.float32, amax_out=word)
    assert bool(torch.isnan(d[:64]).all()) and bool(torch.isinf(d[64:]).all())
    assert float(word) == float("inf")
