"""Every kernel, tile width and cluster size that the GEMM's rule can choose, at sizes with ragged tiles, against a
64-bit matmul of the dequantised operands.  Tolerance: fp32 accumulation of K products whose rounding errors are
independent, about sqrt(K) * 2^-24 of the result's norm, K <= 14336: 7e-6; stated 1e-5."""
import pytest
import torch

from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu

# (tests/test_gemm_rule_cpu.py checks that these reach every choice)
SHAPES = [
    (512, 768, 768), (129, 72, 256), (1, 8, 32), (300, 2088, 544),       # 128 x 64 tiles, odd column halves of a scale group
    (130, 4952, 96), (8, 11600, 2208), (1024, 4104, 992),                # 128 x 128, 128 x 256
    (2040, 776, 3104), (1000, 2584, 2080), (3000, 3000, 800),            # pair, 256 x 128 / 192 / 256, several tiles per pair
    (768, 768, 8192), (300, 520, 8000), (33, 72, 4128), (104, 352, 9248),    # 128 x 64 shared by 2, 4, 4, 8
    (99, 6056, 7136), (8, 3000, 4096), (127, 2000, 8224), (64, 1096, 14336),    # 128 x 128 by 2, 4; 128 x 64 by 4; 128 x 128 by 8
    (11, 9640, 5120), (1574, 400, 11488), (2, 2144, 11296)]              # 128 x 256 by 2, 4, 8


@pytest.fixture(scope="module")
def Q():
    import nvfp4_sm120_b200 as pkg
    return pkg


def _dequant(q):
    rows, k = q.qdata.shape[0], q.qdata.shape[1] * 2
    return O.dequant_parts(q.qdata, q.scale.view(torch.uint8), q.per_tensor_scale, rows, k).double().cuda()


@pytest.mark.parametrize("mnk", SHAPES)
def test_rule_choices_match_the_dequantised_product(Q, mnk):
    m, n, k = mnk
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    qa = Q.quant_nvfp4(torch.randn(m, k, device="cuda", generator=g).bfloat16())
    qb = Q.quant_nvfp4(torch.randn(n, k, device="cuda", generator=g).bfloat16()).t()
    want = _dequant(qa) @ _dequant(qb).t()
    f32 = Q.nvfp4_mm(qa, qb, torch.float32)
    bf16 = Q.nvfp4_mm(qa, qb, torch.bfloat16)
    assert Q.gemm_status() == 0
    assert ((f32.double() - want).norm() / want.norm()).item() < 1e-5
    assert torch.equal(bf16, f32.to(torch.bfloat16))          # one rounding of the same accumulators
    assert torch.equal(f32, Q.nvfp4_mm(qa, qb, torch.float32))     # the same bits on every run
    wide = torch.full((m, n + 8), 7.0, device="cuda")         # nothing is written outside the result
    Q.nvfp4_mm(qa, qb, torch.float32, out=wide[:, :n])
    assert torch.equal(wide[:, :n], f32) and bool((wide[:, n:] == 7.0).all())
