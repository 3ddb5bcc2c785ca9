"""The rotary kernel against the torch operations it stands for (models.apply_rotary under autocast), forward and
backward, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 16), (2, 37, 3, 3, 32), (2, 64, 6, 2, 64), (3, 130, 4, 4, 128)])
def test_rotary_is_the_torch_operations(shape):
    from nvfp4_sm120_b200 import models, rotary
    B, T, hq, hk, D = shape
    g = torch.Generator(device="cuda").manual_seed(T)
    make = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    q0, k0, gq, gk = make(B, T, hq, D), make(B, T, hk, D), make(B, hq, T, D), make(B, hk, T, D)
    cos, sin = models.rotary_tables(T, D, "cuda")
    out = []
    for fused in (True, False):
        q, k = q0.clone().requires_grad_(True), k0.clone().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert rotary.takes(q, k, cos, sin)
            if fused:
                a, b = (t.transpose(1, 2) for t in rotary.rotary(q, k, cos, sin))
            else:
                a, b = (models.apply_rotary(t.transpose(1, 2), cos, sin).to(torch.bfloat16) for t in (q, k))
        torch.autograd.backward([a, b], [gq, gk])
        out.append((a, b, q.grad, k.grad))
    for x, y in zip(*out):
        assert x.dtype == y.dtype and torch.equal(x, y)


def test_calls_that_keep_the_torch_operations():
    from nvfp4_sm120_b200 import models, rotary
    q = torch.randn(1, 8, 2, 32, device="cuda")
    cos, sin = models.rotary_tables(8, 32, "cuda")
    assert not rotary.takes(q.bfloat16(), q.bfloat16(), cos, sin)             # no autocast: the result stays fp32
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert not rotary.takes(q, q, cos, sin)                               # fp32 projections
        assert not rotary.takes(q.bfloat16(), q.bfloat16(), cos[..., :8], sin[..., :8])
    with torch.autocast("cuda", dtype=torch.float16):
        assert not rotary.takes(q.bfloat16(), q.bfloat16(), cos, sin)


def _hessian_vector_product(block, x, v, cos, sin):
    from torch.nn.attention import SDPBackend, sdpa_kernel
    with sdpa_kernel(SDPBackend.MATH), torch.autocast("cuda", dtype=torch.bfloat16):
        loss = block(x, cos, sin).square().sum()
    g, = torch.autograd.grad(loss, x, create_graph=True)
    return torch.autograd.grad((g * v).sum(), x)[0]


def test_dense_blocks_have_second_derivatives(monkeypatch):
    """Without FP4 linears everything in a block is differentiable twice, and takes torch.func transforms."""
    from nvfp4_sm120_b200 import models, rotary
    torch.manual_seed(3)
    block = models.DecoderBlock(64, 2, 2, 128, False, "cuda")
    x, v = torch.randn(1, 16, 64, device="cuda", requires_grad=True), torch.randn(1, 16, 64, device="cuda")
    cos, sin = models.rotary_tables(16, 32, "cuda")
    got = _hessian_vector_product(block, x, v, cos, sin)

    def energy(t):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return block(t, cos, sin).square().sum()

    assert torch.func.grad(energy)(x.detach()).shape == x.shape
    monkeypatch.setattr(rotary, "takes", lambda *a: False)
    assert torch.equal(got, _hessian_vector_product(block, x, v, cos, sin))


def test_the_kernel_differentiates_twice():
    """The rotation is linear: the derivative of its backward is the rotation of the direction."""
    from nvfp4_sm120_b200 import models, rotary
    cos, sin = models.rotary_tables(8, 32, "cuda")
    make = lambda: torch.randn(2, 8, 3, 32, device="cuda").bfloat16()
    q, k = make().requires_grad_(True), make().requires_grad_(True)
    a, b = rotary.rotary(q, k, cos, sin)
    ga, gb, u, w = make().requires_grad_(True), make().requires_grad_(True), make(), make()
    dq, dk = torch.autograd.grad([a, b], [q, k], [ga, gb], create_graph=True)
    got = torch.autograd.grad([dq, dk], [ga, gb], [u, w])
    for x, y in zip(got, rotary.rotary(u, w, cos, sin)):
        assert torch.equal(x, y)
