"""Performance cases of the NVFP4 path, one dict of plain values each.

What a program does with this package, through its public entry points and with the values the path
meets in earnest:

  quant    quant_nvfp4 of one bf16 tensor (any rounding mode, row-wise or transposed)
  mm       a matrix product in FP4: both operands quantized in the call (fp4_matmul), the weight
           quantized beforehand (fp4_mm_preqB), or both (nvfp4_mm)
  linear   FP4Linear forward and backward
  ffn      a SwiGLU feed-forward layer, forward and backward, one optimizer step's microbatches
  block    a decoder block (attention + squared-ReLU MLP), forward and backward under autocast

Sizes are those of this repository's benchmark configurations and tests, or generic ones.  `listed()`
names fixed cases, `draw(rng)` takes one more from the same ranges.  Stochastic rounding is seeded from
the state, so a pass on one state gives the same numbers each time (up to the atomics of attention
backward and of split sums)."""
import math

import torch

import nvfp4_sm120_b200 as Q
from nvfp4_sm120_b200 import parallel
from nvfp4_sm120_b200.ffn import SwiGLUFFN
from nvfp4_sm120_b200.models import DecoderBlock, rotary_tables

SEQ = 1024             # sequence length of the decoder block's benchmark configuration


def _quant(rows, cols, mode, transpose=False):
    return dict(kind="quant", rows=rows, cols=cols, mode=mode, transpose=transpose)


def _mm(m, n, k, form, out="bf16", sr=False):
    return dict(kind="mm", m=m, n=n, k=k, form=form, out=out, sr=sr)


def _linear(tokens, cin, cout, dtype, amortize):
    return dict(kind="linear", tokens=tokens, cin=cin, cout=cout, dtype=dtype, amortize=amortize)


def _ffn(tokens, micro, d, hidden, fuse_gate_up):
    return dict(kind="ffn", tokens=tokens, micro=micro, d=d, hidden=hidden, fuse_gate_up=fuse_gate_up)


def _block(batch, seq, dim, heads, kv_heads):
    return dict(kind="block", batch=batch, seq=seq, dim=dim, heads=heads, kv_heads=kv_heads)


def listed():
    return [
        # the smallest call: an activation of a few tokens; launches and host work count, not bytes
        dict(name="quant_small", **_quant(128, 768, "rne")),
        # the quantizer benchmark's tensor
        dict(name="quant_rne", **_quant(8192, 4096, "rne")),
        # ragged rows (not a multiple of 128: padded scale tiles), stochastic rounding: a gradient
        dict(name="quant_sr_ragged", **_quant(5328, 768, "sr")),
        # the weight-gradient operand dY^T of a wide layer: transposed, Hadamard along the tokens, stochastic
        dict(name="quant_rht_sr_t", **_quant(4096, 14336, "rht_sr", True)),
        # decode: a handful of tokens against a weight quantized once
        dict(name="mm_decode", **_mm(8, 14336, 4096, "preqB")),
        # both operands quantized in the call, the ordinary square size
        dict(name="mm_square", **_mm(4096, 4096, 4096, "matmul")),
        # odd sizes in every dimension, fp32 result, stochastic rounding of the left operand
        dict(name="mm_ragged_f32", **_mm(1000, 2584, 7136, "matmul", "f32", True)),
        # the largest product of the GEMM benchmark that is not square, operands quantized beforehand
        dict(name="mm_large", **_mm(16384, 4096, 14336, "preq")),
        # a small layer, weights quantized in every call (the default)
        dict(name="linear_small", **_linear(512, 768, 768, "bf16", False)),
        # a wide layer with fp32 activations, weights quantized once per optimizer step
        dict(name="linear_wide", **_linear(4096, 4096, 4096, "f32", True)),
        # the feed-forward benchmark: two microbatches of an optimizer step, gradients accumulated
        dict(name="ffn", **_ffn(4096, 2, 4096, 14336, True)),
        # one block of the GPT benchmark model at its training batch
        dict(name="block", **_block(16, SEQ, 768, 12, 12)),
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["quant", "quant", "mm", "mm", "linear", "linear", "ffn", "block"])
    if kind == "quant":
        transpose = rng.random() < 0.4
        while True:
            rows = _log_int(rng, 16, 16384, 16 if transpose else 1)
            cols = _log_int(rng, 64, 14336, 16)
            if rows * cols <= 1 << 26:
                return _quant(rows, cols, rng.choice(["rne", "sr", "rht", "rht_sr"]), transpose)
    if kind == "mm":
        while True:
            form = rng.choice(["matmul", "preqB", "preqB", "preq"])
            m = _log_int(rng, 1, 16384)
            n, k = _log_int(rng, 256, 14336, 8), _log_int(rng, 256, 14336, 32)
            if m * n * k <= 1 << 39:
                return _mm(m, n, k, form, rng.choice(["bf16", "bf16", "f32"]), rng.random() < 0.3 and form != "preq")
    if kind == "linear":
        while True:
            tokens = _log_int(rng, 32, 16384, 32)
            cin, cout = _log_int(rng, 128, 8192, 32), _log_int(rng, 128, 8192, 32)
            if tokens * cin * cout <= 1 << 37:
                return _linear(tokens, cin, cout, rng.choice(["bf16", "bf16", "f32"]), rng.random() < 0.6)
    if kind == "ffn":
        while True:
            tokens, micro = _log_int(rng, 64, 8192, 32), rng.choice([1, 1, 2])
            d, hidden = _log_int(rng, 256, 4096, 32), _log_int(rng, 512, 14336, 32)
            if tokens * micro * d * hidden <= 1 << 38:
                return _ffn(tokens, micro, d, hidden, rng.random() < 0.5)
    while True:
        heads, head_dim = rng.choice([4, 6, 8, 12]), rng.choice([64, 64, 128])
        batch, seq = rng.choice([1, 2, 4, 8, 16]), _log_int(rng, 256, SEQ, 32)
        if batch * seq * heads * head_dim <= 16 * SEQ * 768:
            return _block(batch, seq, heads * head_dim, heads, rng.choice([heads, heads, heads // 2]))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape, dtype=torch.bfloat16, outliers=False):
    """N(0, 1), optionally with 0.1 % of the entries scaled by 50 (the quantizer benchmark's tensor)."""
    x = torch.randn(*shape, device="cuda", generator=g)
    if outliers:
        x = torch.where(torch.rand(*shape, device="cuda", generator=g) < 1e-3, x * 50.0, x)
    return x.to(dtype)


def _leaf(t):
    return t.requires_grad_(True)


def prepare(case, seed):
    g = _gen(seed)
    s = dict(case)
    kind = case["kind"]
    s["seed"] = int(seed) % (1 << 31)
    if kind == "quant":
        s["x"] = _normal(g, case["rows"], case["cols"], outliers=True)
        s["signs"] = (torch.randint(0, 2, (16,), device="cuda", generator=g).float() * 2 - 1) if "rht" in case["mode"] else None
    elif kind == "mm":
        m, n, k = case["m"], case["n"], case["k"]
        a, b = _normal(g, m, k), _normal(g, k, n)
        s["out_dtype"] = torch.float32 if case["out"] == "f32" else torch.bfloat16
        s["a"] = Q.quant_nvfp4(a) if case["form"] == "preq" else a
        if case["form"] == "matmul":
            s["b"] = b
        else:
            s["b"] = Q.quant_nvfp4(b.t().contiguous())
    elif kind == "linear":
        Q.set_amortize(case["amortize"])
        lin = Q.FP4Linear(case["cin"], case["cout"], device="cuda")
        with torch.no_grad():
            lin.weight.normal_(std=0.02, generator=g)
        dtype = torch.float32 if case["dtype"] == "f32" else torch.bfloat16
        s["lin"] = lin
        s["x"] = _leaf(_normal(g, case["tokens"], case["cin"], dtype=dtype))
        s["gy"] = _normal(g, case["tokens"], case["cout"], dtype=dtype) * 1e-3
    elif kind == "ffn":
        Q.set_amortize(True)
        s["ffn"] = SwiGLUFFN(case["d"], case["hidden"], device="cuda", seed=int(seed), fuse_gate_up=case["fuse_gate_up"])
        s["x"] = [_leaf(_normal(g, case["tokens"], case["d"])) for _ in range(case["micro"])]
        s["gy"] = [_normal(g, case["tokens"], case["d"]) * 1e-3 for _ in range(case["micro"])]
    else:
        Q.set_amortize(True)
        dim = case["dim"]
        blk = DecoderBlock(dim, case["heads"], case["kv_heads"], 4 * dim, True, "cuda")
        with torch.no_grad():
            for p in blk.parameters():
                if p.dim() == 2:
                    p.normal_(std=0.02, generator=g)
        s["blk"] = blk
        s["rope"] = rotary_tables(case["seq"], dim // case["heads"], "cuda")
        s["x"] = _leaf(_normal(g, case["batch"], case["seq"], dim, dtype=torch.float32))
        s["gy"] = _normal(g, case["batch"], case["seq"], dim, dtype=torch.float32) * 1e-3
    return s


def _bytes_of(q):
    return [q.qdata, q.scale.view(torch.uint8), q.per_tensor_scale]


def run(s):
    kind = s["kind"]
    if kind == "quant":
        mode = s["mode"]
        q = Q.quant_nvfp4(s["x"], stochastic="sr" in mode, rht="rht" in mode, signs=s["signs"], seed=s["seed"],
                          transpose=s["transpose"])
        return _bytes_of(q)
    if kind == "mm":
        if s["form"] == "matmul":
            return Q.fp4_matmul(s["a"], s["b"], sr_a=s["sr"], seed=s["seed"], out_dtype=s["out_dtype"])
        if s["form"] == "preqB":
            return Q.fp4_mm_preqB(s["a"], s["b"], sr_a=s["sr"], seed=s["seed"], out_dtype=s["out_dtype"])
        return Q.nvfp4_mm(s["a"], s["b"].t(), s["out_dtype"])
    parallel.seed_stochastic_rounding(s["seed"], 0)
    if kind == "linear":
        lin, x = s["lin"], s["x"]
        x.grad = lin.weight.grad = None
        y = lin(x)
        y.backward(s["gy"])
        Q.mark_step()                     # the optimizer has moved the weight
        return [y.detach(), x.grad, lin.weight.grad]
    if kind == "ffn":
        ffn = s["ffn"]
        ffn.zero_grad(set_to_none=True)
        out = []
        for x, gy in zip(s["x"], s["gy"]):
            x.grad = None
            y = ffn(x)
            y.backward(gy)
            out += [y.detach(), x.grad]
        Q.mark_step()
        return out + [p.grad for p in ffn.parameters()]
    blk, x = s["blk"], s["x"]
    blk.zero_grad(set_to_none=True)
    x.grad = None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = blk(x, *s["rope"])
    y.backward(s["gy"])
    Q.mark_step()
    return [y.detach(), x.grad] + [p.grad for p in blk.parameters()]


FP4_BYTES = 0.5 + 1.0 / 16        # a quantized element: half a byte of code, a sixteenth of a scale byte


def work(case):
    kind = case["kind"]
    if kind == "quant":
        n = case["rows"] * case["cols"]
        return {"bytes": n * (2 + FP4_BYTES), "flops": 0}
    if kind == "mm":
        m, n, k = case["m"], case["n"], case["k"]
        a = m * k * (FP4_BYTES if case["form"] == "preq" else 2)
        b = n * k * (2 if case["form"] == "matmul" else FP4_BYTES)
        return {"bytes": a + b + m * n * (4 if case["out"] == "f32" else 2), "flops": 2 * m * n * k}
    if kind == "linear":
        t, ci, co = case["tokens"], case["cin"], case["cout"]
        e = 4 if case["dtype"] == "f32" else 2
        return {"bytes": 2 * t * (ci + co) * e + 2 * ci * co * 4, "flops": 6 * t * ci * co}
    if kind == "ffn":
        t, d, h = case["tokens"] * case["micro"], case["d"], case["hidden"]
        return {"bytes": 4 * t * d * 2 + 2 * 3 * d * h * 4, "flops": 18 * t * d * h}
    t, d = case["batch"] * case["seq"], case["dim"]
    kv = case["kv_heads"] * (d // case["heads"])
    weights = d * d * 2 + 2 * d * kv + 8 * d * d
    attention = 3 * 2 * t * case["seq"] * d       # causal: half of the square, scores and values, backward twice forward
    return {"bytes": 4 * t * d * 4 + 2 * weights * 4, "flops": 6 * t * weights + attention}


def tolerance(case):
    """Measured by adding to every product, before its rounding to bf16, the noise of another summation
    order (3e-7 of the result's root mean square, what the fp32 product differs from an fp64 one by)."""
    kind = case["kind"]
    if kind == "quant":
        return "exact"
    if kind == "mm" and case["out"] == "f32":
        return {"rel": 2e-6, "max": 1e-5}           # seen: 3e-7, 1.7e-6
    if kind in ("mm", "linear"):
        return {"rel": 2e-4, "max": 3.2e-2}         # seen: 5.6e-5, and one bf16 step (7.8e-3)
    if kind == "ffn":
        return {"rel": 5e-3, "max": 0.5}            # seen: 1.1e-3, 0.12 (bf16 steps that the next quantization reads)
    # A bf16 step in the tensor that holds a maximum moves a per-tensor scale, and with it the stochastic
    # rounding of part of the gradient's blocks: seen 1e-3 to 0.1 over the gradients of a block.
    return {"rel": 0.03, "max": 0.95}


def _dequantized(t):
    """What quant_nvfp4(t) (round to nearest) stands for, in 64 bits: 1 x 16 blocks along the rows of t, E4M3
    block scales under one fp32 scale of the tensor, E2M1 codes."""
    x = t.to(torch.bfloat16).float()
    blocks = x.view(x.shape[0], -1, 16)
    top = blocks.abs().amax(-1)
    six, one = torch.full_like(top, 6.0), x.new_ones(())
    pts = torch.clamp(top.max(), min=1e-12) / x.new_tensor(2688.0)
    scale = (top / six / pts).clamp(2.0 ** -6, 448.0).to(torch.float8_e4m3fn).float()
    v = (blocks * (one / pts / scale)[..., None]).clamp(-6.0, 6.0)
    a = v.abs()
    v = torch.where(a < 2, torch.round(v * 2) / 2, torch.where(a < 4, torch.round(v), torch.round(v / 2) * 2))
    return (v.double() * scale[..., None].double() * pts.double()).view(x.shape)


def exact(case, seed):
    """Products of operands that are rounded to nearest; where an operand is rounded stochastically, or a
    rounding to bf16 is quantized again, there is no such value."""
    kind = case["kind"]
    if kind == "mm" and not case["sr"]:
        g = _gen(seed)
        m, n, k = case["m"], case["n"], case["k"]
        a, b = _normal(g, m, k), _normal(g, k, n)
        return _dequantized(a) @ _dequantized(b.t().contiguous()).t()
    if kind == "linear":
        s = prepare(case, seed)
        x, w = s["x"].detach(), s["lin"].weight.detach()
        return [_dequantized(x) @ _dequantized(w).t(), None, None]
    return None
