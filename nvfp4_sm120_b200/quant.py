"""NVFP4 quantizer: the reference's `quant_nvfp4` / `quant_nvfp4_cuda` surface
(nvfp4_gemm.py:30-48, nvfp4_cuda.py:158-187) on top of the sm_100a kernels."""
from __future__ import annotations

import ctypes
import math

import torch

from . import _lib
from .tensor import BLK, NVFP4Tensor

F4_MAX, F8E4M3_MAX, E4M3_EPS = 6.0, 448.0, 0.015625

_M64 = 2 ** 64 - 1   # seeds, offsets and counters are 64-bit words: any integer, modulo 2^64
_SEED = [0]          # auto-advancing seed of stochastic calls, like nvfp4_cuda.py:154,160-162
_H_OK = {}           # H tensors already checked to be the Sylvester matrix / 4


def hadamard16(device="cuda"):
    """Sylvester Hadamard matrix of order 16, divided by 4 (nvfp4_gemm.py:23-27).  The kernels
    apply exactly this transform as an in-register butterfly; the matrix exists for callers
    that pass it around."""
    h = torch.ones(1, 1, device=device, dtype=torch.float32)
    while h.shape[0] < BLK:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    return h / math.sqrt(BLK)


def _check_h(H):
    if H is None:
        return
    key = (H.data_ptr(), H._version, H.device)
    if key not in _H_OK:
        if H.shape != (BLK, BLK) or not torch.equal(H.float().cpu(), hadamard16("cpu")):
            raise ValueError("H must be hadamard16(): the kernels implement the 16-point Sylvester "
                             "Hadamard transform only")
        _H_OK[key] = True


def _signs(signs, device):
    """A sign vector as the kernels read it (the activation and norm wrappers)."""
    s = signs.to(device=device, dtype=torch.float32).contiguous()
    if s.numel() != BLK:
        raise ValueError("signs must have 16 entries")
    return s


def _device_index(device):
    index = None if device is None else torch.device(device).index
    return torch.cuda.current_device() if index is None else index


def _workspace(device):
    """64-byte scratch of the single-launch quantizer, zeroed once, one per (device, stream): every
    launch leaves it ready for the next, and launches on one stream never overlap."""
    return _lib.host().workspace(_device_index(device))


def fused_error(device=None) -> int:
    """Sticky error word of the quantizers (0 = none): the single-launch quantizer's workspace on the current stream, then
    the word that the kernels without a workspace share on the device.  Reading it synchronises."""
    index = _device_index(device)
    ws = _lib.host().workspace_if_any(index)
    code = 0 if ws is None else int(ws[4].item())
    if code == 0:
        word = ctypes.c_int32(0)
        with torch.cuda.device(index):
            _lib.check(_lib.lib().nvfp4_quantize_wait_status(ctypes.byref(word), 0, _stream(index)), "nvfp4_quantize_wait_status")
        code = word.value
    return code


def _stream(device=None):
    """Handle of torch's current stream on `device` (default: the current device)."""
    return torch.cuda.current_stream(device).cuda_stream


def tensor_amax(t, rht=False, signs=None, transpose=False, out=None):
    """Per-tensor |x| maximum of a 2-D tensor as a 1-element fp32 CUDA tensor (after the Hadamard
    transform of its 16-blocks when rht).  No host synchronisation."""
    return _lib.host().amax(t, bool(rht), signs, bool(transpose), out)


def quant_nvfp4(t, stochastic=False, rht=False, H=None, signs=None, seed=None, *,
                transpose=False, amax=None, philox_offset=0, fused=True, counter=None):
    """t: [M, K] -> NVFP4Tensor blocked along K (K % 16 == 0), as nvfp4_gemm.py:30-48.

    transpose=True quantizes t.t() (blocks along the rows of t) without materialising the
    transpose: the result equals quant_nvfp4(t.t().contiguous(), ...).
    amax: optional 1-element fp32 CUDA tensor to use instead of computing the per-tensor
    maximum here (a tensor sharded across GPUs passes the all-reduced maximum).
    seed=None takes the module counter and advances it on stochastic calls.
    fused=False forces the two-launch path (amax kernel, then quantize kernel) where the
    single-launch cooperative kernel would be used; both give the same bytes.
    counter: (pitch, base) of the stochastic-rounding counter when t is a shard of a larger tensor
    (see nvfp4_quantize_shard_bf16 in the C header); needs amax (the group-reduced one)."""
    if counter is not None and amax is None:
        raise ValueError("a sharded tensor is quantized with the group-reduced amax: pass amax=")
    if seed is None:
        seed = _SEED[0]
        if stochastic:
            _SEED[0] += 1
    _check_h(H)
    pitch, base = (0, 0) if counter is None else (int(counter[0]) & _M64, int(counter[1]) & _M64)
    q, s, pts = _lib.host().quantize(t, bool(stochastic), bool(rht), signs, int(seed) & _M64, bool(transpose), amax,
                                     int(philox_offset) & _M64, bool(fused), counter is not None, pitch, base)
    return NVFP4Tensor(q, s, BLK, t.dtype, pts, True)


def quant_weight_nvfp4(w, amax=None, two_d=False):
    """(quant(w), quant(w.t())) of a weight [N, K] from one read of w, round to nearest: the two
    operands FP4Linear needs (nvfp4_train.py:72-78).  two_d=True scales 16 x 16 tiles (the simulator's
    weight scaling, nvfp4_validate.py:68-82), so that both layouts dequantize to the same matrix.
    amax: optional 1-element fp32 CUDA tensor (a sharded weight passes the group-reduced maximum)."""
    q_r, s_r, q_c, s_c, pts = _lib.host().quantize_weight(w, amax, bool(two_d))
    return (NVFP4Tensor(q_r, s_r, BLK, w.dtype, pts, True), NVFP4Tensor(q_c, s_c, BLK, w.dtype, pts, True))


def tensor_amax_both(t, signs):
    """fp32 [2] = (max|t|, max|RHT_rows(t)|) from one read of t [rows, cols] (rows % 16 == 0): what
    tensor_amax(t) and tensor_amax(t, True, signs, transpose=True) find in two."""
    return _lib.host().amax_both(t, signs)


def quant_dual_nvfp4(t, signs, amax_rows=None, amax_cols=None, stochastic_rows=False, stochastic_cols=False,
                     seed_rows=None, seed_cols=None, philox_offset=0, counters=None):
    """(quant_nvfp4(t, stochastic_rows), quant_nvfp4(t, stochastic_cols, rht=True, signs=signs,
    transpose=True)) from ONE read of t [rows, cols]: the operand and its Hadamard-transformed
    transpose, which FP4Linear needs of every activation and gradient (nvfp4_train.py:36-55).
    amax_rows / amax_cols: 1-element fp32 CUDA tensors (the plain maximum and the maximum after the
    Hadamard transform along the rows); both are found in one extra read when either is missing.
    Seeds left None come from the module counter in the order rows, cols, as two separate stochastic
    calls would draw them.  counters: (pitch_rows, base_rows, pitch_cols, base_cols) for a shard."""
    if seed_rows is None:
        seed_rows = _SEED[0]
        if stochastic_rows:
            _SEED[0] += 1
    if seed_cols is None:
        seed_cols = _SEED[0]
        if stochastic_cols:
            _SEED[0] += 1
    q_r, s_r, p_r, q_c, s_c, p_c = _lib.host().quantize_dual(
        t, signs, amax_rows, amax_cols, bool(stochastic_rows), bool(stochastic_cols), int(seed_rows) & _M64, int(seed_cols) & _M64,
        int(philox_offset) & _M64, [] if counters is None else [int(v) & _M64 for v in counters])
    return (NVFP4Tensor(q_r, s_r, BLK, t.dtype, p_r, True), NVFP4Tensor(q_c, s_c, BLK, t.dtype, p_c, True))


# the reference's second name for the same entry (nvfp4_cuda.py:158)
quant_nvfp4_cuda = quant_nvfp4
