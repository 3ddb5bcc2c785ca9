"""The rule that picks the GEMM's kernel, tile width and CTAs per tile is host arithmetic: what it can return is known
here, and the shapes of the GPU tests reach all of it."""
import ctypes
import random

import pytest


@pytest.fixture(scope="module")
def choose():
    from nvfp4_sm120_b200 import _lib, build
    build.build()
    L = _lib.lib()

    def f(m, n, k):
        out = (ctypes.c_int32 * 3)()
        assert L.nvfp4_gemm_choice(m, n, k, out) == 0
        return tuple(out)
    return f


def _reachable(choose):
    rng = random.Random(0)
    size = lambda lo, hi: int(2 ** rng.uniform(lo, hi))
    return {choose(size(0, 13), size(3, 14), (size(5, 14) + 31) // 32 * 32) for _ in range(100000)}


def test_the_gpu_tests_reach_every_choice(choose):
    import test_gemm_outputs_gpu
    import test_gemm_tiles_gpu
    every = _reachable(choose)
    assert every == {(2, w, 1) for w in (128, 192, 256)} | {(1, w, s) for w in (64, 128, 256) for s in (1, 2, 4, 8)}
    assert {choose(*mnk) for mnk in test_gemm_tiles_gpu.SHAPES} == every
    assert {choose(*mnk) for mnk in test_gemm_outputs_gpu.SHAPES} >= {c for c in every if c[2] > 1}


def test_a_shared_tile_has_work_for_every_cta(choose):
    rng = random.Random(1)
    for _ in range(20000):
        m, n, k = (int(2 ** rng.uniform(0, 14)) for _ in range(3))
        _, width, ctas = choose(m, n, k)
        slices = (k + 255) // 256
        per = -(-slices // ctas)
        assert per * (ctas - 1) < slices and width % (4 * ctas) == 0


def test_arguments(choose):
    from nvfp4_sm120_b200 import _lib
    assert _lib.lib().nvfp4_gemm_choice(1, 1, 32, None) == -1
    assert _lib.lib().nvfp4_gemm_choice(0, 1, 32, (ctypes.c_int32 * 3)()) == -2
