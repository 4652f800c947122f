"""Which kernel the fp32 GEMM takes (host only): the shapes by which tests/test_gpu_gemm_f32_split.py means to reach the
tensor-core kernel do, and the ones that the CUDA cores are ahead on do not."""
import ctypes

import pytest

from cavs_b200 import check, lib


def _choice(m, n, k, scratch_bytes=0):
    tile, splits = ctypes.c_int(), ctypes.c_int()
    check(lib().cavs_gemm_f32_choice(m, n, k, ctypes.c_size_t(scratch_bytes), ctypes.byref(tile), ctypes.byref(splits)))
    return tile.value, splits.value


@pytest.mark.parametrize("m,n,k", [(600, 640, 256), (601, 643, 257), (130, 1996, 1028), (3000, 2100, 68), (700, 640, 512), (700, 643, 512)])
def test_shapes_of_the_dispatching_tests_reach_the_tensor_cores(m, n, k):
    tile, splits = _choice(m, n, k)
    assert tile in (64, 128) and splits == 1          # without scratch k is not split


def test_both_tiles_and_the_cuda_cores_are_chosen():
    assert _choice(14474, 10000, 512)[0] == 128
    assert _choice(256, 1536, 512)[0] == 64
    assert _choice(20, 30, 40) == (0, 1)
    assert _choice(64, 64, 0)[0] == 0


def test_splits_fit_the_scratch():
    m, n, k = 256, 1536, 512
    assert _choice(m, n, k, 1 << 30)[1] > 1
    for scratch in (0, m * n * 4, 3 * m * n * 4, 9 * m * n * 4):
        tile, splits = _choice(m, n, k, scratch)
        assert splits == 1 or splits * m * n * 4 <= scratch
