"""What launches ask for, without a GPU."""
from ctypes import c_int, c_int64

import pytest

from dinfer_b200.kernels.lib import library

SM_SHARED, CTA_SHARED = 228 * 1024, 227 * 1024              # of a B200's SM, and of a CTA at most


@pytest.mark.parametrize("a", [0, 1])
@pytest.mark.parametrize("w", [0, 1])
def test_ctas_that_wait_for_one_another_have_an_sm_each(a, w):
    """CTAs of the 32-bit product that share K hold all of tensor memory while they wait for their cluster: two of them never fit
    on one SM, whatever the tile."""
    f = library("gemm_f32").dinfer_gemm_f32_shared
    f.restype, f.argtypes = c_int64, [c_int] * 4
    for bt in range(16, 113, 16):
        assert 0 < f(a, w, bt, 1) <= CTA_SHARED
        for splits in range(2, 9):
            assert SM_SHARED < 2 * f(a, w, bt, splits) and f(a, w, bt, splits) <= CTA_SHARED
    assert f(a, w, 128, 1) == f(a, w, 24, 1) == f(a, w, 16, 9) == -1


@pytest.mark.parametrize("portions, tokens, heads, state, vdim, wide", [
    (1, 2, 64, 128, 64, True), (32, 64, 64, 128, 64, True), (33, 66, 64, 128, 64, False), (64, 64 * 32, 64, 128, 64, False),
    (64, 64 * 33, 64, 128, 64, True), (16, 64, 16, 64, 64, False), (16, 16 * 64, 16, 64, 64, False), (16, 16 * 65, 16, 64, 64, True),
    (1, 255, 16, 64, 64, False), (1, 256, 16, 64, 64, True), (1, 511, 8, 64, 64, False), (1, 512, 8, 64, 64, True),
    (1, 2000, 24, 16, 64, False), (1, 2731, 24, 16, 64, True), (1, 2000, 16, 128, 60, False), (1, 2000, 16, 72, 64, False), (1, 2000, 16, 144, 64, False)])
def test_which_portions_take_chunks_of_128(portions, tokens, heads, state, vdim, wide):
    f = library("state_space").dinfer_state_space_wide
    f.restype, f.argtypes = c_int, [c_int64, c_int64, c_int, c_int, c_int]
    assert bool(f(portions, tokens, heads, state, vdim)) is wide
