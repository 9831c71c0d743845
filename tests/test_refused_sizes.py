"""Sizes that the fold and the products refuse before anything is launched (no GPU needed; the addresses are never used)."""
import ctypes as C

import pytest
import torch


@pytest.mark.parametrize("cols,first,channels", [((2 * 35, 4 * 9), 0, 4), ((2 * 36, 4 * 9 - 1), 0, 4), ((36, 4 * 9), 0, 4), ((2 * 36, 4 * 9), 2, 4),
                                                 ((2 * 36, 4 * 9), -1, 4), ((2, 36, 4 * 9), 0, 4)])
def test_unfolded_gradient_that_does_not_fit_the_image(cols, first, channels):
    from mptorch_b200 import backend as be

    with pytest.raises(ValueError, match="fold_into"):
        be.fold_into(torch.zeros(cols), torch.zeros(2, 5, 6, 6), first, channels, (3, 3), (1, 1), (1, 1), (1, 1))
    assert be.fold_into(torch.zeros(2 * 36, 36), torch.zeros(2, 5, 6, 6), 1, 4, (3, 3), (1, 1), (1, 1), (1, 1)) is False      # on the CPU


def refused(rc):
    from mptorch_b200 import _cabi

    return rc == 1 and b"too large" in _cabi.lib().mpt_last_error()


@pytest.mark.parametrize("size,kernel,stride,pad,dil", [(3, 1, 1 << 30, 1 << 30, 1), (1, 1, 1, 0x7FFFFFFF, 1), (3, 1, 0x7FFFFFFF, 0, 1),
                                                        (1, 3, 1, 1 << 30, 1 << 30)])
def test_fold_of_images_past_32_bits(size, kernel, stride, pad, dil):
    from mptorch_b200 import _cabi

    fold = _cabi.lib().mpt_fold
    p = C.c_void_p(16)
    assert refused(fold(p, p, 1, 1, size, 1, kernel, 1, stride, 1, pad, 0, dil, 1, size, None))
    assert refused(fold(p, p, 1, 1, 1, size, 1, kernel, 1, stride, 0, pad, 1, dil, size, None))


@pytest.mark.parametrize("M,N,K", [(1, 0x7FFFFFFF, 1), (1, 0x7FFFFFFF - 255, 4), (1, 1, 0x7FFFFFFF), (4, 8, 0x7FFFFFFF - 100)])
def test_products_past_32_bits(M, N, K):
    from mptorch_b200 import _cabi

    p = C.c_void_p(16)
    assert refused(_cabi.lib().mpt_float_mm_nearest(p, p, p, 1, M, N, K, 10, 5, 3, 4, 1, 0, 0, 1, p, 256, None))
