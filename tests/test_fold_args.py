"""Sizes that the fold and the products refuse before anything is launched (no GPU needed)."""

import pytest
import torch


@pytest.mark.parametrize("cols,first,channels", [((2 * 35, 4 * 9), 0, 4), ((2 * 36, 4 * 9 - 1), 0, 4), ((36, 4 * 9), 0, 4), ((2 * 36, 4 * 9), 2, 4),
                                                 ((2 * 36, 4 * 9), -1, 4), ((2, 36, 4 * 9), 0, 4)])
def test_unfolded_gradient_that_does_not_fit_the_image(cols, first, channels):
    from mptorch_b200 import backend as be

    with pytest.raises(ValueError, match="fold_into"):
        be.fold_into(torch.zeros(cols), torch.zeros(2, 5, 6, 6), first, channels, (3, 3), (1, 1), (1, 1), (1, 1))
    assert be.fold_into(torch.zeros(2 * 36, 36), torch.zeros(2, 5, 6, 6), 1, 4, (3, 3), (1, 1), (1, 1), (1, 1)) is False      # on the CPU
