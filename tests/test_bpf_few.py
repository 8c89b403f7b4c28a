"""BPF's 2-D filter of few slices: launches of few CTAs take their transforms
with passes over shared memory of their own, others with passes that ride on the
stages.  The arithmetic is the same, so the bits are."""
import numpy as np
import pytest
import torch

from algotom_b200.rec import reconstruction as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,pad", [(1, 1), (17, 2), (100, 15), (64, 9),
                                      (301, 45)])
def test_bits_do_not_depend_on_the_number_of_slices(cuda, ncol, pad):
    n = 2 * (600 // (ncol + 2 * pad) + 2)
    x = torch.from_numpy(np.random.default_rng(ncol).uniform(
        0.1, 1.0, (ncol, n, ncol)).astype(np.float32)).to(cuda)
    many = R._circular_filter(x, None, "hann", pad, "edge")
    few = R._circular_filter(x[:, :2], None, "hann", pad, "edge")
    assert torch.equal(many[:, :2], few)
