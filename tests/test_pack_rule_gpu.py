"""Small dims run one run per warp while every run has a warp of its own, and packed
pairs beyond: the same bits on both sides of the line, for odd and even counts and
batches that end in the middle of a pair or of 32 runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_same_bits_on_both_sides_of_the_line(engine, dim, precision):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = (12 if precision == 0 else 16) * sms
    big = engine.eigs_seeded(3, dim, 300, 5, line + 35, precision=precision)  # packed
    for n in (1, 31, 33, line - 1, line, line + 1):
        assert np.array_equal(engine.eigs_seeded(3, dim, 300, 5, n, precision=precision), big[:n]), n
