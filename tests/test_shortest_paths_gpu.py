"""FP64 paths of at most one tile (32 steps), summed in FP64 multiply-adds: every dim and
model against the general path on the same increments, one model alone against the pass
that serves all five (which sums every moment), and runs taken from the counter or
through the no-allocation entry against runs computed alone.

Tolerance (per run, normwise): both sides sum T products in FP64; the explicit matrices
carry one rounding per increment (dB = z / sqrt(T)), 2^-53 relative, amplified by the
pencil's condition (up to ~10^4 on 24 steps at dim 12): 1e-11 holds 2^-53 10^4 with a
factor of about ten."""
import numpy as np
import pytest

from conftest import normwise_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", range(1, 13))
def test_every_dim_and_model(engine, jne, dim):
    for steps in (24, 32):
        dB, _ = engine.export_increments(dim, steps, 3, 7)
        every = engine.eigs_seeded_models(range(5), dim, steps, 3, 7, precision=jne.PREC_FP64)
        for model in range(5):
            got = engine.eigs_seeded(model, dim, steps, 3, 7, precision=jne.PREC_FP64)
            ref = engine.eigs_from_increments(model, dB, precision=jne.PREC_FP64)
            assert normwise_err(got, ref) < 1e-11, (model, dim, steps)
            assert normwise_err(got, every[model]) < 1e-11, (model, dim, steps)


@pytest.mark.parametrize("dim", [1, 4, 12])
def test_bits_do_not_depend_on_the_batch(engine, jne, dim):
    big = engine.eigs_seeded(3, dim, 30, 1, 20011, precision=jne.PREC_FP64)
    assert np.array_equal(big[20000:], engine.eigs_seeded(3, dim, 30, 20001, 11, precision=jne.PREC_FP64))
    mixed = engine.eigs_seeded(3, dim, 30, 20001, 11, precision=jne.PREC_MIXED)  # short paths run in FP64
    assert np.array_equal(big[20000:], mixed)
