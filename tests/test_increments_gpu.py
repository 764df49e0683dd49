"""The FP64 walk of explicit increments (several lanes per feature, by dim) against
the oracle: every dim, tile edges and partial tiles, and a walk whose increments
cancel exactly."""
import numpy as np
import pytest

from conftest import normwise_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", range(1, 13))
def test_every_dim_and_tile_edge(engine, oracle, jne, dim):
    rng = np.random.default_rng(dim)
    for steps in (31, 32, 33, 63, 65, 250):
        dB = rng.standard_normal((3, steps, dim)) * 10.0 ** rng.integers(-3, 4)
        for model in range(5):
            if steps <= jne.eigen_count(model, dim) + 1:
                continue
            ref = oracle.c_eigs_from_increments(model, dB)
            got = engine.eigs_from_increments(model, dB, precision=jne.PREC_FP64)
            assert normwise_err(got, ref) < 1e-9, (steps, model)
