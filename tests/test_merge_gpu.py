"""The mixed kernel's merge takes the moments a model needs only: a single-model
request (its own kinds of sums) equals the same model out of a pass over all five
(every kind) bit for bit, for packed and unpacked dims, one and several chunks, and
in a ragged batch whose neighbours need other kinds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", range(1, 13))
def test_single_model_equals_all_models(engine, jne, dim):
    import torch

    for steps in (256, 1000, 2503):
        full = engine.eigs_seeded_models(range(5), dim, steps, 3, 37, precision=jne.PREC_MIXED)
        reqs = [dict(model=m, dim=dim, steps=steps, seed_first=3, n_runs=37) for m in (4, 0, 3, 1, 2)]
        outs = [torch.empty((37, jne.eigen_count(r["model"], dim)), dtype=torch.float64, device="cuda") for r in reqs]
        engine.run_batch(reqs, [o.data_ptr() for o in outs])
        engine.sync()
        for r, o in zip(reqs, outs):
            m = r["model"]
            assert np.array_equal(engine.eigs_seeded(m, dim, steps, 3, 37, precision=jne.PREC_MIXED), full[m]), (m, steps)
            assert np.array_equal(o.cpu().numpy(), full[m]), (m, steps)
