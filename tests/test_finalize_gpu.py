"""The finalize's own branches: eigenvalues outside FP32's range (the QL shift's
correction then stays in FP64), non-finite moments, and several models in one launch.

Scaling the increments by c scales S11 and S10'S10 alike up to a factor c^2 of the
eigenvalues, exactly for a power of two; 1e-9 is the FP64 tolerance of the parity
tests."""
import numpy as np
import pytest

from conftest import normwise_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2_c", [-90, -70, 70, 90])
def test_eigenvalues_outside_fp32_range(engine, oracle, jne, log2_c):
    c = 2.0 ** log2_c  # eigenvalues of 2^-180 .. 2^180, FP32 ends at 2^128
    for dim in (1, 2, 7, 12):
        dB, _ = engine.export_increments(dim, 300, 4, 3)
        for model in range(5):
            ref = oracle.c_eigs_from_increments(model, dB) * c * c
            got = engine.eigs_from_increments(model, dB * c, precision=jne.PREC_FP64)
            assert normwise_err(got, ref) < 1e-9, (model, dim)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_non_finite_increments_are_reported(engine, jne, precision):
    for bad in (np.inf, np.nan):
        for step in (0, 150, 299):  # the last increment enters S10 only
            dB, _ = engine.export_increments(3, 300, 4, 2)
            dB[1, step, 1] = bad
            with pytest.raises(jne.JneError) as ei:
                engine.eigs_from_increments(0, dB, precision=precision)
            assert ei.value.code == jne.JNE_ERR_NUMERIC


@pytest.mark.parametrize("models", [(4,), (1, 3), (0, 2, 4, 1), (0, 1, 2, 3, 4)])
def test_models_of_one_launch_equal_single_calls(engine, models):
    for precision in (0, 1):
        outs = engine.eigs_seeded_models(models, 6, 700, 3, 131, precision=precision)
        for m in models:
            assert np.array_equal(outs[m], engine.eigs_seeded(m, 6, 700, 3, 131, precision=precision)), m
