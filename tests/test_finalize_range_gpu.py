"""The finalize near the bottom of the FP64 range: explicit increments so small that the Householder step's squared
norm is subnormal.  1 / x is then still finite (above 2^-1024) and the eigenvalues those of the unscaled increments
times c^2.

Tolerance: squares below 2^-1074 are lost, that is rotations among values 2^-537 and smaller, 2^-26 of the matrix's
2^-511; some fifty such rotations stay within 1e-6."""
import numpy as np
import pytest

from conftest import normwise_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [-1022.5, -1023.0, -1023.5])
def test_subnormal_householder_norm(engine, oracle, jne, bits):
    dB, _ = engine.export_increments(3, 300, 4, 8)
    ref = oracle.c_eigs_from_increments(0, dB)
    for run in range(len(dB)):
        # the pencil of model 0 as the engine forms it: F = the walk, C = E'E with E = S10 L^-T, all unscaled
        F = np.cumsum(dB[run], axis=0) - dB[run]
        E = np.linalg.solve(np.linalg.cholesky(F.T @ F), (dB[run].T @ F).T).T
        C = E.T @ E
        r2 = C[0, 1] ** 2 + C[0, 2] ** 2
        c = 2.0 ** ((bits - np.log2(np.sqrt(r2) * abs(C[0, 1]) + r2)) / 4)  # C scales with c^2, its squares with c^4
        got = engine.eigs_from_increments(0, dB[run:run + 1] * c, precision=jne.PREC_FP64)
        assert normwise_err(got / c / c, ref[run:run + 1]) < 1e-6, run


@pytest.mark.parametrize("log2_c", [-480, -300, -264, -256, -250, -201, -200, 200, 201, 250, 254, 256, 300, 480])
def test_increments_of_any_scale(engine, oracle, jne, log2_c):
    # S11 scales with c^2, C = E'E and the eigenvalues too, by an exact power of two: all normal numbers down to
    # c = 2^-480 and up to 2^480 (1e-9: the FP64 tolerance against the oracle)
    c = 2.0 ** log2_c
    for dim in (1, 2, 3, 5, 12):
        for steps in (40, 2000):
            dB, _ = engine.export_increments(dim, steps, 4, 3)
            for model in range(5):
                one = engine.eigs_from_increments(model, dB, precision=jne.PREC_FP64)
                got = engine.eigs_from_increments(model, dB * c, precision=jne.PREC_FP64)
                assert normwise_err(got / c / c, one) < 1e-9, (model, dim, steps)
                assert normwise_err(one, oracle.c_eigs_from_increments(model, dB)) < 1e-9, (model, dim, steps)


@pytest.mark.parametrize("steps", [40, 64, 300, 320])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_a_single_non_finite_eigenvalue_is_reported(engine, jne, steps, precision):
    dB, _ = engine.export_increments(1, steps, 4, 2)
    for bad in (np.nan, np.inf, -np.inf):
        for step in (0, steps // 2, steps - 1):  # the last increment enters S10 only
            b = dB.copy()
            b[1, step, 0] = bad
            for model in (0, 2, 4):  # one eigenvalue at dim 1
                with pytest.raises(jne.JneError) as ei:
                    engine.eigs_from_increments(model, b, precision=precision)
                assert ei.value.code == jne.JNE_ERR_NUMERIC, (model, bad, step)
