"""The FP64 accumulation in exact digits (the engine's own increments) against the
general FP64 path, which takes the same increments as explicit matrices and
accumulates them by multiply-adds: edges of its tiles, chunks and digit scales,
packed and unpacked dims, odd run counts.

Tolerance (per run, normwise): the two round differently, the multiply-adds once
per step: T 2^-53 relative to a moment at most, amplified by the pencil's
condition (up to ~10^4 at dim 12); the explicit matrices also carry one rounding
per increment (dB = z / sqrt(T)).  1e-10 holds T 2^-53 10^4 with a factor of
about ten at T = 10^3 and 2 at 5,000."""
import numpy as np
import pytest

from conftest import normwise_err

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize("dim", range(1, 13))
def test_every_dim_against_the_general_path(engine, jne, dim):
    for steps in (33, 500, 1100, 2500):  # the three chunk lengths and digit scales
        for n in (1, 3):
            dB, _ = engine.export_increments(dim, steps, 9, n)
            for model in range(5):
                if steps <= jne.eigen_count(model, dim) + 1:
                    continue
                ref = engine.eigs_from_increments(model, dB, precision=jne.PREC_FP64)
                got = engine.eigs_seeded(model, dim, steps, 9, n, precision=jne.PREC_FP64)
                assert normwise_err(got, ref) < TOL, (model, dim, steps, n)


@pytest.mark.parametrize("steps", [15, 31, 32, 64, 127, 128, 129, 255, 257, 511, 512, 513, 767, 769, 2047, 2048, 2049,
                                   2559, 2561, 5000])
def test_edges_of_tiles_chunks_and_scales(engine, jne, steps):
    for dim in (2, 5, 12):
        dB, _ = engine.export_increments(dim, steps, 2, 5)
        for model in range(5):
            if steps <= jne.eigen_count(model, dim) + 1:
                continue
            ref = engine.eigs_from_increments(model, dB, precision=jne.PREC_FP64)
            got = engine.eigs_seeded(model, dim, steps, 2, 5, precision=jne.PREC_FP64)
            assert normwise_err(got, ref) < TOL, (model, dim, steps)


def test_more_runs_than_warps(engine, jne):
    # runs taken from the counter give the bits of runs computed alone
    big = engine.eigs_seeded(3, 5, 200, 1, 5001, precision=jne.PREC_FP64)
    assert np.array_equal(big[4990:], engine.eigs_seeded(3, 5, 200, 4991, 11, precision=jne.PREC_FP64))
    pair = engine.eigs_seeded(1, 2, 200, 1, 9001, precision=jne.PREC_FP64)
    assert np.array_equal(pair[8999:], engine.eigs_seeded(1, 2, 200, 9000, 2, precision=jne.PREC_FP64))
