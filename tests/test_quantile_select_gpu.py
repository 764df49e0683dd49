"""The device select's own branches against the host rule (bit-identical): rows in
16-byte loads or not (odd k, a table off by 8 bytes), NaN and infinities under the
maximum, bins of the first pass by the number of ranks, keys that differ in their
last bits only, heavy ties, and ranges up to the largest doubles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(jne, engine, eigs, stats=("trace", "maxeig"), ps=(0.01, 0.05, 0.1, 0.5, 0.9, 0.95, 0.99), offset=0):
    import torch

    n, k = eigs.shape
    buf = torch.empty(n * k + offset, dtype=torch.float64, device="cuda")
    buf[offset:] = torch.from_numpy(np.ascontiguousarray(eigs).reshape(-1)).cuda()
    torch.cuda.synchronize()
    for stat in stats:
        got = engine.percentiles_device(buf.data_ptr() + 8 * offset, n, k, stat, list(ps))
        assert got == jne.percentiles(eigs, stat, list(ps)), (stat, n, k, offset)


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 12, 13, 16])
def test_row_lengths_and_alignment(jne, engine, k):
    eigs = np.random.default_rng(k).gamma(2.0, 3.0, size=(3001, k))
    _check(jne, engine, eigs)
    _check(jne, engine, eigs, offset=1)


@pytest.mark.parametrize("n_ps", [1, 2, 3, 5, 8, 9, 16, 17, 33])
def test_number_of_ranks(jne, engine, n_ps):
    eigs = np.random.default_rng(n_ps).standard_normal((50_001, 2)) * 7.0
    _check(jne, engine, eigs, ps=np.linspace(0.0, 1.0, n_ps))


def test_last_bits_ties_and_range(jne, engine):
    rng = np.random.default_rng(5)
    one = np.nextafter(1.0, 2.0) - 1.0
    _check(jne, engine, 1.0 + one * rng.integers(0, 300, size=(100_000, 1)))  # keys in a range of 300
    _check(jne, engine, rng.integers(0, 3, size=(100_000, 1)).astype(float))  # every bin above 64 keys
    _check(jne, engine, np.full((70_000, 1), 2.5))
    wide = rng.standard_normal((100_000, 1)) * 10.0 ** rng.integers(-300, 300, size=(100_000, 1))
    _check(jne, engine, wide)
    clustered = np.concatenate([1.0 + one * rng.integers(0, 2**40, size=(99_990, 1)), rng.standard_normal((10, 1)) * 1e307])
    _check(jne, engine, clustered)


def test_nan_and_infinities_under_the_maximum(jne, engine):
    eigs = np.random.default_rng(6).standard_normal((5000, 4))
    eigs[::7, 1] = np.nan
    eigs[3, :] = np.nan  # folds to the start value
    eigs[10, 0], eigs[11, 2], eigs[12, :] = np.inf, -np.inf, -np.inf
    _check(jne, engine, eigs, stats=("maxeig",), ps=(0.0, 0.25, 0.5, 0.999))
    inf = np.random.default_rng(7).standard_normal((5000, 3))
    inf[:100, 0] = np.inf
    _check(jne, engine, inf, ps=(0.0, 0.5, 0.95))
