"""The device select over the ranges that keys were found in, against the host rule (bit-identical): ties beyond a list's
length with and without neighbours one bit away, clusters inside clusters (each pass finds a range far below its bin),
ranks on both sides of a wide gap, one key alone at either end, and more ranks than a group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(jne, engine, v, ps):
    import torch

    t = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    torch.cuda.synchronize()
    got = engine.percentiles_device(t.data_ptr(), len(v), 1, "trace", list(ps))
    assert got == jne.percentiles(v[:, None], "trace", list(ps))


@pytest.mark.parametrize("n", [64, 65, 129, 2049, 70_001])
def test_ties_and_neighbours(jne, engine, n):
    rng = np.random.default_rng(n)
    ps = np.linspace(0.0, 1.0, 37)
    base = rng.choice([-3.0, 1.0, 1.0 + 2.0**-52, 7.5], n)
    _check(jne, engine, base, ps)
    base[rng.integers(0, n, 5)] = np.nextafter(7.5, 8.0)
    base[rng.integers(0, n, 2)] = [-1e300, 1e300]
    _check(jne, engine, base, ps)
    _check(jne, engine, np.where(rng.random(n) < 0.5, -0.5, 0.5), (0.0, 0.25, 0.49, 0.5, 0.51, 1.0))


@pytest.mark.parametrize("n", [1000, 100_000])
def test_clusters_inside_clusters(jne, engine, n):
    rng = np.random.default_rng(n)
    depth = rng.integers(1, 51, n)  # distances of 2^-1 to 2^-50 from one value
    v = 1.0 + 2.0 ** -depth.astype(float) * np.where(rng.random(n) < 0.3, 1.0, rng.random(n))
    for extra in ([], [np.inf], [-np.inf, np.inf], [5e-324, -5e-324, 1.7e308]):
        _check(jne, engine, np.concatenate([v, extra]), np.linspace(0.0, 1.0, 21))
