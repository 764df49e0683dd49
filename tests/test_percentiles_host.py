"""The host percentiles' two ways (sorted below 32 values a percentile, selected from there on) and the ranges of equal
values they skip: the values of a plain sort and the reference's interpolation, bit for bit."""
import math

import numpy as np
import pytest


def _plain(agg, ps):
    v = np.sort(agg)
    out = []
    for p in ps:
        rank = p * (len(v) - 1)
        lo, hi = math.floor(rank), math.ceil(rank)
        out.append(v[lo] if lo == hi else v[lo] * (1.0 - (rank - lo)) + v[hi] * (rank - lo))
    return [float(x) for x in out]


@pytest.mark.parametrize("n_ps", [1, 7, 101])
@pytest.mark.parametrize("per", [1, 31, 32, 33, 200])
def test_both_sides_of_the_line(jne, n_ps, per):
    rng = np.random.default_rng(n_ps * 1000 + per)
    n = n_ps * per
    ps = list(rng.uniform(0.0, 1.0, n_ps - 1)) + [1.0]
    few = rng.integers(0, 3, n).astype(float)
    blocks = np.repeat(rng.standard_normal(max(1, n // 16 + 1)), 16)[:n]
    for agg in (rng.standard_normal(n), few, np.full(n, 2.5), blocks, np.sort(few), -np.sort(-blocks),
                np.where(rng.random(n) < 0.1, np.inf, few)):
        assert jne.percentiles(agg[:, None], "maxeig", ps) == _plain(agg, ps)
