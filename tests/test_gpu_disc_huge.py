"""The general discrete path beyond 2^31 samples, where the products of two counts leave 64-bit
signed integers: the statistic of one skewed pair against its exact value."""
from fractions import Fraction

import numpy as np
import pytest
from scipy.stats import chi2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1 << 31) - 16, 3_200_000_016])
def test_level0_of_billions_of_samples(cuda, n):
    from gpucsl_gb300 import engine

    rare, both = n // 32, n // 1024 + 3000  # codes 1 of each column, and of both
    s = engine.DiscreteSolver(2, n, 0, 2)
    s.data.zero_()
    s.data[0, :rare] = 1
    s.data[1, rare - both:2 * rare - both] = 1
    s.dims.fill_(2)
    s.run(1e-9)
    G, _, pmax = s.to_host()
    N = [[n - 2 * rare + both, rare - both], [rare - both, both]]
    m = [n - rare, rare]
    x = sum(Fraction((N[a][b] * n - m[a] * m[b]) ** 2, m[a] * m[b] * n) for a in range(2) for b in range(2))
    want = float(chi2.sf(float(x), 1))
    assert 1e-9 < want < 0.5 and G[0, 1] == 0
    # the normal tail is a published polynomial (absolute error below 1e-6)
    assert abs(pmax[0, 1] - want) < 2e-6
