"""Discrete tests of few samples, whose chi-squared is a small fraction and often lies exactly on a
jump of the published p-value (a change of branch) or whose p-value on alpha: decisions and p-values
are the oracle's, which evaluates in the published order.  At alpha = 1 the last bit of exp and log
decides, which the host's and the device's need not share: there planes and tables have to agree."""
import numpy as np
import pytest

from test_gpu_discrete import assert_parity, oracle_discrete, run_gpu

pytestmark = pytest.mark.gpu


def few_samples(p, n, card, seed):
    rng = np.random.default_rng(seed)
    mix, hidden = float(rng.choice([0.0, 0.3, 0.7])), rng.random(n)
    codes = np.empty((p, n), np.uint8)
    for v in range(p):
        d = int(rng.integers(1, card + 1))
        codes[v] = np.minimum(((hidden * mix + rng.random(n) * (1 - mix)) * d).astype(int), d - 1)
    return codes, codes.max(1).astype(np.uint8) + 1


@pytest.mark.parametrize("alpha", [0.5, 0.01])
@pytest.mark.parametrize("p,n,card,level", [
    (26, 6, 33, 0), (55, 5, 40, 0), (31, 17, 40, 1), (12, 38, 11, 2), (27, 12, 16, 0), (45, 9, 16, 1), (29, 9, 24, 0),
    (56, 14, 9, 1), (40, 8, 2, 1), (40, 16, 3, 1), (60, 24, 4, 1), (60, 40, 5, 1), (64, 36, 2, 1), (150, 20, 6, 0),
])
def test_decisions_on_the_jumps(cuda, p, n, card, level, alpha):
    for seed in range(6):
        codes, dims = few_samples(p, n, card, 100 * seed + p + n)
        assert_parity(run_gpu(codes, dims, alpha, level), oracle_discrete(codes, dims, alpha, level))


@pytest.mark.parametrize("p,n,card", [(40, 8, 2), (40, 16, 3), (60, 24, 4), (60, 40, 5), (64, 36, 2), (64, 14, 9)])
def test_planes_and_tables_agree_at_one(cuda, p, n, card):
    from test_gpu_disc_routes import solve

    for seed in range(6):
        codes, dims = few_samples(p, n, card, 100 * seed + p + n)
        a, b = (solve(cuda, codes, dims, 1, general, 1.0) for general in (False, True))
        assert all(np.array_equal(x, y) for x, y in zip(a[:2], b[:2]))
        assert (np.abs(a[2] - b[2]) <= 1e-9 * np.abs(b[2])).all()
