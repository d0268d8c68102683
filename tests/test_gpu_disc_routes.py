"""Discrete levels 0 and 1 whichever way they are counted, on bit planes or with a table for each
test: the same results on both sides of every line between the two (cardinality, variables,
samples, sparse and dense graphs), and with every graph the oracle's where it is quick."""
import numpy as np
import pytest

from test_gpu_disc_bits import dependent_codes
from test_gpu_discrete import assert_parity, oracle_discrete

pytestmark = pytest.mark.gpu


def independent_codes(p, n, card, seed):
    """Columns in pairs: the graph has p / 2 edges."""
    rng = np.random.default_rng(seed)
    codes = rng.integers(0, card, (p, n)).astype(np.uint8)
    half = codes[1::2]
    half[:] = np.where(rng.random(half.shape) < 0.5, codes[:p - p % 2:2], half)
    codes[:, :card] = np.arange(card)
    return codes, np.full(p, card, np.uint8)


def solve(torch, codes, dims, level, general, alpha=0.05):
    from gpucsl_gb300 import _lib, engine

    p, n = codes.shape
    s = engine.DiscreteSolver(p, n, level, int(dims.max()))
    if general:  # no room for the planes
        s.workspace = s.workspace[:int(_lib.lib().gcsl_disc_workspace_bytes(p, n, level, 1))]
    s.load(codes, dims)
    st = s.run(alpha)
    return (*s.to_host(), st)


@pytest.mark.parametrize("make", [dependent_codes, independent_codes])
@pytest.mark.parametrize("p,n,card", [
    (9, 700, 2), (10, 700, 2), (13, 1025, 3), (14, 1023, 3), (18, 2500, 4), (33, 900, 8), (34, 900, 8), (41, 31, 6),
    (40, 20011, 5), (63, 800, 9), (64, 800, 9), (127, 400, 11), (128, 16384, 11), (128, 16385, 11), (130, 90, 16),
    (20, 65000, 4), (64, 4097, 2),
])
def test_both_ways_agree(cuda, make, p, n, card):
    codes, dims = make(p, n, card, 31 * p + n)
    a, b = solve(cuda, codes, dims, 1, False), solve(cuda, codes, dims, 1, True)
    assert (a[0] == b[0]).all() and (a[1] == b[1]).all()
    assert a[3].raw["tests"] == b[3].raw["tests"] and a[3].raw["removed"] == b[3].raw["removed"]
    assert (np.abs(a[2] - b[2]) <= 1e-9 * np.abs(b[2])).all()
    if p * p * p * n < 3e9:
        assert_parity(a, oracle_discrete(codes, dims, 0.05, 1))
