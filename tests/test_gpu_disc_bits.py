"""Bit-plane path of discrete levels 0 and 1 against the C oracle at its edges: ends of the
512-sample steps, cardinalities from binary to the widest it takes (and one more, which
leaves it), neighbour groups of several tasks, constant columns, and cardinalities above
the announced maximum (repeated on the general path)."""
import numpy as np
import pytest

from test_gpu_discrete import assert_parity, oracle_discrete, run_gpu

pytestmark = pytest.mark.gpu


def dependent_codes(p, n, card, seed):
    """Columns of cardinality up to `card` that share two hidden causes, so that degrees are
    high; the first column takes every value."""
    rng = np.random.default_rng(seed)
    hidden = rng.random((2, n))
    codes = np.empty((p, n), np.uint8)
    for v in range(p):
        d = int(rng.integers(1 if v % 7 == 3 else 2, card + 1)) if v else card
        x = hidden[v % 2] * 0.35 + rng.random(n) * 0.65
        codes[v] = np.minimum((x * d).astype(np.int64), d - 1)
    codes[0, :card] = np.arange(min(card, n))[:n]
    dims = codes.max(1).astype(np.uint8) + 1
    return codes, dims


@pytest.mark.parametrize("p,n,card,level", [
    (2, 1, 2, 1), (3, 15, 2, 1), (9, 511, 3, 2), (9, 512, 4, 2), (10, 513, 5, 2), (70, 1600, 2, 1), (60, 2100, 3, 1),
    (40, 9001, 5, 2), (14, 4000, 16, 1), (9, 3000, 17, 1), (17, 33000, 9, 1),
])
def test_bit_plane_levels_match_oracle(cuda, p, n, card, level):
    codes, dims = dependent_codes(p, n, card, 100 * p + n)
    assert_parity(run_gpu(codes, dims, 0.05, level), oracle_discrete(codes, dims, 0.05, level))


def test_cardinality_above_the_announced_maximum(cuda):
    """dims beyond max_dim: the general path takes them when its tables fit (level 0 here) and
    refuses them otherwise (level 1: three strata where two were announced)."""
    from gpucsl_gb300 import _lib, engine

    codes, dims = dependent_codes(8, 900, 3, 5)
    s = engine.DiscreteSolver(8, 900, 0, 2)  # announced 2, the data hold 3
    s.load(codes, dims)
    st = s.run(0.05)
    G, sep, pmax = s.to_host()
    assert_parity((G, sep, pmax, st), oracle_discrete(codes, dims, 0.05, 0))
    s = engine.DiscreteSolver(8, 900, 1, 2)
    s.load(codes, dims)
    with pytest.raises(_lib.GcslError) as e:
        s.run(0.05)
    assert e.value.code == _lib.GCSL_ERR_UNSUPPORTED
