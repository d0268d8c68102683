"""p-values of kept pairs over many rounds a block, all of them gathered for the dense evaluation
(a block flushes after every fourth round), against erfc in closed form: the single solve and a
batch, with the table of removed pairs in use and without it."""
import numpy as np
import pytest
from scipy.special import erfc

pytestmark = pytest.mark.gpu


def correlations(p, seed):
    """A dense matrix whose pairs are all far from independent."""
    rng = np.random.default_rng(seed)
    C = np.triu(rng.uniform(0.2, 0.6, (p, p)) * rng.choice([-1.0, 1.0], (p, p)), 1)
    return C + C.T + np.eye(p)


def check(G, pmax, C, n):
    p = C.shape[0]
    iu = np.triu_indices(p, 1)
    assert (G == 1 - np.eye(p, dtype=np.uint16)).all()
    want = erfc(np.sqrt(n - 3) * np.arctanh(np.abs(C[iu])) / np.sqrt(2.0))
    assert (np.abs(pmax[iu] - want) <= 1e-9 * want).all()
    assert (pmax[np.tril_indices(p)] == -1).all()


# n = 903: at 0.05 the table covers the removed pairs, at 1e-6 its range (c atanh <= 3) ends before
@pytest.mark.parametrize("alpha", [0.05, 1e-6])
def test_single_solve(cuda, alpha):
    from gpucsl_gb300 import engine

    n = 903
    for p in (900, 1030):  # 5.2 and 6.8 rounds of 304 blocks of 256 pairs
        C = correlations(p, p)
        s = engine.GaussianSolver(p, 0)
        s.run(cuda.from_numpy(C).cuda(), n, engine.gaussian_thresholds(n, alpha))
        G, _, pmax = s.to_host()
        check(G, pmax, C, n)


@pytest.mark.parametrize("alpha", [0.05, 1e-6])
def test_batch(cuda, alpha):
    from gpucsl_gb300.batch import GaussianBatch

    n, ps = 903, [400, 131, 640, 3, 183]  # 39, 4.2, 100, 1 and 8.1 rounds of 8 blocks
    Cs = [correlations(p, p) for p in ps]
    b = GaussianBatch(ps, [n] * len(ps), alpha, 0)
    b.set_correlations([cuda.from_numpy(C).cuda() for C in Cs])
    b.run()
    for k, C in enumerate(Cs):
        G, _, pmax = b.to_host(k)
        check(G, pmax, C, n)
