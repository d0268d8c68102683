"""Batched levels whose edges fill the chip several times over, so that a group of lanes takes
runs of two to eight consecutive edges: results of every instance equal its own solve's, with
instances without edges in between and runs that end in the middle of a row or an instance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def samples(p, n, share, rng):
    X = rng.standard_normal((n, p))
    k = int(round(share * p))  # so many variables share a factor: nearly all their pairs are kept
    X[:, :k] += 0.5 * rng.standard_normal((n, 1)) * rng.uniform(0.5, 1.5, k)
    return X


# 78k to 156k edges make runs of two, 312k and more runs of eight
@pytest.mark.parametrize("sizes", [[(420, 1.0), (30, 0.0), (2, 1.0), (301, 0.5)],
                                   [(1, 1.0), (505, 0.9), (33, 0.0), (640, 1.0), (511, 0.4)],
                                   [(700, 1.0), (31, 0.3), (720, 0.8)]])
@pytest.mark.parametrize("precision", ["f64", "split"])
def test_runs_equal_single_solves(cuda, sizes, precision):
    from gpucsl_gb300 import engine
    from gpucsl_gb300.batch import GaussianBatch

    torch = cuda
    rng = np.random.default_rng(len(sizes))
    n, alpha, maxl = 900, 0.01, 1
    Xs = [torch.from_numpy(samples(p, n, share, rng)).cuda() for p, share in sizes]
    b = GaussianBatch([p for p, _ in sizes], [n] * len(sizes), alpha, maxl, precision)
    b.bind_samples(Xs)
    res = b.run()
    for k, (p, _) in enumerate(sizes):
        assert res[k].status == 0
        G, sep, pmax = b.to_host(k)
        if p == 1:
            continue
        s = engine.GaussianSolver(p, maxl)
        one = s.run(engine.correlation(Xs[k]), n, engine.gaussian_thresholds(n, alpha))
        G1, sep1, pmax1 = s.to_host()
        assert np.array_equal(G, G1)
        assert np.array_equal(sep, sep1)
        if precision == "f64":
            assert np.array_equal(pmax, pmax1)
            assert res[k].tests == one.tests
