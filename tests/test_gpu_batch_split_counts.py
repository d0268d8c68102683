"""Split-precision batches with runs of consecutive edges: test counts of every instance equal its
own solve's and every kept pair has its p-value, within the FP32 error of the test statistic."""
import numpy as np
import pytest

from test_gpu_batch_runs import samples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(420, 1.0), (30, 0.0), (2, 1.0), (301, 0.5)], [(700, 1.0), (31, 0.3), (720, 0.8)]])
def test_counts_and_pmax(cuda, sizes):
    from gpucsl_gb300 import engine
    from gpucsl_gb300.batch import GaussianBatch

    torch = cuda
    rng = np.random.default_rng(len(sizes))
    n, alpha = 900, 0.01
    Xs = [torch.from_numpy(samples(p, n, share, rng)).cuda() for p, share in sizes]
    b = GaussianBatch([p for p, _ in sizes], [n] * len(sizes), alpha, 1, "split")
    b.bind_samples(Xs)
    res = b.run()
    for k, (p, _) in enumerate(sizes):
        pmax = b.to_host(k)[2]
        s = engine.GaussianSolver(p, 1)
        one = s.run(engine.correlation(Xs[k]), n, engine.gaussian_thresholds(n, alpha))
        pmax1 = s.to_host()[2]
        assert res[k].tests == one.tests
        assert ((pmax == -1) == (pmax1 == -1)).all()
        assert (np.abs(pmax - pmax1) <= 1e-4).all()
