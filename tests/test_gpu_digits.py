"""The digit-split correlation at the ends of its exactness argument: columns whose every
sample has the largest magnitude (the shortest chunks between drains), columns of a single
outlier (the longest), and shapes at the edges of tiles, 64-sample windows and K splits.

Bound: I is rounded to 2^-49 of the column's range and pairs below 2^-49 are dropped, so an
entry of C is off by at most 4 * 2^-49 w, w = n / sum y^2 of its columns in units of the range
(1 .. 6 for most, up to 2.5 n for the outlier columns), plus the FP64 roundings of both sides
(1e-13 allowed).  One lost unit in the leading digit group is at least 2^-18 w / n."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def columns(n, p, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, p))
    kind = np.arange(p) % 5
    for j in range(p):
        if kind[j] == 1:
            X[:, j] = rng.choice([-1.0, 1.0], n)  # every |y| near the top of the range
        elif kind[j] == 2:
            X[:, j] = np.where(rng.random(n) < 0.5, -0.999999, 1.0) * 2.0 ** (j % 41 - 20)
        elif kind[j] == 3:
            X[:, j] *= 1e-6
            X[rng.integers(0, n), j] = 5.0
        elif kind[j] == 4:
            X[:, j] = rng.integers(0, 7, n) + 1000.0
    return X


@pytest.mark.parametrize("n,p", [(2, 3), (31, 5), (64, 20), (65, 64), (513, 65), (2100, 129), (2049, 40), (9000, 257)])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_extreme_columns(cuda, n, p, dtype):
    from gpucsl_gb300 import engine

    X = columns(n, p, n + p).astype(dtype)
    X64 = X.astype(np.float64)
    ok = X64.std(0) > 0
    ref = np.corrcoef(X64, rowvar=False)
    C = engine.correlation(cuda.from_numpy(X).cuda()).cpu().numpy()
    both = ok[:, None] & ok[None, :]
    assert np.array_equal(C, C.T)
    y = X64 - X64.mean(0)
    top = np.abs(y).max(0)
    w = n / np.maximum((np.ldexp(y, -np.frexp(np.where(top > 0, top, 1.0))[1]) ** 2).sum(0), 1e-300)
    tol = 1e-13 + 4 * 2.0 ** -49 * np.maximum(w[:, None], w[None, :])
    assert (np.abs(C - ref) <= tol)[both].all()


def test_batch_equals_single(cuda):
    """Batched jobs and single ones, whose K splits differ, give the same bits."""
    from gpucsl_gb300 import engine
    from gpucsl_gb300.batch import GaussianBatch

    shapes = [(40, 700), (129, 2049), (65, 5000), (300, 1111)]
    Xs = [cuda.from_numpy(columns(n, p, 7 * p)).cuda() for p, n in shapes]
    b = GaussianBatch([s[0] for s in shapes], [s[1] for s in shapes], 0.01, 1, "f64")
    b.bind_samples(Xs)
    b.run()
    for k, X in enumerate(Xs):
        assert cuda.equal(b.C[k], engine.correlation(X))


@pytest.mark.parametrize("n,p", [(9, 5), (64, 33), (577, 65), (1531, 40)])
def test_floats_widen_exactly(cuda, n, p):
    """FP32 samples with zeros, subnormals and the largest finite values give the bits of the
    same samples held in FP64."""
    from gpucsl_gb300 import engine

    rng = np.random.default_rng(n + p)
    X = (rng.standard_normal((n, p)) * 10.0 ** rng.integers(-30, 30, p)).astype(np.float32)
    odd = np.array([0.0, -0.0, 1e-45, -1e-45, 1.1e-38, -1.1e-38, 1.1754944e-38, 3.4e38, -3.4e38], np.float32)
    hit = rng.random((n, p)) < 0.05
    X[hit] = rng.choice(odd, int(hit.sum()))
    X[:, 0] = (rng.integers(-3, 4, n) * np.float32(1e-45)).astype(np.float32)  # subnormal throughout
    X[0, 0] = np.float32(5e-45)
    x32 = cuda.from_numpy(X).cuda()
    assert cuda.equal(engine.correlation(x32), engine.correlation(cuda.from_numpy(X.astype(np.float64)).cuda()))
