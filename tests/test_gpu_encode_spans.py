"""Device ordinal encoding at the spans where its kernels change form (32, 64, 4096 values
from minimum to maximum), around zero and the bitmap's end, at the edges of 64-row steps and
32-column strips.  Exact against the host encoder."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def table(n, p, span, low, rng):
    cols = []
    for j in range(p):
        s = span if j % 3 else min(span, 5)
        k = int(min(s, 255, rng.integers(2, 300)))
        vals = np.concatenate([[0, s - 1], rng.choice(s, size=k, replace=False)])[: k + 1] if s > 1 else np.zeros(1)
        vals = np.unique(vals)[:255]
        cols.append(low + rng.choice(vals, size=n))
    return np.stack(cols, axis=1)


@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.uint8, np.float64])
@pytest.mark.parametrize("span", [1, 2, 31, 32, 33, 63, 64, 65, 200, 4095, 4096])
def test_spans(cuda, dtype, span):
    from gpucsl_gb300 import engine

    rng = np.random.default_rng(span)
    if dtype == np.uint8 and span > 256:
        span = 256
    for n, p in [(1, 1), (63, 31), (64, 33), (65, 40), (1900, 70), (40001, 3)]:
        for low in [0] if dtype == np.uint8 else [0, -17, 4080, -2**31, 10**6 - 3]:
            data = table(n, p, span, low, rng).astype(dtype)
            codes, dims = engine.ordinal_encode(data)
            ld = n + 5  # columns off the 8-byte boundary
            cdev, ddev = engine.ordinal_encode_device(cuda.from_numpy(data).cuda(), ld=ld)
            assert np.array_equal(ddev.cpu().numpy(), dims)
            assert np.array_equal(cdev.cpu().numpy()[:, :n], codes)
            assert not cdev.cpu().numpy()[:, n:].any()


def test_float_integers(cuda):
    """Whole FP64 values of every exponent pass, the nearest fractions do not."""
    from gpucsl_gb300 import _lib, engine

    for e in list(range(0, 63)):
        v = 2.0 ** e
        data = np.array([[v, -v], [v + 1.0 if e < 53 else v, -v], [v, -0.0 if e == 0 else -v]])
        codes, dims = engine.ordinal_encode(data)
        cdev, ddev = engine.ordinal_encode_device(cuda.from_numpy(data).cuda())
        assert np.array_equal(ddev.cpu().numpy(), dims) and np.array_equal(cdev.cpu().numpy()[:, :3], codes)
        if e < 52:
            for bad in (np.nextafter(v, 0.0), np.nextafter(v, np.inf), -np.nextafter(v, np.inf)):
                data[1, 0] = bad
                with pytest.raises(_lib.GcslError):
                    engine.ordinal_encode_device(cuda.from_numpy(data).cuda())
    for bad in (np.nan, np.inf, -np.inf, 5e-324, 0.5, -0.25, 2.0 ** 63):
        with pytest.raises(_lib.GcslError):
            engine.ordinal_encode_device(cuda.from_numpy(np.array([[1.0], [bad]])).cuda())
