"""DiscreteSolver refuses code and cardinality tensors that its kernels could not read as they are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_codes_and_dims_are_checked(cuda):
    from gpucsl_gb300 import engine

    torch = cuda
    p, n, ld = 7, 40, 48

    def codes(dtype=torch.uint8, device="cuda", shape=(p, ld)):
        return torch.zeros(shape, dtype=dtype, device=device)

    def dims(dtype=torch.uint8, device="cuda", count=p):
        return torch.full((count,), 2, dtype=dtype, device=device)

    for c, d in [(codes(torch.int16), dims()), (codes(device="cpu"), dims()), (codes(shape=(p, ld - 16)), dims()),
                 (codes(), dims(count=p - 1)), (codes(), dims(torch.int32)), (codes(), dims(device="cpu")),
                 (codes(), dims(count=2 * p)[::2]), (None, dims(count=p - 1)), (codes(torch.int8), None)]:
        with pytest.raises(ValueError):
            engine.DiscreteSolver(p, n, 1, 2, codes=c, dims=d)
    c, d = codes(), dims()
    c[0, :n // 2] = 1
    c[1, :n // 2] = 1
    s = engine.DiscreteSolver(p, n, 1, 2, codes=c, dims=d)
    assert s.data is c and s.dims is d
    s.run(0.05)
    G, _, _ = s.to_host()
    want = np.zeros((p, p), np.uint16)
    want[0, 1] = want[1, 0] = 1
    assert (G == want).all()
