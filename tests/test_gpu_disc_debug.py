"""The bounds-checked build on the bit-plane kernels: complete graphs whose level 1 has many tasks of
several neighbour groups, ragged last passes and mixed cardinalities; no check fires, and the results
are the release build's bit for bit, in permuted work orders too."""
import numpy as np
import pytest

from test_gpu_disc_bits import dependent_codes
from test_gpu_debug import disc_solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,n,card", [(40, 700, 2), (37, 2500, 3), (40, 4100, 5), (66, 600, 9)])
def test_checked_bit_planes_agree(cuda, p, n, card):
    from gpucsl_gb300 import engine

    codes, dims = dependent_codes(p, n, card, 7 * p + n)
    base = disc_solve(codes, dims, n, 0.05, 1, debug=False)
    assert base[3].raw["tests"][1] > 4000
    for seed in (0, 11):
        with engine.debug_work_order(seed):
            got = disc_solve(codes, dims, n, 0.05, 1, debug=True)
        assert got[3].raw["status"] == 0 and got[3].raw["debug_site"] == 0, (got[3].raw["status"], got[3].raw["debug_site"])
        for a, b in zip(got[:3], base[:3]):
            assert np.array_equal(a, b), seed
