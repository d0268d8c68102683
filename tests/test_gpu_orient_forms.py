"""Edge orientation in its two forms, one cooperative kernel (sparse skeletons) and separate
kernels (a sum of cubed degrees above 2^26), on random graphs and sets against the sequential
oracle: vertices at the edges of blocks, hubs, empty rows, dense graphs on both sides of the
line."""
import numpy as np
import pytest

from oracle import orient as oo

pytestmark = pytest.mark.gpu


def graph(p, prob, L, seed, hub=False, keep=0.97):
    rng = np.random.default_rng(seed)
    S = np.triu(rng.random((p, p)) < prob, 1)
    if hub:
        S[0, 1:] = rng.random(p - 1) < 0.8
    S = (S | S.T).astype(np.uint16)
    sep = np.full((p, p, max(L, 1)), -1, np.int32)
    for a, b in zip(*np.nonzero(np.triu(S == 0, 1))):
        common = np.nonzero(S[a] & S[b])[0]  # sets that leave most triples to the rules
        if common.size and common.size <= L and rng.random() < keep:
            sep[a, b, :common.size] = common
        elif L:
            sep[b, a, 0] = rng.integers(p)
    return S, sep


@pytest.mark.parametrize("p,prob,L,hub", [(1, 0.0, 1, False), (2, 1.0, 1, False), (7, 0.5, 4, False),
                                          (8, 0.4, 5, False), (33, 0.1, 6, False), (65, 0.05, 9, True),
                                          (150, 0.02, 6, False), (300, 0.01, 4, False), (70, 0.6, 40, False),
                                          (96, 0.85, 96, False), (120, 0.85, 120, False)])
def test_orientation_forms(cuda, p, prob, L, hub):
    from gpucsl_gb300.orient import orient_matrix

    for seed in range(3):
        S, sep = graph(p, prob, L, 100 * p + seed, hub, 0.97 if prob < 0.5 else 0.998)
        D, passes = orient_matrix(S, sep)
        ref, ref_passes = oo.orient(S, sep)
        assert np.array_equal(D, ref)
        assert passes == ref_passes
