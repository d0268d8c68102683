"""The C entry point of the discrete solve with a dense separation-set buffer, against the C
oracle: a cardinality above the announced maximum must leave nothing of its first attempt behind,
and a workspace without room for the optional buffers is enough."""
import ctypes as ct

import numpy as np
import pytest

from test_gpu_discrete import assert_parity, oracle_discrete

pytestmark = pytest.mark.gpu


def run_entry(torch, codes, dims, alpha, L, max_dim, ws_bytes=None):
    """(status, (G, dense sepsets, pmax, stats)) of one call."""
    from gpucsl_gb300 import _lib
    from gpucsl_gb300.engine import SolveStats

    p, n = codes.shape
    ld = (n + 15) // 16 * 16
    data = torch.zeros((p, ld), dtype=torch.uint8, device="cuda")
    data[:, :n].copy_(torch.from_numpy(codes))
    dd = torch.from_numpy(dims).cuda()
    G = torch.empty((p, p), dtype=torch.int16, device="cuda")
    pmax = torch.empty((p, p), dtype=torch.float64, device="cuda")
    sep = torch.full((p, p, L), -1, dtype=torch.int32, device="cuda")
    lib = _lib.lib()
    size = int(lib.gcsl_disc_workspace_bytes(p, n, L, max_dim)) if ws_bytes is None else ws_bytes
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    st = _lib.GcslStats()
    rc = lib.gcsl_disc_skeleton(data.data_ptr(), ld, n, p, dd.data_ptr(), max_dim, alpha, L, G.data_ptr(),
                                sep.data_ptr(), None, 0, pmax.data_ptr(), ct.byref(st), ws.data_ptr(), size,
                                _lib.stream_ptr())
    torch.cuda.synchronize()
    return rc, (G.cpu().numpy().view(np.uint16), sep.cpu().numpy(), pmax.cpu().numpy(), SolveStats(st.as_dict()))


def test_sets_of_a_repeated_solve(cuda):
    """w = 0, 1, 2 has the independent causes a, b and is announced as binary.  With its last two
    values merged a - w is removed given b; with all three it is kept (b - w is in both)."""
    rng = np.random.default_rng(3)
    n = 800
    a, b = rng.integers(0, 2, n), rng.integers(0, 2, n)
    w = (rng.random(n) < 0.35 + 0.3 * b + 0.07 * a).astype(int)
    w = np.where(w == 1, 1 + (rng.random(n) < 0.2 + 0.6 * a), 0)
    # constant columns beside them: enough variables for the bit planes
    codes = np.concatenate([np.stack([a, b, w]), np.zeros((37, n), np.int64)]).astype(np.uint8)
    merged = oracle_discrete(np.minimum(codes, 1), np.minimum(codes.max(1) + 1, 2).astype(np.uint8), 0.05, 1)
    assert merged[0][0, 2] == 0 and merged[1][0, 2, 0] == 1  # what the first attempt finds
    dims = codes.max(1).astype(np.uint8) + 1
    rc, got = run_entry(cuda, codes, dims, 0.05, 1, 2)
    assert rc == 0
    assert_parity(got, oracle_discrete(codes, dims, 0.05, 1))


def test_workspace_of_the_general_path(cuda):
    """The bit planes are optional: a workspace that holds the other buffers is accepted."""
    from test_gpu_disc_bits import dependent_codes
    from gpucsl_gb300 import _lib

    codes, dims = dependent_codes(40, 1500, 4, 77)
    small = int(_lib.lib().gcsl_disc_workspace_bytes(40, 1500, 2, 1))  # no planes for constant columns
    assert small < int(_lib.lib().gcsl_disc_workspace_bytes(40, 1500, 2, 4))
    ref = oracle_discrete(codes, dims, 0.05, 2)
    rc, got = run_entry(cuda, codes, dims, 0.05, 2, 4, small)
    assert rc == 0
    assert_parity(got, ref)
    assert run_entry(cuda, codes, dims, 0.05, 2, 4, small - 1)[0] == _lib.GCSL_ERR_WORKSPACE
