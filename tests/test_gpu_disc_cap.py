"""The cap on resident blocks holds for every long kernel of a discrete solve (launch shapes as the
profiler records them), and results do not depend on it."""
import json

import numpy as np
import pytest

from test_gpu_disc_bits import dependent_codes

pytestmark = pytest.mark.gpu

# the kernels of levels 0 and 1; grids in threads
STRIDED = ("disc_planes_kernel", "disc_pair_counts_kernel", "disc_level0_kernel", "disc_bits_level1_kernel")


def solve(torch, codes, dims, cap, tmp_path):
    from torch.profiler import ProfilerActivity, profile
    from gpucsl_gb300 import _lib, engine

    s = engine.DiscreteSolver(codes.shape[0], codes.shape[1], 2, int(dims.max()))
    s.load(codes, dims)
    _lib.check(_lib.lib().gcsl_set_blocks_per_sm_cap(cap), "gcsl_set_blocks_per_sm_cap")
    try:
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            s.run(0.05)
            torch.cuda.synchronize()
    finally:
        _lib.lib().gcsl_set_blocks_per_sm_cap(0)
    path = tmp_path / f"trace{cap}.json"
    prof.export_chrome_trace(str(path))
    grids = {}
    for e in json.loads(path.read_text())["traceEvents"]:
        if e.get("cat") == "kernel":
            name = next((k for k in STRIDED if k in e["name"]), None)
            if name:
                blocks, threads = int(np.prod(e["args"]["grid"])), int(np.prod(e["args"]["block"]))
                grids[name] = blocks * threads
    return s.to_host(), grids


@pytest.mark.parametrize("cap", [1, 2])
def test_cap_bounds_the_grids(cuda, tmp_path, cap):
    codes, dims = dependent_codes(150, 30000, 5, 9)
    solve(cuda, codes, dims, 0, tmp_path)  # the profiler may miss launches while it starts
    free, grids0 = solve(cuda, codes, dims, 0, tmp_path)
    held, grids = solve(cuda, codes, dims, cap, tmp_path)
    for a, b in zip(free, held):
        assert np.array_equal(a, b)
    if set(grids) != set(STRIDED) or set(grids0) != set(STRIDED):
        pytest.skip("no kernel records from the profiler")
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    for name in STRIDED:
        assert grids[name] <= sms * cap * 256, (name, grids[name])
        assert grids0[name] > sms * cap * 256 or cap > 1, name  # the shape needs the cap
