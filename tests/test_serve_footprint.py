"""Admission counts what the engine allocates (no GPU): the library's own sizes for the correlation
and the level loop, whatever they are, beside the request's tensors."""
import pytest

from gpucsl_gb300 import _lib, serve


class Sizes:
    """Library sizes of a device whose product cuts its K range into five splits."""

    @staticmethod
    def gcsl_corr_tc_workspace_bytes(n, p):
        pad = (p + 127) // 128 * 128
        return 14 * pad * ((n + 31) // 32 * 32) + 5 * 16 * pad * pad + 8 * p * ((n + 511) // 512) + 4096

    @staticmethod
    def gcsl_gauss_state_bytes(p):
        return 30 * p * p

    @staticmethod
    def gcsl_gauss_workspace_bytes(p, max_level):
        return 50 * p * p


@pytest.mark.parametrize("p,n", [(20, 1000), (211, 7919), (1999, 49999)])
def test_footprint_holds_what_a_request_allocates(monkeypatch, p, n):
    monkeypatch.setattr(_lib, "lib", lambda debug=False: Sizes)
    tensors = 4 * n * p + 8 * p * p + 2 * p * p + 8 * p * p + 4 * max(1024, 64 * p)
    allocated = tensors + Sizes.gcsl_corr_tc_workspace_bytes(n, p) + Sizes.gcsl_gauss_workspace_bytes(p, 3)
    assert serve.gaussian_footprint(p, n, 3) >= allocated
