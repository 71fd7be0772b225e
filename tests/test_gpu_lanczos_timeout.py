"""The plain Lanczos driver when a barrier of its fused step gives up waiting."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flush", [False, True])
def test_error_word_is_seen_and_nothing_stays_in_flight(flush):
    """ctn_selftest_lanczos_timeout: barriers that wait for one arrival more than the grid has.  The error word
    is the integer 1, which a thread that flushes denormals must see too; the driver comes back with the
    stream idle (the self-test refuses otherwise) and the context stays usable."""
    from cytnx_b200 import _lib, workloads as W
    import cytnx_b200 as c

    lib = _lib.lib()
    torch.set_flush_denormal(flush)
    try:
        rc = lib.ctn_selftest_lanczos_timeout(1 << 12, _lib.stream_ptr())
    finally:
        torch.set_flush_denormal(False)
    assert rc == 4, (rc, lib.ctn_last_error())
    assert b"gave up waiting" in lib.ctn_last_error()
    psi, L, M1, M2, R = W.build_two_site(W.xxz_spec(16), W.xxz_mpo_values(), seed=1, device=0)
    e, _, it = c.TwoSiteHeff(L, M1, M2, R, psi).lanczos(psi, maxiter=4, cvgcrit=1e-300)
    assert it == 4 and e == e
