"""The CTAs of the one-launch Gram-Schmidt step (host arithmetic of the library): all of
them wait on one another, so there are never more than the device has SMs."""
import pytest


@pytest.mark.parametrize("sms", [1, 7, 100, 148, 152, 160])
def test_fused_step_fits_the_device(sms):
    from pytreenet_gb300 import _lib
    lib = _lib.load()
    most = min(sms, 152)
    for n in (1, 127, 128, 129, 4394, 19456, 131072, 12800 * most, 12800 * most + 1, 1 << 20, 1900000, 1 << 25):
        g = int(lib.ptn_krylov_fused_ctas(n, sms))
        assert 0 <= g <= most
        assert (g == 0) == (n > 12800 * most)           # w in 200 KB of shared memory a CTA
        if g:
            assert -(-n // g) <= 12800
            # mailboxes of three exchanges of 2 * 16 + 1 values, 16 bytes each, as partial's entries
            assert 3 * 33 * g <= int(lib.ptn_krylov_partials(n))
    assert int(lib.ptn_krylov_fused_ctas(0, sms)) == 0 and int(lib.ptn_krylov_fused_ctas(10, 0)) == 0
