"""The encoders' limits, checked before any device call: a fragment whose
windows do not fit one warp's shared memory is refused, however many come."""
import ctypes

import pytest

from rotormap._lib import R2M_EINVAL, lib

# longest fragment that is accepted: histogram + 2.5 bytes a base <= 200 KiB less 32 bytes
LIMITS = [(5, 1, 5), (8, 4, 4), (6, 3, 2), (8, 8, 3)]


def one_warp_bytes(k, s, m, c):
    nw, words = k - s + 1, (k + 15) // 16
    return (2 * m * 4 ** c + 31) // 32 * 128 + (nw + 7) // 8 * 16 + (words + 5) // 4 * 32 + 32


@pytest.mark.parametrize("s,m,c", LIMITS)
@pytest.mark.parametrize("n", [1, 100, 10_000])
@pytest.mark.parametrize("kind", [0, 2, 3])
def test_overlong_fragments_are_refused(s, m, c, n, kind):
    k = next(k for k in range(90_000, s, -1) if one_warp_bytes(k, s, m, c) <= 200 * 1024) + 1
    dummy = (ctypes.c_uint8 * 64)()
    p = (ctypes.addressof(dummy) + 15) // 16 * 16
    for bases in (k, 100_000, 200_000):
        rc = lib().r2m_encode_frag_real_batch(p, kind, p, p, p, n, bases, s, m, c, 0, None)
        assert rc == R2M_EINVAL and "does not fit" in lib().r2m_last_error().decode()
        rc = lib().r2m_encode_ref_windows(p, kind, p, p, p, p, n, 64, bases, s, m, c, 0, None)
        assert rc == R2M_EINVAL and "does not fit" in lib().r2m_last_error().decode()
