"""Sizes the encoder takes: past the 34 GB at which a
block's slots need more than 32 bits to count.  No device memory is touched:
the calls name a workspace that is too small."""
import ctypes

import pytest


@pytest.mark.parametrize("n", [1, 64 << 20, (1 << 28) * 128, (1 << 28) * 128 + 1, 40_000_000_001,
                               (1 << 31) * 64 - 64])
@pytest.mark.parametrize("L", [1024, 4096])
def test_large_inputs_are_taken(mg, n, L):
    from multians_gb300 import encode
    lib = encode._sig()
    cap = lib.mans_encode_max_units(n, L)
    at = ctypes.c_void_p(0x100000)   # never dereferenced
    rc = lib.mans_encode(at, n, at, L, at, cap, at, 0, 0, None)
    assert rc == mg.Status.ERR_AUX_SMALL
    # 16 slots of two words, an entry and a share of a tile per block of 128 bytes at most
    assert lib.mans_encode_aux_size(n, 0) <= (-(-n // 64)) * 138 + 4096
