"""GPU encoder parity at the edges of its blocks (64 and 128 bytes), groups of
32 blocks and scan tiles (1024 blocks), at the smallest tables, where byte 0
has a single state, and on data whose encodes meet late or never, so that the
true path is repaired or the encode is planned again with wider spacing.  The
units equal the host encoder's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(mg, O, sym, L, chunk=0):
    from multians_gb300 import encode
    st = O.encode(sym, L)
    units, n_units, fb, fs, dec = encode.encode(sym, L, chunk=chunk)
    assert np.array_equal(dec, st.table)
    assert (n_units, fb, fs) == (st.n_units, st.first_bit, st.first_state)
    got = units.cpu().numpy().view(np.uint32)
    assert np.array_equal(got, st.units), np.nonzero(got != st.units)[0][:10]


@pytest.mark.parametrize("L", [2, 16, 256, 1024, 4096, 8192])
def test_block_and_group_edges(mg, oracle_lib, L):
    O = oracle_lib
    for n in (1, 63, 64, 65, 127, 128, 129, 2047, 2048, 2049, 4095, 4096, 4097):
        sym = O.gen_symbols(n + L, 0.3 if L < 256 else 0.02, n)
        if L < 256:
            sym = (sym % L).astype(np.uint8)
        _check(mg, O, sym, L)


@pytest.mark.parametrize("n", [65_535, 65_537, 131_071, 131_073, (1 << 20) + 1])
def test_tile_edges(mg, oracle_lib, n):
    for L in (1024, 2048):
        _check(mg, oracle_lib, oracle_lib.gen_symbols(n, 0.2, n), L)


def test_every_symbol_has_one_state(mg, oracle_lib):
    """L = 256 with all byte values: every code is eight bits, byte 0's first
    slot is slot 0."""
    rng = np.random.default_rng(4)
    for n in (256, 999, 50_000):
        sym = np.concatenate([np.arange(256), rng.integers(0, 256, n)]).astype(np.uint8)
        _check(mg, oracle_lib, sym, 256)


@pytest.mark.parametrize("K,L,n", [(3, 1024, 200_000), (3, 4096, 3_000_000), (2, 8192, 500_000),
                                   (8, 1024, 16_000), (8, 1024, 1_000_000)])
def test_late_meeting_data(mg, oracle_lib, K, L, n):
    rng = np.random.default_rng(K + L)
    _check(mg, oracle_lib, rng.integers(0, K, n).astype(np.uint8), L)


@pytest.mark.parametrize("chunk", [64, 1000, 1 << 20])
def test_spacing_hints(mg, oracle_lib, chunk):
    _check(mg, oracle_lib, oracle_lib.gen_symbols(chunk, 0.05, 150_001), 1024, chunk=chunk)
