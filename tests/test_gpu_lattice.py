"""GPU parity of the lattice decode (the planner's own plan without symbol
capture): streams at the edges of its blocks (4, 8, 16, 32 units), scan tiles
(1024 blocks), slot counts (4, 8, 12) and warp widths, in both output orders
and at odd output addresses, and data whose trajectories meet later than the
planner expects, so that the true path runs out of slots and is repaired.
Integer work: the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LATTICE = 0x80
REPAIRED = 256 + 5 * 4   # byte of the workspace counter of repaired blocks


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).to("cuda")


def _decode(mg, st, n_out=None, shift=0, source_order=False):
    """One asynchronous decode with the planner's plan; the output and
    whether the path was repaired."""
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    n_out = st.n if n_out is None else n_out
    plan = mg.plan(st.n_units, n_out, st.L)
    assert plan["flags"] & LATTICE
    if source_order:
        plan["flags"] |= mg.DECODE_SOURCE_ORDER
    aux = torch.full((mg.aux_size(st.n_units, plan),), 0x5A, dtype=torch.uint8, device="cuda")
    big = torch.full((n_out + 64,), 0xCD, dtype=torch.uint8, device="cuda")
    decode_async(_dev(st.units), st.n_units, big[shift:], n_out, _dev(st.table), st.L,
                 st.first_state, st.first_bit, aux, plan)
    status = aux_status(aux)
    assert status & ~mg.DEV_DEGENERATE == 0, hex(status)
    repaired = bool(aux[REPAIRED: REPAIRED + 4].cpu().numpy().any())
    b = big.cpu().numpy()
    assert (b[:shift] == 0xCD).all() and (b[shift + n_out:] == 0xCD).all()
    return b[shift: shift + n_out], repaired


@pytest.mark.parametrize("L,lam", [(2, 2.0), (64, 1.0), (256, 0.05), (1024, 0.005), (1024, 0.2),
                                   (2048, 1.0), (4096, 2.0), (8192, 0.05)])
def test_block_edges(mg, oracle_lib, L, lam):
    """Unit counts around multiples of 4, 8 and 16 and tiny streams."""
    O = oracle_lib
    for n in (1, 2, 5, 17, 63, 64, 65, 130, 511, 1021, 4099):
        sym = O.gen_symbols(n * 3 + L, lam, n)
        if L < 256:
            sym = (sym % min(L, 4)).astype(np.uint8)
        st = O.encode(sym, L)
        want = sym[::-1]
        for shift, so in ((0, False), (3, False), (0, True), (5, True)):
            got, _ = _decode(mg, st, shift=shift, source_order=so)
            assert np.array_equal(got[::-1] if so else got, want), (n, shift, so)


@pytest.mark.parametrize("tiles", [1, 2, 33])
@pytest.mark.parametrize("d", [-1, 0, 1])
@pytest.mark.parametrize("lam,bits,block", [(0.05, 6.0, 32), (0.2, 3.83, 16)])
def test_scan_tile_edges(mg, oracle_lib, tiles, d, lam, bits, block):
    """Streams of about 1024 blocks per scan tile, one unit around the edge,
    and a look-back longer than 32 tiles."""
    O = oracle_lib
    n_units = tiles * 1024 * block + d
    st = O.make_stream(seed=tiles * 10 + d, lam=lam, n=int(n_units * 32 / bits), L=1024)
    got, _ = _decode(mg, st)
    assert np.array_equal(got[::-1], st.symbols)


@pytest.mark.parametrize("lam,L,n", [(0.005, 1024, 24_000_000), (0.05, 1024, 18_000_001),
                                     (0.2, 4096, 16_000_003), (2.0, 1024, 30_000_000)])
def test_long_streams(mg, lam, L, n):
    """The larger spacings and the slot counts they go with (4, 8, 12)."""
    from multians_gb300 import host
    st = host.make_stream(77, lam, n, L)
    got, _ = _decode(mg, st, shift=1)
    assert np.array_equal(got[::-1], st.symbols)


def test_short_output(mg, oracle_lib):
    O = oracle_lib
    st = O.make_stream(seed=9, lam=0.05, n=50_000, L=1024)
    want = st.symbols[::-1]
    for short in (1, 4097, 49_963):
        for so in (False, True):
            got, _ = _decode(mg, st, n_out=short, source_order=so)
            assert np.array_equal(got[::-1] if so else got, want[:short])


@pytest.mark.parametrize("K,L,n", [(2, 1024, 400_000), (8, 1024, 60_000), (8, 1024, 3_000_000),
                                   (8, 4096, 2_000_000), (32, 1024, 3_000_000)])
def test_slow_meeting_data(mg, oracle_lib, K, L, n):
    """K equally frequent symbols with a rare other one: code lengths are
    almost all the same, trajectories at different bit phases run side by
    side for long."""
    O = oracle_lib
    rng = np.random.default_rng(K * 1000 + L)
    sym = rng.integers(0, K, n).astype(np.uint8)
    sym[rng.random(n) < 0.002] = 200
    st = O.encode(sym, L)
    got, _ = _decode(mg, st)
    assert np.array_equal(got[::-1], sym)


def test_repaired_path(mg, oracle_lib):
    """The same kind of data, where the true path does run out of slots: on
    streams short enough for any number of repairs."""
    O = oracle_lib
    ran = 0
    for seed in range(12):
        rng = np.random.default_rng(seed)
        n = 600_000
        sym = rng.integers(0, 2, n).astype(np.uint8)
        sym[rng.random(n) < 0.0002 * (seed % 2)] = 200
        st = O.encode(sym, 1024)
        assert st.n_units <= 32768
        got, repaired = _decode(mg, st)
        assert np.array_equal(got[::-1], sym), seed
        ran += repaired
    assert ran > 0
