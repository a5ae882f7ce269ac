"""GPU parity of the lattice decode at the exact edges of its blocks, of the 32
blocks a warp decodes in the final pass, and of its scan tiles: streams of
exactly the wanted number of units, and the number of blocks the decode
reports tells the block size.  Set bits in the memory behind the stream.
Integer work: the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# lambda, L, units per block at the sizes below
SIZES = [(0.05, 4096, 32), (0.05, 1024, 16), (0.6, 1024, 8), (2.0, 1024, 4)]


def stream_of_units(O, lam, L, target):
    """A stream of exactly `target` units: a prefix of one generated run,
    encoded with the table of the whole run, so that its length grows with the
    prefix."""
    bits = {0.05: 6.0, 0.6: 2.3, 2.0: 0.67}[lam]
    pool = O.gen_symbols(target, lam, int(target * 32 / bits * 1.2) + 2000)
    enc, dec, ml, _ = O.build_tables(pool, L, O.TABLE_SEED)

    def encode(n):
        buf = O._padded(pool[:n])
        units = np.zeros(O.lib().mo_max_units(ml, n) + 4, dtype=np.uint32)
        fb, fs = np.zeros(1, dtype=np.uint32), np.zeros(1, dtype=np.uint32)
        nu = O.lib().mo_encode(O._ptr(enc, O._u32p), L, ml, O._ptr(buf, O._u8p), n,
                               O._ptr(units, O._u32p), units.size, O._ptr(fb, O._u32p),
                               O._ptr(fs, O._u32p))
        return O.Stream(pool[:n].copy(), units[: nu + 4].copy(), int(nu), int(fb[0]), int(fs[0]),
                        dec, L)

    lo, hi, n = 0, pool.size + 1, pool.size
    while True:
        st = encode(n)
        if st.n_units == target:
            return st
        lo, hi = (n, hi) if st.n_units < target else (lo, n)
        assert hi - lo > 1, f"no prefix of {target} units"
        guess = n + round((target - st.n_units) * n / st.n_units)
        n = guess if lo < guess < hi else (lo + hi) // 2


def check(mg, st, block, source_order):
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    units = torch.full((st.n_units + 64,), -1, dtype=torch.int32, device="cuda")
    units[: st.n_units] = torch.from_numpy(np.ascontiguousarray(st.units[: st.n_units]).view(np.int32))
    table = torch.from_numpy(np.ascontiguousarray(st.table).view(np.int32)).to("cuda")
    cfg = {"flags": mg.DECODE_SOURCE_ORDER if source_order else 0}
    aux = torch.full((mg.aux_size(st.n_units, mg.plan(st.n_units, st.n, st.L, cfg)),), 0x5A,
                     dtype=torch.uint8, device="cuda")
    out = torch.full((st.n + 32,), 0xCD, dtype=torch.uint8, device="cuda")
    decode_async(units, st.n_units, out, st.n, table, st.L, st.first_state, st.first_bit, aux, cfg)
    assert aux_status(aux) == 0
    stats = mg._lib.sync_stats(aux.data_ptr(), aux.numel(), st.n_units, st.n, st.L, cfg)
    assert stats["blocks"] == st.n_units // block + 1
    b = out.cpu().numpy()
    want = st.symbols if source_order else st.symbols[::-1]
    assert np.array_equal(b[: st.n], want), st.n_units
    assert (b[st.n:] == 0xCD).all()


@pytest.mark.parametrize("lam,L,block", SIZES)
def test_rows(mg, oracle_lib, lam, L, block):
    """Around a warp's 32 blocks, and around a block's end inside the next."""
    edge = 32 * block
    for target in [edge + d for d in (-4, -3, -1, 0, 1, 2, 3, 4, 5)] + \
            [edge + block + d for d in (-1, 0, 1)] + [2 * edge, 2 * edge + block + 3]:
        st = stream_of_units(oracle_lib, lam, L, target)
        for so in (False, True):
            check(mg, st, block, so)


@pytest.mark.parametrize("tiles", [1, 2, 33])
@pytest.mark.parametrize("lam,L,block", SIZES[:2])
def test_tiles(mg, oracle_lib, lam, L, block, tiles):
    """A block short of a whole tile, a whole tile, and one block in the next:
    its last unit, and none at all."""
    whole = 1024 * tiles
    for target, blocks in ((block * (whole - 1) - 1, whole - 1), (block * whole - 1, whole),
                           (block * (whole - 1), whole), (block * whole, whole + 1),
                           (block * whole + 1, whole + 1)):
        st = stream_of_units(oracle_lib, lam, L, target)
        assert st.n_units // block + 1 == blocks
        check(mg, st, block, bool(target & 1))
