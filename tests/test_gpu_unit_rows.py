"""GPU parity of the lattice decode's final pass where it copies units in rows
of a block each: with each block size (32, 16, 8, 4 units by the bits per
symbol), streams a few units short of, at and beyond a warp's 32 blocks, with
set bits in the memory behind the stream.  Integer work: the tolerance is
zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lam,block,bits", [(0.05, 32, 6.0), (0.2, 16, 3.83), (0.6, 8, 2.3),
                                            (2.0, 4, 0.9)])
def test_row_edges(mg, oracle_lib, lam, block, bits):
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    O = oracle_lib
    edge = 32 * block
    for units in (1, 3, block - 1, edge - 3, edge - 1, edge, edge + 1, edge + 2, edge + 4,
                  edge + 5, 2 * edge + block + 5):
        sym = O.gen_symbols(units, lam, max(int(units * 32 / bits), 2))
        st = O.encode(sym, 1024)
        units_dev = torch.full((st.n_units + 64,), -1, dtype=torch.int32, device="cuda")
        units_dev[: st.n_units] = torch.from_numpy(
            np.ascontiguousarray(st.units[: st.n_units]).view(np.int32))
        table = torch.from_numpy(np.ascontiguousarray(st.table).view(np.int32)).to("cuda")
        plan = mg.plan(st.n_units, st.n, 1024)
        aux = torch.full((mg.aux_size(st.n_units, plan),), 0x5A, dtype=torch.uint8, device="cuda")
        out = torch.full((st.n + 32,), 0xCD, dtype=torch.uint8, device="cuda")
        decode_async(units_dev, st.n_units, out, st.n, table, st.L, st.first_state,
                     st.first_bit, aux, plan)
        assert aux_status(aux) & ~mg.DEV_DEGENERATE == 0
        b = out.cpu().numpy()
        assert np.array_equal(b[: st.n], sym[::-1]), units
        assert (b[st.n:] == 0xCD).all()
