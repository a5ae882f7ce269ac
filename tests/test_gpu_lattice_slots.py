"""GPU parity of the lattice decode on tables of a few states, where a block
has four slots and narrow warps look at more than that ahead: every slot of a
block gets taken.  Integer work: the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [2, 4, 8, 16, 32])
@pytest.mark.parametrize("n", [700, 20_000, 300_000])
def test_few_slots(mg, oracle_lib, L, n):
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    rng = np.random.default_rng(L * 7 + n)
    sym = rng.integers(0, max(L // 2, 2), n).astype(np.uint8)
    st = oracle_lib.encode(sym, L)
    units = torch.from_numpy(np.ascontiguousarray(st.units).view(np.int32)).to("cuda")
    table = torch.from_numpy(np.ascontiguousarray(st.table).view(np.int32)).to("cuda")
    plan = mg.plan(st.n_units, n, L)
    aux = torch.full((mg.aux_size(st.n_units, plan),), 0x5A, dtype=torch.uint8, device="cuda")
    out = torch.full((n + 32,), 0xCD, dtype=torch.uint8, device="cuda")
    for _ in range(3):
        decode_async(units, st.n_units, out, n, table, L, st.first_state, st.first_bit, aux, plan)
        assert aux_status(aux) & ~mg.DEV_DEGENERATE == 0
        b = out.cpu().numpy()
        assert np.array_equal(b[:n], sym[::-1])
        assert (b[n:] == 0xCD).all()
