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


@pytest.mark.parametrize("n,lam,L", [(40_000, 0.3, 4096), (146_000, 0.33, 4096),
                                     (219_000, 1.95, 4096), (1_000_000, 1.0, 2048),
                                     (5_000_001, 0.5, 4096)])
def test_many_slots(mg, oracle_lib, n, lam, L):
    """Streams that get 32 slots a block: one and several scan tiles."""
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    sym = oracle_lib.gen_symbols(n, lam, n)
    st = oracle_lib.encode(sym, L)
    units = torch.from_numpy(np.ascontiguousarray(st.units).view(np.int32)).to("cuda")
    table = torch.from_numpy(np.ascontiguousarray(st.table).view(np.int32)).to("cuda")
    for flags in (0, mg.DECODE_SOURCE_ORDER):
        plan = mg.plan(st.n_units, n, L, {"flags": flags})
        aux = torch.full((mg.aux_size(st.n_units, plan),), 0x5A, dtype=torch.uint8, device="cuda")
        out = torch.full((n + 32,), 0xCD, dtype=torch.uint8, device="cuda")
        decode_async(units, st.n_units, out, n, table, L, st.first_state, st.first_bit, aux, plan)
        assert aux_status(aux) == 0
        b = out.cpu().numpy()
        assert np.array_equal(b[:n], sym if flags else sym[::-1])
        assert (b[n:] == 0xCD).all()


def test_many_slots_in_batches(mg, oracle_lib):
    """The same next to streams with fewer slots, in batches that fill narrow
    and full warps."""
    import torch
    from multians_gb300 import batch
    for specs in ([(146_000, 0.33, 4096), (9_000, 0.1, 1024), (219_000, 1.95, 4096)],
                  [(5_000_000, 0.5, 4096), (3_000_000, 0.05, 1024)]):
        keep, descs, want = [], [], []
        for i, (n, lam, L) in enumerate(specs):
            sym = oracle_lib.gen_symbols(n + i, lam, n)
            st = oracle_lib.encode(sym, L)
            units = torch.from_numpy(np.ascontiguousarray(st.units).view(np.int32)).to("cuda")
            table = torch.from_numpy(np.ascontiguousarray(st.table).view(np.int32)).to("cuda")
            out = torch.full((n,), 0xCD, dtype=torch.uint8, device="cuda")
            keep.append((units, table, out))
            want.append(sym[::-1])
            descs.append(batch.desc(units, st.n_units, out, n, table, L, st.first_state, st.first_bit))
        batch.decode_batch(descs)
        torch.cuda.synchronize()
        for (_, _, out), w in zip(keep, want):
            assert np.array_equal(out.cpu().numpy(), w)
