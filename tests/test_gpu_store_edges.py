"""The final passes' store of a warp's output range where the range ends
within the first 16-byte line of an unaligned output: in source order the
stream's last blocks, a handful of symbols, land at the start of the
buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).to("cuda")


@pytest.mark.parametrize("cfg", [{"block_units": 4, "region_blocks": 9, "walk_slots": 4},
                                 {"block_units": 16, "region_blocks": 9, "walk_slots": 4}])
def test_short_last_group_at_unaligned_output(mg, oracle_lib, cfg):
    import torch
    O = oracle_lib
    # these streams are 1024 .. 1026 units long: the last group of 32 blocks
    # (128 or 512 units) holds at most two units
    for n in (3808, 3815, 3818, 3820, 3821, 3824, 3827, 3837, 3840):
        st = O.make_stream(seed=n, lam=0.005, n=n, L=1024)
        assert st.n_units % (32 * cfg["block_units"]) <= 2
        for shift in (1, 3, 13):
            big = torch.full((n + 64,), 0xCD, dtype=torch.uint8, device="cuda")
            mg.decode(_dev(st.units), st.n_units, n, _dev(st.table), st.first_state,
                      st.first_bit, L=st.L, out=big[shift: shift + n], cfg=cfg,
                      source_order=True)
            b = big.cpu().numpy()
            assert np.array_equal(b[shift: shift + n], st.symbols), (n, shift)
            assert (b[:shift] == 0xCD).all() and (b[shift + n:] == 0xCD).all()


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [50_001, 400_003])
def test_ranges_past_the_staging(mg, oracle_lib, n, shift):
    """Data of a few bits per block's dozens of symbols: a warp's output range
    does not fit its staging buffer, and lanes store words of their own
    between bytes at their ends."""
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    sym = oracle_lib.gen_symbols(n + shift, 5.0, n)
    st = oracle_lib.encode(sym, 1024)
    assert n / st.n_units > 110      # 4 units a block, 32 blocks, 16 KB
    units, table = _dev(st.units), _dev(st.table)
    for flags in (0, mg.DECODE_SOURCE_ORDER):
        plan = mg.plan(st.n_units, n, 1024, {"flags": flags})
        aux = torch.full((mg.aux_size(st.n_units, plan),), 0x5A, dtype=torch.uint8, device="cuda")
        out = torch.full((n + 64,), 0xCD, dtype=torch.uint8, device="cuda")
        decode_async(units, st.n_units, out[shift:], n, table, 1024, st.first_state,
                     st.first_bit, aux, plan)
        assert aux_status(aux) == 0
        b = out.cpu().numpy()
        assert np.array_equal(b[shift: shift + n], sym if flags else sym[::-1])
        assert (b[:shift] == 0xCD).all() and (b[shift + n:] == 0xCD).all()
