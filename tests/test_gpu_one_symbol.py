"""GPU decodes of streams of a single symbol (no bits at all), whose outputs are
filled with 16-byte stores: lengths around multiples of 16 at every offset from
a 16-byte line, alone and in batches.  Byte for byte, with guards."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [4, 1024])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 4097, 1_000_003])
def test_fill(mg, oracle_lib, n, L):
    import torch
    from multians_gb300 import batch
    from multians_gb300.decoder import aux_status, decode_async
    st = oracle_lib.encode(np.full(n, 201, dtype=np.uint8), L)
    units = torch.from_numpy(np.ascontiguousarray(st.units).view(np.int32)).to("cuda")
    table = torch.from_numpy(np.ascontiguousarray(st.table).view(np.int32)).to("cuda")
    aux = torch.empty(mg.aux_size(st.n_units, mg.plan(st.n_units, n, L)), dtype=torch.uint8,
                      device="cuda")
    cs = torch.cuda.current_stream()
    for shift in range(17):
        for way in ("plain", "batch"):
            big = torch.full((n + 64,), 0xCD, dtype=torch.uint8, device="cuda")
            out = big[shift: shift + n]
            args = (units, st.n_units, out, n, table, L, st.first_state, st.first_bit)
            if way == "plain":
                decode_async(*args, aux, {"flags": shift & 1})
                assert aux_status(aux) == mg.DEV_DEGENERATE
            else:
                acc, _ = batch.decode_batch([batch.desc(*args)], stream=cs)
                assert acc == mg.DEV_DEGENERATE
            b = big.cpu().numpy()
            assert (b[shift: shift + n] == 201).all(), (shift, way)
            assert (b[:shift] == 0xCD).all() and (b[shift + n:] == 0xCD).all(), (shift, way)
