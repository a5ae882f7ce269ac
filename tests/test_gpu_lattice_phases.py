"""GPU parity of the lattice decode on tables of a few states whose codes have
nearly all the same length (a symbol other than the frequent one is rare, and
the frequent one has one state): trajectories at different bit phases run side
by side for tens of thousands of symbols.  They all have a slot: nothing is
repaired.  Byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPAIRED = 256 + 5 * 4   # byte of the workspace counter of repaired blocks


@pytest.mark.parametrize("L,rare,n", [(8, 0.002, 16 << 20), (8, 0.012, 128 << 20), (16, 0.004, 16 << 20),
                                      (16, 0.006, 16 << 20), (16, 0.002, 32 << 20),
                                      (32, 0.002, 16 << 20)])
def test_phases(mg, L, rare, n):
    import torch
    from multians_gb300 import encode
    from multians_gb300.decoder import aux_status, decode_async
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    u = torch.rand(n, generator=g, device="cuda")
    # floor(-ln(1 - u) / rare), cut off at L / 4 - 1
    sym = (1.0 - u).log_().neg_().div_(rare).floor_().clamp_(max=L // 4 - 1).to(torch.uint8)
    units, n_units, first_bit, first_state, dec = encode.encode(sym, L)
    assert 32 * n_units > 0.95 * (L.bit_length() - 1) * n
    table = torch.from_numpy(dec.view(np.int32)).cuda()
    aux = torch.empty(mg.aux_size(n_units, mg.plan(n_units, n, L)), dtype=torch.uint8, device="cuda")
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    for flags in (0, mg.DECODE_SOURCE_ORDER):
        decode_async(units, n_units, out, n, table, L, first_state, first_bit, aux, {"flags": flags})
        assert aux_status(aux) == 0
        assert int(aux[REPAIRED: REPAIRED + 4].cpu().numpy().view(np.uint32)[0]) == 0
        assert torch.equal(out if flags else out.flip(0), sym)
