"""Short decodes and encodes, whose kernels are launched before the ones ahead
of them have ended: many in a row on one stream through one workspace, each
overwriting the last one's tables and slots, and replays of a captured decode
whose input changes in between.  Integer work: the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).to("cuda")


@pytest.mark.parametrize("n", [1, 40, 4099, 131_071, 700_001])
def test_calls_in_a_row(mg, oracle_lib, n):
    import torch
    O = oracle_lib
    lams, Ls = (0.05, 0.3, 1.5, 0.01), (1024, 4096, 2048, 1024)
    sts = [O.make_stream(seed=40 + i, lam=lams[i], n=n + i, L=Ls[i]) for i in range(4)]
    plans = [mg.plan(s.n_units, s.n, s.L) for s in sts]
    need = max(mg.aux_size(s.n_units, p) for s, p in zip(sts, plans))
    aux = torch.empty(need, dtype=torch.uint8, device="cuda")
    dev = [(_dev(s.units), _dev(s.table)) for s in sts]
    outs = [torch.zeros(sts[i % 4].n, dtype=torch.uint8, device="cuda") for i in range(40)]
    for i, out in enumerate(outs):
        s = sts[i % 4]
        mg.decode_async(dev[i % 4][0], s.n_units, out, s.n, dev[i % 4][1], s.L, s.first_state,
                        s.first_bit, aux, plans[i % 4])
    for i, out in enumerate(outs):
        assert np.array_equal(out.cpu().numpy(), sts[i % 4].symbols[::-1]), i


def test_captured_decode(mg, oracle_lib):
    import torch
    O = oracle_lib
    sts = [O.make_stream(seed=50 + i, lam=0.2, n=20_000, L=1024) for i in range(3)]
    n_units = max(s.n_units for s in sts)
    st = sts[0]
    plan = mg.plan(st.n_units, st.n, st.L)
    aux = torch.empty(mg.aux_size(st.n_units, plan), dtype=torch.uint8, device="cuda")
    units = torch.zeros(n_units + 4, dtype=torch.int32, device="cuda")
    table = torch.zeros(1024, dtype=torch.int32, device="cuda")
    out = torch.zeros(st.n, dtype=torch.uint8, device="cuda")

    def decode():
        mg.decode_async(units, st.n_units, out, st.n, table, st.L, st.first_state, st.first_bit,
                        aux, plan)

    def load(s):
        units.zero_()
        units[: s.n_units] = _dev(s.units[: s.n_units])
        table.copy_(_dev(s.table))

    load(st)
    decode()   # first calls set attributes, outside the capture
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        decode()
    for _ in range(3):
        out.zero_()
        g.replay()
        g.replay()
        assert np.array_equal(out.cpu().numpy(), st.symbols[::-1])
    # another stream's symbols under the first one's start: as the call gives them
    load(sts[1])
    g.replay()
    got = out.cpu().numpy().copy()
    decode()
    assert np.array_equal(got, out.cpu().numpy())


@pytest.mark.parametrize("n", [1, 65, 4096, 100_001, 1_300_000])
def test_encodes_in_a_row(mg, oracle_lib, n):
    import torch
    from multians_gb300 import encode
    O = oracle_lib
    for i in range(6):
        L = (1024, 4096)[i % 2]
        sym = O.gen_symbols(60 + i, (0.05, 0.5, 2.0)[i % 3], n + i)
        want = O.encode(sym, L)
        units, n_units, first_bit, first_state, table = encode.encode(
            torch.from_numpy(sym.copy()).cuda(), L)
        assert (n_units, first_bit, first_state) == (want.n_units, want.first_bit, want.first_state)
        assert np.array_equal(units.cpu().numpy().view(np.uint32)[:n_units], want.units[:n_units])
