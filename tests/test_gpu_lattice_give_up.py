"""The lattice decode on data whose trajectories meet so late that the true
path runs out of slots again and again: it gives up after a number of blocks
(256 at L = 1024, 512 at 4096) decoded one after the other, says so, and every blocking call decodes the stream
all the same.  Byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPAIRED = 256 + 5 * 4   # byte of the workspace counter of repaired blocks
TILE = 1024              # blocks


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).to("cuda")


def _late(oracle_lib, K=4, L=1024, n=1 << 20, rare=0.0):
    rng = np.random.default_rng(K * 100 + L + n)
    sym = rng.integers(0, K, n).astype(np.uint8)
    if rare:
        sym[rng.random(n) < rare] = 200
    return oracle_lib.encode(sym, L)


def _counter(aux):
    return int(aux[REPAIRED: REPAIRED + 4].cpu().numpy().view(np.uint32)[0])


@pytest.mark.parametrize("K,L,n", [(4, 1024, 1 << 20), (8, 1024, 16 << 20), (4, 4096, 4 << 20),
                                   (2, 4096, 16 << 20)])
def test_gives_up_early(mg, oracle_lib, K, L, n):
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    st = _late(oracle_lib, K, L, n, 1e-4 if n == 4 << 20 else 0.0)
    plan = mg.plan(st.n_units, n, L)
    aux = torch.empty(mg.aux_size(st.n_units, plan), dtype=torch.uint8, device="cuda")
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    decode_async(_dev(st.units), st.n_units, out, n, _dev(st.table), L, st.first_state,
                 st.first_bit, aux, plan)
    assert aux_status(aux) & mg.DEV_SYNC_OVERFLOW
    limit = {1024: 256, 4096: 512}[L]
    assert _counter(aux) == limit + 1


@pytest.mark.parametrize("source_order", [False, True])
@pytest.mark.parametrize("start_offset", [False, True])
def test_blocking_calls(mg, oracle_lib, source_order, start_offset):
    import torch
    from multians_gb300 import batch
    st = _late(oracle_lib)
    other = oracle_lib.make_stream(seed=8, lam=0.05, n=70_001, L=1024)
    flags = (mg.DECODE_SOURCE_ORDER if source_order else 0) | \
        (mg._lib.DECODE_START_OFFSET if start_offset else 0)
    bit = lambda s: 32 - s.first_bit if start_offset else s.first_bit  # noqa: E731
    dev = [(_dev(s.units), _dev(s.table)) for s in (st, other)]

    def right(out, s):
        b = out.cpu().numpy()
        return np.array_equal(b if source_order else b[::-1], s.symbols)

    aux = torch.empty(mg.aux_size(st.n_units, mg.plan(st.n_units, st.n, 1024)), dtype=torch.uint8,
                      device="cuda")
    got = mg.decode(*[dev[0][0], st.n_units, st.n, dev[0][1], st.first_state, bit(st)], L=1024, aux=aux,
                    cfg={"flags": flags})
    assert right(got, st)
    outs = [torch.full((s.n,), 0xCD, dtype=torch.uint8, device="cuda") for s in (st, other)]
    descs = []
    for s, (u, t), o in zip((st, other), dev, outs):
        d = batch.desc(u, s.n_units, o, s.n, t, s.L, s.first_state, bit(s), source_order=source_order)
        d.flags |= flags
        descs.append(d)
    bt = batch.Batch(descs)
    cs = torch.cuda.current_stream()
    bt.graph_decode(cs)
    _, per = bt.status(cs)
    assert per[0] & mg.DEV_SYNC_OVERFLOW and per[1] == 0
    assert bt.fixup(cs) == 1 and bt.status(cs)[1] == [0, 0]
    assert all(right(o, s) for o, s in zip(outs, (st, other)))
    bt.close()
    for o in outs:
        o.fill_(0xCD)
    acc, per = batch.decode_batch(descs, stream=cs)
    assert acc == 0 and per == [0, 0]
    assert all(right(o, s) for o, s in zip(outs, (st, other)))


def test_served(mg, oracle_lib):
    """Pinned and pageable outputs: what was copied out before the second
    decode is copied again."""
    import torch
    from multians_gb300 import serve
    sts = [_late(oracle_lib), oracle_lib.make_stream(seed=8, lam=0.05, n=70_001, L=1024)]
    srv = serve.Server(budget_bytes=1 << 30)
    reqs, keep = [], []
    for i in range(6):
        st = sts[i % 2]
        out = torch.full((st.n,), 0xCD, dtype=torch.uint8)
        units = torch.from_numpy(np.ascontiguousarray(st.units[: st.n_units]).view(np.int32))
        if i < 4:
            out, units = out.pin_memory(), units.pin_memory()
        keep.append((st, units, out))
        reqs.append(serve.request(units, st.n_units, out, st.n, srv.add_table(st.table),
                                  st.first_state, st.first_bit, tag=i))
    srv.submit(reqs)
    assert all(c.status == 0 for c in srv.wait(len(reqs)))
    for st, _, out in keep:
        assert np.array_equal(out.numpy()[::-1], st.symbols)
    assert srv.stats()["streams_redone"] == 3
    srv.close()


@pytest.mark.parametrize("n,rare", [(1 << 20, 0.0), (4 << 20, 1e-4)])
def test_repairs_over_tiles(mg, oracle_lib, n, rare):
    """Repairs in a lattice of 32 slots a block over many scan tiles: the end
    of each tile, with or without a slot, is handed to the next."""
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    L = 4096
    st = _late(oracle_lib, 8, L, n, rare)
    aux = torch.empty(mg.aux_size_max_any(st.n_units), dtype=torch.uint8, device="cuda")
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    decode_async(_dev(st.units), st.n_units, out, n, _dev(st.table), L, st.first_state,
                 st.first_bit, aux)
    assert aux_status(aux) == 0
    assert np.array_equal(out.cpu().numpy()[::-1], st.symbols)
    assert _counter(aux) > 0
    stats = mg._lib.sync_stats(aux.data_ptr(), aux.numel(), st.n_units, n, L)
    assert stats["blocks"] > 4 * TILE
