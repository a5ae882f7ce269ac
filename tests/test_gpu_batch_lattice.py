"""Batches that mix lattice streams with streams on the region kernels: a
stream that asks for capture, a single-symbol table, data that meets late,
streams of a few units, both output orders and unaligned outputs; launched
directly, as a graph and in the one-call form.  Byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).to("cuda")


@pytest.mark.parametrize("capture", [False, True])
def test_mixed_batch(mg, oracle_lib, capture):
    import torch

    from multians_gb300 import batch
    O = oracle_lib
    rng = np.random.default_rng(6)
    late = rng.integers(0, 8, 150_000).astype(np.uint8)
    sts = [O.make_stream(seed=50 + i, lam=lam, n=n, L=L)
           for i, (lam, n, L) in enumerate([(0.05, 200_000, 1024), (2.0, 150_000, 4096),
                                            (0.2, 1, 1024), (0.005, 33, 256), (1.0, 4_097, 8192),
                                            (0.2, 700_001, 2048), (0.05, 5, 1024)])]
    sts += [O.encode(late, 1024), O.encode(np.full(9_000, 17, dtype=np.uint8), 1024)]
    total = sum(st.n for st in sts) + 64
    big = torch.empty(total, dtype=torch.uint8, device="cuda")
    keep, descs, spans, at = [], [], [], 3
    for i, st in enumerate(sts):
        u, t = _dev(st.units), _dev(st.table)
        keep.append((u, t))
        d = batch.desc(u, st.n_units, big[at: at + st.n], st.n, t, st.L, st.first_state,
                       st.first_bit, source_order=bool(i % 2))
        if capture and i in (0, 5):
            d.flags |= mg.DECODE_CAPTURE
        descs.append(d)
        spans.append((at, at + st.n))
        at += st.n

    def check(what):
        b = big.cpu().numpy()
        assert (b[:3] == 0xCD).all() and (b[at:] == 0xCD).all()
        for i, (st, (x, y)) in enumerate(zip(sts, spans)):
            got = b[x:y]
            assert np.array_equal(got if i % 2 else got[::-1], st.symbols), (what, i)

    s = torch.cuda.current_stream()
    bt = batch.Batch(descs)
    for what in ("direct", "graph", "graph again"):
        big.fill_(0xCD)
        (bt.decode if what == "direct" else bt.graph_decode)(s)
        acc, per = bt.status(s)
        assert acc & ~mg.DEV_DEGENERATE == 0, per
        check(what)
    bt.close()
    big.fill_(0xCD)
    acc, per = batch.decode_batch(descs, stream=s)
    assert acc & ~mg.DEV_DEGENERATE == 0, per
    check("one call")
