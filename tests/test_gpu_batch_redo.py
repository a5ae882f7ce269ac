"""Streams of a batch whose path runs out of slots are decoded again, also
where their slice is smaller than the workspace of a plain decode (which has
room for seeded walks on top).  Byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).to("cuda")


@pytest.mark.parametrize("K,L,n", [(2, 1024, 250_007), (4, 1024, 250_007)])
@pytest.mark.parametrize("source_order", [False, True])
def test_region_streams(mg, oracle_lib, K, L, n, source_order):
    """Two or four equally frequent symbols and a rare one: merge walks take
    tens of thousands of units.  The hint keeps the batch on the region
    kernels."""
    import torch
    from multians_gb300 import batch
    rng = np.random.default_rng(K * 100 + L + n)
    late = rng.integers(0, K, n).astype(np.uint8)
    late[rng.random(n) < 0.0001] = 200
    sts = [oracle_lib.encode(late, L), oracle_lib.make_stream(seed=3, lam=0.05, n=80_000, L=1024)]
    keep, descs = [], []
    for st in sts:
        u, t = _dev(st.units), _dev(st.table)
        out = torch.full((st.n,), 0xCD, dtype=torch.uint8, device="cuda")
        keep.append((u, t, out))
        descs.append(batch.desc(u, st.n_units, out, st.n, t, st.L, st.first_state, st.first_bit,
                                source_order=source_order))
    hint = {"flags": mg.DECODE_NO_CAPTURE}
    bt = batch.Batch(descs, hint)
    s = torch.cuda.current_stream()
    bt.decode(s)
    _, per = bt.status(s)
    assert per[0] & mg.DEV_SYNC_OVERFLOW and per[1] == 0
    assert bt.fixup(s) == 1
    assert bt.status(s)[1] == [0, 0]
    bt.close()
    for st, (_, _, out) in zip(sts, keep):
        got = out.cpu().numpy()
        assert np.array_equal(got if source_order else got[::-1], st.symbols)
        out.fill_(0xCD)
    acc, per = batch.decode_batch(descs, hint=hint, stream=s)
    assert acc == 0 and per == [0, 0]
    for st, (_, _, out) in zip(sts, keep):
        got = out.cpu().numpy()
        assert np.array_equal(got if source_order else got[::-1], st.symbols)
