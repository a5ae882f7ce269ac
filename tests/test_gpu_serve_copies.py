"""Served requests whose pinned buffers are copied by one launch: outputs at
every offset from a 16-byte line and of lengths around multiples of 16, units
at every word offset, buffers on both sides of the size up to which that is
done, and more requests than one launch takes.  Byte for byte, with guards
around every output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_small_copies(mg, oracle_lib):
    import torch
    from multians_gb300 import serve
    O = oracle_lib
    sizes = [1, 2, 15, 16, 17, 31, 33, 255, 4095, 4096, 4097, 70_001, (256 << 10) - 1, 256 << 10,
             (256 << 10) + 1, 400_003]
    sts = [O.make_stream(seed=300 + i, lam=0.05 if i % 2 else 0.3, n=n, L=1024)
           for i, n in enumerate(sizes)]
    srv = serve.Server(budget_bytes=1 << 30)
    reqs, keep = [], []
    for i in range(16 * 17):
        st = sts[i % 16]
        shift, words = (i // 16) % 16, i % 4
        out = torch.full((st.n + 64,), 0xCD, dtype=torch.uint8).pin_memory()
        units = torch.zeros(st.n_units + 4, dtype=torch.int32).pin_memory()
        units[words: words + st.n_units] = torch.from_numpy(
            np.ascontiguousarray(st.units[: st.n_units]).view(np.int32))
        keep.append((st, units, out, shift))
        reqs.append(serve.request(units[words:], st.n_units, out[shift: shift + st.n], st.n,
                                  srv.add_table(st.table), st.first_state, st.first_bit, tag=i))
    for _ in range(2):
        for _, _, out, _ in keep:
            out.fill_(0xCD)
        srv.submit(reqs)
        done = srv.wait(len(reqs))
        assert all(c.status == 0 for c in done)
        for st, _, out, shift in keep:
            b = out.numpy()
            assert np.array_equal(b[shift: shift + st.n], st.symbols[::-1]), (st.n, shift)
            assert (b[:shift] == 0xCD).all() and (b[shift + st.n:] == 0xCD).all()
    srv.close()
