"""Decodes in workspaces smaller than the planner's first choice: the lattice
where it fits without the room for symbol capture, and the region plan's own
size, which plain decodes always took.  Byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).to("cuda")


def _run(mg, st, size, blocking):
    import torch
    from multians_gb300.decoder import aux_status, decode_async
    aux = torch.empty(size, dtype=torch.uint8, device="cuda")
    out = torch.full((st.n + 16,), 0xCD, dtype=torch.uint8, device="cuda")
    args = (_dev(st.units), st.n_units, out, st.n, _dev(st.table), st.L, st.first_state, st.first_bit)
    if blocking:
        mg.decode(args[0], st.n_units, st.n, args[4], st.first_state, st.first_bit, L=st.L, aux=aux,
                  out=out)
    else:
        decode_async(*args, aux)
        assert aux_status(aux) == 0
    launches = int(mg.lib().mans_last_launch_count())
    stats = mg._lib.sync_stats(aux.data_ptr(), size, st.n_units, st.n, st.L)
    b = out.cpu().numpy()
    assert np.array_equal(b[:st.n][::-1], st.symbols) and (b[st.n:] == 0xCD).all()
    return launches, stats


@pytest.mark.parametrize("blocking", [False, True])
def test_lattice_without_room_for_capture(mg, blocking):
    """A stream long enough for capture, in a workspace without its slices."""
    from multians_gb300 import host
    st = host.make_stream(31, 0.2, 150_000_001, 1024)
    plan = mg.plan(st.n_units, st.n, st.L)
    size = mg.aux_size(st.n_units, dict(plan, capture_bytes=0))
    assert plan["capture_bytes"] and mg.aux_size(st.n_units, plan) > size
    launches, stats = _run(mg, st, size, blocking)
    assert launches == 4   # tables, sync, scan, final: the lattice's kernels
    assert stats["open_walks"] == 0 and stats["fallback_warps"] == 0


@pytest.mark.parametrize("blocking", [False, True])
@pytest.mark.parametrize("n,lam,L", [(400_000, 0.2, 1024), (3_000_000, 0.05, 1024),
                                     (3_000_000, 0.2, 4096), (9_000, 0.005, 256),
                                     (12_000_000, 2.0, 2048)])
def test_region_plan_size(mg, oracle_lib, n, lam, L, blocking):
    st = oracle_lib.make_stream(seed=n, lam=lam, n=n, L=L)
    plan = mg.plan(st.n_units, n, L)
    regions = mg.plan(st.n_units, n, L, dict(plan, flags=plan["flags"] & ~mg.DECODE_LATTICE,
                                             walk_slots=0))
    size = mg.aux_size(st.n_units, regions)
    assert size < mg.aux_size(st.n_units, plan)
    _run(mg, st, size, blocking)
