"""Each stream's own workspace inside a batch against the slice planned for it
alone (mans_batch_slice_size): a batch decoded in given slices writes up to the
former, so it must never exceed the latter, stream by stream and up to
outputs of 2 GB, where the planner lengthens regions and deepens lattices
differently alone and in company.  Sizing calls only, no device memory."""
import ctypes

import numpy as np
import pytest


def _arr(batch, specs):
    ds = []
    for i, (n_units, n_out, L, flags) in enumerate(specs):
        base = 0x100000 * (i + 1)   # placeholder addresses, never dereferenced
        ds.append(batch.StreamDesc(base, n_units, base + 0x80000, n_out, base + 0x40000, L, L, 32,
                                   flags))
    return (batch.StreamDesc * len(ds))(*ds)


def _inside(mg, specs):
    """Bytes of each stream in the batch, and the descriptors."""
    from multians_gb300 import batch
    lib = batch._sig()
    vp, sz = ctypes.c_void_p, ctypes.POINTER(ctypes.c_size_t)
    lib.mans_batch_data_sizes.argtypes = [vp, ctypes.c_uint32, vp, sz]
    arr = _arr(batch, specs)
    inside = (ctypes.c_size_t * len(specs))()
    assert lib.mans_batch_data_sizes(arr, len(specs), None, inside) == 0
    return list(inside), arr


def _check(mg, specs):
    inside, arr = _inside(mg, specs)
    lib = mg.lib()
    lib.mans_batch_slice_size.argtypes = [ctypes.c_void_p, ctypes.c_void_p,
                                          ctypes.POINTER(ctypes.c_size_t)]
    v = ctypes.c_size_t()
    for i in range(len(specs)):
        assert lib.mans_batch_slice_size(ctypes.byref(arr[i]), None, ctypes.byref(v)) == 0
        assert inside[i] <= v.value, (i, specs[i], inside[i], v.value)


def test_sparse_stream_in_company(mg):
    """One stream of 58 M units beside twelve of far more symbols per unit: its
    share of the lanes is small, its chain long."""
    _check(mg, [(58_198_146, 935_418_631, 1024, 0)] + [(1_500_000, 800_000_000, 1024, 0)] * 12)


@pytest.mark.parametrize("flags", [0, 2, 4])   # planner's choice, without, with symbol capture
@pytest.mark.parametrize("seed", range(4))
def test_random_batches(mg, seed, flags):
    rng = np.random.default_rng(seed)
    for _ in range(250):
        specs = []
        for _ in range(int(rng.integers(1, 66))):
            n_out = int(np.exp(rng.uniform(np.log(4_000), np.log(2 << 30))))
            bps = float(np.exp(rng.uniform(np.log(0.05), np.log(8.6))))
            specs.append((max(1, int(n_out * bps / 32)), n_out,
                          int(rng.choice([64, 1024, 2048, 4096, 8192])), flags))
        _check(mg, specs)


@pytest.mark.parametrize("k,deep", [(0.1, True), (0.25, False), (1.0, False)])
def test_long_streams_have_no_deep_lattice(mg, k, deep):
    """The sparse company above asks for 32 slots a block (blocks of 16 units,
    eight bytes a slot), whose scan goes from tile to tile in order: not past
    512 tiles of 1024 blocks."""
    n_units = int(58_198_146 * k)
    inside, _ = _inside(mg, [(n_units, int(935_418_631 * k), 1024, 0)] +
                        [(int(1_500_000 * k), int(800_000_000 * k), 1024, 0)] * 12)
    assert (n_units // 16 <= 512 * 1024) == deep
    assert (inside[0] >= n_units // 16 * 32 * 8) == deep
