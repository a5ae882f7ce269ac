"""Long streams whose codes are eight bits long (a unit holds four) keep symbol capture;
below that, and where capture is not planned, the lattice
decodes."""
import pytest


@pytest.mark.parametrize("n,bps,L,lattice", [
    (128 << 20, 8.0, 256, False), (512 << 20, 8.0, 256, False), (32 << 20, 8.0, 256, True),
    (128 << 20, 7.996, 256, True),
    (128 << 20, 7.0, 256, True), (512 << 20, 8.77, 512, True), (512 << 20, 8.6, 1024, True),
    (128 << 20, 6.99, 128, True), (512 << 20, 8.6, 4096, True)])
def test_capture_keeps_one_length_codes(mg, n, bps, L, lattice):
    n_units = int(n * bps / 32) + 1
    plan = mg.plan(n_units, n, L)
    assert bool(plan["flags"] & mg.DECODE_LATTICE) == lattice
    if not lattice:
        assert plan["capture_bytes"] > 0
        assert mg.plan(n_units, n, L, plan) == plan
