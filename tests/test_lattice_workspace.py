"""Workspace of plans that decode through the lattice: the lattice and the
region decode that stands in for it use the same memory, one at a time."""
import pytest


@pytest.mark.parametrize("n_units,n_out,L", [
    (50_339_428, 268_435_456, 1024), (144_000_000, 536_870_913, 4096), (6_376_000, 134_217_805, 4096),
    (17_000_000, 90_000_000, 1024), (3_146_214, 16 << 20, 1024), (32_000, 131_071, 1024), (900, 4099, 1024)])
def test_lattice_shares_the_regions_memory(mg, n_units, n_out, L):
    plan = mg.plan(n_units, n_out, L)
    assert plan["flags"] & mg.DECODE_LATTICE
    regions = mg.aux_size(n_units, dict(plan, flags=plan["flags"] & ~mg.DECODE_LATTICE))
    bare = mg.aux_size(n_units, dict(plan, capture_bytes=0))
    assert mg.aux_size(n_units, plan) == max(regions, bare)
