"""The planner sweep times region plans: every candidate decodes by regions
with exactly its geometry, capture choice and walk slots when it is handed to
a decode, and the candidates differ."""
import pytest


@pytest.mark.parametrize("n_units,n,L", [(50_339_428, 256 << 20, 1024), (12_800_000, 256 << 20, 4096),
                                         (3_146_214, 16 << 20, 1024), (800_000, 16 << 20, 8192)])
def test_candidates_are_region_plans(mg, n_units, n, L):
    from multians_gb300 import tune
    cands = tune.candidates(mg, n_units, n, L)
    assert len(cands) >= 6
    seen = set()
    for c in cands:
        cfg = c["cfg"]
        assert not cfg["flags"] & mg.DECODE_LATTICE
        assert cfg["block_units"] == c["block_units"]
        assert (cfg["capture_bytes"] > 0) == c["capture"]
        # what a decode makes of it
        assert mg.plan(n_units, n, L, cfg) == cfg
        # as many walk slots as its regions take, like a plan whose geometry
        # is fixed by hand
        by_hand = mg.plan(n_units, n, L, {"block_units": cfg["block_units"],
                                          "region_blocks": cfg["region_blocks"]})
        assert cfg["walk_slots"] == by_hand["walk_slots"]
        seen.add((cfg["block_units"], cfg["region_blocks"], cfg["capture_bytes"] > 0))
    assert len(seen) == len(cands)
