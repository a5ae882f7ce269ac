"""bench.py's planner report says which decode ran: a lattice with its own
geometry, or regions with the plan's."""
import argparse
import importlib.util
import os
import types

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_planner_report(mg):
    bench = _bench()
    n, n_units, L = 256 << 20, 50_339_428, 1024
    st = types.SimpleNamespace(L=L, n=n, n_units=n_units, bits_per_symbol=32 * n_units / n)
    args = argparse.Namespace(no_capture=False)
    plan = mg.plan(n_units, n, L)
    r = bench.planner_report(mg, st, args, plan, {"blocks": n_units // 32 + 1, "regions": 77_826})
    assert r["decode"] == "lattice" and "entry" not in r
    assert r["lattice"] == {"blocks": n_units // 32 + 1, "starts": 77_826, "units_per_block": 32}
    assert r["regions"]["entry"]["block_units"] == plan["block_units"]
    assert bench.planner_report(mg, st, args, plan, {"error": "x"})["lattice"] is None
    regions = dict(plan, flags=plan["flags"] & ~mg.DECODE_LATTICE)
    r = bench.planner_report(mg, st, args, regions, {"blocks": 1})
    assert r["decode"] == "regions" and r["source"] == "measured table"
