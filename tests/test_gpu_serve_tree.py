"""Served QSAT jobs around the tile geometry: units inside a part of a tile, of
a part, a tile and larger; the tree on the device, and the host's reducer
where the tree has no room; against the oracle."""
import random

import pytest

from naivesat_b200 import api
from naivesat_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def jobs():
    rng = random.Random(12)
    for n, first in [(9, 2), (13, 4), (16, 8), (16, 6), (17, 5), (17, 4), (17, 3), (17, 2), (18, 2), (18, 17), (20, 1),
                     (20, 3), (21, 6), (22, 2), (23, 4), (24, 1)]:
        for longest in (1, 3, 9):
            ch = rng.choice("AE")
            q = ch * first
            while len(q) < n:
                ch = "E" if ch == "A" else "A"
                q += ch * rng.randint(1, longest)
            c = W.random_dag(rng.randrange(1 << 30), n, rng.randint(12, 220), output="live")
            yield c, q[:n]


@pytest.mark.parametrize("shape,arena", [(1, 0), (5, 0), (1, 3072)])
def test_quantifier_trees(ctx, shape, arena):
    # 3 KB of arena: a small job's program fits, the larger trees do not
    cases = [(c, q) for c, q in jobs() if not arena or c.num_gates < 60]
    assert cases
    srv = api.Server(ctx, shape=shape, arena_bytes=arena, tier_min_ms=0xffffffff)
    try:
        for i, (c, q) in enumerate(cases):
            srv.submit("qsat", c, quants=q, tag=i)
        got = {r["tag"]: r for r in srv.run_all()}
    finally:
        srv.close()
    for i, (c, q) in enumerate(cases):
        exp = O.qsat(O.Circuit(c.n, c.gates, c.outputs), q, mode=1)
        assert got[i]["status"] == 0
        assert {k: got[i][k] for k in exp} == exp, (c.n, q)


@pytest.mark.parametrize("rollover", [False, True])
def test_counts_and_tables_by_parts(ctx, rollover):
    """Every assignment once, whichever way tiles are claimed: exact counts,
    lowest witnesses, and SATOSTOP answers."""
    srv = api.Server(ctx, rollover=rollover, first_slice_tiles=3)
    try:
        cs = [W.random_dag(70 + n, n, 30 + 9 * n, output="live") for n in (8, 13, 14, 15, 16, 19, 22)]
        ms = [W.lfsr_stop(n, n, 60) for n in (5, 10, 12, 13, 15, 16, 18)]
        for i, c in enumerate(cs):
            srv.submit("sat", c, tag=i, find_all=True)
        for i, c in enumerate(ms):
            srv.submit("stop", c, unknowns=c.n, tag=100 + i)
        got = {r["tag"]: r for r in srv.run_all()}
    finally:
        srv.close()
    for i, c in enumerate(cs):
        assert (got[i]["count"], got[i]["witness"]) == O.sat_range(O.Circuit(c.n, c.gates, c.outputs)), c.n
    for i, c in enumerate(ms):
        exp = O.stop_solve(c.n, c.n, O.stop_table(O.Circuit(c.n, c.gates, c.outputs)), mode=1)
        r = got[100 + i]
        assert r["found"] == (exp is not None)
        if exp is not None:
            assert (r["start"], r["end"], r["steps"]) == (exp["start"], exp["end"], exp["steps"])
