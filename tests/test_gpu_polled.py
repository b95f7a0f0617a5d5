"""Short launches, whose results the host polls for: past the wrap of the
launch number, mixed with launches timed by events, at the sizes around the
lines between the two, and with handles freed straight after a solve."""
import numpy as np
import pytest

from naivesat_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def oc(c):
    return O.Circuit(c.n, c.gates, c.outputs)


def test_launch_numbers_wrap(ctx):
    a, b = W.random_dag(61, 11, 40, output="live"), W.planted_dag(62, 13, 80, plant_bits=7)
    q = "AE" * 10
    qc = W.random_dag(63, 20, 60, output="live")
    s = W.lfsr_stop(64, 10, 60)
    want = [O.sat_range(oc(a)), O.sat_range(oc(b))]
    ha, hb, hq, hs = (ctx.circuit(x) for x in (a, b, qc, s))
    events = hq.qsat(q, chunk_bits=15)          # several launches: timed by events
    table = O.stop_table(oc(s)).astype(np.uint64)
    first = hs.stop_table(want_steps=True).solve(10, mode=1)
    for i in range(16500):                       # four launches each
        for h, (cnt, low) in ((ha, want[0]), (hb, want[1])):
            r = h.sat(find_all=True)
            assert (r["count"], r["witness"]) == (cnt, low)
        if i % 1500:
            r = hq.qsat(q)
            assert (r["value"], r["solution_bits"]) == (events["value"], events["solution_bits"])
            continue
        assert hb.sat(find_all=True, chunk_bits=10)["count"] == want[1][0]
        t = hs.stop_table(want_steps=True)
        assert (t.read() == table).all()
        r = t.solve(10, mode=1)
        assert [r.get(k) for k in ("found", "start", "end", "steps", "rounds")] == \
               [first.get(k) for k in ("found", "start", "end", "steps", "rounds")]
        assert r["build_ms"] < 1.0 and r["join_ms"] < 2.2


@pytest.mark.parametrize("n,gates", [(10, 20), (15, 60), (24, 3000), (28, 60), (28, 700), (29, 300), (31, 40), (32, 40)])
def test_both_sides_of_the_line(ctx, n, gates):
    c = W.random_dag(n * 1000 + gates, n, gates, output="live")
    q = ("AEE" * n)[:n]
    for _ in range(2):
        h = ctx.circuit(c)
        one = h.sat(find_all=True)
        halves = [h.sat(find_all=True, begin=k << (n - 1), end=(k + 1) << (n - 1), chunk_bits=min(n - 1, 24))
                  for k in range(2)] if n > 10 else [one, {"count": 0, "satisfiable": False}]
        assert one["count"] == sum(r["count"] for r in halves)
        low = [r["witness"] for r in halves if r["satisfiable"]]
        assert one["satisfiable"] == bool(low) and (not low or one["witness"] == low[0])
        a = h.qsat(q)
        h.close()                                # its kernel may still be returning
        b = ctx.circuit(c).qsat(q, chunk_bits=min(n, max(15, n - 5)))
        assert [a[k] for k in ("value", "solution")] == [b[k] for k in ("value", "solution")]


@pytest.mark.parametrize("n", [2, 5, 14, 15, 20, 21])
def test_table_builds(ctx, n):
    c = W.counter_stop(n)
    want = O.stop_table(oc(c)).astype(np.uint64)
    for steps in (False, True):
        t = ctx.circuit(c).stop_table(want_steps=steps)
        assert (t.read() == want).all()
        t.solve(n, mode=1)


@pytest.mark.parametrize("n", [14, 15, 16, 17, 18, 19, 20, 21])
def test_one_launch_doubling(ctx, n):
    """Plain rounds in numpy against the solves of one launch and, at n = 21, a
    launch a round; twice, as each leaves the next one's state."""
    c = W.lfsr_stop(n, n, 80)
    table = O.stop_table(oc(c))
    for mode in (0, 1, 0):
        for u in (0, 3, n):
            want = O.stop_solve(n, u, table, mode=mode)
            for steps in (False, True):
                t = ctx.circuit(c).stop_table(want_steps=steps)
                r = t.solve(u, mode=mode)
                assert r["found"] == (want is not None)
                if want:
                    assert (r["start"], r["end"], r["rounds"]) == (want["start"], want["end"], want["rounds"])
                    if steps:
                        assert r["steps"] == want["steps"]
                # the table left behind: 2^rounds evaluations on
                after = table.copy()
                for _ in range(r["rounds"]):
                    stop = (after >> np.uint64(n)) != 0
                    after = np.where(stop, after, after[np.where(stop, 0, after).astype(np.int64)])
                assert r["rounds"] == 0 or (t.read() == after).all()


@pytest.mark.parametrize("n,gates,threads", [(11, 30, 32), (14, 60, 64), (16, 90, 32), (18, 400, 64), (19, 700, 256)])
def test_iterations_together(n, gates, threads):
    """Fewer CTAs, so more iterations per warp, than the default shape's, padded
    inputs included (n < 15), against the oracle."""
    from naivesat_b200 import api
    c = W.random_dag(n * 100 + gates, n, gates, output="live")
    cnt, low = O.sat_range(oc(c))
    q = ("AEEA" * n)[:n]
    with api.Context(0, block_threads=threads) as small:
        h = small.circuit(c)
        want = h.qsat(q)
        for kind, qs in (("sat", None), ("qsat", q)):
            h.autotune(kind, quants=qs)
        r = h.sat(find_all=True)
        assert (r["count"], r["witness"]) == (cnt, low)
        got = h.qsat(q)
        assert [got[k] for k in ("value", "solution")] == [want[k] for k in ("value", "solution")]
