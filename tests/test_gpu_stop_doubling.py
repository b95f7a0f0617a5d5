"""Doubling of 32-bit tables against the plain rounds in numpy: the one-CTA
solve (up to 2^14 entries), plain rounds, and contracted domains of one and
two levels (from 2^20 entries), on maps with shrinking and full images."""
import numpy as np
import pytest

from naivesat_b200 import workloads as W

pytestmark = pytest.mark.gpu


def machine(seed, n, stop_bits):
    """lfsr_stop's register halting on a pattern of its low stop_bits bits."""
    base = W.lfsr_stop(seed, n, max(60, n + 1))
    gates = base.gates.tolist()
    pat = W.SplitMix64(seed ^ 0x57).next()
    acc = None
    for i in range(stop_bits):
        if (pat >> i) & 1:
            gates.append([W.AND, i, i if acc is None else acc])
        elif acc is None:
            gates.append([W.NOR, i, i])
        else:
            gates.append([W.NIMPL, acc, i])
        acc = n + len(gates) - 1
    return W.Circuit(n, gates, base.outputs.tolist()[:n] + [[acc, 0]])


def doubling(table, dist, n, unknowns, mode):
    """Plain synchronous rounds: (table, dist, rounds, lowest start or None)."""
    stop = np.uint32(1 << n)
    starts = np.arange(1 << unknowns, dtype=np.int64) << (n - unknowns)
    best = None
    for r in range(1, n + 1):
        open_ = (table & stop) == 0
        nx = np.where(open_, table, 0)
        dist = np.where(open_, dist + dist[nx], dist)
        table = np.where(open_, table[nx], table)
        hit = np.nonzero(table[starts] & stop)[0]
        best = int(starts[hit[0]]) if len(hit) else None
        if best is not None and (mode == 0 or best == 0):
            return table, dist, r, best
    return table, dist, n, best


@pytest.mark.parametrize("steps", [False, True])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,kind,unknowns", [
    (2, "counter", 2), (5, 2, 0), (11, 4, 11), (12, 8, 6), (13, 11, 5), (14, 14, 7), (15, 3, 15), (16, 16, 9), (17, "counter", 6),
    (20, 20, 10), (20, 9, 20), (21, 14, 1), (21, "counter", 0), (23, 23, 12), (24, 13, 3),
])
def test_rounds_match_plain_doubling(ctx, n, kind, unknowns, mode, steps):
    c = W.counter_stop(n) if kind == "counter" else machine(n * 7 + unknowns, n, kind)
    t = ctx.circuit(c).stop_table(want_steps=steps)
    table = t.read().astype(np.uint32)
    dist = np.ones(1 << n, dtype=np.int64)
    for u in (unknowns, n):                 # the second solve starts from the first one's table
        before = np.nonzero(table >> np.uint32(n))[0]
        r = t.solve(u, mode=mode)
        if len(before) == 0:
            assert not r["found"]
            break
        table, dist, rounds, best = doubling(table, dist, n, u, mode)
        assert r["rounds"] == rounds and r["found"] == (best is not None)
        if best is not None:
            assert r["start"] == best and r["end"] == int(table[best]) & ((1 << n) - 1)
            assert r["steps"] == (int(dist[best]) if steps else 0)
        np.testing.assert_array_equal(t.read(), table.astype(np.uint64))
    t.close()


@pytest.mark.parametrize("n,stop_bits,unknowns,partitions", [
    (11, 3, 11, 2), (11, 8, 4, 32), (12, 12, 12, 64), (13, 10, 7, 16), (16, 2, 16, 1024), (18, 13, 3, 4),
    (19, 19, 19, 8), (21, 12, 0, 2),
])
def test_device_table_steps_match_host_image(ctx, n, stop_bits, unknowns, partitions):
    """The two-kernel steps over a device table against one kernel per join
    over a host image, up to the smallest partitions (64 entries)."""
    h = ctx.circuit(machine(n + stop_bits, n, stop_bits))
    a = h.greedy_partitioned(unknowns, partitions)
    b = h.greedy_partitioned(unknowns, partitions, device_bytes=1)
    assert (a["storage"], b["storage"]) == (0, 1)
    keys = ("found", "start", "end", "stage", "partition", "joins", "load_bits")
    assert {k: a[k] for k in keys} == {k: b[k] for k in keys}


@pytest.mark.parametrize("n", [5, 9, 10, 11, 15, 17, 20])
def test_table_words(ctx, n):
    """Tables below and above the staged size."""
    c = machine(n, n, 3)
    t = ctx.circuit(c).stop_table()
    got = t.read()
    t.close()
    s = np.arange(1 << n, dtype=np.uint32)
    w = [((s >> np.uint32(i)) & 1).astype(bool) for i in range(n)]
    for f, a, b in c.gates.tolist():
        w.append([w[a] & w[b], ~(w[a] | w[b]), w[a] & ~w[b], w[a] ^ w[b]][f])
    exp = np.zeros(1 << n, dtype=np.uint64)
    for k, (o, neg) in enumerate(c.outputs.tolist()):
        exp |= (w[o] ^ bool(neg)).astype(np.uint64) << np.uint64(k)
    np.testing.assert_array_equal(got, exp)
