"""Doubling of tables large enough that their contracted domains contract
again, and of one whose image shrinks too late for the first look at it,
against plain rounds in torch: whole tables, steps, and answers before, between
and after the contractions.  The levels that a solve makes follow from the
images and stop_join.cpp's thresholds; they are asserted, so that a change of
the thresholds cannot empty the test."""
import os
import re

import pytest
import torch

from naivesat_b200 import workloads as W
from test_gpu_stop_doubling import machine

pytestmark = pytest.mark.gpu

SOURCE = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "naivesat_b200", "csrc",
                           "stop_join.cpp")).read()


def constant(name):
    m = re.search(r"constexpr \w+ %s = (?:1ull << (\d+)|([\d.]+));" % name, SOURCE)
    return 1 << int(m.group(1)) if m.group(1) else float(m.group(2))


def contractions(n, images):
    """Rounds after which a solve that runs on contracts; images[r]: distinct
    successors after round r that have not stopped."""
    size = 1 << n
    assert "entries * 4 <= (64ull << 20) ? 5 : 4" in SOURCE
    assert "looks[2] = {{1, first_rounds(N), 0.85}, {6, 8, kKeepMost}}" in SOURCE
    left, keep = constant("kRoundsLeft"), constant("kKeepMost")
    at = None
    if size >= constant("kTableLeast"):
        looks = [(1, 5 if size * 4 <= 64 << 20 else 4, 0.85)]
        if size >= constant("kSecondLook"):
            looks.append((6, 8, keep))
        for sampled, r, most in looks:
            assert abs(images[sampled] / size - most) > 0.05      # not the sample's decision by chance
            if n > r + left and images[sampled] <= most * size:
                at = r
                break
    made, items = [], size
    while at is not None and images[at] <= keep * items:
        made.append(at)
        items = images[at]
        step = int(constant("kRoundsPerLevel"))
        at = at + step if items >= constant("kContractLeast") and n > at + step + left else None
    return made


def late(n, low):
    """The low bits count up and stay at all ones, the others count round and
    halt at a pattern: 2^-low of the states remain, but only after 2^low steps."""
    rb = W.RawBuilder(n)

    def chain(first, count):
        carry, bits = None, []
        for i in range(first, first + count):
            bits.append((i, None) if carry is None else (rb.gate(W.XOR, i, carry), carry))
            carry = i if carry is None else rb.gate(W.AND, i, carry)
        return bits, carry
    bits, full = chain(0, low)
    for k, (w, _) in enumerate(bits):
        rb.output(rb.gate(W.NOR, w, full, 1 if k == 0 else 0, 0), 1)       # incremented, or all ones
    bits, _ = chain(low, n - low)
    for k, (w, _) in enumerate(bits):
        rb.output(w, 1 if k == 0 else 0)
    acc = None
    for i in range(low, n):
        acc = i if acc is None else rb.gate(W.AND, acc, i, 0, (0x2b5d >> (i % 14)) & 1)
    rb.output(acc)
    return rb.fold()


CASES = [
    # circuit, unknowns and the rounds between which answers have to lie
    ("two levels", 25, lambda: machine(25 * 7 + 3 + 1000, 25, 12), (0, 1, 3, 5, 6, 7, 8, 11, 25), [4, 7]),
    ("three levels", 26, lambda: machine(26 * 7 + 2 + 3000, 26, 17), (0, 1, 9, 10, 12, 14, 19), [4, 7, 10]),
    ("second look", 25, lambda: late(25, 6), (0, 3, 9, 12, 16, 19, 25), [8]),
]


@pytest.mark.parametrize("name,n,circuit,unknowns,levels", CASES, ids=[c[0] for c in CASES])
def test_levels_match_plain_rounds(ctx, name, n, circuit, unknowns, levels):
    h = ctx.circuit(circuit())
    t = h.stop_table()
    size, stop = 1 << n, 1 << n
    tables = [torch.from_numpy(t.read().view("int64")).cuda().int()]
    t.close()
    dist = torch.ones(size, dtype=torch.int64, device="cuda")     # of the entries that have stopped
    images = [0]
    for r in range(1, n + 1):
        v = tables[-1]
        going = v < stop
        nx = torch.where(going, v, 0).long()
        w = torch.where(going, v[nx], v)
        dist = torch.where(going & (w >= stop), (1 << (r - 1)) + dist[nx], dist)
        tables.append(w)
        mark = torch.zeros(size, dtype=torch.bool, device="cuda")
        mark[w[w < stop].long()] = True
        images.append(int(mark.sum()))
    assert contractions(n, images) == levels
    answered = set()
    for u in unknowns:
        starts = torch.arange(1 << u, device="cuda") << (n - u)
        for mode in (0, 1):
            for r in range(1, n + 1):
                hit = torch.nonzero(tables[r][starts] >= stop)
                best = int(starts[hit[0, 0]]) if len(hit) else None
                if best is not None and (mode == 0 or best == 0):
                    break
            answered.add(sum(r > x for x in levels))
            for steps in (False, True):
                t = h.stop_table(want_steps=steps)
                got = t.solve(u, mode=mode)
                assert got["rounds"] == r and got["found"] == (best is not None)
                if best is not None:
                    assert got["start"] == best and got["end"] == int(tables[r][best]) - stop
                    assert got["steps"] == (int(dist[best]) if steps else 0)
                after = torch.from_numpy(t.read().view("int64")).cuda()
                assert torch.equal(after, tables[r].long())
                t.close()
    assert answered == set(range(len(levels) + 1))      # answers before, between and after the contractions
