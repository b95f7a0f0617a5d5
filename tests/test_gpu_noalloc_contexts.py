"""nsat_qsat_solve_noalloc from several contexts of one device, one call after
another: they share the static area."""
import ctypes as C

import pytest

from naivesat_b200 import api
from naivesat_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_contexts_take_turns():
    # short solves with many nodes and with few, under different trees
    cases = []
    for seed, n, gates, longest in ((71, 22, 40, 2), (72, 22, 60, 5), (73, 20, 50, 1), (74, 21, 90, 3)):
        c = W.random_dag(seed, n, gates, output="live")
        q = W.alternating_quants(seed, n, longest)
        cases.append((c, q, O.qsat(O.Circuit(c.n, c.gates, c.outputs), q, mode=1)))
    with api.Context(0) as a, api.Context(0, block_threads=64) as b:
        handles = [[x.circuit(c) for c, _, _ in cases] for x in (a, b)]
        for i in range(4000):
            k = (i * 7 + i // 5) % len(cases)
            got = handles[i & 1][k].qsat_noalloc(cases[k][1])
            exp = cases[k][2]
            assert {x: got[x] for x in exp} == exp, i


def test_area_left_dirty(ctx):
    """What the static area holds before a call does not reach the call's answer."""
    fill = api.lib().nsat_test_fill_noalloc
    fill.argtypes = [C.c_void_p, C.c_int]
    # trees from many nodes to none (units inside a chunk), one launch and several
    for seed, n, gates, longest, chunk in ((81, 22, 40, 2, 0), (82, 24, 300, 6, 0), (83, 22, 60, 21, 0), (84, 16, 50, 3, 0),
                                           (85, 24, 200, 2, 20)):
        c = W.random_dag(seed, n, gates, output="live")
        q = W.alternating_quants(seed, n, longest)
        exp = O.qsat(O.Circuit(c.n, c.gates, c.outputs), q, mode=1)
        h = ctx.circuit(c)
        for byte in (0x00, 0x80, 0xff, 0x01):
            assert fill(ctx.h, byte) == 0
            got = h.qsat_noalloc(q, chunk_bits=chunk)
            assert {x: got[x] for x in exp} == exp, (seed, byte)
