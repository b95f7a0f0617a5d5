"""Launch numbers past the end of their 32 bits: 0 is left out, and every kind
of short launch, mixed with launches timed by events, answers across it."""
import ctypes as C

import pytest

from naivesat_b200 import api
from naivesat_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", range(15))
def test_numbers_start_again(before):
    number = api.lib().nsat_test_launch_number
    number.argtypes = [C.c_void_p, C.c_uint32]
    oc = [O.Circuit(c.n, c.gates, c.outputs) for c in
          (W.planted_dag(62, 13, 80, plant_bits=7), W.random_dag(63, 18, 60, output="live"), W.lfsr_stop(64, 10, 60),
           W.counter_stop(16))]
    q = "AEE" * 6
    want = [O.sat_range(oc[0]), O.qsat(oc[1], q, mode=1), O.stop_solve(10, 5, O.stop_table(oc[2]), mode=1)]
    with api.Context(0) as ctx:
        h = [ctx.circuit(c) for c in
             (W.planted_dag(62, 13, 80, plant_bits=7), W.random_dag(63, 18, 60, output="live"), W.lfsr_stop(64, 10, 60),
              W.counter_stop(16))]
        for start in (None, 0xffffffff - before, None):
            # the second pass meets the end at another launch for each `before`;
            # the third has numbers that the first used
            if start is not None:
                assert number(ctx.h, start) == 0
            for _ in range(2):
                r = h[0].sat(find_all=True)
                assert (r["count"], r["witness"]) == want[0]
                got = h[1].qsat(q)
                assert {k: got[k] for k in want[1]} == want[1]
                got = h[1].qsat(q, chunk_bits=15)                     # events
                assert {k: got[k] for k in want[1]} == want[1]
                t = h[2].stop_table(want_steps=True)                  # one CTA
                r = t.solve(5, mode=1)
                assert r["found"] == (want[2] is not None)
                if want[2] is not None:
                    assert all(r[k] == want[2][k] for k in ("start", "end", "steps", "rounds"))
                r = h[3].stop_table(want_steps=True).solve(8, mode=1)  # one cooperative launch
                assert (r["start"], r["end"], r["steps"]) == (0, 0, 1 << 16)
