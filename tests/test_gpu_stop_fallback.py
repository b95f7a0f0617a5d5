"""Solves of 2^15 .. 2^20 states whose one cooperative launch gives up at its
grid barrier: the rounds start again, a launch each, from the table as built."""
import ctypes as C

import numpy as np
import pytest

from naivesat_b200 import api
from naivesat_b200 import workloads as W
from test_gpu_stop_doubling import doubling, machine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [False, True])
@pytest.mark.parametrize("n,kind,unknowns", [(15, "counter", 4), (16, 4, 16), (17, 16, 0), (18, 9, 7), (20, 20, 5)])
def test_rounds_after_a_barrier_that_gave_up(n, kind, unknowns, steps):
    c = W.counter_stop(n) if kind == "counter" else machine(n * 5 + unknowns, n, kind)
    spins = api.lib().nsat_test_grid_spins
    spins.argtypes = [C.c_void_p, C.c_uint32]
    with api.Context(0) as ctx:
        h = ctx.circuit(c)
        # 1: the CTAs that arrive first give up at once; many: the launch goes through
        gave_up = []
        for limit in (1, 1 << 22, 1):
            gave_up.append(spins(ctx.h, limit))
            t = h.stop_table(want_steps=steps)
            table, dist = t.read().astype(np.uint32), np.ones(1 << n, dtype=np.int64)
            for mode in (1, 0):                     # the second solve starts from the first one's table
                if not (table >> np.uint32(n)).any():
                    break
                r = t.solve(unknowns, mode=mode)
                table, dist, rounds, best = doubling(table, dist, n, unknowns, mode)
                assert r["rounds"] == rounds and r["found"] == (best is not None)
                if best is not None:
                    assert r["start"] == best and r["end"] == int(table[best]) & ((1 << n) - 1)
                    assert r["steps"] == (int(dist[best]) if steps else 0)
                np.testing.assert_array_equal(t.read(), table.astype(np.uint64))
            t.close()
        gave_up.append(spins(ctx.h, 1))
        assert gave_up[0] == 0 and gave_up[1] + gave_up[3] >= 1 and gave_up[2] == 0
