"""Buffers that the pool refuses: the calls that can do without one answer as
before."""
import ctypes as C

import numpy as np
import pytest

from naivesat_b200 import api
from naivesat_b200 import workloads as W
from test_gpu_stop_doubling import doubling, machine

pytestmark = pytest.mark.gpu


def fail_alloc(ctx, k):
    f = api.lib().nsat_test_fail_alloc
    f.argtypes = [C.c_void_p, C.c_uint32]
    return f(ctx.h, k)


@pytest.mark.parametrize("k", [1, 2, 3])
@pytest.mark.parametrize("n,partitions", [(14, 4), (18, 16)])
def test_partitioned_solve_when_the_pool_is_in_pieces(n, partitions, k):
    """A repeated solve counts on what the first one gave back to the pool; when
    a buffer does not come out of that, it goes by the free memory."""
    with api.Context(0) as ctx:
        h = ctx.circuit(machine(n, n, 6))
        first = h.greedy_partitioned(n // 2, partitions)
        assert first["storage"] == 0
        fail_alloc(ctx, k)
        again = h.greedy_partitioned(n // 2, partitions)
        assert fail_alloc(ctx, 0) == 0             # the refusal was met
        keys = ("found", "start", "end", "stage", "partition", "joins", "load_bits", "storage")
        assert {x: again[x] for x in keys} == {x: first[x] for x in keys}


@pytest.mark.parametrize("steps", [False, True])
@pytest.mark.parametrize("n,kind,unknowns,buffers", [(16, 5, 9, 1), (21, 14, 4, 0), (24, 13, 3, 3)])
def test_solves_without_one_of_their_buffers(n, kind, unknowns, buffers, steps):
    """Distances, the copy of the table, the sample, and each buffer of a
    contraction in turn."""
    with api.Context(0) as ctx:
        h = ctx.circuit(machine(n + 3 * unknowns, n, kind))
        t = h.stop_table(want_steps=steps)
        built = t.read().astype(np.uint32)
        t.close()
        table, dist, rounds, best = doubling(built, np.ones(1 << n, dtype=np.int64), n, unknowns, 1)
        for k in range(1, 10):
            t = h.stop_table(want_steps=steps)
            fail_alloc(ctx, k)
            r = t.solve(unknowns, mode=1)
            met = fail_alloc(ctx, 0) == 0
            assert r["rounds"] == rounds and r["found"] == (best is not None)
            if best is not None:
                assert r["start"] == best and r["end"] == int(table[best]) & ((1 << n) - 1)
                assert r["steps"] == (int(dist[best]) if steps else 0)
            np.testing.assert_array_equal(t.read(), table.astype(np.uint64))
            t.close()
            if not met:
                break
        assert k - 1 >= buffers + steps            # refusals met
