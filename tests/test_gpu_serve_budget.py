"""A served SATOSTOP job works in the server's own memory: the doubling's
buffers come out of the arena, or it does without them."""
import ctypes as C

import numpy as np
import pytest

from naivesat_b200 import api
from test_gpu_stop_doubling import doubling, machine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("room", [False, True])
@pytest.mark.parametrize("n,stop_bits,unknowns", [(12, 6, 5), (16, 9, 7), (22, 12, 6)])
def test_doubling_takes_nothing_beside_the_arena(n, stop_bits, unknowns, room):
    c = machine(5 * n, n, stop_bits)
    # without room: the job's two areas and its program fit, and little else
    arena = 0 if room else (16 << n) + (64 << 10)
    with api.Context(0) as ctx:
        f = api.lib().nsat_test_fail_alloc
        f.argtypes = [C.c_void_p, C.c_uint32]
        t = ctx.circuit(c).stop_table()
        table, dist, _, best = doubling(t.read().astype(np.uint32), np.ones(1 << n, dtype=np.int64), n, unknowns, 1)
        t.close()
        srv = api.Server(ctx, arena_bytes=arena)
        try:
            f(ctx.h, 1000)
            for i in range(3):
                srv.submit("stop", c, unknowns=unknowns, tag=i)
            got = srv.run_all()
            assert f(ctx.h, 0) == 1000             # the context's pool was not asked
        finally:
            srv.close()
    assert len(got) == 3
    for r in got:
        assert r["status"] == 0 and r["found"] == (best is not None)
        if best is not None:
            assert (r["start"], r["end"], r["steps"]) == (best, int(table[best]) & ((1 << n) - 1), int(dist[best]))
