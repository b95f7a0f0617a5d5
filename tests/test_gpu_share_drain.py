"""A shared queue that runs out while launches are in flight: their results
count."""
import pytest

from naivesat_b200 import api
from naivesat_b200 import workloads as W

pytestmark = pytest.mark.gpu


def only_solution(n, value):
    """Satisfied by the assignment `value` alone."""
    gates = []
    acc = None
    for i in range(n):
        bit = (value >> i) & 1
        if acc is None:
            gates.append((W.AND, i, i) if bit else (W.NOR, i, i))
        else:
            gates.append((W.AND, acc, i) if bit else (W.NIMPL, acc, i))
        acc = n + len(gates) - 1
    return W.Circuit(n, gates, [(acc, 0)])


@pytest.mark.parametrize("left", [1, 2, 3, 4, 7])
def test_launches_in_flight_when_the_queue_runs_out(ctx, left):
    n, chunk_bits = 24, 18
    chunks = 1 << (n - chunk_bits)
    for back in range(1, left + 1):            # the solution's chunk, counted from the last
        value = ((chunks - back) << chunk_bits) | 0x2a5f3
        share = api.SatShare()
        share.next = chunks - left
        r = ctx.circuit(only_solution(n, value)).sat(find_all=False, chunk_bits=chunk_bits, share=share)
        assert r["satisfiable"] and r["witness"] == value
        # chunks above the solution's are not claimed once it is known
        assert left - back + 1 <= r["launches"] <= left and r["scanned"] == r["launches"] << chunk_bits
        assert left > 4 or r["launches"] == left           # all in flight at once


def test_launches_in_flight_when_the_stop_lands(ctx):
    """Nobody claims a chunk at or above the stop; those below it count."""
    n, chunk_bits = 24, 18
    value = (2 << chunk_bits) | 0x1234
    share = api.SatShare()
    share.stop_plus1 = 1 + 3
    r = ctx.circuit(only_solution(n, value)).sat(find_all=False, chunk_bits=chunk_bits, share=share)
    assert r["witness"] == value and r["launches"] == 3
