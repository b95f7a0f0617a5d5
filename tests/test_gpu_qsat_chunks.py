"""The tree above the chunks of the QSAT kernel: decided nodes end their other
chunks, whichever order the chunks finish in, for every cut of the levels into
blocks and several CTA shapes, against the oracle's reducer."""
import random

import numpy as np
import pytest

from naivesat_b200 import api
from naivesat_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def quants(rng, n, longest):
    q, ch = "", rng.choice("AE")
    while len(q) < n:
        q += ch * rng.randint(1, longest)
        ch = "E" if ch == "A" else "A"
    return q[:n]


def items(rng, n, q):
    """2^n item bits, each node of the quantifier tree true or false with
    equal odds: children that decide it are few, the rest are neutral."""
    v = np.array([rng.random() < 0.5])
    nprng = np.random.default_rng(rng.randrange(1 << 30))
    for ch in q:
        # a node under All is true when both halves are, false when one is not
        other = nprng.random(len(v)) < 0.5
        side = nprng.random(len(v)) < 0.5
        free = np.where(v == (ch == "A"), v, other)      # the half that need not carry the value
        v = np.where(side, np.stack([v, free]), np.stack([free, v])).T.reshape(-1)
    return np.packbits(v, bitorder="little").view(np.uint32)


@pytest.mark.parametrize("threads", [32, 256, 512])
@pytest.mark.parametrize("n,longest", [(15, 3), (17, 1), (18, 6), (20, 2), (20, 17), (21, 4), (22, 10)])
def test_words_match_the_reducer(n, longest, threads):
    rng = random.Random(n * 100 + longest)
    with api.Context(0, block_threads=threads) as ctx:
        for _ in range(4):
            q = quants(rng, n, longest)
            w = items(rng, n, q)
            qr = O.QuantReducer(q)
            qr.push_words(w)
            got = ctx.qsat_reduce_words(q, w)
            exp = qr.final_result()
            assert {k: got[k] for k in exp} == exp, (q, threads)


@pytest.mark.parametrize("n,gates,chunk_bits", [(21, 40, 0), (24, 700, 0), (25, 90, 0), (24, 200, 20), (26, 150, 0)])
def test_circuits_match_the_reducer(ctx, n, gates, chunk_bits):
    rng = random.Random(n + gates)
    c = W.random_dag(n * gates, n, gates, output="live")
    h = ctx.circuit(c)
    for longest in (2, 5, 12):
        q = quants(rng, n, longest)
        exp = O.qsat(O.Circuit(c.n, c.gates, c.outputs), q, mode=1)
        for _ in range(2):                # the second run finds the nodes as the first left them
            got = h.qsat(q, chunk_bits=chunk_bits)
            assert {k: got[k] for k in exp} == exp, q
        if n <= 24:
            got = h.qsat_noalloc(q, chunk_bits=chunk_bits)
            assert {k: got[k] for k in exp} == exp, q
