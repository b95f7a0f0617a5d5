"""Performance cases: what users of the solver have it do, by size and kind.

The four command-line tools are one call each of the Python API (a SAT search,
a QSAT solve, a SATOSTOP table with its doubling solve, the partitioned greedy
solve); a serving process drives a Server.  The listed cases span each of
them from the smallest calls, where launches and host time count, to the
benchmark configurations; `draw` gives others of the same ranges.

A case is a dict of plain values:
  kind   sat | planted | qsat | adder | lfsr | machine | counter | greedy | serve
  n      inputs (state bits for the SATOSTOP kinds)
and per kind: gates, find_all (sat, planted), max_block (qsat: longest
quantifier block), key_bits (adder), unknowns, steps and mode (SATOSTOP),
stop_bits (state bits that the STOP condition looks at), partitions (greedy),
jobs (serve).
Circuits follow from the case and the seed; sizes follow from the case alone.
"""
import math

import numpy as np

from naivesat_b200 import api
from naivesat_b200 import workloads as W

_CTX = None


def _context():
    """One context per process, as a program that solves many circuits keeps."""
    global _CTX
    if _CTX is None:
        _CTX = api.Context(0)
    return _CTX


def listed():
    return [
        # a small SAT circuit, counted: the cost of a call (launch, copies, result)
        {"name": "sat_16", "kind": "sat", "n": 16, "gates": 100, "find_all": True},
        # naivesat's own use: the first witness of a 24-input, 500-gate circuit
        {"name": "sat_find_24", "kind": "sat", "n": 24, "gates": 500, "find_all": False},
        # the headline benchmark: 36 inputs, 3018 gates, a planted block, every assignment counted
        {"name": "sat_36", "kind": "planted", "n": 36, "gates": 3000, "find_all": True},
        # a small quantified formula with short alternating blocks
        {"name": "qsat_16", "kind": "qsat", "n": 16, "gates": 150, "max_block": 4},
        # exists a key, forall a, exists b: a + b == target over two 14-bit words: long blocks
        {"name": "qsat_adder_32", "kind": "adder", "n": 32, "key_bits": 4},
        # a 30-input, 1500-gate formula with alternating blocks of up to six
        {"name": "qsat_30", "kind": "qsat", "n": 30, "gates": 1500, "max_block": 6},
        # a small state machine, as a server's SATOSTOP requests: lowest stopping start with its steps
        {"name": "stop_12", "kind": "machine", "n": 12, "gates": 100, "stop_bits": 8, "unknowns": 6, "steps": True,
         "mode": 1},
        # greedysatostop on a 24-bit register with a mixer: a table that fits the L2 cache
        {"name": "stop_lfsr_24", "kind": "lfsr", "n": 24, "gates": 300, "unknowns": 12, "steps": False, "mode": 0},
        # naivesatostop on a 24-bit counter: every state stops, the furthest after 2^24 steps
        {"name": "stop_counter_24", "kind": "counter", "n": 24, "unknowns": 16, "steps": True, "mode": 1},
        # a 28-bit register: a table well beyond the L2 cache
        {"name": "stop_lfsr_28", "kind": "lfsr", "n": 28, "gates": 400, "unknowns": 20, "steps": False, "mode": 0},
        # greedysatostop -p 4 on a 26-bit machine, the packed image in device memory
        {"name": "greedy_26", "kind": "greedy", "n": 26, "gates": 300, "stop_bits": 12, "unknowns": 3,
         "partitions": 4},
        # a serving process answering a batch of mixed requests
        {"name": "serve_64", "kind": "serve", "n": 30, "gates": 2000, "jobs": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sat", "planted", "qsat", "adder", "lfsr", "machine", "counter", "greedy", "serve"])
    if kind == "sat":
        return {"kind": kind, "n": rng.randint(12, 34), "gates": _log_int(rng, 60, 4000),
                "find_all": rng.random() < 0.5}
    if kind == "planted":
        return {"kind": kind, "n": rng.randint(20, 35), "gates": _log_int(rng, 300, 3000),
                "find_all": rng.random() < 0.5}
    if kind == "qsat":
        return {"kind": kind, "n": rng.randint(12, 33), "gates": _log_int(rng, 60, 3000),
                "max_block": rng.randint(2, 12)}
    if kind == "adder":
        key = rng.randint(2, 7)
        return {"kind": kind, "n": key + 2 * rng.randint(6, 13), "key_bits": key}
    if kind == "lfsr":
        n = rng.randint(11, 27)
        return {"kind": kind, "n": n, "gates": _log_int(rng, 50, 600), "unknowns": rng.randint(2, n),
                "steps": rng.random() < 0.5, "mode": rng.randint(0, 1)}
    if kind == "machine":
        n = rng.randint(11, 26)
        return {"kind": kind, "n": n, "gates": _log_int(rng, 50, 600), "stop_bits": rng.randint(4, n),
                "unknowns": rng.randint(2, n), "steps": rng.random() < 0.5, "mode": rng.randint(0, 1)}
    if kind == "counter":
        n = rng.randint(11, 26)
        return {"kind": kind, "n": n, "unknowns": rng.randint(2, n), "steps": rng.random() < 0.5,
                "mode": rng.randint(0, 1)}
    if kind == "greedy":
        n = rng.randint(14, 26)
        return {"kind": kind, "n": n, "gates": _log_int(rng, 50, 600), "stop_bits": rng.randint(4, n),
                "unknowns": rng.randint(2, n), "partitions": rng.choice([2, 4, 8, 16])}
    return {"kind": "serve", "n": rng.randint(22, 30), "gates": _log_int(rng, 200, 2000),
            "jobs": rng.randint(8, 64)}


# ---------------------------------------------------------------------------
# circuits


def _literal_and(n, gates, literals):
    """Appends AND gates over (wire, negated) literals; returns the last wire."""
    (a, na), (b, nb) = literals[0], literals[1]
    gates.append((W.NOR, a, b) if na and nb else (W.NIMPL, b, a) if na else (W.NIMPL, a, b) if nb else (W.AND, a, b))
    for w, neg in literals[2:]:
        acc = n + len(gates) - 1
        gates.append((W.NIMPL if neg else W.AND, acc, w))
    return n + len(gates) - 1


def _machine(seed, n, mixer_gates, stop_bits):
    """A register with a random mixer that halts on a pattern of its low bits."""
    base = W.lfsr_stop(seed, n, max(mixer_gates, n + 1))
    gates = [tuple(g) for g in base.gates.tolist()]
    pattern = W.SplitMix64(seed ^ 0x57A7E).next()
    stop = _literal_and(n, gates, [(i, ((pattern >> i) & 1) == 0) for i in range(max(2, stop_bits))])
    return W.Circuit(n, gates, base.outputs.tolist()[:n] + [[stop, 0]])


def _counter(seed, n):
    """next = s + 1 mod 2^n, STOP on a seeded value."""
    pattern = W.SplitMix64(seed).next() & ((1 << n) - 1)
    rb = W.RawBuilder(n)
    outs = [(0, 1)]
    carry = 0
    for i in range(1, n):
        outs.append((rb.gate(W.XOR, i, carry), 0))
        if i < n - 1:
            carry = rb.gate(W.AND, i, carry)
    acc = rb.gate(W.AND, 0, 1, not pattern & 1, not (pattern >> 1) & 1)
    for i in range(2, n):
        acc = rb.gate(W.AND, acc, i, 0, not (pattern >> i) & 1)
    for w, neg in outs + [(acc, 0)]:
        rb.output(w, neg)
    return rb.fold()


def _keyed(n, gates, out, keys, bits, value):
    """(out AND the first block equals keys[0]) OR the first block equals
    keys[1]; with value 0 the dual.  The first block's witness
    (counterexample) is one of the keys.  Returns the output."""
    def match(key):
        return [(i, ((key >> i) & 1) == 0) for i in range(bits)]
    wire, neg = out
    first = _literal_and(n, gates, [(wire, neg != (not value))] + match(keys[0]))
    second = _literal_and(n, gates, match(keys[1]))
    gates.append((W.NOR, first, second))
    return [n + len(gates) - 1, value]


def _qsat(seed, n, num_gates, max_block):
    """A random DAG under seeded alternating quantifier blocks of up to
    max_block inputs, the first of at least two, whose inputs have to match
    one of two seeded keys (one with the DAG, one without)."""
    c = W.random_dag(seed, n, num_gates, output="live")
    rng = W.SplitMix64(seed ^ 0x5157A7)
    q, quants, first = ("A", "E")[rng.below(2)], "", 0
    while len(quants) < n:
        k = 1 + rng.below(max_block)
        if not first:
            first = k = max(2, k)
        quants += q * k
        q = "E" if q == "A" else "A"
    gates = [tuple(g) for g in c.gates.tolist()]
    first = min(first, n)
    out = _keyed(n, gates, c.outputs.tolist()[0], (rng.next(), rng.next()), first, 1 if quants[0] == "E" else 0)
    return W.Circuit(n, gates, [out]), quants[:n]


def _adder(seed, n, key_bits):
    """exists key, forall a, exists b: key == K and (a + b) mod 2^w == target."""
    w = (n - key_bits) // 2
    rng = W.SplitMix64(seed)
    target, key = rng.next(), rng.next()
    rb = W.RawBuilder(n)
    lits, carry = [], None      # carry: (wire, negated)
    for i in range(w):
        a, b = key_bits + i, key_bits + w + i
        t = rb.gate(W.XOR, a, b)
        s = t if carry is None else rb.gate(W.XOR, t, carry[0], 0, carry[1])
        if i < w - 1:
            g = rb.gate(W.AND, a, b)
            carry = (g, 0) if carry is None else (rb.gate(W.NOR, g, rb.gate(W.AND, t, carry[0], 0, carry[1])), 1)
        lits.append((s, 0 if (target >> i) & 1 else 1))
    lits += [(i, 0 if (key >> i) & 1 else 1) for i in range(key_bits)]
    acc = rb.gate(W.AND, lits[0][0], lits[1][0], lits[0][1], lits[1][1])
    for s, neg in lits[2:]:
        acc = rb.gate(W.AND, acc, s, 0, neg)
    rb.output(acc)
    return rb.fold(), "E" * key_bits + "A" * w + "E" * w


def _requests(case, seed):
    """A batch in the serving trace's proportions: per ten jobs seven SAT, two
    QSAT and one SATOSTOP; sizes spread over the case's range, the same for
    every seed."""
    rng = W.SplitMix64(seed)
    reqs = []
    for i in range(case["jobs"]):
        u = (i * 0.6180339887498949) % 1.0
        v = (i * 0.7548776662466927) % 1.0
        rseed = rng.next() & 0xFFFFFFFF
        kind = "stop" if i % 10 == 9 else "qsat" if i % 5 == 2 else "sat"
        if kind == "stop":
            n = 12 + int(u * 9)
            reqs.append((kind, W.lfsr_stop(rseed, n, max(n + 1, int(50 * 20 ** v))), None, n // 2))
            continue
        n = 18 + int(u * (case["n"] - 17))
        c = W.random_dag(rseed, n, int(100 * (case["gates"] / 100.0) ** v), output="live")
        quants = None
        if kind == "qsat":
            q = W.SplitMix64(rseed ^ 0xA5A5)
            quants = "".join("A" if q.below(2) else "E" for _ in range(n))
        reqs.append((kind, c, quants, 0))
    return reqs


# ---------------------------------------------------------------------------


def prepare(case, seed):
    """The circuit handle a program keeps (the server and its requests for
    serving)."""
    ctx = _context()
    kind, n = case["kind"], case["n"]
    st = dict(case, ctx=ctx)
    if kind == "serve":
        st["server"] = api.Server(ctx)
        st["requests"] = _requests(case, seed)
        return st
    if kind == "sat":
        c = W.random_dag(seed, n, case["gates"], output="live")
    elif kind == "planted":
        c = W.planted_dag(seed, n, case["gates"], plant_bits=min(18, n))
    elif kind == "qsat":
        c, st["quants"] = _qsat(seed, n, case["gates"], case["max_block"])
    elif kind == "adder":
        c, st["quants"] = _adder(seed, n, case["key_bits"])
    elif kind == "lfsr":
        c = W.lfsr_stop(seed, n, max(case["gates"], n + 1))
    elif kind == "counter":
        c = _counter(seed, n)
    else:
        c = _machine(seed, n, case["gates"], case["stop_bits"])
    st["circuit"] = ctx.circuit(c)
    return st


def _pick(r, keys):
    """The answer's numbers, -1 where it has none (no witness, no start)."""
    return {k: -1 if r.get(k) is None else r[k] for k in keys}


def run(st):
    kind = st["kind"]
    if kind in ("sat", "planted"):
        return _pick(st["circuit"].sat(find_all=st["find_all"]), ("satisfiable", "witness", "count", "scanned"))
    if kind in ("qsat", "adder"):
        return _pick(st["circuit"].qsat(st["quants"]),
                     ("reversed", "solution_bits", "solution", "value", "launches", "chunk_bits", "scanned"))
    if kind in ("lfsr", "machine", "counter"):
        table = st["circuit"].stop_table(want_steps=st["steps"])
        r = table.solve(st["unknowns"], mode=st["mode"])
        # where the first states have got to after the last round
        ends = table.read(0, min(1 << st["n"], 4096))
        table.close()
        return dict(_pick(r, ("found", "start", "end", "steps", "rounds")), ends=ends.astype(np.int64))
    if kind == "greedy":
        return _pick(st["circuit"].greedy_partitioned(st["unknowns"], st["partitions"]),
                     ("found", "start", "end", "stage", "partition", "load_bits", "storage", "joins"))
    server = st["server"]
    for i, (k, c, quants, unknowns) in enumerate(st["requests"]):
        server.submit(k, c, quants=quants, unknowns=unknowns, tag=i)
    answers = server.run_all()
    # per request: status, a truth value, and up to three numbers of its answer (-1: none)
    out = np.full((len(answers), 5), -1, dtype=np.int64)
    for a in answers:
        keys = {"sat": ("satisfiable", "witness"), "qsat": ("value", "solution", "solution_bits"),
                "stop": ("found", "start", "end", "steps")}[a["kind"]]
        out[a["tag"], 0] = a["status"]
        for j, key in enumerate(keys):
            if a[key] is not None:
                out[a["tag"], 1 + j] = int(a[key])
    return out


# ---------------------------------------------------------------------------


def work(case):
    """flops: 32-bit word operations, one per gate and 32 assignments (and one
    per table entry and doubling round); bytes: tables written once when
    built, read and written once when solved, and circuits read once."""
    kind, n = case["kind"], case["n"]
    size = 1 << n
    gates = case.get("gates", 0)
    if kind in ("sat", "planted", "qsat"):
        return {"bytes": 12 * gates + 64, "flops": size / 32 * gates}
    if kind == "adder":
        return {"bytes": 12 * 3 * n + 64, "flops": size / 32 * 3 * n}
    if kind in ("lfsr", "machine", "counter"):
        entry = 8 if case["steps"] else 4
        return {"bytes": 3 * entry * size, "flops": size / 32 * (gates or 3 * n) + size}
    if kind == "greedy":
        return {"bytes": 3 * size * (n + 1) / 8, "flops": size / 32 * gates + size}
    ops = nbytes = 0.0
    for i in range(case["jobs"]):
        u = (i * 0.6180339887498949) % 1.0
        v = (i * 0.7548776662466927) % 1.0
        g = int(100 * (case["gates"] / 100.0) ** v)
        if i % 10 == 9:
            s = 12 + int(u * 9)
            ops += (1 << s) / 32 * int(50 * 20 ** v)
            nbytes += 3 * 8 * (1 << s)
        elif i % 5 == 2:
            ops += (1 << (18 + int(u * (case["n"] - 17)))) / 32 * g
        else:
            ops += (1 << 18) / 32 * g       # a SAT request ends at its first witness
        nbytes += 12 * g
    return {"bytes": nbytes, "flops": ops}
