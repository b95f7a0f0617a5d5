"""A tuned QSAT shape keeps the chunks that it was timed with."""
import statistics

import pytest

from naivesat_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("persist", [False, True])
def test_tuned_solves_reach_the_rate_reported(ctx, tmp_path, monkeypatch, persist):
    monkeypatch.setenv("NSAT_JIT_CACHE", str(tmp_path))
    c = W.config("c2b")           # decided early: small chunks leave most of it out
    h = ctx.circuit(c)

    def rate():
        r = [h.qsat(c.quants) for _ in range(40)][5:]
        return r[0]["scanned"] / (statistics.median(x["device_ms"] for x in r) * 1e-3)
    default = rate()
    t = h.autotune("qsat", quants=c.quants, sample_ms=20, persist=persist)
    # without its chunks the solve takes 1.5 times as long
    assert rate() > 0.8 * t["best_rate"] and rate() > 0.9 * default
    if persist:
        h = ctx.circuit(c)
        again = h.autotune("qsat", quants=c.quants, persist=True)
        assert again["from_cache"] and again["cta_bits_max"] == t["cta_bits_max"]
        assert rate() > 0.8 * t["best_rate"] and rate() > 0.9 * default
