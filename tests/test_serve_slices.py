"""The cap of a job's slice: whatever the caller asks for, the parts of a slice
and one claim beyond it by every warp are counted in 32 bits."""
import os
import shutil
import subprocess

import pytest

CHECK = r"""
#include <cstdint>
#include <cstdio>
#include "serve_common.h"
int main() {
    const uint32_t wanted[] = {0, 1, 4096, 1u << 20, (1u << 28) - 1, 1u << 28, 1u << 30, 0xffffffffu};
    for (uint32_t w : wanted) printf("%u %llu\n", w, (unsigned long long)srv_slice_cap(w) << SRV_SUB_BITS);
    return 0;
}
"""


def test_parts_of_a_slice_fit_their_counter(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "naivesat_b200", "csrc")
    src = tmp_path / "slices.cpp"
    src.write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-I", csrc, "-I", "/usr/local/cuda/include", str(src), "-o", str(tmp_path / "slices")], check=True)
    out = subprocess.run([str(tmp_path / "slices")], capture_output=True, text=True, check=True).stdout
    parts = dict(tuple(int(x) for x in line.split()) for line in out.splitlines())
    warps = 1024 * 64                       # more than any device keeps resident
    for wanted, count in parts.items():
        assert 0 < count and count + warps < 1 << 32
        assert count >> 2 == (wanted or 4096) or wanted > 1 << 28
    server = open(os.path.join(csrc, "serve.cpp")).read()
    assert "s->opts.max_slice_tiles = srv_slice_cap(s->opts.max_slice_tiles);" in server
