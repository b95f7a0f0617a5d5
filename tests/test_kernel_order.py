"""Orderings that the kernels' sources have to state, checked on their text: a
run would show a missing one only by chance."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "naivesat_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def test_nodes_are_zero_before_the_host_is_released():
    """The last CTA's threads all put QSAT nodes back to zero; the words that
    release the host (after which another context may use shared nodes) follow a
    fence by each thread and a barrier."""
    text = source("device_template.cuh")
    tail = text[text.index("nodes[i] = 0u;"):]
    tail = tail[:tail.index("nsat_publish(")]
    assert re.search(r"if \(shared\) \{\s*__threadfence\(\);\s*__syncthreads\(\);\s*\}\s*if \(threadIdx\.x == 0\)", tail)
    assert "uint32_t shared = fixed_scratch ? 1 : 0;" in source("nsat_api.cpp")


def test_overlapped_kernels_take_no_const_restrict():
    """A kernel that waits for its predecessor by pdl_wait can be resident while
    its inputs are still being written, so none of them may be read through the
    non-coherent path."""
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = source(name)
        for k in re.finditer(r"__global__[^{;]*\)\s*\{", text):
            body = text[k.end():]
            body = body[:body.index("\n}\n")]
            if "pdl_wait()" not in body:
                continue
            seen += 1
            assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", k.group(0)), k.group(0)
            assert "__ldg(" not in body
    assert seen == 4
