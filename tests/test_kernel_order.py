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
    release the host (after which another context may use the nodes) follow a
    fence by each thread and a barrier."""
    text = source("device_template.cuh")
    tail = text[text.index("nodes[i] = 0u;"):]
    tail = tail[:tail.index("nsat_publish(")]
    assert re.search(r"__threadfence\(\);\s*__syncthreads\(\);\s*if \(threadIdx\.x == 0\)", tail)
