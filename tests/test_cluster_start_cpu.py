"""The cluster form of the one-kernel solves writes other blocks' shared memory in every exchange, which is
defined only once all blocks of the cluster are known to run: each kernel announces its start and waits for
the others' before its first exchange. Read from the source: nothing is run."""
import os
import re

import pytest

from conftest import ROOT

SOURCE = os.path.join(ROOT, "hethyppar_gb300", "csrc", "hhp_small.cuh")


def _body(text, name):
    at = re.search(r"__global__ [^;{]*\b" + name + r"\(", text).end()
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i]
    raise AssertionError(f"{name}: unbalanced braces")


@pytest.mark.parametrize("kernel", ["k_small", "k_small_mix"])
def test_blocks_are_running_before_the_first_remote_write(kernel):
    with open(SOURCE) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert "barrier.cluster.arrive" in re.search(r"void cluster_start\(\) \{([^}]*)\}", text).group(1)
    assert "barrier.cluster.wait" in re.search(r"void cluster_started\(\) \{([^}]*)\}", text).group(1)
    body = _body(text, kernel)
    start, started = body.find("cluster_start();"), body.find("cluster_started();")
    assert 0 <= start < started < body.index("exchange<")
    assert body.count("cluster_start();") == 1 and body.count("cluster_started();") == 1
    # under the same condition, and outside any other branch or loop
    for at in (start, started):
        line = body[body.rfind("\n", 0, at) + 1:body.find("\n", at)]
        assert line.strip().startswith("if constexpr (CLUSTER)")
        assert body.count("{", 0, at) - body.count("}", 0, at) == 1
    # no other remote write anywhere than in exchange()
    assert "mapa" not in body and "st.shared::cluster" not in body
