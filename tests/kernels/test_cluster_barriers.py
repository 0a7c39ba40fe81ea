"""A cluster barrier in its aligned form is undefined for a warp whose lanes have not met again after a branch, and no wait on it has a limit:
the one function that holds it gathers the warp first. Read from the sources, no GPU."""

import re

from nanonemo_b200.csrc import build

BARRIER = "barrier.cluster.arrive"


def _function_around(text, at):
    start = max(m.start() for m in re.finditer(r"^__device__[^\n]*\{$", text, re.M) if m.start() < at)
    return text[start:text.index("\n}", at)]


def test_attention_backward_meets_through_the_function_that_gathers_the_warp():
    header = (build.HERE / "sm100.cuh").read_text()
    found = [m.start() for m in re.finditer(re.escape(BARRIER), header)]
    assert found
    for at in found:
        body = _function_around(header, at)
        assert body.index("__syncwarp();") < body.index(BARRIER), body
    for name in ("flash_bwd.cu", "flash_bwd_t.cu"):
        text = (build.HERE / name).read_text()
        assert "cluster_sync();" in text and "barrier.cluster" not in text


def test_other_cluster_barriers_follow_a_block_barrier():
    text = (build.HERE / "gemm2.cu").read_text()
    calls = [m.start() for m in re.finditer(r"^\s*cluster_sync_all\(\);", text, re.M)]
    assert calls
    for at in calls:
        assert text[:at].rstrip().endswith("__syncthreads();")
