"""Waits whose absence a GPU test would rarely see, or only by hanging: they are read from the sources."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "interattn_b200", "csrc")


def _body(file, signature):
    """The function that starts at `signature`, without comments."""
    with open(os.path.join(CSRC, file)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    start = text.index("{", text.index(signature))
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i]
    raise AssertionError(f"no end of {signature}")


@pytest.mark.parametrize("file,signature,remote_store", [
    ("llama_step.cu", "llama_argmax_parts_kernel(const PartsView", "st.shared::cluster"),
    ("select_kernel.cuh", "select_body(const SelectParams& p)", "st_cluster_f32("),
    ("select_kernel.cuh", "select_body(const SelectParams& p)", "map_to_rank("),
])
def test_no_remote_store_before_the_whole_cluster_runs(file, signature, remote_store):
    """A CTA of a cluster may touch another one's shared memory only once that CTA is known to run: a kernel that stores
    into a peer's shared memory announces itself to the cluster at its start and waits for all others before that."""
    body = _body(file, signature)
    at = [body.find(s) for s in ("cluster_arrive_started()", "cluster_wait_started()", remote_store)]
    assert 0 <= at[0] < at[1] < at[2], at


def test_waits_of_the_streamed_projections_end():
    """try_wait may park a thread for as long as the hardware likes, so its loop is bounded by the clock and not by a
    number of polls; after a wait that ran out no further copy or MMA is issued, and the copies in flight are awaited
    before the CTA ends (read from the source: making these waits run out would take a faulty kernel)."""
    assert "global_timer_ns() - start < kParkedWaitNs" in _body("skinny_gemm.cu", "bool mbar_wait_parked(")
    body = _body("skinny_gemm.cu", "llama_stream_gemm_kernel(const __grid_constant__")
    producer, consumer = body[body.index("if (warp == 0) {"):].split("} else if (warp == 1) {")
    issuer = consumer[:consumer.index("} else {")]
    failed = r"if \([^;{]*!mbar_wait\(&%s[^;{]*\{[^}]*DEV_STATUS_GEMM_WAIT_TIMEOUT\);\s*break;"
    assert re.search(failed % "empty_bar", producer) and re.search(failed % "acc_empty", issuer)
    assert re.search(failed % "full_bar", issuer)
    assert producer.rindex("mbar_wait(&full_bar[s]") > producer.rindex("load_x(")
    assert issuer.rindex("mbar_wait(&empty_bar[last_stage]") > issuer.rindex("umma_commit(")
