"""A CTA of a cluster may touch another one's shared memory only once that CTA is known to run.  A kernel that stores
into a peer's shared memory therefore announces itself to the cluster at its start and waits for all others before the
first such store.  The order is read from the sources: breaking it is a race that a GPU test would rarely see."""

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
    body = _body(file, signature)
    at = [body.find(s) for s in ("cluster_arrive_started()", "cluster_wait_started()", remote_store)]
    assert 0 <= at[0] < at[1] < at[2], at
