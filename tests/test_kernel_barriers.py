"""Barriers in the kernel sources that threads of one warp may reach apart (no
GPU needed: a barrier that waits for good is not run to see it)."""
import os

from tile_processor_gpu_b200 import build


def test_cluster_barrier_takes_divergent_threads():
    """k_texture_list's phases end in loops that lanes leave one by one, so its
    cluster barrier must not be the form that wants whole warps."""
    with open(os.path.join(build.CSRC, "tp_list.cuh")) as f:
        text = f.read()
    uses = [line for line in text.splitlines() if "barrier.cluster." in line]
    assert uses and not any(".aligned" in line for line in uses)
