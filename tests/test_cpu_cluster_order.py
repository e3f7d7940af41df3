"""Stores into another CTA's shared memory, by their source: the next thing in the kernel that hands anything over is the
cluster's barrier, which orders them for every thread of the cluster.

An mbarrier arrive of the default form or a commit of the tensor core's instructions orders at the scope of its own CTA; what
they announce may be seen elsewhere before such a store.  A run shows none of that, so it is shown here."""
import re

import pytest

from tests.test_cpu_overlapped_kernels import KERNELS

STORE = re.compile(r"\bst_cluster_\w+\s*\(")
HAND_OVER = re.compile(r"\b(cluster_sync|cluster_arrive|mbar_arrive\w*|tc_commit\w*|team_agrees|__syncthreads|__syncwarp)\s*(?:<[^>]*>)?\(")
STORING = sorted(name for name, (_, body) in KERNELS.items() if STORE.search(body))


def test_the_kernels_that_store_into_other_ctas_are_found():
    assert {"gemm_tiles_kernel", "gemm_f32_kernel"} <= set(STORING)


@pytest.mark.parametrize("name", STORING)
def test_a_barrier_of_the_cluster_comes_before_any_other_hand_over(name):
    body = KERNELS[name][1]
    for store in STORE.finditer(body):
        after = [m.group(1) for m in HAND_OVER.finditer(body, store.end())]
        # __syncwarp gathers the lanes in front of a barrier that a whole warp arrives at
        assert next((m for m in after if m != "__syncwarp"), None) in ("cluster_sync", "cluster_arrive"), after[:3]
