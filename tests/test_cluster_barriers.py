"""Cluster barriers in their .aligned form need all lanes of a warp together.  A lane that comes late can hang the GPU, so
this is checked in the source: what follows lane-dependent code must meet first."""
import os
import re

import drops_gb300

CSRC = os.path.join(os.path.dirname(drops_gb300.__file__), "csrc")


def test_aligned_cluster_barriers_follow_a_warp_barrier():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        for hit in re.finditer(r'asm volatile\("barrier\.cluster\.\w+\.\w+\.aligned', text):
            found += 1
            before = text[:hit.start()].rstrip()
            assert before.endswith("__syncwarp();"), (name, text.count("\n", 0, hit.start()) + 1)
    assert found >= 2
