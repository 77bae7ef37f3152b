"""Argument checks of the re-clusterization that end a call before any GPU work."""
import numpy as np

import meshoptimizer_gb300 as mg


def test_no_vertices_is_refused_on_the_host():
    """The kernel puts vertex 0 in the place of a bad index, so there has to be one."""
    from meshoptimizer_gb300 import build

    build.build()
    off = np.array([0, 3], np.uint64)
    for positions, vertex_count in ((0, 0), (4096, 0), (0, 5)):
        try:
            mg.build_meshlets_flex_groups_device(4096, 4096, 4096, mg.meshlet_rows(off, 64, 16), 4096, off, positions, vertex_count, 12, 64, 16, 64)
            raise AssertionError("not refused")
        except mg.SimplifyError as e:
            assert e.status == mg.STATUS_INVALID_ARGUMENT
