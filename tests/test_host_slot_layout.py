"""Where the red-black solves put the slots of a pack's instances (host arithmetic,
no GPU): a cluster copies its rows of J as whole warp tiles of 32 slots, so it may
take a pack only when every instance starts on one."""
import ctypes

import numpy as np
import pytest


def _layout(shapes):
    from tcad_b200 import _lib
    lib = _lib.load(require_gpu=False)
    s = np.array([tuple(q) + (1,) * (3 - len(q)) for q in shapes], dtype=np.int32)
    start = np.full(len(shapes) + 1, -1, dtype=np.int64)
    cluster = ctypes.c_int32(-1)
    n = int(np.prod(s, axis=1, dtype=np.int64).sum())
    rc = lib.tcad_slot_layout_test(s.ctypes.data, len(shapes), n, len(shapes[0]),
                                   start.ctypes.data, ctypes.byref(cluster))
    return rc, start, cluster.value, n


PACKS = [[(5, 3)] * 2, [(3, 3)] * 2, [(41, 21), (5, 3), (5, 3)], [(5, 3), (41, 21)],
         [(64, 41), (21, 10), (2, 2)], [(9, 7, 5), (24, 16, 13)], [(5, 3, 1)] * 2]


@pytest.mark.parametrize("shapes", PACKS, ids=lambda q: "+".join(str(s) for s in q))
def test_clusters_start_on_warp_tiles(shapes):
    rc, start, cluster, _ = _layout(shapes)
    assert rc == 0
    assert cluster == 0 or not (start[:-1] % 32).any()


def test_single_instances_keep_their_cluster():
    for shape, ctas in (((2, 2), 8), ((5, 3), 8), ((81, 41), 8), ((9, 7, 5), 8),
                        ((120, 120), 16), ((31, 22, 16), 16), ((201, 101), 0)):
        rc, start, cluster, _ = _layout([shape])
        assert (rc, start[0], cluster) == (0, 0, ctas), shape
