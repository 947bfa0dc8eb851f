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


PACKS = [[(5, 5)] * 3, [(5, 11)] * 4, [(2, 2)] * 8, [(3, 3, 3)] * 3, [(9, 7)] * 64,
         [(5, 3), (3, 3), (5, 3)], [(5, 3)] * 2, [(3, 3)] * 2, [(41, 21), (5, 3), (5, 3)], [(5, 3), (41, 21)],
         [(64, 41), (21, 10), (2, 2)], [(9, 7, 5), (24, 16, 13)], [(5, 3, 1)] * 2]


@pytest.mark.parametrize("shapes", PACKS, ids=lambda q: f"{len(q)}x{q[0]}")
def test_clusters_start_on_warp_tiles(shapes):
    rc, start, cluster, _ = _layout(shapes)
    assert rc == 0
    assert cluster == 0 or not (start[:-1] % 32).any()


def test_any_pack_fits():
    """Half the nodes and a slot per odd row: without gaps the slots of any pack are in
    n_nodes, in order and without overlap."""
    rng = np.random.default_rng(7)
    for _ in range(400):
        dim, ni = int(rng.integers(2, 4)), int(rng.integers(1, 40))
        top = int(rng.choice([4, 8, 20, 70]))
        shapes = [tuple(int(v) for v in rng.integers(2, top, dim)) for _ in range(ni)]
        rc, start, cluster, n = _layout(shapes)
        slots = [(s[0] + 1) // 2 * int(np.prod(s[1:])) for s in shapes]
        assert rc == 0 and start[0] == 0 and start[-1] <= n, shapes
        assert (np.diff(start) >= slots).all(), shapes
        assert cluster == 0 or not (start[:-1] % 32).any(), shapes


def test_single_instances_keep_their_cluster():
    for shape, ctas in (((2, 2), 8), ((5, 3), 8), ((81, 41), 8), ((9, 7, 5), 8),
                        ((120, 120), 16), ((31, 22, 16), 16), ((201, 101), 0)):
        rc, start, cluster, _ = _layout([shape])
        assert (rc, start[0], cluster) == (0, 0, ctas), shape


@pytest.mark.parametrize("shape,n,ctas", [((20, 20), 2, 8), ((20, 20), 18, 8), ((20, 20), 19, 4),
                                          ((20, 20), 64, 2), ((20, 20), 1024, 1),
                                          ((60, 40), 16, 8), ((60, 40), 256, 4),
                                          ((120, 60), 16, 8), ((120, 60), 512, 8),
                                          ((118, 120), 2, 16), ((118, 120), 64, 16),
                                          ((14, 10, 9), 256, 2), ((30, 22, 16), 4, 16)])
def test_cluster_size_looks_at_the_batch(shape, n, ctas):
    """A batch's clusters all run at once (148 CTAs) unless they are the smallest that
    hold its largest instance (480 slots a CTA in 2D, 352 in 3D)."""
    rc, _, cluster, _ = _layout([shape] * n)
    slots, most = (shape[0] + 1) // 2 * int(np.prod(shape[1:])), 480 if len(shape) == 2 else 352
    assert (rc, cluster) == (0, ctas)
    assert slots <= cluster * most
    assert n * cluster <= 148 or cluster == 1 or slots > cluster // 2 * most
