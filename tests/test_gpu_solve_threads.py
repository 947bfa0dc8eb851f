"""Solves of different sizes from several host threads at once: the dynamic shared
memory that one thread's launch asks for is not limited by another's, so every solve
keeps its single launch (and the bits it has alone)."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [((81, 41), (21, 10), (64, 41), (9, 9)),
                                    ((181, 120), (221, 160), (170, 130), (251, 150))],
                         ids=["clusters", "grid"])
def test_threads_keep_the_single_launch(shapes):
    import torch
    from tcad_b200 import _lib
    from test_gpu_redblack import _scaled_system
    from test_gpu_resident import _device
    packs = [_scaled_system(_device("mosfet", s)) for s in shapes]
    lib, rounds, bad = packs[0].lib, 1500, []

    def solve(pk, x, stream):
        it, st, rr = ctypes.c_int32(0), ctypes.c_int32(0), ctypes.c_double(0.0)
        return lib.tcad_block_krylov(pk.pref, _lib.ptr(pk.J), _lib.ptr(pk.F), _lib.ptr(x), 2,
                                     1e-30, 1, 0, _lib.ptr(pk.work), pk.work.numel(),
                                     ctypes.byref(it), ctypes.byref(st), ctypes.byref(rr),
                                     ctypes.c_void_p(stream.cuda_stream))

    xs = [torch.full_like(pk.du, float("nan")) for pk in packs]
    streams = [torch.cuda.Stream() for _ in packs]
    torch.cuda.synchronize()
    for pk, x, s in zip(packs, xs, streams):
        _lib.check(solve(pk, x, s), "krylov")
    torch.cuda.synchronize()
    want = [x.cpu().numpy() for x in xs]
    n0 = lib.tcad_launch_count()

    def work(i):
        for _ in range(rounds):
            rc = solve(packs[i], xs[i], streams[i])
            if rc != _lib.TCAD_OK:
                bad.append(rc)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(packs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert not bad
    assert lib.tcad_launch_count() - n0 == 2 * len(packs) * rounds  # colour repack + solve
    for x, w in zip(xs, want):
        assert np.array_equal(x.cpu().numpy(), w)
