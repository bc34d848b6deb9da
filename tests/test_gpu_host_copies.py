"""Host volumes and host results large enough for the threaded copies through pinned
slots (from 8 MiB, in 2 MiB pieces): the bits of the device-memory call, for sizes at
the edges of a piece, pinned memory (copied directly), a slice that starts at an odd
address, and several contexts at once."""
import threading

import numpy as np
import pytest

from ctl_b200 import geometry as G
from ctl_b200.projector import Context, Settings, VoxelVolume

pytestmark = pytest.mark.gpu


def _volume(shape_xyz, seed):
    return np.random.default_rng(seed).uniform(0.0, 0.05, shape_xyz[::-1]).astype(np.float32)


def _device(vol, P, C, R):
    import torch
    d, p = torch.from_numpy(vol).cuda(), torch.from_numpy(P).cuda()
    torch.cuda.synchronize()
    with Context(0) as c:
        v = c.volume(VoxelVolume(d, (1.0, 1.0, 1.0)))
        return c.project(v, p, C, R, Settings()).cpu().numpy()


@pytest.mark.parametrize("shape,views,C,R", [
    ((40, 40, 40), 32, 256, 256),     # result 8 MiB, volume copied directly
    ((40, 40, 40), 71, 331, 97),      # several chunks, ragged pieces
    ((128, 128, 128), 3, 64, 64),     # volume 8 MiB, result copied directly
    ((161, 133, 127), 9, 512, 513),   # both, ragged
])
def test_pageable_memory_gives_the_device_calls_bits(shape, views, C, R):
    vol = _volume(shape, 1)
    P = G.circular_flat(views, 750.0, 1000.0, G.FlatDetector(C, R, 0.7, 0.7))
    want = _device(vol, P, C, R)
    with Context(0) as c:
        for _ in range(2):
            np.testing.assert_array_equal(c.project_volume(VoxelVolume(vol, (1.0, 1.0, 1.0)), P, C, R), want)
        # a result behind other data, at an address that is no multiple of 16
        room = np.full(want.size + 8, np.float32(7.0))
        out = room[5:5 + want.size].reshape(want.shape)
        c.project_volume(VoxelVolume(vol, (1.0, 1.0, 1.0)), P, C, R, out=out)
        np.testing.assert_array_equal(out, want)
        assert (room[:5] == 7.0).all() and (room[5 + want.size:] == 7.0).all()


def test_pinned_memory_gives_the_same_bits():
    import torch
    vol = _volume((140, 120, 130), 2)
    P = G.circular_flat(30, 750.0, 1000.0, G.FlatDetector(300, 256, 0.8, 0.8))
    want = _device(vol, P, 300, 256)
    out = torch.empty(want.shape, dtype=torch.float32, pin_memory=True)
    with Context(0) as c:
        c.project_volume(VoxelVolume(torch.from_numpy(vol).pin_memory(), (1.0, 1.0, 1.0)), P, 300, 256, out=out)
    np.testing.assert_array_equal(out.numpy(), want)


def test_contexts_in_several_threads_copy_at_once():
    jobs = []
    for k in range(3):
        vol = _volume((130, 129, 128 + k), 10 + k)
        P = G.circular_flat(24 + k, 750.0, 1000.0, G.FlatDetector(320, 300, 0.8, 0.8), start=0.3 * k)
        jobs.append((vol, P, _device(vol, P, 320, 300)))
    got = [None] * len(jobs)

    def run(k):
        vol, P, _ = jobs[k]
        with Context(0) as c:
            got[k] = [c.project_volume(VoxelVolume(vol, (1.0, 1.0, 1.0)), P, 320, 300) for _ in range(3)]

    ts = [threading.Thread(target=run, args=(k,)) for k in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k, (_, _, want) in enumerate(jobs):
        for g in got[k]:
            np.testing.assert_array_equal(g, want)
