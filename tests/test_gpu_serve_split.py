"""A wave is closed at its request limit while requests wait, whatever the speed of the submitting thread."""
import time

import pytest
import torch

import distance_transform_benchmarks_b200 as dtb
from distance_transform_benchmarks_b200 import workloads as wl
from oracle import oracle as orc
from tests.helpers import assert_images_eq, ns_fixpoint_violations

pytestmark = pytest.mark.gpu


def test_waves_split_while_a_large_image_runs():
    """The 4096 x 4096 maze takes several milliseconds on the device; the first small image takes the engine's second wave
    behind it, and the others wait until the maze is done: the next wave is closed at one request with others left."""
    maze, mmask, mg = wl.config1()
    small = wl.config3(seed=58, n=8, smin=100, smax=300)
    srv = dtb.Server(1 << 30, max_wave_requests=1)
    pin = [(torch.from_numpy(i).pin_memory(), torch.from_numpy(m).pin_memory(), g) for i, m, g in [(maze, mmask, mg)] + small]
    outs = [torch.empty(p[0].shape[:2], dtype=torch.float32).pin_memory() for p in pin]
    for k, ((i, m, g), out) in enumerate(zip(pin, outs)):
        srv.submit_image(k, i, m, g, out)
    left, t0 = len(pin), time.time()
    while left and time.time() - t0 < 60:
        for c in srv.poll(wait_ms=50):
            assert c["status"] == 0
            left -= 1
    assert left == 0
    st = srv.stats()
    assert st["waves"] == len(pin) and st["failed"] == 0 and st["waves_split"] >= 1, st
    for k, (i, m, g) in enumerate(small):
        assert_images_eq(outs[1 + k], orc.ggdt_ns(i, m, g), "small image %d" % k)
    assert ns_fixpoint_violations(pin[0][0].cuda(), pin[0][1].cuda(), mg, 1e10, outs[0].cuda())[:2] == (0, 0)
    srv.close()
