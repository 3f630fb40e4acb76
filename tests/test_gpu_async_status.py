"""An asynchronous device call and host-buffer batches open at the same time: one sync waits for both, no error is lost, and
the statistics are those of the call that came last."""
import numpy as np
import pytest
import torch

import distance_transform_benchmarks_b200 as dtb
from distance_transform_benchmarks_b200 import workloads as wl
from oracle import oracle as orc
from tests.helpers import assert_images_eq

pytestmark = pytest.mark.gpu

DTB_ERR_TIMEOUT = 4


@pytest.fixture
def work():
    """A context, a device picture of 256 tiles with its map, and a host batch with its maps."""
    c = dtb.Context(0)
    img, mask, gamma = wl.config0()
    batch = wl.config3(seed=71, n=5, smin=30, smax=200)
    hi, hm, hd = dtb.host_batch_arena([b[0] for b in batch], [b[1] for b in batch])
    ti, tm = torch.from_numpy(img).cuda(), torch.from_numpy(mask).cuda()
    dist = torch.empty(img.shape, device="cuda")

    def device(asynchronous):
        dtb.geodesic_distance_transform_batch([ti], [tm], [gamma], dists=[dist], ctx=c, asynchronous=asynchronous)

    def host(asynchronous):
        dtb.geodesic_distance_transform_batch(hi, hm, [b[2] for b in batch], dists=hd, ctx=c, asynchronous=asynchronous)

    def check():
        assert_images_eq(dist, orc.ggdt_ns(img, mask, gamma), "device map")
        for k, b in enumerate(batch):
            assert_images_eq(hd[k], orc.ggdt_ns(*b), "host map %d" % k)

    tiles = sum(-(-b[0].shape[0] // 32) * -(-b[0].shape[1] // 32) for b in batch)
    yield c, device, host, check, tiles
    c.close()


def test_a_stalled_device_call_is_reported_past_a_host_batch(work):
    c, device, host, check, tiles = work
    for asynchronous in (True, False):
        c.inject_queue_stall(100)
        device(True)
        host(asynchronous)
        with pytest.raises(dtb.DtbError) as e:
            c.sync()
        assert e.value.status == DTB_ERR_TIMEOUT and "no progress" in str(e.value)
        c.sync()  # reported once
        device(True)
        host(True)
        c.sync()
        assert c.stats()["tiles"] == tiles  # of the batch, which came last
        check()


def test_a_device_call_after_an_open_host_batch_has_its_own_statistics(work):
    c, device, host, check, tiles = work
    host(True)
    device(False)
    assert c.stats()["tiles"] == 256 and c.stats()["rounds"] == 1
    check()
    host(True)
    device(True)
    c.sync()
    assert c.stats()["tiles"] == 256
    check()
    host(False)
    assert c.stats()["tiles"] == tiles


def test_a_call_on_another_stream_follows_an_open_one(work):
    """The device call leaves its scratch to the next stream's call only when it has ended, a host batch in between or not."""
    c, device, host, check, tiles = work
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(6):
        with torch.cuda.stream(streams[k % 2]):
            device(True)
            if k % 3 == 0:
                host(True)
    c.sync()
    torch.cuda.synchronize()
    check()
