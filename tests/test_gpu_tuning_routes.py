"""Which kernel a call takes after which tuning, and host batches of many chunks through either kernel."""
import numpy as np
import pytest
import torch

import distance_transform_benchmarks_b200 as dtb
from distance_transform_benchmarks_b200 import workloads as wl
from oracle import oracle as orc
from tests.helpers import assert_images_eq

pytestmark = pytest.mark.gpu


def kernel_of(stats, images):
    """The kernel that made maps of wholly reached pictures with one seeded tile each: the tile kernel activates every other
    tile at least once, the block kernel crosses the tiles of its 64 x 64 blocks without (in these tests it needs fewer
    activations than there are tiles)."""
    return "blocks" if stats["activations"] < stats["tiles"] - images else "tiles"


def set_nothing(c):
    pass


def set_chunk(c):
    c.set_tuning(host_chunk_kpx=24)


def set_launch(c):
    c.set_tuning(ctas_per_sm=3, host_chunk_kpx=24)


def set_and_return(c):
    defaults = c.get_tuning()
    c.set_tuning(ctas_per_sm=3, queue_buckets=16)
    c.set_tuning(**dict(defaults, host_chunk_kpx=24))


def set_launch_then_chunk(c):
    c.set_tuning(ctas_per_sm=2)
    c.set_tuning(host_chunk_kpx=24)


@pytest.mark.parametrize("change,kernel", [(set_nothing, "blocks"), (set_chunk, "blocks"), (set_launch, "tiles"),
                                           (set_and_return, "blocks"), (set_launch_then_chunk, "tiles")])
def test_the_chunk_size_alone_keeps_the_choice_by_size(change, kernel):
    c = dtb.Context(0)
    change(c)
    img = wl.blobs_gray(3, 64, 64)
    mask = np.zeros((64, 64), np.uint8)
    mask[20, 40] = 1
    want = orc.ggdt_ns(img, mask, 0.1)
    d = dtb.geodesic_distance_transform(torch.from_numpy(img).cuda(), torch.from_numpy(mask).cuda(), 0.1, ctx=c)
    assert_images_eq(d, want, "device call")
    assert kernel_of(c.stats(), 1) == kernel
    hi, hm, hd = dtb.host_batch_arena([img] * 9, [mask] * 9)
    dtb.geodesic_distance_transform_batch(hi, hm, [0.1] * 9, dists=hd, ctx=c)
    assert kernel_of(c.stats(), 9) == kernel
    for k in range(9):
        assert_images_eq(hd[k], want, "host image %d" % k)
    c.close()


@pytest.mark.parametrize("tile_kernel", [False, True])
@pytest.mark.parametrize("chunk_kpx", [8, 64, 16384])
def test_host_batches_of_many_chunks(chunk_kpx, tile_kernel):
    """Synchronous calls (their last chunks shrink) and asynchronous ones behind each other, arenas and single planes, batches
    of few and of many images; a stalled call in between is reported and the next calls are right."""
    c = dtb.Context(0)
    c.set_tuning(host_chunk_kpx=chunk_kpx, ctas_per_sm=2 if tile_kernel else 0)
    batches = [wl.config3(seed=60 + k, n=n, smin=16, smax=smax) for k, (n, smax) in enumerate(((3, 500), (40, 150), (17, 300)))]
    want = [[orc.ggdt_ns(*b) for b in batch] for batch in batches]
    arenas = [dtb.host_batch_arena([b[0] for b in batch], [b[1] for b in batch]) for batch in batches]
    arenas[2][0][4] = torch.from_numpy(batches[2][4][0].copy())

    def call(k, asynchronous):
        hi, hm, hd = arenas[k]
        dtb.geodesic_distance_transform_batch(hi, hm, [b[2] for b in batches[k]], dists=hd, ctx=c, asynchronous=asynchronous)

    def check(what):
        for k, (_, _, hd) in enumerate(arenas):
            for j, d in enumerate(hd):
                assert_images_eq(d, want[k][j], "%s: batch %d image %d" % (what, k, j))
                d.fill_(-1.0)

    for k in range(3):
        call(k, False)
        if chunk_kpx == 8:
            assert c.stats()["rounds"] >= 3  # chunks (of three images or more)
    check("synchronous")
    for k in (2, 0, 1):
        call(k, True)
    c.sync()
    check("asynchronous")
    c.inject_queue_stall(100)
    with pytest.raises(dtb.DtbError) as e:
        call(1, False)
    assert e.value.status == 4
    for k in range(3):
        call(k, False)
    check("after the stall")
    c.close()
