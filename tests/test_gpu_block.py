"""The block kernel (calls and plans of a context whose tuning was never set, up to about 38 Mpx) around the edges of its
64 x 64 blocks and of what one CTA owns, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import distance_transform_benchmarks_b200 as dtb
from distance_transform_benchmarks_b200 import workloads as wl
from oracle import oracle as orc
from tests.helpers import assert_images_eq, ns_fixpoint_violations

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fresh():
    c = dtb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("h,w", [(1, 65), (63, 64), (64, 63), (65, 129), (96, 160), (127, 1), (193, 257)])
@pytest.mark.parametrize("rgb", [False, True])
def test_block_edges_match_the_oracle(fresh, h, w, rgb):
    rng = np.random.default_rng(h * 1000 + w)
    img = rng.integers(0, 256, (h, w, 3) if rgb else (h, w), dtype=np.uint8)
    for k, v in ((1, 1e10), (5, 40.0), (0, 7.0)):  # 40 is reached, so part of the picture keeps v; no seed: all of it
        mask = np.zeros((h, w), np.uint8)
        for _ in range(k):
            mask[rng.integers(0, h), rng.integers(0, w)] = 255
        for gamma in (0.5, 0.0):
            d = dtb.geodesic_distance_transform(torch.from_numpy(img).cuda(), torch.from_numpy(mask).cuda(), gamma, v=v, ctx=fresh)
            assert_images_eq(d, orc.ggdt_ns(img, mask, gamma, v=v), "%dx%d seeds %d v %g gamma %g" % (h, w, k, v, gamma))


@pytest.mark.parametrize("n,smin,smax", [(1, 1200, 1300), (40, 2, 70), (700, 2, 100), (24, 64, 700)])
def test_ragged_batches_call_and_plan(fresh, n, smin, smax):
    """One image of more blocks than CTAs, and batches of up to several blocks per CTA, one image without seeds among
    them; a second run on the same buffers gives the same maps."""
    batch = [wl.make_image(s) for s in wl.config3_specs(n, n, smin, smax)]
    batch = [(i, np.zeros_like(m) if k == 3 else m, g) for k, (i, m, g) in enumerate(batch)]
    imgs = [dtb.pitched_from(b[0]) for b in batch]
    masks = [dtb.pitched_from(b[1]) for b in batch]
    gam = [b[2] for b in batch]
    want = [orc.ggdt_ns(*b) for b in batch]
    dists = [dtb.pitched_empty(b[1].shape[0], b[1].shape[1], 1, torch.float32) for b in batch]
    plan = dtb.BatchPlan(imgs, masks, gam, dists=dists, ctx=fresh)
    for run in range(2):
        dtb.geodesic_distance_transform_batch(imgs, masks, gam, dists=dists, ctx=fresh)
        for k in range(n):
            assert_images_eq(dists[k], want[k], "call %d image %d" % (run, k))
            dists[k].fill_(-1.0)
        plan.run()
        st = plan.wait()
        assert st["device_error"] == 0 and st["tile_visits"] > 0
        for k in range(n):
            assert_images_eq(dists[k], want[k], "plan run %d image %d" % (run, k))
            dists[k].fill_(-1.0)


def test_both_sides_of_the_size_rule_are_fixpoints():
    """6208 x 6208 has 9409 blocks (block kernel), 6272 x 6272 has 9604 (tile kernel, on 148 SMs)."""
    for side in (6208, 6272):
        img, mask, gamma = wl.config2(5, side, side)
        c = dtb.Context(0)
        ti, tm = dtb.pitched_from(img), dtb.pitched_from(mask)
        d = dtb.geodesic_distance_transform(ti, tm, gamma, ctx=c)
        va, vb, _ = ns_fixpoint_violations(ti, tm, gamma, 1e10, d)
        assert (va, vb) == (0, 0), "side %d: %d pixels could fall, %d have no source" % (side, va, vb)
        c.close()


@pytest.mark.parametrize("h,w", [(1, 1), (1, 65), (33, 31), (63, 64), (64, 64), (65, 129), (96, 160), (193, 257)])
@pytest.mark.parametrize("lam", [0.0, 0.3, 1.0])
def test_ref_mode_blocks_tiles_and_rounds(fresh, h, w, lam):
    """Reference weight: the block kernel, the tile kernel (a context with a tuning of its own) and the host-driven rounds,
    with and without FMA, from seeds in each corner (fronts that cross blocks over their corners) and none."""
    rng = np.random.default_rng(h * 1000 + w)
    tiles = dtb.Context(0)
    tiles.set_tuning(ctas_per_sm=2)
    for kind in ("noise", "flat", "steps"):
        img = (rng.integers(0, 256, (h, w)) if kind == "noise" else np.zeros((h, w)) if kind == "flat"
               else np.add.outer(np.arange(h) // 7 * 40, np.arange(w) // 5 * 30) % 256).astype(np.uint8)
        for y, x, v in ((0, 0, 1e10), (h - 1, 0, 1e10), (0, w - 1, 60.0), (h - 1, w - 1, 1e10), (-1, -1, 5.0)):
            mask = np.zeros((h, w), np.uint8)
            if y >= 0:
                mask[y, x] = 1
            ti, tm = torch.from_numpy(img).cuda(), torch.from_numpy(mask).cuda()
            for fma in (True, False):
                want = orc.ggdt_ref(img, mask, lam, v, fma)
                what = "%s %dx%d lambda %g seed (%d, %d) fma %d: " % (kind, h, w, lam, y, x, fma)
                assert_images_eq(dtb.generalised_distance_transform_task(ti, tm, lam, v, ctx=fresh, fma=fma), want, what + "blocks of tiles")
                assert_images_eq(dtb.generalised_distance_transform_task(ti, tm, lam, v, ctx=tiles, fma=fma), want, what + "tiles")
                assert_images_eq(dtb.generalised_distance_transform_blocks(ti, tm, lam, v, ctx=fresh, fma=fma), want, what + "rounds")
    tiles.close()


@pytest.mark.parametrize("tuned", [False, True])
def test_wave_edits_through_either_kernel(tuned):
    """Serve waves run the block kernel under the default tuning and the tile kernel under one of the caller's: new images
    and repeated seed edits (inside, across blocks, on old seeds, outside the picture) equal cold runs on all seeds."""
    c = dtb.Context(0)
    if tuned:
        c.set_tuning(ctas_per_sm=2)
    srv = dtb.Server(1 << 28, ctx=c)
    rng = np.random.default_rng(4)
    imgs = [rng.integers(0, 256, (150, 333, 3), dtype=np.uint8), rng.integers(0, 256, (64, 65), dtype=np.uint8)]
    masks = [np.zeros(i.shape[:2], np.uint8) for i in imgs]
    masks[0][5, 7] = masks[1][63, 0] = 1

    def ask(n, outs):
        for _ in range(n):
            for a in srv.poll(8, wait_ms=5000):
                assert a["status"] == 0
                n -= 1
            if n <= 0:
                break
        for k, o in outs:
            assert_images_eq(o, orc.ggdt_ns(imgs[k], masks[k], 0.2), "image %d tuned %d" % (k, tuned))

    outs = [(k, torch.empty(imgs[k].shape[:2])) for k in range(2)]
    for k, o in outs:
        srv.submit_image(k, imgs[k], masks[k], 0.2, o)
    ask(2, outs)
    for disks in ([(330, 149, 2)], [(64, 63, 3)], [(7, 5, 0)], [(500, 500, 4)], [(0, 0, 1), (63, 64, 2)]):
        outs = []
        for k in range(2):
            h, w = masks[k].shape
            yy, xx = np.mgrid[:h, :w]
            for x, y, r in disks:
                masks[k][(xx - x) ** 2 + (yy - y) ** 2 <= r * r] = 1
            outs.append((k, torch.empty((h, w))))
            srv.submit_edit(k, disks, outs[-1][1])
        ask(2, outs)
    srv.close()
    c.close()


def test_large_batch_defaults_are_fixpoints():
    """A plan above the size at which untuned batches change their launch shape and queue policy (96k tiles, 32 images):
    every map passes the fixpoint check, and a call on the same images gives the same maps."""
    specs = wl.config3_specs(9, 260, 512, 2048)
    c = dtb.Context(0)
    batch = [wl.make_image(s) for s in specs]
    assert sum(-(-b[1].shape[0] // 32) * -(-b[1].shape[1] // 32) for b in batch) >= 96 * 1024
    imgs, masks = [dtb.pitched_from(b[0]) for b in batch], [dtb.pitched_from(b[1]) for b in batch]
    gam = [b[2] for b in batch]
    dists = [dtb.pitched_empty(b[1].shape[0], b[1].shape[1], 1, torch.float32) for b in batch]
    plan = dtb.BatchPlan(imgs, masks, gam, dists=dists, ctx=c)
    plan.run()
    assert plan.wait()["device_error"] == 0
    first = [d.clone() for d in dists]
    for k in range(len(batch)):
        assert ns_fixpoint_violations(imgs[k], masks[k], gam[k], 1e10, dists[k])[:2] == (0, 0), k
        dists[k].fill_(-1.0)
    dtb.geodesic_distance_transform_batch(imgs, masks, gam, dists=dists, ctx=c)
    assert all(torch.equal(a, b) for a, b in zip(first, dists))
    plan.close()
    c.close()
