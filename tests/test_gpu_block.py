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
