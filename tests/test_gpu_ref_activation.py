"""Reference weight: a visit activates the neighbours that its border can lower, and no others, also from tiles that the
picture fills in part."""
import numpy as np
import pytest
import torch

import distance_transform_benchmarks_b200 as dtb
from oracle import oracle as orc
from tests.helpers import assert_images_eq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(64, 33), (33, 64), (65, 40), (70, 31), (31, 70), (64, 64), (95, 95)])
@pytest.mark.parametrize("lam", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("fma", [True, False])
def test_nothing_is_activated_where_no_pixel_can_fall(ctx, h, w, lam, fma):
    """v = 0: every pixel begins at 0, so every seeded tile is visited once and brings nothing to anybody."""
    img = np.random.default_rng(h * w).integers(0, 256, (h, w), dtype=np.uint8)
    mask = np.ones((h, w), np.uint8)
    d = dtb.generalised_distance_transform_task(torch.from_numpy(img).cuda(), torch.from_numpy(mask).cuda(), lam, 0.0, ctx=ctx, fma=fma)
    assert_images_eq(d, np.zeros((h, w), np.float32))
    st = ctx.stats()
    assert st["activations"] == 0 and st["tile_visits"] == st["tiles"], st


@pytest.mark.parametrize("h,w", [(97, 33), (33, 97), (65, 65), (40, 100), (34, 66)])
@pytest.mark.parametrize("v", [1e10, float("inf"), 30.0])
def test_maps_of_pictures_with_partial_tiles(ctx, h, w, v):
    """Fronts that reach the partial tiles and come back out of them over their corners, and pixels that stay at v."""
    rng = np.random.default_rng(h + 1000 * w)
    for img in (rng.integers(0, 256, (h, w), dtype=np.uint8), np.full((h, w), 9, np.uint8)):
        for y, x in ((0, 0), (h - 1, w - 1), (h - 1, 0), (0, w - 1), (h // 2, w - 1), (h - 1, w // 2)):
            mask = np.zeros((h, w), np.uint8)
            mask[y, x] = 1
            for lam in (0.0, 0.4, 1.0):
                d = dtb.generalised_distance_transform_task(torch.from_numpy(img).cuda(), torch.from_numpy(mask).cuda(), lam, v, ctx=ctx)
                assert_images_eq(d, orc.ggdt_ref(img, mask, lam, v), "%dx%d seed (%d, %d) lambda %g v %g" % (h, w, y, x, lam, v))
