"""The tile sweeps where they can go wrong: fronts that enter a tile at each corner and along each side, paths inside
a tile that turn many times (spirals and serpentines, which need many rounds and both skewed layouts), and sides
around the tile size, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import distance_transform_benchmarks_b200 as dtb
from oracle import oracle as orc
from tests.helpers import assert_images_eq

pytestmark = pytest.mark.gpu


def spiral(h, w):
    """Walls of 255 on 0, one pixel wide, winding towards the middle with corridors of one pixel."""
    img = np.zeros((h, w), np.uint8)
    y0, x0, y1, x1 = 0, 0, h - 1, w - 1
    while y1 - y0 >= 4 and x1 - x0 >= 4:
        img[y0 + 1, x0:x1] = 255
        img[y0 + 1:y1, x1 - 1] = 255
        img[y1 - 1, x0 + 1:x1] = 255
        img[y0 + 3:y1, x0 + 1] = 255
        y0, x0, y1, x1 = y0 + 2, x0 + 2, y1 - 2, x1 - 2
    return img


def serpentine(h, w):
    img = np.zeros((h, w), np.uint8)
    for k, y in enumerate(range(1, h, 2)):
        img[y] = 255
        img[y, 0 if k % 2 else w - 1] = 0
    return img


def picture(content, h, w, seed):
    rng = np.random.default_rng(seed)
    if content == "spiral":
        return spiral(h, w)
    if content == "serpentine":
        return serpentine(h, w)
    if content == "columns":
        return np.ascontiguousarray(serpentine(w, h).T)
    if content == "noise_rgb":
        return rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    return rng.integers(0, 256, (h, w), dtype=np.uint8)


@pytest.mark.parametrize("h,w", [(1, 1), (2, 33), (33, 2), (31, 31), (32, 32), (33, 33), (32, 64), (97, 95)])
@pytest.mark.parametrize("content", ["spiral", "serpentine", "columns", "noise", "noise_rgb"])
def test_sweeps_from_every_corner_and_side(ctx, content, h, w):
    img = picture(content, h, w, 17 * h + w)
    seeds = {(0, 0), (h - 1, 0), (0, w - 1), (h - 1, w - 1), (h // 2, 0), (0, w // 2), (h // 2, w - 1), (h - 1, w // 2)}
    for gamma in (1.0, 0.02):
        for y, x in sorted(seeds):
            mask = np.zeros((h, w), np.uint8)
            mask[y, x] = 1
            d = dtb.geodesic_distance_transform(torch.from_numpy(img).cuda(), torch.from_numpy(mask).cuda(), gamma, ctx=ctx)
            assert_images_eq(d, orc.ggdt_ns(img, mask, gamma), "%s %dx%d gamma %g seed (%d, %d)" % (content, h, w, gamma, y, x))
