"""The autotuner's two kernels: the block kernel competes once, with the tuning the plan began with, and a result saved for
the tile kernel does not shut it out."""
import json

import numpy as np
import pytest
import torch

import distance_transform_benchmarks_b200 as dtb
from oracle import oracle as orc
from tests.helpers import assert_images_eq
from tests.test_gpu_tuning_routes import kernel_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def picture():
    """One even picture of 1024 blocks: the block kernel takes about half the tile kernel's time, and about 2800 activations
    for its 4096 tiles."""
    img, mask = np.full((2048, 2048), 9, np.uint8), np.zeros((2048, 2048), np.uint8)
    mask[700, 900] = 1
    return img, mask, 0.1, orc.ggdt_ns(img, mask, 0.1)


def plan_of(picture, c):
    img, mask, gamma, _ = picture
    return dtb.BatchPlan([dtb.pitched_from(img)], [dtb.pitched_from(mask)], [gamma], ctx=c)


def entry(path):
    entries = json.loads(path.read_text())["entries"]
    assert len(entries) == 1
    return entries[0]


def check(plan, picture, kernel):
    plan.dists[0].fill_(-1.0)
    plan.run()
    assert kernel_of(plan.wait(), 1) == kernel
    assert_images_eq(plan.dists[0], picture[3], kernel)


def test_the_block_kernel_wins_with_the_tuning_unchanged(picture, tmp_path):
    path = tmp_path / "tune.json"
    c = dtb.Context(0)
    c.set_tuning_cache(path)
    plan = plan_of(picture, c)
    before = plan.tuning()
    assert plan.autotune(reps=3) == before
    check(plan, picture, "blocks")
    assert entry(path)["blocks"] == 1
    plan.close()
    c.close()
    c = dtb.Context(0)  # and a program that loads the file runs the same
    c.set_tuning_cache(path)
    plan = plan_of(picture, c)
    assert plan.tuning() == before
    check(plan, picture, "blocks")
    plan.close()
    c.close()


def test_a_saved_tile_result_is_used_as_saved_and_does_not_shut_the_block_kernel_out(picture, tmp_path):
    path = tmp_path / "tune.json"
    saved = {"gpu": torch.cuda.get_device_name(0), "images_pow2": 1, "tiles_pow2": 4096, "ctas_per_sm": 3, "staging": 1,
             "warps_per_cta": 4, "grid_percent": 50, "queue_buckets": 16, "bucket_width_pct": 25, "ms": 0.5}
    path.write_text(json.dumps({"format": "dtb-autotune-1", "entries": [saved]}, indent=1))
    c = dtb.Context(0)
    c.set_tuning_cache(path)
    plan = plan_of(picture, c)
    assert plan.tuning()["queue_buckets"] == 16 and plan.tuning()["grid_percent"] == 50
    check(plan, picture, "tiles")
    plan.autotune(reps=3)
    check(plan, picture, "blocks")
    assert entry(path)["blocks"] == 1
    plan.close()
    c.close()


def test_the_callers_tuning_keeps_the_tile_kernel(picture, tmp_path):
    path = tmp_path / "tune.json"
    c = dtb.Context(0)
    c.set_tuning(ctas_per_sm=3)
    c.set_tuning_cache(path)
    plan = plan_of(picture, c)
    plan.autotune(reps=1)
    check(plan, picture, "tiles")
    assert entry(path)["blocks"] == 0
    plan.close()
    c.close()
