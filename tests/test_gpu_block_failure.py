"""What the block kernel does after an error: no block is claimed any more, ready or not, and the visit cap also ends a run
whose CTAs never wait.  The kernel is launched from a test library that sets its launch words (no device fault)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

import distance_transform_benchmarks_b200 as dtb
from distance_transform_benchmarks_b200 import build as dtb_build
from distance_transform_benchmarks_b200 import workloads as wl
from oracle import oracle as orc
from tests.helpers import assert_images_eq

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DERR_TMA_TIMEOUT, DERR_VISIT_LIMIT = 2, 5


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cuda") / "libblock_checks.so")
    cmd = [dtb_build._nvcc()] + dtb_build.ARCH + dtb_build.NVCC_FLAGS + [
        "-I" + dtb_build.INCLUDE, "-I" + dtb_build.CSRC, "-shared", "-o", out, os.path.join(ROOT, "tests", "cuda", "block_checks.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    torch.zeros(1, device="cuda")  # the library launches in torch's context
    return ctypes.CDLL(out)


def run(checks, img, mask, gamma, error=0, max_visits=0xF0000000):
    h, w = img.shape
    ti, tm = dtb.pitched_from(img), dtb.pitched_from(mask)
    d = dtb.pitched_empty(h, w, 1, torch.float32)
    d.fill_(-1.0)
    torch.cuda.synchronize()
    out = (ctypes.c_uint32 * 4)()
    p = ctypes.c_void_p
    i64 = ctypes.c_int64
    rc = checks.block_run(p(ti.data_ptr()), i64(ti.stride(0)), p(tm.data_ptr()), i64(tm.stride(0)), p(d.data_ptr()),
                          i64(4 * d.stride(0)), w, h, ctypes.c_float(np.float32(gamma) * np.float32(gamma)), ctypes.c_float(1e10),
                          ctypes.c_uint32(error), ctypes.c_uint32(max_visits), out)
    assert rc == 0, rc
    return d, dict(zip(("error", "info", "visits", "blocks"), out))


def test_no_block_is_visited_after_an_error(checks):
    img, mask, gamma = wl.config0()
    d, st = run(checks, img, mask, gamma)
    assert st["error"] == 0 and st["visits"] >= st["blocks"]
    assert_images_eq(d, orc.ggdt_ns(img, mask, gamma), "run without an error")
    _, st = run(checks, img, mask, gamma, error=DERR_TMA_TIMEOUT)
    assert st["error"] == DERR_TMA_TIMEOUT and st["visits"] == 0, st


def test_the_visit_cap_ends_a_run_whose_ctas_never_wait(checks):
    """A seed in each of the 94 x 94 blocks: every CTA has about 30 blocks ready from the start."""
    side = 94 * 64
    img = np.random.default_rng(3).integers(0, 256, (side, side), dtype=np.uint8)
    mask = np.zeros((side, side), np.uint8)
    mask[10::64, 20::64] = 1
    _, st = run(checks, img, mask, 0.1, max_visits=64)
    # A CTA looks at the cap at its 16th visit at the latest, and then nobody claims another block.
    assert st["error"] == DERR_VISIT_LIMIT and st["info"] > 64, st
    assert st["visits"] < 4 * 0.75 * st["blocks"], st  # a visit sweeps up to four tiles


def test_a_copy_that_does_not_arrive_ends_the_warp(checks):
    out = (ctypes.c_uint32 * 4)()
    assert checks.lost_copy(out) == 0
    assert tuple(out) == (0, 1, DERR_TMA_TIMEOUT, 77)
