"""sqrt_ge1, the root in every ns-mode weight, is the correctly rounded one for each float it can be given."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

from distance_transform_benchmarks_b200 import build as dtb_build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_float_from_one_to_infinity(tmp_path):
    out = str(tmp_path / "libsqrt_checks.so")
    cmd = [dtb_build._nvcc()] + dtb_build.ARCH + dtb_build.NVCC_FLAGS + ["-I" + dtb_build.CSRC, "-shared", "-o", out,
                                                                       os.path.join(ROOT, "tests", "cuda", "sqrt_checks.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    torch.zeros(1, device="cuda")
    first, last = (int(np.float32(x).view(np.uint32)) for x in (1.0, np.inf))
    assert last - first + 1 == 1073741825  # all of them: 128 binades of 2^23 floats, and infinity
    res = (ctypes.c_ulonglong * 2)()
    assert ctypes.CDLL(out).sqrt_mismatches(ctypes.c_uint32(first), ctypes.c_uint32(last), res) == 0
    assert res[0] == 0, "%d roots differ, the first of 0x%08x" % (res[0], res[1])
