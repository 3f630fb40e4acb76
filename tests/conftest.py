import os
import sys

import pytest

# The oracle's OpenMP threads would spin on every core for a while after each call (about 1.5 ms on 16 cores): a thread that
# then submits requests gets a time slice only when the serving engine's worker sleeps (100 us a submission instead of
# 8), which is not what a program that feeds the engine sees.  Read by the OpenMP runtime when it is loaded.
os.environ.setdefault("OMP_WAIT_POLICY", "passive")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs an sm_100 GPU (run with -m gpu on a B200)")
    config.addinivalue_line("markers", "slow: full-size workload")


@pytest.fixture(scope="session")
def ctx():
    import distance_transform_benchmarks_b200 as dtb
    c = dtb.Context(0)
    yield c
    c.close()
