"""The one-launch layer kernel (decode_fused.cu) on layers that are small enough for the three launches of few_one.cu,
which take them by default.  The path is pinned by an environment variable that is read once: a child process runs the
tests; a layer the pinned path does not take is an error there."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

TESTS = [
    "test_gpu_configs.py::test_decode_three_bit_run_remainders",       # parts that end inside a 5-group run
    "test_gpu_configs.py::test_decode_wait_limit_expires_and_is_reported",
    "test_gpu_configs.py::test_expert_id_out_of_range_is_reported_not_used",
    "test_gpu_configs.py::test_config2_deepseek_real_shape",           # a shared slot, 64 experts routed outside
    "test_gpu_configs.py::test_decode_layer_is_bit_reproducible_over_many_graph_replays",
    "test_gpu_moe.py::test_mixtral_one_token_small",                   # routed inside, fewer CTAs than the chip has
]


def test_layer_tests_on_the_one_launch_kernel():
    ids = [os.path.join(ROOT, "tests", t) for t in TESTS]
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", "-p", "no:cacheprovider", *ids], cwd=ROOT,
                       env={**os.environ, "GEMQ_B200_DECODE": "persistent"}, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
    assert " passed" in r.stdout and "skipped" not in r.stdout, r.stdout[-500:]
