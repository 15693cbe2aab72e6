"""The one-launch layer kernel (decode_fused.cu) on layers that are small enough for the three launches of few_one.cu,
which take them by default.  The path is pinned by an environment variable that is read once: a child process runs the
tests; a layer the pinned path does not take is an error there."""
import os
import subprocess
import sys

import pytest
import torch

from conftest import REL_FRO_TOL, ROOT, rel_fro

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


@pytest.mark.parametrize("hidden,ffn,top_k,n_shared", [
    (512, 24576, 6, 0),    # the down launch's tables leave no room for two stages
    (2048, 256, 2, 112),   # ... those of the shared expert
    (512, 21504, 6, 0),    # two stages fit, three do not
    (512, 16384, 6, 0),    # three fit
])
def test_layer_at_the_limit_of_shared_memory(hidden, ffn, top_k, n_shared):
    """Layers the few-row launches cannot hold go on to the other one-token paths."""
    from gemq_b200 import synth
    from test_gpu_configs import f16_abs_bound, max_abs, reference_rows
    if n_shared:
        blk, mode = synth.deepseek_block(seed=1, bits=[3, 2, 1], hidden_size=hidden, moe_intermediate_size=ffn, n_routed_experts=3,
                                         n_shared_experts=n_shared, num_experts_per_tok=top_k, shared_bits=3), 2
    else:
        blk, mode = synth.mixtral_block(seed=1, bits=[3, 1, 3, 2, 4, 3, 2], hidden_size=hidden, intermediate_size=ffn,
                                        num_local_experts=7, num_experts_per_tok=top_k), 0
    x = torch.randn(1, hidden, generator=torch.Generator().manual_seed(ffn)).half()
    out = blk(x.cuda().view(1, 1, -1))
    out = out[0] if isinstance(out, tuple) else out
    assert blk.decode_error_code() == 0
    _, gw, gi = blk._decode(x.cuda(), mode)
    ref = reference_rows(blk, x, gw.cpu(), gi.cpu(), hidden, ffn, shared_ffn=n_shared * ffn)
    got = out.view(1, -1).float().cpu().numpy()
    assert rel_fro(got, ref) < REL_FRO_TOL, rel_fro(got, ref)
    assert max_abs(got, ref) < f16_abs_bound(ref)
