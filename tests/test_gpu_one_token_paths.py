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


@pytest.mark.parametrize("D,Fd,SF,A,E", [
    (128, 128, 0, 1, 2),       # one slot; fewer stages than warps
    (256, 384, 0, 2, 4),
    (640, 256, 128, 1, 3),     # the shared expert is the shorter one; 3-bit runs that end inside a stage
    (384, 256, 896, 2, 5),     # ... the longer one
    (256, 1408, 512, 6, 40),   # seven slots: one part each
    (512, 384, 384, 7, 9),     # eight slots
    (256, 2048, 0, 8, 8),
    (2048, 1024, 0, 2, 44),
])
@pytest.mark.parametrize("shared_bits", [3, 4])
def test_few_row_launches_at_their_edges(D, Fd, SF, A, E, shared_bits):
    """Slots, cluster sizes and reduction lengths of the one-token few-row launches, routed and shared."""
    import numpy as np
    import moe_fixtures as MF
    from oracle import gemq_oracle as O
    if not SF and shared_bits == 4:
        pytest.skip("no shared expert")
    bits = [(3, 1, 4, 2)[e % 4] for e in range(E)]
    layer = MF.make_layer("mixtral", D=D, Fd=Fd, E=E, A=A, bits=bits, seed=D + Fd + A, gate_std=0.1)
    mode = 0
    if SF:
        rng = np.random.default_rng(SF)
        layer["shared"] = (MF.draw_linear(rng, SF, D, shared_bits), MF.draw_linear(rng, D, SF, shared_bits),
                           MF.draw_linear(rng, SF, D, shared_bits))
        c = layer["cfg"]
        c.moe_intermediate_size, c.n_routed_experts, c.n_shared_experts, c.norm_topk_prob = Fd, E, 1, False
        layer["family"], mode = "deepseek", 2
    blk = MF.gpu_block(layer)
    w1, w3, w2, sh = MF.oracle_parts(layer)
    x = torch.randn(3, D, generator=torch.Generator().manual_seed(A)).half()
    for t in range(3):
        out = blk(x[t].cuda().view(1, 1, -1))
        out = (out[0] if isinstance(out, tuple) else out).view(1, -1)
        assert blk.decode_error_code() == 0
        _, gw, gi = blk._decode(x[t:t + 1].cuda(), mode)
        ref = np.asarray(O.moe_reference_fp32(x[t:t + 1], gw.float().cpu(), gi.cpu(), w1, w3, w2, *([sh] if sh else [])), dtype=np.float32)
        assert rel_fro(out.float().cpu().numpy(), ref) < REL_FRO_TOL
