"""Which calls the decode step's own kernels take: decided on the host, so it can be asked without a GPU."""
from types import SimpleNamespace

import pytest
import torch
import torch.nn as nn

from gemq_b200.inference import QuantFusedMixtralMoEBlock, StaticCache
from gemq_b200.inference import decoder as D

CFG = dict(hidden_size=256, intermediate_size=512, num_local_experts=4, num_experts_per_tok=2, num_hidden_layers=3,
           num_attention_heads=4, num_key_value_heads=2, head_dim=64, vocab_size=96, rms_norm_eps=1e-5, rope_theta=1e6)


def model(dtype=torch.bfloat16):
    """The modules of a decoder without the quantised weights of its blocks."""
    m = D.MixtralDecoder.__new__(D.MixtralDecoder)
    nn.Module.__init__(m)
    m.config = SimpleNamespace(**CFG)
    lin = lambda n, k: nn.Linear(k, n, bias=False)
    m.embed_tokens = nn.Embedding(96, 256)
    m.layers = nn.ModuleList(D.DecoderLayer(m.config, i, QuantFusedMixtralMoEBlock(m.config), lin) for i in range(3))
    m.norm, m.lm_head = D.RMSNorm(256, 1e-5), lin(96, 256)
    m.to(dtype)
    m._init_rotary("cpu")
    return m


def cache(n=3, dtype=torch.bfloat16):
    c = StaticCache(SimpleNamespace(num_hidden_layers=n), 40)
    for layer in c.layers:
        layer.lazy_initialization(torch.zeros(1, 2, 1, 64, dtype=dtype), torch.zeros(1, 2, 1, 64, dtype=dtype))
    return c


def ok(m, c, pos=None):
    return m._step_ok(torch.zeros(1, 1, 256, dtype=torch.bfloat16), c, torch.tensor([5]) if pos is None else pos)


def test_cache_layers_are_found_by_the_layers_own_index():
    m = model()
    assert ok(m, cache()) and ok(m, cache(4))
    assert not ok(m, cache(2))          # the tensor operations raise for the third layer
    m.layers = m.layers[1:]             # layers 1 and 2 are left
    c = cache()
    assert ok(m, c)
    c.layers[0].is_initialized = False  # nobody's
    assert ok(m, c)
    c.layers[2].is_initialized = False
    assert not ok(m, c)


MODULES = [lambda m: m.layers[1], lambda m: m.layers[1].self_attn, lambda m: m.layers[1].self_attn.q_proj,
           lambda m: m.layers[1].self_attn.o_proj, lambda m: m.layers[1].input_layernorm,
           lambda m: m.layers[1].post_attention_layernorm, lambda m: m.layers[1].block_sparse_moe, lambda m: m.norm,
           lambda m: m.lm_head]


@pytest.mark.parametrize("pick", MODULES)
def test_modules_that_somebody_hooked_are_called(pick):
    m, c = model(), cache()
    sub = pick(m)
    for register in (sub.register_forward_hook, sub.register_forward_pre_hook):
        handle = register(lambda *a: None)
        assert not ok(m, c)
        handle.remove()
    assert ok(m, c)
    sub.forward = lambda *a: None  # an instance's own
    assert not ok(m, c)
    del sub.forward
    assert ok(m, c)


def test_replaced_modules_settings_and_caches_are_not_the_kernels():
    m, c = model(), cache()

    class Other(D.Attention):
        pass

    m.layers[1].self_attn.__class__ = Other
    assert not ok(m, c)
    m.layers[1].self_attn.__class__ = D.Attention
    moe, m.layers[0].block_sparse_moe = m.layers[0].block_sparse_moe, nn.Identity()
    assert not ok(m, c)
    m.layers[0].block_sparse_moe = moe
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    assert not ok(m, c)
    handle.remove()
    with torch.autocast("cuda", dtype=torch.float16, enabled=True):
        auto = torch.is_autocast_enabled("cuda")  # not without a device
        assert ok(m, c) != auto
    m.config.rope_theta = 1e4  # the tensor operations follow the configuration
    assert not ok(m, c)
    m.config.rope_theta = 1e6

    class OtherCache(StaticCache):
        def update(self, *a):
            raise NotImplementedError

    c.__class__ = OtherCache
    assert not ok(m, c)
    c.__class__ = StaticCache
    assert ok(m, c) and not ok(m, c, torch.tensor([5, 6])) and not ok(m, c, torch.tensor([5], dtype=torch.int32))
