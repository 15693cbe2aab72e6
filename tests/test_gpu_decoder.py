"""The one-token decode step's own kernels against the decoder's tensor operations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hidden,heads,kv_heads,hd,cache_len,positions", [
    (256, 4, 2, 64, 40, (0, 1, 31, 39)),              # shorter than one piece of the attention
    (512, 4, 4, 128, 1100, (63, 64, 511, 512, 1099)),  # one query head a key head; edges of a piece and of a round
    (768, 16, 2, 64, 600, (600 - 1,)),                 # eight query heads a key head
    (4096, 32, 8, 128, 700, (575, 640)),
])
def test_step_kernels_equal_tensor_operations(hidden, heads, kv_heads, hd, cache_len, positions, dtype):
    from gemq_b200.inference import MixtralDecoder, StaticCache
    model = MixtralDecoder(seed=5, dtype=dtype, hidden_size=hidden, intermediate_size=512, num_local_experts=4,
                           num_experts_per_tok=2, num_hidden_layers=2, num_attention_heads=heads,
                           num_key_value_heads=kv_heads, head_dim=hd, vocab_size=1000)
    gen = torch.Generator(device="cuda").manual_seed(7)
    for p in positions:
        caches = [StaticCache(model.config, cache_len) for _ in range(2)]
        for a, b in zip(*(c.layers for c in caches)):
            kv = torch.randn(2, 1, kv_heads, cache_len, hd, device="cuda", generator=gen).to(dtype)
            for layer in (a, b):
                layer.lazy_initialization(kv[0], kv[1])
                layer.keys.copy_(kv[0])
                layer.values.copy_(kv[1])
        tok = torch.randint(0, 1000, (1, 1), device="cuda", generator=gen)
        pos = torch.tensor([p], device="cuda")
        assert model._step_ok(model.embed_tokens(tok), caches[0], pos)
        got = model(tok, caches[0], pos).double()
        model._step_ok = lambda *a: False
        want = model(tok, caches[1], pos).double()
        del model._step_ok
        # both round the same values to `dtype` at the same places (per layer: two normalisations, the projections,
        # the rotation, the attention, its projection, the block, two sums); a place where the sums before it
        # fall on two sides of a rounding boundary differs by one unit in the last place, eps relative
        eps = torch.finfo(dtype).eps
        assert got.shape == want.shape
        assert float((got - want).norm() / want.norm()) < 2 * 9 * eps
        for a, b in zip(*(c.layers for c in caches)):
            for x, y in ((a.keys, b.keys), (a.values, b.values)):
                assert float((x.double() - y.double()).norm() / y.double().norm()) < 2 * 9 * eps
                rest = [i for i in range(cache_len) if i != p]
                assert torch.equal(x[:, :, rest], y[:, :, rest])


def test_step_writes_the_cache_of_the_layers_own_index():
    """A decoder whose first layer was dropped: prefill and step agree on the cache layers, and one layer short of
    cache is an error in both."""
    from gemq_b200.inference import MixtralDecoder, StaticCache
    model = MixtralDecoder(seed=5, hidden_size=256, intermediate_size=512, num_local_experts=4, num_experts_per_tok=2,
                           num_hidden_layers=3, num_attention_heads=4, num_key_value_heads=2, head_dim=64, vocab_size=96)
    model.layers = model.layers[1:]
    gen = torch.Generator(device="cuda").manual_seed(7)
    prompt, tok, pos = torch.randint(0, 96, (1, 9), device="cuda", generator=gen), torch.tensor([[3]], device="cuda"), \
        torch.tensor([9], device="cuda")
    caches = [StaticCache(model.config, 40) for _ in range(2)]
    for c in caches:
        model(prompt, c, torch.arange(9, device="cuda"))
        c.layers[0].lazy_initialization(*(torch.zeros(1, 2, 1, 64, dtype=torch.bfloat16, device="cuda") for _ in range(2)))
    assert model._step_ok(model.embed_tokens(tok), caches[0], pos)
    got = model(tok, caches[0], pos).double()
    model._step_ok = lambda *a: False
    want = model(tok, caches[1], pos).double()
    del model._step_ok
    assert not caches[0].layers[0].keys.any()
    assert float((got - want).norm() / want.norm()) < 2 * 9 * torch.finfo(torch.bfloat16).eps
    assert not torch.equal(caches[0].layers[2].keys[:, :, 9], torch.zeros_like(caches[0].layers[2].keys[:, :, 9]))
    caches[0].layers = caches[0].layers[:2]
    with pytest.raises(IndexError):
        model(tok, caches[0], pos)


def test_hooks_see_the_modules_of_a_step():
    """A hook that changes what a projection returns changes the step, as it does with the tensor operations."""
    from gemq_b200.inference import MixtralDecoder, StaticCache
    model = MixtralDecoder(seed=5, hidden_size=256, intermediate_size=512, num_local_experts=4, num_experts_per_tok=2,
                           num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=64, vocab_size=96)
    tok, pos = torch.tensor([[3]], device="cuda"), torch.tensor([4], device="cuda")
    outs = []
    for hooked, own in ((False, True), (True, True), (True, False)):
        c = StaticCache(model.config, 40)
        for layer in c.layers:
            layer.lazy_initialization(*(torch.zeros(1, 2, 1, 64, dtype=torch.bfloat16, device="cuda") for _ in range(2)))
        handle = model.layers[1].self_attn.v_proj.register_forward_hook(lambda m, a, y: -y) if hooked else None
        if not own:
            model._step_ok = lambda *a: False
        outs.append(model(tok, c, pos))
        if hooked:
            handle.remove()
    del model._step_ok
    assert not torch.equal(outs[0], outs[1]) and torch.equal(outs[1], outs[2])


@pytest.mark.parametrize("position", [-1, 40, 2 ** 40])
def test_position_outside_the_cache_is_visible(position):
    """The tensor operations refuse such a position; the step's kernels store nothing and give no numbers."""
    from gemq_b200.inference import MixtralDecoder, StaticCache
    model = MixtralDecoder(seed=5, hidden_size=256, intermediate_size=512, num_local_experts=4, num_experts_per_tok=2,
                           num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=64, vocab_size=96)
    c = StaticCache(model.config, 40)
    for layer in c.layers:
        layer.lazy_initialization(*(torch.zeros(1, 2, 1, 64, dtype=torch.bfloat16, device="cuda") for _ in range(2)))
    out = model(torch.tensor([[3]], device="cuda"), c, torch.tensor([position], device="cuda"))
    assert torch.isnan(out).all()
    assert not any(t.any() for layer in c.layers for t in (layer.keys, layer.values))
    assert all(layer.block_sparse_moe.decode_error_code() == 0 for layer in model.layers)
    assert torch.isfinite(model(torch.tensor([[3]], device="cuda"), c, torch.tensor([39], device="cuda"))).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,kv_heads,hd,cache_len,positions", [
    (4, 2, 64, 40, (0, 1, 31, 39)),                   # shorter than one piece of the attention
    (4, 4, 128, 1100, (63, 64, 511, 512, 1099)),      # one query head a key head; edges of a piece and of a round
    (6, 2, 128, 600, (0, 65, 448, 599)),              # three of four query heads
    (16, 2, 64, 600, (64, 599)),                      # eight query heads a key head
    (32, 8, 128, 700, (575, 576, 640)),
])
def test_step_attention_against_fp64(heads, kv_heads, hd, cache_len, positions, dtype):
    """The attention by itself: one position left out of 600 changes it by 4 %, the bound is one rounding."""
    from gemq_b200 import _capi
    from gemq_b200.inference.decoder import inverse_frequencies
    from gemq_b200.kernels._runtime import stream_ptr
    gen = torch.Generator(device="cuda").manual_seed(heads * cache_len)
    inv, G = inverse_frequencies(hd, 1e6, "cuda"), heads // kv_heads
    eps = torch.finfo(dtype).eps
    for p in positions:
        qkv = torch.randn((heads + 2 * kv_heads) * hd, device="cuda", generator=gen).to(dtype)
        keys, values = (torch.randn(kv_heads, cache_len, hd, device="cuda", generator=gen).to(dtype) for _ in range(2))
        k2, v2, out = keys.clone(), values.clone(), qkv.new_empty(heads * hd)
        pos = torch.tensor([p], device="cuda")
        assert _capi.lib.gemq_step_attention(qkv.data_ptr(), inv.data_ptr(), pos.data_ptr(), k2.data_ptr(), v2.data_ptr(), out.data_ptr(),
                                             heads, kv_heads, hd, cache_len, int(dtype == torch.bfloat16), stream_ptr(out.device)) == 0
        q, k, v = qkv.double().view(-1, hd).split([heads, kv_heads, kv_heads])
        ang = (float(p) * inv).double()  # an fp32 product, like the kernel's
        cos, sin = torch.cat([ang.cos()] * 2), torch.cat([ang.sin()] * 2)
        rot = lambda t: (t * cos + torch.cat([-t[:, hd // 2:], t[:, :hd // 2]], 1) * sin).to(dtype).double()
        q, k = rot(q), rot(k)
        # stored: the value itself, the rotated key up to a rounding that falls to the other side
        assert torch.equal(v2[:, p].double(), v) and ((k2[:, p].double() - k).abs() <= eps * k.abs() + 2.0 ** -20).all()
        rest = [i for i in range(cache_len) if i != p]
        assert torch.equal(k2[:, rest], keys[:, rest]) and torch.equal(v2[:, rest], values[:, rest])
        K, V = k2[:, :p + 1].double().repeat_interleave(G, 0), v2[:, :p + 1].double().repeat_interleave(G, 0)
        s = (K @ q[:, :, None])[:, :, 0] * hd ** -0.5
        want = (s.softmax(1)[:, None] @ V)[:, 0]
        # the output's rounding is at most eps / 2 of each value.  A rotated query element that was rounded to the other
        # side (one in some thousands) moves its head's scores by eps / sqrt(hd) of a product of order one; fp32 sums and
        # the fast exponential are below 2^-12.
        err = (out.double().view(heads, hd) - want).norm(dim=1) / want.norm(dim=1)
        assert float(err.max()) < 0.5 * eps + 2.0 ** -12 + eps * hd ** -0.5, (p, err.max())
