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
