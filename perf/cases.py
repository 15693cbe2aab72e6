"""The work whose speed is measured: calls a user of the package makes, over the range in which they are used.

Every case goes through the package's public entry points only: the quantised MoE blocks
(``QuantFusedMixtralMoEBlock``, ``QuantFusedDeepseekV2MoEBlock``), the quantised dense layer
(``QuantLinear``), the one-row operator (``dequant_splitk_gemv``) and the captured decode step of
``MixtralDecoder``.  Weights are drawn like the benchmark layers in ``gemq_b200.synth``: uniform codes,
group 128 along the reduction, fp16 scale and offset, 1 to 4 bits per expert.
"""
from __future__ import annotations

import random
from types import SimpleNamespace

import torch

from gemq_b200 import synth
from gemq_b200.inference import (MixtralDecoder, QuantFusedDeepseekV2MoEBlock, QuantFusedMixtralMoEBlock, QuantLinear,
                                 StaticCache)
from gemq_b200.kernels import dequant_splitk_gemv

GROUP = 128
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
# Bit widths of eight experts, mean 2.0: the middle of the 1.5 .. 2.5 bits per expert the layers are quantised to.
EXPERT_BITS = (2, 1, 3, 2, 1, 4, 2, 1)

MIXTRAL = dict(kind="mixtral", hidden=4096, ffn=14336, experts=8, top_k=2)
DEEPSEEK = dict(kind="deepseek", hidden=2048, ffn=1408, experts=64, shared=2, top_k=6, norm=False)


def listed():
    return [
        # A key / value projection quantised to 4 bits, one decoded token: the smallest call a decode step makes.
        dict(name="linear_kv_1", kind="linear", rows=1, inf=4096, outf=1024, bits=4, dtype="bf16", bias=False),
        # One expert's gate projection at 2 bits for one token, called as an operator.
        dict(name="gemv_expert_1", kind="gemv", inf=4096, outf=14336, bits=2),
        # A 4-bit attention projection under a small decode batch (an odd number of sequences).
        dict(name="linear_rows_13", kind="linear", rows=13, inf=4096, outf=4096, bits=4, dtype="bf16", bias=False),
        # The same projection over a prompt.
        dict(name="linear_rows_1000", kind="linear", rows=1000, inf=4096, outf=4096, bits=4, dtype="bf16", bias=False),
        # Mixtral-8x7B MoE layer, decode with one sequence: the layer the package exists for.
        dict(name="mixtral_token_1", **MIXTRAL, tokens=1, dtype="fp16", skew=0.0),
        # ... with 32 sequences: every expert is read for a handful of rows.
        dict(name="mixtral_batch_32", **MIXTRAL, tokens=32, dtype="bf16", skew=0.0),
        # ... a prompt of ordinary, odd length.
        dict(name="mixtral_prompt_509", **MIXTRAL, tokens=509, dtype="fp16", skew=0.0),
        # ... a large prefill batch with uneven expert popularity: the largest call.
        dict(name="mixtral_prompt_4096", **MIXTRAL, tokens=4096, dtype="bf16", skew=0.5),
        # DeepSeek-V2-Lite MoE layer (64 small experts, 6 per token, two shared ones): one token,
        dict(name="deepseek_token_1", **DEEPSEEK, tokens=1, dtype="fp16", skew=0.0),
        # ... a decode batch,
        dict(name="deepseek_batch_16", **DEEPSEEK, tokens=16, dtype="bf16", skew=0.0),
        # ... a prompt.
        dict(name="deepseek_prompt_2000", **DEEPSEEK, tokens=2000, dtype="bf16", skew=0.5),
        # A captured decode step of a Mixtral-architecture decoder, one sequence with 600 tokens of context.  Two
        # layers and the output head: a layer costs the same in a deeper stack.
        dict(name="decoder_step_600", kind="decoder", layers=2, hidden=4096, ffn=14336, context=600, cache=1024),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng: random.Random):
    kind = rng.choice(("linear", "linear", "gemv", "mixtral", "mixtral", "mixtral", "deepseek", "deepseek", "decoder"))
    if kind == "linear":
        return dict(kind="linear", rows=_log_int(rng, 1, 4096), inf=rng.choice((512, 1408, 2048, 2816, 4096, 4096, 14336)),
                    outf=rng.choice((576, 1024, 1408, 2048, 2816, 4096, 4096, 14336)), bits=rng.choice((1, 2, 3, 4, 4, 4)),
                    dtype=rng.choice(("fp16", "bf16")), bias=rng.random() < 0.2)
    if kind == "gemv":
        return dict(kind="gemv", inf=rng.choice((1408, 2048, 4096, 14336)), outf=rng.choice((1024, 1408, 2048, 4096, 14336)),
                    bits=rng.choice((1, 2, 3, 4)))
    if kind == "mixtral":
        return dict(kind="mixtral", hidden=rng.choice((2048, 4096, 4096)), ffn=rng.choice((3456, 7168, 14336, 14336)),
                    experts=rng.choice((8, 8, 16)), top_k=2, tokens=_log_int(rng, 1, 4096), dtype=rng.choice(("fp16", "bf16")),
                    skew=rng.choice((0.0, 0.5, 2.0)))
    if kind == "deepseek":
        return dict(kind="deepseek", hidden=2048, ffn=1408, experts=rng.choice((32, 64, 64)), shared=2, top_k=6,
                    norm=rng.random() < 0.3, tokens=_log_int(rng, 1, 4096), dtype=rng.choice(("fp16", "bf16")),
                    skew=rng.choice((0.0, 0.5, 2.0)))
    cache = rng.choice((512, 1024, 2048, 4096))
    return dict(kind="decoder", layers=rng.choice((1, 2)), hidden=rng.choice((2048, 4096)), ffn=rng.choice((7168, 14336)),
                context=_log_int(rng, 32, cache - 1), cache=cache)


# ---- what a user's program has in hand ------------------------------------------------------------
def _expert_bits(n: int, seed: int):
    bits = [EXPERT_BITS[i % len(EXPERT_BITS)] for i in range(n)]
    random.Random(seed).shuffle(bits)
    return bits


def _gate_and_input(case, seed: int, gate_std: float, gen: torch.Generator):
    """Router matrix and hidden states.  ``skew`` > 0: expert popularity follows a Dirichlet(skew) draw, through a
    component that all hidden states share and that the router rows weigh differently."""
    E, D, T = case["experts"], case["hidden"], case["tokens"]
    gate = torch.randn(E, D, device="cuda", generator=gen) * gate_std
    x = torch.randn(T, D, device="cuda", generator=gen)
    if case["skew"] > 0:
        r = random.Random(seed)
        p = [r.gammavariate(case["skew"], 1.0) for _ in range(E)]
        logp = torch.tensor([max(v / sum(p), 1e-3) for v in p], device="cuda").log()
        m = 0.3 * torch.randn(D, device="cuda", generator=gen)
        x = x + m
        gate = gate + (logp - logp.mean())[:, None] * (m / m.square().sum())[None, :]
    return gate.to(torch.float16), x.to(DTYPES[case["dtype"]])


def _experts(bits, out_f: int, in_f: int, gen: torch.Generator):
    return [synth.make_linear(out_f, in_f, b, GROUP, gen, "cuda") for b in bits]


def prepare(case, seed):
    gen = synth.generator(seed, "cuda")
    kind = case["kind"]
    if kind in ("linear", "gemv"):
        packed = synth.make_linear(case["outf"], case["inf"], case["bits"], GROUP, gen, "cuda")
        rows = case.get("rows", 1)
        x = torch.randn(rows, case["inf"], device="cuda", generator=gen).to(DTYPES[case.get("dtype", "fp16")])
        if kind == "gemv":
            return SimpleNamespace(kind=kind, w=packed, x=x)
        bias = torch.randn(case["outf"], device="cuda", generator=gen).to(x.dtype) if case["bias"] else None
        return SimpleNamespace(kind=kind, layer=QuantLinear(packed, bias), x=x)
    if kind == "mixtral":
        E, D, Fd = case["experts"], case["hidden"], case["ffn"]
        gate, x = _gate_and_input(case, seed, 0.02, gen)
        bits = _expert_bits(E, seed)
        cfg = SimpleNamespace(hidden_size=D, intermediate_size=Fd, num_local_experts=E, num_experts_per_tok=case["top_k"])
        layer = QuantFusedMixtralMoEBlock.from_linears(cfg, gate, _experts(bits, Fd, D, gen), _experts(bits, D, Fd, gen),
                                                       _experts(bits, Fd, D, gen))
        return SimpleNamespace(kind=kind, layer=layer, x=x.unsqueeze(0))
    if kind == "deepseek":
        E, D, Fd = case["experts"], case["hidden"], case["ffn"]
        gate, x = _gate_and_input(case, seed, D ** -0.5, gen)
        bits = _expert_bits(E, seed)
        cfg = SimpleNamespace(hidden_size=D, moe_intermediate_size=Fd, n_routed_experts=E, n_shared_experts=case["shared"],
                              num_experts_per_tok=case["top_k"], norm_topk_prob=case["norm"])
        SF = case["shared"] * Fd
        shared = tuple(synth.make_linear(n, k, 4, GROUP, gen, "cuda") for n, k in ((SF, D), (D, SF), (SF, D)))
        layer = QuantFusedDeepseekV2MoEBlock.from_linears(cfg, gate, _experts(bits, Fd, D, gen), _experts(bits, D, Fd, gen),
                                                          _experts(bits, Fd, D, gen), shared)
        return SimpleNamespace(kind=kind, layer=layer, x=x.unsqueeze(0))
    # decoder: model, a cache that holds the context, and the decode step captured in a graph
    torch.manual_seed(seed)
    model = MixtralDecoder(device="cuda", seed=seed % 100003, num_hidden_layers=case["layers"], hidden_size=case["hidden"],
                           intermediate_size=case["ffn"], num_attention_heads=case["hidden"] // 128)
    cfg = model.config
    cache = StaticCache(cfg, case["cache"])
    for layer in cache.layers:
        kv = torch.randn(2, 1, cfg.num_key_value_heads, case["context"], cfg.head_dim, device="cuda", generator=gen)
        layer.lazy_initialization(kv[0].to(torch.bfloat16), kv[1].to(torch.bfloat16))
        layer.keys[:, :, :case["context"]] = kv[0]
        layer.values[:, :, :case["context"]] = kv[1]
    st = SimpleNamespace(kind=kind, model=model, cache=cache)
    st.next_tok = torch.randint(0, cfg.vocab_size, (1, 1), device="cuda", generator=gen)
    st.next_pos = torch.tensor([case["context"]], device="cuda")
    st.tok, st.pos = st.next_tok.clone(), st.next_pos.clone()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(2):
            model(st.tok, cache, st.pos)
        torch.cuda.synchronize()
        st.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st.graph, stream=side):
            st.logits = model(st.tok, cache, st.pos)
    torch.cuda.synchronize()
    return st


# ---- one pass -------------------------------------------------------------------------------------
def run(state):
    if state.kind == "gemv":
        w = state.w
        return dequant_splitk_gemv(state.x, w.W_q, w.scales, w.zeros, w.W_nbits, w.group_size)
    if state.kind == "decoder":
        state.tok.copy_(state.next_tok)
        state.pos.copy_(state.next_pos)
        state.graph.replay()
        return [state.logits] + [t for layer in state.cache.layers for t in (layer.keys, layer.values)]
    return state.layer(state.x)


# ---- what a pass cannot do without ----------------------------------------------------------------
def _packed_bytes(n: float, bits: float) -> float:
    return n * (bits + 32.0 / GROUP) / 8.0  # codes, and an fp16 scale and offset per group


def _moe_work(hidden, ffn, experts, top_k, tokens, bits, shared_ffn=0):
    touched = experts * (1.0 - (1.0 - top_k / experts) ** tokens)  # distinct experts of `tokens` independent choices
    byts = touched * _packed_bytes(3.0 * hidden * ffn, bits) + _packed_bytes(3.0 * hidden * shared_ffn, 4)
    byts += 2.0 * hidden * experts + 2.0 * 2.0 * tokens * hidden
    flops = 2.0 * tokens * hidden * (3.0 * (ffn * top_k + shared_ffn) + experts)
    return byts, flops


def work(case):
    kind = case["kind"]
    if kind in ("linear", "gemv"):
        rows, K, N = case.get("rows", 1), case["inf"], case["outf"]
        return {"bytes": _packed_bytes(float(K) * N, case["bits"]) + 2.0 * rows * (K + N), "flops": 2.0 * rows * K * N}
    mean = sum(EXPERT_BITS) / len(EXPERT_BITS)
    if kind == "decoder":
        D, hd, kv_heads, vocab = case["hidden"], 128, 8, 32000
        byts, flops = _moe_work(D, case["ffn"], 8, 2, 1, 2.0)
        attn = D * hd * (2 * (D // hd) + 2 * kv_heads)  # q, k, v, o projections, bf16
        kv = 2.0 * kv_heads * hd * (case["context"] + 1)
        return {"bytes": case["layers"] * (byts + 2.0 * attn + 2.0 * kv) + 2.0 * vocab * D,
                "flops": case["layers"] * (flops + 2.0 * attn + 4.0 * D * (case["context"] + 1)) + 2.0 * vocab * D}
    shared = case["shared"] * case["ffn"] if kind == "deepseek" else 0
    byts, flops = _moe_work(case["hidden"], case["ffn"], case["experts"], case["top_k"], case["tokens"], mean, shared)
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    # One rounding of the output type per stage: gate and up projections, their product, the down projection and
    # the weighted sum are each rounded, and the sums before them may be taken in any order.
    return {"rel": 1e-2 if case.get("dtype") == "bf16" or case["kind"] == "decoder" else 5e-3}
