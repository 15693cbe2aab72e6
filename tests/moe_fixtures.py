"""Build the same seeded quantised MoE layer twice: as oracle tensors and as a GPU block."""
from types import SimpleNamespace

import numpy as np
import torch

from oracle import gemq_oracle as O


def draw_linear(rng, out_f, in_f, b, G=128):
    q = rng.integers(0, 2 ** b, (out_f, in_f), dtype=np.uint8)
    s = (np.abs(rng.standard_normal((in_f // G, out_f))) * 0.01 + 1e-3).astype(np.float16)
    zp = (rng.random((in_f // G, out_f)) * (2 ** b - 1)).astype(np.float16)
    return dict(wq=O.pack_kernel_form(q, b), s=s, z=O.kernel_form_offset(s, zp), b=b, G=G, i=in_f, o=out_f)


def to_packed(lin, device):
    from gemq_b200.inference import PackedLinear
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)
    return PackedLinear(t(lin["wq"]), t(lin["s"]), t(lin["z"]), lin["b"], lin["G"], lin["i"], lin["o"])


def stacked(lins):
    return O.StackedExperts([l["wq"] for l in lins], [l["s"] for l in lins], [l["z"] for l in lins],
                            [l["b"] for l in lins], lins[0]["G"])


def make_layer(family, D, Fd, E, A, bits, seed, gate_std, n_shared=0, shared_bits=4, norm_topk_prob=False):
    rng = np.random.default_rng(seed)
    gate = (rng.standard_normal((E, D)) * gate_std).astype(np.float16)
    w1 = [draw_linear(rng, Fd, D, b) for b in bits]
    w3 = [draw_linear(rng, Fd, D, b) for b in bits]
    w2 = [draw_linear(rng, D, Fd, b) for b in bits]
    shared = None
    if n_shared:
        SF = n_shared * Fd
        shared = (draw_linear(rng, SF, D, shared_bits), draw_linear(rng, D, SF, shared_bits),
                  draw_linear(rng, SF, D, shared_bits))  # gate_proj, down_proj, up_proj
    if family == "mixtral":
        cfg = SimpleNamespace(hidden_size=D, intermediate_size=Fd, num_local_experts=E, num_experts_per_tok=A)
    else:
        cfg = SimpleNamespace(hidden_size=D, moe_intermediate_size=Fd, n_routed_experts=E, n_shared_experts=n_shared,
                              num_experts_per_tok=A, norm_topk_prob=norm_topk_prob)
    return dict(family=family, cfg=cfg, gate=gate, w1=w1, w2=w2, w3=w3, shared=shared, A=A)


def oracle_parts(layer):
    sh = None
    if layer["shared"]:
        s1, s2, s3 = layer["shared"]
        trip = lambda l: (l["wq"], l["s"], l["z"])
        sh = (trip(s1), trip(s3), trip(s2), s1["b"], s1["G"])
    return stacked(layer["w1"]), stacked(layer["w3"]), stacked(layer["w2"]), sh


def gpu_block(layer, device="cuda"):
    from gemq_b200.inference import QuantFusedDeepseekV2MoEBlock, QuantFusedMixtralMoEBlock
    gate = torch.from_numpy(layer["gate"]).to(device)
    p = lambda lins: [to_packed(l, device) for l in lins]
    if layer["family"] == "mixtral":
        return QuantFusedMixtralMoEBlock.from_linears(layer["cfg"], gate, p(layer["w1"]), p(layer["w2"]), p(layer["w3"]))
    s1, s2, s3 = layer["shared"]
    return QuantFusedDeepseekV2MoEBlock.from_linears(layer["cfg"], gate, p(layer["w1"]), p(layer["w2"]), p(layer["w3"]),
                                                     (to_packed(s1, device), to_packed(s2, device), to_packed(s3, device)))


def shift_experts(blk, words, scales, which=None):
    """The block's experts moved off their places: `words` int32 and `scales` fp16 elements ahead of each, or of those in
    `which` only, the others at whole rows."""
    for name in ("w1", "w2", "w3"):
        for suffix, table, gap in (("wq", "wq_strides", words), ("scales", "zs_strides", scales), ("zeros", "zs_strides", scales)):
            old = getattr(blk, f"{name}_{suffix}")
            at, N = getattr(blk, f"{name}_{table}").tolist() + [old.numel()], old.shape[1]
            places, end = [], 0
            for e in range(len(at) - 1):
                places.append(end + gap if which is None or e in which else -(-end // N) * N)
                end = places[-1] + at[e + 1] - at[e]
            new = torch.zeros(-(-end // N), N, dtype=old.dtype, device=old.device)
            for e, p in enumerate(places):
                new.view(-1)[p:p + at[e + 1] - at[e]] = old.reshape(-1)[at[e]:at[e + 1]]
            setattr(blk, f"{name}_{suffix}", new)
            if suffix != "scales":  # the offsets, next, lie like the scales
                setattr(blk, f"{name}_{table}", torch.tensor(places, dtype=torch.int32, device=old.device))
    blk._build_layer(blk._layer.route_mode, bool(blk._layer.renorm), blk._layer.shared_ffn)


def takes_few_rows(layer, T):
    """Whether a batch of T tokens takes the few-row launches: they report experts off a whole row, which the GEMM loads."""
    blk, A = gpu_block(layer), layer["A"]
    shift_experts(blk, 5, 0)
    E, D = layer["gate"].shape
    routing = (torch.full((T, A), 0.5, dtype=torch.float16, device="cuda"), (torch.arange(T * A).view(T, A) % E).cuda())
    blk._prefill(torch.ones(T, D, dtype=torch.float16, device="cuda"), 1, True, routing=routing)
    code = blk.prefill_error_code(T)
    assert code in (0, 22)
    return code == 22
