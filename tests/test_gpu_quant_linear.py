"""Loader side on the GPU: an HQQ-format layer (gemq/inference/patch.py:23-68) converted to the
kernel form and run as a quantised linear, against fp32 math on the de-quantised weight
W = (Q - zero) * scale (gemq/quantizers/gptq.py:446-450)."""
import pytest
import torch

from conftest import MAX_ABS_TOL, REL_FRO_TOL, max_abs, rel_fro

pytestmark = pytest.mark.gpu


def _hqq_layer(seed, out_f, in_f, nbits, G):
    from gemq_b200.quant.hqq_format import hqq_pack
    g = torch.Generator().manual_seed(seed)
    codes = torch.randint(0, 2 ** nbits, (out_f, in_f), generator=g, dtype=torch.uint8)
    groups = out_f * in_f // G
    scale = (torch.randn(groups, 1, generator=g).abs() * 0.01 + 1e-3).half()
    zero = (torch.rand(groups, 1, generator=g) * (2 ** nbits - 1)).half()
    meta = dict(shape=(out_f, in_f), nbits=nbits, group_size=G, axis=1, scale=scale, zero=zero)
    return hqq_pack(codes.reshape(groups, G), nbits), meta, codes, scale, zero


@pytest.mark.parametrize("nbits", [1, 2, 3, 4])
@pytest.mark.parametrize("rows", [1, 64])
def test_hqq_layer_as_quant_linear(nbits, rows):
    from gemq_b200.inference import QuantLinear
    from gemq_b200.quant.emit import check_packing
    from gemq_b200.quant.hqq_format import packed_linear_from_hqq
    out_f, in_f, G = 384, 512, 128
    W_q, meta, codes, scale, zero = _hqq_layer(10 * nbits + rows, out_f, in_f, nbits, G)
    packed = packed_linear_from_hqq(W_q, meta)
    check_packing(packed, codes=codes)          # the integers survive the conversion bit-exactly
    lin = QuantLinear(packed)
    for name in ("W_q", "scales", "zeros"):
        setattr(lin, name, getattr(lin, name).cuda())
    x = torch.randn(rows, in_f, generator=torch.Generator().manual_seed(3)).half()
    y = lin(x.cuda()).float().cpu().numpy()
    s = scale.float().reshape(out_f, in_f // G).repeat_interleave(G, dim=1)
    z = zero.float().reshape(out_f, in_f // G).repeat_interleave(G, dim=1)
    W = (codes.float() - z) * s
    ref = (x.float() @ W.t()).numpy()
    assert y.shape == (rows, out_f)
    assert rel_fro(y, ref) < REL_FRO_TOL, rel_fro(y, ref)
    assert max_abs(y, ref) < MAX_ABS_TOL, max_abs(y, ref)


@pytest.mark.parametrize("rows", [1, 13, 200])
@pytest.mark.parametrize("nbits", [2, 3])
def test_weights_written_by_the_launch_before(rows, nbits):
    """The matrix, its scales and its offsets are results of the launches right before the call, whose kernels start
    before those have ended: the call waits for them (few-row kernel and tcgen05 GEMM)."""
    from gemq_b200 import synth
    from gemq_b200.inference import PackedLinear, QuantLinear
    gen = synth.generator(rows + nbits, "cuda")
    srcs = [synth.make_linear(4096, 2048, nbits, 128, gen, "cuda") for _ in range(2)]
    x = torch.randn(rows, 2048, device="cuda", generator=gen).to(torch.bfloat16)
    want = [QuantLinear(s)(x) for s in srcs]
    own = PackedLinear(srcs[0].W_q.clone(), srcs[0].scales.clone(), srcs[0].zeros.clone(), nbits, 128, 2048, 4096)
    layer = QuantLinear(own)
    torch.cuda.synchronize()
    got = []
    for i in range(40):
        s = srcs[i % 2]
        for dst, src in (((own.scales, s.scales), (own.zeros, s.zeros), (own.W_q, s.W_q)) if i % 4 < 2 else
                         ((own.W_q, s.W_q), (own.zeros, s.zeros), (own.scales, s.scales))):
            torch.add(src, 0, out=dst)  # a kernel, not a copy
        got.append(layer(x))
    assert all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))
