"""The few-row kernels at the edges of their tiles: one to seventeen rows around the 8- and 16-row blocks,
column counts that end inside a 64-column tile, reduction lengths that end inside a stage or a 3-bit run,
and MoE batches whose experts get no row, one row or more than a tile."""
import numpy as np
import pytest
import torch

from oracle import gemq_oracle as O
from conftest import REL_FRO_TOL, rel_fro
import moe_fixtures as MF

pytestmark = pytest.mark.gpu

# One rounding of the output: 2^-11 (fp16) or 2^-8 (bf16) of each value at most; the sums before it are fp32.
OUT_TOL = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("b", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(32, 128), (96, 640), (576, 1408), (160, 4096)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_linear_rows_edges(b, N, K, dtype):
    from gemq_b200.kernels._runtime import error_word
    from gemq_b200.kernels.dequant_gemm import quant_linear
    rng = np.random.default_rng(b * 100 + N)
    lin = MF.draw_linear(rng, N, K, b)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    wq, s, z = t(lin["wq"]), t(lin["s"]), t(lin["z"])
    W = O.dequantize(lin["wq"], lin["s"], lin["z"], b, 128, K).astype(np.float64)
    bias = torch.from_numpy(rng.standard_normal(N)).to(dtype).cuda()
    for M in (1, 7, 8, 9, 16, 17):
        x = torch.from_numpy(rng.standard_normal((M, K))).to(dtype).cuda()
        y = quant_linear(x, wq, s, z, b, 128, None)
        assert y.dtype == dtype and torch.equal(y, quant_linear(x, wq, s, z, b, 128, None))
        want = x.double().cpu().numpy() @ W
        # the de-quantised reference weights carry an fp16 rounding (2^-11) that the exact codes do not
        assert rel_fro(y.double().cpu().numpy(), want) < OUT_TOL[dtype] + 2.0 ** -11, (M, rel_fro(y.double().cpu().numpy(), want))
        yb = quant_linear(x, wq, s, z, b, 128, bias)
        assert torch.equal(yb, y + bias)
    # rows of a wider tensor, not 16-byte aligned
    wide = torch.from_numpy(rng.standard_normal((5, K + 3))).to(dtype).cuda()[:, 1:K + 1]
    assert torch.equal(quant_linear(wide, wq, s, z, b, 128, None), quant_linear(wide.contiguous(), wq, s, z, b, 128, None))
    assert int(error_word(y.device).item()) == 0


@pytest.mark.parametrize("bits", [[1, 2, 3, 4], [3, 3, 3, 3], [1, 1, 4, 1]])
@pytest.mark.parametrize("D,Fd", [(256, 512), (640, 384), (1408, 896)])
def test_moe_few_rows_edges(bits, D, Fd):
    layer = MF.make_layer("mixtral", D=D, Fd=Fd, E=4, A=2, bits=bits, seed=9, gate_std=0.02)
    blk = MF.gpu_block(layer)
    w1, w3, w2, _ = MF.oracle_parts(layer)
    g = torch.Generator().manual_seed(D)
    for T, one in ((2, False), (5, True), (9, True), (17, True), (24, False)):
        x = torch.randn(T, D, generator=g).half()
        # `one`: every token picks expert 2 and one other, so one expert crosses the tile sizes
        sel = torch.stack([torch.tensor([2, int(torch.randint(0, 2, (1,), generator=g))]) if one
                           else torch.randperm(4, generator=g)[:2] for _ in range(T)])
        w = torch.softmax(torch.randn(T, 2, generator=g), -1).half()
        out = blk._prefill(x.cuda(), 1, True, routing=(w.cuda(), sel.cuda()))[0]
        assert blk.prefill_error_code(T) == 0
        ref = O.moe_reference_fp32(x, w.float(), sel, w1, w3, w2).numpy()
        assert rel_fro(out.float().cpu().numpy(), ref) < REL_FRO_TOL
        assert torch.equal(out, blk._prefill(x.cuda(), 1, True, routing=(w.cuda(), sel.cuda()))[0])


@pytest.mark.parametrize("b", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(32, 128), (288, 640), (576, 1408)])
def test_gemm_tile_edges(b, N, K):
    """The tcgen05 GEMM where the last 256-column pair of CTAs is partly or half empty, the k-blocks are fewer
    than the ring's stages or no multiple of them, and the token count ends inside a 32-row box, fills a tile
    or goes one past it."""
    from gemq_b200.kernels import dequant_gemm
    from gemq_b200.kernels._runtime import error_word
    from gemq_b200.kernels.dequant_gemm import _gemm_tc
    rng = np.random.default_rng(b * 10 + N)
    lin = MF.draw_linear(rng, N, K, b)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    wq, s, z = t(lin["wq"]), t(lin["s"]), t(lin["z"])
    W = O.dequantize(lin["wq"], lin["s"], lin["z"], b, 128, K).astype(np.float64)
    bias = torch.from_numpy(rng.standard_normal(N)).cuda()
    for M in (32, 33, 255, 256, 257):
        for dtype in (torch.float16, torch.bfloat16):
            x = torch.from_numpy(rng.standard_normal((M, K))).to(dtype).cuda()
            y = dequant_gemm(x, wq, s, z, b, 128)
            want = x.double().cpu().numpy() @ W
            # fp16: one rounding of the result.  bf16: the weights are rounded to bf16 as well, errors 2^-9 rms at most
            # each way
            tol = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8 + 2.0 ** -9
            assert rel_fro(y.double().cpu().numpy(), want) < tol, (M, dtype, rel_fro(y.double().cpu().numpy(), want))
            assert torch.equal(_gemm_tc(x, wq, s, z, b, 128, bias.to(dtype)), y + bias.to(dtype))
    assert int(error_word(wq.device).item()) == 0


@pytest.mark.parametrize("M,N,K,b,gemm", [(3, 2816, 14336, 3, 0), (4, 6912, 4224, 3, 0), (128, 576, 4096, 4, 1), (15, 1152, 384, 1, 1),
                                          (21, 4096, 512, 1, 1), (13, 4096, 4096, 4, 0), (64, 4096, 4096, 4, 1)])
def test_linear_line(M, N, K, b, gemm):
    """Which kernel a linear takes decides how its weights are rounded.  Calls at which other constants of the GEMM's estimate
    would draw the line elsewhere: on the few-row kernel a bf16 result carries one rounding of its own (2^-9 of a value at
    most), in the GEMM one of every weight, too."""
    from gemq_b200 import _capi
    from gemq_b200.kernels.dequant_gemm import quant_linear
    assert _capi.lib.gemq_linear_takes_gemm(M, N, K, b) == gemm
    if gemm:
        return
    lin = MF.draw_linear(np.random.default_rng(N), N, K, b)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    wq, s, z = t(lin["wq"]), t(lin["s"]), t(lin["z"])
    W = torch.from_numpy(O.dequantize(lin["wq"], lin["s"], lin["z"], b, 128, K).astype(np.float64)).cuda()
    scale, zero = s.double().repeat_interleave(128, 0), z.double().repeat_interleave(128, 0)
    W = ((W - zero) / scale).round() * scale + zero  # without the rounding to fp16
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).bfloat16().cuda()
    y = quant_linear(x, wq, s, z, b, 128, None)
    assert rel_fro(y.double().cpu().numpy(), (x.double() @ W).cpu().numpy()) < 2.0 ** -9


@pytest.mark.parametrize("b", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K,M", [(288, 2176, 1), (96, 4096, 33), (1024, 5376, 100)])
def test_gemm_split_k(b, N, K, M):
    """The tcgen05 GEMM with k in parts: an odd number of k-blocks, a last part shorter than the others, 3-bit parts that
    begin at every place of a packed word, fewer rows than a tile."""
    from gemq_b200 import _capi
    from gemq_b200.kernels._runtime import error_word
    from gemq_b200.kernels.dequant_gemm import _gemm_tc
    assert _capi.lib.gemq_linear_gemm_scratch_bytes(M, N, K, b) >= 2 * 4 * M * N
    rng = np.random.default_rng(b * 10 + N)
    lin = MF.draw_linear(rng, N, K, b)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    wq, s, z = t(lin["wq"]), t(lin["s"]), t(lin["z"])
    W = O.dequantize(lin["wq"], lin["s"], lin["z"], b, 128, K).astype(np.float64)
    bias = torch.from_numpy(rng.standard_normal(N)).cuda()
    for dtype in (torch.float16, torch.bfloat16):
        x = torch.from_numpy(rng.standard_normal((M, K))).to(dtype).cuda()
        y = _gemm_tc(x, wq, s, z, b, 128, None)
        want = x.double().cpu().numpy() @ W
        tol = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8 + 2.0 ** -9  # as in the test above
        assert rel_fro(y.double().cpu().numpy(), want) < tol, (dtype, rel_fro(y.double().cpu().numpy(), want))
        assert torch.equal(_gemm_tc(x, wq, s, z, b, 128, bias.to(dtype)), y + bias.to(dtype))
    assert int(error_word(wq.device).item()) == 0


@pytest.mark.parametrize("rows", [[49, 1, 0, 60], [256, 257, 16, 17], [600, 0, 0, 1]])
@pytest.mark.parametrize("bits", [[1, 2, 3, 4], [3, 4, 1, 2]])
def test_moe_large_tiles(rows, bits):
    """Experts with fewer rows than a 32-row box, exactly a tile, one more than a tile, an uneven number of
    16-row blocks; the second CTA of a pair past the last column (384 = 256 + 128)."""
    D, Fd = 384, 640
    layer = MF.make_layer("mixtral", D=D, Fd=Fd, E=4, A=1, bits=bits, seed=5, gate_std=0.02)
    blk = MF.gpu_block(layer)
    w1, w3, w2, _ = MF.oracle_parts(layer)
    g = torch.Generator().manual_seed(sum(rows))
    sel = torch.cat([torch.full((n,), e, dtype=torch.int64) for e, n in enumerate(rows)])
    T = sel.numel()
    sel = sel[torch.randperm(T, generator=g)].view(T, 1)
    w = (torch.rand(T, 1, generator=g) * 0.5 + 0.5).half()
    for dtype in (torch.float16, torch.bfloat16):
        x = torch.randn(T, D, generator=g).to(dtype)
        out = blk._prefill(x.cuda(), 1, True, routing=(w.to(dtype).cuda(), sel.cuda()))[0]
        assert blk.prefill_error_code(T) == 0
        ref = O.moe_reference_fp32(x.float(), w.to(dtype).float(), sel, w1, w3, w2).numpy()
        assert rel_fro(out.float().cpu().numpy(), ref) < REL_FRO_TOL


@pytest.mark.parametrize("D,Fd,E", [(128, 10240, 16), (10240, 128, 32)])
def test_moe_many_tiles_per_pair(D, Fd, E):
    """More than sixteen tiles for every pair of CTAs with k of one stage, the shortest there is: barriers whose phases run through
    the ring many times within a launch, tiles of all widths in turn (and in the other launch, k of eighty stages)."""
    bits = [1, 2, 3, 4] * (E // 4)
    layer = MF.make_layer("mixtral", D=D, Fd=Fd, E=E, A=1, bits=bits, seed=11, gate_std=0.02)
    blk = MF.gpu_block(layer)
    w1, w3, w2, _ = MF.oracle_parts(layer)
    g = torch.Generator().manual_seed(D)
    T = 26 * E  # above 24 rows per expert: the GEMMs
    sel = torch.randint(0, E, (T, 1), generator=g)
    w = (torch.rand(T, 1, generator=g) * 0.5 + 0.5).half()
    x = torch.randn(T, D, generator=g).half()
    out = blk._prefill(x.cuda(), 1, True, routing=(w.cuda(), sel.cuda()))[0]
    assert blk.prefill_error_code(T) == 0
    ref = O.moe_reference_fp32(x, w.float(), sel, w1, w3, w2).numpy()
    assert rel_fro(out.float().cpu().numpy(), ref) < REL_FRO_TOL
    assert torch.equal(out, blk._prefill(x.cuda(), 1, True, routing=(w.cuda(), sel.cuda()))[0])


@pytest.mark.parametrize("rows", [[128, 129, 40, 7], [192, 193, 130, 33], [161, 177, 224, 192]])
@pytest.mark.parametrize("bits", [[1, 2, 3, 4], [3, 4, 1, 2], [4, 4, 4, 3]])
def test_moe_staged_words(rows, bits):
    """Tiles of 7 to 224 rows, at and next to multiples of 32, whose packed words come through shared memory, every width at every
    size; reduction lengths that end inside a 3-bit word."""
    g = torch.Generator().manual_seed(sum(rows))
    sel = torch.cat([torch.full((n,), e, dtype=torch.int64) for e, n in enumerate(rows)])
    T = sel.numel()
    sel = sel[torch.randperm(T, generator=g)].view(T, 1)
    w = (torch.rand(T, 1, generator=g) * 0.5 + 0.5).half()
    for D, Fd in ((384, 1408), (1664, 128)):
        layer = MF.make_layer("mixtral", D=D, Fd=Fd, E=4, A=1, bits=bits, seed=5, gate_std=0.02)
        blk = MF.gpu_block(layer)
        w1, w3, w2, _ = MF.oracle_parts(layer)
        for dtype in (torch.float16, torch.bfloat16):
            x = torch.randn(T, D, generator=g).to(dtype)
            out = blk._prefill(x.cuda(), 1, True, routing=(w.to(dtype).cuda(), sel.cuda()))[0]
            assert blk.prefill_error_code(T) == 0
            ref = O.moe_reference_fp32(x.float(), w.to(dtype).float(), sel, w1, w3, w2).numpy()
            assert rel_fro(out.float().cpu().numpy(), ref) < REL_FRO_TOL


def _reference(layer, x, w, sel):
    """Layer output in fp32 for one expert per token, an expert's rows at a time."""
    deq = lambda l: torch.from_numpy(O.dequantize(l["wq"], l["s"], l["z"], l["b"], 128, l["i"]).astype(np.float32))
    ffn = lambda x, w1, w3, w2: (torch.nn.functional.silu(x @ deq(w1)) * (x @ deq(w3))) @ deq(w2)
    x, out = x.float(), torch.zeros(x.shape)
    for e, mats in enumerate(zip(layer["w1"], layer["w3"], layer["w2"])):
        rows = sel[:, 0] == e
        out[rows] = w.float()[rows] * ffn(x[rows], *mats)
    if layer["shared"]:
        s1, s2, s3 = layer["shared"]
        out += ffn(x, s1, s3, s2)
    return out.numpy()


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("D,Fd", [(1280, 1024), (2560, 256)])
def test_moe_long_words_before_short(D, Fd, shared):
    """Every pair of CTAs gets 4-bit tiles of 256 rows, whose packed words fill a whole place of the ring, and then tiles of
    shorter words: routed experts of 2 and 1 bits behind a 4-bit one, or 3 bits behind the shared expert, whose tiles lead the list.
    Reduction lengths of two stages (a use of every second stage) to twenty."""
    g = torch.Generator().manual_seed(D)
    if shared:
        T = 5120
        layer = MF.make_layer("deepseek", D=D, Fd=Fd, E=2, A=1, bits=[3, 1], seed=3, gate_std=0.02, n_shared=1)
        sel = (torch.arange(T) >= 2560).long()
    else:
        layer = MF.make_layer("mixtral", D=D, Fd=Fd, E=3, A=1, bits=[4, 2, 1], seed=3, gate_std=0.02)
        sel = torch.tensor([0] * 5120 + [1] * 2560 + [2] * 2560)
        T = sel.numel()
    blk = MF.gpu_block(layer)
    sel = sel[torch.randperm(T, generator=g)].view(T, 1)
    w = (torch.rand(T, 1, generator=g) * 0.5 + 0.5).half()
    x = torch.randn(T, D, generator=g).half()
    args = (x.cuda(), 1, True)
    out = blk._prefill(*args, routing=(w.cuda(), sel.cuda()))[0]
    assert blk.prefill_error_code(T) == 0
    assert rel_fro(out.float().cpu().numpy(), _reference(layer, x, w, sel)) < REL_FRO_TOL
    for _ in range(20):
        assert torch.equal(out, blk._prefill(*args, routing=(w.cuda(), sel.cuda()))[0])


@pytest.mark.parametrize("D,Fd,bits", [(128, 2048, [4, 3, 1, 2, 4, 3]), (2048, 128, [2, 4, 3, 4, 1, 2]), (4096, 128, [1, 3, 4, 3, 2, 1])])
def test_moe_many_short_tiles(D, Fd, bits):
    """Gate/up or down tiles of one stage, some nine or more a pair of CTAs: the slots of tile descriptions and the ring of words go
    round while a tile is over before the next one's description is made.  Tiles of 1, 17, 65 and 128 rows, which use the halves of
    the accumulators in turn, between those of some 240 to 256, which take all of them."""
    g = torch.Generator().manual_seed(D + Fd)
    layer = MF.make_layer("mixtral", D=D, Fd=Fd, E=6, A=1, bits=bits, seed=5, gate_std=0.02)
    rows = (5121, 129, 5000, 1, 17, 128)
    sel = torch.cat([torch.full((n,), e) for e, n in enumerate(rows)])
    T = sel.numel()
    blk = MF.gpu_block(layer)
    sel = sel[torch.randperm(T, generator=g)].view(T, 1)
    w = (torch.rand(T, 1, generator=g) * 0.5 + 0.5).half()
    x = torch.randn(T, D, generator=g).half()
    args = (x.cuda(), 1, True)
    out = blk._prefill(*args, routing=(w.cuda(), sel.cuda()))[0]
    assert blk.prefill_error_code(T) == 0
    assert rel_fro(out.float().cpu().numpy(), _reference(layer, x, w, sel)) < REL_FRO_TOL
    for _ in range(10):
        assert torch.equal(out, blk._prefill(*args, routing=(w.cuda(), sel.cuda()))[0])


@pytest.mark.parametrize("shared", [0, 2])
def test_moe_few_rows_one_behind_the_other(shared):
    """Decode batches on one scratch with nothing in between but kernels that write their weights: the products read the plan, which
    replaces that of the call before at the same place, and their first weights ahead of their waits.  Routings with one tile, with
    a tile for every expert, with tiles of many rows and (ids out of range) with none."""
    E, A, D, Fd = 16, 2, 512, 384
    make = lambda seed: MF.make_layer("deepseek" if shared else "mixtral", D=D, Fd=Fd, E=E, A=A, bits=[1, 2, 3, 4] * 4, seed=seed,
                                      gate_std=0.02, n_shared=shared)
    blk, other = MF.gpu_block(make(1)), MF.gpu_block(make(2))
    names = [n for n in vars(blk) if n.endswith(("_wq", "_scales", "_zeros")) and getattr(blk, n) is not None]
    weights = [{n: getattr(b, n).clone() for n in names} for b in (blk, other)]
    g = torch.Generator().manual_seed(shared)
    calls = []
    for i in range(24):
        T = (24, 24, 24, 9, 40, 24)[i % 6]
        sel = (torch.full((T, A), i % E), torch.randint(0, E, (T, A), generator=g), torch.arange(T * A).view(T, A) % E,
               torch.randint(0, 3, (T, A), generator=g), torch.full((T, A), E + 1), torch.randint(8, E, (T, A), generator=g))[i % 6]
        w = torch.softmax(torch.randn(T, A, generator=g), -1).half().cuda()
        calls.append((torch.randn(T, D, generator=g).half().cuda(), w, sel.cuda(), (i // 6 + i) % 2))

    def write(which):
        for n in names:  # kernels, not copies
            torch.add(weights[which][n], 0, out=getattr(blk, n))

    for rewritten in (True, False):
        want = []
        for x, w, sel, which in calls:
            write(which if rewritten else 0)
            torch.cuda.synchronize()
            want.append(blk._prefill(x, 1, True, routing=(w, sel))[0].clone())
            torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = []
            for x, w, sel, which in calls:
                if rewritten:
                    write(which)
                got.append(blk._prefill(x, 1, True, routing=(w, sel))[0])
        for _ in range(10):
            for y in got:
                y.fill_(float("nan"))
            graph.replay()
            assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("T", [40, 400])  # few-row launches and the GEMM
def test_moe_bit_width_tables(T):
    """Widths on the device are clamped before they choose a map of packed words, and the shared expert's third matrix is read with
    the first one's width."""
    layer = MF.make_layer("deepseek", D=256, Fd=384, E=4, A=2, bits=[4, 4, 1, 4], seed=1, gate_std=0.02, n_shared=1)
    assert MF.takes_few_rows(layer, T) == (T == 40)
    blk = MF.gpu_block(layer)
    x = torch.randn(T, 256, generator=torch.Generator().manual_seed(T)).half().cuda()
    want = blk._prefill(x, 2, False)[0].clone()
    for name in ("w1", "w2", "w3"):
        getattr(blk, f"{name}_nbits").copy_(torch.tensor([4, 7, -3, 33]))
    blk._layer.s3.nbits = 3
    assert torch.equal(blk._prefill(x, 2, False)[0], want)
    assert blk.prefill_error_code(T) == 0


@pytest.mark.parametrize("words,scales", [(0, 8), (5, 0), (32, 0), (0, 3), (9, 1)])
def test_moe_experts_off_whole_rows(words, scales):
    """Experts that begin off a whole row of words or a 16-byte boundary of scales: the GEMM's producers load them, few-row launches
    leave them out and say so.  Eight scales more are a boundary."""
    layer = MF.make_layer("mixtral", D=384, Fd=256, E=4, A=1, bits=[1, 2, 3, 4], seed=7, gate_std=0.02)
    blk, moved = MF.gpu_block(layer), MF.gpu_block(layer)
    MF.shift_experts(moved, words, scales)
    g = torch.Generator().manual_seed(words + scales)
    for T in (16, 300, 1200):
        x, w = torch.randn(T, 384, generator=g).half().cuda(), torch.rand(T, 1, generator=g).half().cuda()
        sel = torch.randint(0, 4, (T, 1), generator=g).cuda()
        want = blk._prefill(x, 1, True, routing=(w, sel))[0]
        got = moved._prefill(x, 1, True, routing=(w, sel))[0]
        if T == 16 and (words or scales % 8):
            assert moved.prefill_error_code(T) == 22 and not got.any()
        else:
            assert moved.prefill_error_code(T) == 0 and torch.equal(got, want)
        assert blk.prefill_error_code(T) == 0


@pytest.mark.parametrize("rows", [17, 18, 21, 22, 24, 25])
def test_moe_few_rows_line(rows):
    """Up to 24 rows per expert on average the codes are used as they are: weights are not rounded to fp16, and bf16
    activations beyond fp16's range count (gate and up weights of their group are 2^-8 of the others: h stays in range)."""
    E, A, D, Fd = 4, 2, 256, 384
    T = rows * E // A
    layer = MF.make_layer("mixtral", D=D, Fd=Fd, E=E, A=A, bits=[1, 2, 3, 4], seed=rows, gate_std=0.02)
    assert MF.takes_few_rows(layer, T) == (rows <= 24)
    if rows > 24:
        return
    for mats in (layer["w1"], layer["w3"]):
        for lin in mats:
            lin["s"][0] *= np.float16(2.0 ** -8)
            lin["z"][0] *= np.float16(2.0 ** -8)
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(T, D, generator=g).bfloat16()
    x[T // 2, 7] = 90000.0
    sel = torch.stack([torch.randperm(E, generator=g)[:A] for _ in range(T)])
    w = torch.softmax(torch.randn(T, A, generator=g), -1).bfloat16()
    blk = MF.gpu_block(layer)
    out = blk._prefill(x.cuda(), 1, True, routing=(w.cuda(), sel.cuda()))[0]
    assert blk.prefill_error_code(T) == 0 and out.isfinite().all()
    w1, w3, w2, _ = MF.oracle_parts(layer)
    ref = O.moe_reference_fp32(x.float(), w.float(), sel, w1, w3, w2).numpy()
    got, large = out.float().cpu().numpy(), np.arange(T) == T // 2
    assert rel_fro(got[large], ref[large]) < REL_FRO_TOL and rel_fro(got[~large], ref[~large]) < REL_FRO_TOL


@pytest.mark.parametrize("moved", [(0,), (1,), (0, 2), (1, 2), (0, 1, 2)])
@pytest.mark.parametrize("D,Fd,shared", [(128, 2560, False), (256, 1280, True), (384, 2560, False), (2560, 1024, True)])
def test_moe_staged_and_unstaged_tiles(D, Fd, shared, moved):
    """Tiles of experts off their boundaries, whose words the producers load, before, between and behind those of experts (and of
    the shared one, whose tiles lead) whose words come through shared memory, some eleven a pair of CTAs and of 1, 2, 3, 8, 10 and 20
    stages: the two kinds pass the same barriers."""
    g = torch.Generator().manual_seed(D + len(moved))
    layer = MF.make_layer("deepseek" if shared else "mixtral", D=D, Fd=Fd, E=3, A=1, bits=[4, 3, 1], seed=3, gate_std=0.02, n_shared=int(shared))
    blk, other = MF.gpu_block(layer), MF.gpu_block(layer)
    MF.shift_experts(other, 5, 8, moved)
    sel = torch.tensor([0] * 5120 + [1] * 2700 + [2] * 2420)
    T = sel.numel()
    args = (torch.randn(T, D, generator=g).half().cuda(), 1, True)
    routing = ((torch.rand(T, 1, generator=g) * 0.5 + 0.5).half().cuda(), sel[torch.randperm(T, generator=g)].view(T, 1).cuda())
    want = blk._prefill(*args, routing=routing)[0]
    for _ in range(10):
        assert torch.equal(other._prefill(*args, routing=routing)[0], want)
    assert blk.prefill_error_code(T) == 0 and other.prefill_error_code(T) == 0


@pytest.mark.parametrize("b", [1, 2, 3, 4])
def test_gemm_of_unaligned_views(b):
    """A dense matrix whose words, scales or offsets begin off a 16-byte boundary is loaded by the GEMM's producers: the same sums."""
    from gemq_b200.kernels import dequant_gemm
    from gemq_b200.kernels._runtime import error_word
    N, K, M = 288, 1408, 200
    lin = MF.draw_linear(np.random.default_rng(b), N, K, b)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    mats = [t(lin["wq"]), t(lin["s"]), t(lin["z"])]
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(b)).half().cuda()
    want = dequant_gemm(x, *mats, b, 128)
    W = O.dequantize(lin["wq"], lin["s"], lin["z"], b, 128, K).astype(np.float64)
    assert rel_fro(want.double().cpu().numpy(), x.double().cpu().numpy() @ W) < 2.0 ** -11  # one rounding of the result
    for which in range(3):
        m = list(mats)
        flat = torch.empty(m[which].numel() + 1, dtype=m[which].dtype, device="cuda")
        m[which] = flat[1:].view_as(m[which]).copy_(m[which])
        assert m[which].data_ptr() % 16 and torch.equal(dequant_gemm(x, *m, b, 128), want)
    assert int(error_word(x.device).item()) == 0
