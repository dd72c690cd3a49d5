"""The linear layers that run on pairs of SMs (csrc/gemm_pair.cu), at the edges of their tiles: token tiles of 32 .. 256 rows, weight tiles of 256 rows
of which the last may be half or partly empty, stages of two k-blocks of which the last may hold one."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from onnxruntime_genai_b200 import ops
    from onnxruntime_genai_b200.ops.fp4 import Fp4Experts
    from onnxruntime_genai_b200.ops.w4 import W4Weight


def _rows(m, k, seed, scale=0.5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(m, k, generator=g, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("m,n,k,tiles", [(1, 8, 8, 1), (129, 256, 64, 1), (256, 257, 128, 1), (257, 384, 200, 2), (300, 1000, 136, 5), (777, 640, 320, 4),
                                         (4096, 264, 72, 16), (2500, 19000, 192, 10)])
@pytest.mark.parametrize("out_fp32", [False, True])
def test_pair_product(m, n, k, tiles, out_fp32):
    x, w = _rows(m, k, 1), _rows(n, k, 2)
    bias = _rows(1, n, 3)[0]
    res = _rows(m, n, 4).float() if out_fp32 else _rows(m, n, 4)
    got = ops.linear(x, w, bias, residual=res, out_fp32=out_fp32, splits=-tiles)
    ops.check_kernel_status()
    ref = x.double() @ w.double().t() + bias.double() + res.double()
    # fp32 accumulation of k products of values below 2.5: k * 2^-24 * 6 ; a bf16 result adds half a unit of its last place
    bound = k * 2.0 ** -24 * 6.25 + (0 if out_fp32 else 1) * 2.0 ** -8 * ref.abs()
    assert ((got.double() - ref).abs() <= bound + 1e-6).all()


@pytest.mark.parametrize("act", ["silu", "relu", "gelu"])
def test_pair_gated(act):
    m, n, k = 301, 384, 328
    x, w = _rows(m, k, 5), _rows(2 * n, k, 6, 0.2)
    got = ops.gate_up_act(x, w, None, act, interleaved=True)
    ops.check_kernel_status()
    y = (x.double() @ w.double().t()).view(m, n // 64, 2, 64)
    g, u = y[:, :, 0].reshape(m, n), y[:, :, 1].reshape(m, n)
    g = {"silu": lambda t: t * torch.sigmoid(t), "relu": torch.relu, "gelu": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}[act](g)
    ref = g * u
    assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-3).all()


@pytest.mark.parametrize("m,n,k,tiles", [(65, 128, 64, 1), (130, 384, 192, 3), (257, 200, 320, 2), (777, 3072, 448, 4)])
def test_pair_int4_equals_the_split_kernel(m, n, k, tiles):
    g = torch.Generator().manual_seed(7)
    q = torch.randint(0, 16, (n, k), generator=g, dtype=torch.uint8)
    scale = (torch.rand(n, k // 32, generator=g) * 0.01 + 0.001).half()
    zero = torch.randint(0, 16, (n, k // 32), generator=g, dtype=torch.uint8)
    w = W4Weight.from_quantized(q, scale, zero, "cuda")
    x = _rows(m, k, 8)
    one = ops.linear(x, w, out_fp32=True, splits=1)
    pair = ops.linear(x, w, out_fp32=True, splits=-tiles)
    ops.check_kernel_status()
    assert torch.equal(one, pair)       # the same bf16 weights, summed in the same order
    ref = x.double() @ w.dequantize().double().cuda().t()
    assert ((pair.double() - ref).abs() <= k * 2.0 ** -24 * 2 + 1e-6).all()


@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("tokens,tile", [(40, 32), (90, 64), (300, 128), (500, 256)])
@pytest.mark.parametrize("n,k", [(384, 192), (256, 128)])
def test_pair_experts(half, tokens, tile, n, k):
    experts, top = 5, 2
    g = torch.Generator(device="cuda").manual_seed(9)
    codes = torch.randint(0, 16, (experts, n, k), generator=g, device="cuda", dtype=torch.uint8)
    scales = torch.randint(118, 124, (experts, n, k // 32), generator=g, device="cuda", dtype=torch.uint8)
    w = Fp4Experts.from_codes(codes, scales, "cuda", half=half)
    bias = _rows(experts, n, 10)
    plan = ops.moe_route(torch.randn(tokens, experts, generator=g, device="cuda"), top, token_tile=tile)
    x = _rows(tokens * top, k, 11)
    x = x.half() if half else x
    got = ops.moe_gemm(x, w, plan, bias)
    ops.check_kernel_status()
    grid = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device="cuda")
    full = torch.cat([grid, -grid])[codes.long()] * torch.exp2(scales.double() - 127).repeat_interleave(32, -1)
    offs = plan.expert_offsets.tolist()
    for e in range(experts):
        rows = slice(offs[e], offs[e + 1])
        ref = x[rows].double() @ full[e].t() + bias[e].double()
        assert ((got[rows].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()


# ---- several tiles per cluster: barriers, stages, records and accumulators carry on from one tile to the next, over tiles that end on a stage of one k-block
def _within(got, x, w, add=None, out_bits=None):
    """`got` against x @ w.T (+ add): the bound of 32-bit sums over k in any order, and half a place of the result's type (out_bits: its significand)."""
    ref = x.double() @ w.double().t()
    bound = x.shape[1] * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())
    if add is not None:
        ref = ref + add.double()
    if out_bits:
        bound = bound + 2.0 ** -out_bits * ref.abs()
    return bool(((got.double() - ref).abs() <= bound + 2.0 ** -22 * ref.abs() + 1e-30).all())


def _int4(n, k, seed, interleaved=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randint(0, 16, (n, k), generator=g, device="cuda", dtype=torch.uint8)
    scale = (torch.rand(n, k // 32, generator=g, device="cuda") * 0.01 + 0.001).half()
    zero = torch.randint(0, 16, (n, k // 32), generator=g, device="cuda", dtype=torch.uint8)
    return W4Weight.from_quantized(q, scale, zero, "cuda", interleaved=interleaved)


@pytest.mark.parametrize("m,n,k,tiles", [(300, 20000, 1216, 2), (70, 40000, 64, 1), (1000, 5000, 704, 8), (2500, 3072, 3072, 10)])
def test_pair_int4_many_tiles(m, n, k, tiles):
    w, x = _int4(n, k, 21), _rows(m, k, 22)
    pair = ops.linear(x, w, out_fp32=True, splits=-tiles)
    ops.check_kernel_status()
    assert torch.equal(pair, ops.linear(x, w, out_fp32=True, splits=1))      # the same bf16 weights, summed in the same order
    assert _within(pair, x, w.dequantize())


def test_pair_int4_epilogues():
    m, n, k = 333, 1480, 576
    w, x, bias, res = _int4(n, k, 23), _rows(m, k, 24), _rows(1, n, 25)[0], _rows(m, n, 26)
    full = w.dequantize()
    got = ops.linear(x, w, bias, residual=res, splits=-3)
    ops.check_kernel_status()
    assert _within(got, x, full, bias + res.double(), out_bits=8)
    gated = _int4(2 * 768, k, 27, interleaved=True)
    got = ops.gate_up_act(x, gated, _rows(1, 2 * 768, 28)[0], "silu", splits=-2)
    one = ops.gate_up_act(x, gated, _rows(1, 2 * 768, 28)[0], "silu", splits=1)
    ops.check_kernel_status()
    assert torch.equal(got, one)
    y = (x.double() @ gated.dequantize().double().t() + _rows(1, 2 * 768, 28)[0].double()).view(m, 12, 2, 64)
    g, u = y[:, :, 0].reshape(m, -1), y[:, :, 1].reshape(m, -1)
    ref = torch.nn.functional.silu(g) * u
    # sums within k * 2^-23 of the sums of magnitudes (below 60), silu with a slope of at most 1.1, half a place of bf16
    assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + k * 2.0 ** -23 * 60 * (1.1 * u.abs() + g.abs() + 1)).all()


@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("tokens,tile,n,k", [(400, 32, 1280, 1216), (900, 64, 1408, 704), (3000, 256, 640, 576)])
def test_pair_experts_many_tiles(half, tokens, tile, n, k):
    experts, top = 40, 4
    g = torch.Generator(device="cuda").manual_seed(29)
    codes = torch.randint(0, 16, (experts, n, k), generator=g, device="cuda", dtype=torch.uint8)
    scales = torch.randint(118, 124, (experts, n, k // 32), generator=g, device="cuda", dtype=torch.uint8)
    w = Fp4Experts.from_codes(codes, scales, "cuda", keep_host=False, half=half)
    plan = ops.moe_route(torch.randn(tokens, experts, generator=g, device="cuda"), top, token_tile=tile)
    assert int(plan.num_tiles) * -(-n // 256) > 2 * 74
    x = _rows(tokens * top, k, 30)
    x = x.half() if half else x
    got = ops.moe_gemm(x, w, plan)
    ops.check_kernel_status()
    grid = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device="cuda")
    grid = torch.cat([grid, -grid])
    offs = plan.expert_offsets.tolist()
    for e in range(experts):
        rows = slice(offs[e], offs[e + 1])
        assert _within(got[rows], x[rows], grid[codes[e].long()] * torch.exp2(scales[e].double() - 127).repeat_interleave(32, -1), out_bits=8)


# ---- results whose rows do not start on 16 bytes, column ranges, and an activation of every column
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("shift,pitch", [(0, 0), (1, 5), (8, 8), (3, 13)])
def test_pair_rows_of_any_alignment(fp32, shift, pitch):
    m, n, k = 290, 520, 200
    x, w, bias = _rows(m, k, 31), _rows(n, k, 32), _rows(1, n, 33)[0]
    res = _rows(m, n + pitch + shift, 34)[:, shift:shift + n]
    res = res.float() if fp32 else res
    wide = torch.full((m, n + pitch + shift), 3.0, dtype=torch.float32 if fp32 else torch.bfloat16, device="cuda")
    out = wide[:, shift:shift + n]
    ops.linear(x, w, bias, residual=res, out_fp32=fp32, out=out, splits=-2)
    ops.check_kernel_status()
    assert _within(out, x, w, bias.double() + res.double(), out_bits=None if fp32 else 8)
    assert (wide[:, :shift] == 3).all() and (wide[:, shift + n:] == 3).all()


@pytest.mark.parametrize("act", ["silu", "gelu", "relu", "gelu_erf", "relu2"])
def test_pair_activation_of_every_column(act):
    m, n, k = 290, 520, 200
    x, w = _rows(m, k, 35), _rows(n, k, 36)
    wide = torch.zeros(m, n + 3, dtype=torch.bfloat16, device="cuda")
    out = wide[:, 3:]
    ops._gemm(x, w, out, None, None, (1 + ops._ACT[act]) << 8, -2)
    ops.check_kernel_status()
    f = torch.nn.functional
    ref = {"silu": f.silu, "gelu": lambda t: f.gelu(t, approximate="tanh"), "relu": torch.relu, "gelu_erf": f.gelu,
           "relu2": lambda t: torch.relu(t) ** 2}[act](x.double() @ w.double().t())
    # the sums within k * 2^-23 of their magnitudes (below 60), slopes of at most 1.2 (squares: 2 * 30), fast exponentials and tanh within 2^-11 of half an argument below 8 (beyond, they saturate)
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + k * 2.0 ** -23 * 60 * (60 if act == "relu2" else 1.2) + 2e-3).all()
    assert (wide[:, :3] == 0).all()
