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
