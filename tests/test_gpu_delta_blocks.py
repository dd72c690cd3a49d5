"""The prompt kernel of the gated delta rule (csrc/linear_attention.cu), which walks tokens in blocks of four: lengths around a block and a chunk, empty requests,
head sizes around its tiles, against the recurrence in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from onnxruntime_genai_b200 import ops


def _recurrence(q, k, v, g, beta, state, lens, past, slots):
    out = torch.zeros(v.shape, dtype=torch.float64)
    rep, at = v.shape[1] // q.shape[1], 0
    for r, n in enumerate(lens):
        S = state[slots[r]].double() if past[r] else torch.zeros_like(state[slots[r]]).double()
        for t in range(at, at + n):
            kt, qt = (x[t].double().repeat_interleave(rep, 0) for x in (k, q))
            S = S * torch.exp(g[t].double())[:, None, None]
            d = (v[t].double() - torch.einsum("hij,hi->hj", S, kt)) * beta[t].double()[:, None]
            S = S + kt[:, :, None] * d[:, None, :]
            out[t] = torch.einsum("hij,hi->hj", S, qt)
        if n:
            state[slots[r]] = S.to(state.dtype)
        at += n
    return out


@pytest.mark.parametrize("Hk,Hv,dk,dv", [(1, 2, 8, 5), (2, 2, 64, 17), (1, 3, 65, 16), (2, 4, 128, 40), (1, 1, 136, 33), (1, 2, 256, 16), (1, 1, 20, 3)])
@pytest.mark.parametrize("lens", [[1], [4, 3, 0, 5], [33, 2, 31, 32], [70]])
def test_blocks_follow_the_recurrence(Hk, Hv, dk, dv, lens):
    gen = torch.Generator().manual_seed(sum(lens) + dk)
    T, B = sum(lens), len(lens)
    unit = lambda *s: torch.nn.functional.normalize(torch.randn(*s, generator=gen), dim=-1).to(torch.bfloat16)  # noqa: E731
    q, k, v = unit(T, Hk, dk), unit(T, Hk, dk), torch.randn(T, Hv, dv, generator=gen).to(torch.bfloat16)
    g, beta = -torch.rand(T, Hv, generator=gen), torch.rand(T, Hv, generator=gen)
    state = torch.randn(B + 1, Hv, dk, dv, generator=gen) * 0.3
    slots = torch.randperm(B + 1, generator=gen)[:B].to(torch.int32)
    past = [3 * (r % 2) for r in range(B)]
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    dev_state = state.cuda()
    got = ops.gated_delta(q.cuda(), k.cuda(), v.cuda(), g.cuda(), beta.cuda(), dev_state, slots.cuda(), cu, torch.tensor(past, dtype=torch.int32).cuda())
    ops.check_kernel_status()
    want = _recurrence(q, k, v, g, beta, state, lens, past, slots.tolist())
    # unit keys contract the state: 32-bit sums of dk products per token, at most 70 of them, on values of the order of 1 .. 10; half a place of bf16
    assert ((got.cpu().double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
    assert torch.allclose(dev_state.cpu(), state, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("Hk,Hv,dk,dv,B", [(2, 4, 64, 128, 11), (2, 4, 40, 65, 20), (2, 4, 128, 128, 11), (4, 4, 100, 130, 11), (2, 2, 200, 64, 40), (1, 4, 256, 128, 11)])
@pytest.mark.parametrize("longest", [2, 5, 9, 17, 50])
def test_many_requests(Hk, Hv, dk, dv, B, longest):
    """More column tiles than fit the GPU at once (the form with eight warps), and portions of a few tokens, which are walked one at a time."""
    gen = torch.Generator().manual_seed(dk + longest)
    lens = [longest] + [int(n) for n in torch.randint(0, longest + 1, (B - 1,), generator=gen)]
    T = sum(lens)
    unit = lambda *s: torch.nn.functional.normalize(torch.randn(*s, generator=gen), dim=-1).to(torch.bfloat16)  # noqa: E731
    q, k, v = unit(T, Hk, dk), unit(T, Hk, dk), torch.randn(T, Hv, dv, generator=gen).to(torch.bfloat16)
    g, beta = -torch.rand(T, Hv, generator=gen), torch.rand(T, Hv, generator=gen)
    state = torch.randn(B + 1, Hv, dk, dv, generator=gen) * 0.3
    slots = torch.randperm(B + 1, generator=gen)[:B].to(torch.int32)
    past = [3 * (r % 2) for r in range(B)]
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    dev_state = state.cuda()
    got = ops.gated_delta(q.cuda(), k.cuda(), v.cuda(), g.cuda(), beta.cuda(), dev_state, slots.cuda(), cu, torch.tensor(past, dtype=torch.int32).cuda(), longest)
    ops.check_kernel_status()
    want = _recurrence(q, k, v, g, beta, state, lens, past, slots.tolist())
    # as above: at most 50 tokens
    assert ((got.cpu().double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
    assert torch.allclose(dev_state.cpu(), state, rtol=1e-4, atol=1e-4)


def test_a_later_token_that_is_not_finite_leaves_earlier_ones_alone():
    gen = torch.Generator().manual_seed(5)
    T, H, d = 8, 1, 64
    unit = lambda *s: torch.nn.functional.normalize(torch.randn(*s, generator=gen), dim=-1).to(torch.bfloat16).cuda()  # noqa: E731
    q, k, v = unit(T, H, d), unit(T, H, d), unit(T, H, d)
    g, beta = torch.full((T, H), -0.1).cuda(), torch.full((T, H), 0.5).cuda()
    one = lambda x: torch.tensor(x, dtype=torch.int32).cuda()  # noqa: E731
    run = lambda vv: ops.gated_delta(q, k, vv, g, beta, torch.zeros(1, H, d, d).cuda(), one([0]), one([0, T]), one([0]))  # noqa: E731
    clean = run(v)
    bad = v.clone()
    bad[6] = float("nan")
    got = run(bad)
    assert torch.equal(got[:6], clean[:6]) and torch.isnan(got[6:]).all()
