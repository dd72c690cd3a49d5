"""The vector form of rotary embedding and cache append (csrc/elementwise.cu): one CTA per token or per pass over the heads, idle threads, several passes, partial
rotation, skipped slots, and the calls that fall back to the general form, against the rotation in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from onnxruntime_genai_b200 import ops


def _rotate(x, c, s):
    h = c.shape[-1]
    a, b = x[..., :h], x[..., h:2 * h]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * h:]], -1)


@pytest.mark.parametrize("T", [1, 63, 64, 130])
@pytest.mark.parametrize("Hq,Hkv,D,rot", [(32, 32, 96, 96), (32, 8, 256, 256), (40, 8, 80, 64), (4, 1, 16, 16), (64, 8, 64, 32), (3, 1, 128, 0), (0, 5, 128, 128)])
@pytest.mark.parametrize("pitch,cached", [(0, True), (8, True), (3, True), (0, False)])
def test_rotation_and_append(T, Hq, Hkv, D, rot, pitch, cached):
    g = torch.Generator(device="cuda").manual_seed(T + D)
    heads, places = Hq + 2 * Hkv, T + 7
    # a pitch of 3 elements takes the general form: the same results
    wide = torch.randn(T, heads * D + pitch, generator=g, device="cuda").to(torch.bfloat16)
    qkv = wide[:, :heads * D]
    whole = wide.clone()
    before = whole[:, :heads * D]
    pos = torch.randint(-2, 60, (T,), generator=g, device="cuda", dtype=torch.int32)      # positions are clamped to the tables
    slots = torch.randperm(places, generator=g, device="cuda")[:T].to(torch.int32)
    slots[T // 2] = -1
    cos, sin = (torch.rand(50, max(1, rot // 2), generator=g, device="cuda") * 2 - 1 for _ in range(2))
    kc, vc = (torch.full((places, Hkv, D), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.rope_kv_append(qkv, pos, slots if cached else None, cos if rot else None, sin if rot else None, kc, vc, Hq, Hkv, D, rot)
    ops.check_kernel_status()
    x_bits = before.reshape(T, heads, D)
    x = x_bits.double()
    at = pos.long().clamp(0, 49)
    c, s = (t[at].double()[:, None, :rot // 2] for t in (cos, sin))
    want_q, want_k = _rotate(x[:, :Hq], c, s), _rotate(x[:, Hq:Hq + Hkv], c, s)
    # three roundings of values below 8 in 32 bits, and the rounding to bf16
    close = lambda got, want: ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -19).all()  # noqa: E731
    after = qkv.reshape(T, heads, D)
    assert close(after[:, :Hq], want_q)
    assert torch.equal(wide[:, Hq * D:], whole[:, Hq * D:])
    kept = slots >= 0 if cached else torch.zeros(T, dtype=torch.bool, device="cuda")
    rows = slots[kept].long()
    assert close(kc[rows], want_k[kept])
    assert torch.equal(vc[rows], x_bits[kept, Hq + Hkv:])
    others = torch.ones(places, dtype=torch.bool, device="cuda")
    others[rows] = False
    assert (kc[others] == 7).all() and (vc[others] == 7).all()
