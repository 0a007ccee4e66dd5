"""The rotation of a training or scoring block: every token at its own position, as the block's caller
gives them, or inside the QKV product where these are promised to be in order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rotated(x, freqs, pos):
    """Interleaved pairs of x [T, H, D] at positions pos [T], in fp32."""
    f = freqs.float()[pos.long()][:, None]
    a, b = x.float()[..., 0::2], x.float()[..., 1::2]
    return torch.stack([a * f[..., 0] - b * f[..., 1], b * f[..., 0] + a * f[..., 1]], -1).flatten(2)


@pytest.mark.parametrize("B,S", [(1, 1), (2, 5), (3, 40), (2, 129), (5, 130)])
@pytest.mark.parametrize("H,G,D", [(4, 2, 64), (2, 2, 128)])
@pytest.mark.parametrize("in_order", [False, True])
def test_sequences_may_start_anywhere(B, S, H, G, D, in_order):
    """Left-padded rows, positions that repeat, sequences that start at different ones; the same with
    the promise that all start at one position. Bound: the fp32 sum and its rotation may each differ
    by one bf16 step."""
    from easy_to_hard_b200.models import fused_block as fb
    from easy_to_hard_b200.ops import _lib, functional as Fn, reference
    dim, T = H * D, B * S
    g = torch.Generator(device="cuda").manual_seed(T)

    def mk(*shape):
        return (torch.randn(*shape, device="cuda", generator=g) * shape[-1] ** -0.5).bfloat16()
    w = dict(wqkv=mk((H + 2 * G) * D, dim), wo=mk(dim, dim), w1=mk(96, dim), w3=mk(96, dim),
             w2=mk(dim, 96), attention_norm=torch.ones(dim, device="cuda").bfloat16(),
             ffn_norm=torch.ones(dim, device="cuda").bfloat16())
    x = torch.randn(T, dim, device="cuda", generator=g).bfloat16()
    freqs = reference.precompute_freqs_cis(300, D, 10000.0, device="cuda")
    start = torch.randint(-S, 150, (B, 1), device="cuda", generator=g)
    pos = (start + torch.arange(S, device="cuda")).clamp_min(0).to(torch.int32).flatten().contiguous()
    if in_order:
        pos = (7 + torch.arange(S, device="cuda", dtype=torch.int32)).repeat(B)
    shape = fb.BlockShape(B, S, H, G, D, 1e-5, in_order=in_order)
    _, a = fb.block_forward(x, w, freqs, pos, shape, keep=True)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    raw = (a["xn1f"].float() @ w["wqkv"].float().T).bfloat16().view(T, H + 2 * G, D)
    want = raw.float()
    want[:, : H + G] = _rotated(raw[:, : H + G], freqs, pos)
    got = a["qkv"].float().view(T, H + 2 * G, D)
    assert bool(((got - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -8 * want.abs().max()).all())
    # and what the backward undoes: the same rotation as the separate kernel's
    apart = Fn.rope(raw.reshape(T, -1).contiguous(), freqs, pos, H + G, D).view(T, H + 2 * G, D)
    assert bool(((apart.float()[:, : H + G] - want[:, : H + G]).abs()
                 <= 2.0 ** -7 * want.abs().max()).all())
