"""Decode attention with few (sequence, head) pairs: contexts on both sides of the line up to which one CTA takes
a pair by itself, mixed in one launch, against 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,G,D", [(1, 32, 32, 128), (3, 4, 4, 64), (2, 16, 2, 128), (2, 8, 2, 128),
                                     (1, 8, 2, 64), (5, 40, 40, 128)])
@pytest.mark.parametrize("pos", [0, 31, 63, 64, 127, 159, 160, 161, 319, 320, 321, 500])
def test_contexts(B, H, G, D, pos):
    from easy_to_hard_b200.ops import _lib, functional as Fn
    S = 512
    g = torch.Generator(device="cuda").manual_seed(pos + H)
    kc, vc = (torch.randn(B, G, S, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    q = torch.randn(B, H * D, device="cuda", generator=g).bfloat16()
    pads = torch.tensor([min(pos, 37 * b * b) for b in range(B)], device="cuda", dtype=torch.int32)
    p = torch.tensor([pos], device="cuda", dtype=torch.int32)
    for _ in range(2):                                    # (tickets are zero again after a launch)
        got = Fn.attn_decode(q, kc, vc, p, pads, H).double().view(B, H, D)
        for b in range(B):
            k, v = (t[b, :, int(pads[b]):pos + 1].double().repeat_interleave(H // G, 0) for t in (kc, vc))
            w = torch.softmax((k @ q[b].view(H, D, 1).double())[..., 0] / math.sqrt(D), -1)
            want = (w[..., None] * v).sum(1)
            mass = (w[..., None] * v.abs()).sum(1)
            # fp32 scores and sums, one rounding to bf16
            assert bool(((got[b] - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * mass + 1e-7).all())
    assert _lib.read_status() == 0
