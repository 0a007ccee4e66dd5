"""Forward flash attention against 64 bits: sizes at the edges of its tiles (128 queries, 64 keys), items of one
and of two query tiles, pairs of heads, several items per CTA, left pads up to whole rows, either sign
of the scale."""
import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _want(q, k, v, left, scale):
    B, Sq, H, D = q.shape
    Sk, G = k.shape[1], k.shape[2]
    q, k, v = (t.double().transpose(1, 2) for t in (q, k, v))
    k, v = (t.repeat_interleave(H // G, 1) for t in (k, v))
    i = torch.arange(Sq, device="cuda")[:, None] + Sk - Sq
    j = torch.arange(Sk, device="cuda")[None]
    ok = ((j <= i)[None] & (j[None] >= left[:, None, None])) | (j == i)[None]
    s = (q @ k.transpose(2, 3) * scale).masked_fill(~ok[:, None], -math.inf)
    p = torch.softmax(s, -1).nan_to_num(0.0)        # (a row that sees nothing: zeros)
    return (p @ v).transpose(1, 2), (p @ v.abs()).transpose(1, 2), torch.logsumexp(s, -1)


def _check(out, lse, q, k, v, left, scale):
    want, mass, lse_want = _want(q, k, v, left, scale)
    # probabilities and the result are rounded to bf16 (2^-8 of p and of o at most); fp32 scores of D products
    # and base-2 exponentials are far below
    tol = 2.0 ** -8 * (mass + want.abs()) * 1.02 + 1e-4 * mass
    assert bool(((out.double() - want).abs() <= tol).all())
    seen = lse_want > -math.inf
    err = (lse.double() - lse_want)[seen].abs()
    assert bool((err <= 1e-4 + 2.0 ** -20 * lse_want[seen].abs()).all())


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("B,H,G,Sq,Sk", [
    (1, 1, 1, 1, 1), (2, 2, 2, 1, 200), (1, 3, 3, 63, 63), (2, 2, 2, 64, 64), (1, 2, 2, 65, 65),
    (2, 3, 1, 127, 127), (1, 2, 2, 128, 129), (1, 2, 1, 129, 129), (1, 4, 4, 191, 191), (1, 4, 4, 193, 193),
    (2, 8, 2, 256, 256), (1, 8, 1, 257, 300), (3, 5, 5, 385, 385), (20, 16, 16, 320, 320),
    (9, 32, 8, 450, 450), (1, 2, 2, 300, 200)])
def test_forward(B, H, G, Sq, Sk, D):
    from easy_to_hard_b200.ops import _lib, flash
    g = torch.Generator(device="cuda").manual_seed(Sq * 7 + Sk + D)
    q = torch.randn(B, Sq, H, D, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(B, Sk, G, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    q[:, Sq // 2:] *= 6                              # rows whose maximum grows far enough to be raised
    for left in (torch.zeros(B, device="cuda", dtype=torch.int32),
                 torch.randint(0, Sk + 1, (B,), device="cuda", generator=g, dtype=torch.int32)):
        out, lse = flash.flash_fwd(q, k, v, left if bool(left.any()) else None, return_lse=True)
        _check(out, lse, q, k, v, left, 1.0 / math.sqrt(D))
    assert _lib.read_status() == 0


def test_negative_scale():
    from easy_to_hard_b200.ops import _lib
    B, H, S, D = 2, 2, 200, 128
    q, k, v = (torch.randn(B, S, H, D, device="cuda").bfloat16() for _ in range(3))
    out = torch.empty_like(q)
    lse = torch.empty(B, H, S, device="cuda")
    st = (S * H * D, H * D, D)
    rc = _lib.lib().e2h_flash_fwd(q.data_ptr(), *st, k.data_ptr(), v.data_ptr(), *st, out.data_ptr(), *st,
                                  lse.data_ptr(), None, B, H, H, S, S, D, C.c_float(-0.07),
                                  _lib.status_word(q.device).data_ptr(), _lib.stream())
    assert rc == 0
    _check(out, lse, q, k, v, torch.zeros(B, device="cuda", dtype=torch.int32), -0.07)
    assert _lib.read_status() == 0
