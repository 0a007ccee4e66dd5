"""Grouped products whose feature tiles are lower than 128 rows: the last tile of a group ends inside the
tile (its box reaches into the next group's matrix, or past the last one), groups without rows, one token."""
import pytest
import torch

from easy_to_hard_b200.ops import gemm

U = 2.0 ** -8                       # half a unit of the last of the 8 bits of bf16

# features, K, groups, tokens, choices per token
CASES = [(2752, 2048, 4, 32, 2), (1368, 192, 4, 32, 2), (712, 256, 16, 64, 4), (1032, 128, 4, 1, 2),
         (904, 128, 8, 1, 3), (3456, 320, 4, 64, 2), (1104, 512, 5, 33, 2)]


@pytest.mark.parametrize("F,K,n,tokens,top", CASES)
def test_heights_are_low(F, K, n, tokens, top):
    th = gemm.group_height(F, n, tokens, tokens * top)
    assert th is not None and 64 <= th < 128 and th % 8 == 0
    live = min(n, top) if tokens == 1 else n
    assert -(-F // th) * live <= 148 * (1 if tokens == 1 else 2)


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("F,K,n,tokens,top", CASES)
def test_low_tiles(F, K, n, tokens, top, gated):
    gen = torch.Generator(device="cuda").manual_seed(F + K)
    host = torch.Generator().manual_seed(tokens)
    sel = torch.stack([torch.randperm(n, generator=host)[:top] for _ in range(tokens)]).flatten()
    if n == 5:
        sel = torch.where(sel == 2, torch.tensor(0), sel)      # a group without rows among the others
        sel = sel.clamp(max=3)                                 # and the last one
    count = torch.bincount(sel, minlength=n).clamp(max=tokens)
    off = torch.zeros(n + 1, dtype=torch.int32)
    off[1:] = count.cumsum(0)
    T = tokens * top
    x = torch.randn(T, K, device="cuda", generator=gen).bfloat16()
    w1, w3 = ((torch.randn(n * F, K, device="cuda", generator=gen) / K ** 0.5).bfloat16()
              for _ in range(2))
    out = torch.full((T, F), 7.0, device="cuda").bfloat16()
    group_off = off.cuda()
    if gated:
        gemm.grouped_swiglu(x, w1, w3, out, group_off, n, tokens)
    else:
        gemm.grouped_linear(x, w1, out, group_off, n, tokens)
    for g in range(n):
        a, b = int(off[g]), int(off[g + 1])
        if a == b:
            continue
        xs, wa = x[a:b].double(), w1[g * F:(g + 1) * F].double()
        want = xs @ wa.T
        slack = 2.0 ** -23 * K * (xs.abs() @ wa.abs().T)       # fp32 sums of K products
        tol = U * want.abs() + slack
        if gated:
            up = xs @ w3[g * F:(g + 1) * F].double().T
            ups = 2.0 ** -23 * K * (xs.abs() @ w3[g * F:(g + 1) * F].double().abs().T)
            sig = torch.sigmoid(want)
            # |silu'| < 1.1: gate rounded, SiLU rounded, up rounded, product rounded
            dsilu = 1.1 * (U * want.abs() + slack) + 1.01 * U * (want * sig).abs()
            dup = U * up.abs() + ups
            want = want * sig
            tol = dsilu * (up.abs() + dup) + want.abs() * dup
            want = want * up
            tol = tol + U * (want.abs() + tol)
        assert ((out[a:b].double() - want).abs() <= 1.001 * tol + 1e-30).all()
    assert (out[int(off[-1]):] == 7.0).all()                   # rows of no group stay as they were


# token tiles of 128 and of 256 rows, at their edges
WIDE = [(2752, 256, 4, 65, 2), (904, 192, 8, 100, 2), (1776, 128, 8, 128, 2), (1368, 320, 4, 129, 3),
        (2752, 128, 4, 200, 2), (1104, 128, 5, 256, 2)]


@pytest.mark.parametrize("F,K,n,tokens,top", WIDE)
def test_heights_are_low_for_wide_token_tiles(F, K, n, tokens, top):
    test_heights_are_low(F, K, n, tokens, top)


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("F,K,n,tokens,top", WIDE)
def test_low_tiles_of_many_tokens(F, K, n, tokens, top, gated):
    test_low_tiles(F, K, n, tokens, top, gated)


def test_heights_that_gain_nothing_are_left_out():
    """Groups whose tiles of 128 rows cover the SMs nearly as well keep them."""
    for F in range(64, 6000, 8):
        for n in (1, 4, 5, 8, 16):
            th = gemm.group_height(F, n, 32, 32 * n)
            assert th is None or 64 <= th <= 112
    assert gemm.group_height(2048, 8, 16, 32) is None
