"""Products of up to 16 rows (ops/csrc/gemm_rows.cu) against fp32 matmuls and against the tcgen05
kernels, which an explicit split factor selects."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _status_ok():
    from easy_to_hard_b200.ops import _lib
    torch.cuda.synchronize()
    assert _lib.read_status() == 0


def _weight(F, K, bits, seed, pad=0):
    """(operand, per-feature scale or None, the bf16-exact matrix it stands for, in fp32)"""
    from easy_to_hard_b200.ops.gemm import Int4Weight
    g = torch.Generator(device="cuda").manual_seed(seed)
    if bits == 16:
        w = torch.randn(F, K + pad, device="cuda", generator=g).bfloat16()[:, :K]
        return w, None, w.float()
    if bits == 8:
        w = torch.randint(-128, 128, (F, K + 2 * pad), device="cuda", generator=g, dtype=torch.int8)
        w, s = w[:, :K], torch.rand(F, device="cuda", generator=g) * 0.01 + 0.001
        return w, s, w.float() * s[:, None]
    codes = torch.randint(0, 16, (F, K), device="cuda", generator=g, dtype=torch.int32)
    sz = (torch.rand(K // 64, F, 2, device="cuda", generator=g) * 0.1).bfloat16()
    w = Int4Weight.from_int(codes, sz, 64)
    return w, None, w.dequant().float()


def _bound(x, w):
    """fp32 sums of K products in any order differ from the exact sum by at most K 2^-23 sum |x w|
    (truncating adders included)."""
    return x.shape[1] * 2.0 ** -23 * (x.float().abs() @ w.abs().t()) + 1e-30


@pytest.mark.parametrize("T", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("bits,F,K", [(16, 16, 8), (16, 130, 72), (16, 4096, 1032), (16, 9504, 512),
                                      (8, 40, 16), (8, 256, 1040), (8, 9504, 4096), (4, 17, 128),
                                      (4, 384, 1408), (4, 9504, 1024), (16, 4744, 2056),
                                      (8, 4744, 2064), (4, 4744, 2176)])
def test_linear(T, bits, F, K):
    from easy_to_hard_b200.ops import gemm
    w, s, wf = _weight(F, K, bits, T + F, pad=8)
    x = torch.randn(T, K + 16, device="cuda").bfloat16()[:, 8:8 + K]      # rows on 16-byte boundaries
    assert gemm.rows_rule(w, None, x, gemm.EPI_STORE_F32)
    want = x.double() @ wf.double().t()
    out = torch.full((T, F + 3), 7.0, device="cuda")
    gemm.linear(x, w, out=out[:, :F], scale=s)
    _status_ok()
    assert bool(((out[:, :F] - want).abs() <= _bound(x, wf)).all())
    assert bool((out[:, F:] == 7.0).all())
    got = gemm.linear(x, w, scale=s)
    tol = _bound(x, wf) + want.abs() * 2.0 ** -8
    assert bool(((got - want).abs() <= tol).all())


@pytest.mark.parametrize("T", [1, 8, 11])
@pytest.mark.parametrize("bits", [16, 8, 4])
def test_epilogues_match_the_wide_kernels(T, bits):
    """bf16 results of two correct fp32 sums differ by a rounding (2^-8 of the value) at most, here
    after one more bf16 rounding and a product of two."""
    from easy_to_hard_b200.ops import gemm
    F, K = 640, 1024
    w, s, _ = _weight(F, K, bits, 3)
    w3, s3, _ = _weight(F, K, bits, 4)
    x = (torch.randn(T, K, device="cuda") * 0.05).bfloat16()
    res = torch.randn(T, F, device="cuda").bfloat16()
    both = None if s is None else torch.cat([s, s3])

    def close(a, b):
        a, b = a.float(), b.float()
        assert bool(((a - b).abs() <= 2.0 ** -6 * b.abs() + 2.0 ** -8 * b.abs().mean()).all())
    kw = dict(splitk=1)
    close(gemm.linear_residual(x, w, res, scale=s), gemm.linear_residual(x, w, res, scale=s, **kw))
    close(gemm.linear_swiglu(x, w, w3, scale=both), gemm.linear_swiglu(x, w, w3, scale=both, **kw))
    if bits == 16:
        for a, b in zip(gemm.linear_dual(x, w, w3), gemm.linear_dual(x, w, w3, **kw)):
            close(a, b)
        acc = torch.randn(T, F, device="cuda")
        other = acc.clone()
        gemm.gemm(w, x, epi=gemm.EPI_RESIDUAL_F32, out=acc, aux=acc)
        gemm.gemm(w, x, epi=gemm.EPI_RESIDUAL_F32, out=other, aux=other, **kw)
        close(acc, other)
        bias = torch.randn(F, device="cuda")
        y, t = torch.empty(T, 512, device="cuda").bfloat16(), torch.empty(T, 128, device="cuda")
        y2, t2 = torch.empty_like(y), torch.empty_like(t)
        gemm.linear_packed(x, w, y, bias=bias, act_from=256, tail=t, act="gelu")
        gemm.gemm(w, x, epi=gemm.EPI_STORE_BF16, out=y2, bias=bias, act_from=256, tail=t2,
                  tail_from=512, act="gelu", **kw)
        close(y, y2)
        close(t, t2)
    _status_ok()


@pytest.mark.parametrize("T,sq,pos", [(1, 1, 0), (8, 1, 37), (16, 1, 63), (12, 6, 3), (5, 1, 64)])
@pytest.mark.parametrize("bits", [16, 8, 4])
def test_rope_and_cache(T, sq, pos, bits):
    """The last position case lies outside the cache: nothing is rotated, no key or value is kept."""
    from easy_to_hard_b200.ops import gemm, reference
    H, G, D, S, K = 4, 2, 64, 64, 256
    w, s, _ = _weight((H + 2 * G) * D, K, bits, 5)
    x = (torch.randn(T, K, device="cuda") * 0.05).bfloat16()
    freqs = reference.precompute_freqs_cis(S, D, 10000.0, dtype=torch.bfloat16, device="cuda")
    at = torch.tensor([pos], dtype=torch.int32, device="cuda")
    outs = []
    for kw in ({}, dict(splitk=1)):
        q = torch.zeros(T, H * D, device="cuda").bfloat16()
        kc, vc = (torch.zeros(T // sq, G, S, D, device="cuda").bfloat16() for _ in range(2))
        gemm.linear_qkv_rope(x, w, q, freqs=freqs, pos_base=at, sq=sq, n_head=H, n_kv=G, head_dim=D,
                             kcache=kc, vcache=vc, scale=s, **kw)
        outs.append((q.float(), kc.float(), vc.float()))
    _status_ok()
    for a, b in zip(*outs):
        assert bool(((a - b).abs() <= 2.0 ** -6 * b.abs() + 2.0 ** -7 * b.abs().max()).all())
    assert bool((outs[0][1] == 0).all()) == (pos >= S)


@pytest.mark.parametrize("T", [1, 8, 11, 16])
@pytest.mark.parametrize("bits", [16, 8, 4])
def test_epilogues(T, bits):
    """Against products in 64 bits. One rounding to bf16 (2^-9 of the value, 2^-8 here) at each value that
    the epilogue rounds; silu(a) b moves by at most 1.1 |b| per unit of a and |a| per unit of b."""
    from easy_to_hard_b200.ops import gemm
    F, K, one = 640, 1024, 2.0 ** -8
    w, s, wf = _weight(F, K, bits, 3)
    w3, s3, wf3 = _weight(F, K, bits, 4)
    x = (torch.randn(T, K, device="cuda") * 0.05).bfloat16()
    res = torch.randn(T, F, device="cuda").bfloat16()
    both = None if s is None else torch.cat([s, s3])
    a, b = x.double() @ wf.double().t(), x.double() @ wf3.double().t()
    ta, tb = _bound(x, wf), _bound(x, wf3)
    want = res.double() + a
    got = gemm.linear_residual(x, w, res, scale=s)
    assert bool(((got - want).abs() <= ta + one * (a.abs() + want.abs())).all())
    want = torch.nn.functional.silu(a) * b
    got = gemm.linear_swiglu(x, w, w3, scale=both)
    tol = 1.1 * b.abs() * (ta + one * a.abs()) + a.abs() * (tb + one * b.abs()) + 3 * one * want.abs()
    assert bool(((got - want).abs() <= 1.1 * tol + 1e-6).all())
    if bits == 16:
        for got, want, tol in zip(gemm.linear_dual(x, w, w3), (a, b), (ta, tb)):
            assert bool(((got - want).abs() <= tol + one * want.abs()).all())
        acc = torch.randn(T, F, device="cuda")
        want = acc.double() + a
        gemm.gemm(w, x, epi=gemm.EPI_RESIDUAL_F32, out=acc, aux=acc)
        assert bool(((acc - want).abs() <= ta + 2.0 ** -22 * (a.abs() + want.abs())).all())
        bias = torch.randn(F, device="cuda")
        y, t = torch.empty(T, 512, device="cuda").bfloat16(), torch.empty(T, 128, device="cuda")
        gemm.linear_packed(x, w, y, bias=bias, act_from=256, tail=t, act="gelu")
        z = a + bias.double()
        want = torch.cat([z[:, :256], torch.nn.functional.gelu(z[:, 256:512], approximate="tanh")], 1)
        assert bool(((y - want).abs() <= 1.2 * ta[:, :512] + one * want.abs() + 2.0 ** -10).all())
        assert bool(((t - z[:, 512:]).abs() <= ta[:, 512:] + 2.0 ** -22 * z[:, 512:].abs()).all())
    _status_ok()


def _rope_reference(x, wf, freqs, positions, H, G, D):
    """q, k, v [T, heads, D] of x: the products rounded to bf16, queries and keys rotated in 32 bits."""
    raw = (x.double() @ wf.double().t()).to(torch.bfloat16).float().view(x.shape[0], H + 2 * G, D)
    f = freqs.float()[positions.long()][:, None]
    a, b = raw[:, : H + G, 0::2], raw[:, : H + G, 1::2]
    turned = torch.stack([a * f[..., 0] - b * f[..., 1], b * f[..., 0] + a * f[..., 1]], -1).flatten(2)
    return turned[:, :H], turned[:, H:], raw[:, H + G:]


@pytest.mark.parametrize("T,sq,pos", [(1, 1, 0), (8, 1, 37), (16, 1, 63), (12, 6, 3)])
@pytest.mark.parametrize("bits", [16, 8, 4])
def test_rope_and_cache_against_the_rotation(T, sq, pos, bits):
    """The fp32 sum and its rotation may each differ by one bf16 step, of the larger of the pair."""
    from easy_to_hard_b200.ops import gemm, reference
    H, G, D, S, K = 4, 2, 64, 64, 256
    w, s, wf = _weight((H + 2 * G) * D, K, bits, 5)
    x = (torch.randn(T, K, device="cuda") * 0.05).bfloat16()
    freqs = reference.precompute_freqs_cis(S, D, 10000.0, dtype=torch.bfloat16, device="cuda")
    at = torch.tensor([pos], dtype=torch.int32, device="cuda")
    q = torch.zeros(T, H * D, device="cuda").bfloat16()
    kc, vc = (torch.zeros(T // sq, G, S, D, device="cuda").bfloat16() for _ in range(2))
    gemm.linear_qkv_rope(x, w, q, freqs=freqs, pos_base=at, sq=sq, n_head=H, n_kv=G, head_dim=D,
                         kcache=kc, vcache=vc, scale=s)
    _status_ok()
    positions = pos + torch.arange(T, device="cuda") % sq
    seq = torch.arange(T, device="cuda") // sq
    wants = _rope_reference(x, wf, freqs, positions, H, G, D)
    for got, want in zip((q.view(T, H, D), kc[seq, :, positions], vc[seq, :, positions]), wants):
        assert bool(((got.float() - want).abs() <= 2.0 ** -6 * want.abs().max()).all())
        assert float((got.float() - want).norm()) <= 2.0 ** -8 * float(want.norm())
    live = torch.zeros(T // sq, S, dtype=torch.bool, device="cuda")
    live[seq, positions] = True
    assert not kc.transpose(1, 2)[~live].any() and not vc.transpose(1, 2)[~live].any()
