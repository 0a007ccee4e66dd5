"""One token tile, more than 16 rows (ops/csrc/gemm_umma.cu with the epilogue compiled in): the widths
at which the tile plan changes, contractions off the 64-wide blocks, both ring sizes, every epilogue,
against fp32 matmuls."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _status_ok():
    from easy_to_hard_b200.ops import _lib
    torch.cuda.synchronize()
    assert _lib.read_status() == 0


# widths: one tile, split-K of 4 and 2, plan of 64 to 120 rows with K in two, more tiles than SMs, more
# than two tiles per SM; contractions: 64-wide blocks, 8 past them, fewer blocks than stages
@pytest.mark.parametrize("T", [17, 64, 65, 128])
@pytest.mark.parametrize("F,K", [(96, 256), (2048, 2048), (5000, 512), (9600, 520), (12296, 1024),
                                 (19080, 264), (32016, 128), (40000, 72)])
def test_widths(T, F, K):
    """fp32 out: at most K 2^-23 sum |x w| from the exact sum; bf16 out: one more rounding of 2^-8."""
    from easy_to_hard_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(F + T)
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(F, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    want = x.double() @ w.double().t()
    tol = K * 2.0 ** -23 * (x.float().abs() @ w.float().abs().t())
    out = torch.full((T, F + 8), 7.0, device="cuda")
    gemm.linear(x, w, out=out[:, :F])
    _status_ok()
    assert bool(((out[:, :F] - want).abs() <= tol).all()) and bool((out[:, F:] == 7.0).all())
    got = gemm.linear(x, w)
    assert bool(((got - want).abs() <= tol + 2.0 ** -8 * want.abs()).all())
    res = torch.randn(T, F, device="cuda", generator=g).bfloat16()
    got = gemm.linear_residual(x, w, res)
    ref = res.double() + want
    assert bool(((got - ref).abs() <= tol + 2.0 ** -8 * (want.abs() + ref.abs())).all())
    acc = res.float()
    gemm.gemm(w, x, epi=gemm.EPI_RESIDUAL_F32, out=acc, aux=acc)
    assert bool(((acc - ref).abs() <= tol + 2.0 ** -22 * (want.abs() + ref.abs())).all())
    _status_ok()


@pytest.mark.parametrize("T", [17, 64, 100])
@pytest.mark.parametrize("F,K", [(688, 256), (11008, 136), (19200, 128), (22016, 192)])
def test_gated(T, F, K):
    from easy_to_hard_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(F + T)
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w1, w3 = ((torch.randn(F, K, device="cuda", generator=g) * K ** -0.5).bfloat16() for _ in range(2))
    got = gemm.linear_swiglu(x, w1, w3)
    _status_ok()
    a, b = x.double() @ w1.double().t(), x.double() @ w3.double().t()
    want = torch.nn.functional.silu(a) * b
    # three roundings to bf16 before the last one; silu changes by at most 1.1 times its input
    tol = 2.0 ** -8 * (2.2 * (a.abs() * b.abs()) + 2 * want.abs()) + 1e-3
    assert bool(((got - want).abs() <= tol).all())


@pytest.mark.parametrize("H,G,D,K", [(32, 32, 128, 256), (64, 8, 128, 192), (8, 2, 64, 264)])
@pytest.mark.parametrize("T,pos", [(17, 0), (64, 39), (33, 40)])
def test_rope_and_cache(T, pos, H, G, D, K):
    """Against the form of the kernel without a compiled-in epilogue (64-row tiles); position 40 lies
    behind the cache."""
    from easy_to_hard_b200.ops import gemm, reference
    S = 40
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn((H + 2 * G) * D, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    freqs = reference.precompute_freqs_cis(S, D, 10000.0, dtype=torch.bfloat16, device="cuda")
    at = torch.tensor([pos], dtype=torch.int32, device="cuda")
    outs = []
    for kw in ({}, dict(tf=64, splitk=1)):
        q = torch.zeros(T, H * D, device="cuda").bfloat16()
        kc, vc = (torch.zeros(T, G, S, D, device="cuda").bfloat16() for _ in range(2))
        gemm.linear_qkv_rope(x, w, q, freqs=freqs, pos_base=at, sq=1, n_head=H, n_kv=G, head_dim=D,
                             kcache=kc, vcache=vc, **kw)
        outs.append((q.float(), kc.float(), vc.float()))
    _status_ok()
    for a, b in zip(*outs):        # two bf16 roundings of sums in another order
        assert bool(((a - b).abs() <= 2.0 ** -6 * b.abs() + 2.0 ** -7).all())
    assert bool((outs[0][1] == 0).all()) == (pos >= S)


@pytest.mark.parametrize("H,G,D,K", [(32, 32, 128, 256), (64, 8, 128, 192), (8, 2, 64, 264)])
@pytest.mark.parametrize("T,pos", [(17, 0), (64, 39), (128, 7)])
def test_rope_and_cache_against_the_rotation(T, pos, H, G, D, K):
    """The fp32 sum and its rotation may each differ by one bf16 step, of the larger of the pair."""
    from easy_to_hard_b200.ops import gemm, reference
    S = 40
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn((H + 2 * G) * D, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    freqs = reference.precompute_freqs_cis(S, D, 10000.0, dtype=torch.bfloat16, device="cuda")
    at = torch.tensor([pos], dtype=torch.int32, device="cuda")
    q = torch.zeros(T, H * D, device="cuda").bfloat16()
    kc, vc = (torch.zeros(T, G, S, D, device="cuda").bfloat16() for _ in range(2))
    gemm.linear_qkv_rope(x, w, q, freqs=freqs, pos_base=at, sq=1, n_head=H, n_kv=G, head_dim=D,
                         kcache=kc, vcache=vc)
    _status_ok()
    raw = (x.double() @ w.double().t()).to(torch.bfloat16).view(T, 1, H + 2 * G, D)
    f = freqs[pos:pos + 1]
    wants = (reference.apply_rotary_emb(raw[:, :, :H], f), reference.apply_rotary_emb(raw[:, :, H:H + G], f),
             raw[:, :, H + G:])
    for got, want in zip((q.view(T, H, D), kc[:, :, pos], vc[:, :, pos]), wants):
        want = want[:, 0].float()
        assert bool(((got.float() - want).abs() <= 2.0 ** -6 * want.abs().max()).all())
        assert float((got.float() - want).norm()) <= 2.0 ** -8 * float(want.norm())
    other = torch.arange(S, device="cuda") != pos
    assert not kc[:, :, other].any() and not vc[:, :, other].any()
