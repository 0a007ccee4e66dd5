"""Products of few rows whose CTAs take equal shares of the features: widths on both sides of the lines where
the split changes, odd widths, the rotation's pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
SM = 148


@pytest.mark.parametrize("T", [1, 8, 9, 16])
@pytest.mark.parametrize("bits", [16, 8])
@pytest.mark.parametrize("F", [16 * SM * 2, 16 * SM * 2 + 1, 5120, 16 * SM * 3 + 2, 16 * SM * 4, 16 * SM * 4 + 3,
                               32 * SM * 2, 12288, 32 * SM * 3 + 1, 32 * SM * 4 - 2, 32 * SM * 6 + 1])
@pytest.mark.parametrize("K", [64, 528, 4096])
def test_shares(T, bits, F, K):
    from easy_to_hard_b200.ops import _lib, gemm
    g = torch.Generator(device="cuda").manual_seed(F + K + T)
    if bits == 16:
        w, s = torch.randn(F, K, device="cuda", generator=g).bfloat16(), None
        wf = w.double()
    else:
        w = torch.randint(-128, 128, (F, K), device="cuda", generator=g, dtype=torch.int8)
        s = torch.rand(F, device="cuda", generator=g) + 0.5
        wf = w.double() * s.double()[:, None]
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    out = torch.full((T, F + 5), 7.0, device="cuda")
    gemm.gemm(w, x, epi=gemm.EPI_STORE_F32, out=out[:, :F], scale=s)
    want = x.double() @ wf.t()
    # fp32 sums of K products (and one product with the scale)
    tol = (K + 2) * 2.0 ** -23 * (x.double().abs() @ wf.abs().t()) + 1e-30
    assert bool(((out[:, :F].double() - want).abs() <= tol).all())
    assert bool((out[:, F:] == 7.0).all())
    assert _lib.read_status() == 0


@pytest.mark.parametrize("H,G,D", [(32, 32, 128), (40, 40, 64), (20, 10, 128)])
def test_rotation(H, G, D):
    """Against the unrotated product of the same kernel, turned pair by pair."""
    from easy_to_hard_b200.models.engine import _freqs
    from easy_to_hard_b200.ops import gemm
    T, K, S, pos = 5, 1024, 32, 11
    F = (H + 2 * G) * D
    w = torch.randn(F, K, device="cuda").bfloat16()
    x = (torch.randn(T, K, device="cuda") * 0.1).bfloat16()
    freqs = _freqs(S, D, 10000.0, torch.device("cuda"))
    kc, vc = (torch.zeros(T, G, S, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    q = torch.empty(T, H * D, device="cuda", dtype=torch.bfloat16)
    gemm.linear_qkv_rope(x, w, q, freqs=freqs, pos_base=torch.tensor([pos], device="cuda", dtype=torch.int32),
                         sq=1, n_head=H, n_kv=G, head_dim=D, kcache=kc, vcache=vc)
    y = x.double() @ w.double().t()
    c, s = freqs[pos].double().view(-1, 2).unbind(-1)
    z = y[:, : (H + G) * D].reshape(T, H + G, D // 2, 2)
    turned = torch.stack([z[..., 0] * c - z[..., 1] * s, z[..., 1] * c + z[..., 0] * s], -1).flatten(1)
    got = torch.cat([q, kc[:, :, pos].flatten(1)], 1).double()
    # the product is rounded to bf16 before it is turned, and the result once more
    mag = (z.abs().amax(-1, keepdim=True) * 2).expand_as(z).flatten(1)
    assert bool(((got - turned).abs() <= 2.0 ** -8 * (mag + turned.abs()) + 1e-3).all())
    assert bool(((vc[:, :, pos].flatten(1).double() - y[:, (H + G) * D:]).abs()
                 <= 2.0 ** -8 * y[:, (H + G) * D:].abs() + 1e-3).all())


@pytest.mark.parametrize("T", [1, 16])
@pytest.mark.parametrize("bits", [16, 8])
@pytest.mark.parametrize("F", [16 * SM * 3, 16 * SM * 4 - 1, 32 * SM * 3, 32 * SM * 4 - 2])
@pytest.mark.parametrize("K", [2048, 8192, 8208, 12288])
def test_shares_of_long_sums(T, bits, F, K):
    """On both sides of the lengths at which a product leaves the shares or takes eight warps."""
    test_shares(T, bits, F, K)
