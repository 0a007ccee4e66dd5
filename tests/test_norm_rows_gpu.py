"""RMSNorm kernels whose blocks stay and walk the rows: rows around the resident blocks, widths with idle
threads, embedding rows, in-place gradients."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = [1, 255, 256, 257, 2367, 2369, 5015]
DIMS = [8, 256, 1000, 1032, 4096, 5120, 8192]
U = 2.0 ** -8                       # half a unit of the last of the 8 bits of bf16


def _data(T, d, n, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + T * 31 + d)
    return [torch.randn(T, d, device="cuda", generator=g).bfloat16() for _ in range(n)] + \
        [(1 + 0.1 * torch.randn(d, device="cuda", generator=g)).bfloat16()]


def _check_forward(got, x, w, eps):
    x64 = x.double()
    want = x64 * torch.rsqrt(x64.pow(2).mean(-1, keepdim=True) + eps) * w.double()
    # two roundings to bf16; the fp32 sum of d squares is off by d 2^-24 at most, its root by half
    tol = ((1 + U) ** 2 - 1 + x.shape[1] * 2.0 ** -24 + 2.0 ** -21) * want.abs()
    assert bool(((got.double() - want).abs() <= tol).all())


@pytest.mark.parametrize("T", ROWS)
@pytest.mark.parametrize("d", DIMS)
def test_rows(T, d):
    from easy_to_hard_b200.ops import _lib, functional as Fn
    x, dy, res, w = _data(T, d, 3)
    _check_forward(Fn.rmsnorm(x, w, 1e-5), x, w, 1e-5)
    x64, g64 = x.double(), dy.double() * w.double()
    rstd = torch.rsqrt(x64.pow(2).mean(-1, keepdim=True) + 1e-5)
    a = g64 * rstd
    b = x64 * rstd.pow(3) / d * (g64 * x64).sum(-1, keepdim=True)
    b_abs = x64.abs() * rstd.pow(3) / d * (g64 * x64).abs().sum(-1, keepdim=True)
    for r in (None, res):
        want = a - b + (0 if r is None else r.double())
        fp32 = (d + 16) * 2.0 ** -24 * (a.abs() + 3 * b_abs + (0 if r is None else r.double().abs()))
        tol = U * (want.abs() + fp32) + fp32
        got = Fn.rmsnorm_bwd(x, dy, w, 1e-5, dres=r)
        assert bool(((got.double() - want).abs() <= tol).all())
    assert _lib.read_status() == 0


@pytest.mark.parametrize("T,d", [(1, 4096), (255, 256), (256, 1032), (2369, 4096), (600, 8192)])
def test_embedding_rows(T, d):
    from easy_to_hard_b200.ops import _lib, functional as Fn
    emb, w = _data(301, d, 1)
    tok = torch.randint(0, 301, (T,), device="cuda", dtype=torch.int32)
    h, x = (torch.empty(T, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    Fn.fused_residual_rmsnorm(None, w, 1e-5, tokens=tok, emb=emb, h_out=h, x_out=x)
    assert torch.equal(h, emb[tok.long()])
    _check_forward(x, h, w, 1e-5)
    assert _lib.read_status() == 0
    tok[T // 2], tok[-1] = 301, -1                      # outside the table: zero rows, reported
    Fn.fused_residual_rmsnorm(None, w, 1e-5, tokens=tok, emb=emb, h_out=h, x_out=x)
    for t in (T // 2, T - 1):
        assert not h[t].any() and not x[t].any()
    assert _lib.read_status() == 106


@pytest.mark.parametrize("T", [1, 255, 257, 2369, 5015])
@pytest.mark.parametrize("d", [256, 1032, 4096, 8192])
def test_in_place(T, d):
    """The result over one of its inputs: each block loads its next row before it stores this one, and no
    row is another block's."""
    from easy_to_hard_b200.ops import _lib, functional as Fn
    x, dy, res, w = _data(T, d, 3)
    p = lambda t: t.data_ptr()

    def bwd(a, b, r, out):
        _lib.check(_lib.lib().e2h_rmsnorm_bwd(p(a), p(b), p(w), p(r), p(out), T, d, 1e-5, _lib.stream()), "bwd")
        return out
    want = bwd(x, dy, res, torch.empty_like(x))
    for k in range(3):
        args = [x.clone(), dy.clone(), res.clone()]
        assert torch.equal(bwd(*args, args[k]), want)
    want = Fn.rmsnorm(x, w, 1e-5)
    y = x.clone()
    _lib.check(_lib.lib().e2h_rmsnorm_fwd(p(y), None, None, 0, None, 0, p(w), None, p(y), None, T, d, 1e-5,
                                          None, None, None, _lib.status_word(x.device).data_ptr(),
                                          _lib.stream()), "fwd")
    assert torch.equal(y, want)
    assert _lib.read_status() == 0
