"""The 16-byte forms of the optimizer, cast and cross-entropy kernels and the forms for rows that do not
start on a 16-byte boundary, at the edges of both."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _adam64(p, g, m, v, kw):
    """The step in 64 bits with the kernel's roundings: to the type of the state after every operation on
    it, to the type of the parameter where that is used. Returns (p, m, v, the step taken by p)."""
    tp, ts = p.dtype, m.dtype
    p, g, m, v = (t.double() for t in (p, g, m, v))

    def rp(t):
        return t.to(tp).double() if tp == torch.bfloat16 else t

    def rs(t):
        return t.to(ts).double() if ts == torch.bfloat16 else t
    p = rp(p * (1 - kw["lr"] * kw["weight_decay"]))
    g = rs(g)
    m = rs(rs(kw["beta1"] * m) + (1 - kw["beta1"]) * g)
    v = rs(rs(kw["beta2"] * v) + (1 - kw["beta2"]) * g * g)
    b1, b2 = 1 - kw["beta1"] ** kw["step"], 1 - kw["beta2"] ** kw["step"]
    step = kw["lr"] / b1 * rp(m) / rp(rs(rs(v.sqrt() / b2 ** 0.5) + kw["eps"]))
    return p - step, m, v, step


@pytest.mark.parametrize("n", [1, 4, 1027, 500003])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dts", [("f", "f", "f"), ("f", "b", "f"), ("b", "f", "b"), ("b", "b", "b")])
def test_adamw(n, offset, dts):
    """Element by element. fp32: a dozen roundings of 2^-24. bf16: the same roundings as the reference's, of
    which fp32 arithmetic may turn one over at each (2^-8 of the value; in the step three of them and
    their quotient). The step and the decay are a hundred times the bounds."""
    from easy_to_hard_b200.utils.memory_efficient_adam import fused_adamw_
    dt = {"f": torch.float32, "b": torch.bfloat16}
    g0 = torch.Generator(device="cuda").manual_seed(n)

    def mk(kind, scale, positive=False):
        t = torch.randn(n + offset, device="cuda", generator=g0) * scale
        return (t.abs() + 1e-2 * scale if positive else t).to(dt[kind])[offset:]
    p, g, m, v = mk(dts[0], 1.0), mk(dts[1], 1.0), mk(dts[2], 0.1), mk(dts[2], 0.1, True)
    kw = dict(lr=0.5, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.2, step=3)
    wp, wm, wv, step = _adam64(p, g, m, v, kw)
    copy = torch.zeros(n + offset, device="cuda", dtype=torch.bfloat16)[offset:]
    fused_adamw_(p, g, m, v, bf16_copy=copy, **kw)
    torch.cuda.synchronize()
    one = 2.0 ** -20 if dts[0] == dts[2] == "f" else 2.0 ** -7
    terms = 0.1 * g.double().abs() + wm.abs()        # what the sum of the first moment is made of
    assert bool(((m.double() - wm).abs() <= 2 * one * terms).all())
    assert bool(((v.double() - wv).abs() <= 2 * one * wv).all())
    tol = one * (wp.abs() + step.abs() + p.double().abs()) + 4 * one * step.abs()
    tol = tol + 2 * one * step.abs() / wm.abs().clamp_min(1e-30) * terms
    assert bool(((p.double() - wp).abs() <= tol).all())
    assert torch.equal(copy, p.to(torch.bfloat16))


@pytest.mark.parametrize("n,offset", [(1, 0), (7, 4), (4099, 0), (1 << 20, 8), (33, 1)])
def test_widening_is_exact(n, offset):
    from easy_to_hard_b200.parallel.fsdp import _as_dtype
    x = torch.randn(n + offset, device="cuda").bfloat16()[offset:]
    assert torch.equal(_as_dtype(x, torch.float32), x.float())


@pytest.mark.parametrize("vocab,pad", [(1, 3), (5, 0), (1000, 8), (8200, 1), (32016, 0)])
def test_cross_entropy_rows(vocab, pad):
    """fp32 sums of ``vocab`` terms and a few exponentials of 2 ulp: 1e-5; bf16 gradients: 2^-8."""
    from easy_to_hard_b200.ops import loss
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = (torch.randn(6, vocab + pad, device="cuda", generator=g) * 5)[:, :vocab]
    x[1] = -80.0
    x[2, vocab // 2] = 60.0
    t = torch.randint(0, vocab, (6,), device="cuda", generator=g)
    z = x.double() / 0.7
    lse = torch.logsumexp(z, -1)
    p = torch.exp(z - lse[:, None])
    st = loss.ce_stats(x, t, 0.7)
    L, tgt, H = loss._combine_stats(st, None, 1)
    assert float((L - lse).abs().max()) < 1e-5 * float(lse.abs().max().clamp_min(1))
    assert float((tgt - z.gather(1, t[:, None])[:, 0]).abs().max()) < 1e-4
    ent = lse - (p * z).sum(-1)
    assert float((H - ent).abs().max()) < 1e-4 * float(lse.abs().max().clamp_min(1))
    glp, gen = torch.randn(6, device="cuda"), torch.randn(6, device="cuda")
    for ge in (None, gen):
        d = loss.ce_grad(x, t, L, H, glp, ge, 0.7)
        hot = torch.nn.functional.one_hot(t, vocab).double()
        want = glp.double()[:, None] * (hot - p)
        if ge is not None:
            want = want - ge.double()[:, None] * p * (z - lse[:, None] + ent[:, None])
        want = want / 0.7
        assert float((d.double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) + 1e-4


@pytest.mark.parametrize("vocab,pad", [(5, 0), (1000, 8), (4096, 0), (8200, 1), (32016, 0)])
def test_cross_entropy_of_masked_rows(vocab, pad):
    """Entries at the lowest finite value add nothing, wherever they lie and however many threads meet
    nothing else; a NaN or an infinite entry still shows. Bounds as above."""
    from easy_to_hard_b200.ops import loss
    low = torch.finfo(torch.float32).min
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = (torch.randn(7, vocab + pad, device="cuda", generator=g) * 5)[:, :vocab]
    drop = torch.rand(7, vocab, device="cuda", generator=g)
    x[0, drop[0] < 0.75] = low
    x[1, : vocab - 1] = low
    x[2, 1:] = low
    x[3, ::2] = low
    x[4, : vocab // 2] = low
    x[5] = low
    x[5, vocab // 3] = -1e30
    x[:, vocab // 2] = torch.where(x[:, vocab // 2] == low, x[:, vocab // 2], 3.0)
    t = torch.full((7,), vocab // 2, device="cuda")
    z = x.double()
    lse = torch.logsumexp(z, -1)
    p = torch.exp(z - lse[:, None])
    L, tgt, H = loss._combine_stats(loss.ce_stats(x, t), None, 1)
    scale = lse.abs().clamp_min(1)
    assert float(((L - lse).abs() / scale).max()) < 1e-5
    ent = -(p * torch.where(p > 0, z - lse[:, None], 0.0)).sum(-1)
    assert float(((H - ent).abs() / scale).max()) < 1e-4
    d = loss.ce_grad(x, t, L, H, torch.ones(7, device="cuda"), torch.ones(7, device="cuda"))
    assert bool(torch.isfinite(d).all())
    for bad in (float("nan"), float("inf")):
        y = x.clone()
        y[:, 0], y[:, -1] = bad, 500.0
        L, _, H = loss._combine_stats(loss.ce_stats(y, t), None, 1)
        assert bool(torch.isnan(L).all()) and bool(torch.isnan(H).all())
