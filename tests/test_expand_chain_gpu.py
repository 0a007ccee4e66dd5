"""Products over weights that the call itself expands to bf16, in a captured chain with programmatic
launches: the product may start before the expansion has finished, but must not read its result."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weight(F, K, bits, seed):
    """(operand, per-feature scale or None, the matrix it stands for, in fp32)"""
    from easy_to_hard_b200.ops.gemm import Int4Weight
    g = torch.Generator(device="cuda").manual_seed(seed)
    if bits == 8:
        w = torch.randint(-128, 128, (F, K), device="cuda", generator=g, dtype=torch.int8)
        s = torch.rand(F, device="cuda", generator=g) * 0.01 + 0.001
        return w, s, w.float() * s[:, None]
    group = 16 if K % 32 else 32
    codes = torch.randint(0, 16, (F, K), device="cuda", generator=g, dtype=torch.int32)
    sz = (torch.rand(K // group, F, 2, device="cuda", generator=g) * 0.1).bfloat16()
    w = Int4Weight.from_int(codes, sz, group)
    return w, None, w.dequant().float()


def _captured(step):
    """A graph of ``step`` with programmatic launches, as a decode step is captured."""
    from easy_to_hard_b200.ops import _lib
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        step()
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    old = _lib.lib().e2h_set_pdl(1)
    try:
        with torch.cuda.graph(g):
            step()
    finally:
        _lib.lib().e2h_set_pdl(old)
    return g


def _close(got, want, x, wf):
    """fp32 sums of K products: K 2^-23 sum |x w|; one rounding to bf16."""
    tol = x.shape[1] * 2.0 ** -23 * (x.float().abs() @ wf.abs().t()) + 2.0 ** -8 * want.abs()
    assert bool(((got.double() - want).abs() <= tol + 1e-30).all())


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("T,K", [(17, 688), (64, 688), (17, 1376), (64, 1376), (200, 1024)])
def test_products_alternate_through_the_expansion(bits, T, K):
    from easy_to_hard_b200.ops import _lib, gemm
    ws = [_weight(F, K, bits, 7 + F) for F in (4096, 1000, 4096)]
    x = torch.randn(T, K, device="cuda").bfloat16()
    outs = [torch.empty(T, w.shape[0], device="cuda", dtype=torch.bfloat16) for w, _, _ in ws]

    def step():
        for (w, s, _), out in zip(ws, outs):
            gemm.linear(x, w, out=out, scale=s)
    g = _captured(step)
    for _ in range(3):
        for out in outs:
            out.fill_(float("nan"))
        x.copy_(torch.randn(T, K, device="cuda"))
        g.replay()
        torch.cuda.synchronize()
        for (_, _, wf), out in zip(ws, outs):
            _close(out, x.double() @ wf.double().t(), x, wf)
    assert _lib.read_status() == 0
