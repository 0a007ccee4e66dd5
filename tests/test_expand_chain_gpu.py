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


@pytest.mark.parametrize("bits", [8, 4])
def test_a_captured_step_keeps_its_image(bits):
    """A larger matrix is expanded after the capture, and memory that comes free is taken and filled:
    the step still gives its product, and writes into nothing else."""
    from easy_to_hard_b200.ops import _lib, gemm
    T, K = 160, 1024
    w, s, wf = _weight(512, K, bits, 1)
    x = torch.randn(T, K, device="cuda").bfloat16()
    out = torch.empty(T, 512, device="cuda", dtype=torch.bfloat16)
    g = _captured(lambda: gemm.linear(x, w, out=out, scale=s))
    big, sb, bf = _weight(9000, K, bits, 2)
    got = gemm.linear(x, big, scale=sb)
    _close(got, x.double() @ bf.double().t(), x, bf)
    torch.cuda.synchronize()
    taken = [torch.full((n * K,), 7.0, device="cuda", dtype=torch.bfloat16)
             for n in (512, 512, 512, 9000)]
    x.copy_(torch.randn(T, K, device="cuda"))
    g.replay()
    torch.cuda.synchronize()
    _close(out, x.double() @ wf.double().t(), x, wf)
    assert all(bool((t == 7.0).all()) for t in taken)
    assert _lib.read_status() == 0


def test_two_streams_expand_at_once():
    from easy_to_hard_b200.ops import _lib, gemm
    T, K = 160, 2048
    ws = [_weight(8192, K, 8, n) for n in (3, 4)]
    x = torch.randn(T, K, device="cuda").bfloat16()
    want = [x.double() @ wf.double().t() for _, _, wf in ws]
    streams = [torch.cuda.Stream() for _ in ws]
    outs = [torch.empty(20, T, 8192, device="cuda", dtype=torch.bfloat16) for _ in ws]
    torch.cuda.synchronize()
    for i in range(20):
        for (w, s, _), st, out in zip(ws, streams, outs):
            with torch.cuda.stream(st):
                gemm.linear(x, w, out=out[i], scale=s)
    torch.cuda.synchronize()
    for (_, _, wf), out, ref in zip(ws, outs, want):
        for i in range(20):
            _close(out[i], ref, x, wf)
    assert _lib.read_status() == 0


@pytest.mark.parametrize("T", [4, 64, 200])
def test_strided_pairs(T):
    from easy_to_hard_b200.ops import _lib, gemm
    F, K, group = 96, 512, 64
    dense, _, wf = _weight(F, K, 4, 5)
    sz = torch.rand(K // group, F, 4, device="cuda").bfloat16()[..., ::2]
    w = gemm.Int4Weight(dense.q, sz, group, (F, K))
    wf = w.dequant().float()
    assert torch.equal(gemm._expand_int4(w, 0), w.dequant())
    x = torch.randn(T, K, device="cuda").bfloat16()
    got = gemm.linear(x, w)
    torch.cuda.synchronize()
    _close(got, x.double() @ wf.double().t(), x, wf)
    assert _lib.read_status() == 0
