"""Quantised products whose converters take turns: numbers of stages around the line between one group and two,
odd and even, fewer stages than buffers, K split or not, gated; every int8 code."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weight(F, K, bits, g):
    from easy_to_hard_b200.ops.gemm import Int4Weight
    if bits == 8:
        w = torch.randint(-128, 128, (F, K), device="cuda", generator=g, dtype=torch.int8)
        return w, (torch.rand(F, device="cuda", generator=g) + 0.5), w.double()
    codes = torch.randint(0, 16, (F, K), device="cuda", generator=g, dtype=torch.int32)
    sz = (torch.rand(K // 128, F, 2, device="cuda", generator=g) * 0.1).bfloat16()
    w = Int4Weight.from_int(codes, sz, 128)
    return w, None, w.dequant().double()


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("T", [17, 64, 65, 128])
@pytest.mark.parametrize("F,stages", [(12000, 1), (12000, 7), (12000, 8), (12000, 9), (12000, 33), (2048, 31),
                                      (2048, 32), (2048, 36), (300, 8), (300, 64)])
def test_stages(bits, T, F, stages):
    from easy_to_hard_b200.ops import _lib, gemm
    K = 128 * stages
    g = torch.Generator(device="cuda").manual_seed(F + K + T)
    w, s, wf = _weight(F, K, bits, g)
    if s is not None:
        wf = wf * s.double()[:, None]
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    out = torch.empty(T, F, device="cuda")
    for _ in range(2):
        gemm.linear(x, w, out=out, scale=s)
        want = x.double() @ wf.t()
        tol = (K + 2) * 2.0 ** -23 * (x.double().abs() @ wf.abs().t()) + 1e-30   # fp32 sums of K products
        assert bool(((out.double() - want).abs() <= tol).all())
    assert _lib.read_status() == 0


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("T", [40, 100])
@pytest.mark.parametrize("F,stages", [(11008, 7), (11008, 8), (11008, 32), (1376, 9)])
def test_gated(bits, T, F, stages):
    from easy_to_hard_b200.ops import _lib, gemm
    K = 128 * stages
    g = torch.Generator(device="cuda").manual_seed(F + K + T)
    (w1, s1, f1), (w3, s3, f3) = (_weight(F, K, bits, g) for _ in range(2))
    x = (torch.randn(T, K, device="cuda", generator=g) / (30 * K ** 0.5 if bits == 8 else K ** 0.5)).bfloat16()
    sc = None
    if bits == 8:
        sc = torch.cat([s1, s3])
        f1, f3 = f1 * s1.double()[:, None], f3 * s3.double()[:, None]
    got = gemm.linear_swiglu(x, w1, w3, scale=sc).double()
    a, b = x.double() @ f1.t(), x.double() @ f3.t()
    want = torch.nn.functional.silu(a) * b
    # silu(bf16(a)), bf16(b) and their product rounded to bf16: four relative errors of 2^-8, silu's slope
    # against its value (1.1 |a| at most), and the fp32 sums
    u = 2.0 ** -8
    ta, tb = (K * 2.0 ** -23 * (x.double().abs() @ f.abs().t()) for f in (f1, f3))
    tol = 1.1 * b.abs() * (ta + u * a.abs()) + 1.1 * a.abs() * (tb + u * b.abs()) + 3 * u * want.abs() + 1e-6
    assert bool(((got - want).abs() <= 1.05 * tol).all())
    assert _lib.read_status() == 0


def test_every_code():
    from easy_to_hard_b200.ops import gemm
    w = torch.arange(-128, 128, device="cuda", dtype=torch.int32).to(torch.int8)
    w = w.repeat(256, 8)                                   # [256, 2048]
    out = torch.empty(64, 256, device="cuda")
    for first in range(0, 2048, 64):                       # one-hot rows read the codes back
        x = torch.zeros(64, 2048, device="cuda", dtype=torch.bfloat16)
        x[torch.arange(64), first + torch.arange(64)] = 1
        gemm.linear(x, w, out=out, scale=torch.ones(256, device="cuda"))
        assert torch.equal(out, w[0, first:first + 64].float()[:, None].expand(64, 256))


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("dual,T", [(False, 40), (False, 100), (True, 64)])
@pytest.mark.parametrize("ring", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("trips", [8, 19])
def test_rings(bits, dual, T, ring, trips):
    """Rings of so many stages (all of them fit): odd ones, and ones with fewer stages than converted-tile
    buffers. A stage converted before its load has landed gives what an earlier trip held."""
    from easy_to_hard_b200.ops import _lib, gemm
    F, K = 9600, 128 * trips
    g = torch.Generator(device="cuda").manual_seed(K + T)
    ws = [_weight(F, K, bits, g) for _ in range(1 + dual)]
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    scale = torch.cat([s for _, s, _ in ws]) if bits == 8 else None
    wf = [f if s is None else f * s.double()[:, None] for _, s, f in ws]
    outs = [torch.empty(T, F, device="cuda", dtype=torch.bfloat16 if dual else torch.float32) for _ in ws]
    for _ in range(4):
        if dual:
            gemm.gemm(ws[0][0], x, epi=gemm.EPI_DUAL_STORE, a2=ws[1][0], out=outs[0], out2=outs[1], scale=scale,
                      stages=ring)
        else:
            gemm.gemm(ws[0][0], x, epi=gemm.EPI_STORE_F32, out=outs[0], scale=scale, stages=ring)
        for out, f in zip(outs, wf):
            want = x.double() @ f.t()
            tol = (K + 2) * 2.0 ** -23 * (x.double().abs() @ f.abs().t()) + 2.0 ** -8 * dual * want.abs()
            assert bool(((out.double() - want).abs() <= 1.01 * tol + 1e-30).all())
    assert _lib.read_status() == 0


@pytest.mark.parametrize("F,K,T,bits", [(12288, 4096, 128, 8), (15360, 5120, 80, 8), (12288, 4096, 128, 4),
                                        (2752, 4096, 64, 8), (2752, 8192, 64, 8)])
def test_odd_rings_as_dispatched(F, K, T, bits):
    """Shapes whose own ring has an odd number of stages (tests/test_gemm_w8_ring_cpu.py): 5 beside 4 buffers,
    and gated with K in four (2752 features) 3 beside 3."""
    from easy_to_hard_b200.ops import _lib, gemm
    dual = F == 2752
    g = torch.Generator(device="cuda").manual_seed(F + K)
    ws = [_weight(F, K, bits, g) for _ in range(1 + dual)]
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    scale = torch.cat([s for _, s, _ in ws]) if bits == 8 else None
    outs = [torch.empty(T, F, device="cuda", dtype=torch.bfloat16 if dual else torch.float32) for _ in ws]
    for _ in range(8):
        if dual:
            gemm.gemm(ws[0][0], x, epi=gemm.EPI_DUAL_STORE, a2=ws[1][0], out=outs[0], out2=outs[1], scale=scale)
        else:
            gemm.linear(x, ws[0][0], out=outs[0], scale=scale)
        for out, (_, s, f) in zip(outs, ws):
            f = f if s is None else f * s.double()[:, None]
            want = x.double() @ f.t()
            tol = (K + 2) * 2.0 ** -23 * (x.double().abs() @ f.abs().t()) + 2.0 ** -8 * dual * want.abs()
            assert bool(((out.double() - want).abs() <= 1.01 * tol + 1e-30).all())
    assert _lib.read_status() == 0
