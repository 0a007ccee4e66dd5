"""The residual stream's norm over many rows (rows in registers): widths around the vectors of a warp and of a
block, rows around the blocks, bad ids, picked rows."""
import pytest
import torch

from easy_to_hard_b200.ops import _lib, hybrid as hy

pytestmark = pytest.mark.gpu

U = {torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}


def _want(row, weight, offset, eps):
    rstd = 1.0 / torch.sqrt((row * row).mean(-1, keepdim=True) + eps)
    return row * rstd * (offset + weight.double())


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("W", [4, 508, 512, 516, 1024, 1028, 2044, 2048, 2052, 4096, 4100, 8192])
@pytest.mark.parametrize("n", [1024, 1027])
def test_many_rows(n, W, dt):
    g = torch.Generator(device="cuda").manual_seed(W + n)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    weight, eps, top = rnd(W), 1e-5, 2
    # W values summed in 32 bits, a division and a square root; then one rounding of the result
    rel = U[dt] + (W + 16) * 2.0 ** -24

    # start of the stream: embeddings
    emb, tok = rnd(50, W).to(dt), torch.randint(0, 50, (n,), device="cuda", generator=g).int()
    x, out = torch.empty(n, W, device="cuda"), torch.empty(n, W, device="cuda", dtype=dt)
    pos, pad = torch.empty(n, device="cuda").int(), torch.arange(n, device="cuda").int()
    hy.stream_norm(x, weight, out, eps=eps, offset=1.0, tokens=tok, emb=emb, emb_scale=3.0,
                   col=torch.tensor([100], device="cuda").int(), left_pad=pad, pos_out=pos)
    assert torch.equal(x, emb[tok.long()].float() * 3.0)
    assert torch.equal(pos, (100 - pad).clamp(min=0))
    want = _want(x.double(), weight, 1.0, eps)
    assert ((out.double() - want).abs() <= rel * want.abs() + 1e-30).all()

    # expert outputs come in
    y = rnd(n * top, W).to(dt)
    place = torch.randperm(n * top, device="cuda", generator=g).int().view(n, top)
    ew = rnd(n, top).abs()
    new = torch.empty_like(x).copy_(x)
    hy.stream_norm(new, weight, out, eps=eps, experts=(y, place, ew))
    terms = y[place.long()].double() * ew.double()[..., None]
    row = x.double() + terms.sum(1)
    slack = 4 * 2.0 ** -24 * (x.double().abs() + terms.abs().sum(1))
    assert ((new.double() - row).abs() <= slack).all()
    want = _want(new.double(), weight, 0.0, eps)
    assert ((out.double() - want).abs() <= rel * want.abs() + 1e-30).all()

    # picked rows leave the stream alone
    rows = torch.randint(0, n, (n,), device="cuda", generator=g).int()
    keep = new.clone()
    hy.stream_norm(new, weight, out, eps=eps, rows=rows)
    want = _want(keep[rows.long()].double(), weight, 0.0, eps)
    assert torch.equal(new, keep)
    assert ((out.double() - want).abs() <= rel * want.abs() + 1e-30).all()


def test_bad_ids_are_reported():
    n, W = 1030, 128
    status = _lib.status_word(torch.device("cuda", torch.cuda.current_device()))
    emb, weight = torch.randn(8, W, device="cuda").bfloat16(), torch.ones(W, device="cuda")
    x, out = torch.empty(n, W, device="cuda"), torch.empty(n, W, device="cuda").bfloat16()
    for bad in (-1, 8):
        tok = torch.zeros(n, device="cuda", dtype=torch.int32)
        tok[1028] = bad
        status.zero_()
        hy.stream_norm(x, weight, out, eps=1e-5, tokens=tok, emb=emb)
        assert int(status) != 0 and torch.equal(x[1028], emb[0].float())
        rows = torch.zeros(n, device="cuda", dtype=torch.int32)
        rows[1027] = n if bad > 0 else -1
        status.zero_()
        hy.stream_norm(x, weight, out, eps=1e-5, rows=rows)
        assert int(status) != 0 and torch.equal(out[1027], out[0])
    status.zero_()
