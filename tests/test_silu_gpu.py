"""SiLU of every bf16 number against 64 bits: the fast division has to hold where its divisor leaves the
range that the instruction divides by, and for infinities, NaN and the two zeros."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [0, 1])
def test_silu_all_inputs(sign):
    from easy_to_hard_b200.ops import functional as F
    bits = (torch.arange(32768, dtype=torch.int32) + 32768 * sign).to(torch.int16)
    g = bits.view(torch.bfloat16).cuda()
    got = F.swiglu(g, torch.ones_like(g)).cpu().double()
    x = bits.view(torch.bfloat16).double()
    e = torch.exp(-x)
    want = x / (1 + e)
    nan = torch.isnan(x) | (x == -float("inf"))
    assert torch.isnan(got)[nan].all() and not torch.isnan(got)[~nan].any()
    # exp(-x) is infinite in 32 bits below -88.73: zero there, and within the bound everywhere else
    gone = (x < -88.73) & ~nan
    assert (got[gone] == 0).all()
    rest = ~nan & ~gone
    assert torch.equal(got[rest & torch.isinf(x)], x[rest & torch.isinf(x)])
    rest &= ~torch.isinf(x)
    # one rounding to bf16 (2^-8), the exponential (2 + 1.173 |x| units of 2^-23, as documented), the sum,
    # the division (2 units) and the scale; tiny results also lose what lies below the smallest bf16
    rel = 2.0 ** -8 + (2 + 1.173 * x.abs().clamp(max=128) + 4) * 2.0 ** -23
    err = (got - want).abs()
    assert (err[rest] <= (rel * want.abs() * (1 + 2.0 ** -8) + 2.0 ** -133)[rest]).all()
    assert torch.equal(torch.signbit(got[rest]), torch.signbit(x[rest]))
