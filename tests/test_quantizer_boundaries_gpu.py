"""The quantiser's fast path decides most codes and hands the rest to the written-down formula;
the dequantiser divides through corrected reciprocals.  Both against the oracle, bit for bit, on
inputs that lie on and next to the rounding boundaries, on extreme groups and for every code."""

import pytest
import torch

from flashoptim_b200.ops import oracle
from flashoptim_b200.ops.quant import dequantize, quantize

pytestmark = pytest.mark.gpu

RECIPES = [(a, b, c) for a in (True, False) for b in (True, False) for c in (True, False)]


def _boundary_groups(signed, sqrt, softsign):
    """Groups of absmax a (element 0) whose other 31 elements sit within a few ulps of the input at
    which the code steps from q to q + 1."""
    qmax = 127 if signed else 255
    g = torch.Generator().manual_seed(5)
    a = torch.exp(torch.empty(64).uniform_(-20, 5, generator=g))[:, None]
    t = (torch.arange(0, qmax).float() + 0.5) / qmax
    n = t / (2.0 - t) if softsign else t  # inverse of 2n / (1 + n)
    x = a * n[None, :]
    x = torch.cat([x + k * x * 2.0**-24 for k in range(-6, 7)], dim=1)
    if signed and not sqrt:
        x = torch.where(torch.rand(x.shape, generator=g) < 0.5, x, -x)
    if sqrt:
        a, x = a * a, x * x
    x = torch.cat([x, x[:, :-x.shape[1] % 31]], dim=1).reshape(a.shape[0], -1, 31)
    return torch.cat([a[:, None].expand(-1, x.shape[1], 1), x], dim=2).reshape(-1)


@pytest.mark.parametrize("signed,sqrt,softsign", RECIPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_codes_next_to_a_rounding_boundary(signed, sqrt, softsign, dtype):
    x = _boundary_groups(signed, sqrt, softsign).to(dtype)
    q, s = quantize(x.cuda(), signed=signed, sqrt=sqrt, softsign=softsign)
    q_ref, s_ref = oracle.quantize_ref(x, signed=signed, sqrt=sqrt, softsign=softsign)
    assert torch.equal(q.cpu(), q_ref) and torch.equal(s.cpu(), s_ref)


@pytest.mark.parametrize("signed,sqrt,softsign", RECIPES)
def test_extreme_group_maxima(signed, sqrt, softsign):
    """Largest, smallest, subnormal and infinite maxima (by the formula an infinity's own code is
    that of inf / inf, no number, stored as 0)."""
    tops = torch.tensor([3.4028234663852886e38, 1e30, 1.0, 1e-12, 1e-13, 1e-38, 1e-45, 0.0])
    x = (tops[:, None] * torch.linspace(0, 1, 32)[None, :]).reshape(-1)
    q, s = quantize(x.cuda(), signed=signed, sqrt=sqrt, softsign=softsign)
    q_ref, s_ref = oracle.quantize_ref(x, signed=signed, sqrt=sqrt, softsign=softsign)
    assert torch.equal(q.cpu(), q_ref) and torch.equal(s.cpu(), s_ref)
    x = torch.linspace(0, 3e38, 64)
    x[5] = float("inf")
    q, s = quantize(x.cuda(), signed=signed, sqrt=sqrt, softsign=softsign)
    assert (q[:32] == 0).all() and torch.isinf(s[0])
    q_ref, _ = oracle.quantize_ref(x[32:], signed=signed, sqrt=sqrt, softsign=softsign)
    assert torch.equal(q[32:].cpu(), q_ref)


@pytest.mark.parametrize("n", [4095, 4097, 148 * 64 * 4096 + 4097])  # one chunk, two, more than the grid
@pytest.mark.parametrize("signed,sqrt,softsign", RECIPES)
def test_every_code_dequantises_to_the_formula(n, signed, sqrt, softsign):
    q = torch.arange(n, dtype=torch.int32).mul_(37).bitwise_and_(255).to(torch.uint8)
    q = q.view(torch.int8) if signed else q
    s = torch.linspace(0, 60000, (n + 31) // 32).half()
    got = dequantize(q.cuda(), s.cuda(), signed=signed, sqrt=sqrt, softsign=softsign)
    assert torch.equal(got.cpu(), oracle.dequantize_ref(q, s, signed=signed, sqrt=sqrt, softsign=softsign))
