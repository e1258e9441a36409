"""Conversions of many tensors by one launch (checkpoints, fp32 export and import): the same bits
as the oracle and torch's own conversions, nothing written outside a tensor."""

import pytest
import torch
import torch.nn as nn

from flashoptim_b200 import FlashAdamW
from flashoptim_b200.ops import oracle
from flashoptim_b200.ops.quant import Conversions

pytestmark = pytest.mark.gpu

# more rows than one launch takes; sizes around a quad, a tile and a chunk, a large one in between
SIZES = [1, 3, 4, 5, 255, 257, 4095, 4096, 4097, 1_000_003] * 7


def _views(buf, skew):
    """Back to back and unaligned, or each at a multiple of 32 elements with a gap behind it."""
    out, at = [], skew
    for n in SIZES:
        out.append(buf[at:at + n])
        at += n if skew else -(-(n + 1) // 32) * 32
    return out


def _buffer(fill, dtype):
    return torch.full((sum(SIZES) + 64 * len(SIZES),), fill, dtype=dtype, device="cuda")


@pytest.mark.parametrize("skew", [0, 1])
@pytest.mark.parametrize("signed,sqrt,softsign", [(True, False, True), (False, True, False)])
def test_moments_as_bf16(skew, signed, sqrt, softsign):
    codes = _views(torch.randint(0, 256, _buffer(0, torch.uint8).shape, device="cuda").to(torch.uint8), skew)
    codes = [c.view(torch.int8) if signed else c for c in codes]
    scales = [torch.rand((n + 31) // 32, device="cuda").half() for n in SIZES]
    conv = Conversions()
    got = [conv.dequantize_bf16(c, s, signed, sqrt, softsign) for c, s in zip(codes, scales)]
    conv.launch()
    for c, s, out in zip(codes, scales, got):
        ref = oracle.dequantize_ref(c.cpu(), s.cpu(), signed=signed, sqrt=sqrt, softsign=softsign)
        assert torch.equal(out.cpu(), ref.to(torch.bfloat16))


@pytest.mark.parametrize("skew", [0, 1])
def test_quantise_lists(skew):
    values = _views(torch.randn(_buffer(0, torch.float32).shape, device="cuda").bfloat16(), skew)
    conv = Conversions()
    got = [conv.quantize(x, True, False, True) for x in values]
    conv.launch()
    for x, (q, s) in zip(values, got):
        q_ref, s_ref = oracle.quantize_ref(x.cpu())
        assert torch.equal(q.cpu(), q_ref) and torch.equal(s.cpu(), s_ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_codes_in_the_parameters_dtype_convert_as_torch_does(dtype):
    every = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).cuda().view(dtype)  # NaN and infinities too
    codes = torch.arange(-128, 128, dtype=torch.int32).to(torch.int8).cuda()
    conv = Conversions()
    pairs = [(t, d, conv.codes_as(t, d)) for skew in (0, 1, 3)
             for t, d in ((every[skew:], torch.int8), (codes[skew:], dtype))]
    conv.launch()
    for t, d, got in pairs:
        assert got.dtype == d and torch.equal(got, t.to(d))


@pytest.mark.parametrize("skew", [0, 1])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("code_dtype", [torch.int8, torch.int16])
def test_split_and_merge_of_lists(skew, dtype, code_dtype):
    x = torch.randn(_buffer(0, torch.float32).shape, device="cuda") * 0.05
    x[::7] *= 1e-30 if dtype == torch.bfloat16 else 1e-6
    x[::11] = 0
    values = _views(x, skew)
    buf, want = _buffer(-7.0, dtype), _buffer(-7.0, dtype)
    params = _views(buf, skew)
    conv = Conversions()
    codes = [conv.split(v, p, torch.empty(p.shape, dtype=code_dtype, device="cuda")) for v, p in zip(values, params)]
    conv.launch()
    masters = [conv.reconstruct_fp32_param(p, c) for p, c in zip(params, codes)]
    conv.launch()
    for v, c, m, w in zip(values, codes, masters, _views(want, skew)):
        w.copy_(v.to(dtype))
        ref = oracle.ecc_encode_ref(v.cpu(), w.cpu(), 1 if code_dtype == torch.int8 else 2)
        assert torch.equal(c.cpu(), ref)
        assert torch.equal(m.cpu(), oracle.ecc_decode_ref(w.cpu(), ref))
    assert torch.equal(buf, want)  # the parameters, and nothing between them


def test_what_the_list_kernels_do_not_serve_is_converted_all_the_same():
    """Strided parameters, values of another layout, a dtype without list kernel, and an error on
    the way (what came before it has been set)."""
    class Net(nn.Module):
        def __init__(self):
            super().__init__()
            self.a = nn.Parameter(torch.randn(33, 65, device="cuda").bfloat16())
            self.b = nn.Parameter(torch.randn(65, 33, device="cuda").bfloat16().t())
            self.c = nn.Parameter(torch.randn(17, device="cuda"))

    net = Net()
    opt = FlashAdamW(net.parameters(), lr=1e-3, fused=False)
    for p in net.parameters():
        p.grad = torch.randn_like(p) * 1e-2
    opt.step()
    values = {k: torch.randn(v.shape[::-1], device="cuda").t() if v.dim() == 2 else torch.randn(17, device="cuda")
              for k, v in net.named_parameters()}
    opt.set_fp32_model_state_dict(net, values)
    out = opt.get_fp32_model_state_dict(net)
    assert list(out) == list(net.state_dict())
    for k, p in net.named_parameters():
        assert torch.equal(p.detach(), values[k].to(p.dtype))
        want = values[k]
        if "error_bits" in opt.state[p]:
            want = oracle.ecc_decode_ref(p.detach(), oracle.ecc_encode_ref(values[k], p.detach(), 1))
        assert torch.equal(out[k], want)
    bad = dict(values, a=torch.ones(33, 65, device="cuda"), b=torch.ones(33, 65, device="cuda").half())
    with pytest.raises(ValueError, match="Expected fp32"):
        opt.set_fp32_model_state_dict(net, bad)
    assert (net.a == 1).all() and (opt.state[net.a]["error_bits"] == 0).all()


def test_import_from_host_memory_holds_few_copies_on_the_device():
    """24 fp32 tensors of 16 MB: 384 MB if every device copy waited for one launch at the end."""
    net = nn.ParameterList([nn.Parameter(torch.zeros(1 << 22, device="cuda", dtype=torch.bfloat16)) for _ in range(24)])
    opt = FlashAdamW(net.parameters(), lr=1e-3)
    for p in net:
        p.grad = torch.zeros_like(p)
    opt.step()
    opt.zero_grad()
    values = {k: torch.full((1 << 22,), 1.0 + i) for i, k in enumerate(net.state_dict())}
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    opt.set_fp32_model_state_dict(net, values)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - base < 24 * (4 << 20) + 96 * (1 << 20)  # new codes, and the copies in hand
    assert all((p == 1.0 + i).all() for i, p in enumerate(net))


def _trained(count, numel):
    net = nn.ParameterList([nn.Parameter(torch.full((numel,), 1.0, device="cuda").bfloat16()) for _ in range(count)])
    opt = FlashAdamW(net.parameters(), lr=1e-3)
    for p in net:
        p.grad = torch.full_like(p, 1e-3)
    opt.step()
    opt.zero_grad()
    return net, opt


def _peak(fn):
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    fn()
    torch.cuda.synchronize()
    return torch.cuda.max_memory_allocated() - base


@pytest.mark.parametrize("what", ["checkpoint", "fp32 weights"])
def test_host_memory_is_taken_in_with_few_copies_more_than_a_loop_holds(what, monkeypatch):
    """192 MB of moments, or 384 MB of fp32 weights, in host memory: beyond what a loop over tensors
    (a limit of nothing) holds, the limit and the tensors of the parameter in hand."""
    net, opt = _trained(24, 1 << 22)
    saved = opt.state_dict()
    saved["state"] = {k: {n: v.cpu() for n, v in st.items()} for k, st in saved["state"].items()}
    values = {k: torch.full((1 << 22,), 1.0 + i) for i, k in enumerate(net.state_dict())}

    def run():
        if what == "checkpoint":
            opt.load_state_dict(saved)
        else:
            opt.set_fp32_model_state_dict(net, values)

    run()
    peak = _peak(run)
    monkeypatch.setattr(Conversions, "HELD", 0)
    assert peak - _peak(run) <= (32 << 20) + 3 * (16 << 20)


def test_inputs_that_live_anyway_do_not_cut_a_list(monkeypatch):
    monkeypatch.setattr(Conversions, "HELD", 1)
    x = torch.randn(100, 64, device="cuda")
    conv = Conversions()
    codes, scales = conv.quantize(x, True, False, True)
    conv.dequantize_bf16(codes, scales, True, False, True)
    param = x.bfloat16()
    error_bits = torch.empty(x.shape, dtype=torch.int8, device="cuda")
    conv.split(x, param, error_bits)
    conv.reconstruct_fp32_param(param, error_bits)
    conv.codes_as(error_bits, torch.bfloat16)
    assert len(conv._lists) == 5
    codes, scales = conv.quantize(x.t(), True, False, True)  # of another layout: a copy, launched with the rest
    assert not conv._lists
    q_ref, s_ref = oracle.quantize_ref(x.t().cpu())
    torch.cuda.synchronize()
    assert torch.equal(codes.cpu(), q_ref) and torch.equal(scales.cpu(), s_ref)
