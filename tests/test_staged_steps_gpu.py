"""The staged step kernels against the register-path kernels (which test_kernels_gpu.py compares
with the oracle): the same expressions per element, so the same bits, whatever the layout."""

import numpy as np
import pytest
import torch

from flashoptim_b200.ops import native
from flashoptim_b200.ops.step import (
    AdamHyper, MomentumHyper, SegmentTable, launch_adam, launch_momentum, make_rows, set_step_variant,
)

pytestmark = pytest.mark.gpu

# long enough together for the staged kernels to be chosen; tails of every kind behind them
SIZES = (1, 2047, 2048, 2049, 31, 1_500_017, 4096, 65_537, 33, 500_000)
MANY = (1024,) * 700 + (2048,) * 40 + (5,) * 30 + (1_300_003,)  # segment look-up over many tensors


def _streams(sizes, dtype, err, n_states, skew, seed):
    """Every stream is one buffer; the gradients lie back to back, `skew` elements into theirs."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    starts = np.concatenate([[0], np.cumsum([-(-n // 256) * 256 for n in sizes])])
    total = int(starts[-1])

    def codes(t, lo, hi):
        return torch.randint(lo, hi, (total,), device="cuda", generator=g, dtype=t)

    p = (torch.randn(total, device="cuda", generator=g) * 0.02).to(dtype)
    grad = (torch.randn(sum(sizes) + skew, device="cuda", generator=g) * 1e-3).to(dtype)
    ecc = {0: None, 1: torch.int8, 2: torch.int16}[err]
    ecc = None if ecc is None else codes(ecc, -127, 128)
    s = [codes(torch.int8, -127, 128), codes(torch.uint8, 0, 256)][:n_states]
    sc = [torch.rand(total // 32, device="cuda", generator=g).mul_(1e-3).half() for _ in s]

    def views(buf, div=1):
        if buf is None:
            return [None] * len(sizes)
        return [buf[a // div:a // div + -(-n // div)] for a, n in zip(starts.tolist(), sizes)]

    at = np.concatenate([[0], np.cumsum(sizes)]) + skew
    grads = [grad[a:a + n] for a, n in zip(at.tolist(), sizes)]
    none = [None] * len(sizes)
    st = [(views(a), views(b, 32)) for a, b in zip(s, sc)] + [(none, none)] * (2 - n_states)
    rows = make_rows(views(p), grads, views(ecc), st[0][0], st[0][1], st[1][0], st[1][1])
    return rows, [t for t in (p, ecc, *s, *sc) if t is not None], grad


def _run(rows, dtype, err, n_states, variant):
    set_step_variant(variant)
    try:
        table = SegmentTable(torch.device("cuda", torch.cuda.current_device()))
        if n_states == 2:
            h = AdamHyper(lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=1e-5, step=7, decoupled=True)
            launch_adam(table, rows, dtype, err, True, h)
        else:
            h = MomentumHyper(lr=1e-3, mom_coef=0.9, update_coef=1.0, weight_decay=1e-5, nesterov=True, decoupled=True)
            launch_momentum(table, rows, dtype, err, native.FO_STATE_Q8, h)
        torch.cuda.synchronize()
    finally:
        set_step_variant(1)


@pytest.mark.parametrize("skew", range(8))
@pytest.mark.parametrize("dtype,err,n_states", [
    (torch.bfloat16, 1, 2), (torch.bfloat16, 0, 1), (torch.float16, 2, 2), (torch.float16, 2, 1),
    (torch.float32, 0, 2), (torch.float32, 0, 1),
])
def test_staged_equals_register_path(dtype, err, n_states, skew):
    results = []
    for variant in (0, 1):
        rows, bufs, grad = _streams(SIZES, dtype, err, n_states, skew, seed=skew)
        keep = grad.clone()
        _run(rows, dtype, err, n_states, variant)
        assert torch.equal(grad, keep)
        results.append(bufs)
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("count", [len(MANY), 17, 33, 64])
def test_segment_look_up_over_many_tensors(count):
    sizes = MANY[-count:]
    # more chunks than the register path has CTAs: the staged kernel is the one that runs
    chunk = native.chunk_elems()
    assert sum(-(-n // chunk) for n in sizes) > native.load().fo_step_grid(torch.cuda.current_device())
    results = []
    for variant in (0, 1):
        rows, bufs, _ = _streams(sizes, torch.bfloat16, 1, 2, 0, seed=3)
        if variant == 0:  # one launch per tensor: no look-up to get wrong
            for i in range(count):
                _run(rows[i:i + 1].copy(), torch.bfloat16, 1, 2, 0)
        else:
            _run(rows, torch.bfloat16, 1, 2, 1)
        results.append(bufs)
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("variant", [0, 1])
def test_steps_back_to_back_and_in_a_graph(variant):
    """A step's grid may become resident while the one before it drains: without waiting in between,
    and replayed from a graph, the steps leave what they leave one at a time."""
    results = []
    for how in ("apart", "together", "graph"):
        rows, bufs, _ = _streams((1_500_017, 70_001, 33), torch.bfloat16, 1, 2, 0, seed=1)
        table = SegmentTable(torch.device("cuda", torch.cuda.current_device()))
        h = AdamHyper(lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=1e-5, step=7, decoupled=True)

        def steps(n):
            for _ in range(n):
                launch_adam(table, rows, torch.bfloat16, 1, True, h)
                if how == "apart":
                    torch.cuda.synchronize()

        set_step_variant(variant)
        try:
            torch.cuda.synchronize()
            if how == "graph":
                steps(1)  # what is set up on first use is there before the capture
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    steps(3)
                for _ in range(13):
                    graph.replay()
            else:
                steps(40)
            torch.cuda.synchronize()
        finally:
            set_step_variant(1)
        results.append(bufs)
    for other in results[1:]:
        for a, b in zip(results[0], other):
            assert torch.equal(a, b)
