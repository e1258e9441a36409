"""The native walk over a parameter group against the Python walk: same kernels, so same bits."""

import copy

import pytest
import torch
import torch.nn as nn

import flashoptim_b200 as fo
from flashoptim_b200.ops import step as fo_step

pytestmark = pytest.mark.gpu


def _state_tensors(opt):
    out = []
    for group in opt.param_groups:
        for p in group["params"]:
            for key, v in sorted(opt.state[p].items()):
                parts = [v] if isinstance(v, torch.Tensor) else [v.quantized, v.scales] if v.is_quantized() else [v.data]
                out += [(key, t.cpu()) for t in parts]
            out.append(("param", p.detach().cpu()))
    return out


def _make(cls, kw, dtypes, count, seed=0):
    g = torch.Generator().manual_seed(seed)
    params = []
    for i in range(count):
        n = (1, 33, 4097, 64, 31, 8192)[i % 6]
        params.append(nn.Parameter(torch.randn(n, generator=g).to(dtypes[i % len(dtypes)]).cuda()))
    params[1].requires_grad_(False)
    params.append(nn.Parameter(torch.zeros(0, dtype=dtypes[0], device="cuda")))
    return params, cls([dict(params=params[:count // 2]), dict(params=params[count // 2:], lr=0.02)], lr=0.01, **kw)


def _grads(params, seed, skip):
    g = torch.Generator().manual_seed(seed)
    for i, p in enumerate(params):
        grad = torch.randn(p.shape, generator=g).to(p.dtype).cuda()
        p.grad = grad if p.requires_grad and i not in skip else None


@pytest.mark.parametrize("cls,kw", [
    (fo.FlashAdamW, {}), (fo.FlashAdam, dict(weight_decay=0.1, quantize=False, master_weight_bits=32)),
    (fo.FlashLion, dict(weight_decay=0.1, master_weight_bits=32)), (fo.FlashSGDW, dict(momentum=0.9, nesterov=True)),
    (fo.FlashSGD, {}), (fo.FlashAdamW, dict(check_numerics=True)),
])
@pytest.mark.parametrize("count", [6, 44])  # table inside the kernel parameters, table on the device
def test_native_walk_equals_python_walk(cls, kw, count, monkeypatch):
    dtypes = (torch.bfloat16, torch.bfloat16, torch.float32, torch.float16)
    results = []
    for native in (True, False):
        params, opt = _make(cls, kw, dtypes, count)
        if not native:
            monkeypatch.setattr(opt, "_native_step_group", lambda *a: False)
        for it in range(4):
            # other parameters lack a gradient each time (step counts diverge), addresses move
            _grads(params, 10 + it, {it, it + 3})
            if it == 2:  # a state that was replaced, and one that was emptied
                opt.state[params[0]] = copy.copy(opt.state[params[0]])
                opt.state[params[4]] = {}
            n0 = fo_step.launch_count()
            opt.step()
            assert fo_step.launch_count() > n0
        assert native == (opt._walker is not None)
        torch.cuda.synchronize()
        results.append(_state_tensors(opt))
    assert len(results[0]) == len(results[1])
    for (ka, a), (kb, b) in zip(*results):
        assert ka == kb and torch.equal(a, b), ka


def test_step_param_skips_what_a_collective_updated_once():
    p = nn.Parameter(torch.randn(100, device="cuda").bfloat16())
    opt = fo.FlashAdamW([p], lr=0.1)
    p.grad = torch.ones_like(p)
    opt._peer_stepped.add(id(p))
    before = p.detach().clone()
    opt.step_param(p)
    assert torch.equal(p, before) and not opt._peer_stepped
    opt.step_param(p, opt.param_groups[0])
    assert not torch.equal(p, before) and opt.state[p]["step"].item() == 1


def test_refusals_come_from_the_python_walk():
    p = nn.Parameter(torch.randn(8, 8, device="cuda").bfloat16())
    opt = fo.FlashAdamW([p], lr=0.1)
    p.grad = torch.ones(8, 8, device="cuda", dtype=torch.bfloat16).t()[:, ::1].t().t()
    with pytest.raises(RuntimeError, match="contiguous gradient"):
        opt.step()
    p.grad = torch.ones_like(p)
    opt.step()
    opt.state[p]["exp_avg"]._quantized = torch.zeros(63, dtype=torch.int8, device="cuda")
    with pytest.raises(ValueError, match="63 codes"):
        opt.step()


def test_hooks_and_profiler_still_see_the_step():
    p = nn.Parameter(torch.randn(100, device="cuda").bfloat16())
    opt = fo.FlashAdamW([p], lr=0.1)
    p.grad = torch.ones_like(p)
    opt.step()
    calls = []
    h = opt.register_step_pre_hook(lambda *a: calls.append("pre"))
    opt.register_step_post_hook(lambda *a: calls.append("post"))
    opt.step()
    assert calls == ["pre", "post"]
    h.remove()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        opt.step()
    assert any("Optimizer.step#FlashAdamW" in e.key for e in prof.key_averages())
    sched = torch.optim.lr_scheduler.StepLR(opt, 1)
    opt.step()
    sched.step()


def test_an_allocation_that_fails_in_a_step_is_an_exception_and_leaves_the_step_undone():
    """The address table of a long list does not fit any more: out of memory, raised as such, with
    parameters, states and step counts as they were; the next step is made as if nothing had been."""
    results = []
    for short_of_memory in (True, False):
        params, opt = _make(fo.FlashAdamW, {}, (torch.bfloat16,), 44)
        _grads(params, 1, ())
        opt.step()
        _grads(params, 2, (4, 5))  # another number of rows, at other addresses
        if short_of_memory:
            before = _state_tensors(opt)
            fill = []
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            torch.cuda.set_per_process_memory_fraction(0.0)
            try:
                with pytest.raises(torch.OutOfMemoryError):
                    while True:  # what is left in the allocator's small blocks
                        fill.append(torch.empty(512, dtype=torch.uint8, device="cuda"))
                with pytest.raises(torch.OutOfMemoryError):
                    opt.step()
            finally:
                torch.cuda.set_per_process_memory_fraction(1.0)
            for (_, a), (_, b) in zip(before, _state_tensors(opt)):
                assert torch.equal(a, b)
        opt.step()
        results.append(_state_tensors(opt))
    for (ka, a), (kb, b) in zip(*results):
        assert ka == kb and torch.equal(a, b), ka


def test_address_tables_are_not_freed_or_shared_under_a_launch_on_another_stream():
    """Parameters come and go while steps run on two streams: every stream and number of rows keeps
    its own table, and what the steps leave is what they leave on one stream."""
    results = []
    for streams in (2, 1):
        params = [nn.Parameter(torch.linspace(-1, 1, 700 + i, device="cuda").bfloat16()) for i in range(40)]
        opt = fo.FlashLion(params, lr=0.01)
        other = torch.cuda.Stream() if streams == 2 else torch.cuda.current_stream()
        seen = []
        for it, (count, stream) in enumerate([(20, None), (20, other), (24, other), (20, other), (24, None), (40, other)]):
            _grads(params, it, range(count, 40))
            side = stream if stream is not None else torch.cuda.current_stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                torch.cuda._sleep(2_000_000)  # about a millisecond: the launches behind it are still to come
                opt.step()
            seen.append(dict.fromkeys(opt._walker.tables()))
            assert all(t in seen[-1] for before in seen for t in before)
            # nothing of a table's size that is allocated now lies where a table does
            blocks = [torch.empty(n * 68 + 4, dtype=torch.uint8, device="cuda") for n in (20, 24) * 4]
            assert not {b.data_ptr() for b in blocks} & {t[1] for t in seen[-1]}
            torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        if streams == 2:
            assert sorted(t[0] for t in seen[-1]) == [20, 20, 24, 24, 40]
        results.append(_state_tensors(opt))
    for (ka, a), (kb, b) in zip(*results):
        assert ka == kb and torch.equal(a, b), ka


@pytest.mark.parametrize("native", [True, False])
def test_a_captured_step_keeps_its_address_table(native, monkeypatch):
    """Steps between capture and replay, on other gradients and with another number of rows, change
    nothing about what a replay updates from, and a replay nothing about what the next step does."""
    results = []
    for capture in (True, False):
        params = [nn.Parameter(torch.linspace(-1, 1, 700 + i, device="cuda").bfloat16()) for i in range(30)]
        opt = fo.FlashLion(params, lr=0.01)
        if not native:
            monkeypatch.setattr(opt, "_native_step_group", lambda *a: False)

        def step(seed, count):
            _grads(params, seed, range(count, 30))
            opt.step()

        step(0, 20)
        _grads(params, 1, range(20, 30))
        held = [p.grad for p in params]  # the captured step's gradients
        if capture:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                opt.step()
                opt.step()

        def replay():
            if capture:
                graph.replay()
                return
            now = [p.grad for p in params]
            for again in (0, 1):
                for p, g in zip(params, held):
                    p.grad = g
                opt.step()
            for p, g in zip(params, now):
                p.grad = g

        opt.step()  # the rows of the captured step, before its copies have run once
        step(2, 24)
        if capture and native:
            kept = {t[2] for t in opt._walker.tables()} - {0}
            assert len(kept) == 2
            blocks = [torch.empty(20 * 68 + 4, dtype=torch.uint8).pin_memory() for _ in range(8)]
            assert not {b.data_ptr() for b in blocks} & kept
        replay()
        step(3, 20)
        replay()
        opt.step()
        replay()
        replay()
        torch.cuda.synchronize()
        results.append(_state_tensors(opt))
    for (ka, a), (kb, b) in zip(*results):
        assert ka == kb and torch.equal(a, b), ka


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("betas,count,error", [
    ((0.9, 1.5), 1.0, ValueError), ((1.5, 0.9), 1e6, OverflowError), ((0.9, 1.0), 1.0, ZeroDivisionError),
    ((0.9, 0.999), -3.0, ValueError), ((0.9, 0.999), float("nan"), ValueError),
])
def test_moment_factors_and_step_counts_without_a_bias_correction_are_refused(native, betas, count, error, monkeypatch):
    p = nn.Parameter(torch.ones(100, device="cuda").bfloat16())
    opt = fo.FlashAdamW([p], lr=0.1)
    if not native:
        monkeypatch.setattr(opt, "_native_step_group", lambda *a: False)
    p.grad = torch.ones_like(p)
    opt.step()
    before = p.detach().clone()
    opt.param_groups[0]["betas"] = betas
    opt.state[p]["step"].fill_(count)
    with pytest.raises(error):
        opt.step()
    assert torch.equal(p, before)


def test_a_step_count_that_parameters_share(monkeypatch):
    results = []
    for native in (True, False):
        params = [nn.Parameter(torch.linspace(-1, 1, 700 + i, device="cuda").bfloat16()) for i in range(5)]
        opt = fo.FlashAdamW(params, lr=0.01)
        if not native:
            monkeypatch.setattr(opt, "_native_step_group", lambda *a: False)
        for it in range(3):
            _grads(params, it, ())
            opt.step()
            for p in params[1:3]:
                opt.state[p]["step"] = opt.state[params[0]]["step"]
        results.append(_state_tensors(opt))
    for (ka, a), (kb, b) in zip(*results):
        assert ka == kb and torch.equal(a, b), ka


@pytest.mark.parametrize("lost", ["gradient", "state"])
def test_what_goes_during_the_walk_is_kept_until_the_launch(lost, monkeypatch):
    """A method that the walk calls drops a gradient, or replaces a state, that was looked at before,
    and its memory is used again at once."""
    results = []
    for native in (True, False):
        class Lion(fo.FlashLion):
            def _check_param_numerics(self, p, *args):
                if p is params[2] and armed:
                    if lost == "gradient":
                        params[0].grad = None
                    else:
                        self.state[params[0]] = {}
                    armed.append([torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(8)])

        params = [nn.Parameter(torch.linspace(-1, 1, 1 << 21, device="cuda").bfloat16()) for _ in range(4)]
        opt = Lion(params, lr=0.01, check_numerics=True)
        if not native:
            monkeypatch.setattr(opt, "_native_step_group", lambda *a: False)
        armed = []
        for p in params:
            p.grad = torch.linspace(-1, 1, 1 << 21, device="cuda").bfloat16()
        opt.step()
        armed.append(True)
        opt.step()
        torch.cuda.synchronize()
        results.append([p.detach().cpu() for p in params])
    for a, b in zip(*results):
        assert torch.equal(a, b)


def test_sharded_parameters_are_walked_as_in_python(monkeypatch):
    """DTensors (parameters and gradients) on a mesh of one, with more rows than fit the parameters."""
    import torch.distributed as dist
    from torch.distributed.device_mesh import init_device_mesh
    from torch.distributed.tensor import DTensor, Replicate, Shard

    dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    try:
        mesh = init_device_mesh("cuda", (1,))
        results = []
        for native in (True, False):
            g = torch.Generator().manual_seed(5)

            def sharded(i, dtype):
                t = torch.randn((33, 1025, 4096, 7)[i % 4] + i, generator=g).to(dtype).cuda()
                return DTensor.from_local(t, mesh, [Shard(0) if i % 3 else Replicate()])

            dtypes = [torch.float32 if i % 5 == 4 else torch.bfloat16 for i in range(24)]
            params = [nn.Parameter(sharded(i, d)) for i, d in enumerate(dtypes)]
            opt = fo.FlashAdamW(params, lr=0.01)
            if not native:
                monkeypatch.setattr(opt, "_native_step_group", lambda *a: False)
            for _ in range(3):
                for i, (p, d) in enumerate(zip(params, dtypes)):
                    p.grad = sharded(i, d)
                opt.step()
            assert native == bool(opt._walker is not None and opt._walker.tables())
            torch.cuda.synchronize()
            results.append([(k, t.to_local() if isinstance(t, DTensor) else t) for k, t in _state_tensors(opt)])
        for (ka, a), (kb, b) in zip(*results):
            assert ka == kb and torch.equal(a, b), ka
    finally:
        dist.destroy_process_group()
