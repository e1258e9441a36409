"""Step hooks see every step, whoever wrapped or overrode ``step()``, and the wrapper that skips
torch's bookkeeping does so only while nobody listens."""

import functools
import types

import pytest
import torch
import torch.nn as nn
from torch.optim.optimizer import register_optimizer_step_post_hook, register_optimizer_step_pre_hook

import flashoptim_b200 as fo
from flashoptim_b200.ops import host


@pytest.fixture(params=["extension loaded", "extension not loaded"])
def extension(request, monkeypatch):
    mod = types.SimpleNamespace(watched=False, observed=lambda: mod.watched, launches=lambda: 0)
    monkeypatch.setattr(host, "_module", mod if request.param == "extension loaded" else None)
    return mod


def _opt(cls):
    p = nn.Parameter(torch.ones(40))
    p.grad = torch.ones(40)
    return cls([p], lr=0.1, master_weight_bits=None)


def _hooked_calls(opt, **step_kwargs):
    calls = []
    opt.register_step_pre_hook(lambda o, args, kwargs: calls.append(("pre", args[1:], kwargs)))
    opt.register_step_post_hook(lambda o, args, kwargs: calls.append(("post", args[1:], kwargs)))
    opt.step(**step_kwargs)
    return calls


ONCE = [("pre", (), {}), ("post", (), {})]


def _logging(step, log):
    @functools.wraps(step)
    def wrapper(self, *args, **kwargs):
        log.append("wrapper")
        return step(self, *args, **kwargs)

    return wrapper


def test_hooks_get_the_arguments_of_the_call(extension):
    class Lion(fo.FlashLion):
        pass

    assert _hooked_calls(_opt(Lion)) == ONCE
    closure = lambda: None  # noqa: E731
    assert _hooked_calls(_opt(Lion), closure=closure) == [("pre", (), {"closure": closure}), ("post", (), {"closure": closure})]


@pytest.mark.parametrize("when", ["before the first instance", "after it"])
def test_a_class_whose_step_is_wrapped_still_runs_the_hooks(extension, when):
    class Lion(fo.FlashLion):
        pass

    if when == "after it":
        opt = _opt(Lion)
    log = []
    Lion.step = _logging(Lion.step, log)
    for o in ([opt] if when == "after it" else []) + [_opt(Lion)]:
        log.clear()
        assert _hooked_calls(o) == ONCE and log == ["wrapper"]


def test_an_override_that_copies_the_attributes_of_step_runs_the_hooks(extension):
    class Base(fo.FlashLion):
        pass

    class Lion(Base):
        @functools.wraps(Base.step)
        def step(self, closure=None):
            log.append("override")
            return super().step(closure)

    log = []
    assert [c[0] for c in _hooked_calls(_opt(Lion))] == ["pre", "post"] and log == ["override"]


def test_an_override_that_does_all_by_itself_runs_the_hooks(extension):
    class Lion(fo.FlashLion):
        def step(self, closure=None):
            return 7

    calls = _hooked_calls(opt := _opt(Lion))
    assert calls == ONCE and opt.step() == 7


def test_hooks_of_every_optimizer(extension):
    calls = []
    handles = [register_optimizer_step_pre_hook(lambda *a: calls.append("pre")),
               register_optimizer_step_post_hook(lambda *a: calls.append("post"))]
    try:
        _opt(fo.FlashLion).step()
    finally:
        for h in handles:
            h.remove()
    _opt(fo.FlashLion).step()
    assert calls == ["pre", "post"]


def test_torch_wraps_nothing_around_a_step_that_nobody_watches(extension, monkeypatch):
    names = []
    real = torch.autograd.profiler.record_function

    class Recorded(real):
        def __init__(self, name, *args):
            names.append(name)
            super().__init__(name, *args)

    monkeypatch.setattr(torch.autograd.profiler, "record_function", Recorded)
    opt = _opt(fo.FlashLion)
    opt.step()
    assert bool(names) == (host._module is None)
    extension.watched = True
    names.clear()
    opt.step()
    assert names == ["Optimizer.step#FlashLion.step"]
