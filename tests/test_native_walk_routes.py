"""Which steps the native walk may take: what a subclass, a patch or an instance overrides is called."""

import pytest
import torch
import torch.nn as nn

import flashoptim_b200 as fo
from flashoptim_b200 import build
from flashoptim_b200.ops import host, native

OVERRIDES = ["_pre_step", "_pre_step_many", "_fused_step", "_step_group", "_ensure_state_initialized"]
CLASSES = [fo.FlashAdam, fo.FlashAdamW, fo.FlashLion, fo.FlashSGD, fo.FlashSGDW]


def _param(device="cpu"):
    return nn.Parameter(torch.ones(100, device=device).bfloat16())


def _counting(cls, name, calls):
    def method(self, *args, **kwargs):
        calls.append(name)
        return getattr(super(sub, self), name)(*args, **kwargs)

    sub = type("Sub", (cls,), {name: method})
    return sub


@pytest.mark.parametrize("cls", CLASSES)
@pytest.mark.parametrize("name", OVERRIDES)
def test_an_override_keeps_the_native_walk_out(cls, name, monkeypatch):
    assert not host.load().overrides(cls([_param()], lr=0.1))
    assert not host.load().overrides(type("Plain", (cls,), {})([_param()], lr=0.1))
    sub = _counting(cls, name, [])
    assert host.load().overrides(sub([_param()], lr=0.1))
    assert host.load().overrides(type("SubSub", (sub,), {})([_param()], lr=0.1))
    opt = cls([_param()], lr=0.1)
    setattr(opt, name, getattr(opt, name))
    assert host.load().overrides(opt)
    opt = cls([_param()], lr=0.1)
    original = getattr(cls, name)
    monkeypatch.setattr(cls, name, lambda *a, **k: original(*a, **k))
    assert host.load().overrides(opt)


@pytest.mark.gpu
def test_a_class_or_an_optimizer_that_changes_between_steps(monkeypatch):
    """The look at a class is remembered until the class, or one above it, changes."""
    class Lion(fo.FlashLion):
        pass

    calls = []
    p = _param("cuda")
    opt = Lion([p], lr=0.1)

    def steps():
        calls.clear()
        for _ in range(2):
            p.grad = torch.ones_like(p)
            opt.step()
        return len(calls)

    original = fo.FlashLion._pre_step
    patched = lambda self, state: calls.append(original(self, state))  # noqa: E731
    assert steps() == 0
    for owner in (Lion, fo.FlashLion, opt):
        with monkeypatch.context() as m:
            m.setattr(owner, "_pre_step", patched if owner is not opt else lambda state: calls.append(state))
            assert steps() == 2
        assert steps() == 0


def test_a_class_that_says_what_it_does_is_walked_natively():
    class Own(fo.FlashLion):
        def _pre_step_many(self, param_states):
            pass

        def _native_step_args(self, hparams):
            return super()._native_step_args(hparams)

    assert not host.load().overrides(Own([_param()], lr=0.1))


@pytest.mark.gpu
@pytest.mark.parametrize("cls", [fo.FlashAdamW, fo.FlashLion, fo.FlashSGDW])
@pytest.mark.parametrize("name", OVERRIDES)
def test_an_override_is_called_on_the_gpu_as_on_the_cpu(cls, name):
    calls = {"cpu": [], "cuda": []}
    for device, seen in calls.items():
        p = _param(device)
        opt = _counting(cls, name, seen)([p], lr=0.1)
        for _ in range(2):
            p.grad = torch.ones_like(p)
            opt.step()
            opt.step_param(p)
    if name == "_pre_step" and cls is fo.FlashAdamW:
        return  # Adam counts the steps of a fused launch in _pre_step_many; _pre_step is the eager path's
    if name in ("_pre_step_many", "_fused_step"):
        assert len(calls["cuda"]) == 4 and not calls["cpu"]
    else:
        assert len(calls["cuda"]) == len(calls["cpu"]) == 4


def _no_extension(monkeypatch, tried):
    def build_host(*args, **kwargs):
        tried.append(1)
        raise RuntimeError("no C++ compiler")

    monkeypatch.setattr(host, "_module", None)
    monkeypatch.setattr(host, "_unavailable", False)
    monkeypatch.setattr(build, "host_is_current", lambda: False)
    monkeypatch.setattr(build, "build_host", build_host)


def test_an_extension_that_cannot_be_built_is_reported_once(monkeypatch):
    tried = []
    _no_extension(monkeypatch, tried)
    monkeypatch.setattr(native, "load", lambda path=None: None)
    with pytest.warns(UserWarning, match="no C\\+\\+ compiler"):
        assert host.available() is None
    assert host.available() is None and len(tried) == 1  # neither warned of nor tried again


def test_kernels_that_cannot_be_loaded_are_an_error(monkeypatch):
    def load(path=None):
        raise native.NativeError("missing")

    _no_extension(monkeypatch, [])
    monkeypatch.setattr(native, "load", load)
    with pytest.raises(native.NativeError, match="missing"):
        host.available()


@pytest.mark.gpu
def test_steps_without_the_extension_are_the_same_steps(monkeypatch):
    results = []
    for extension in (True, False):
        if not extension:
            _no_extension(monkeypatch, [])
        params = [nn.Parameter(torch.linspace(-1, 1, 700 + i, device="cuda").bfloat16()) for i in range(20)]
        opt = fo.FlashAdamW(params, lr=0.1)
        for p in params:
            p.grad = torch.ones_like(p)
        if extension:
            opt.step()
        else:
            with pytest.warns(UserWarning, match="Python walk"):
                opt.step()
        opt.step_param(params[0])
        assert extension == (opt._walker is not None)
        results.append(torch.cat([p.detach() for p in params]))
    assert torch.equal(*results)


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_what_a_step_calls_runs_without_gradients(device):
    modes = {}

    class Lion(fo.FlashLion):
        def _initial_value_for_state_var(self, param, key):
            modes["state"] = torch.is_grad_enabled()
            return torch.zeros_like(param)

        def _check_param_numerics(self, *args):
            modes["check"] = torch.is_grad_enabled()

    for how in ("step", "step_param"):
        p = _param(device)
        opt = Lion([p], lr=0.1, check_numerics=True)
        opt._local_update_listeners.append(lambda params: modes.update(listener=torch.is_grad_enabled()))
        opt._post_step_callbacks.append(lambda: modes.update(callback=torch.is_grad_enabled()))
        p.grad = torch.ones_like(p)
        modes.clear()
        opt.step() if how == "step" else opt.step_param(p)
        assert torch.is_grad_enabled() and not any(modes.values())
        assert set(modes) == {"state", "check", "listener"} | ({"callback"} if how == "step" else set())
