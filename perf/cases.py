"""Timed workloads of this library, through its public entry points.

A case is a dict of plain values.  ``kind`` says which call is timed:

* ``step``        ``optimizer.step()`` on a whole parameter list whose gradients are in place;
* ``step_param``  ``optimizer.step_param()`` tensor by tensor, as gradient release drives it;
* ``save`` / ``load``      ``state_dict()`` / ``load_state_dict()``, plain or compressed flavour;
* ``export`` / ``import``  fp32 master weights out of / into the narrow model;
* ``quantize``    the group quantiser and its inverse on one tensor.

Optimizers start as a resumed run does: from a checkpoint at step 1000 with moments, scales and
correction codes of trained magnitude.  A list of tensors is laid out as views of one buffer per
stream (parameters, codes, scales, moments), every tensor at a 512-byte boundary as the caching
allocator would place it, so that what a step wrote can be handed back whole.
"""

from __future__ import annotations

import math
from typing import Any

import torch

import flashoptim_b200 as fo

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
WIDTH = {"bf16": 2, "fp16": 2, "fp32": 4}
STATES = {"adam": 2, "adamw": 2, "lion": 1, "sgd": 1, "sgdw": 1}
ALIGN = 8192  # elements; the narrowest stream, one fp16 scale per 32 elements, then starts at 512 bytes too
MOST_BYTES = 12.2e9  # of a drawn case: the largest listed one needs 12.3e9


def _step(name: str, **kw: Any) -> dict[str, Any]:
    case = dict(name=name, kind="step", optimizer="adamw", dtype="bf16", bits=24, quantize=True, groups=1,
                grads="separate")
    case.update(kw)
    return case


def listed() -> list[dict[str, Any]]:
    return [
        # the 784-256-10 classifier of the training example: four tensors, all latency
        _step("mlp_adamw24", layout="mlp", d_in=784, hidden=256, depth=1, d_out=10),
        # a GPT-2-medium list as it is usually trained: weight decay on matrices only, two groups
        _step("gpt2_medium_adamw24", layout="gpt", layers=24, width=1024, ffn=4096, vocab=50257, context=1024,
              groups=2),
        # one rank's share of Llama-3-8B under FSDP2 on eight GPUs: 291 tensors, 1.0 B elements
        _step("llama8b_shard_adamw24", layout="decoder", layers=32, width=4096, kv=1024, ffn=14336, vocab=128256,
              shard=8),
        # gradient release over one Llama-3-70B layer's shards on eight GPUs: Lion, 32-bit masters
        _step("llama70b_layer_lion32_release", kind="step_param", optimizer="lion", bits=32, layout="block",
              layers=1, width=8192, kv=1024, ffn=28672, shard=8),
        # a cast convolutional network: batch norms stay fp32, everything else is bf16
        _step("resnet18_sgdw24", optimizer="sgdw", layout="resnet18", d_out=10),
        # fp32 training with 8-bit states only, no narrow parameters (12 layers of width 768)
        _step("fp32_adamw8", dtype="fp32", bits=None, layout="gpt", layers=12, width=768, ffn=3072, vocab=50257,
              context=1024),
        # odd widths, fp16, gradients as views of a DDP bucket (back to back, at any offset)
        _step("ragged_adam32_bucket", optimizer="adam", dtype="fp16", bits=32, layout="gpt", layers=6, width=1021,
              ffn=4093, vocab=32003, context=509, grads="bucket"),
        # writing a checkpoint in the flavour that stock optimizers read, and reading one back
        _step("save_plain", kind="save", compressed=False, layout="block", layers=1, width=4096, kv=1024, ffn=14336,
              shard=1),
        _step("load_plain", kind="load", compressed=False, layout="block", layers=1, width=4096, kv=1024, ffn=14336,
              shard=1),
        # fp32 masters for evaluation or conversion, and back into the training run
        _step("export_fp32", kind="export", layout="block", layers=2, width=4096, kv=1024, ffn=14336, shard=1),
        _step("import_fp32", kind="import", layout="block", layers=2, width=4096, kv=1024, ffn=14336, shard=1),
        # the tensor functions on their own, at a length that is no multiple of anything
        dict(name="quantize_round_trip", kind="quantize", dtype="bf16", n=100_000_007, signed=True, sqrt=False,
             softsign=True),
    ]


# ------------------------------------------------------------------ parameter lists
def _shapes(case: dict[str, Any]) -> list[tuple[int, ...]]:
    layout = case["layout"]
    if layout == "mlp":
        widths = [case["d_in"]] + [case["hidden"]] * case["depth"] + [case["d_out"]]
        return [s for a, b in zip(widths, widths[1:]) for s in ((b, a), (b,))]
    if layout == "resnet18":
        shapes: list[tuple[int, ...]] = [(64, 3, 7, 7), (64,), (64,)]
        c_in = 64
        for c in (64, 128, 256, 512):
            for block in range(2):
                shapes += [(c, c_in, 3, 3), (c,), (c,), (c, c, 3, 3), (c,), (c,)]
                if block == 0 and c != c_in:
                    shapes += [(c, c_in, 1, 1), (c,), (c,)]
                c_in = c
        return shapes + [(case["d_out"], 512), (case["d_out"],)]
    d, f = case["width"], case["ffn"]
    if layout == "gpt":
        shapes = [(case["vocab"], d), (case["context"], d)]
        for _ in range(case["layers"]):
            shapes += [(d,), (d,), (3 * d, d), (3 * d,), (d, d), (d,), (d,), (d,), (f, d), (f,), (d, f), (d,)]
        return shapes + [(d,), (d,)]
    kv = case["kv"]
    shapes = []
    for _ in range(case["layers"]):
        shapes += [(d, d), (kv, d), (kv, d), (d, d), (f, d), (f, d), (d, f), (d,), (d,)]
    if layout == "decoder":
        shapes = [(case["vocab"], d)] + shapes + [(d,), (case["vocab"], d)]
    return [(-(-s[0] // case["shard"]), *s[1:]) for s in shapes]


def _dtype_of(case: dict[str, Any], shape: tuple[int, ...], index: int, last: int) -> str:
    """Batch-norm vectors of the convolutional network stay fp32 (``cast_model`` keeps them)."""
    if case["layout"] == "resnet18" and len(shape) == 1 and index != last:
        return "fp32"
    return case["dtype"]


def _tensors(case: dict[str, Any]) -> list[tuple[tuple[int, ...], str]]:
    shapes = _shapes(case)
    return [(s, _dtype_of(case, s, i, len(shapes) - 1)) for i, s in enumerate(shapes)]


def _code_bytes(dtype: str, bits: int | None) -> int:
    return 0 if bits is None else max(0, bits // 8 - WIDTH[dtype])


def work(case: dict[str, Any]) -> dict[str, float]:
    if case["kind"] == "quantize":
        n = case["n"]
        scales = -(-n // 32) * 2
        return {"bytes": n * (WIDTH[case["dtype"]] + 2 + 4) + 2 * scales, "flops": 14 * n}
    total = flops = 0
    for shape, dt in _tensors(case):
        n, w, e = math.prod(shape), WIDTH[dt], _code_bytes(dt, case["bits"])
        scales = -(-n // 32) * 2
        k = STATES[case["optimizer"]]
        state = n + scales if case["quantize"] else n * w
        if case["kind"] in ("step", "step_param"):
            total += n * (3 * w + 2 * e) + 2 * k * state
            flops += n * (12 * k + 4)
        elif case["kind"] in ("save", "load"):
            # moments: codes + scales on one side, bf16 on the other; the compressed flavour hands
            # the codes over as they are.  Corrections travel in the parameter's dtype.
            total += (0 if case["compressed"] else k * (state + 2 * n)) + (n * (e + w) if e != w else 0)
            flops += 0 if case["compressed"] else 6 * n * k
        else:
            total += n * (w + e + 4)
            flops += 4 * n
    return {"bytes": max(total, 64), "flops": flops}


def tolerance(case: dict[str, Any]) -> Any:
    if case["kind"] in ("save", "load", "export", "import", "quantize"):
        return "exact"  # one defined rounding each: bit for bit the written-down formulas
    # narrow parameters: half a unit in the last place of their mantissa.  fp32 parameters: fp32
    # sums; the fp16 group scales beside them may round the other way at a tie.
    rel = {"bf16": 4e-3, "fp16": 5e-4, "fp32": 1e-4}[case["dtype"]]
    # codes: a value next to a rounding boundary may fall on either side of it
    return {"rel": rel, "differ": 0.01}


# ------------------------------------------------------------------ what a program has in hand
class _Arena:
    """The tensors of one dtype: buffers of every stream, and each tensor's place in them."""

    def __init__(self, case: dict[str, Any], dtype: str, shapes: list[tuple[int, ...]], gen: torch.Generator):
        self.dtype, self.shapes = DTYPES[dtype], shapes
        self.starts, total = [], 0
        for s in shapes:
            self.starts.append(total)
            total += -(-math.prod(s) // ALIGN) * ALIGN
        self.adam = STATES[case["optimizer"]] == 2
        self.quantize = case["quantize"]
        master = torch.empty(total, device="cuda").normal_(0.0, 0.02, generator=gen)
        self.param = master.to(self.dtype)
        self.code_bytes = _code_bytes(dtype, case["bits"])
        self.ecc = None
        if self.code_bytes:
            self.ecc = fo.compute_ecc_bits(master, self.param, master_bytewidth=case["bits"] // 8)
        del master
        self.m = torch.empty(total, device="cuda").normal_(0.0, 3e-4, generator=gen)
        self.v = torch.empty(total, device="cuda").normal_(0.0, 1e-3, generator=gen).square_() if self.adam else None
        self.ms = self.vs = None
        if self.quantize:
            self.m, self.ms = fo.quantize(self.m)
            if self.adam:
                self.v, self.vs = fo.quantize(self.v, signed=False, sqrt=True, softsign=False)
        else:
            self.m = self.m.to(self.dtype)
            self.v = self.v.to(self.dtype) if self.adam else None
        self.bucket = case.get("grads") == "bucket"
        g_total = sum(math.prod(s) for s in shapes) if self.bucket else total
        self.grad = torch.empty(g_total, device="cuda", dtype=self.dtype).normal_(0.0, 1e-3, generator=gen)

    def view(self, buf: torch.Tensor, i: int) -> torch.Tensor:
        n = math.prod(self.shapes[i])
        return buf[self.starts[i]:self.starts[i] + n].view(self.shapes[i])

    def scales(self, buf: torch.Tensor, i: int) -> torch.Tensor:
        at = self.starts[i] // 32
        return buf[at:at + -(-math.prod(self.shapes[i]) // 32)]

    def grad_view(self, i: int) -> torch.Tensor:
        if not self.bucket:
            return self.view(self.grad, i)
        # a bucket holds gradients in the order in which backward produces them: last tensor first
        at = sum(math.prod(s) for s in self.shapes[i + 1:])
        return self.grad[at:at + math.prod(self.shapes[i])].view(self.shapes[i])

    def checkpoint_entry(self, case: dict[str, Any], i: int) -> dict[str, torch.Tensor]:
        first = "momentum_buffer" if case["optimizer"].startswith("sgd") else "exp_avg"
        out: dict[str, torch.Tensor] = {}
        moments = [(first, self.m, self.ms)] + ([("exp_avg_sq", self.v, self.vs)] if self.adam else [])
        for name, codes, sc in moments:
            if self.quantize:
                out[name + "::quantized"] = self.view(codes, i)
                out[name + "::scales"] = self.scales(sc, i)
            else:
                out[name] = self.view(codes, i)
        if self.adam:
            out["step"] = torch.tensor(1000.0)
        if self.ecc is not None:
            e = self.view(self.ecc, i)
            out["error_bits"] = e.to(self.dtype) if self.code_bytes == 1 else e.view(self.dtype)
        return out

    def outputs(self) -> dict[str, torch.Tensor]:
        named = dict(param=self.param, ecc=self.ecc, m=self.m, ms=self.ms, v=self.v, vs=self.vs)
        return {k: t for k, t in named.items() if t is not None}


def _optimizer(case: dict[str, Any], params: list[torch.nn.Parameter], compressed: bool) -> Any:
    groups: Any = params
    if case["groups"] == 2:
        groups = [dict(params=[p for p in params if p.dim() >= 2]),
                  dict(params=[p for p in params if p.dim() < 2], weight_decay=0.0)]
    kw = dict(lr=3e-4, weight_decay=0.01, master_weight_bits=case["bits"], quantize=case["quantize"],
              compress_state_dict=compressed)
    name = case["optimizer"]
    if name.startswith("sgd"):
        kw.update(momentum=0.9, nesterov=bool(case.get("nesterov", False)))
    if name == "lion":
        kw.update(lr=1e-4)
    cls = dict(adam=fo.FlashAdam, adamw=fo.FlashAdamW, lion=fo.FlashLion, sgd=fo.FlashSGD, sgdw=fo.FlashSGDW)[name]
    return cls(groups, **kw)


def _resumed(case: dict[str, Any], seed: int) -> dict[str, Any]:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    tensors = _tensors(case)
    arenas, place, count = {}, [], {}
    for _, dt in tensors:
        place.append((dt, count.setdefault(dt, 0)))
        count[dt] += 1
    for dt in count:
        arenas[dt] = _Arena(case, dt, [s for s, d in tensors if d == dt], gen)
    params = [torch.nn.Parameter(arenas[dt].view(arenas[dt].param, i)) for dt, i in place]
    grads = [arenas[dt].grad_view(i) for dt, i in place]
    opt = _optimizer(case, params, bool(case.get("compressed", False)))
    where = {id(p): at for p, at in zip(params, place)}
    ordered = [p for g in opt.param_groups for p in g["params"]]
    checkpoint = opt.state_dict()
    checkpoint["state"] = {k: arenas[where[id(p)][0]].checkpoint_entry(case, where[id(p)][1])
                           for k, p in enumerate(ordered)}
    opt.load_state_dict(checkpoint)  # 8-bit codes and scales stay where the checkpoint has them
    for p in ordered:
        dt, i = where[id(p)]
        if arenas[dt].ecc is not None:
            opt.state[p]["error_bits"] = arenas[dt].view(arenas[dt].ecc, i)
    return dict(case=case, opt=opt, params=params, grads=grads, arenas=arenas)


def prepare(case: dict[str, Any], seed: int) -> dict[str, Any]:
    if case["kind"] == "quantize":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.empty(case["n"], device="cuda").normal_(0.0, 1e-3, generator=gen)
        x = (x.square_() if case["sqrt"] else x).to(DTYPES[case["dtype"]])
        return dict(case=case, x=x, how=dict(signed=case["signed"], sqrt=case["sqrt"], softsign=case["softsign"]))
    state = _resumed(case, seed)
    kind = case["kind"]
    if kind == "step":
        for p, g in zip(state["params"], state["grads"]):
            p.grad = g
    elif kind == "step_param":
        opt = state["opt"]
        group_of = {id(p): g for g in opt.param_groups for p in g["params"]}
        # backward finishes the last tensor first
        state["order"] = [(p, g, group_of[id(p)]) for p, g in zip(state["params"], state["grads"])][::-1]
    else:
        state["grads"] = None
        for a in state["arenas"].values():
            a.grad = None
        state["model"] = torch.nn.ParameterList(state["params"])
        if kind == "load":
            state["checkpoint"] = state["opt"].state_dict()
        if kind == "import":
            state["fp32"] = state["opt"].get_fp32_model_state_dict(state["model"])
    return state


def _state_tensors(opt: Any, params: list[torch.nn.Parameter]) -> list[dict[str, Any]]:
    out = []
    for p in params:
        entry = {}
        for key, value in opt.state[p].items():
            if isinstance(value, torch.Tensor):
                entry[key] = value
            elif value.is_quantized():
                entry[key] = [value.quantized, value.scales]
            else:
                entry[key] = value.data
        out.append(entry)
    return out


# ------------------------------------------------------------------ the timed call
def run(state: dict[str, Any]) -> Any:
    kind = state["case"]["kind"]
    if kind == "quantize":
        codes, scales = fo.quantize(state["x"], **state["how"])
        return codes, scales, fo.dequantize(codes, scales, **state["how"])
    opt = state["opt"]
    if kind == "step":
        opt.step()
        return {dt: a.outputs() for dt, a in state["arenas"].items()}
    if kind == "step_param":
        for p, g, group in state["order"]:
            p.grad = g
            opt.step_param(p, group)
            p.grad = None
        return {dt: a.outputs() for dt, a in state["arenas"].items()}
    if kind == "save":
        return opt.state_dict()["state"]
    if kind == "load":
        opt.load_state_dict(state["checkpoint"])
        return _state_tensors(opt, state["params"])
    if kind == "export":
        return opt.get_fp32_model_state_dict(state["model"])
    opt.set_fp32_model_state_dict(state["model"], state["fp32"])
    return [[p, opt.state[p].get("error_bits")] for p in state["params"]]


# ------------------------------------------------------------------ more cases of the same ranges
def _log_int(rng: Any, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _width(rng: Any, low: int, high: int) -> int:
    """A layer width: usually a multiple of 64, sometimes any number."""
    w = _log_int(rng, low, high)
    return w if rng.random() < 0.35 else max(64, (w + 32) // 64 * 64)


def _draw_layout(rng: Any, few: bool) -> dict[str, Any]:
    """``few``: at most ten tensors (checkpoint and export cases hand every tensor back)."""
    pick = rng.random()
    if pick < (0.4 if few else 0.25):
        return dict(layout="mlp", d_in=_width(rng, 32, 4096), hidden=_width(rng, 64, 8192),
                    depth=rng.randint(1, 3 if few else 6), d_out=_log_int(rng, 2, 1000))
    if few or pick < 0.4:
        d = _width(rng, 256, 8192)
        return dict(layout="block", layers=1, width=d, kv=max(64, d // rng.choice([1, 4, 8])),
                    ffn=_width(rng, 2 * d, 4 * d), shard=rng.choice([1, 1, 2, 4, 8]))
    if not few and pick < 0.45:
        return dict(layout="resnet18", d_out=_log_int(rng, 2, 1000))
    d = _width(rng, 128, 4096)
    if pick < 0.75:
        return dict(layout="gpt", layers=_log_int(rng, 2, 32), width=d, ffn=4 * d, vocab=_log_int(rng, 500, 60000),
                    context=_log_int(rng, 64, 2048))
    return dict(layout="decoder", layers=_log_int(rng, 2, 32), width=d, kv=max(64, d // rng.choice([1, 4, 8])),
                ffn=_width(rng, 2 * d, 4 * d), vocab=_log_int(rng, 500, 130000), shard=rng.choice([1, 2, 4, 8]))


def draw(rng: Any) -> dict[str, Any]:
    pick = rng.random()
    if pick < 0.06:
        signed = rng.random() < 0.5
        return dict(kind="quantize", dtype=rng.choice(["bf16", "fp16", "fp32"]), n=_log_int(rng, 1000, 400_000_000),
                    signed=signed, sqrt=not signed, softsign=signed)
    kind = ("step" if pick < 0.68 else "step_param" if pick < 0.8 else "save" if pick < 0.85 else
            "load" if pick < 0.9 else "export" if pick < 0.95 else "import")
    checkpointing = kind in ("save", "load", "export", "import")
    while True:
        case = dict(kind=kind, optimizer=rng.choice(["adamw", "adamw", "adamw", "adam", "lion", "sgd", "sgdw"]))
        case["dtype"] = "bf16" if checkpointing else rng.choice(["bf16", "bf16", "bf16", "bf16", "fp16", "fp32"])
        case["bits"] = None if case["dtype"] == "fp32" else rng.choice([24, 24, 32] if checkpointing else [24, 24, 32, None])
        case["quantize"] = checkpointing or case["dtype"] == "fp16" or rng.random() < 0.85
        case["groups"] = rng.choice([1, 1, 2])
        case["grads"] = "bucket" if kind == "step" and rng.random() < 0.3 else "separate"
        if case["optimizer"].startswith("sgd"):
            case["nesterov"] = rng.random() < 0.3
        if kind in ("save", "load"):
            case["compressed"] = rng.random() < 0.3
        case.update(_draw_layout(rng, few=checkpointing))
        if case["layout"] == "resnet18":
            case["dtype"], case["bits"] = "bf16", 24
        if work(case)["bytes"] <= MOST_BYTES:
            return case
