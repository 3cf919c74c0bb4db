"""The work that users of this package have it do, as timed cases.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare(case, seed)`` makes what a
program has in hand before the call, ``run(state)`` is one pass through the public entry points, ``work(case)`` the
bytes and operations of a pass that no implementation can do without, ``tolerance(case)`` how far another correct
implementation of the same precision may be off.

Kinds of cases:

``core``    ``ssd_forward``: the SSD scan alone (prefill), optionally with dt, initial states in and final states out
``mixer``   what a layer does between its two projections: ``conv1d_silu``, ``dt_prologue`` and ``ssd_forward`` with the
            skip and the gate, on column slices of the projection's output
``conv``    ``conv1d_silu`` alone
``step``    ``ssd_step``: one token, the state carried in place; with ``views`` as a decode loop calls it, after
            ``dt_prologue`` and with z, B and C as columns of the projection's output
``host``    ``HostRunner.run``: a forward from and to pinned host memory
``model``   the drop-in ``Model``: a whole forward
"""
import math

import torch

import workloadsuite_b200 as W
from workloadsuite_b200 import mamba_model

DEVICE = "cuda"
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZES = {"f32": 4, "f16": 2, "bf16": 2}
P = 64   # head dimension of every configuration


def listed():
    return [
        # the reference's small fp32 shape: B/C per head, decays of both signs; latency and launches count
        {"name": "core_fp32_small", "kind": "core", "b": 16, "s": 128, "h": 8, "n": 16, "g": 8, "chunk": 64,
         "dtype": "f32", "decay": "normal", "dt": False, "init": False, "final": False},
        # prefill of a small model's layer: fewer sequences than SMs
        {"name": "core_130m", "kind": "core", "b": 8, "s": 2048, "h": 24, "n": 128, "g": 1, "chunk": 256,
         "dtype": "bf16", "decay": "mamba", "dt": False, "init": False, "final": False},
        # prefill of a large model's layer: the benchmark's default workload
        {"name": "core_2p7b", "kind": "core", "b": 4, "s": 8192, "h": 80, "n": 128, "g": 1, "chunk": 256,
         "dtype": "bf16", "decay": "mamba", "dt": False, "init": False, "final": False},
        # one document of 128K tokens
        {"name": "core_128k", "kind": "core", "b": 1, "s": 131072, "h": 32, "n": 128, "g": 1, "chunk": 256,
         "dtype": "bf16", "decay": "mamba", "dt": False, "init": False, "final": False},
        # many short continuations with grouped B/C and carried states, in and out
        {"name": "core_short_seqs", "kind": "core", "b": 256, "s": 512, "h": 48, "n": 64, "g": 8, "chunk": 128,
         "dtype": "bf16", "decay": "mamba", "dt": False, "init": True, "final": True},
        # a pair of prompts of no round length, whose final state starts a decode loop
        {"name": "core_ragged_prefill", "kind": "core", "b": 2, "s": 3001, "h": 80, "n": 128, "g": 1, "chunk": 1,
         "dtype": "bf16", "decay": "mamba", "dt": True, "init": False, "final": True},
        # the 1.3B layer between its projections
        {"name": "mixer_1p3b", "kind": "mixer", "b": 8, "s": 2048, "h": 128, "n": 128, "g": 8, "chunk": 64,
         "dtype": "f16"},
        # the producer of the core's X at the large model's width
        {"name": "conv_2p7b", "kind": "conv", "b": 4, "s": 8192, "h": 80, "taps": 4, "dtype": "bf16"},
        # one token of one sequence, small model: the smallest call there is
        {"name": "step_130m", "kind": "step", "b": 1, "h": 24, "n": 128, "g": 1, "dtype": "bf16", "views": False},
        # one token of a batch in a decode loop over the 1.3B layer
        {"name": "decode_1p3b", "kind": "step", "b": 8, "h": 128, "n": 128, "g": 8, "dtype": "f16", "views": True},
        # end to end over PCIe
        {"name": "host_130m", "kind": "host", "b": 8, "s": 2048, "h": 24, "n": 128, "g": 1, "chunk": 256,
         "dtype": "bf16"},
        # the whole 24-layer model at its production batch
        {"name": "model_1p3b", "kind": "model", "b": 8, "s": 2048, "d_model": 2048, "layers": 24, "n": 128, "g": 8,
         "chunk": 64},
    ]


def _log(rng, low, high):
    """A whole number, spread evenly over the logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _chunk(s):
    """The longest block length up to 256, a power of two, that divides the sequence."""
    return math.gcd(s, 256)


def _heads(rng, low=2):
    """Heads and B/C groups: ordinary counts and odd ones."""
    h = rng.choice([k for k in (2, 8, 15, 24, 32, 48, 64, 80, 112, 128) if k >= low])
    return h, rng.choice([g for g in (1, 1, 2, 8) if h % g == 0])


def _length(rng, low, high):
    """A sequence length: half of them whole tiles of 128 tokens, half as they come."""
    s = _log(rng, low, high)
    return max(128, s // 128 * 128) if rng.random() < 0.5 and s >= 96 else s


def draw(rng):
    kind = rng.choice(["core"] * 5 + ["mixer", "mixer", "conv", "step", "step", "host", "model"])
    if kind == "core":
        if rng.random() < 0.15:
            h, g = _heads(rng)
            return {"kind": "core", "b": _log(rng, 1, 32), "s": rng.choice([64, 128]), "h": min(h, 32) if g == 1 else h,
                    "n": rng.choice([16, 64, 128]), "g": g, "chunk": 64, "dtype": "f32",
                    "decay": rng.choice(["normal", "mamba"]), "dt": rng.random() < 0.3, "init": rng.random() < 0.3,
                    "final": rng.random() < 0.3}
        h, g = _heads(rng)
        s = _length(rng, 17, 131072)
        most = 256 * 512 * 48 // (s * h)      # no more than the many short sequences hold
        b = _log(rng, 1, max(1, min(256, most)))
        return {"kind": "core", "b": b, "s": s, "h": h, "n": rng.choice([64, 128, 128]), "g": g, "chunk": _chunk(s),
                "dtype": rng.choice(["bf16", "bf16", "f16"]), "decay": "mamba", "dt": rng.random() < 0.4,
                "init": rng.random() < 0.3, "final": rng.random() < 0.5}
    if kind == "mixer":
        h = rng.choice([24, 48, 80, 128])
        s = _length(rng, 64, 8192)
        return {"kind": "mixer", "b": _log(rng, 1, max(1, min(16, 16384 * 128 // (s * h)))), "s": s, "h": h,
                "n": rng.choice([64, 128, 128]), "g": rng.choice([1, 8]), "chunk": _chunk(s),
                "dtype": rng.choice(["f16", "bf16"])}
    if kind == "conv":
        h = rng.choice([24, 32, 48, 80, 128])
        s = _log(rng, 1, 16384)
        return {"kind": "conv", "b": _log(rng, 1, max(1, min(16, 4 * 8192 * 80 // (s * h)))), "s": s, "h": h,
                "taps": rng.choice([2, 3, 4, 4, 4]), "dtype": rng.choice(["bf16", "bf16", "f16", "f32"])}
    if kind == "step":
        h, g = _heads(rng, 8)
        return {"kind": "step", "b": _log(rng, 1, 64), "h": h, "n": rng.choice([64, 128, 128, 256]), "g": g,
                "dtype": rng.choice(["bf16", "f16"]), "views": rng.random() < 0.5}
    if kind == "host":
        h = rng.choice([8, 24, 48, 80])
        s = _length(rng, 128, 8192)
        return {"kind": "host", "b": _log(rng, 1, max(1, min(16, 8 * 2048 * 48 // (s * h)))), "s": s, "h": h,
                "n": rng.choice([64, 128]), "g": 1, "chunk": _chunk(s), "dtype": rng.choice(["bf16", "f16"])}
    d = rng.choice([512, 768, 1024, 2048])   # 4 d / 64 heads, as the 24-layer configuration has
    s = 64 * _log(rng, 1, 64)
    return {"kind": "model", "b": _log(rng, 1, max(1, min(8, 16384 // s))), "s": s, "d_model": d,
            "layers": _log(rng, 2, 24), "n": rng.choice([64, 128]), "g": rng.choice([1, 8]), "chunk": 64}


# ---------------------------------------------------------------------------------------------------- what is in hand

def _randn(gen, *shape, dtype=torch.float32, mean=0.0, std=1.0):
    t = torch.empty(shape, dtype=dtype, device=DEVICE).normal_(0.0, 1.0, generator=gen)
    return t if mean == 0.0 and std == 1.0 else t.mul_(std).add_(mean)


def _rates(gen, h):
    """A_log per head, uniform over [0, log 16]."""
    return torch.empty(h, device=DEVICE).uniform_(0.0, math.log(16.0), generator=gen)


def _steps(gen, *shape):
    """Discretised time steps, softplus(N(-4, 1))."""
    return torch.nn.functional.softplus(_randn(gen, *shape, mean=-4.0))


def _core_inputs(gen, case):
    b, s, h, n, g, dtype = case["b"], case["s"], case["h"], case["n"], case["g"], DTYPES[case["dtype"]]
    st = {"X": _randn(gen, b, s, h, P, dtype=dtype),
          "B": _randn(gen, b, s, g, n, dtype=dtype), "C": _randn(gen, b, s, g, n, dtype=dtype)}
    dt = _steps(gen, b, s, h)
    if case.get("dt"):
        st["dt"] = dt.to(dtype)
        dt = st["dt"].float()
    if case.get("decay", "mamba") == "normal":
        st["A"] = _randn(gen, b, s, h)
    else:
        st["A"] = -dt * torch.exp(_rates(gen, h))     # log-decay per token
    if case.get("init"):
        st["init"] = _randn(gen, b, h, n, P, std=0.1)
    return st


def _projection(gen, tokens, h, gn, dtype):
    """An input projection's output rows (z, x, B, C and dt side by side), dt around the layer's operating point."""
    return _randn(gen, *tokens, 2 * h * P + 2 * gn + h, dtype=dtype)


def _layer_weights(gen, h, dtype, taps=4):
    d = h * P
    return {"weight": _randn(gen, d, 1, taps, dtype=dtype, std=0.3), "bias": _randn(gen, d, dtype=dtype, std=0.1),
            "A_log": _rates(gen, h), "D": _randn(gen, h, dtype=dtype, mean=1.0, std=0.1),
            "dt_bias": _randn(gen, h, dtype=dtype, mean=-4.0, std=0.3)}


def prepare(case, seed):
    gen = torch.Generator(DEVICE).manual_seed(int(seed))
    kind, b = case["kind"], case["b"]
    st = {"case": case}
    if kind == "core":
        st.update(_core_inputs(gen, case))
    elif kind == "mixer":
        dtype, h = DTYPES[case["dtype"]], case["h"]
        st["proj"] = _projection(gen, (b, case["s"]), h, case["g"] * case["n"], dtype)
        st.update(_layer_weights(gen, h, dtype))
    elif kind == "conv":
        dtype, d = DTYPES[case["dtype"]], case["h"] * P
        st["proj"] = _randn(gen, b, case["s"], 2 * d, dtype=dtype)
        st.update(_layer_weights(gen, case["h"], dtype, case["taps"]))
    elif kind == "step":
        dtype, h, n, g = DTYPES[case["dtype"]], case["h"], case["n"], case["g"]
        st["x"] = _randn(gen, b, h, P, dtype=dtype)
        st["state"] = _randn(gen, b, h, n, P)
        st.update(_layer_weights(gen, h, dtype))
        if case["views"]:
            st["proj"] = _projection(gen, (b,), h, g * n, dtype)
        else:
            st["a"] = -_steps(gen, b, h) * torch.exp(st["A_log"])
            st["B"], st["C"] = _randn(gen, b, g, n, dtype=dtype), _randn(gen, b, g, n, dtype=dtype)
    elif kind == "host":
        inputs = _core_inputs(gen, case)
        st.update({k: torch.empty(v.shape, dtype=v.dtype, pin_memory=True).copy_(v) for k, v in inputs.items()})
        st["out"] = torch.empty(inputs["X"].shape, dtype=inputs["X"].dtype, pin_memory=True)
        st["runner"] = W.HostRunner(b, case["s"], case["h"], P, case["n"], case["g"], case["chunk"],
                                    DTYPES[case["dtype"]], device="cuda:0")
    else:
        d = case["d_model"]
        with torch.random.fork_rng(devices=[torch.cuda.current_device()]), torch.device(DEVICE):
            torch.manual_seed(int(seed))
            st["model"] = mamba_model.Model(d, case["layers"], 4 * d // P, case["n"], P, case["g"], case["chunk"]).eval()
        st["u"] = _randn(gen, b, case["s"], d, dtype=torch.float16)
    return st


# --------------------------------------------------------------------------------------------------------- one pass

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "core":
        return W.ssd_forward(st["X"], st["A"], st["B"], st["C"], case["chunk"], dt=st.get("dt"),
                             initial_states=st.get("init"), return_final_state=case["final"])
    if kind == "mixer":
        b, s, h, n, g = case["b"], case["s"], case["h"], case["n"], case["g"]
        x, z, B, C, dt = torch.split(st["proj"], [h * P, h * P, g * n, g * n, h], dim=-1)
        x = W.conv1d_silu(x, st["weight"], st["bias"]).view(b, s, h, P)
        dt, A = W.dt_prologue(dt, st["dt_bias"], st["A_log"])
        return W.ssd_forward(x, A, B.unflatten(-1, (g, n)), C.unflatten(-1, (g, n)), case["chunk"], dt=dt, D=st["D"],
                             z=z.unflatten(-1, (h, P)))
    if kind == "conv":
        return W.conv1d_silu(st["proj"][..., :case["h"] * P], st["weight"], st["bias"])
    if kind == "step":
        if not case["views"]:
            return W.ssd_step(st["x"], st["a"], st["B"], st["C"], st["state"]), st["state"]
        h, n, g = case["h"], case["n"], case["g"]
        _, z, B, C, dt = torch.split(st["proj"], [h * P, h * P, g * n, g * n, h], dim=-1)
        dt, A = W.dt_prologue(dt.unsqueeze(1), st["dt_bias"], st["A_log"])
        y = W.ssd_step(st["x"], A.squeeze(1), B.unflatten(-1, (g, n)), C.unflatten(-1, (g, n)), st["state"],
                       dt=dt.squeeze(1), D=st["D"], z=z.unflatten(-1, (h, P)))
        return y, st["state"]
    if kind == "host":
        return st["runner"].run(st["X"], st["A"], st["B"], st["C"], st["out"])
    with torch.inference_mode():
        return st["model"](st["u"])


# ------------------------------------------------------------------------------------------------- what it costs

def work(case):
    kind, b, e = case["kind"], case["b"], SIZES[case.get("dtype", "f16")]
    if kind == "step":
        h, n, g = case["h"], case["n"], case["g"]
        state = b * h * n * P
        small = e * (2 * b * h * P + 2 * b * g * n) + (e * b * (h * P + h) if case["views"] else 4 * b * h)
        return {"bytes": 2 * 4 * state + small, "flops": 5 * state}
    t, s = b * case["s"], case["s"]
    if kind == "conv":
        d = case["h"] * P
        return {"bytes": e * (2 * t * d + d * (case["taps"] + 1)), "flops": t * d * (2 * case["taps"] + 4)}
    if kind == "model":
        d, n, g, h = case["d_model"], case["n"], case["g"], 4 * case["d_model"] // P
        weights = d * (2 * h * P + 2 * g * n + h) + h * P * d
        layer = 2 * t * weights + 4 * t * h * P * n
        return {"bytes": 2 * (2 * t * d + case["layers"] * weights), "flops": case["layers"] * layer}
    h, n, g = case["h"], case["n"], case["g"]
    flops = 4 * t * h * P * n      # the recurrence: update of the state and read-out
    if kind == "mixer":
        return {"bytes": e * t * (3 * h * P + 2 * g * n + h), "flops": flops + t * h * P * 18}
    moved = t * (2 * e * h * P + 2 * e * g * n + 4 * h + (e * h if case.get("dt") else 0))
    moved += 4 * b * h * n * P * (bool(case.get("init")) + bool(case.get("final")))
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["kind"] == "model":        # fp16 through all layers
        return {"rel": 1e-2}
    return {"rel": {"f32": 1e-5, "f16": 4e-3, "bf16": 1e-2}[case["dtype"]]}
