"""The work that a user of the NVFP4 projection engine has it do, as measurable cases.

A case is a dict of plain values; `prepare` builds what a host program holds before the call (weights repacked on the
GPU, activations, work lists, scratch), `run` makes one pass through the public entry points of `qwen35x_b200.engine`
and returns the outputs whole, `work` says which bytes and operations the pass cannot do without, `tolerance` how far
another correct implementation at the same precision may be off.

Kinds of pass
  step         one decode step: the work list over every projection of `layers` layers (GemvBatch), m = 1..8 tokens
  gemv         one decode projection on its own (gemv_w4a16, or gemv_w4a16_f32 with x = "f32")
  decode_mlp   one layer's MLP block at decode: gate/up with the SiLU epilogue, then down + residual after it, one list
  prefill      one prefill projection: activation quantisation and the W4A4 GEMM, optionally with a residual
  prefill_mlp  one layer's MLP block at prefill: quantise, gate/up writing NVFP4, down + residual

Weights are N(0, 0.02) (single projections: one row in 128 scaled by 8), activations N(0, 1) with one channel in a
thousand scaled by 20, as in the per-shape report.
"""
import math

import torch

from qwen35x_b200 import engine as q

# (N, K) of the projections of one layer, from the benchmark: mixer input and output, MLP gate+up, MLP down
LAYER_0P8B = [(4096, 1024), (1024, 2048), (7168, 1024), (1024, 3584)]
LAYER_4B = [(18432, 2560), (2560, 9216), (10240, 2560), (2560, 4096)]

MAX_STEP_WEIGHTS = 3_500_000_000        # weights of one decode step, the 4B-class step's 3.45e9 rounded up
MAX_PREFILL_MACS = 4096 * 18432 * 2560  # the largest listed projection; the MLP block is 1.5 times this


def listed():
    return [
        # The smallest call there is: one projection of the small model, one token, nothing to batch it with.
        {"name": "gemv_3584x1024_m1", "kind": "gemv", "n": 3584, "k": 1024, "m": 1, "x": "bf16"},
        # A wide single projection (an output head's width) for a few sequences at once.
        {"name": "gemv_32768x2560_m3", "kind": "gemv", "n": 32768, "k": 2560, "m": 3, "x": "bf16"},
        # The headline: every projection of a decode step of the small model, one token.
        {"name": "step_0p8b_m1", "kind": "step", "hidden": 1024, "mix_in": 4096, "mix_out": 2048, "inter": 3584, "layers": 24, "m": 1},
        # The same step with the largest decode batch.
        {"name": "step_0p8b_m8", "kind": "step", "hidden": 1024, "mix_in": 4096, "mix_out": 2048, "inter": 3584, "layers": 24, "m": 8},
        # Decode step of the larger model, one token: the largest weight stream.
        {"name": "step_4b_m1", "kind": "step", "hidden": 2560, "mix_in": 10240, "mix_out": 4096, "inter": 9216, "layers": 32, "m": 1},
        # ... and with a batch of four.
        {"name": "step_4b_m4", "kind": "step", "hidden": 2560, "mix_in": 10240, "mix_out": 4096, "inter": 9216, "layers": 32, "m": 4},
        # One layer's MLP block at decode, as a host runs it between two attention layers: dependent items.
        {"name": "decode_mlp_4b_m2", "kind": "decode_mlp", "hidden": 2560, "inter": 9216, "m": 2},
        # A short prompt or a block of drafted tokens.
        {"name": "prefill_9216x2560_m16", "kind": "prefill", "n": 9216, "k": 2560, "m": 16, "x": "bf16", "given_scale": False, "residual": False},
        # A prompt of about a hundred tokens through a down projection, residual added in the epilogue.
        {"name": "prefill_2560x9216_m100", "kind": "prefill", "n": 2560, "k": 9216, "m": 100, "x": "bf16", "given_scale": False, "residual": True},
        # A ragged chunk of fp32 activations with the checkpoint's stored input scale.
        {"name": "prefill_3584x1024_m1000_f32", "kind": "prefill", "n": 3584, "k": 1024, "m": 1000, "x": "f32", "given_scale": True, "residual": False},
        # The benchmark's prefill shape: gate+up of the larger model over a full chunk.
        {"name": "prefill_18432x2560_m4096", "kind": "prefill", "n": 18432, "k": 2560, "m": 4096, "x": "bf16", "given_scale": False, "residual": False},
        # The whole prefill MLP block of the larger model over a full chunk.
        {"name": "prefill_mlp_4b_m4096", "kind": "prefill_mlp", "hidden": 2560, "inter": 9216, "m": 4096},
    ]


def _log_int(rng, lo, hi, multiple=1):
    """An integer spread over the logarithm of [lo, hi], rounded to a multiple."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / multiple)) * multiple))


def draw(rng):
    kind = rng.choice(["step", "gemv", "decode_mlp", "prefill", "prefill", "prefill_mlp"])
    if kind == "step":
        # the work list takes K in multiples of 256; rows are free
        while True:
            c = {"kind": kind, "hidden": _log_int(rng, 512, 4096, 256), "mix_in": _log_int(rng, 1000, 10240, 8),
                 "mix_out": _log_int(rng, 512, 4096, 256), "inter": _log_int(rng, 1024, 9216, 256),
                 "layers": _log_int(rng, 2, 32), "m": rng.randint(1, 8)}
            if c["layers"] * sum(n * k for n, k in _layer(c)) <= MAX_STEP_WEIGHTS:
                return c
    if kind == "gemv":
        x = rng.choice(["bf16", "bf16", "bf16", "f32"])
        return {"kind": kind, "n": _log_int(rng, 100, 32768), "k": _log_int(rng, 256, 9216, rng.choice([16, 32, 256])),
                "m": 1 if x == "f32" else rng.randint(1, 8), "x": x}
    if kind == "decode_mlp":
        return {"kind": kind, "hidden": _log_int(rng, 512, 4096, 256), "inter": _log_int(rng, 1024, 9216, 256), "m": rng.randint(1, 8)}
    if kind == "prefill":
        while True:
            c = {"kind": kind, "n": _log_int(rng, 100, 32768), "k": _log_int(rng, 512, 9216, 64), "m": _log_int(rng, 1, 4096),
                 "x": rng.choice(["bf16", "bf16", "f32"]), "given_scale": rng.random() < 0.4, "residual": rng.random() < 0.3}
            if c["m"] * c["n"] * c["k"] <= MAX_PREFILL_MACS:
                return c
    while True:
        c = {"kind": kind, "hidden": _log_int(rng, 512, 4096, 64), "inter": _log_int(rng, 1024, 9216, 64), "m": _log_int(rng, 16, 4096)}
        if 3 * c["m"] * c["hidden"] * c["inter"] <= 3 * MAX_PREFILL_MACS // 2:
            return c


def _layer(c):
    """(N, K) of one layer's projections of a decode step."""
    return [(c["mix_in"], c["hidden"]), (c["hidden"], c["mix_out"]), (2 * c["inter"], c["hidden"]), (c["hidden"], c["inter"])]


def _weight_bytes(n, k):
    return n * k // 2 + n * k // 16


# ---- what the host program holds before the call ---------------------------------------------------------------


def _fp4(gen, n, k, outlier_rows):
    w = torch.empty((n, k), device="cuda").normal_(0.0, 0.02, generator=gen)
    if outlier_rows:
        w[int(torch.randint(0, 128, (1,), generator=gen, device="cuda")):: 128] *= 8.0
    return q.quantize_weight(w)


def _weight(gen, n, k, outlier_rows=False):
    codes, scales, s2 = _fp4(gen, n, k, outlier_rows)
    return q.Nvfp4Weight.from_device(codes, scales, s2)


def _gate_up_weight(gen, inter, hidden):
    args = []
    for _ in range(2):
        codes, scales, s2 = _fp4(gen, inter, hidden, False)
        args += [codes.cpu().numpy(), scales.cpu().numpy(), s2]
    return q.Nvfp4Weight.gate_up_from_host(*args)


def _activations(gen, m, k, dtype=torch.bfloat16):
    x = torch.randn((m, k), generator=gen, device="cuda")
    x[:, int(torch.randint(0, 1000, (1,), generator=gen, device="cuda")) % k:: 1000] *= 20.0
    return x.to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, m = case["kind"], case["m"]
    if kind == "step":
        shapes = _layer(case) * case["layers"]
        y = torch.zeros(m * sum(n for n, _ in shapes), dtype=torch.bfloat16, device="cuda")
        items, at = [], 0
        for n, k in shapes:
            items.append((_weight(gen, n, k), _activations(gen, m, k), y[at: at + m * n].view(m, n)))
            at += m * n
        return {"kind": kind, "list": q.GemvBatch(items, m), "y": y}
    if kind == "gemv":
        dtype = torch.float32 if case["x"] == "f32" else torch.bfloat16
        x = _activations(gen, m, case["k"], dtype)
        return {"kind": kind, "w": _weight(gen, case["n"], case["k"], True), "x": x[0].contiguous() if case["x"] == "f32" else x,
                "f32": case["x"] == "f32"}
    hidden, inter = case.get("hidden"), case.get("inter")
    if kind == "decode_mlp":
        gate_up, down = _gate_up_weight(gen, inter, hidden), _weight(gen, hidden, inter)
        x, residual = _activations(gen, m, hidden), _activations(gen, m, hidden)
        h = torch.zeros((m, inter), dtype=torch.bfloat16, device="cuda")
        y = torch.zeros((m, hidden), dtype=torch.bfloat16, device="cuda")
        return {"kind": kind, "list": q.GemvBatch([(gate_up, x, h), (down, h, y, residual, 0)], m), "h": h, "y": y}
    if kind == "prefill":
        n, k = case["n"], case["k"]
        x = _activations(gen, m, k, torch.float32 if case["x"] == "f32" else torch.bfloat16)
        return {"kind": kind, "w": _weight(gen, n, k, True), "x": x, "scratch": q.act_scratch(m, k, x.device),
                # a stored input scale: the amax of a calibration run, here 20 * 4.5 sigma
                "scale": 90.0 / 2688.0 if case["given_scale"] else 0.0,
                "residual": torch.randn((m, n), generator=gen, device="cuda").to(torch.bfloat16) if case["residual"] else None}
    x = _activations(gen, m, hidden)
    # a stored input scale of the down projection: gate and up are N(0, sigma), their SiLU product stays below 20 sigma^2
    sigma2 = 0.02 ** 2 * hidden * 1.4
    return {"kind": kind, "m": m, "gate_up": _gate_up_weight(gen, inter, hidden), "down": _weight(gen, hidden, inter), "x": x,
            "residual": torch.randn((m, hidden), generator=gen, device="cuda").to(torch.bfloat16),
            "h_scale": torch.full((1,), 20.0 * sigma2 / 2688.0, device="cuda"),
            "x_scratch": q.act_scratch(m, hidden, x.device), "h_scratch": q.act_scratch(m, inter, x.device)}


# ---- one pass ---------------------------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["list"].run()
        return state["y"]
    if kind == "gemv":
        return (q.gemv_w4a16_f32 if state["f32"] else q.gemv_w4a16)(state["w"], state["x"])
    if kind == "decode_mlp":
        state["list"].run()
        return {"h": state["h"], "y": state["y"]}
    if kind == "prefill":
        return q.project_prefill(state["w"], state["x"], scratch=state["scratch"], global_scale=state["scale"], residual=state["residual"])
    m = state["m"]
    codes, scales, g = q.quantize_activations(state["x"], 0.0, state["x_scratch"])
    h_codes, h_scales, h_g = q.gemm_w4a4_gate_up_quant(state["gate_up"], codes, scales, g, m, state["h_scale"], state["h_scratch"])
    return q.gemm_w4a4(state["down"], h_codes, h_scales, h_g, m, residual=state["residual"])


# ---- what a pass cannot do without, and how close results have to be ---------------------------------------------


def work(case):
    kind, m = case["kind"], case["m"]
    if kind == "step":
        shapes = _layer(case) * case["layers"]
        return {"bytes": sum(_weight_bytes(n, k) + 2 * m * (n + k) for n, k in shapes), "flops": 2 * m * sum(n * k for n, k in shapes)}
    if kind in ("decode_mlp", "prefill_mlp"):
        hidden, inter = case["hidden"], case["inter"]
        # x and the residual in, the block's output out; decode also hands out the intermediate activation
        act = 2 * m * 3 * hidden + (2 * m * inter if kind == "decode_mlp" else 0)
        return {"bytes": 3 * _weight_bytes(inter, hidden) + act, "flops": 6 * m * hidden * inter}
    n, k = case["n"], case["k"]
    x_bytes = 4 if case["x"] == "f32" else 2
    y_bytes = 4 if kind == "gemv" and case["x"] == "f32" else 2
    return {"bytes": _weight_bytes(n, k) + m * k * x_bytes + m * n * (y_bytes + (2 if case.get("residual") else 0)), "flops": 2 * m * n * k}


def tolerance(case):
    # Measured against the same pass in 64 bits rounded to the output type at the same points: 2e-7 for fp32 output;
    # for BF16 output up to 2e-5 for one projection (a few sums land on the other side of a rounding boundary), 7e-5
    # for the prefill block and 3.4e-4 for the decode block, whose second projection reads the first one's rounded
    # output; the largest single difference is one BF16 step (0.008), or in the prefill block one FP4 code of the
    # intermediate activation (0.011).  A result of few values shows one flipped rounding more than these do.
    if case["kind"] == "gemv" and case["x"] == "f32":
        return {"rel": 1e-6}
    return {"rel": 1e-3, "max": 0.04}


# ---- the same results in 64 bits ---------------------------------------------------------------------------------

E2M1_LEVELS = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]
UE4M3_LEVELS = [(b & 7) * 2.0 ** -9 if b < 8 else (8 + (b & 7)) * 2.0 ** ((b >> 3) - 10) for b in range(0x7f)]


def _nearest(v, levels):
    """The nearest of the ascending levels, the lower one of a tie."""
    table = torch.tensor(levels, dtype=torch.float64, device=v.device)
    return table[torch.bucketize(v.double(), (table[1:] + table[:-1]) / 2)]


def _nvfp4(x, g=None):
    """What NVFP4 codes of x stand for, in 64 bits; the quantiser's own steps are 32-bit by contract (scale of the tensor
    amax / 2688, scale of a block amax / 6 over that as unsigned E4M3, ties down).  Divisors are tensors: a division by a
    Python number would become a multiplication by its reciprocal."""
    word = lambda v: torch.tensor(v, dtype=torch.float32, device=x.device)  # noqa: E731
    x = x.float()
    g = x.abs().max() / word(2688.0) if g is None else word(g)
    out = torch.empty(x.shape, dtype=torch.float64, device=x.device)
    for at in range(0, x.shape[0], 2048):
        b = x[at: at + 2048].view(-1, x.shape[1] // 16, 16)
        t = b.abs().amax(dim=2, keepdim=True) / word(6.0)
        scale = _nearest((t / g).clamp_min(1e-8), UE4M3_LEVELS).float()
        q = b / (scale.clamp_min(1e-8) * g)
        out[at: at + 2048] = (_nearest(q.abs(), E2M1_LEVELS).copysign(q.double()) * (scale.double() * g.double())).view(-1, x.shape[1])
    return out


def _exact_weight(gen, n, k, outlier_rows=False):
    w = torch.empty((n, k), device="cuda").normal_(0.0, 0.02, generator=gen)
    if outlier_rows:
        w[int(torch.randint(0, 128, (1,), generator=gen, device="cuda")):: 128] *= 8.0
    return _nvfp4(w)


def _silu_product(x, gate, up):
    a = x @ gate.T
    return a / (1.0 + torch.exp(-a)) * (x @ up.T)


def exact(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, m = case["kind"], case["m"]
    if kind == "step":
        parts = []
        for n, k in _layer(case) * case["layers"]:
            w = _exact_weight(gen, n, k)
            parts.append((_activations(gen, m, k).double() @ w.T).reshape(-1))
        return torch.cat(parts)
    if kind == "gemv":
        dtype = torch.float32 if case["x"] == "f32" else torch.bfloat16
        x = _activations(gen, m, case["k"], dtype).double()
        y = x @ _exact_weight(gen, case["n"], case["k"], True).T
        return y[0] if case["x"] == "f32" else y
    hidden, inter = case.get("hidden"), case.get("inter")
    if kind == "decode_mlp":
        gate, up, down = (_exact_weight(gen, *shape) for shape in ((inter, hidden), (inter, hidden), (hidden, inter)))
        x, residual = _activations(gen, m, hidden).double(), _activations(gen, m, hidden).double()
        h = _silu_product(x, gate, up)
        # the intermediate activation is handed out, and read by the second projection, as BF16
        return {"h": h, "y": h.to(torch.bfloat16).double() @ down.T + residual}
    if kind == "prefill":
        n, k = case["n"], case["k"]
        x = _activations(gen, m, k, torch.float32 if case["x"] == "f32" else torch.bfloat16)
        y = _nvfp4(x, 90.0 / 2688.0 if case["given_scale"] else None) @ _exact_weight(gen, n, k, True).T
        return y + torch.randn((m, n), generator=gen, device="cuda").to(torch.bfloat16).double() if case["residual"] else y
    x = _activations(gen, m, hidden)
    gate, up, down = (_exact_weight(gen, *shape) for shape in ((inter, hidden), (inter, hidden), (hidden, inter)))
    residual = torch.randn((m, hidden), generator=gen, device="cuda").to(torch.bfloat16).double()
    h = _silu_product(_nvfp4(x), gate, up)
    # the epilogue rounds the intermediate activation to BF16 before it quantises it
    return _nvfp4(h.to(torch.bfloat16), 20.0 * (0.02 ** 2 * hidden * 1.4) / 2688.0) @ down.T + residual
