"""Performance cases of the state-space path: what programs built on this package have it do, through the calls they
make.

  prefill    a byte LM (24 blocks, d_model 768, bf16) reads a batch of prompts of one length and keeps the decode state
  prompts    the same model working through a queue: host buffers in and out, one prompt after another, each of its own
             length
  generate   the same model: prefill of a short prompt, then single-token decode steps
  block      one Mamba block on tensors, with the state a decode step continues from
  module     MambaBlock as a module (host array in, host array out), f32: the reference's own way of using it
  scan       the fused selective scan by itself
  s4         the diagonal S4 recurrence by itself
  s4_ssm     S4Block::forward_ssm, the recurrence the reference computes, as a module

A case is a dict of plain values; listed() holds the fixed ones and draw() gives more of the same ranges."""
from __future__ import annotations

import math

import numpy as np
import torch

from helixml_b200 import nn, ops

LAYERS, WIDTH, STATE, TAPS, VOCAB = 24, 768, 16, 4, 256   # the byte LM of bench.py's default workload
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}

_lm = None


def byte_lm():
    """The model a serving program loads once and keeps: random-init weights under a fixed seed (drawing them on the
    host takes seconds)."""
    global _lm
    if _lm is None:
        nn.manual_seed(3)
        _lm = nn.ByteLM(LAYERS, WIDTH, STATE, TAPS, 2)
    return _lm


def listed():
    return [
        # a full batch of long prompts: bench.py's default workload on one GPU
        {"name": "prefill 32x2048", "kind": "prefill", "batch": 32, "seq_len": 2048},
        # what one of eight GPUs gets of that batch; also a small serving batch
        {"name": "prefill 4x2048", "kind": "prefill", "batch": 4, "seq_len": 2048},
        # a queue of requests worked through one by one, prompts of 60 to 731 bytes
        {"name": "prompts 12x60..731", "kind": "prompts", "count": 12, "longest": 731},
        # one user's completion: latency of every single step
        {"name": "generate 1", "kind": "generate", "batch": 1, "prompt": 100, "steps": 32},
        # a batch of completions
        {"name": "generate 32", "kind": "generate", "batch": 32, "prompt": 128, "steps": 64},
        # one block of a wider model with trained decays (no closed form over the states), ragged length
        {"name": "block bf16 6x1500x1024", "kind": "block", "batch": 6, "seq_len": 1500, "d_model": 1024, "dtype": "bf16",
         "trained": True},
        # the smallest call: the parity configuration [100, 64] with d_state 16
        {"name": "module 100x64", "kind": "module", "batch": 1, "seq_len": 100, "d_model": 64, "d_state": 16},
        # the reference's own criterion shape, MambaBlock::new(512, 64, 4, 2) on [256, 512]
        {"name": "module 256x512 N64", "kind": "module", "batch": 1, "seq_len": 256, "d_model": 512, "d_state": 64},
        # bench.py's stand-alone scan, planned once as bench.py does
        {"name": "scan bf16 16x4096x1536", "kind": "scan", "batch": 16, "seq_len": 4096, "d_inner": 1536, "dtype": "bf16",
         "trained": False, "planned": True},
        # f32, trained decays, a ragged length, every argument at its default
        {"name": "scan f32 3x1111x640", "kind": "scan", "batch": 3, "seq_len": 1111, "d_inner": 640, "dtype": "f32",
         "trained": True, "planned": False},
        # diagonal S4 at bench.py's shape
        {"name": "s4 8x2048x256", "kind": "s4", "batch": 8, "seq_len": 2048, "d_model": 256, "d_state": 64},
        # the reference's literal recurrence, [d_model, L] in, [L, d_model] out
        {"name": "s4_ssm 256x2048", "kind": "s4_ssm", "d_model": 256, "seq_len": 2048, "d_state": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prefill", "prefill", "prompts", "generate", "generate", "block", "block", "module", "scan", "scan",
                       "s4", "s4_ssm"])
    if kind == "prefill":
        batch = _log_int(rng, 1, 32)
        return {"kind": kind, "batch": batch, "seq_len": _log_int(rng, 16, 2048)}
    if kind == "prompts":
        return {"kind": kind, "count": rng.randint(4, 12), "longest": _log_int(rng, 64, 731)}
    if kind == "generate":
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "prompt": _log_int(rng, 8, 400), "steps": rng.randint(8, 64)}
    if kind == "block":
        seq_len = _log_int(rng, 32, 4096)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, 32768 // seq_len)), "seq_len": seq_len,
                "d_model": 64 * rng.randint(2, 20), "dtype": rng.choice(["bf16", "bf16", "f32"]), "trained": rng.random() < 0.5}
    if kind == "module":
        return {"kind": kind, "batch": rng.randint(1, 4), "seq_len": _log_int(rng, 32, 512), "d_model": 32 * rng.randint(2, 16),
                "d_state": rng.choice([16, 16, 64])}
    if kind == "scan":
        seq_len = _log_int(rng, 64, 8192)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, 65536 // seq_len)), "seq_len": seq_len,
                "d_inner": 32 * rng.randint(4, 64), "dtype": rng.choice(["bf16", "bf16", "f32"]), "trained": rng.random() < 0.5,
                "planned": rng.random() < 0.5}
    if kind == "s4":
        return {"kind": kind, "batch": _log_int(rng, 1, 16), "seq_len": _log_int(rng, 64, 4096), "d_model": 32 * rng.randint(2, 16),
                "d_state": rng.choice([16, 64, 64])}
    return {"kind": kind, "d_model": 32 * rng.randint(2, 16), "seq_len": _log_int(rng, 64, 4096), "d_state": rng.choice([16, 64])}


def _lengths(case):
    """Prompt lengths of a `prompts` case: spread over (0, longest], in no sorted order, odd and even."""
    n, top = case["count"], case["longest"]
    order = sorted(range(n), key=lambda i: (i * 7919 + 3) % (2 * n + 1))
    return [max(1, top * (i + 1) // n - (i * 5) % 3 * (i + 1 < n)) for i in order]


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _decays(rows, d_state, trained, g):
    """A = -(n + 1), the initial value of every channel; `trained` scales each entry by its own factor around 1."""
    a = -torch.arange(1, d_state + 1, device="cuda", dtype=torch.float32).repeat(rows, 1)
    return a * torch.exp(0.2 * torch.randn(rows, d_state, device="cuda", generator=g)) if trained else a


def _dt_bias(rows, g):
    """softplus^-1 of a step that is log-uniform in [1e-3, 1e-1]."""
    dt = torch.exp(math.log(1e-3) + torch.rand(rows, device="cuda", generator=g) * math.log(100.0))
    return dt + torch.log(-torch.expm1(-dt))


def _tokens(shape, seed):
    return torch.randint(0, VOCAB, shape, device="cuda", dtype=torch.uint8, generator=_gen(seed))


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    s = {"case": case}
    if kind == "prefill":
        B, L = case["batch"], case["seq_len"]
        s.update(lm=byte_lm(), tokens=_tokens((B, L), seed), logits=torch.empty(B, L, VOCAB, device="cuda", dtype=torch.bfloat16))
    elif kind == "prompts":
        rng = np.random.default_rng(seed)
        s.update(lm=byte_lm(), tokens=[], logits=[])
        for n in _lengths(case):
            s["tokens"].append(torch.from_numpy(rng.integers(0, VOCAB, (1, n), dtype=np.uint8)).pin_memory())
            s["logits"].append(torch.empty(1, n, VOCAB, dtype=torch.bfloat16).pin_memory())
    elif kind == "generate":
        B, L, n = case["batch"], case["prompt"], case["steps"]
        # the continuation is given (as when scoring one), so every step's input is the same for any arithmetic
        s.update(lm=byte_lm(), tokens=_tokens((B, L), seed), next=_tokens((n, B), seed + 1),
                 logits=torch.empty(B, L, VOCAB, device="cuda", dtype=torch.bfloat16),
                 step_logits=torch.empty(n, B, VOCAB, device="cuda", dtype=torch.bfloat16))
    elif kind == "block":
        B, L, M, dt = case["batch"], case["seq_len"], case["d_model"], DTYPES[case["dtype"]]
        E, R = 2 * M, (M + 15) // 16
        w = lambda out, inner: (torch.randn(out, inner, device="cuda", generator=g) * inner ** -0.5).to(dt)
        s.update(x=torch.randn(B, L, M, device="cuda", generator=g).to(dt), h=torch.empty(B, E, STATE, device="cuda"),
                 conv_state=torch.empty(B, 3, E, device="cuda", dtype=dt))
        s["w"] = {"W_in": w(2 * E, M), "W_x": w(R + 2 * STATE, E), "W_dt": w(E, R), "W_out": w(M, E),
                  "conv_w": torch.rand(E, TAPS, device="cuda", generator=g) - 0.5,
                  "conv_b": torch.rand(E, device="cuda", generator=g) - 0.5, "b_dt": _dt_bias(E, g),
                  "A": _decays(E, STATE, case["trained"], g), "D": torch.ones(E, device="cuda")}
    elif kind == "module":
        nn.manual_seed(seed)
        s["module"] = nn.MambaBlock(case["d_model"], case["d_state"], TAPS, 2)
        rng = np.random.default_rng(seed)
        s["x"] = rng.uniform(-1, 1, (case["batch"], case["seq_len"], case["d_model"])).astype(np.float32)
    elif kind == "scan":
        B, L, D, dt = case["batch"], case["seq_len"], case["d_inner"], DTYPES[case["dtype"]]
        rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g).to(dt)
        s.update(x=rnd(B, L, D), z=rnd(B, L, D), B=rnd(B, L, STATE), C=rnd(B, L, STATE),
                 dt=(torch.rand(B, L, D, device="cuda", generator=g) * 3 - 4).to(dt), A=_decays(D, STATE, case["trained"], g),
                 D=torch.ones(D, device="cuda"), conv_w=torch.rand(D, TAPS, device="cuda", generator=g) - 0.5, plan={})
        if case["planned"]:
            splits = ops.suggest_splits(B, L, D, dt, a_geometric=not case["trained"])
            s["plan"] = {"a_geometric": ops.check_geometric(s["A"]), "seq_splits": splits, "out": torch.empty_like(s["x"])}
            if splits > 1:
                n = ops.scan_workspace_bytes(B, L, D, dt, splits)
                s["plan"]["workspace"] = torch.empty(n, dtype=torch.uint8, device="cuda")
    elif kind == "s4":
        B, L, D, N = case["batch"], case["seq_len"], case["d_model"], case["d_state"]
        s.update(u=torch.randn(B, L, D, device="cuda", generator=g),
                 A=-0.5 * torch.arange(1, N + 1, device="cuda", dtype=torch.float32).repeat(D, 1),
                 B=torch.randn(D, N, device="cuda", generator=g) * N ** -0.5,
                 C=torch.randn(D, N, device="cuda", generator=g) * N ** -0.5,
                 delta=torch.exp(math.log(1e-3) + torch.rand(D, device="cuda", generator=g) * math.log(100.0)),
                 D=torch.ones(D, device="cuda"))
    else:
        nn.manual_seed(seed)
        s["module"] = nn.S4Block(case["d_model"], case["d_state"])
        s["u"] = np.random.default_rng(seed).standard_normal((case["d_model"], case["seq_len"]), dtype=np.float32)
    return s


# ------------------------------------------------------------------------------------------------ the calls
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "prefill":
        s["lm"].prefill_device(s["tokens"].data_ptr(), s["logits"].data_ptr(), case["batch"], case["seq_len"])
        return s["logits"]
    if kind == "prompts":
        for tok, out in zip(s["tokens"], s["logits"]):
            s["lm"].forward_host(tok.data_ptr(), out.data_ptr(), 1, tok.shape[1])
        return s["logits"]
    if kind == "generate":
        B = case["batch"]
        s["lm"].prefill_device(s["tokens"].data_ptr(), s["logits"].data_ptr(), B, case["prompt"])
        for i in range(case["steps"]):
            s["lm"].decode_step_device(s["next"][i].data_ptr(), s["step_logits"][i].data_ptr(), B)
        return s["logits"], s["step_logits"]
    if kind == "block":
        y = ops.mamba_block(s["x"], s["w"], STATE, TAPS, h_last=s["h"], conv_state=s["conv_state"])
        return y, s["h"], s["conv_state"]
    if kind == "module":
        return s["module"].forward(nn.Tensor.from_numpy(s["x"])).numpy()
    if kind == "scan":
        return ops.selective_scan(s["x"], s["dt"], s["A"], s["B"], s["C"], D=s["D"], z=s["z"], conv_w=s["conv_w"], **s["plan"])
    if kind == "s4":
        return ops.s4_diag(s["u"], s["A"], s["B"], s["C"], s["delta"], s["D"])
    return s["module"].forward_ssm(nn.Tensor.from_numpy(s["u"])).numpy()


# ------------------------------------------------------------------------------------------------ what they need
def _scan_flops(points, d_state):
    # per state: decay power, input product, state update (2), output product and sum (2); about 20 point-wise
    return points * (6 * d_state + 20)


def _block_flops(tokens, M, N):
    E, R = 2 * M, (M + 15) // 16
    return 2 * tokens * (2 * E * M + (R + 2 * N) * E + E * R + M * E) + 2 * tokens * E * TAPS + _scan_flops(tokens * E, N)


def _block_weight_bytes(M, N, es):
    E, R = 2 * M, (M + 15) // 16
    return es * (2 * E * M + (R + 2 * N) * E + E * R + M * E) + 4 * (E * TAPS + 3 * E + E * N)


def _lm_work(tokens, passes, states):
    """`passes` readings of the weights, `tokens` bytes in and rows of logits out, `states` decode states written."""
    weights = LAYERS * (_block_weight_bytes(WIDTH, STATE, 2) + 4 * WIDTH) + 2 * VOCAB * WIDTH
    state = LAYERS * 2 * WIDTH * (4 * STATE + 2 * 3)
    return {"bytes": passes * weights + tokens * (1 + 2 * VOCAB) + states * state,
            "flops": LAYERS * _block_flops(tokens, WIDTH, STATE) + 2 * tokens * WIDTH * VOCAB}


def work(case):
    kind = case["kind"]
    if kind == "prefill":
        return _lm_work(case["batch"] * case["seq_len"], 1, case["batch"])
    if kind == "prompts":
        return _lm_work(sum(_lengths(case)), case["count"], 0)
    if kind == "generate":
        # a step reads and writes the state of every sequence
        return _lm_work(case["batch"] * (case["prompt"] + case["steps"]), 1 + case["steps"], case["batch"] * (1 + 2 * case["steps"]))
    if kind == "block":
        es, M = DTYPES[case["dtype"]].itemsize, case["d_model"]
        T = case["batch"] * case["seq_len"]
        return {"bytes": 2 * T * M * es + _block_weight_bytes(M, STATE, es) + case["batch"] * 2 * M * (4 * STATE + 3 * es),
                "flops": _block_flops(T, M, STATE)}
    if kind == "module":
        T, M, N = case["batch"] * case["seq_len"], case["d_model"], case["d_state"]
        return {"bytes": 2 * T * M * 4 + _block_weight_bytes(M, N, 4), "flops": _block_flops(T, M, N)}
    if kind == "scan":
        es, T, D = DTYPES[case["dtype"]].itemsize, case["batch"] * case["seq_len"], case["d_inner"]
        return {"bytes": es * (4 * T * D + 2 * T * STATE) + 4 * D * (STATE + TAPS + 1), "flops": _scan_flops(T * D, STATE) + 2 * T * D * TAPS}
    if kind == "s4":
        T, D, N = case["batch"] * case["seq_len"], case["d_model"], case["d_state"]
        return {"bytes": 8 * T * D + 4 * D * (3 * N + 2), "flops": 4 * T * D * N}
    L, M, N = case["seq_len"], case["d_model"], case["d_state"]
    return {"bytes": 8 * L * M + 4 * (2 * N * M + 2 * N + M), "flops": 4 * L * M * N + 4 * L * N}


def tolerance(case):
    if case["kind"] in ("prefill", "prompts", "generate"):
        # 24 layers that store bf16 activations are 1.97e-2 from exact arithmetic by that rounding alone; two correct
        # implementations that round in different places are sqrt(2) of it apart
        return {"rel": 3e-2}
    # one block rounds five times on its way (block input products, u, x_proj row, scan output, result)
    return {"rel": 1e-2 if case.get("dtype") == "bf16" else 1e-5}
