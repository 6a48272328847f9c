"""The calls this framework is measured by: whole-model prefill and decode, the composed scan and the
scan with its epilogue, each through its public entry point.

Two models: "135m" is the 135M-class model of the benchmark (hidden 768, 24 layers, 24 heads of 64,
128 modes, chunk 256, vocabulary 50280); "default" is `FracConfig()` as it stands (12 heads of 128,
8 modes, chunk 32, vocabulary 32000).  Weights and inputs are random, drawn from the seed on the GPU.
"""

from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "frac-ssm-kernels_b200"))
from frac_ssm_b200 import frac_scan  # noqa: E402
from frac_ssm_b200.layers import scan_epilogue  # noqa: E402
from frac_ssm_b200.models import FracConfig, FracForCausalLM  # noqa: E402

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
MODELS = {
    "135m": dict(vocab_size=50280, hidden_size=768, num_hidden_layers=24, num_attention_heads=24, frac_expand=2.0,
                 frac_num_modes=128, frac_chunk_size=256),
    "default": dict(),
}


def decode(model, batch, dtype="bf16"):
    return dict(kind="decode", model=model, batch=batch, dtype=dtype)


def prefill(model, batch, length, cache, masked, dtype="bf16"):
    return dict(kind="prefill", model=model, batch=batch, length=length, cache=cache, masked=masked, dtype=dtype)


def scan(rows, length, R, M, chunk, dtype="bf16", coeff="bf16", initial=False, final=False):
    return dict(kind="scan", rows=rows, length=length, R=R, M=M, chunk=chunk, dtype=dtype, coeff=coeff,
                initial=initial, final=final)


def layer(batch, heads, length):
    return dict(kind="layer", batch=batch, heads=heads, length=length)


def listed():
    named = {
        # one user's chat: one token at a time through the whole model, its cache given and handed back
        "decode_135m_b1": decode("135m", 1),
        # a serving batch of such users
        "decode_135m_b32": decode("135m", 32),
        # the same step of the model a user gets from FracConfig()
        "decode_default_b8": decode("default", 8),
        # a prompt of ordinary, odd length whose cache is kept for the tokens to come
        "prefill_135m_prompt": prefill("135m", 1, 397, cache=True, masked=False),
        # scoring a large batch of full-length sequences: the benchmark's whole-model prefill
        "prefill_135m_b16_l4096": prefill("135m", 16, 4096, cache=False, masked=False),
        # a batch of prompts of different lengths, padded on the left, through the default model
        "prefill_default_padded": prefill("default", 4, 1000, cache=True, masked=True),
        # one layer's scan at the benchmark's headline shape (batch 8 x 24 heads)
        "scan_135m_b8_l8192": scan(192, 8192, 64, 128, 256),
        # the scan inside the model's prefill of a next piece of a long text: float32 coefficients as the
        # parameter prep emits them, a ragged length, a state that comes in and one that goes out
        "scan_f32_coeff_ragged": scan(96, 5003, 64, 128, 256, coeff="f32", initial=True, final=True),
        # one million-token text, 24 heads: few rows, each very long
        "scan_long_context": scan(24, 1048576, 64, 128, 256),
        # the reference benchmark's own default: two rows, 128 features, 16 modes
        "scan_16_modes": scan(2, 32768, 128, 16, 64),
        # all-float32 check of a single small sequence (8 heads, 64 modes)
        "scan_f32_l1024": scan(8, 1024, 64, 64, 64, dtype="f32", coeff="f32", final=True),
        # a wide layer: scan, skip connection and gated norm over 64 heads
        "layer_64_heads": layer(4, 64, 16384),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "prefill", "scan", "scan_small", "scan_long", "layer"])
    name = rng.choice(["135m", "135m", "default"])
    if kind == "decode":
        return decode(name, _log_int(rng, 1, 64))
    if kind == "prefill":
        length = _log_int(rng, 5, 4096)
        batch = _log_int(rng, 1, max(1, min(16, 65536 // length)))
        return prefill(name, batch, length, cache=rng.random() < 0.5, masked=rng.random() < 0.4)
    if kind == "scan":
        length = _log_int(rng, 100, 16384)
        rows = _log_int(rng, 4, min(384, (192 * 8192) // length))
        return scan(rows, length, 64, 128, rng.choice([64, 128, 256]), coeff=rng.choice(["bf16", "f32"]),
                    initial=rng.random() < 0.5, final=rng.random() < 0.5)
    if kind == "scan_small":
        dtype = rng.choice(["bf16", "bf16", "f32"])
        length = _log_int(rng, 100, 32768)
        rows = _log_int(rng, 1, max(1, min(96, 131072 // length)))
        return scan(rows, length, rng.choice([64, 128]), rng.choice([8, 16, 64]), rng.choice([32, 64]), dtype=dtype,
                    coeff=dtype if rng.random() < 0.7 else "f32", initial=rng.random() < 0.5, final=rng.random() < 0.5)
    if kind == "scan_long":
        return scan(rng.choice([8, 12, 24]), _log_int(rng, 32768, 524288), 64, 128, 256, final=rng.random() < 0.5)
    return layer(_log_int(rng, 1, 4), rng.choice([16, 24, 32, 64]), _log_int(rng, 200, 16384))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _model(case, g):
    cfg = FracConfig(**MODELS[case["model"]])
    with torch.device(DEV):
        model = FracForCausalLM(cfg)
    model = model.to(DTYPES[case["dtype"]]).eval()
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name.endswith("conv1d.weight"):
                p.uniform_(-0.5, 0.5, generator=g)
            elif name.endswith(("norm.weight", "out_norm.weight")):
                p.uniform_(0.8, 1.2, generator=g)
            elif name.endswith(("mixer.D", "dt_bias", "conv1d.bias", "dyn_proj.bias")):
                p.normal_(0.0, 0.3, generator=g)
            elif p.dim() == 2:
                # a trained projection keeps its input's scale: 1/sqrt(fan in)
                p.normal_(0.0, 0.02 if "embed" in name else p.shape[1] ** -0.5, generator=g)
    return cfg, model


def _scan_inputs(rows, L, R, M, dtype, coeff, g):
    """u ~ N(0, 1); c and kappa softmax weights over the modes (kappa times 1 - rho), rho = exp(-dt rate / tau)
    with dt = softplus(N(0, 1) - 4), tau from 1 to 65536 and one rate per row: what the parameter prep emits."""
    u = torch.empty(rows, L, R, device=DEV, dtype=dtype)
    c = torch.empty(rows, L, M, device=DEV, dtype=coeff)
    kappa = torch.empty(rows, L, M, device=DEV, dtype=coeff)
    rho = torch.empty(rows, L, M, device=DEV, dtype=torch.float32)
    log_tau = torch.linspace(0.0, math.log(65536.0), M, device=DEV)
    inv_tau = torch.exp(-log_tau)
    rate = torch.exp(torch.rand(rows, device=DEV, generator=g) * math.log(16.0))
    alpha = 0.3 + 0.6 * torch.rand(rows, device=DEV, generator=g)
    step = max(1, (1 << 21) // M)
    for b in range(rows):       # a row and a stretch of it at a time: bounds the float32 temporaries
        for t in range(0, L, step):
            sl = slice(t, min(t + step, L))
            n = sl.stop - sl.start
            u[b, sl] = torch.randn(n, R, device=DEV, generator=g)
            dt = torch.nn.functional.softplus(torch.randn(n, 1, device=DEV, generator=g) - 4.0)
            r = torch.exp(-dt * rate[b] ** (1.0 / alpha[b]) * inv_tau).clamp_(1e-6, 1 - 1e-6)
            noise = torch.randn(2, n, M, device=DEV, generator=g)
            weights = torch.softmax(noise - alpha[b] * log_tau, dim=-1)
            rho[b, sl] = r
            c[b, sl] = weights[0]
            kappa[b, sl] = (1 - r) * weights[1]
    return u, c, kappa, rho


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        cfg, model = _model(case, g)
        B = case["batch"]
        L = case.get("length", 1)
        ids = torch.randint(1, cfg.vocab_size, (B, L), device=DEV, generator=g)
        s = dict(kind=kind, model=model, ids=ids)
        if kind == "decode":
            # what a prefill leaves behind: per layer the state and the last inputs of the convolution
            shape = (B, cfg.num_attention_heads, cfg.frac_num_modes, cfg.frac_head_dim)
            s["past"] = tuple(
                (0.02 * torch.randn(shape, device=DEV, generator=g),
                 torch.randn(B, cfg.intermediate_size, cfg.frac_conv_kernel - 1, device=DEV, generator=g).to(
                     DTYPES[case["dtype"]]))
                for _ in range(cfg.num_hidden_layers))
        else:
            s["mask"] = None
            if case["masked"]:
                pad = torch.randint(0, max(1, L // 2), (B, 1), device=DEV, generator=g)
                pad[0] = 0
                s["mask"] = (torch.arange(L, device=DEV)[None] >= pad).long()
            s["cache"] = case["cache"]
        return s
    if kind == "scan":
        R, M = case["R"], case["M"]
        u, c, kappa, rho = _scan_inputs(case["rows"], case["length"], R, M, DTYPES[case["dtype"]],
                                        DTYPES[case["coeff"]], g)
        init = 0.05 * torch.randn(case["rows"], R, M, device=DEV, generator=g) if case["initial"] else None
        return dict(kind=kind, args=(u, c, kappa, rho, case["chunk"], init, case["final"]))
    B, H, L, R = case["batch"], case["heads"], case["length"], 64
    u, c, kappa, rho = _scan_inputs(B * H, L, R, 128, torch.bfloat16, torch.bfloat16, g)
    x_conv = u.view(B, H, L, R).permute(0, 2, 1, 3).reshape(B, L, H * R)
    gate = torch.randn(B, L, H * R, device=DEV, generator=g).bfloat16()
    D = torch.randn(H, R, device=DEV, generator=g)
    weight = torch.empty(H * R, device=DEV).uniform_(0.8, 1.2, generator=g).bfloat16()
    return dict(kind=kind, args=(u, c, kappa, rho, 256), x_conv=x_conv, gate=gate, D=D, weight=weight, H=H, R=R)


def run(state):
    kind = state["kind"]
    if kind == "decode":
        return state["model"](state["ids"], past_key_values=state["past"], use_cache=True)
    if kind == "prefill":
        return state["model"](state["ids"], attention_mask=state["mask"], use_cache=state["cache"])
    if kind == "scan":
        return frac_scan(*state["args"])
    h = frac_scan(*state["args"])
    return scan_epilogue(h, state["x_conv"], state["gate"], state["D"], state["weight"], state["H"], state["R"])


def work(case):
    kind = case["kind"]
    if kind == "scan":
        n, R, M = case["rows"] * case["length"], case["R"], case["M"]
        e, k = (4 if case["dtype"] == "f32" else 2), (4 if case["coeff"] == "f32" else 2)
        state = case["rows"] * R * M
        fin = 2 if case["dtype"] == "bf16" else 4
        return {"bytes": n * (2 * R * e + 2 * M * k + 4 * M) + state * (4 * case["initial"] + fin * case["final"]),
                "flops": 5 * n * R * M}
    if kind == "layer":
        # u, x_conv, gate and the output, then c, kappa and rho
        n, R, M = case["batch"] * case["heads"] * case["length"], 64, 128
        return {"bytes": n * (4 * R * 2 + 2 * M * 2 + 4 * M), "flops": 5 * n * R * M + 12 * n * R}
    cfg = FracConfig(**MODELS[case["model"]])
    e = 4 if case["dtype"] == "f32" else 2
    d, di, H, M, R = (cfg.hidden_size, cfg.intermediate_size, cfg.num_attention_heads, cfg.frac_num_modes,
                      cfg.frac_head_dim)
    tokens = case["batch"] * case.get("length", 1)
    matmul = cfg.num_hidden_layers * (d * 2 * di + di * 3 * H + di * 2 * H * M + di * d) + d * cfg.vocab_size
    cache = cfg.num_hidden_layers * case["batch"] * (4 * H * M * R + e * di * (cfg.frac_conv_kernel - 1))
    passes = 2 if kind == "decode" else int(case["cache"])
    return {"bytes": matmul * e + cache * passes + tokens * (cfg.vocab_size * e + 8 + d * e),
            "flops": tokens * (2 * matmul + cfg.num_hidden_layers * 5 * H * R * M)}


def tolerance(case):
    if case["kind"] in ("decode", "prefill"):
        # 24 layers of bf16 activations: against the same weights run in float32 the logits and caches
        # are off by rel 0.016 to 0.019, max 0.11 to 0.16 (decode), and by rel 0.023 to 0.029, max 0.27 to
        # 0.47 (prefill); two bf16 runs may differ by that much again
        return {"rel": 0.03, "max": 0.6 if case["kind"] == "decode" else 0.95}
    if case["kind"] == "scan" and case["dtype"] == "f32":
        # against the token recurrence in float64: rel 8e-7, max 3e-5 at 1024 tokens
        return {"rel": 1e-5, "max": 3e-4}
    # bf16 outputs against the token recurrence in float64: rel 1.6e-3 to 2.6e-3, max 4e-3 to 2.6e-2;
    # the layer's output against its oracle: rel 1.7e-3, max 4e-3
    return {"rel": 0.01, "max": 0.1}
