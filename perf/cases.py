"""The operator calls whose speed matters to a user of this library, over the sizes they are made with.

One case is one pass through the public entry points on the GPU: a WKV7 call (decode, prefill, training), the
token-shift mixing and the two epilogues around it, the channel mixer, the LM-head cross entropy.  Widths are those of
the benchmark configurations (head size 64; 12, 32, 40 and 64 heads; vocabulary 65 536); batch and context length are
what a server or a trainer sends, ragged lengths among them.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from __graft_entry__ import load_package

pkg = load_package()
from rwkv_rs_stable_b200 import cell_forward, workloads  # noqa: E402  (the package is loaded under this name)

N = 64
HEADS = (12, 16, 32, 40, 64)
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
# No drawn case is larger than the largest listed ones.
MAX_TOKEN_HEADS = 16 * 8192 * 32
MAX_FLOPS = 2.2e12


def listed():
    return [
        # One user's chat: the next token of one sequence, one layer of the 32-head model.  Latency of a call.
        dict(name="decode_one", op="decode", B=1, T=1, H=32),
        # A loaded server: one layer-step of the decode configuration, 1024 sequences of 40 heads.
        dict(name="decode_batch", op="decode", B=1024, T=1, H=40),
        # A chat prompt of odd length, state carried on; decays as the model initialises them.
        dict(name="prefill_prompt", op="prefill", B=1, T=333, H=32, dtype="bf16", decay="model"),
        # The headline prefill configuration.
        dict(name="prefill_batch", op="prefill", B=8, T=4096, H=12, dtype="bf16", decay="uniform"),
        # A few documents cut at an odd length, decays as the model initialises them.
        dict(name="prefill_documents", op="prefill", B=3, T=2047, H=32, dtype="bf16", decay="model"),
        # One layer of the whole-model prefill configuration, the largest call.
        dict(name="prefill_layer", op="prefill", B=16, T=8192, H=32, dtype="bf16", decay="uniform"),
        # fp32 tensors, the element type of the reference's own tests.
        dict(name="prefill_f32", op="prefill", B=2, T=1000, H=12, dtype="f32", decay="uniform"),
        # A training step of the layer: forward with autograd, then backward.
        dict(name="train_batch", op="train", B=8, T=4096, H=12, state=False),
        # Everything this library does around WKV7 in a decode step of 16 sequences: five launches of small work.
        dict(name="around_decode", op="around", B=16, T=1, H=32),
        # The same around a prefill, odd number of tokens.
        dict(name="around_prefill", op="around", B=4, T=2049, H=32),
        # The feed-forward half of a layer during prefill.
        dict(name="channel_mixer", op="channel_mixer", B=2, T=2048, C=2048, F=8192),
        # Loss over one ragged batch of rows against the whole vocabulary.
        dict(name="lm_head", op="lm_head", R=8191, C=2048, V=65536),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng):
    op = rng.choice(("decode", "prefill", "prefill", "prefill_f32", "train", "around", "channel_mixer", "lm_head"))
    H = rng.choice(HEADS)
    if op == "decode":
        # (up to four tokens at a time: speculative steps; one token is by far the usual step)
        return dict(op=op, B=_log(rng, 1, 40960 // H), T=rng.choice((1, 1, 1, 1, 2, 3, 4)), H=H)
    if op == "prefill":
        decay = rng.choice(("uniform", "model"))
        most = MAX_TOKEN_HEADS if decay == "uniform" else MAX_TOKEN_HEADS // 4
        T = _log(rng, 5, 16384)
        return dict(op=op, B=_log(rng, 1, max(1, min(64, most // (T * H)))), T=T, H=H, dtype="bf16", decay=decay)
    if op == "prefill_f32":
        T = _log(rng, 16, 4096)
        return dict(op="prefill", B=_log(rng, 1, max(1, min(16, MAX_TOKEN_HEADS // 8 // (T * H)))), T=T, H=H, dtype="f32",
                    decay=rng.choice(("uniform", "uniform", "model")))
    if op == "train":
        T = 16 * _log(rng, 4, 256)
        return dict(op=op, B=_log(rng, 1, max(1, min(16, 8 * 4096 * 12 // (T * H)))), T=T, H=H, state=rng.random() < 0.5)
    if op == "around":
        T = 1 if rng.random() < 0.5 else _log(rng, 2, 8192)
        return dict(op=op, B=_log(rng, 1, max(1, min(512, 16384 * 32 // (T * H)))), T=T, H=H)
    if op == "channel_mixer":
        C = rng.choice((768, 1024, 2048, 2560, 4096))
        rows = _log(rng, 1, int(MAX_FLOPS / (16 * C * C)))
        B = _log(rng, 1, min(rows, 64))
        return dict(op=op, B=B, T=max(1, rows // B), C=C, F=4 * C)
    C = rng.choice((768, 1024, 2048, 2560, 4096))
    V = rng.choice((65536, 65536, 32768, 8192))     # the whole vocabulary, or one GPU's shard of it
    return dict(op=op, R=_log(rng, 16, int(MAX_FLOPS / (2 * C * V))), C=C, V=V)


def _model_decay(shape, seed, dtype):
    """``-softplus(-d) - 0.5`` with ``d`` at the reference's initial decay speeds of a middle layer, moved per token."""
    B, T, H, n = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(7 + 1009 * seed)
    bias = cell_forward.decay_speed_bias(24, H * n, n, 12).cuda().view(1, 1, H, n)
    d = bias + 0.3 * torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
    return (-F.softplus(-d) - 0.5).to(dtype)


def _sequence(x):
    return pkg.Wkv7PretrainForwardInputs(x["r"], x["w"], x["k"], x["v"], x["a"], x["b"])


def prepare(case, seed):
    op = case["op"]
    if op in ("decode", "prefill", "train"):
        shape = (case["B"], case["T"], case["H"], N)
        dtype = DTYPES[case.get("dtype", "bf16")]
        x = workloads.wkv7_inputs(*shape, seed=seed, dtype=dtype, device="cuda",
                                  state="normal" if case.get("state", True) else None)
        if case.get("decay") == "model":
            x["w"] = _model_decay(shape, seed, dtype)
        s = dict(op=op, state=x.get("s0"))
        if op == "train":
            g = torch.Generator(device="cuda")
            g.manual_seed(11 + 1013 * seed)
            s["dy"] = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(dtype)
            s["leaves"] = [x[n].requires_grad_() for n in ("r", "w", "k", "v", "a", "b")]
            if s["state"] is not None:
                s["dstate"] = 0.1 * torch.randn(s["state"].shape, generator=g, device="cuda", dtype=torch.float32)
                s["leaves"].append(s["state"].requires_grad_())
        s["sequence"] = _sequence(x)
        return s
    if op == "around":
        B, T, H = case["B"], case["T"], case["H"]
        x, scales = workloads.mix_inputs(B, T, H * N, seed=seed, dtype=torch.bfloat16, device="cuda")
        s = dict(op=op, x=x, scales=scales, H=H, step=T == 1,
                 e=workloads.time_mixer_epilogue_inputs(B, T, H, N, seed=seed, dtype=torch.bfloat16, device="cuda"))
        if s["step"]:
            g = torch.Generator(device="cuda")
            g.manual_seed(13 + 1019 * seed)
            # a server keeps more slots than it steps: the last token of every sequence, picked by batch_ids
            s["slots"] = torch.randn((2 * B, H * N), generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)
            s["ids"] = torch.randperm(2 * B, generator=g, device="cuda")[:B].to(torch.int32)
        return s
    if op == "channel_mixer":
        args = workloads.channel_mixer_inputs(case["B"], case["T"], case["C"], case["F"], seed=seed, device="cuda")
    else:
        args = workloads.lm_head_inputs(case["R"], case["C"], case["V"], seed=seed, device="cuda")
    return dict(op=op, args=args)


def run(s):
    op = s["op"]
    if op == "decode":      # the state is updated in place, as a server's cache is
        out = pkg.wkv7_statepass(s["state"], s["sequence"], reference_contract=False, next_state=s["state"])
        return out.output, out.next_state
    if op == "prefill":
        out = pkg.wkv7_statepass(s["state"], s["sequence"], reference_contract=False)
        return out.output, out.next_state
    if op == "train":
        y, state = pkg.wkv7_statepass_autograd(s["state"], s["sequence"])
        if s["state"] is None:
            return y.detach(), torch.autograd.grad(y, s["leaves"], s["dy"])
        return y.detach(), state.detach(), torch.autograd.grad((y, state), s["leaves"], (s["dy"], s["dstate"]))
    if op == "around":
        x, scales, e = s["x"], s["scales"], s["e"]
        if s["step"]:
            shift = pkg.token_shift_diff(x, s["slots"], s["ids"])
            mixed = dict(pkg.addcmul5(x, shift.token_shifted_diff, *scales[:5]), diff=shift.token_shifted_diff,
                         slots=shift.next_token_shift)
        else:
            mixed = pkg.mix6(x, *scales)
        w = pkg.weight_prepare_epilogue(e["key_precursor"], e["learning_rate_lora"], e["weight_decay_lora"],
                                        e["key_removal"], e["key_replacement"], s["H"],
                                        value_precursor=e["value_precursor"],
                                        value_from_first_cell=e["value_from_first_cell"],
                                        value_residual_lora=e["value_residual_lora"])
        out = pkg.gated_readout_epilogue(e["wkv7_output"], e["receptance"], w.replacement_key, w.value, e["gate"],
                                         e["group_norm_gamma"], e["group_norm_beta"], e["receptance_key_bonus"], s["H"])
        return dict(mixed, weight_decay=w.weight_decay, key=w.replacement_key, value=w.value,
                    removal=w.removal_key_normalized, replacement=w.replacement, readout=out)
    if op == "channel_mixer":
        return pkg.channel_mixer(*s["args"])
    return pkg.lm_head_ce(*s["args"])


def work(case):
    op = case["op"]
    if op in ("decode", "prefill", "train"):
        chains, th = case["B"] * case["H"], case["B"] * case["T"] * case["H"]
        row = N * DTYPES[case.get("dtype", "bf16")].itemsize
        state = 4 * N * N * chains
        if op == "train":       # six inputs and the output gradient in, the output and six gradients out
            return {"bytes": 14 * row * th + (4 if case["state"] else 1) * state, "flops": 27 * N * N * th}
        # the recurrence itself: S·a, S·diag, + sa bᵀ, + v kᵀ, S·r
        return {"bytes": 7 * row * th + 2 * state, "flops": 9 * N * N * th}
    if op == "around":
        elements = case["B"] * case["T"] * case["H"] * N
        carried = 4 * case["B"] * case["H"] * N if case["T"] == 1 else 0
        return {"bytes": 2 * (22 * elements + 2 * carried), "flops": 60 * elements}
    if op == "channel_mixer":
        rows, C, Fd = case["B"] * case["T"], case["C"], case["F"]
        return {"bytes": 2 * (2 * rows * C + 2 * C * Fd), "flops": 4 * rows * C * Fd}
    R, C, V = case["R"], case["C"], case["V"]
    return {"bytes": 2 * (R * C + V * C) + 16 * R, "flops": 2 * R * C * V}


def tolerance(case):
    op = case["op"]
    if op == "lm_head":                 # exact bf16 products, fp32 sums and logarithm
        return {"rel": 1e-5}
    if op == "prefill" and case["dtype"] == "f32":
        return {"rel": 1e-3}            # (long sequences go through operands of 11 significant bits)
    if op == "train":
        return {"rel": 1e-2}            # bf16 gradients, bf16 saved tensors
    return {"rel": 5e-3}                # one rounding to bf16
