"""Calls whose inputs and weights other kernels write right in front of them, and overwrite right behind them, on the same stream and in a
captured graph.  Most kernels here take their places while the one before them finishes; what they read must be there all the same.  The
arithmetic is the same as in a call on its own, so results are compared bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

bf16, f32 = torch.bfloat16, torch.float32


def _wkv7(shape, dtype):
    def make(pkg, workloads, seed):
        x = workloads.wkv7_inputs(*shape, seed=seed, dtype=dtype, device="cuda", state="normal")

        def call(x):
            out = pkg.wkv7_statepass(x["s0"], pkg.Wkv7PretrainForwardInputs(*[x[n] for n in "rwkvab"]), reference_contract=False)
            return out.output, out.next_state
        return x, call
    return make


def _training(pkg, workloads, seed):
    x = workloads.wkv7_inputs(2, 320, 12, 64, seed=seed, dtype=bf16, device="cuda", state="normal")
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x["dy"] = torch.randn((2, 320, 12, 64), generator=g, device="cuda").to(bf16)

    def call(x):
        leaves = [x[n].detach().requires_grad_() for n in ("r", "w", "k", "v", "a", "b", "s0")]
        y, state = pkg.wkv7_statepass_autograd(leaves[6], pkg.Wkv7PretrainForwardInputs(*leaves[:6]))
        dy = x["dy"] + 0    # (right in front of the backward pass)
        return (y.detach(), state.detach(), *torch.autograd.grad((y, state), leaves, (dy, state.detach())))
    return x, call


def _mix6(pkg, workloads, seed):
    x, mus = workloads.mix_inputs(2, 600, 768, seed=seed, dtype=bf16, device="cuda")
    return dict(x=x, **{"m%d" % i: m for i, m in enumerate(mus)}), lambda x: tuple(pkg.mix6(x["x"], *[x["m%d" % i] for i in range(6)]).values())


def _token_shift(pkg, workloads, seed):
    x, mus = workloads.mix_inputs(16, 1, 768, seed=seed, dtype=bf16, device="cuda", nscale=5)
    slots = workloads.mix_inputs(1, 32, 768, seed=seed + 9, dtype=bf16, device="cuda")[0][0]
    ids = torch.arange(16, dtype=torch.int32, device="cuda") * 2 + seed % 2

    def call(x):
        shift = pkg.token_shift_diff(x["x"], x["slots"], x["ids"])
        mixed = pkg.addcmul5(x["x"], shift.token_shifted_diff, *[x["m%d" % i] for i in range(5)])
        return (shift.token_shifted_diff, shift.next_token_shift, *mixed.values())
    return dict(x=x, slots=slots, ids=ids, **{"m%d" % i: m for i, m in enumerate(mus)}), call


def _epilogues(pkg, workloads, seed):
    def call(e):
        w = pkg.weight_prepare_epilogue(e["key_precursor"], e["learning_rate_lora"], e["weight_decay_lora"], e["key_removal"], e["key_replacement"], 12,
                                        value_precursor=e["value_precursor"], value_from_first_cell=e["value_from_first_cell"],
                                        value_residual_lora=e["value_residual_lora"])
        return (w.replacement_key, w.value, w.weight_decay, w.removal_key_normalized, w.replacement,
                pkg.gated_readout_epilogue(e["wkv7_output"], e["receptance"], w.replacement_key, w.value, e["gate"], e["group_norm_gamma"],
                                           e["group_norm_beta"], e["receptance_key_bonus"], 12))
    return workloads.time_mixer_epilogue_inputs(2, 300, 12, 64, seed=seed, dtype=bf16, device="cuda"), call


def _channel_mixer(rows):
    def make(pkg, workloads, seed):
        x = dict(zip(("x", "scale", "kw", "vw"), workloads.channel_mixer_inputs(1, rows, 768, 3072, seed=seed, device="cuda")))
        return x, lambda x: (pkg.channel_mixer(x["x"], x["scale"], x["kw"], x["vw"]),)
    return make


def _lm_head(rows):
    def make(pkg, workloads, seed):
        x = dict(zip(("x", "w", "targets"), workloads.lm_head_inputs(rows, 2048, 4100, seed=seed, device="cuda")))
        return x, lambda x: tuple(pkg.lm_head_ce(x["x"], x["w"], x["targets"]))
    return make


CALLS = {
    "decode": _wkv7((16, 1, 12, 64), bf16), "sequential": _wkv7((2, 40, 4, 64), bf16), "prefill": _wkv7((1, 333, 12, 64), bf16),
    "prefill_many_chunks": _wkv7((4, 4096, 12, 64), bf16), "prefill_fp32": _wkv7((1, 700, 12, 64), f32), "sequential_fp32": _wkv7((1, 100, 12, 64), f32),
    "training": _training, "mix6": _mix6, "token_shift_addcmul5": _token_shift, "epilogues": _epilogues,
    "channel_mixer_pieces": _channel_mixer(16), "channel_mixer": _channel_mixer(300), "channel_mixer_pairs": _channel_mixer(3000),
    "lm_head": _lm_head(100), "lm_head_pairs": _lm_head(500),
}


def _fill(to, source):
    for name, t in to.items():
        torch.add(source[name], 0, out=t)   # (a kernel, where copy_ may be a copy engine's work)


@pytest.mark.parametrize("name", CALLS)
def test_inputs_written_right_in_front(pkg, workloads, cuda, name):
    old, call = CALLS[name](pkg, workloads, 1)
    new, _ = CALLS[name](pkg, workloads, 2)
    expected = [t.clone() for t in call(new)]
    x = {n: t.clone() for n, t in old.items()}
    for _ in range(3):
        stale = call(x)
        _fill(x, new)
        got = call(x)
        _fill(x, old)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, expected))
        assert not torch.equal(stale[0], got[0])
    assert pkg.read_device_status(0) == 0


@pytest.mark.parametrize("name", [n for n in CALLS if n != "training"])
def test_inputs_written_right_in_front_in_a_graph(pkg, workloads, cuda, name):
    old, call = CALLS[name](pkg, workloads, 1)
    new, _ = CALLS[name](pkg, workloads, 2)
    expected = [t.clone() for t in call(new)]
    x = {n: t.clone() for n, t in old.items()}
    torch.cuda.synchronize()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        call(x)
        _fill(x, new)
        got = call(x)
        _fill(x, old)
    for _ in range(3):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, expected))
    assert pkg.read_device_status(0) == 0


@pytest.mark.parametrize("rows", [16, 300, 3000])
def test_weights_from_a_kernel_that_lets_the_next_one_in_early(pkg, workloads, cuda, rows):
    """mix6 lets its successor start before it has written the weights."""
    x, scale, kw, vw = workloads.channel_mixer_inputs(1, rows, 768, 3072, seed=3, device="cuda")
    h, w, targets = workloads.lm_head_inputs(rows, 768, 4100, seed=4, device="cuda")
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    rates = {n: [torch.rand((1, 1, t.shape[-1]), generator=g, device="cuda").to(bf16) for _ in range(6)] for n, t in (("kw", kw), ("vw", vw), ("w", w))}

    def updated(name, weight):
        return pkg.mix6(weight[None], *rates[name])["learning_rate_input"][0]

    def calls(pause):
        out = []
        for first, second in (("kw", "vw"), ("vw", "kw")):
            new = {}
            for n in (first, second):
                new[n] = updated(n, kw if n == "kw" else vw)
            pause()
            out.append(pkg.channel_mixer(x, scale, new["kw"], new["vw"]))
        new = updated("w", w)
        pause()
        return out + list(pkg.lm_head_ce(h, new, targets))
    expected = [t.clone() for t in calls(torch.cuda.synchronize)]
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(calls(lambda: None), expected))
    assert pkg.read_device_status(0) == 0
