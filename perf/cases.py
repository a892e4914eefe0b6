"""What the performance of this framework is measured on: its public entry points at the sizes they are used at.

    step       one timestep of streamed inference with the step's vectors on the device (`StreamState.step`, `state_update`)
    host_step  one rollout timestep with the step's vectors in pinned host memory (`HostStep.step`)
    prefill    forward only, the state kept for the steps that follow (`forward`)
    train      forward and backward (`forward` + `backward` on kept buffers, or `ssd_scan` under autograd)
    mixer      forward and backward of a whole mixer layer core: conv + scan + gate + norm (`mamba2_mixer_core`)

Head shapes (heads, headdim, dstate, groups): "policy" is the trading policy's layer, "layer" a 130M-parameter model's layer,
"small" the fp32 parity shape, "wide" and "grouped" two shapes with several B/C groups or a wider state.  Value distributions are
the benchmark's: x, z, dy ~ N(0,1), B, C ~ N(0,1)/sqrt(dstate), step sizes around a log-uniform [1e-3, 1e-1] bias, decay rates
-exp(U(0, log 16)).
"""
import math

import torch
import torch.nn.functional as F

import trading_bot_0_b200 as T
from trading_bot_0_b200 import host, prepost, ssd, stream

DEV = "cuda:0"
HEADS = {"policy": (8, 32, 64, 1), "layer": (24, 64, 128, 1), "small": (4, 32, 16, 1), "wide": (8, 32, 128, 2), "grouped": (4, 64, 64, 2)}
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
LARGEST_ELEMS = 2 * 131072 * 24 * 64      # batch * seqlen * heads * headdim of the largest listed case


def listed():
    return [
        # live trading: one stream per ticker, every step waited for by the decision that follows: pure latency
        dict(name="step_live_4", kind="step", heads="policy", dtype="bf16", streams=4, gate=False, preact=False),
        # a language-model-sized layer serving 192 sequences, with the gate and the softplus(dt + bias) of the layer fused in
        dict(name="step_layer_192", kind="step", heads="layer", dtype="bf16", streams=192, gate=True, preact=True),
        # the rollout benchmark: 8192 environment streams, state in HBM read and written once
        dict(name="step_rollout_8192", kind="step", heads="policy", dtype="bf16", streams=8192, gate=False, preact=False),
        # the rollout loop with environments on the host: 256 environments x 4 tickers, vectors in and outputs out over PCIe
        dict(name="host_step_1024", kind="host_step", heads="policy", dtype="bf16", streams=1024),
        # a live session starts: four tickers' histories of any length from a carried state
        dict(name="prefill_live_4x333", kind="prefill", heads="policy", dtype="bf16", batch=4, seqlen=333, chunk=128, gate=False,
             init=True),
        # prompts of a serving batch: ragged length, gated
        dict(name="prefill_layer_4x4000", kind="prefill", heads="layer", dtype="bf16", batch=4, seqlen=4000, chunk=256, gate=True,
             init=False),
        # the fp32 parity configuration: small, launch-bound
        dict(name="train_fp32_4x256", kind="train", heads="small", dtype="fp32", batch=4, seqlen=256, chunk=64, gate=False,
             init=False, api="autograd"),
        # the policy in fp32: a debugging or fine-tuning batch
        dict(name="train_fp32_16x1000", kind="train", heads="policy", dtype="fp32", batch=16, seqlen=1000, chunk=128, gate=False,
             init=False, api="autograd"),
        # policy-scale training batch (128 environments x 4 tickers), the headline configuration
        dict(name="train_policy_512x1024", kind="train", heads="policy", dtype="bf16", batch=512, seqlen=1024, chunk=128, gate=False,
             init=False, api="calls"),
        # layer shapes of a 130M-parameter model, gated, under autograd
        dict(name="train_layer_16x4096", kind="train", heads="layer", dtype="bf16", batch=16, seqlen=4096, chunk=256, gate=True,
             init=False, api="autograd"),
        # long-sequence training, all of it on one GPU
        dict(name="train_long_2x131072", kind="train", heads="layer", dtype="bf16", batch=2, seqlen=131072, chunk=256, gate=False,
             init=False, api="calls"),
        # a whole mixer of the policy on one minibatch (16 environments x 4 tickers)
        dict(name="mixer_policy_64x1024", kind="mixer", heads="policy", dtype="bf16", batch=64, seqlen=1024, chunk=128),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _batch(rng, heads, seqlen, most_elems, most_batch):
    h, p, _, _ = HEADS[heads]
    return _log_int(rng, 1, max(1, min(most_batch, most_elems // (seqlen * h * p))))


def draw(rng):
    kind = rng.choice(["step", "host_step", "prefill", "train_bf16", "train_bf16", "train_fp32", "mixer"])
    if kind == "step":
        heads = rng.choice(["policy", "policy", "layer", "wide"])
        return dict(kind="step", heads=heads, dtype=rng.choice(["bf16", "bf16", "bf16", "fp32"]),
                    streams=_log_int(rng, 1, 1024 if heads == "layer" else 8192), gate=rng.random() < 0.5, preact=rng.random() < 0.5)
    if kind == "host_step":
        return dict(kind="host_step", heads="policy", dtype="bf16", streams=_log_int(rng, 16, 8192))
    if kind == "prefill":
        heads = rng.choice(["policy", "layer"])
        seqlen = _log_int(rng, 32, 8192)
        return dict(kind="prefill", heads=heads, dtype="bf16", batch=_batch(rng, heads, seqlen, LARGEST_ELEMS // 8, 64), seqlen=seqlen,
                    chunk=128 if heads == "policy" else 256, gate=rng.random() < 0.5, init=rng.random() < 0.5)
    if kind == "train_fp32":
        heads = rng.choice(["small", "policy"])
        seqlen = _log_int(rng, 64, 2048)
        return dict(kind="train", heads=heads, dtype="fp32", batch=_batch(rng, heads, seqlen, 1 << 23, 64), seqlen=seqlen,
                    chunk=64 if heads == "small" else 128, gate=rng.random() < 0.25, init=rng.random() < 0.25, api="autograd")
    if kind == "train_bf16":
        heads = rng.choice(["policy", "policy", "layer", "layer", "wide", "grouped"])
        seqlen = 128 * _log_int(rng, 1, 128)                       # training batches are cut to whole chunks ...
        if rng.random() < 0.25:
            seqlen = max(96, seqlen - rng.randrange(1, 128))       # ... most of the time
        return dict(kind="train", heads=heads, dtype="bf16", batch=_batch(rng, heads, seqlen, LARGEST_ELEMS // 3, 512), seqlen=seqlen,
                    chunk=256 if heads == "layer" else 128, gate=rng.random() < 0.5, init=rng.random() < 0.25,
                    api=rng.choice(["calls", "autograd"]))
    heads = rng.choice(["policy", "policy", "layer"])
    seqlen = 128 * _log_int(rng, 1, 32)
    return dict(kind="mixer", heads=heads, dtype="bf16", batch=_batch(rng, heads, seqlen, LARGEST_ELEMS // 8, 256), seqlen=seqlen,
                chunk=128 if heads == "policy" else 256)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _head_parameters(g, H):
    """Per-head decay rate, and the bias whose softplus is log-uniform in [1e-3, 1e-1]."""
    dt0 = torch.exp(math.log(1e-3) + torch.rand(H, generator=g, device=DEV) * math.log(100.0))
    A = -torch.exp(torch.rand(H, generator=g, device=DEV) * math.log(16.0))
    return A, dt0 + torch.log(-torch.expm1(-dt0)), torch.ones(H, device=DEV)


def _prepare_step(c, g):
    H, P, N, G = HEADS[c["heads"]]
    S, dt = c["streams"], DTYPES[c["dtype"]]
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    A, bias, D = _head_parameters(g, H)
    raw = 0.5 * r(S, H)
    st = stream.init_stream_state_batched(S, H, P, N, DEV, std=0.1, generator=g)
    a = dict(x=r(S, H, P).to(dt), dt=(raw if c["preact"] else F.softplus(raw + bias)).to(dt), A=A,
             Bm=(r(S, G, N) / math.sqrt(N)).to(dt), Cm=(r(S, G, N) / math.sqrt(N)).to(dt), D=D,
             z=r(S, H, P).to(dt) if c["gate"] else None)
    return dict(stream=st, args=a, preact=dict(dt_bias=bias, dt_softplus=True) if c["preact"] else None)


def _prepare_host_step(c, g):
    H, P, N, G = HEADS[c["heads"]]
    S, dt = c["streams"], DTYPES[c["dtype"]]
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    A, bias, D = _head_parameters(g, H)
    st = stream.init_stream_state_batched(S, H, P, N, DEV, std=0.1, generator=g)
    hs = host.HostStep(st.state, G, dt)
    hs.load_inputs(r(S, H, P).to(dt), F.softplus(0.5 * r(S, H) + bias).to(dt), (r(S, G, N) / math.sqrt(N)).to(dt),
                   (r(S, G, N) / math.sqrt(N)).to(dt))
    return dict(host=hs, A=A, D=D)


def _prepare_sequence(c, g):
    H, P, N, G = HEADS[c["heads"]]
    B, L, dt = c["batch"], c["seqlen"], DTYPES[c["dtype"]]
    train = c["kind"] == "train"
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    A, bias, D = _head_parameters(g, H)
    t = dict(x=r(B, L, H, P).to(dt), dt=F.softplus(0.5 * r(B, L, H) + bias).to(dt), A=A, Bm=(r(B, L, G, N) / math.sqrt(N)).to(dt),
             Cm=(r(B, L, G, N) / math.sqrt(N)).to(dt), D=D, z=r(B, L, H, P).to(dt) if c["gate"] else None,
             init_state=0.1 * r(B, H, P, N) if c["init"] else None)
    s = dict(args=t, dy=r(B, L, H, P).to(dt) if train else None)
    if train and c["api"] == "autograd":
        s["leaves"] = [v.requires_grad_() for v in t.values() if v is not None]
    else:   # a program that calls the operator keeps its workspace and output buffers
        d = ssd.make_dims(t["x"], t["dt"], t["Bm"], t["Cm"], c["chunk"], z=t["z"])
        s["workspace"] = ssd.alloc_workspace(d, DEV, backward=train)
        s["y"], s["final"] = torch.empty_like(t["x"]), torch.empty(B, H, P, N, device=DEV)
        s["out"] = {}
    return s


def _prepare_mixer(c, g):
    H, P, N, G = HEADS[c["heads"]]
    B, L, dt = c["batch"], c["seqlen"], DTYPES[c["dtype"]]
    C = H * P + 2 * G * N
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    A, bias, D = _head_parameters(g, H)
    t = dict(xBC=r(B, L, C).to(dt), dt=(0.5 * r(B, L, H)).to(dt), z=r(B, L, H, P).to(dt), conv_weight=r(C, 4) / 2, conv_bias=0.1 * r(C),
             dt_bias=bias, A=A, D=D, norm_weight=1 + 0.1 * r(H * P))
    return dict(args=t, leaves=[v.requires_grad_() for v in t.values()], dout=r(B, L, H * P).to(dt),
                shape=dict(nheads=H, headdim=P, dstate=N, ngroups=G, chunk=c["chunk"]))


def prepare(case, seed):
    g = _generator(seed)
    make = {"step": _prepare_step, "host_step": _prepare_host_step, "prefill": _prepare_sequence, "train": _prepare_sequence,
            "mixer": _prepare_mixer}[case["kind"]]
    return dict(make(case, g), case=case)


def run(state):
    c = state["case"]
    if c["kind"] == "step":
        st, a = state["stream"], state["args"]
        if state["preact"]:
            y = T.state_update(st.state, a["x"], a["dt"], a["A"], a["Bm"], a["Cm"], a["D"], a["z"], **state["preact"])
        else:
            y = st.step(a["x"], a["dt"], a["A"], a["Bm"], a["Cm"], a["D"], a["z"])
        return [y, st.state]
    if c["kind"] == "host_step":
        h = state["host"]
        h.step(state["A"], state["D"])
        return [h.hy, h.state]
    if c["kind"] == "mixer":
        out, fin = prepost.mamba2_mixer_core(**state["args"], **state["shape"])
        return [out.detach(), fin.detach(), *torch.autograd.grad(out, state["leaves"], state["dout"])]
    a = state["args"]
    if c["kind"] == "train" and c["api"] == "autograd":
        y, fin = T.ssd_scan(**a, chunk=c["chunk"])
        return [y.detach(), fin.detach(), *torch.autograd.grad(y, state["leaves"], state["dy"])]
    train = c["kind"] == "train"
    y, fin, ws = T.forward(**a, chunk=c["chunk"], workspace=state["workspace"], y=state["y"], final_state=state["final"],
                           for_backward=train)
    if not train:
        return [y, fin]
    g = T.backward(state["dy"], **a, chunk=c["chunk"], workspace=ws, fwd_saved=True, out=state["out"])
    return [y, fin] + [g[k] for k in ("dx", "ddt", "dA", "dB", "dC", "dD", "dz", "dinit") if k in g]


def work(case):
    """Bytes: every input read once, every output written once.  Flops: the recurrence's multiply-adds (rank-one update and
    read-out of the state; backward: the same for the two adjoint products and the four gradients)."""
    H, P, N, G = HEADS[case["heads"]]
    e = 2 if case["dtype"] == "bf16" else 4
    hp, gn, st = H * P, G * N, H * P * N * 4
    if case["kind"] in ("step", "host_step"):
        S, z = case["streams"], hp if case.get("gate") else 0
        return {"bytes": S * (2 * st + (2 * hp + H + 2 * gn + z) * e), "flops": S * 5.0 * H * P * N}
    B, tokens = case["batch"], case["batch"] * case["seqlen"]
    fwd_flops, bwd_flops = 5.0 * H * P * N, 12.0 * H * P * N
    if case["kind"] == "mixer":
        C = hp + 2 * gn
        io = C + H + hp                                            # xBC, dt, z
        return {"bytes": tokens * e * (io + hp + io + hp + io) + B * st, "flops": tokens * (fwd_flops + bwd_flops)}
    z = hp if case["gate"] else 0
    io = hp + H + 2 * gn + z
    fwd = tokens * e * (io + hp) + B * st * (2 if case["init"] else 1)
    if case["kind"] == "prefill":
        return {"bytes": fwd, "flops": tokens * fwd_flops}
    bwd = tokens * (e * (io + hp) + e * (io - H) + 4 * H) + (2 * B * st if case["init"] else 0)
    return {"bytes": fwd + bwd, "flops": tokens * (fwd_flops + bwd_flops)}


def tolerance(case):
    """bf16 outputs agree to 1e-2.  A training pass also returns dA (and d(dt bias)): token sums of terms that mostly cancel, in
    which two evaluations of the same bf16 inputs differ by up to a few percent.  fp32: long sums in another order (dA shows
    1.3e-5 between two chunk lengths)."""
    if case["dtype"] == "fp32":
        return {"rel": 3e-5}
    return {"rel": 3e-2} if case["kind"] in ("train", "mixer") else {"rel": 1e-2}
