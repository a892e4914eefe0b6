"""Streamed-rollout step: parity with the oracle recurrence, prefill/step equivalence, reset."""
import pytest
import torch

from oracle import ssd_oracle as O
from tests._util import assert_close, cfg_like, to_dev

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def oracle_steps(inp, steps, z=None):
    S = inp["state"].double()
    ys = []
    for t in range(steps):
        y, S = O.state_update(S, inp["x"][t], inp["dt"][t], inp["A"], inp["B"][t], inp["C"][t], inp["D"],
                              None if z is None else z[t])
        ys.append(y)
    return torch.stack(ys), S


@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
@pytest.mark.parametrize("H,P,N,G", [(8, 32, 64, 1), (4, 32, 16, 1), (24, 64, 128, 1), (2, 16, 256, 2),
                                     (6, 24, 40, 3), (4, 20, 32, 2)])
def test_state_update_matches_oracle(lib, dtype, H, P, N, G):
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("dec", 33, 1, H, P, N, G, 1, dtype)
    steps = 12
    inp = O.make_decode_inputs(cfg, steps)
    z = torch.randn(steps, 33, H, P, generator=torch.Generator().manual_seed(3)).to(O.torch_dtype(dtype))
    ref_y, ref_S = oracle_steps(inp, steps, z)
    d = to_dev(inp, DEV)
    zd = z.to(DEV)
    st = T.StreamState(d["state"].clone())
    ys = [st.step(d["x"][t], d["dt"][t], d["A"], d["B"][t], d["C"][t], d["D"], zd[t]) for t in range(steps)]
    assert_close("y", torch.stack(ys), ref_y, dtype)
    assert_close("state", st.state, ref_S, "fp32" if dtype == "fp32" else "bf16")


def test_prefill_then_steps_equals_full(lib):
    """chunk-scan over the first k tokens, then L-k single steps, equals the chunk-scan over all L
    (the SSD analogue of `cached_forward_matches_full_forward`,
    trading_bots/src/torch/world_model.rs:2683-2718: prefill 32, then 32 steps, max-abs < 1e-4)."""
    import trading_bot_0_b200 as T
    cfg = cfg_like(0, seqlen=64, chunk=32)
    d = to_dev(O.make_inputs(cfg), DEV)
    y_full, fin_full, _ = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], chunk=cfg.chunk)
    k = 32
    y_pre, fin, _ = T.forward(d["x"][:, :k], d["dt"][:, :k], d["A"], d["B"][:, :k], d["C"][:, :k], d["D"],
                              chunk=cfg.chunk)
    st = T.StreamState(fin)
    ys = [y_pre]
    for t in range(k, cfg.seqlen):
        ys.append(st.step(d["x"][:, t], d["dt"][:, t], d["A"], d["B"][:, t], d["C"][:, t], d["D"])[:, None])
    y_cat = torch.cat(ys, 1)
    assert (y_cat - y_full).abs().max().item() < 1e-4
    assert (st.state - fin_full).abs().max().item() < 1e-4


def test_batched_equals_per_stream(lib):
    """Batched step == each stream stepped alone (mirror of the windowed-replay-vs-sequential test,
    trading_bots/src/torch/model/stream/replay.rs:263-353)."""
    import trading_bot_0_b200 as T
    cfg = cfg_like(2, batch=5, dtype="fp32")
    d = to_dev(O.make_decode_inputs(cfg, 3), DEV)
    st = T.StreamState(d["state"].clone())
    singles = [T.StreamState(d["state"][s:s + 1].clone()) for s in range(5)]
    for t in range(3):
        y = st.step(d["x"][t], d["dt"][t], d["A"], d["B"][t], d["C"][t], d["D"])
        for s in range(5):
            ys = singles[s].step(d["x"][t, s:s + 1], d["dt"][t, s:s + 1], d["A"], d["B"][t, s:s + 1],
                                 d["C"][t, s:s + 1], d["D"])
            assert torch.equal(ys[0], y[s])
    for s in range(5):
        assert torch.equal(singles[s].state[0], st.state[s])


def test_mid_rollout_stream_reset(lib):
    """Zeroing selected streams between steps == restarting those streams from a zero state
    (mirror of the mid-chunk env reset test, trading_bots/src/torch/model/stream/replay.rs:360-485)."""
    import trading_bot_0_b200 as T
    cfg = cfg_like(2, batch=9, dtype="fp32")
    d = to_dev(O.make_decode_inputs(cfg, 4), DEV)
    st = T.StreamState(d["state"].clone())
    fresh = T.init_stream_state_batched(9, cfg.nheads, cfg.headdim, cfg.dstate, DEV)
    idx = torch.tensor([1, 4, 8], device=DEV)
    for t in range(2):
        st.step(d["x"][t], d["dt"][t], d["A"], d["B"][t], d["C"][t], d["D"])
    st.reset_streams(idx)
    assert st.state[idx].abs().max().item() == 0.0 and st.state[0].abs().max().item() > 0.0
    for t in range(2, 4):
        y = st.step(d["x"][t], d["dt"][t], d["A"], d["B"][t], d["C"][t], d["D"])
        yf = fresh.step(d["x"][t], d["dt"][t], d["A"], d["B"][t], d["C"][t], d["D"])
    assert torch.equal(y[idx], yf[idx])
    st.reset()
    assert st.state.abs().max().item() == 0.0


@pytest.mark.parametrize("groups,graph", [(1, False), (3, True), (8, True)])
def test_host_step_groups_match_oracle(lib, groups, graph):
    """The host-buffer rollout step (pinned staging buffers, streams cut into row groups that overlap on three CUDA
    streams, the step replayed from a CUDA graph) gives the oracle's outputs and state, whatever the number of groups
    (33 streams: ragged last group)."""
    from trading_bot_0_b200.host import HostStep
    cfg = O.SsdConfig("dec", 33, 1, 8, 32, 64, 1, 1, "bf16")
    steps = 6
    inp = O.make_decode_inputs(cfg, steps)
    ref_y, ref_S = oracle_steps(inp, steps)
    d = to_dev(inp, DEV)
    state = d["state"].clone()
    hs = HostStep(state, cfg.ngroups, groups=groups, graph=graph, in_place=False)
    ys = []
    for t in range(steps):
        hs.load_inputs(inp["x"][t], inp["dt"][t], inp["B"][t], inp["C"][t])
        hs.step(d["A"], d["D"])
        torch.cuda.synchronize()
        ys.append(hs.hy.clone())
    assert (hs._graph is not None) == graph and (len(hs.ranges) > 1) == (groups > 1)
    assert_close("y", torch.stack(ys).to(DEV), ref_y, "bf16")
    assert_close("state", state, ref_S, "bf16")


@pytest.mark.parametrize("in_place", [True, False])
@pytest.mark.parametrize("N", [64, 40])
def test_host_step_device_copies(lib, in_place, N):
    """x, dt, Bm, Cm hold the step's vectors on the device after a step of either kind (N = 40 copies anyway)."""
    from trading_bot_0_b200.host import HostStep
    inp = O.make_decode_inputs(O.SsdConfig("dec", 33, 1, 8, 32, N, 1, 1, "bf16"), 2)
    d = to_dev(inp, DEV)
    hs = HostStep(d["state"].clone(), 1, in_place=in_place)
    for t in range(2):
        hs.load_inputs(inp["x"][t], inp["dt"][t], inp["B"][t], inp["C"][t])
        hs.step(d["A"], d["D"])
        for k, v in (("x", hs.x), ("dt", hs.dt), ("B", hs.Bm), ("C", hs.Cm)):
            assert v.is_cuda and torch.equal(v.cpu(), inp[k][t]), k
        torch.cuda.synchronize()
        assert torch.equal(hs.y.cpu(), hs.hy)


@pytest.mark.parametrize("S,H,P,N,G,dtype", [(1, 8, 32, 64, 1, "bf16"), (33, 8, 32, 64, 1, "fp32"), (1201, 8, 32, 64, 2, "bf16"),
                                             (5, 24, 64, 128, 1, "bf16"), (70, 8, 32, 128, 2, "bf16"), (9, 4, 64, 64, 2, "fp32"),
                                             (3, 6, 24, 40, 3, "bf16")])
def test_host_memory_step_matches_oracle(lib, S, H, P, N, G, dtype):
    """The one-kernel host-memory step (and, for the last shape, the copies it leaves to): one stream, fewer and more units than
    resident blocks, several groups, several tiles per head, rows of one and two pieces per thread."""
    from trading_bot_0_b200.host import HostStep
    cfg = O.SsdConfig("dec", S, 1, H, P, N, G, 1, dtype)
    inp = O.make_decode_inputs(cfg, 3)
    ref_y, ref_S = oracle_steps(inp, 3)
    d = to_dev(inp, DEV)
    state = d["state"].clone()
    hs = HostStep(state, G, O.torch_dtype(dtype))
    ys = []
    for t in range(3):
        hs.load_inputs(inp["x"][t], inp["dt"][t], inp["B"][t], inp["C"][t])
        hs.step(d["A"], d["D"])
        torch.cuda.synchronize()
        ys.append(hs.hy.clone())
        assert torch.equal(hs.y.cpu(), hs.hy)
    assert hs._in_place == (N != 40)
    assert_close("y", torch.stack(ys).to(DEV), ref_y, dtype)
    assert_close("state", state, ref_S, dtype)


@pytest.mark.parametrize("P,N,dtype", [(64, 64, "bf16"), (16, 128, "fp32"), (32, 256, "bf16"), (8, 256, "fp32"), (16, 64, "bf16"), (24, 128, "bf16")])
@pytest.mark.parametrize("S", [1, 401])
def test_state_tiles_of_every_width(lib, S, P, N, dtype):
    """Heads of one, several and half tiles of the ring kernel, a single stream and more tiles than the grid has blocks, with
    the gate and the fused step-size activation."""
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("dec", S, 1, 6, P, N, 2, 1, dtype)
    inp = O.make_decode_inputs(cfg, 1)
    g = torch.Generator().manual_seed(5)
    z = torch.randn(S, 6, P, generator=g).to(O.torch_dtype(dtype))
    bias = torch.full((6,), -1.0)
    d = to_dev(inp, DEV)
    state = d["state"].clone()
    y = T.state_update(state, d["x"][0], d["dt"][0], d["A"], d["B"][0], d["C"][0], d["D"], z.to(DEV), dt_bias=bias.to(DEV), dt_softplus=True)
    dt = torch.nn.functional.softplus(inp["dt"][0].double() + bias.double())
    yr, Sr = O.state_update(inp["state"].double(), inp["x"][0], dt, inp["A"], inp["B"][0], inp["C"][0], inp["D"], z)
    assert_close("y", y, yr, dtype)
    assert_close("state", state, Sr, dtype)


def test_state_update_checks_the_callers_y(lib):
    """A y that the kernel would overrun (short, another type or device, inner dims or rows that do not fit) is refused before
    anything is launched; rows that lie apart are written and nothing between them."""
    import trading_bot_0_b200 as T
    S, H, P, N = 6, 8, 32, 64
    inp = O.make_decode_inputs(O.SsdConfig("dec", S, 1, H, P, N, 1, 1, "bf16"), 1)
    d = to_dev(inp, DEV)
    a = lambda st: (st, d["x"][0], d["dt"][0], d["A"], d["B"][0], d["C"][0], d["D"])
    bf = dict(dtype=torch.bfloat16, device=DEV)
    bad = [torch.empty(S - 1, H, P, **bf), torch.empty(S, H, P - 1, **bf), torch.empty(S * H * P, **bf),
           torch.empty(S, H, P, dtype=torch.float16, device=DEV), torch.empty(S, H, P, device=DEV), torch.empty(S, H, P, dtype=torch.bfloat16),
           torch.empty(S, H, 2 * P, **bf)[:, :, ::2], torch.empty(S, H, 2 * P, **bf)[:, :, :P], torch.empty(S, P, H, **bf).transpose(1, 2),
           torch.empty(1, H, P, **bf).expand(S, H, P)]
    state = d["state"].clone()
    for y in bad:
        with pytest.raises(ValueError, match="y: "):
            T.state_update(*a(state), y=y)
    assert torch.equal(state, d["state"])
    ref = T.state_update(*a(state))
    buf = torch.full((S, H + 1, P), 7.0, **bf)
    y = T.state_update(*a(d["state"].clone()), y=buf[:, :H])
    assert torch.equal(y, ref) and (buf[:, H] == 7.0).all()
