"""Full workload sizes.  (1) Parity against the CPU oracle on SAMPLED batch rows / streams of a full-size launch: rows are
independent, so the oracle evaluates only the sampled rows (seconds of CPU time) while the kernels run the whole problem
and meet everything that only shows at size (many tiles per persistent CTA, ring wrap-around, L2 eviction).
(2) Size-independent properties where the oracle would take minutes: the operator is linear in x, in B and in C separately,
so forward and backward must be adjoint; a sequence may be cut anywhere and resumed from the carried state; batch rows are
independent; chunk-scan prefill followed by single steps equals the full chunk-scan.
Inputs come from the benchmark's generator (`bench.make_inputs`), the one place the workload distributions are drawn on
the device."""
import math

import pytest
import torch
import torch.nn.functional as F

import bench
from oracle import ssd_oracle as O
from tests._util import assert_close, assert_close_dA_few_rows, oracle_all

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CFGS = {"cfg1": bench.CFGS["cfg1"], "cfg3": bench.CFGS["cfg3"], "cfg4_one_gpu": bench.CFGS["cfg4"]}


def draw(c, seed=bench.SEED, L=None, B=None):
    return bench.make_inputs(c, DEV, seed, batch=B, seqlen=L)


def rows_to_cpu(d, rows):
    out = {k: d[k][rows].cpu() for k in ("x", "dt", "B", "C", "dy") + (("z",) if "z" in d else ())}
    out.update(A=d["A"].cpu(), D=d["D"].cpu())
    return out


def oracle_chunked64(inp, grads=True, dfinal=None):
    """fp64 oracle through the chunked evaluation (equal to the sequential form to 1e-10, checked on CPU) for rows too
    long for the per-timestep loops."""
    if not grads:
        y, fin = O.ssd_chunked(inp["x"], inp["dt"], inp["A"], inp["B"], inp["C"], inp["D"], inp.get("z"),
                               inp.get("init_state"), chunk=128, dtype=torch.float64)
        return dict(y=y, final_state=fin)
    return O.ssd_grads_autograd(O.ssd_chunked, inp["x"], inp["dt"], inp["A"], inp["B"], inp["C"], inp["D"], inp["dy"],
                                inp.get("z"), inp.get("init_state"), dfinal, dtype=torch.float64, chunk=128)


def test_cfg1_full_size_sampled_rows_match_oracle(lib):
    """B512 L1024 H8 P32 N64 forward + backward in one launch each; rows 0, 255, 511 against the fp64 oracle.  dA and dD sum
    over the batch, so they are gated on a re-run restricted to the sampled rows, and the full-size values against the sum
    of eight re-runs over a partition of the batch (the sums are linear in the batch)."""
    import trading_bot_0_b200 as T
    c = CFGS["cfg1"]
    d = draw(c)
    rows = [0, 255, 511]
    args = lambda sl: (d["x"][sl], d["dt"][sl], d["A"], d["B"][sl], d["C"][sl], d["D"])
    y, fin, ws = T.forward(*args(slice(None)), chunk=c["Q"], for_backward=True, check=True)
    g = T.backward(d["dy"], *args(slice(None)), chunk=c["Q"], workspace=ws, fwd_saved=True, check=True)
    ref = oracle_all(rows_to_cpu(d, rows))
    assert_close("y", y[rows], ref["y"], "bf16")
    assert_close("final_state", fin[rows], ref["final_state"], "bf16")
    for k in ("dx", "ddt", "dB", "dC"):
        assert_close(k, g[k][rows], ref[k], "bf16")
    gs = T.backward(d["dy"][rows], *args(rows), chunk=c["Q"], check=True)
    for k in ("dA", "dD"):
        assert_close(k + " (sampled rows)", gs[k], ref[k], "bf16")
    parts = [T.backward(d["dy"][i:i + 64], *args(slice(i, i + 64)), chunk=c["Q"]) for i in range(0, c["B"], 64)]
    for k in ("dA", "dD"):
        tot = sum(p[k].double() for p in parts)
        assert rel(g[k], tot) <= 1e-3, (k, g[k], tot)


def test_cfg3_full_size_sampled_row_matches_oracle(lib):
    """B16 L4096 H24 P64 N128 chunk 256 with the y*silu(z) gate; one row against the fp64 oracle, all gradients."""
    import trading_bot_0_b200 as T
    c = CFGS["cfg3"]
    d = draw(c)
    row = [9]
    args = lambda sl: (d["x"][sl], d["dt"][sl], d["A"], d["B"][sl], d["C"][sl], d["D"], d["z"][sl])
    y, fin, ws = T.forward(*args(slice(None)), chunk=c["Q"], for_backward=True, check=True)
    g = T.backward(d["dy"], *args(slice(None)), chunk=c["Q"], workspace=ws, fwd_saved=True, check=True)
    ref = oracle_chunked64(rows_to_cpu(d, row))
    assert_close("y", y[row], ref["y"], "bf16")
    assert_close("final_state", fin[row], ref["final_state"], "bf16")
    for k in ("dx", "ddt", "dB", "dC", "dz"):
        assert_close(k, g[k][row], ref[k], "bf16")
    gs = T.backward(d["dy"][row], *args(row), chunk=c["Q"], check=True)
    assert_close_dA_few_rows("dA (sampled row)", gs["dA"], ref["dA"])
    assert_close("dD (sampled row)", gs["dD"], ref["dD"], "bf16")


def test_cfg4_rank_share_sampled_row_matches_oracle(lib):
    """The long-sequence workload at the share one of eight ranks holds (B2, L 16,384, H24 P64 N128, chunk 256): forward of
    the whole share, row 1 against the fp64 oracle; gradients of a 4,096-token launch of the same shapes, row 0."""
    import trading_bot_0_b200 as T
    c = CFGS["cfg4_one_gpu"]
    d = draw(c, L=16384)
    args = lambda sl, t: (d["x"][sl, :t], d["dt"][sl, :t], d["A"], d["B"][sl, :t], d["C"][sl, :t], d["D"])
    y, fin, ws = T.forward(*args(slice(None), 16384), chunk=c["Q"], check=True)
    inp = rows_to_cpu(d, [1])
    ref = oracle_chunked64(inp, grads=False)
    assert_close("y", y[[1]], ref["y"], "bf16")
    assert_close("final_state", fin[[1]], ref["final_state"], "bf16")
    Lg = 4096
    g = T.backward(d["dy"][:, :Lg], *args(slice(None), Lg), chunk=c["Q"], check=True)
    inp = {k: (v[:, :Lg] if k in ("x", "dt", "B", "C", "dy") else v) for k, v in rows_to_cpu(d, [0]).items()}
    ref = oracle_chunked64(inp)
    for k in ("dx", "ddt", "dB", "dC"):
        assert_close(k, g[k][[0]], ref[k], "bf16")
    gs = T.backward(d["dy"][[0], :Lg], *args([0], Lg), chunk=c["Q"], check=True)
    assert_close_dA_few_rows("dA (sampled row)", gs["dA"], ref["dA"])
    assert_close("dD (sampled row)", gs["dD"], ref["dD"], "bf16")


def test_cfg2_full_width_sampled_streams_match_oracle(lib):
    """8192 streams, 8 consecutive steps with fresh draws; 32 sampled streams against the oracle's one-step update."""
    import trading_bot_0_b200 as T
    cfg = O.CONFIGS[2]
    steps = 8
    dec = O.make_decode_inputs(cfg, steps)
    dd = {k: v.to(DEV) for k, v in dec.items()}
    pick = torch.linspace(0, cfg.batch - 1, 32).long()
    st = T.StreamState(dd["state"].clone())
    S = dec["state"][pick].double()
    for t in range(steps):
        y = st.step(dd["x"][t], dd["dt"][t], dd["A"], dd["B"][t], dd["C"][t], dd["D"])
        yr, S = O.state_update(S, dec["x"][t][pick], dec["dt"][t][pick], dec["A"], dec["B"][t][pick], dec["C"][t][pick], dec["D"])
        assert_close(f"y step {t}", y[pick.to(DEV)], yr, "bf16")
    assert_close("state", st.state[pick.to(DEV)], S, "fp32")


def rel(a, b):
    return float((a.double() - b.double()).abs().max() / (b.double().abs().max() + 1e-30))


@pytest.mark.parametrize("name", ["cfg1", "cfg3", "cfg4_one_gpu"])
def test_forward_backward_are_adjoint(lib, name):
    """<dy, F(v)> == <F^T(dy), v> for the maps x -> y, B -> y and C -> y (ungated, D = 0, so each
    map is exactly linear); bf16 outputs bound the agreement to about 1e-2."""
    import trading_bot_0_b200 as T
    c = CFGS[name]
    d = draw(c)
    g = T.backward(d["dy"], d["x"], d["dt"], d["A"], d["B"], d["C"], None, None, chunk=c["Q"])
    y, _, _ = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], None, None, chunk=c["Q"])
    lhs = float((d["dy"].double() * y.double()).sum())
    for key, grad in (("x", "dx"), ("B", "dB"), ("C", "dC")):
        rhs = float((g[grad].double() * d[key].double()).sum())
        # the bf16 roundings of y and of the gradient are independent with relative size 2^-9 per element: the two sums differ by
        # at most 2^-9 * sqrt(sum of squared terms) in standard deviation; the bound is six of those, relative to the data alone
        terms = (d["dy"].double() * y.double())
        tgrad = (g[grad].double() * d[key].double())
        sigma = 2.0 ** -9 * math.sqrt(float((terms * terms).sum()) + float((tgrad * tgrad).sum()))
        assert abs(lhs - rhs) <= 6.0 * sigma, (name, key, lhs, rhs, sigma)


@pytest.mark.parametrize("name", ["cfg1", "cfg3", "cfg4_one_gpu"])
def test_cut_and_resume_from_carried_state(lib, name):
    import trading_bot_0_b200 as T
    c = CFGS[name]
    d = draw(c)
    z = d.get("z")
    y, fin, _ = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], z, chunk=c["Q"])
    k = c["L"] // 2
    cut = lambda t, a, b: None if t is None else t[:, a:b]
    y1, s1, _ = T.forward(cut(d["x"], 0, k), cut(d["dt"], 0, k), d["A"], cut(d["B"], 0, k), cut(d["C"], 0, k), d["D"],
                          cut(z, 0, k), chunk=c["Q"])
    y2, s2, _ = T.forward(cut(d["x"], k, None), cut(d["dt"], k, None), d["A"], cut(d["B"], k, None),
                          cut(d["C"], k, None), d["D"], cut(z, k, None), s1, chunk=c["Q"])
    assert torch.equal(y[:, :k], y1)
    assert (y[:, k:].float() - y2.float()).abs().max().item() <= 2e-2 * max(1.0, y.float().abs().max().item())
    assert rel(s2, fin) <= 1e-3


@pytest.mark.parametrize("name,B,L", [("cfg1", 128, 1024), ("cfg3", 4, 4096), ("cfg4_one_gpu", 2, 16384)])
def test_repeated_runs_are_bit_identical(lib, name, B, L):
    """Every kernel adds in a fixed order, so a second and a third run over the same buffers must reproduce every output
    bit for bit; a hand-off that lets a consumer read a buffer before it has fully arrived shows up here as a difference."""
    import trading_bot_0_b200 as T
    c = CFGS[name]
    d = draw(c, L=L, B=B)
    z = d.get("z")

    def run():
        y, fin, ws = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], z, chunk=c["Q"], for_backward=True)
        g = T.backward(d["dy"], d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], z, chunk=c["Q"], workspace=ws, fwd_saved=True)
        torch.cuda.synchronize()
        return dict(y=y.clone(), fin=fin.clone(), **{k: v.clone() for k, v in g.items() if isinstance(v, torch.Tensor) and k != "workspace"})

    first = run()
    for _ in range(3):
        again = run()
        for k, v in first.items():
            assert torch.equal(v, again[k]), k


@pytest.mark.parametrize("name,B,lengths", [("cfg4_one_gpu", 2, (65536, 16384)), ("cfg1", 128, (1024, 512))])
def test_forward_is_bit_stable_between_other_launches(lib, name, B, lengths):
    """A few hundred forwards of two lengths, a forward + backward of another shape between every third pair, each output
    compared bit for bit with the first run of its length.  With one tile per CTA the whole pass is the start-up of the
    persistent kernels' rings, where a wait that a role passes one phase early shows as a few wrong rows of one head about
    once in a hundred launches: a table ring shared between decay groups did exactly that at the shorter cfg4 length."""
    import trading_bot_0_b200 as T
    c = CFGS[name]
    d = draw(c, L=max(lengths), B=B)
    o = draw(CFGS["cfg3"], L=2048, B=2, seed=7)

    def fwd(L):
        cut = lambda t: t[:, :L]
        return T.forward(cut(d["x"]), cut(d["dt"]), d["A"], cut(d["B"]), cut(d["C"]), d["D"], None, chunk=c["Q"])[0]

    def other():
        y, _, ws = T.forward(o["x"], o["dt"], o["A"], o["B"], o["C"], o["D"], o["z"], chunk=256, for_backward=True)
        T.backward(o["dy"], o["x"], o["dt"], o["A"], o["B"], o["C"], o["D"], o["z"], chunk=256, workspace=ws, fwd_saved=True)

    first = {L: fwd(L).clone() for L in lengths}
    for it in range(200):
        if it % 3 == 0:
            other()
        for L in lengths:
            y = fwd(L)
            assert torch.equal(y, first[L]), f"iteration {it}, length {L}: {int((y != first[L]).sum())} outputs differ"


def test_batch_rows_are_independent(lib):
    import trading_bot_0_b200 as T
    c = CFGS["cfg1"]
    d = draw(c)
    y, fin, _ = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], chunk=c["Q"])
    sl = slice(100, 108)
    ys, fs, _ = T.forward(d["x"][sl], d["dt"][sl], d["A"], d["B"][sl], d["C"][sl], d["D"], chunk=c["Q"])
    assert torch.equal(y[sl], ys) and torch.equal(fin[sl], fs)
    g = T.backward(d["dy"], d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], chunk=c["Q"])
    gs = T.backward(d["dy"][sl], d["x"][sl], d["dt"][sl], d["A"], d["B"][sl], d["C"][sl], d["D"], chunk=c["Q"])
    for k in ("dx", "ddt", "dB", "dC"):
        assert torch.equal(g[k][sl], gs[k]), k


@pytest.mark.parametrize("H,P,N,G,L,rows", [
    (24, 64, 128, 1, 17 * 128, (1, 4, 8, 14)),         # 12 units a row: two kernels, with few and many blocks; walks; even shares
    (8, 32, 64, 1, 40 * 128 + 70, (1, 50, 90)),        # 2 units a row: the same three, a ragged last chunk
    (24, 64, 128, 1, 40 * 128, (2, 6, 13)),
    (8, 32, 128, 2, 3 * 128, (1, 45, 100)),
    (4, 32, 64, 1, 200 * 128 + 5, (1, 90, 180)),       # long ones
    (2, 64, 128, 1, 300 * 128, (1, 70)),
])
def test_row_bits_do_not_depend_on_the_batch(lib, H, P, N, G, L, rows):
    """The state scans are run in another way for few rows, for about as many units as SMs, and for more; a row's results are
    the same bits in each, with states entering at both ends."""
    import trading_bot_0_b200 as T
    B = max(rows)
    d = bench.make_inputs(dict(bench.CFGS["cfg1"], H=H, P=P, N=N, G=G, Q=128), DEV, 11, batch=B, seqlen=L)
    g = torch.Generator(device=DEV).manual_seed(5)
    init, dfin = (0.1 * torch.randn(B, H, P, N, generator=g, device=DEV) for _ in range(2))

    def run(n):   # the last n rows
        s = slice(B - n, B)
        a = (d["x"][s], d["dt"][s], d["A"], d["B"][s], d["C"][s], d["D"], None, init[s])
        y, fin, ws = T.forward(*a, chunk=128, for_backward=True, check=True)
        o = T.backward(d["dy"][s], *a, dfin[s], chunk=128, workspace=ws, fwd_saved=True, check=True)
        return {"y": y, "final_state": fin, **{k: o[k] for k in ("dx", "ddt", "dB", "dC", "dinit")}}

    whole = run(B)
    for n in rows[:-1]:
        part = run(n)
        for k, v in part.items():
            assert torch.equal(whole[k][B - n:], v), (n, k)


@pytest.mark.parametrize("H,P,N,L,cut", [(8, 32, 64, 60 * 128, 7), (24, 64, 128, 300 * 128, 150), (2, 64, 128, 300 * 128, 1)])
def test_prefix_bits_do_not_depend_on_the_length(lib, H, P, N, L, cut):
    """The state scans run a short and a long sequence in different ways; the outputs of the first chunks are the same bits."""
    import trading_bot_0_b200 as T
    d = bench.make_inputs(dict(bench.CFGS["cfg1"], H=H, P=P, N=N), DEV, 13, batch=1, seqlen=L)
    y = [T.forward(d["x"][:, :n], d["dt"][:, :n], d["A"], d["B"][:, :n], d["C"][:, :n], d["D"], chunk=128)[0] for n in (L, cut * 128)]
    assert torch.equal(y[0][:, :cut * 128], y[1])


@pytest.mark.parametrize("H,P,N,L", [(4, 32, 64, 256 * 128), (2, 64, 128, 300 * 128)])
def test_long_sequences_match_oracle(lib, H, P, N, L):
    """A few rows of several hundred chunks, states entering at both ends: the first row against the fp64 oracle."""
    import trading_bot_0_b200 as T
    d = bench.make_inputs(dict(bench.CFGS["cfg1"], H=H, P=P, N=N), DEV, 12, batch=3, seqlen=L)
    g = torch.Generator(device=DEV).manual_seed(6)
    init, dfin = (0.1 * torch.randn(3, H, P, N, generator=g, device=DEV) for _ in range(2))
    a = (d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], None, init)
    y, fin, ws = T.forward(*a, chunk=128, for_backward=True, check=True)
    o = T.backward(d["dy"], *a, dfin, chunk=128, workspace=ws, fwd_saved=True, check=True)
    ref = oracle_chunked64(dict(rows_to_cpu(d, [0]), init_state=init[:1].cpu()), dfinal=dfin[:1].cpu())
    for k, v in (("y", y), ("final_state", fin), *((k, o[k]) for k in ("dx", "ddt", "dB", "dC", "dinit"))):
        assert_close(k, v[:1], ref[k], "bf16")


def test_prefill_then_steps_at_full_batch(lib):
    """cfg1 batch: chunk-scan over 896 tokens, then 128 single steps over all 512 x 8 states, against
    the chunk-scan over all 1024 tokens."""
    import trading_bot_0_b200 as T
    c = CFGS["cfg1"]
    d = draw(c)
    y, fin, _ = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], chunk=c["Q"])
    k = 896
    _, s, _ = T.forward(d["x"][:, :k], d["dt"][:, :k], d["A"], d["B"][:, :k], d["C"][:, :k], d["D"], chunk=c["Q"])
    st = T.StreamState(s)
    worst = 0.0
    for t in range(k, c["L"]):
        yt = st.step(d["x"][:, t], d["dt"][:, t], d["A"], d["B"][:, t], d["C"][:, t], d["D"])
        worst = max(worst, (yt.float() - y[:, t].float()).abs().max().item())
    assert worst <= 2e-2 * max(1.0, y[:, k:].float().abs().max().item())   # the bf16 gate, scaled like every other use of it
    assert rel(st.state, fin) <= 1e-3


def test_decode_full_rollout_width(lib):
    """8192 streams: one batched step equals the same step done in two halves (stream sharding)."""
    import trading_bot_0_b200 as T
    g = torch.Generator(device=DEV).manual_seed(3)
    S, H, P, N = 8192, 8, 32, 64
    st = 0.1 * torch.randn(S, H, P, N, generator=g, device=DEV)
    x = torch.randn(S, H, P, generator=g, device=DEV).bfloat16()
    dt = F.softplus(torch.randn(S, H, generator=g, device=DEV) - 3).bfloat16()
    A = -torch.exp(torch.rand(H, generator=g, device=DEV) * math.log(16.0))
    Bm = (torch.randn(S, 1, N, generator=g, device=DEV) / 8).bfloat16()
    Cm = (torch.randn(S, 1, N, generator=g, device=DEV) / 8).bfloat16()
    full = st.clone()
    y = T.state_update(full, x, dt, A, Bm, Cm, torch.ones(H, device=DEV))
    halves = [st[:4096].clone(), st[4096:].clone()]
    ys = [T.state_update(halves[i], x[i * 4096:(i + 1) * 4096], dt[i * 4096:(i + 1) * 4096], A,
                         Bm[i * 4096:(i + 1) * 4096], Cm[i * 4096:(i + 1) * 4096], torch.ones(H, device=DEV)) for i in range(2)]
    assert torch.equal(y, torch.cat(ys)) and torch.equal(full, torch.cat(halves))
