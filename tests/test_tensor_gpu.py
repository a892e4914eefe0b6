"""Parity of the tcgen05 tensor-core kernels (bf16 storage, chunk 128) against the CPU oracle,
and against the exact-fp32 CUDA-core family on the same inputs."""
import pytest
import torch

from oracle import ssd_oracle as O
from tests._util import assert_close, assert_close_dA_few_rows, mean_rel, oracle_all, to_dev

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GRADS = ("dx", "ddt", "dA", "dB", "dC")


def status_word(ws):
    return int(ws[:4].view(torch.int32).item())


@pytest.mark.parametrize("H,P,N,G", [(8, 32, 64, 1), (24, 64, 128, 1), (8, 32, 128, 2), (4, 64, 64, 2)])
@pytest.mark.parametrize("has_z,use_D,with_state", [(False, True, False), (True, True, True), (False, False, True)])
def test_tensor_forward_backward_matches_oracle(lib, H, P, N, G, has_z, use_D, with_state):
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("tc", 3, 384, H, P, N, G, 128, "bf16", has_z)
    inp = O.make_inputs(cfg, with_init_state=with_state)
    if not use_D:
        inp["D"] = None
    # gradient entering the final state at the magnitude of the state itself (N(0, 0.1)): dA sums
    # strongly cancelling terms, so an O(1) dfinal only amplifies bf16 rounding of the chunk states
    dfinal = 0.1 * torch.randn(3, H, P, N, generator=torch.Generator().manual_seed(4)) if with_state else None
    ref = oracle_all(inp, dfinal)
    d = to_dev(inp, DEV)
    y, fin, ws = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d.get("D"), d.get("z"), d.get("init_state"),
                           chunk=128, algo="tensor", for_backward=True)
    torch.cuda.synchronize()
    assert status_word(ws) == 0, f"kernel status {status_word(ws)}"
    assert_close("y", y, ref["y"], "bf16")
    assert_close("final_state", fin, ref["final_state"], "bf16")
    g = T.backward(d["dy"], d["x"], d["dt"], d["A"], d["B"], d["C"], d.get("D"), d.get("z"), d.get("init_state"),
                   None if dfinal is None else dfinal.to(DEV), chunk=128, algo="tensor", workspace=ws,
                   fwd_saved=True, want_dinit=True)
    torch.cuda.synchronize()
    assert status_word(ws) == 0
    for k in GRADS + ("dinit",) + (("dD",) if use_D else ()) + (("dz",) if has_z else ()):
        assert_close(k, g[k], ref[k], "bf16")
    # recompute path (no saved forward) gives the same gradients
    g2 = T.backward(d["dy"], d["x"], d["dt"], d["A"], d["B"], d["C"], d.get("D"), d.get("z"), d.get("init_state"),
                    None if dfinal is None else dfinal.to(DEV), chunk=128, algo="tensor", want_dinit=True)
    for k in GRADS:
        assert_close(k + " (recompute)", g2[k], ref[k], "bf16")


@pytest.mark.parametrize("H,P,N,G", [(8, 32, 64, 1), (24, 64, 128, 1), (8, 32, 128, 2), (4, 64, 64, 2)])
@pytest.mark.parametrize("has_z", [False, True])
def test_one_tile_arm_matches_oracle(lib, H, P, N, G, has_z):
    """The one-tile-per-CTA kernels (algo = tensor_onetile), which the default path no longer reaches except for the merged
    backward and dB/dC at dstate 128: same gates as the persistent kernels."""
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("tc", 3, 384, H, P, N, G, 128, "bf16", has_z)
    inp = O.make_inputs(cfg, with_init_state=True)
    dfinal = 0.1 * torch.randn(3, H, P, N, generator=torch.Generator().manual_seed(4))
    ref = oracle_all(inp, dfinal)
    d = to_dev(inp, DEV)
    y, fin, ws = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d.get("D"), d.get("z"), d.get("init_state"),
                           chunk=128, algo="tensor_onetile", for_backward=True)
    g = T.backward(d["dy"], d["x"], d["dt"], d["A"], d["B"], d["C"], d.get("D"), d.get("z"), d.get("init_state"),
                   dfinal.to(DEV), chunk=128, algo="tensor_onetile", workspace=ws, fwd_saved=True, want_dinit=True)
    torch.cuda.synchronize()
    assert status_word(ws) == 0
    assert_close("y", y, ref["y"], "bf16")
    assert_close("final_state", fin, ref["final_state"], "bf16")
    for k in GRADS + ("dinit", "dD") + (("dz",) if has_z else ()):
        assert_close(k, g[k], ref[k], "bf16")


def test_tensor_matches_cuda_core_family(lib):
    """Same bf16 inputs through both kernel families: outputs agree to bf16 rounding."""
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("tc", 4, 512, 8, 32, 64, 1, 128, "bf16")
    d = to_dev(O.make_inputs(cfg, with_init_state=True), DEV)
    outs = {}
    for algo in ("tensor", "fp32_cores"):
        y, fin, ws = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], None, None, d["init_state"], chunk=128, algo=algo)
        outs[algo] = (y.float(), fin)
    assert mean_rel(outs["tensor"][0], outs["fp32_cores"][0]) < 1e-2
    assert mean_rel(outs["tensor"][1], outs["fp32_cores"][1]) < 5e-3


def test_tensor_strided_inputs(lib):
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("tc", 2, 256, 8, 32, 64, 1, 128, "bf16")
    inp = to_dev(O.make_inputs(cfg), DEV)
    views = {}
    for k in ("x", "dt", "B", "C"):
        v = inp[k]
        buf = torch.zeros(v.shape[0] + 1, v.shape[1] + 8, *v.shape[2:], dtype=v.dtype, device=DEV)
        views[k] = buf[1:, 8:8 + cfg.seqlen]
        views[k].copy_(v)
    y0, f0, _ = T.forward(inp["x"], inp["dt"], inp["A"], inp["B"], inp["C"], inp["D"], chunk=128, algo="tensor")
    y1, f1, _ = T.forward(views["x"], views["dt"], inp["A"], views["B"], views["C"], inp["D"], chunk=128, algo="tensor")
    assert torch.equal(y0, y1) and torch.equal(f0, f1)


def test_tensor_request_on_unsupported_dims_is_an_error(lib):
    import trading_bot_0_b200 as T
    from trading_bot_0_b200 import _lib as L
    cfg = O.SsdConfig("tc", 1, 128, 4, 32, 16, 1, 64, "bf16")
    d = to_dev(O.make_inputs(cfg), DEV)
    with pytest.raises(L.SsdError) as ei:
        T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], chunk=64, algo="tensor")
    assert ei.value.code == -3


def test_chunk_256_runs_on_the_tensor_family_as_two_128_chunks(lib):
    """The 130M-layer and long-sequence workloads ask for chunk 256; the result must not depend on it."""
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("tc256", 2, 512, 24, 64, 128, 1, 256, "bf16", True)
    inp = O.make_inputs(cfg, with_init_state=True)
    ref = oracle_all(inp)
    d = to_dev(inp, DEV)
    y, fin, ws = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], d["z"], d["init_state"], chunk=256,
                           algo="tensor", for_backward=True)
    g = T.backward(d["dy"], d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], d["z"], d["init_state"], chunk=256,
                   algo="tensor", workspace=ws, fwd_saved=True, want_dinit=True)
    torch.cuda.synchronize()
    assert status_word(ws) == 0
    assert_close("y", y, ref["y"], "bf16")
    assert_close("final_state", fin, ref["final_state"], "bf16")
    for k in GRADS + ("dD", "dz", "dinit"):
        assert_close(k, g[k], ref[k], "bf16")
    y128, _, _ = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], d["z"], d["init_state"], chunk=128, algo="tensor")
    assert torch.equal(y, y128)


@pytest.mark.parametrize("Bn,L,H,P,G", [(1, 128, 8, 32, 1), (3, 1280, 4, 64, 2), (2, 384, 16, 32, 2), (50, 256, 8, 32, 1)])
def test_fused_state_scan_matches_the_staged_two_kernel_path(lib, Bn, L, H, P, G):
    """A full pass at dstate 64 computes the chunk states inside the scan over chunks (one kernel per pass, running state
    in registers: one chunk, or 100 units of the last case) or, for few units, folds them in a kernel of its own; the staged entry points (sequence-parallel callers) keep chunk-state kernel + scan kernel.  Same inputs,
    both ways, incl. one chunk only, fewer units than SMs, an initial state and a gradient entering the final state:
    results agree to fp32 rounding of the chunk decay (exp2 of the table value against expf of the cumsum) and both match
    the oracle."""
    import trading_bot_0_b200 as T
    from trading_bot_0_b200 import _lib as LL
    cfg = O.SsdConfig("fs", Bn, L, H, P, 64, G, 128, "bf16", False)
    inp = O.make_inputs(cfg, with_init_state=True)
    dfinal = 0.1 * torch.randn(Bn, H, P, 64, generator=torch.Generator().manual_seed(8))
    ref = oracle_all(inp, dfinal)
    d = to_dev(inp, DEV)
    args = (d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], None, d["init_state"])
    res = {}
    for name, stage_list in (("fused", [None]), ("staged", [LL.STAGE_LOCAL, LL.STAGE_FINISH])):
        ws = y = fin = None
        for st in stage_list:
            y, fin, ws = T.forward(*args, chunk=128, algo="tensor", for_backward=True, stages=st, workspace=ws, y=y, final_state=fin)
        g = None
        for st in stage_list:
            g = T.backward(d["dy"], *args, dfinal.to(DEV), chunk=128, algo="tensor", workspace=ws, fwd_saved=True,
                           want_dinit=True, stages=st, out=g)
        torch.cuda.synchronize()
        assert status_word(ws) == 0
        res[name] = dict(y=y, final_state=fin, **{k: g[k] for k in GRADS + ("dD", "dinit")})
    for k, v in res["fused"].items():
        if k == "dA":   # a sum over all tokens of terms that mostly cancel: gated at 6e-2 of its largest entry on these small cases
            for w in (v, res["staged"][k]):
                assert (w.double().cpu() - ref[k]).abs().max() <= 6e-2 * ref[k].abs().max()
        else:
            assert_close(k + " (fused)", v, ref[k], "bf16")
            assert_close(k + " (staged)", res["staged"][k], ref[k], "bf16")
        tol = 2e-2 if k == "dA" else 2e-3
        assert mean_rel(v, res["staged"][k]) < tol, f"{k}: fused and staged paths differ by {mean_rel(v, res['staged'][k]):.3e}"


@pytest.mark.parametrize("L", [1, 100, 129, 255, 383, 641])
@pytest.mark.parametrize("H,P,N,G,has_z", [(8, 32, 64, 1, False), (4, 64, 64, 2, True), (24, 64, 128, 1, True), (8, 32, 128, 2, False)])
def test_ragged_forward_runs_on_the_tensor_family(lib, L, H, P, N, G, has_z):
    """A forward without a backward takes any sequence length: the last chunk's loads zero-fill, its stores drop the rows past
    the end (the neighbouring batch row and the guard rows stay untouched)."""
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("rag", 2, L, H, P, N, G, 128, "bf16", has_z)
    inp = O.make_inputs(cfg, with_init_state=True)
    y_ref, fin_ref = O.ssd_sequential(inp["x"], inp["dt"], inp["A"], inp["B"], inp["C"], inp["D"], inp.get("z"), inp["init_state"])
    d = to_dev(inp, DEV)
    buf = torch.full((2, L + 3, H, P), 7.0, dtype=torch.bfloat16, device=DEV)
    y, fin, ws = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], d.get("z"), d["init_state"], chunk=128, algo="tensor",
                           y=buf[:, :L])
    assert status_word(ws) == 0
    assert_close("y", y, y_ref, "bf16")
    assert_close("final_state", fin, fin_ref, "bf16")
    assert (buf[:, L:] == 7.0).all()


@pytest.mark.parametrize("L", [1, 100, 129, 383])
@pytest.mark.parametrize("H,P,N,G,has_z", [(8, 32, 64, 1, False), (4, 64, 64, 2, True), (24, 64, 128, 1, True), (8, 32, 128, 2, False)])
def test_ragged_training_runs_on_the_tensor_family(lib, L, H, P, N, G, has_z):
    """Forward and backward of any sequence length: outputs of one batch row stop at its end, padded positions add nothing."""
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("rag", 3, L, H, P, N, G, 128, "bf16", has_z)
    inp = O.make_inputs(cfg, with_init_state=True)
    ref = oracle_all(inp)
    d = to_dev(inp, DEV)
    a = (d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], d.get("z"), d["init_state"])
    y, fin, ws = T.forward(*a, chunk=128, algo="tensor", for_backward=True)
    g = T.backward(d["dy"], *a, chunk=128, algo="tensor", workspace=ws, fwd_saved=True, want_dinit=True)
    torch.cuda.synchronize()
    assert status_word(ws) == 0
    assert_close("y", y, ref["y"], "bf16")
    for k in ("dx", "ddt", "dB", "dC", "dD", "dinit") + (("dz",) if has_z else ()):
        assert_close(k, g[k], ref[k], "bf16")
    assert_close_dA_few_rows("dA", g["dA"], ref["dA"])


@pytest.mark.parametrize("which", ["y", "dy", "both", "x"])
@pytest.mark.parametrize("N", [64, 128])
def test_ragged_operands_of_any_alignment(lib, which, N):
    """algo = auto on a ragged sequence takes pointers that TMA cannot address: y goes through the workspace, a backward with
    such a dy recomputes on the CUDA cores, a shared operand moves both passes there."""
    import trading_bot_0_b200 as T
    cfg = O.SsdConfig("al", 2, 200, 8, 32, N, 1, 128, "bf16")
    inp = O.make_inputs(cfg, with_init_state=True)
    ref = oracle_all(inp)
    d = to_dev(inp, DEV)

    def off(t):
        v = torch.zeros(t.numel() + 8, dtype=t.dtype, device=DEV)[3:3 + t.numel()].view_as(t)
        v.copy_(t)
        return v

    x = off(d["x"]) if which == "x" else d["x"]
    a = (x, d["dt"], d["A"], d["B"], d["C"], d["D"], None, d["init_state"])
    y_out = off(torch.zeros_like(d["x"])) if which in ("y", "both") else None
    y, fin, ws = T.forward(*a, chunk=128, for_backward=True, y=y_out)
    dy = off(d["dy"]) if which in ("dy", "both") else d["dy"]
    g = T.backward(dy, *a, chunk=128, workspace=ws, fwd_saved=True, want_dinit=True)
    assert_close("y", y, ref["y"], "bf16")
    assert_close("final_state", fin, ref["final_state"], "bf16")
    for k in ("dx", "ddt", "dB", "dC", "dD", "dinit"):
        assert_close(k, g[k], ref[k], "bf16")


@pytest.mark.parametrize("L", [1921, 2304, 4200])
@pytest.mark.parametrize("H,P,N,G", [(8, 32, 64, 1), (4, 64, 128, 2), (12, 64, 128, 1)])
def test_segmented_state_scan_matches_oracle(lib, L, H, P, N, G):
    """Few units and many chunks: the state scans run as two kernels (a last chunk of one token, fewer and more chunks than the
    fold requests at once)."""
    import trading_bot_0_b200 as T
    Bn = 2
    cfg = O.SsdConfig("seg", Bn, L, H, P, N, G, 128, "bf16", False)
    inp = O.make_inputs(cfg, with_init_state=True)
    dfinal = 0.1 * torch.randn(Bn, H, P, N, generator=torch.Generator().manual_seed(4))
    ref = oracle_all(inp, dfinal)
    d = to_dev(inp, DEV)
    y, fin, ws = T.forward(d["x"], d["dt"], d["A"], d["B"], d["C"], d.get("D"), None, d["init_state"], chunk=128, for_backward=True)
    g = T.backward(d["dy"], d["x"], d["dt"], d["A"], d["B"], d["C"], d.get("D"), None, d["init_state"], dfinal.to(DEV),
                   chunk=128, workspace=ws, fwd_saved=True, want_dinit=True)
    torch.cuda.synchronize()
    assert status_word(ws) == 0
    assert_close("y", y, ref["y"], "bf16")
    assert_close("final_state", fin, ref["final_state"], "bf16")
    for k in GRADS + ("dinit",):
        if k == "dA":
            assert_close_dA_few_rows(k, g[k], ref[k])
        else:
            assert_close(k, g[k], ref[k], "bf16")


@pytest.mark.parametrize("H,P,N,G,Bn", [(6, 64, 64, 1, 35), (18, 64, 128, 1, 40), (12, 32, 64, 1, 60)])
@pytest.mark.parametrize("has_z", [False, True])
def test_split_heads_are_the_same_bits(lib, H, P, N, G, Bn, has_z):
    """The scan kernels cut a group's heads into parts by the number of tiles: a few rows alone (many parts) match the oracle,
    and the rows of a larger batch (fewer parts, an odd number of head blocks in each) match them bit for bit."""
    import trading_bot_0_b200 as T
    inp = O.make_inputs(O.SsdConfig("split", Bn, 256, H, P, N, G, 128, "bf16", has_z))
    per_row = ("x", "dt", "B", "C", "z", "dy")

    def run(v):
        d = to_dev(v, DEV)
        a = (d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], d.get("z"))
        y, _, ws = T.forward(*a, chunk=128, algo="tensor", for_backward=True)
        g = T.backward(d["dy"], *a, chunk=128, algo="tensor", workspace=ws, fwd_saved=True)
        torch.cuda.synchronize()
        assert status_word(ws) == 0
        return {"y": y, **g}

    few = {k: (v[:2].contiguous() if k in per_row and v is not None else v) for k, v in inp.items()}
    got, ref, whole = run(few), oracle_all(few), run(inp)
    for k in ("y", "dx", "ddt", "dB", "dC") + (("dz",) if has_z else ()):
        assert_close(k, got[k], ref[k], "bf16")
        assert torch.equal(got[k], whole[k][:2]), k


@pytest.mark.parametrize("H,P,N,Bn,L", [(24, 64, 128, 14, 1100), (8, 32, 64, 80, 1700)])
def test_balanced_state_scan_is_the_same_bits(lib, H, P, N, Bn, L):
    """More units than SMs and a last wave far from full: units are cut between neighbouring blocks, which hand the running
    state over.  A row's results are those of the row in a small batch, again and again over one forward."""
    import trading_bot_0_b200 as T
    inp = O.make_inputs(O.SsdConfig("bal", Bn, L, H, P, N, 1, 128, "bf16", False), with_init_state=True)
    dfinal = 0.1 * torch.randn(Bn, H, P, N, generator=torch.Generator().manual_seed(4))
    d = to_dev(inp, DEV)

    def run(rows, times):
        a = (d["x"][rows], d["dt"][rows], d["A"], d["B"][rows], d["C"][rows], d["D"], None, d["init_state"][rows])
        y, fin, ws = T.forward(*a, chunk=128, algo="tensor", for_backward=True)
        for _ in range(times):
            g = T.backward(d["dy"][rows], *a, dfinal[rows].to(DEV), chunk=128, algo="tensor", workspace=ws, fwd_saved=True,
                           want_dinit=True)
        torch.cuda.synchronize()
        assert status_word(ws) == 0
        return {"y": y, "final_state": fin, **g}

    whole = run(slice(0, Bn), 3)
    for r in range(0, Bn, max(1, Bn // 10)):
        row = run(slice(r, r + 1), 1)
        for k in ("y", "final_state", "dx", "ddt", "dB", "dC", "dinit"):
            assert torch.equal(whole[k][r:r + 1], row[k]), (k, r)


@pytest.mark.parametrize("H,P,N,G,Bn", [(8, 32, 64, 1, 75), (8, 32, 128, 2, 92)])
def test_more_units_than_sms_and_many_chunks(lib, H, P, N, G, Bn):
    """150 and 184 units of 88 chunks (a last chunk of 64 tokens): even shares and no segments.  The first and the last row
    against the oracle, final state and the gradients of both states included."""
    import trading_bot_0_b200 as T
    L = 87 * 128 + 64
    inp = O.make_inputs(O.SsdConfig("many", Bn, L, H, P, N, G, 128, "bf16", False), with_init_state=True)
    dfinal = 0.1 * torch.randn(Bn, H, P, N, generator=torch.Generator().manual_seed(4))
    d = to_dev(inp, DEV)
    a = (d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], None, d["init_state"])
    y, fin, ws = T.forward(*a, chunk=128, algo="tensor", for_backward=True)
    g = T.backward(d["dy"], *a, dfinal.to(DEV), chunk=128, algo="tensor", workspace=ws, fwd_saved=True, want_dinit=True)
    torch.cuda.synchronize()
    assert status_word(ws) == 0
    for r in (0, Bn - 1):
        row = {k: (v[r:r + 1] if k in ("x", "dt", "B", "C", "dy", "init_state") else v) for k, v in inp.items()}
        ref = oracle_all(row, dfinal[r:r + 1])
        for k, v in (("y", y), ("final_state", fin), *((k, g[k]) for k in ("dx", "ddt", "dB", "dC", "dinit"))):
            assert_close(k, v[r:r + 1], ref[k], "bf16")


def block_errors(v, w, tokens=32):
    """2-norm of the difference over the 2-norm of the reference, for every block of `tokens` rows of one batch row and one head (or
    group); blocks whose reference is small are held to the average block's norm."""
    B, L = v.shape[:2]
    pad = -L % tokens

    def blocks(t):
        t = torch.nn.functional.pad(t.double().reshape(B, L, v.shape[2], -1), (0, 0, 0, 0, 0, pad))
        return t.view(B, (L + pad) // tokens, tokens, v.shape[2], -1).square().sum((2, 4))

    ref = blocks(w)
    return (blocks(v.double() - w.double()) / torch.maximum(ref, ref.mean())).sqrt()


@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("H,P,N,B,L", [
    (2, 64, 128, 200, 512), (4, 64, 128, 200, 475), (6, 64, 128, 40, 512), (10, 64, 128, 150, 512), (10, 64, 128, 150, 475), (12, 64, 128, 200, 512),
    (4, 32, 128, 200, 475), (12, 32, 128, 200, 512), (4, 32, 64, 200, 475), (12, 32, 64, 200, 512), (2, 64, 64, 200, 475), (6, 64, 64, 200, 512)])
def test_rings_at_tile_ends(lib, H, P, N, B, L, gate):
    """Five tiles and more per block (40 rows: two or three), of two to twelve head blocks each - 150 rows of 10 heads run as two parts of five
    blocks, 40 rows of 6 as two parts of three - in whole and in ragged chunks: slots that a tile lends out, pieces and rings that end in
    the middle of a tile, every barrier used many times over.  Against the one-tile kernels, which have no rings, block by block of 32
    rows of a head: a wrong block is off by about its own norm, two roundings of the bf16 operands of a sum (2^-9 each) by less than a
    hundredth.  And twice with the same bits."""
    import trading_bot_0_b200 as T
    bf, Lp = torch.bfloat16, L + -L % 128
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    A = -torch.exp(2 * torch.rand(H, generator=g, device="cuda"))
    seq = [r(B, Lp, H, P).to(bf), torch.nn.functional.softplus(r(B, Lp, H) - 2).to(bf), (r(B, Lp, 1, N) / N ** 0.5).to(bf),
           (r(B, Lp, 1, N) / N ** 0.5).to(bf), r(B, Lp, H, P).to(bf) if gate else None, r(B, Lp, H, P).to(bf)]
    for v in seq:   # the one-tile kernels take whole chunks only: steps of size zero behind the end
        if v is not None:
            v[:, L:] = 0
    out = []
    for algo, n in (("tensor", L), ("tensor", L), ("tensor_onetile", Lp)):
        x, dt, Bm, Cm, z, dy = (v if v is None else v[:, :n].contiguous() for v in seq)
        a = (x, dt, A, Bm, Cm, torch.ones(H, device="cuda"), z)
        y, fin, ws = T.forward(*a, chunk=128, algo=algo, for_backward=True)
        o = T.backward(dy, *a, chunk=128, algo=algo, workspace=ws, fwd_saved=True)
        torch.cuda.synchronize()
        assert status_word(ws) == 0
        keys = ("dx", "ddt", "dB", "dC") + (("dz",) if gate else ())
        out.append({"y": y[:, :L], **{k: o[k][:, :L] for k in keys}, "fin": fin, "dA": o["dA"], "dD": o["dD"]})
    for k, v in out[0].items():
        assert torch.equal(v, out[1][k]), k
        if k not in ("fin", "dA", "dD"):
            e = float(block_errors(v, out[2][k]).max())
            assert e < 5e-2, (k, e)


@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("H,P,N", [(8, 32, 64), (4, 64, 128)])
def test_large_steps_next_to_the_diagonal(lib, H, P, N, gate):
    """A fifth of the steps are state resets, so that a chunk's running sum grows to 2e5 and rounds by a hundredth: decays next to the
    diagonal have to come from the steps.  Errors against fp64 are those of the one-tile kernels, which walk by steps from the diagonal
    on; the persistent ones start every eight columns from the running sum (0.02-0.04 more); with each element taken from the running
    sums it would be 0.2-0.4."""
    import trading_bot_0_b200 as T
    B, L, bf = 2, 384, torch.bfloat16
    g = torch.Generator().manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g)
    dt = torch.where(torch.rand(B, L, H, generator=g) < 0.2, torch.tensor(300.0), torch.nn.functional.softplus(r(B, L, H) - 3)).to(bf)
    inp = dict(x=(r(B, L, H, P) / dt.float().clamp(min=1).unsqueeze(-1)).to(bf), dt=dt, A=torch.full((H,), -16.0), B=(r(B, L, 1, N) / N ** 0.5).to(bf),
               C=(r(B, L, 1, N) / N ** 0.5).to(bf), D=torch.zeros(H), dy=r(B, L, H, P).to(bf), z=r(B, L, H, P).to(bf) if gate else None)
    ref = oracle_all(inp)
    d = to_dev(inp, DEV)
    a = (d["x"], d["dt"], d["A"], d["B"], d["C"], d["D"], d["z"])
    err = []
    for algo in ("tensor", "tensor_onetile"):
        y, _, ws = T.forward(*a, chunk=128, algo=algo, for_backward=True)
        o = T.backward(d["dy"], *a, chunk=128, algo=algo, workspace=ws, fwd_saved=True)
        out = {"y": y, "dx": o["dx"], **({"dz": o["dz"]} if gate else {})}
        err.append({k: float((v.double().cpu() - ref[k]).norm() / ref[k].norm()) for k, v in out.items()})
    for k, e in err[0].items():
        assert e < 1.07 * err[1][k], (k, e, err[1][k])
