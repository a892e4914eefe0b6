"""The operators either side of the scan in a Mamba-2 layer: causal depthwise conv1d (+ silu) over the
(x | B | C) channels before it, RMS norm of the gated output after it, each with its backward, plus a
differentiable composition of the whole mixer core (`mamba2_mixer_core`).

The step-size activation softplus(dt + dt_bias) and the gate y * silu(z) are not here: they run inside
the scan's own kernels (`ssd.forward(..., dt_bias=, dt_softplus=)`, `z=`).  Reference anchors: the 3-tap
causal depthwise convolution on q/k/v (trading_bots/src/torch/model/blocks/gqa.rs:148-178) and the
gain-free RMS norm (trading_bots/src/torch/model/rmsnorm.rs:16-19).
"""
from __future__ import annotations

from typing import Optional, Sequence

import torch

from . import _lib as L
from .ssd import ALGOS


def conv1d_forward(inp, weight, bias=None, *, activation=True, out=None):
    """out[b,t,c] = act(bias[c] + sum_k weight[c,k] * inp[b,t-K+1+k,c]); weight [C,K] fp32, bias [C] fp32."""
    return L.host().conv1d_forward(inp, weight, bias, activation, out)


def conv1d_backward(inp, weight, bias, douts: Sequence[torch.Tensor], *, activation=True):
    """Gradients of conv1d_forward.  `douts`: the gradient w.r.t. the output as 1-3 tensors [B,L,c_i] whose channel
    counts add up to C (the scan's dx, dB, dC, viewed as [B,L,H*P] / [B,L,G*N]).  Returns din, dweight, dbias."""
    return L.host().conv1d_backward(inp, weight, bias, activation, *douts)


def rmsnorm_forward(inp, weight=None, *, eps=1e-5):
    """RMS norm over the last dim (all earlier dims are rows).  Returns out, rstd."""
    return L.host().rmsnorm_forward(inp, weight, eps)


def rmsnorm_backward(inp, weight, rstd, dout, *, eps=1e-5):
    """Returns din (shape of inp) and dweight (or None)."""
    return L.host().rmsnorm_backward(inp, weight, rstd, dout, eps)


class _Conv1d(torch.autograd.Function):
    @staticmethod
    def forward(ctx, inp, weight, bias, activation, splits):
        out = conv1d_forward(inp, weight, bias, activation=activation)
        ctx.save_for_backward(inp, weight, bias)
        ctx.activation, ctx.splits = activation, splits
        return tuple(out.split(splits, dim=2)) if splits else out

    @staticmethod
    def backward(ctx, *gs):
        inp, weight, bias = ctx.saved_tensors
        segs = []
        for g, n in zip(gs, ctx.splits or [inp.shape[2]]):
            if g is None:
                g = torch.zeros(inp.shape[0], inp.shape[1], n, dtype=inp.dtype, device=inp.device)
            g = g.to(inp.dtype)
            segs.append(g if g.stride(2) == 1 and (g.stride(1) * g.element_size()) % 16 == 0 and g.data_ptr() % 16 == 0 else g.contiguous())
        din, dw, db = conv1d_backward(inp, weight, bias, segs, activation=ctx.activation)
        return din, dw, (db if bias is not None else None), None, None


def causal_conv1d(inp, weight, bias=None, *, activation=True, splits: Optional[Sequence[int]] = None):
    """Differentiable causal depthwise conv (+ silu).  With `splits` the output comes back as channel-range views of
    one buffer (what the scan takes as strided x, B, C) and their gradients are consumed as separate segments."""
    return _Conv1d.apply(inp, weight, bias, activation, tuple(splits) if splits else None)


class _RmsNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, inp, weight, eps):
        out, rstd = rmsnorm_forward(inp, weight, eps=eps)
        ctx.save_for_backward(inp, weight, rstd)
        ctx.eps = eps
        return out

    @staticmethod
    def backward(ctx, g):
        inp, weight, rstd = ctx.saved_tensors
        din, dw = rmsnorm_backward(inp, weight, rstd, g.to(inp.dtype), eps=ctx.eps)
        return din, dw, None


def rmsnorm(inp, weight=None, *, eps=1e-5):
    return _RmsNorm.apply(inp.contiguous(), weight, eps)


def mamba2_mixer_core(xBC, dt, z, conv_weight, conv_bias, dt_bias, A, D, norm_weight, *, nheads, headdim, dstate, ngroups,
                      chunk=128, eps=1e-5, algo="auto", init_state=None):
    """The mixer of a Mamba-2 layer between its two projections, differentiable:
        x, B, C = split(silu(causal_conv1d(xBC)));  y = SSD(x, softplus(dt + dt_bias), A, B, C, D) * silu(z);
        out = rmsnorm(y) * norm_weight.
    xBC [B,L,H*P+2*G*N], dt [B,L,H], z [B,L,H,P].  One autograd node over this library's operators: conv, scan (with the
    step-size activation and the gate inside; x, B, C are channel ranges of the conv's output), norm.  `algo` is the
    scan's (see ssd.py)."""
    return L.host().mixer(xBC, dt, z, conv_weight, conv_bias, dt_bias, A, D, norm_weight, init_state, nheads, headdim, dstate,
                          ngroups, chunk, eps, ALGOS[algo])
