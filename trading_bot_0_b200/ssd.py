"""Tensor-in / tensor-out host side of the SSD operator.

Mirrors the safe wrapper a tch caller would write over the C ABI: validate first and raise
(`validate` in trading_bots/src/torch/fa4.rs:145-191 checks rank, device, dtype, unit inner
stride and matching batch before its FFI call), then pass raw device pointers, a caller-owned
workspace and the current stream.  Explicit `forward` / `backward` calls are the contract
(tch-rs has no custom autograd node); `ssd_scan` additionally wraps them in an autograd node so
they take part in `loss.backward()`.  Checks, allocations and the library calls themselves are
native (csrc/ssd_host.cpp): a small call costs a few microseconds of host time.

`algo` of every call picks the kernels.  "auto": bf16 shapes that the tensor-core kernels cover, of any length, are
evaluated with bf16 operands and fp32 sums, everything else in fp32.  "fp32_cores" keeps every intermediate value in
fp32 on bf16 storage too: gradients of step sizes and decay rates (ddt, dA) are then exact to 1e-6 instead of 1e-3 to
1e-2, at several times the time.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from . import _lib as L

ALGOS = {"auto": L.ALGO_AUTO, "fp32_cores": L.ALGO_FP32_CORES, "tensor": L.ALGO_TENSOR,
         "tensor_onetile": L.ALGO_TENSOR_ONETILE}


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else C.c_void_p(t.data_ptr())


def _stream(device) -> C.c_void_p:
    return C.c_void_p(torch.cuda.current_stream(device).cuda_stream)


def make_dims(x, dt, Bm, Cm, chunk, *, z=None, y=None, algo="auto", dt_softplus=False) -> L.SsdDims:
    """Validate the sequence operands and fill the geometry struct."""
    return L.SsdDims.from_buffer_copy(L.host().dims(x, dt, Bm, Cm, chunk, z, y, ALGOS[algo], dt_softplus))


def workspace_bytes(dims: L.SsdDims, backward: bool = False) -> int:
    n = L.load().ssd_workspace_bytes(C.byref(dims), L.PASS_BWD if backward else L.PASS_FWD)
    if n == 0:
        raise L.SsdError(-1, L.load().ssd_last_error().decode())
    return n


def alloc_workspace(dims: L.SsdDims, device, backward: bool = False) -> torch.Tensor:
    return torch.empty(workspace_bytes(dims, backward), dtype=torch.uint8, device=device)


def workspace_status(workspace: torch.Tensor) -> int:
    """Wait for the current stream and read the status word of `workspace`: 0 when healthy; raises SsdError (code
    SSD_ERR_TIMEOUT, wait-site in the message) when a bounded wait inside a pipelined kernel ran out.  The device-side
    counterpart of the error read the reference makes after every FFI call (trading_bots/src/torch/cuda/graph.rs:107-118)."""
    code = C.c_int32(0)
    with torch.cuda.device(workspace.device):
        L.check(L.load().ssd_workspace_status(_ptr(workspace), _stream(workspace.device), C.byref(code)))
    return int(code.value)


def forward(x, dt, A, Bm, Cm, D=None, z=None, init_state=None, *, chunk, algo="auto", workspace=None,
            y=None, final_state=None, return_final_state=True, for_backward=False, stages=None,
            dt_bias=None, dt_softplus=False, check=False):
    """y, final_state, workspace = SSD(x, dt, A, B, C, D, z, init_state).  With `dt_bias` / `dt_softplus` the step
    size is act(dt + dt_bias), evaluated inside the cumsum kernel (the pre-activation of a Mamba-2 layer).
    `check=True` waits for the stream afterwards and raises if a kernel reported a timed-out wait."""
    r = L.host().forward(x, dt, A, Bm, Cm, D, z, init_state, chunk, ALGOS[algo], workspace, y, final_state,
                         return_final_state, for_backward, stages, dt_bias, dt_softplus)
    if check:
        workspace_status(r[2])
    return r


def backward(dy, x, dt, A, Bm, Cm, D=None, z=None, init_state=None, dfinal_state=None, *, chunk, algo="auto",
             workspace=None, fwd_saved=False, want_dinit=False, stages=None, out=None, dt_bias=None,
             dt_softplus=False, check=False):
    """Gradients of `forward`.  Returns a dict with dx, ddt, dA, dB, dC, dD, dz, dinit (and ddt_bias when dt_bias is
    given; ddt is then the gradient w.r.t. the dt passed in, before bias and activation).  A tensor already in `out` is
    written in place: it must be dense, 16-byte aligned and of the right shape."""
    o = L.host().backward(dy, x, dt, A, Bm, Cm, D, z, init_state, dfinal_state, chunk, ALGOS[algo], workspace, fwd_saved,
                          want_dinit, stages, {} if out is None else out, dt_bias, dt_softplus)
    if check:
        workspace_status(o["workspace"])
    return o


def state_update(state, x, dt, A, Bm, Cm, D=None, z=None, *, y=None, dt_bias=None, dt_softplus=False):
    """One timestep over all streams, IN PLACE on `state` [S,H,P,N] fp32.  Returns y [S,H,P].  The step size is
    act(dt + dt_bias) as in `forward`."""
    return L.host().state_update(state, x, dt, A, Bm, Cm, D, z, y, dt_bias, dt_softplus)


def ssd_scan(x, dt, A, Bm, Cm, D=None, z=None, init_state=None, *, chunk=128, algo="auto", dt_bias=None,
             dt_softplus=False):
    """Differentiable SSD: returns (y, final_state)."""
    return L.host().scan(x, dt, A, Bm, Cm, D, z, init_state, chunk, ALGOS[algo], dt_bias, dt_softplus)
