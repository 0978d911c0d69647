"""Mamba-2 SSD forward and backward on B200 behind the reference's public API.

``mamba2_ssd_fwd`` keeps the signature, argument meaning, return convention and
error style of ``ascend_kernel.mamba2_ssd_fwd`` in So-cean/mamba-ascendc
(mamba_ascendc/python/ascend_kernel/ascend_kernel/mamba2.py:1923-2017; alias
``mamba_chunk_scan_combined`` :2020).  Where the reference picks between several
device routes and torch glue, this layer has one route: a ``torch.autograd.Function``
that allocates outputs and scratch tensors with torch and enqueues the C-ABI stages
of libssd_b200.so on the current CUDA stream.  There is no CPU path.

Stages (see include/ssd_b200.h): dt softplus + in-tile cumulative decay, chunk
states (tcgen05) and inter-tile state scan (one fused launch when batch * ngroups
fills the GPU, two tile-parallel launches otherwise), output kernel (tcgen05);
backward: local state gradient (tcgen05) and reverse state scan (fused likewise),
dx + dt stage (tcgen05), dB/dC (tcgen05), ddt/dA finalisation.

``chunk_size`` is validated like the reference does, but the kernels always tile the
sequence by 128 tokens: the SSD result does not depend on the chunk length.
"""
from __future__ import annotations

import contextlib
import ctypes
import math
from typing import Dict, Optional, Tuple, Union

import torch

from . import _capi
from .shapes import run_general

TILE = 128

_status_words: Dict[int, torch.Tensor] = {}


def _status(device: torch.device) -> torch.Tensor:
    """Per-device int32 the kernels set when a bounded wait gives up (see ``check_status``)."""
    idx = device.index if device.index is not None else torch.cuda.current_device()
    word = _status_words.get(idx)
    if word is None:
        word = torch.zeros(1, dtype=torch.int32, device=torch.device("cuda", idx))
        _status_words[idx] = word
    return word


def check_status(device: Optional[torch.device] = None) -> None:
    """Synchronise and raise if any kernel on ``device`` reported a TMA / MMA wait that ran out.

    A kernel whose bounded wait gives up writes no results, and every kernel launched after it returns at
    once, so tensors produced since the last check are not valid until this has been called and returned.
    Raising clears the word: the next call starts clean."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else device
    word = _status(device)
    code = int(word.item())
    if code != 0:
        word.zero_()
        kind = {1: "a TMA load did not arrive", 2: "a tensor-core product or its hand-off did not complete",
                3: "shared memory misaligned"}.get(code & 15, "unknown")
        raise RuntimeError(f"mamba2_ssd: a device-side wait gave up (status {code}: {kind}; source file "
                           f"{code >> 12}, wait {(code >> 4) & 255}); results are invalid")


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _stream() -> int:
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def make_shape(x: torch.Tensor, B: torch.Tensor, dt_softplus: bool,
               dt_limit: Tuple[float, float] = (0.0, float("inf")), valid_len: int = 0) -> _capi.SsdShape:
    b, l, h, p = x.shape
    g, n = B.shape[2], B.shape[3]
    return _capi.SsdShape(b, l, h, p, n, TILE, g, _capi.SSD_FLAG_DT_SOFTPLUS if dt_softplus else 0,
                          float(dt_limit[0]), float(dt_limit[1]), int(valid_len))


def extents_shape(x: torch.Tensor, B: torch.Tensor, heads: int, dt_softplus: bool,
                  dt_limit: Tuple[float, float]) -> _capi.SsdShape:
    """The shape of a call whose tensors keep their real extents (SSD_FLAG_EXTENTS): any length, headdim up to 64 or (as
    ``x`` [B,L,heads * parts,64]) a multiple of 64, state size up to 128."""
    b, l, h, p = x.shape
    g, n = B.shape[2], B.shape[3]
    tiles = (l + TILE - 1) // TILE
    flags = (_capi.SSD_FLAG_EXTENTS | (_capi.SSD_FLAG_DT_SOFTPLUS if dt_softplus else 0) |
             _capi.head_parts_flag(h // heads))
    return _capi.SsdShape(b, tiles * TILE, h, p, n, TILE, g, flags, dt_limit[0], dt_limit[1], l if l % TILE else 0)


# ----------------------------------------------------------------------------- validation
def _check_tensor(t: torch.Tensor, name: str) -> None:
    if t.is_cuda and t.dtype is torch.float32 and t.is_contiguous():
        return
    # mamba_ascendc/csrc/ops/mamba2_ssd_fwd/op_host/mamba2_ssd_fwd.cpp:15-23
    if not t.is_cuda:
        raise RuntimeError(f"mamba2_ssd_fwd: {name} must be a CUDA tensor")
    if t.dtype != torch.float32:
        raise RuntimeError(f"mamba2_ssd_fwd: {name} must be float32")
    if not t.is_contiguous():
        raise RuntimeError(f"mamba2_ssd_fwd: {name} must be contiguous")


def _validate(x, dt, A, B, C, chunk_size, D, z, dt_bias, dt_limit, initial_states) -> None:
    for t, name in ((x, "x"), (dt, "dt"), (A, "A"), (B, "B"), (C, "C")):
        _check_tensor(t, name)
    # mamba2_ssd_fwd.cpp:59-85
    if x.dim() != 4:
        raise RuntimeError("mamba2_ssd_fwd: x must have shape [B,L,H,P]")
    if dt.dim() != 3:
        raise RuntimeError("mamba2_ssd_fwd: dt must have shape [B,L,H]")
    if A.dim() != 1:
        raise RuntimeError("mamba2_ssd_fwd: A must have shape [H]")
    if B.dim() != 4 or C.dim() != 4:
        raise RuntimeError("mamba2_ssd_fwd: B and C must have shape [B,L,G,N]")
    b, l, h, _p = x.shape
    if tuple(dt.shape) != (b, l, h):
        raise RuntimeError("mamba2_ssd_fwd: dt shape must equal [B,L,H]")
    if A.shape[0] != h:
        raise RuntimeError("mamba2_ssd_fwd: A shape must equal [H]")
    if B.shape != C.shape:
        raise RuntimeError("mamba2_ssd_fwd: B and C shapes must match")
    if B.shape[0] != b or B.shape[1] != l:
        raise RuntimeError("mamba2_ssd_fwd: B/C batch and sequence dimensions must match x")
    if h % B.shape[2] != 0:
        raise RuntimeError("mamba2_ssd_fwd: nheads must be divisible by ngroups")
    if int(chunk_size) <= 0:
        raise RuntimeError("mamba2_ssd_fwd: chunk_size must be positive")
    if float(dt_limit[0]) > float(dt_limit[1]):
        raise RuntimeError("mamba2_ssd_fwd: dt_limit min must not exceed max")
    if initial_states is not None:
        _check_tensor(initial_states, "initial_states")
        # mamba2_ssd_fwd.cpp:108-112
        if tuple(initial_states.shape) != (b, h, x.shape[3], B.shape[3]):
            raise RuntimeError("mamba2_ssd_fwd: initial_states shape must equal [B,H,P,N]")
    # mamba2_ssd_fwd.cpp:88-106
    if D is not None:
        _check_tensor(D, "D")
        if not ((D.dim() == 1 and D.shape[0] == h) or (D.dim() == 2 and tuple(D.shape) == (h, x.shape[3]))):
            raise RuntimeError("mamba2_ssd_fwd: D shape must equal [H] or [H,P]")
    if z is not None:
        _check_tensor(z, "z")
        if z.shape != x.shape:
            raise RuntimeError("mamba2_ssd_fwd: z shape must match x")
    if dt_bias is not None:
        _check_tensor(dt_bias, "dt_bias")
        if dt_bias.dim() != 1 or dt_bias.shape[0] != h:
            raise RuntimeError("mamba2_ssd_fwd: dt_bias shape must equal [H]")


# ----------------------------------------------------------------------------- route of the state stages
# The per-tile state products and the inter-tile recurrence run either as two tile-parallel launches
# (ssd_chunk_state + ssd_state_passing_*) or as one launch that walks each (batch, group) in tile order with
# the running state on chip (ssd_chunk_state_scan).  The second moves 2 GiB less per pass at the H256 shape
# but has only batch * ngroups CTAs; "auto" leaves the choice to the library (ssd_use_state_scan).
_state_scan = "auto"
_ROUTES = {"auto": 0, "on": 1, "off": 2}


def set_state_scan(mode: str) -> str:
    """Choose "auto" (default), "on" (whenever the kernel takes the shape) or "off"; returns the previous mode."""
    global _state_scan
    if mode not in ("auto", "on", "off"):
        raise ValueError('state scan mode must be "auto", "on" or "off"')
    previous, _state_scan = _state_scan, mode
    return previous


def _use_state_scan(shape: "_capi.SsdShape", device: torch.device) -> bool:
    """The library's own rule, for ``device``, which is the current one wherever stages are launched."""
    with _device_guard(device):
        return bool(_capi.lib.ssd_use_state_scan(ctypes.byref(shape), _ROUTES[_state_scan]))


def _state_cols(shape: "_capi.SsdShape") -> int:
    """State columns of the internal buffers."""
    return 64 if shape.dstate <= 64 else 128


# ----------------------------------------------------------------------------- stage drivers
# When set to a list, every stage launch is bracketed by CUDA events on the launching stream and
# (name, start, end) is appended; used by bench.py to time individual kernels inside a step.
stage_events = None


def _call(name: str, fn, *args) -> None:
    events = stage_events
    if events is None:
        _capi.check(fn(*args), name)
        return
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    _capi.check(fn(*args), name)
    end.record()
    events.append((name, start, end))


def forward_stages(x, dt, A, B, C, dt_softplus: bool, want_final: bool = True, initial_states=None, dt_bias=None,
                   dt_limit=(0.0, float("inf")), valid_len: int = 0, inflow=None, shape=None, copy=None):
    """Run the four forward stages; returns (out, final_state, q, cs, states_start).

    ``inflow(final0, log_decay) -> initial_states`` (sequence-parallel mode): called once the per-tile states
    exist, with the state this block of tokens would hand on from a zero start ([B,H,P,N]) and the logarithm
    of its total decay ([B,H]); what it returns seeds the recurrence.

    ``shape``: from ``extents_shape``; the default is the kernels' own sizes, whole tiles.  ``copy``: like ``out``, receives its
    values as well."""
    if shape is None:
        shape = make_shape(x, B, dt_softplus, dt_limit, valid_len)
    _capi.check(_capi.lib.ssd_check_shape(ctypes.byref(shape)), "mamba2_ssd_fwd")
    b, l, h = shape.batch, shape.seqlen, shape.nheads
    k = l // TILE
    dev = x.device
    status = _status(dev)
    st = _stream()
    q = torch.empty(b, h, l, device=dev, dtype=torch.float32)
    cs = torch.empty_like(q)
    states = torch.empty(b, h, k, 64, _state_cols(shape), device=dev, dtype=torch.float32)
    out = torch.empty_like(x)
    final = torch.empty(b, h, shape.headdim, shape.dstate, device=dev, dtype=torch.float32) if want_final else None
    lib = _capi.lib
    sp = ctypes.byref(shape)
    _call("mamba2_ssd_dt_cumsum", lib.ssd_dt_cumsum, sp, _ptr(dt), _ptr(dt_bias), _ptr(A), _ptr(q), _ptr(cs), st)
    if inflow is None and _use_state_scan(shape, dev):
        _call("mamba2_ssd_chunk_state_scan", lib.ssd_chunk_state_scan, sp, _ptr(x), _ptr(B), _ptr(q), _ptr(cs),
              _ptr(initial_states), _ptr(states), _ptr(final), 0, _ptr(status), st)
        _call("mamba2_ssd_chunk_scan", lib.ssd_chunk_scan_copy_fwd, sp, _ptr(x), _ptr(B), _ptr(C), _ptr(states), _ptr(q),
              _ptr(cs), _ptr(out), _ptr(copy), _ptr(status), st)
        return out, final, q, cs, states
    _call("mamba2_ssd_chunk_state", lib.ssd_chunk_state, sp, _ptr(x), _ptr(B), _ptr(q), _ptr(cs), _ptr(states), 0, _ptr(status), st)
    if inflow is not None:
        final0 = torch.empty(b, h, shape.headdim, shape.dstate, device=dev, dtype=torch.float32)
        _call("mamba2_ssd_state_fold", lib.ssd_state_fold, sp, _ptr(states), _ptr(cs), None, _ptr(final0), 0, st)
        initial_states = inflow(final0, cs.view(b, h, k, TILE)[..., -1].sum(-1))
    _call("mamba2_ssd_state_passing", lib.ssd_state_passing_fwd, sp, _ptr(states), _ptr(cs), _ptr(initial_states),
          _ptr(final), st)
    _call("mamba2_ssd_chunk_scan", lib.ssd_chunk_scan_copy_fwd, sp, _ptr(x), _ptr(B), _ptr(C), _ptr(states), _ptr(q), _ptr(cs),
          _ptr(out), _ptr(copy), _ptr(status), st)
    return out, final, q, cs, states


def backward_stages(x, dt, A, B, C, out, q, cs, states, dout, dfinal, dt_softplus: bool, want_dinitial: bool = False,
                    dt_bias=None, dt_limit=(0.0, float("inf")), valid_len: int = 0, outflow=None, D=None, ddt_bias=None,
                    shape=None):
    """Run the backward stages; returns (dx, ddt, dA, dB, dC, d_initial_states or None).

    ``outflow(d_initial0) -> extra dfinal or None`` (sequence-parallel mode): called once the local state
    gradients exist, with the gradient this block hands back to its predecessor when nothing comes in from
    its successors; what it returns is added to ``dfinal`` before the reverse recurrence runs.

    ``D``: the skip connection of the gated node; then ``dout`` / ``out`` are the gradient / value of the SSD
    output before skip and gate, and ``D * dout`` is added to dx by the dx kernel.

    ``ddt_bias`` [H]: receives the sum of ddt over batch and tokens."""
    if shape is None:
        shape = make_shape(x, B, dt_softplus, dt_limit, valid_len)
    b, l, h, p, n = shape.batch, shape.seqlen, shape.nheads, shape.headdim, shape.dstate
    k = l // TILE
    dev = x.device
    status = _status(dev)
    st = _stream()
    lib = _capi.lib
    sp = ctypes.byref(shape)
    n_state = _state_cols(shape)
    dstates = torch.empty(b, h, k, 64, n_state, device=dev, dtype=torch.float32)
    g_last = torch.empty(n_state // 64, b, h, k, device=dev, dtype=torch.float32)
    ddt_t = torch.empty(b, h, l, device=dev, dtype=torch.float32)
    dA_part = torch.empty(b, h, k, device=dev, dtype=torch.float64)
    dx = torch.empty_like(x)
    ddt = torch.empty_like(dt)
    dA = torch.empty_like(A)
    dB = torch.empty_like(B)
    dC = torch.empty_like(C)
    d_initial = torch.empty(b, h, p, n, device=dev, dtype=torch.float32) if want_dinitial else None
    # g_last (the gradient of each tile's total decay through the state recurrence) comes out of the dB/dC
    # kernel, which streams the forward's states and dU anyway; the reverse scan then never reads the states.
    fused = outflow is None and _use_state_scan(shape, dev)
    if fused:
        _call("mamba2_ssd_chunk_state_scan_bwd", lib.ssd_chunk_state_scan, sp, _ptr(dout), _ptr(C), _ptr(q), _ptr(cs),
              _ptr(dfinal), _ptr(dstates), _ptr(d_initial), 1, _ptr(status), st)
    else:
        _call("mamba2_ssd_chunk_state_bwd", lib.ssd_chunk_state, sp, _ptr(dout), _ptr(C), _ptr(q), _ptr(cs), _ptr(dstates), 1, _ptr(status), st)
    if outflow is not None:
        d0 = torch.empty(b, h, p, n, device=dev, dtype=torch.float32)
        _call("mamba2_ssd_state_fold", lib.ssd_state_fold, sp, _ptr(dstates), _ptr(cs), _ptr(dfinal), _ptr(d0), 1, st)
        extra = outflow(d0)
        if extra is not None:
            dfinal = extra if dfinal is None else dfinal + extra
    if not fused:
        _call("mamba2_ssd_state_passing_bwd", lib.ssd_state_passing_bwd, sp, _ptr(dstates), None, _ptr(cs), _ptr(dfinal),
              None, _ptr(d_initial), st)
    split = lib.ssd_dbc_split(sp)  # > 1: few work items, the heads of a group are dealt to several
    part = torch.empty(2 * split * B.numel(), device=dev, dtype=torch.float32) if split > 1 else None
    _call("mamba2_ssd_chunk_dbc_bwd", lib.ssd_chunk_dbc_split_bwd, sp, _ptr(x), _ptr(B), _ptr(C), _ptr(dout), _ptr(states),
          _ptr(dstates), _ptr(q), _ptr(cs), _ptr(dB), _ptr(dC), _ptr(g_last), split, _ptr(part), _ptr(status), st)
    _call("mamba2_ssd_chunk_dx_bwd", lib.ssd_chunk_dx_bwd, sp, _ptr(x), _ptr(B), _ptr(C), _ptr(dout), _ptr(out), _ptr(dstates), _ptr(q),
                                     _ptr(cs), _ptr(dt), _ptr(dt_bias), _ptr(A), _ptr(g_last), _ptr(dx), _ptr(ddt_t),
                                     _ptr(dA_part), _ptr(D), _d_mode(D), _ptr(status), st)
    _call("mamba2_ssd_dt_bwd", lib.ssd_dt_finalize_bias_bwd, sp, _ptr(ddt_t), _ptr(dA_part), _ptr(ddt), _ptr(dA),
          _ptr(ddt_bias), st)
    return dx, ddt, dA, dB, dC, d_initial


# ----------------------------------------------------------------------------- D skip and z gate
def _d_mode(D: Optional[torch.Tensor]) -> int:
    return 0 if D is None else D.dim()  # 1: [H], 2: [H,P]


def _gate_shape(x, heads: Optional[int]) -> "_capi.SsdShape":
    b, l, h, p = x.shape
    heads = heads or h  # of D; x may hold several heads of 64 channels for each
    return _capi.SsdShape(b, l, heads, p * (h // heads), 64, TILE, 1, 0, 0.0, 0.0, 0)


def gate_forward(y, x, B, D, z, heads: Optional[int] = None):
    """out = (y + D .* x) .* silu(z) in one pass (ssd_gate_skip_fwd)."""
    shape = _gate_shape(x, heads)
    out = torch.empty_like(y)
    _call("mamba2_ssd_gate", _capi.lib.ssd_gate_skip_fwd, ctypes.byref(shape), _ptr(y), _ptr(x), _ptr(D), _d_mode(D),
          _ptr(z), _ptr(out), _stream())
    return out


def gate_backward(dout, y, x, B, D, z, heads: Optional[int] = None):
    """(dy, dz, dD) of the gate / skip epilogue in one pass; without z, dy is dout itself."""
    shape = _gate_shape(x, heads)
    sp = ctypes.byref(shape)
    dy = torch.empty_like(dout) if z is not None else dout
    dz = torch.empty_like(dout) if z is not None else None
    dD = part = None
    if D is not None:
        dD = torch.empty_like(D)
        part = torch.empty(_capi.lib.ssd_gate_partial_floats(sp), device=dout.device, dtype=torch.float32)
    _call("mamba2_ssd_bwd_gate", _capi.lib.ssd_gate_skip_bwd, sp, _ptr(dout), _ptr(y), _ptr(x), _ptr(D), _d_mode(D),
          _ptr(z), _ptr(dy) if z is not None else None, _ptr(dz), _ptr(part), _ptr(dD), _stream())
    return dy, dz, dD


def _per_channel(D, x, heads: int):
    """D for x [B,L,heads * parts,64 or less] (parts > 1: several heads of x for each of D[H])."""
    if D is None or D.dim() == 2:
        return D
    return D.repeat_interleave(x.shape[2] // heads).unsqueeze(-1) if x.shape[2] != heads else D.unsqueeze(-1)


def _epilogue(y, x, D, z, heads: int):
    """out = (y + D .* x) .* silu(z) as framework operations."""
    out = y if D is None else y + x * _per_channel(D, x, heads)
    return out if z is None else out * torch.nn.functional.silu(z)


def _is_batched(t: torch.Tensor) -> bool:
    """A gradient under vmap, or one of several taken at once (is_grads_batched)."""
    return torch._C._functorch.is_legacy_batchedtensor(t) or torch._C._functorch.is_functorch_wrapped_tensor(t)


def _epilogue_gradients(dout, y, x, D, z, heads: int):
    """(dz, dD) of the epilogue as framework operations; y and x are constants."""
    dy, dz, dD = dout, None, None
    if z is not None:
        s = torch.sigmoid(z)
        dy, dz = dout * (z * s), dout * _epilogue(y, x, D, None, heads) * (s * (1 + z * (1 - s)))
    if D is not None:
        dD = (dy * x).sum(dim=(0, 1))
        dD = dD if D.dim() == 2 else dD.reshape(heads, -1).sum(-1)
    return dz, dD


# ----------------------------------------------------------------------------- whole calls
# The stages of one direction as one foreign call (ssd_forward, ssd_backward).  While stage_events collects, the same
# stages are launched one by one with events around them.
def forward_call(x, dt, A, B, C, D, z, dt_bias, initial_states, shape, want_final: bool, copy: bool = False):
    """(out, final, y, work tensors): ``y`` is the SSD output before the D / z epilogue; without one it is ``out`` itself, or
    with ``copy`` a tensor of its own."""
    gated = D is not None or z is not None
    dev = x.device
    out = torch.empty_like(x)
    if stage_events is not None:
        y, final, *work = forward_stages(x, dt, A, B, C, False, want_final=want_final, initial_states=initial_states,
                                         dt_bias=dt_bias, shape=shape, copy=out if copy else None)
        if gated:
            out = gate_forward(y, x, B, D, z, A.shape[0])
        return (out if gated or copy else y), final, y, work
    y = torch.empty_like(x) if gated or copy else out
    sp = ctypes.byref(shape)
    lib = _capi.lib
    # q, cs and the states: floats, also for saved-tensor hooks that convert what autograd keeps
    work = torch.empty(lib.ssd_forward_work_bytes(sp) // 4, device=dev, dtype=torch.float32)
    final = (torch.empty(shape.batch, shape.nheads, shape.headdim, shape.dstate, device=dev, dtype=torch.float32)
             if want_final else None)
    args = _capi.SsdForwardArgs(
        x.data_ptr(), dt.data_ptr(), _ptr(dt_bias), A.data_ptr(), B.data_ptr(), C.data_ptr(), _ptr(D), _ptr(z),
        _ptr(initial_states), y.data_ptr(), out.data_ptr() if gated or copy else None, _ptr(final), work.data_ptr(),
        _status(dev).data_ptr(), _d_mode(D))
    _capi.check(lib.ssd_forward(sp, ctypes.byref(args), _ROUTES[_state_scan], _stream()), "mamba2_ssd_fwd")
    return out, final, y, (work,)


def backward_call(x, dt, A, B, C, D, z, dt_bias, y, work, dout, dfinal, shape, want_dinitial: bool):
    """(dx, ddt, dA, dB, dC, dD, dz, d_initial, d_dt_bias); ``work`` from ``forward_call``."""
    gated = D is not None or z is not None
    dbias = torch.empty_like(dt_bias) if dt_bias is not None else None  # mamba2_ssd_dt_bwd/design.md:63-77
    if len(work) == 3:  # launched one by one
        dy, dz, dD = gate_backward(dout, y, x, B, D, z, A.shape[0]) if gated else (dout, None, None)
        dx, ddt, dA, dB, dC, dinit = backward_stages(x, dt, A, B, C, y, *work, dy, dfinal, False, want_dinitial=want_dinitial,
                                                     dt_bias=dt_bias, D=D, ddt_bias=dbias, shape=shape)
        return dx, ddt, dA, dB, dC, dD, dz, dinit, dbias
    dev = x.device
    lib = _capi.lib
    sp = ctypes.byref(shape)
    scratch = torch.empty(lib.ssd_backward_work_bytes(sp, D is not None, z is not None), device=dev, dtype=torch.uint8)
    dx, ddt, dA, dB, dC = (torch.empty_like(t) for t in (x, dt, A, B, C))
    dD = torch.empty_like(D) if D is not None else None
    dz = torch.empty_like(z) if z is not None else None
    dinit = (torch.empty(shape.batch, shape.nheads, shape.headdim, shape.dstate, device=dev, dtype=torch.float32)
             if want_dinitial else None)
    args = _capi.SsdBackwardArgs(
        x.data_ptr(), dt.data_ptr(), _ptr(dt_bias), A.data_ptr(), B.data_ptr(), C.data_ptr(), _ptr(D), _ptr(z), y.data_ptr(),
        dout.data_ptr(), _ptr(dfinal), work[0].data_ptr(), dx.data_ptr(), ddt.data_ptr(), dA.data_ptr(), dB.data_ptr(),
        dC.data_ptr(), _ptr(dD), _ptr(dz), _ptr(dbias), _ptr(dinit), scratch.data_ptr(), _status(dev).data_ptr(),
        _d_mode(D))
    _capi.check(lib.ssd_backward(sp, ctypes.byref(args), _ROUTES[_state_scan], _stream()), "mamba2_ssd_bwd")
    return dx, ddt, dA, dB, dC, dD, dz, dinit, dbias


# ----------------------------------------------------------------------------- autograd
def _aligned(t: torch.Tensor) -> torch.Tensor:
    """Contiguous fp32 at an address the tile loads take (a gradient may be a slice of a larger one)."""
    t = t.contiguous().float()
    return t.clone() if t.data_ptr() & 15 else t


def _epilogue_alone(ctx) -> bool:
    """Whether of the inputs of ``_Mamba2SsdAutograd`` only D and z need gradients."""
    needs = ctx.needs_input_grad
    return not (needs[0] or needs[1] or needs[2] or needs[3] or needs[4] or needs[8] or needs[9])


class _Mamba2SsdAutograd(torch.autograd.Function):
    """Counterpart of ``_Mamba2SsdAutogradM1`` (mamba2.py:1661-1838), with the D skip connection and the z gate inside the node:
    the epilogue runs as one fused pass forward and one backward (the reference fuses them into its state-epilogue and
    gate kernels, mamba2_ssd_state_epilogue.cpp:413-482, bwd_gate/design.md:8-13), and the skip connection's share of dx
    is added in the epilogue of the dx kernel.  Saves the inputs plus, under the default policy, q, cs, the tile-start states and
    the SSD output before the epilogue.  ``x`` is [B,L,H * parts,64] for a headdim of 64 * parts."""

    @staticmethod
    def forward(ctx, x, dt, A, B, C, D, z, dt_softplus, initial_states, dt_bias, dt_min, dt_max):
        ctx.set_materialize_grads(False)  # an output without a gradient takes no zeros, the kernels know a null
        ctx.shape = extents_shape(x, B, A.shape[0], dt_softplus, (dt_min, dt_max))
        ctx.recompute = _save_policy == "recompute"
        ctx.has_initial = initial_states is not None
        # Without an epilogue the output is what backward needs.  At the kernels' own sizes it is saved itself, so that
        # changing it in place is an error in backward; elsewhere the caller may change it, and a copy is saved.
        own_sizes = x.shape[3] == 64 and B.shape[3] == 64 and x.shape[1] % TILE == 0 and x.shape[2] == A.shape[0]
        gated = D is not None or z is not None
        ctx.alone = alone = gated and _epilogue_alone(ctx)
        ctx.differentiable = gated and not own_sizes  # see differentiable_backward
        if ctx.differentiable:
            ctx.options = (dt_softplus, dt_min, dt_max)
        copy = not gated and not ctx.recompute and not own_sizes
        out, final, y, work = forward_call(x, dt, A, B, C, D, z, dt_bias, initial_states, ctx.shape, True, copy=copy)
        start = initial_states if ctx.recompute or ctx.differentiable else None
        if ctx.recompute:  # inputs only; y, q, cs and the tile-start states are rebuilt in backward
            ctx.save_for_backward(x, dt, A, B, C, dt_bias, D, z, start)
        else:
            if alone:  # its gradients take y only
                work = ()
            ctx.save_for_backward(x, dt, A, B, C, dt_bias, D, z, start, y, *work)
        if alone and not own_sizes:  # where D and z were framework operations the state never belonged to their graph
            ctx.mark_non_differentiable(final)
        return out, final

    @staticmethod
    def backward(ctx, dout, dfinal):
        x, dt, A, B, C, dt_bias, D, z, initial_states, *rest = ctx.saved_tensors
        y, work = (rest[0], rest[1:]) if rest else (None, None)
        if dout is None:  # loss depends on the final state only (mamba2.py:1801-1802)
            dout = torch.zeros_like(x)
        alone = ctx.alone
        again = ctx.differentiable and (torch.is_grad_enabled() or (alone and _is_batched(dout)))
        if again and not alone:
            return _Mamba2SsdAutograd.differentiable_backward(ctx, dout, dfinal)
        if not again:
            dout = _aligned(dout)
            if dfinal is not None:
                dfinal = _aligned(dfinal)
        with _device_guard(x.device):
            if y is None:
                y, _, _, work = forward_call(x, dt, A, B, C, None, None, dt_bias, initial_states, ctx.shape, False)
            if again:
                dz, dD = _epilogue_gradients(dout, y, x, D, z, A.shape[0])
                return None, None, None, None, None, dD, dz, None, None, None, None, None
            if alone:
                _, dz, dD = gate_backward(dout, y, x, B, D, z, A.shape[0])
                return None, None, None, None, None, dD, dz, None, None, None, None, None
            dx, ddt, dA, dB, dC, dD, dz, dinit, dbias = backward_call(x, dt, A, B, C, D, z, dt_bias, y, work, dout, dfinal,
                                                                      ctx.shape, ctx.has_initial)
        return dx, ddt, dA, dB, dC, dD, dz, None, dinit, dbias, None, None

    @staticmethod
    def differentiable_backward(ctx, dout, dfinal):
        """Gradients that are differentiated again (create_graph).  The kernels' gradients are constants to autograd.  Away
        from the kernels' own sizes D and z are nevertheless differentiable any number of times, as framework
        operations around the plain node; so the call is made again in that form and its gradients are taken."""
        inputs = list(ctx.saved_tensors[:9])  # x, dt, A, B, C, dt_bias, D, z, initial_states
        x, dt, A, B, C, dt_bias, D, z, start = aliases = [None if t is None else t.view_as(t) for t in inputs]
        softplus, lo, hi = ctx.options
        y, final = _Mamba2SsdAutograd.apply(x, dt, A, B, C, None, None, softplus, start, dt_bias, lo, hi)
        outputs, upstream = [_epilogue(y, x, D, z, A.shape[0])], [dout]
        if dfinal is not None:
            outputs, upstream = outputs + [final], upstream + [dfinal]
        wanted = [i for i, k in enumerate((0, 1, 2, 3, 4, 9, 5, 6, 8)) if ctx.needs_input_grad[k]]
        grads = [None] * 9
        for i, g in zip(wanted, torch.autograd.grad(outputs, [aliases[i] for i in wanted], upstream, create_graph=True,
                                                    allow_unused=True)):
            grads[i] = g
        dx, ddt, dA, dB, dC, dbias, dD, dz, dinit = grads
        return dx, ddt, dA, dB, dC, dD, dz, None, dinit, dbias, None, None


class _Mamba2SsdPadded(torch.autograd.Function):
    """The plain SSD node on the kernels' own sizes, for the calls that ``shapes.run_general`` pads or cuts into blocks."""

    @staticmethod
    def forward(ctx, x, dt, A, B, C, dt_softplus, initial_states, dt_bias, dt_min, dt_max, valid_len):
        out, final, q, cs, states = forward_stages(x, dt, A, B, C, dt_softplus, want_final=True,
                                                   initial_states=initial_states, dt_bias=dt_bias,
                                                   dt_limit=(dt_min, dt_max), valid_len=valid_len)
        ctx.valid_len = valid_len
        ctx.recompute = _save_policy == "recompute"
        if ctx.recompute:
            ctx.save_for_backward(x, dt, A, B, C, dt_bias, initial_states)
        else:
            ctx.save_for_backward(x, dt, A, B, C, dt_bias, out, q, cs, states)
        ctx.dt_softplus = dt_softplus
        ctx.has_initial = initial_states is not None
        ctx.dt_limit = (dt_min, dt_max)
        return out, final

    @staticmethod
    def backward(ctx, dout, dfinal):
        if ctx.recompute:
            x, dt, A, B, C, dt_bias, initial_states = ctx.saved_tensors
        else:
            x, dt, A, B, C, dt_bias, out, q, cs, states = ctx.saved_tensors
        if dout is None:
            dout = torch.zeros_like(x)
        dout = dout.contiguous().float()
        if dfinal is not None:
            dfinal = dfinal.contiguous().float()
        with _device_guard(x.device):
            if ctx.recompute:
                out, _, q, cs, states = forward_stages(x, dt, A, B, C, ctx.dt_softplus, want_final=False,
                                                       initial_states=initial_states, dt_bias=dt_bias,
                                                       dt_limit=ctx.dt_limit, valid_len=ctx.valid_len)
            dbias = torch.empty_like(dt_bias) if dt_bias is not None else None
            dx, ddt, dA, dB, dC, dinit = backward_stages(x, dt, A, B, C, out, q, cs, states, dout, dfinal,
                                                         ctx.dt_softplus, want_dinitial=ctx.has_initial,
                                                         dt_bias=dt_bias, dt_limit=ctx.dt_limit,
                                                         valid_len=ctx.valid_len, ddt_bias=dbias)
        return dx, ddt, dA, dB, dC, None, dinit, dbias, None, None, None


# What the autograd function keeps between forward and backward (mamba2_ssd_bwd/design.md:207-223 lists the
# reference's save / recompute choices).  "save": inputs plus out, q, cs and the tile-start states (at the
# H256 shape 3.1 GiB on top of the inputs); "recompute": inputs only, the forward stages run again in backward.
_save_policy = "save"


def set_save_policy(policy: str) -> str:
    """Choose "save" (default) or "recompute"; returns the previous policy."""
    global _save_policy
    if policy not in ("save", "recompute"):
        raise ValueError('save policy must be "save" or "recompute"')
    previous, _save_policy = _save_policy, policy
    return previous


class SavedTensorStats:
    """Bytes autograd holds for backward, counted with saved-tensor hooks (the reference's benchmark counts
    the same way, benchmarks/mamba2_backward_bench.py:168-209): ``logical_bytes`` adds every saved tensor,
    ``unique_bytes`` counts each backing storage once.  Use as ``with stats.hooks(): out = fn(...)``."""

    def __init__(self):
        self.logical_bytes = 0
        self._storages: Dict[Tuple[str, Optional[int], int], int] = {}

    def _pack(self, t: torch.Tensor) -> torch.Tensor:
        self.logical_bytes += t.numel() * t.element_size()
        st = t.untyped_storage()
        key = (t.device.type, t.device.index, st.data_ptr())
        self._storages[key] = max(self._storages.get(key, 0), st.nbytes())
        return t

    def hooks(self):
        return torch.autograd.graph.saved_tensors_hooks(self._pack, lambda t: t)

    @property
    def unique_bytes(self) -> int:
        return sum(self._storages.values())


def _device_guard(device: torch.device):
    """Launches go to the current stream of the tensors' device; a context switch only when that is not the
    current device already (the switch costs several microseconds per call)."""
    if torch.cuda.current_device() == device.index:
        return contextlib.nullcontext()
    return torch.cuda.device(device)


# Longest sequence that takes the recurrence kernel instead of the tile kernels (which treat 128 tokens at a time and so
# cost almost the same for 1 token as for 128).  Device time of both, us, with D, z and an initial state:
#   [batch, heads, P, N, G]    16 tokens    32 tokens    48 tokens    64 tokens
#   [ 1,   4, 64,  64, 1]     8.6 /  22     15 /  22     22 /  22     29 /  24
#   [16,  24, 64, 128, 1]      26 /  58     48 /  59     70 /  59     91 /  59
#   [ 8,  32, 64, 128, 1]      18 /  46     32 /  45     46 /  46     60 /  46
#   [64, 128, 64,  64, 8]     212 / 456    391 / 487    570 / 516    753 / 539
SHORT_SEQUENCE = 32


def _own_sizes(l: int, p: int, n: int, grad: bool) -> bool:
    """The kernels' own sizes, which nothing pads, copies or cuts off."""
    return p == 64 and l % TILE == 0 and (n == 64 or (n == 128 and not grad))


_forward_ad, _transforms_active = torch.autograd.forward_ad, torch._C._are_functorch_transforms_active


def _in_transform() -> bool:
    """Whether forward-mode derivatives or a function transform (vmap, grad, jvp) are being taken, which see framework
    operations only.  Away from the kernels' own sizes D and z are then applied by such operations."""
    return _forward_ad._current_level >= 0 or _transforms_active()


def _short_sequence(x, B, C, D, z, initial_states) -> bool:
    """Whether a call without gradients runs as one recurrence launch (ssd_recurrent_fwd)."""
    n = B.shape[3]
    if not (0 < x.shape[1] <= SHORT_SEQUENCE and 0 < n <= 128 and n % 4 == 0 and min(x.shape) > 0 and B.shape[2] > 0):
        return False
    if x.shape[0] > 65535 or B.shape[2] > 65535 or x.shape[0] * x.shape[2] * ((x.shape[3] + 63) // 64) * 64 >= 1 << 31:
        return False  # beyond the tile kernels' range: refused there
    if _in_transform():
        return False
    return not any(t is not None and t.data_ptr() & 15 for t in (B, C, initial_states))


def _tile_extents(x, B, C, D, z, initial_states, grad: bool = False) -> bool:
    """Whether the tile kernels read and write the caller's tensors as they are: their tile loads and stores cut a tile off
    at the end of a sequence, of a head's channels and of the state's columns, in steps of four floats from 16-byte
    aligned addresses.  What this leaves (other headdims and state sizes) is padded or cut into blocks by shapes.py."""
    sizes, state = x.shape, B.shape
    p, n = sizes[3], state[3]
    if min(sizes) <= 0 or min(state) <= 0 or n % 4 or n > 128 or p > 1024 or (p % 64 if p > 64 else p % 4):
        return False
    if _own_sizes(sizes[1], p, n, grad):
        return True  # unaligned addresses are refused
    if _in_transform():
        return False
    return not any(t is not None and t.data_ptr() & 15 for t in (x, B, C, D, z, initial_states))


def _tile_call(x, dt, A, B, C, D, z, dt_bias, dt_softplus, lim, initial_states, return_final_state, grad):
    b, l, h, p = x.shape
    parts = p // 64 if p > 64 else 1
    if parts > 1:  # a head of 64 * parts channels is that many heads of 64 that share dt, A and the group
        x = x.view(b, l, h * parts, 64)
        z = z.view(x.shape) if z is not None else None
        D = D.view(h * parts, 64) if D is not None and D.dim() == 2 else D
        if initial_states is not None:
            initial_states = initial_states.view(b, h * parts, 64, -1)
    if grad:
        out, final = _Mamba2SsdAutograd.apply(x, dt, A, B, C, D, z, dt_softplus, initial_states, dt_bias, lim[0], lim[1])
    else:
        out, final, _, _ = forward_call(x, dt, A, B, C, D, z, dt_bias, initial_states, extents_shape(x, B, h, dt_softplus, lim),
                                        return_final_state)
    if parts > 1:
        out = out.view(b, l, h, p)
        final = final.view(b, h, p, -1) if final is not None else None
    return (out, final) if return_final_state else out


def recurrent_forward(x, dt, A, B, C, dt_softplus: bool, want_final: bool, initial_states, dt_bias, dt_limit, D, z):
    b, l, h, p = x.shape
    g, n = B.shape[2], B.shape[3]
    shape = _capi.SsdShape(b, l, h, p, n, TILE, g, _capi.SSD_FLAG_DT_SOFTPLUS if dt_softplus else 0, dt_limit[0],
                           dt_limit[1], 0)
    out = torch.empty_like(x)
    final = torch.empty(b, h, p, n, device=x.device, dtype=torch.float32) if want_final else None
    _call("mamba2_ssd_recurrent", _capi.lib.ssd_recurrent_fwd, ctypes.byref(shape), _ptr(x), _ptr(dt), _ptr(dt_bias),
          _ptr(A), _ptr(B), _ptr(C), _ptr(D), _d_mode(D), _ptr(z), _ptr(initial_states), _ptr(out), _ptr(final), _stream())
    return out, final


def _requires_grad(*tensors) -> bool:
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


def mamba2_ssd_fwd(
    x: torch.Tensor,
    dt: torch.Tensor,
    A: torch.Tensor,
    B: torch.Tensor,
    C: torch.Tensor,
    chunk_size: int,
    D: Optional[torch.Tensor] = None,
    z: Optional[torch.Tensor] = None,
    dt_bias: Optional[torch.Tensor] = None,
    dt_softplus: bool = False,
    dt_limit: Tuple[float, float] = (0.0, float("inf")),
    initial_states: Optional[torch.Tensor] = None,
    return_final_state: bool = False,
) -> Union[torch.Tensor, Tuple[torch.Tensor, torch.Tensor]]:
    """Mamba-2 SSD chunk scan: ``out[B,L,H,P]`` and optionally ``final_state[B,H,P,N]``.

    x [B,L,H,P], dt [B,L,H], A [H] (the negative decay value, not its log), B and C [B,L,G,N] with
    head h reading group h // (H/G); all contiguous fp32 CUDA tensors.
    """
    _validate(x, dt, A, B, C, chunk_size, D, z, dt_bias, dt_limit, initial_states)
    lim = (float(dt_limit[0]), float(dt_limit[1]))
    needs_grad = _requires_grad(x, dt, A, B, C, initial_states, dt_bias)

    def core(xk, dtk, Ak, Bk, Ck, init, bias, valid):
        # the fixed-shape call: headdim 64, state size 64 (128 without gradients), whole tiles
        if needs_grad:
            return _Mamba2SsdPadded.apply(xk, dtk, Ak, Bk, Ck, bool(dt_softplus), init, bias, lim[0], lim[1], valid)
        out_k, final_k, *_ = forward_stages(xk, dtk, Ak, Bk, Ck, bool(dt_softplus), want_final=return_final_state,
                                            initial_states=init, dt_bias=bias, dt_limit=lim, valid_len=valid)
        return out_k, final_k

    with _device_guard(x.device):
        grad_anywhere = needs_grad or _requires_grad(D, z)
        if not grad_anywhere and _short_sequence(x, B, C, D, z, initial_states):
            out, final = recurrent_forward(x, dt, A, B, C, bool(dt_softplus), return_final_state, initial_states, dt_bias,
                                           lim, D, z)
            return (out, final) if return_final_state else out
        if _tile_extents(x, B, C, D, z, initial_states, grad_anywhere):
            return _tile_call(x, dt, A, B, C, D, z, dt_bias, bool(dt_softplus), lim, initial_states, return_final_state,
                              grad_anywhere)
        # any other headdim and state size, unaligned addresses: see shapes.py
        out, final = run_general(core, x, dt, A, B, C, initial_states, dt_bias, needs_grad)
        # D skip connection and z gate (ssd_reference.py:300-318) as element-wise epilogue; under autograd
        # their gradients (dD, dz and the extra term of dx) come from these same operations
        out = _epilogue(out, x, D, z, x.shape[2])
    if return_final_state:
        return out, final
    return out


mamba_chunk_scan_combined = mamba2_ssd_fwd
