"""Layer calls through one library entry per direction (``b200gru_layer_forward`` / ``_backward``).

``forward(layer, x, h0)`` runs the input projection and the scan of a dispatchable ``GRULayer`` with
a dense input side and returns ``out``, or ``None`` where the call has a form this path does not take
(other dtypes or devices, widths that are no multiple of 8, quantizers other than the kinds the
kernels implement or with hooks, tracing and function transforms): the caller then goes through the composed path
of ``tc.linear`` and the scan functions, which also words the errors.

One step of one sequence (T = B = 1, 256 x 256) spent 190 us in the composed path's Python: four
concatenations, two autograd functions and a dozen library calls around 23 us of kernels.
"""

from __future__ import annotations

import ctypes
from functools import lru_cache

import torch

from . import _lib
from .quantizers import FakeQuantizePerChannel, FakeQuantizePerGroup, FakeQuantizePerTensor, Identity

_INTS = ctypes.c_int * 10
_FLOATS = ctypes.c_float * 12
_FWD_PTRS = ctypes.c_void_p * 19
_BWD_PTRS = ctypes.c_void_p * 14
_SIZES = ctypes.c_size_t * 3
_GATES = "rzn"
_INPUT_QUANTIZERS = (Identity, FakeQuantizePerTensor, FakeQuantizePerChannel, FakeQuantizePerGroup)


@lru_cache(maxsize=512)
def _plan(kind, T, B, I, H, nblocks, log2_hpad, bits_i, bits_h):
    """``((dims, of the scan's backward, of the projection's), kept bytes, forward scratch, backward scratch)`` of a
    shape, or None if it has none."""
    dims = [_INTS(_lib.KIND[kind], T, B, I, H, nblocks, log2_hpad, bits_i, bits_h, part) for part in range(3)]
    sizes = _SIZES()
    if _lib.load().b200gru_layer_sizes(dims[0], sizes):
        return None
    return (dims, *sizes)


@lru_cache(maxsize=512)
def _quants(qx, qi, qo):
    vals = []
    for q in (qx, qi, qo):
        vals += [1.0, 0.0, 0.0, 0.0] if q is None else [q[0], q[1], q[2], 1.0]
    return _FLOATS(*vals)


def _weight_bits(quantizers):
    """Bit width the weight-preparation kernel implements for these three quantizers (32: identities), else None."""
    a, b, c = quantizers
    if type(a) is Identity and type(b) is Identity and type(c) is Identity:
        return 32
    bits = a.config.bits
    for q in quantizers:
        cfg = q.config
        if (not isinstance(q, FakeQuantizePerChannel) or cfg.axis != 0 or not cfg.symmetric or cfg.mode != "dynamic" or
                cfg.bits != bits or bits > 8):
            return None
    return int(bits)


def _observed(module) -> bool:
    """The module has hooks, or a ``forward`` of the instance's own: it has to be called, once."""
    return bool(module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks or
                "forward" in module.__dict__)


def _plain(t, shape, device):
    return ((type(t) is torch.nn.Parameter or type(t) is torch.Tensor) and t.dtype is torch.float32 and
            t.device == device and t.shape == shape and t.is_contiguous())


def _transformed() -> bool:
    """Function transforms, forward-mode AD and tracing look at every operation: not for one opaque call."""
    return (torch._C._functorch.peek_interpreter_stack() is not None or
            torch.autograd.forward_ad._current_level >= 0 or torch.jit.is_tracing() or torch.compiler.is_compiling())


def _parameters(cell, kind, device, I, H):
    """``(params, nblocks, log2_hpad)``: input weights, hidden weights, input biases, hidden biases per gate (no biases: six)."""
    own, mods = cell._parameters, cell._modules
    wi = [own.get("W_i" + g) for g in _GATES]
    nblocks, log2_hpad = 1, 0
    if kind == "dense":
        wh, shape = [own.get("W_h" + g) for g in _GATES], (H, H)
    else:
        structs = [mods["struct_Wh_" + g] for g in _GATES]
        if kind == "butterfly":
            wh = [s.b.twiddle for s in structs]
            shape = wh[0].shape
            if len(shape) != 6 or shape[0] != 1 or 2 * shape[3] != 1 << shape[2] or 2 * shape[3] < H or tuple(shape[4:]) != (2, 2):
                return None
            nblocks, log2_hpad = shape[1], shape[2]
        else:
            wh = [s.weight for s in structs]
            if kind == "diagonal":
                shape = (H,)
            else:
                nblocks = wh[0].shape[0]
                if nblocks == 0 or H % nblocks:
                    return None
                shape = (nblocks, H // nblocks, H // nblocks)
    biases = [own.get("b_" + s + g) for s in "ih" for g in _GATES]
    if any(b is None for b in biases):
        if any(b is not None for b in biases) or any(getattr(cell, "b_" + s + g, None) is not None for s in "ih" for g in _GATES):
            return None
        biases = None
    elif not all(_plain(b, (H,), device) for b in biases):
        return None
    if not (all(_plain(w, (H, I), device) for w in wi) and all(_plain(w, shape, device) for w in wh)):
        return None
    return wi + wh + (biases or []), nblocks, log2_hpad


def _addresses(params):
    ptrs = [p.data_ptr() for p in params]
    return ptrs if len(ptrs) == 12 else ptrs + [None] * 6


def _run(x, h0, key, quants, params, train):
    """``(out, save, kept, gi)`` of a whole forward call."""
    dims, kept_bytes, scratch_bytes, _ = _plan(*key)
    kind, T, B, I, H = key[:5]
    device = x.device
    out = torch.empty((T, B, H), device=device, dtype=torch.float32)
    # the diagonal backward recomputes its gates from gi, the others read them
    save = torch.empty((4, T, B, H), device=device, dtype=torch.float32) if train and kind != "diagonal" else None
    kept = torch.empty(kept_bytes, device=device, dtype=torch.uint8)
    gi = torch.empty((T, B, 3 * H), device=device, dtype=torch.float32)
    scratch = torch.empty(scratch_bytes, device=device, dtype=torch.uint8)
    ptrs = _FWD_PTRS(x.data_ptr(), h0.data_ptr(), *_addresses(params), out.data_ptr(), None if save is None else save.data_ptr(),
                     kept.data_ptr(), scratch.data_ptr(), gi.data_ptr())
    rc = _call(_lib.load().b200gru_layer_forward, dims[0], quants, ptrs, device)
    if rc:
        _lib._raise(rc, f"{kind} layer forward")
    _lib._after_call()
    return out, save, kept, gi


def _call(fn, dims, quants, ptrs, device):
    index = device.index
    if torch._C._cuda_getDevice() == index:
        return fn(dims, quants, ptrs, torch._C._cuda_getCurrentRawStream(index))
    with torch.cuda.device(index):
        return fn(dims, quants, ptrs, torch._C._cuda_getCurrentRawStream(index))


def _restored(ctx, dtypes):
    """Saved tensors in the form the library reads: saved-tensor hooks may hand back another dtype or layout."""
    device = ctx.device
    return [t if t.dtype is dtype and t.device == device and t.is_contiguous() else t.to(device, dtype).contiguous()
            for t, dtype in zip(ctx.saved_tensors, dtypes)]


# One library call runs the whole forward, but two autograd nodes stand for it, the projection's and the scan's:
# the gradients of the hidden side are complete, and their reduction can start, before the projection's backward runs.
# Both biases belong to the scan's node, whose kernels sum them from one read of dgi.

class ProjectionFunction(torch.autograd.Function):
    """``gi[T,B,3H]``; runs the scan as well and leaves ``(out, save, kept)`` in ``call``, which holds what it needs beside x."""

    @staticmethod
    def forward(ctx, x, key, quants, call, *wi):
        h0, params = call
        out, save, kept, gi = _run(x, h0, key, quants, params, True)
        call[:] = out, save, kept
        ctx.key, ctx.quants, ctx.device = key, quants, x.device
        if any(ctx.needs_input_grad):
            ctx.save_for_backward(x, kept)
        return gi

    @staticmethod
    def backward(ctx, dgi):
        x, kept = _restored(ctx, (torch.float32, torch.uint8))
        need = ctx.needs_input_grad
        kind, T, B, I, H = ctx.key[:5]
        dims, _, _, scratch_bytes = _plan(*ctx.key)
        device = ctx.device
        dgi = dgi.contiguous()
        dx = torch.empty_like(x) if need[0] else None
        dwi = torch.empty((3, H, I), device=device, dtype=torch.float32) if any(need[4:]) else None
        scratch = torch.empty(scratch_bytes, device=device, dtype=torch.uint8)
        ptrs = _BWD_PTRS(x.data_ptr(), None, None, None, None, kept.data_ptr(), scratch.data_ptr(), None if dx is None else dx.data_ptr(),
                         None, None if dwi is None else dwi.data_ptr(), None, None, None, dgi.data_ptr())
        rc = _call(_lib.load().b200gru_layer_backward, dims[2], ctx.quants, ptrs, device)
        if rc:
            _lib._raise(rc, f"{kind} layer backward")
        _lib._after_call()
        grads = dwi.unbind(0) if dwi is not None else (None, None, None)
        return (dx, None, None, None, *(g if n else None for g, n in zip(grads, need[4:])))


class ScanFunction(torch.autograd.Function):
    """``out[T,B,H]`` that the projection's call left in ``call``; ``params``: hidden weights, then (if any) both biases."""

    @staticmethod
    def forward(ctx, gi, h0, key, quants, call, *params):
        out, save, kept = call
        ctx.key, ctx.quants, ctx.nparams, ctx.device = key, quants, len(params), gi.device
        ctx.save_for_backward(h0, out, gi if save is None else save, kept)
        return out

    @staticmethod
    def backward(ctx, dout):
        h0, out, save, kept = _restored(ctx, (torch.float32, torch.float32, torch.float32, torch.uint8))
        need = ctx.needs_input_grad
        kind, T, B, I, H, nblocks, log2_hpad = ctx.key[:7]
        has_bias = ctx.nparams == 9
        want_bi = has_bias and any(need[8:11])
        dims, _, _, scratch_bytes = _plan(*ctx.key)
        device = ctx.device
        dout = dout.contiguous()
        dh0 = torch.empty_like(h0)
        shape = {"dense": (H, H), "diagonal": (H,), "monarch": (nblocks, H // nblocks, H // nblocks),
                 "butterfly": (1, nblocks, log2_hpad, (1 << log2_hpad) // 2, 2, 2)}[kind]
        dwh = torch.empty((3, *shape), device=device, dtype=torch.float32)
        dbi = torch.empty((3, H), device=device, dtype=torch.float32) if want_bi else None
        dbh = torch.empty((3, H), device=device, dtype=torch.float32)
        dgi = torch.empty((T, B, 3 * H), device=device, dtype=torch.float32)
        scratch = torch.empty(scratch_bytes, device=device, dtype=torch.uint8)
        ptrs = _BWD_PTRS(None, h0.data_ptr(), out.data_ptr(), dout.data_ptr(), save.data_ptr(), kept.data_ptr(), scratch.data_ptr(),
                         None, dh0.data_ptr(), None, dwh.data_ptr(), dbi.data_ptr() if want_bi else None, dbh.data_ptr(), dgi.data_ptr())
        rc = _call(_lib.load().b200gru_layer_backward, dims[1], ctx.quants, ptrs, device)
        if rc:
            _lib._raise(rc, f"{kind} layer backward")
        _lib._after_call()
        grads = [dgi, dh0, None, None, None, *dwh.unbind(0)]
        if has_bias:
            grads += [*(dbi.unbind(0) if want_bi else (None, None, None)), *dbh.unbind(0)]
        return tuple(g if n else None for g, n in zip(grads, need))


def forward(layer, x, h0):
    """``out[T,B,H]``, or None where this path does not take the call."""
    from .gru_layer import _extract_h_quant_params
    cell, kind = layer.cell, layer._dispatch_kind
    I, H = cell.input_size, cell.hidden_size
    device = x.device
    if (not cell._input_dense or I % 8 or H % 8 or not _plain_input(x, device) or not _plain_input(h0, device) or
            x.shape[2] != I or h0.dim() != 2 or h0.shape[0] != x.shape[1] or h0.shape[1] != H or _transformed()):
        return None
    mods = cell._modules
    quant_x, quant_wi, quant_wh = mods["quant_x"], [mods["quant_W_i" + g] for g in _GATES], [mods["quant_W_h" + g] for g in _GATES]
    bits_i = _weight_bits(quant_wi)
    bits_h = _weight_bits(quant_wh) if kind == "dense" else 32
    if bits_i is None or bits_h is None:
        return None
    # the composed path calls the input quantizer and, where they are identities, those of dense hidden weights: these are
    # passed by only where nobody could tell
    if (type(quant_x) not in _INPUT_QUANTIZERS or torch.nn.modules.module._has_any_global_hook() or _observed(quant_x) or
            (kind == "dense" and bits_h == 32 and any(map(_observed, quant_wh)))):
        return None
    found = _parameters(cell, kind, device, I, H)
    if found is None:
        return None
    params, nblocks, log2_hpad = found
    T, B = x.shape[0], x.shape[1]
    key = (kind, T, B, I, H, nblocks, log2_hpad, bits_i, bits_h)
    if _plan(*key) is None:
        return None
    grad = torch.is_grad_enabled() and (x.requires_grad or h0.requires_grad or any([p.requires_grad for p in params]))
    qx = None
    if type(quant_x) is not Identity:
        if type(quant_x) is FakeQuantizePerTensor and not grad:
            qx = _extract_h_quant_params(quant_x)
        # the kernel's grid: int8 codes, a scale whose reciprocal is a normal number (the module takes any, negative ones too)
        if qx is None or not 1e-30 < qx[0] < 1e30 or qx[1] < -127 or qx[2] > 127:
            qx, x = None, quant_x(x)
            if not _plain_input(x, device):
                return None
    x, h0 = x.contiguous(), h0.contiguous()
    if x.data_ptr() & 15:
        return None
    quants = _quants(qx, _extract_h_quant_params(mods["quant_h_in"]), _extract_h_quant_params(mods["quant_h_out"]))
    if grad:
        call = [h0, params]
        gi = ProjectionFunction.apply(x, key, quants, call, *params[:3])
        return ScanFunction.apply(gi, h0, key, quants, call, *params[3:])
    return _run(x, h0, key, quants, params, False)[0]


def _plain_input(t, device):
    return type(t) is torch.Tensor and t.dtype is torch.float32 and t.is_cuda and t.device == device
