"""torch custom ops over the C-ABI library: `slotscan::hard_fwd` / `slotscan::hard_bwd` with a registered autograd
formula and fake (meta) implementations, so the op can sit inside torch.compile'd model blocks without a graph
break (the reference calls its scan from compiled blocks, gqa25/train_sh.py:783-793).

torch is plumbing here -- it owns device memory and the stream; every computation is a kernel of libslotscan.so.
"""
import ctypes
from typing import Optional, Tuple

import torch
from torch.utils._device import DeviceContext

from . import _lib

_DT = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16}
# position of each output of hard_fwd
OUT = ("kbuf", "vbuf", "addr", "oold", "kold", "vold", "kfin", "vfin", "ofin", "tfirst", "kiold", "nsqfin", "kinv", "valid")


def _ptr(t):
    return None if t is None or t.numel() == 0 else ctypes.c_void_p(t.data_ptr())


def _stream(dev):
    """The current stream of `dev`, whose index the tensors carry."""
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(dev.index))


class _Here:
    """`with torch.cuda.device(dev)`, free of charge where that device is the current one already."""
    __slots__ = ("dev", "guard")

    def __init__(self, dev):
        self.dev = dev

    def __enter__(self):
        self.guard = None
        if torch._C._cuda_getDevice() != self.dev.index:
            self.guard = torch.cuda.device(self.dev)
            self.guard.__enter__()

    def __exit__(self, *a):
        if self.guard is not None:
            self.guard.__exit__(*a)


# looked up once: plain_call runs in every call
_tracing, _dispatch_modes, _transforms = torch.jit.is_tracing, torch._C._len_torch_dispatch_stack, torch._C._functorch.peek_interpreter_stack
_profiled, _function_modes = torch._C._autograd._profiler_enabled, torch._C._len_torch_function_stack
_is_batched = torch._C._functorch.is_legacy_batchedtensor
_Tensor, _Parameter = torch.Tensor, torch.nn.Parameter


def _modes_watch(n):
    """The mode of `torch.device` and `torch.set_default_device` concerns factory functions alone."""
    return any(type(torch._C._get_function_stack_at(i)) is not DeviceContext for i in range(n))


def plain_call(*ts):
    """True when nothing looks over this call's shoulder and its tensors are ordinary ones: no tracing, compiling, fake or
    functional mode, function mode or profiler; tensors of no other class and no lazy negation.
    The custom op's own wrapping costs about 80 us of host time per call and direction, as much as the kernels of a small
    call take; such a call goes to the same implementation without it, and through an autograd.Function with the same
    backward when a gradient is wanted.  Everything else takes the registered op."""
    if torch.compiler.is_compiling() or _tracing() or _dispatch_modes() or _transforms() is not None or _profiled():
        return False
    modes = _function_modes()
    if modes and _modes_watch(modes):
        return False
    for t in ts:
        if t is not None:
            kind = type(t)
            if kind is not _Tensor and kind is not _Parameter or t.is_neg():
                return False
    return True


def plain_grads(*ts):
    """plain_call for the gradients that come into a backward: also not batched by the older vmap, whose tensors have the
    ordinary class and no memory (`is_grads_batched`, `jacobian(vectorize=True)`)."""
    return plain_call(*ts) and not any(t is not None and _is_batched(t) for t in ts)


def wants_grad(*ts):
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in ts)


def as_flag_bytes(valid):
    """A bool or byte tensor as contiguous bytes; a bool tensor's storage holds them already."""
    valid = valid.contiguous()
    return valid.view(torch.uint8) if valid.dtype == torch.bool else valid.to(torch.uint8)


def _params(k, v, gate, fr, N, G, hard_gate, eps, occ_bin, snap_dtype):
    B, T, H, DK = k.shape
    return _lib.Params(B, T, H, N, DK, v.shape[-1], G, int(hard_gate), int(occ_bin), int(fr.dim() == 3),
                       _DT[k.dtype], _DT[snap_dtype], float(eps))


def _require_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("slotscan ops run on CUDA tensors only: there is no CPU implementation in this package "
                               "(the CPU oracle lives in the test tree)")


def _addr(t):
    return 0 if t is None or t.numel() == 0 else t.data_ptr()


def _fwd_shapes(k, v, N, G, snap_bf16, want_norm, undo_log, new):
    """The output tensors of hard_fwd; `new(shape, dtype)` allocates (real or fake).  Outputs that were not asked
    for have zero elements."""
    B, T, H, DK = k.shape
    DV = v.shape[-1]
    NB = (T + G - 1) // G
    sdt = torch.bfloat16 if snap_bf16 else torch.float32
    f32, i32 = torch.float32, torch.int32
    return (new((B, NB, H, N, DK), sdt), new((B, NB, H, N, DV), sdt), new((B, T, H), i32), new((B, T, H), f32),
            new((B, T, H, DK) if undo_log else (0,), f32), new((B, T, H, DV) if undo_log else (0,), f32),
            new((B * H, N, DK), f32), new((B * H, N, DV), f32), new((B * H, N), f32), new((B * H, N), i32),
            new((B, T, H), f32), new((B * H, N), torch.float64),
            new((B, NB, H, N) if want_norm else (0,), f32), new((B, NB, H, N) if want_norm else (0,), torch.uint8))


def _hard_fwd(k: torch.Tensor, q: Optional[torch.Tensor], v: torch.Tensor, gate: torch.Tensor, fr: torch.Tensor,
             temp: torch.Tensor, K0: Optional[torch.Tensor], V0: Optional[torch.Tensor], o0: Optional[torch.Tensor],
             nsq0: Optional[torch.Tensor], N: int, G: int, hard_gate: bool, eps: float, occ_bin: bool,
             snap_bf16: bool, want_norm: bool, undo_log: bool, qbits: int = 0, qgroup: int = 16
             ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor,
                        torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """k, q, v: contiguous f32 or bf16 (same dtype); gate, fr, temp: contiguous f32.  K0, V0, o0 (f32), nsq0 (f64):
    the state carried in from the preceding chunk, or None.  qbits, qgroup: the storage quantiser of the emitted
    snapshots (codes of slotscan_epilogue_params, 0: none); kinv and valid are then the quantised rows'.  Returns, in the order of `OUT`: kbuf, vbuf, the log
    (addr, oold, kold, vold, kfin, vfin, ofin, tfirst, kiold; include/slotscan.h), nsqfin, kinv, valid."""
    _require_cuda(k, q, v, gate, fr, temp, K0, V0, o0, nsq0)
    dev = k.device
    out = _fwd_shapes(k, v, N, G, snap_bf16, want_norm, undo_log, lambda s, dt: torch.empty(s, device=dev, dtype=dt))
    kbuf, vbuf, addr, oold, kold, vold, kfin, vfin, ofin, tfirst, kiold, nsqfin, kinv, valid = out
    p = _params(k, v, gate, fr, N, G, hard_gate, eps, occ_bin, kbuf.dtype)
    log = _lib.Log(*(_addr(t) for t in (addr, oold, kold, vold, kfin, vfin, ofin, tfirst, kiold)))
    c = lambda t, dt: None if t is None else t.contiguous().to(dt)
    K0, V0, o0, nsq0 = c(K0, torch.float32), c(V0, torch.float32), c(o0, torch.float32), c(nsq0, torch.float64)
    ex = _lib.FwdExtra(_addr(K0), _addr(V0), _addr(o0), _addr(nsq0), _addr(nsqfin), _addr(kinv), _addr(valid),
                       0 if undo_log else 1)
    with _Here(dev):
        rc = _lib.lib().slotscan_hard_fwd_q(ctypes.byref(p), _ptr(k), _ptr(q), _ptr(v), _ptr(gate), _ptr(fr), _ptr(temp),
                                            _ptr(kbuf), _ptr(vbuf), ctypes.byref(log), ctypes.byref(ex),
                                            ctypes.byref(_lib.Storage(qbits, qgroup)), _stream(dev))
    _lib.check(rc, "slotscan_hard_fwd_q")
    return out


hard_fwd = torch.library.custom_op("slotscan::hard_fwd", mutates_args=())(_hard_fwd)


@hard_fwd.register_fake
def _(k, q, v, gate, fr, temp, K0, V0, o0, nsq0, N, G, hard_gate, eps, occ_bin, snap_bf16, want_norm, undo_log, qbits=0,
      qgroup=16):
    return _fwd_shapes(k, v, N, G, snap_bf16, want_norm, undo_log, lambda s, dt: k.new_empty(s, dtype=dt))


def _hard_bwd(k: torch.Tensor, q: Optional[torch.Tensor], v: torch.Tensor, gate: torch.Tensor, fr: torch.Tensor,
             temp: torch.Tensor, addr: torch.Tensor, oold: torch.Tensor, kold: torch.Tensor, vold: torch.Tensor,
             kfin: torch.Tensor, vfin: torch.Tensor, ofin: torch.Tensor, tfirst: torch.Tensor, kiold: torch.Tensor,
             dkbuf: Optional[torch.Tensor], dvbuf: Optional[torch.Tensor], dkinv: Optional[torch.Tensor], N: int, G: int,
             hard_gate: bool, eps: float, occ_bin: bool, snap_bf16: bool, qbits: int = 0, qgroup: int = 16
             ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """Returns dk, dq, dv (dtype of k), dgate (B,T,H) f32, dfr (shape of fr) f32, dtemp (1,) f32.
    With q None, dq holds the search-path part, which the kernel has already added into dk.
    dkinv: the gradient that reached the kinv output of the forward (B,NB,H,N) f32, or None."""
    _require_cuda(k, v)
    if kold.numel() == 0 or vold.numel() == 0:
        raise RuntimeError("slotscan: this forward was run without its undo log (forward-only mode); it has no backward")
    dev = k.device
    sdt = torch.bfloat16 if snap_bf16 else torch.float32
    p = _params(k, v, gate, fr, N, G, hard_gate, eps, occ_bin, sdt)
    L = _lib.lib()
    nbytes = L.slotscan_hard_bwd_scratch_bytes(ctypes.byref(p))
    scratch = torch.empty(nbytes, device=dev, dtype=torch.uint8)
    dk, dq, dv = torch.empty_like(k), torch.empty_like(k), torch.empty_like(v)
    dgate = torch.empty(gate.shape, device=dev, dtype=torch.float32)
    dfr = torch.empty(fr.shape, device=dev, dtype=torch.float32)
    dtemp = torch.empty(1, device=dev, dtype=torch.float32)
    log = _lib.Log(*(t.data_ptr() for t in (addr, oold, kold, vold, kfin, vfin, ofin, tfirst, kiold)))
    with _Here(dev):
        rc = L.slotscan_hard_bwd_q(ctypes.byref(p), _ptr(k), _ptr(q), _ptr(v), _ptr(gate), _ptr(fr), _ptr(temp),
                                   ctypes.byref(log), _ptr(dkbuf), _ptr(dvbuf), _ptr(dkinv),
                                   ctypes.byref(_lib.Storage(qbits, qgroup)), _ptr(scratch), nbytes, _ptr(dk), _ptr(dq),
                                   _ptr(dv), _ptr(dgate), _ptr(dfr), _ptr(dtemp), _stream(dev))
    _lib.check(rc, "slotscan_hard_bwd_q")
    return dk, dq, dv, dgate, dfr, dtemp


hard_bwd = torch.library.custom_op("slotscan::hard_bwd", mutates_args=())(_hard_bwd)


@hard_bwd.register_fake
def _(k, q, v, gate, fr, temp, addr, oold, kold, vold, kfin, vfin, ofin, tfirst, kiold, dkbuf, dvbuf, dkinv, N, G,
      hard_gate, eps, occ_bin, snap_bf16, qbits=0, qgroup=16):
    f = lambda t: t.new_empty(t.shape, dtype=torch.float32)
    return torch.empty_like(k), torch.empty_like(k), torch.empty_like(v), f(gate), f(fr), gate.new_empty(1)


def _setup(ctx, inputs, output):
    k, q, v, gate, fr, temp, K0, V0, o0, nsq0, N, G, hard_gate, eps, occ_bin, snap_bf16, want_norm, undo_log, qbits, qgroup = inputs
    ctx.save_for_backward(k, q, v, gate, fr, temp, *output[2:11])
    ctx.meta = (N, G, hard_gate, eps, occ_bin, snap_bf16, qbits, qgroup)
    ctx.set_materialize_grads(False)


def _backward(ctx, *grads, bwd=None):
    dkbuf, dvbuf, dkinv = grads[0], grads[1], grads[12]
    k, q, v, gate, fr, temp, addr, oold, kold, vold, kfin, vfin, ofin, tfirst, kiold = ctx.saved_tensors
    N, G, hard_gate, eps, occ_bin, snap_bf16, qbits, qgroup = ctx.meta
    sdt = torch.bfloat16 if snap_bf16 else torch.float32
    c = lambda g, dt: None if g is None else g.contiguous().to(dt)
    dk, dq, dv, dgate, dfr, dtemp = (bwd or hard_bwd)(k, q, v, gate, fr, temp, addr, oold, kold, vold, kfin, vfin, ofin, tfirst,
                                             kiold, c(dkbuf, sdt), c(dvbuf, sdt), c(dkinv, torch.float32), N, G, hard_gate,
                                             eps, occ_bin, snap_bf16, qbits, qgroup)
    # no gradient for the carried-in state (K0, V0, o0, nsq0) nor for the integer / flag arguments
    return (dk, (None if q is None else dq), dv, dgate, dfr, dtemp) + (None,) * 14


hard_fwd.register_autograd(_backward, setup_context=_setup)


class _HardScan(torch.autograd.Function):
    """hard_fwd and its backward for a plain_call."""

    @staticmethod
    def forward(ctx, *inputs):
        out = _hard_fwd(*inputs)
        _setup(ctx, inputs, out)
        return out

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, *grads):
        return _backward(ctx, *grads, bwd=_hard_bwd if plain_grads(*grads) else None)


def run_hard_fwd(*args):
    """hard_fwd with every argument given, by the shorter way where that is the same thing."""
    ts = args[:10]
    if not plain_call(*ts):
        return hard_fwd(*args)
    return _HardScan.apply(*args) if wants_grad(*ts) else _hard_fwd(*args)


# ------------------------------------------------------------------------------------------------------------------
# The general scan (soft address, attached address gradient): slotscan_dense_fwd / slotscan_dense_bwd.
def _dense_params(k, v, gate, fr, N, G, hard, hard_gate, eps, detach_addr, occ_bin):
    base = _params(k, v, gate, fr, N, G, hard_gate, eps, occ_bin, torch.float32)
    return _lib.DenseParams(base, int(hard), int(detach_addr))


def _dense_fwd(k: torch.Tensor, q: Optional[torch.Tensor], v: torch.Tensor, gate: torch.Tensor, fr: torch.Tensor,
              temp: torch.Tensor, N: int, G: int, hard: bool, hard_gate: bool, eps: float, detach_addr: bool,
              occ_bin: bool) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor,
                                      torch.Tensor]:
    """Any mode of the scan.  Returns kbuf, vbuf (float32), obuf (B,NB,H,N), addr (B,T,H) int32, kfin, vfin, ofin."""
    _require_cuda(k, q, v, gate, fr, temp)
    B, T, H, DK = k.shape
    DV = v.shape[-1]
    NB = (T + G - 1) // G
    dev = k.device
    e = lambda *s, dt=torch.float32: torch.empty(*s, device=dev, dtype=dt)
    kbuf, vbuf, obuf = e(B, NB, H, N, DK), e(B, NB, H, N, DV), e(B, NB, H, N)
    addr = e(B, T, H, dt=torch.int32)
    kfin, vfin, ofin = e(B * H, N, DK), e(B * H, N, DV), e(B * H, N)
    p = _dense_params(k, v, gate, fr, N, G, hard, hard_gate, eps, detach_addr, occ_bin)
    _lib.check(_lib.lib().slotscan_dense_check(ctypes.byref(p)), "slotscan_dense_check")
    with _Here(dev):
        rc = _lib.lib().slotscan_dense_fwd(ctypes.byref(p), _ptr(k), _ptr(q), _ptr(v), _ptr(gate), _ptr(fr), _ptr(temp),
                                           _ptr(kbuf), _ptr(vbuf), _ptr(obuf), _ptr(addr), _ptr(kfin), _ptr(vfin),
                                           _ptr(ofin), _stream(dev))
    _lib.check(rc, "slotscan_dense_fwd")
    return kbuf, vbuf, obuf, addr, kfin, vfin, ofin


dense_fwd = torch.library.custom_op("slotscan::dense_fwd", mutates_args=())(_dense_fwd)


@dense_fwd.register_fake
def _(k, q, v, gate, fr, temp, N, G, hard, hard_gate, eps, detach_addr, occ_bin):
    B, T, H, DK = k.shape
    DV = v.shape[-1]
    NB = (T + G - 1) // G
    e = lambda *s, dt=torch.float32: k.new_empty(s, dtype=dt)
    return (e(B, NB, H, N, DK), e(B, NB, H, N, DV), e(B, NB, H, N), e(B, T, H, dt=torch.int32), e(B * H, N, DK),
            e(B * H, N, DV), e(B * H, N))


def _dense_bwd(k: torch.Tensor, q: Optional[torch.Tensor], v: torch.Tensor, gate: torch.Tensor, fr: torch.Tensor,
              temp: torch.Tensor, kbuf: torch.Tensor, vbuf: torch.Tensor, obuf: torch.Tensor,
              dkbuf: Optional[torch.Tensor], dvbuf: Optional[torch.Tensor], N: int, G: int, hard: bool, hard_gate: bool,
              eps: float, detach_addr: bool, occ_bin: bool
              ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """dk, dq, dv (dtype of k), dgate, dfr (shape of fr), dtemp (1,).  With q None the search-path part in dq has
    already been added into dk."""
    _require_cuda(k, v, kbuf)
    dev = k.device
    p = _dense_params(k, v, gate, fr, N, G, hard, hard_gate, eps, detach_addr, occ_bin)
    L = _lib.lib()
    nbytes = L.slotscan_dense_bwd_scratch_bytes(ctypes.byref(p))
    scratch = torch.empty(nbytes, device=dev, dtype=torch.uint8)
    dk, dq, dv = torch.empty_like(k), torch.empty_like(k), torch.empty_like(v)
    dgate = torch.empty(gate.shape, device=dev, dtype=torch.float32)
    dfr = torch.empty(fr.shape, device=dev, dtype=torch.float32)
    dtemp = torch.empty(1, device=dev, dtype=torch.float32)
    with _Here(dev):
        rc = L.slotscan_dense_bwd(ctypes.byref(p), _ptr(k), _ptr(q), _ptr(v), _ptr(gate), _ptr(fr), _ptr(temp), _ptr(kbuf),
                                  _ptr(vbuf), _ptr(obuf), _ptr(dkbuf), _ptr(dvbuf), _ptr(scratch), nbytes, _ptr(dk),
                                  _ptr(dq), _ptr(dv), _ptr(dgate), _ptr(dfr), _ptr(dtemp), _stream(dev))
    _lib.check(rc, "slotscan_dense_bwd")
    return dk, dq, dv, dgate, dfr, dtemp


dense_bwd = torch.library.custom_op("slotscan::dense_bwd", mutates_args=())(_dense_bwd)


@dense_bwd.register_fake
def _(k, q, v, gate, fr, temp, kbuf, vbuf, obuf, dkbuf, dvbuf, N, G, hard, hard_gate, eps, detach_addr, occ_bin):
    f = lambda t: t.new_empty(t.shape, dtype=torch.float32)
    return torch.empty_like(k), torch.empty_like(k), torch.empty_like(v), f(gate), f(fr), gate.new_empty(1)


def _dense_setup(ctx, inputs, output):
    k, q, v, gate, fr, temp, N, G, hard, hard_gate, eps, detach_addr, occ_bin = inputs
    ctx.save_for_backward(k, q, v, gate, fr, temp, output[0], output[1], output[2])
    ctx.meta = (N, G, hard, hard_gate, eps, detach_addr, occ_bin)
    ctx.set_materialize_grads(False)


def _dense_backward(ctx, dkbuf, dvbuf, *unused, bwd=None):
    k, q, v, gate, fr, temp, kbuf, vbuf, obuf = ctx.saved_tensors
    c = lambda g: None if g is None else g.contiguous().to(torch.float32)
    dk, dq, dv, dgate, dfr, dtemp = (bwd or dense_bwd)(k, q, v, gate, fr, temp, kbuf, vbuf, obuf, c(dkbuf), c(dvbuf), *ctx.meta)
    return (dk, (None if q is None else dq), dv, dgate, dfr, dtemp) + (None,) * 7


dense_fwd.register_autograd(_dense_backward, setup_context=_dense_setup)


class _DenseScan(torch.autograd.Function):
    """dense_fwd and its backward for a plain_call."""

    @staticmethod
    def forward(ctx, *inputs):
        out = _dense_fwd(*inputs)
        _dense_setup(ctx, inputs, out)
        return out

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, *grads):
        return _dense_backward(ctx, *grads, bwd=_dense_bwd if plain_grads(*grads) else None)


def run_dense_fwd(*args):
    """dense_fwd by the shorter way where that is the same thing."""
    ts = args[:6]
    if not plain_call(*ts):
        return dense_fwd(*args)
    return _DenseScan.apply(*args) if wants_grad(*ts) else _dense_fwd(*args)
