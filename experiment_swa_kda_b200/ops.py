"""Tensor-level operators over the C ABI: allocation, stream and autograd plumbing only.

PyTorch is used for device memory, the current CUDA stream and autograd bookkeeping;
every arithmetic step runs in libkda_b200.so.  Nothing here falls back to PyTorch math.
The differentiable operators are C++ (_native); the functions that call the C ABI through
ctypes are its thin binding for callers that manage workspaces themselves.
"""

from __future__ import annotations

import contextlib
from typing import Optional, Tuple

import torch

from . import _lib, _native

Tensor = torch.Tensor

_DT = {torch.float32: _lib.DTYPE_F32, torch.bfloat16: _lib.DTYPE_BF16}


def _dt(t: Tensor) -> int:
    try:
        return _DT[t.dtype]
    except KeyError:
        raise RuntimeError(f"KDA kernels take float32 or bfloat16 tensors, got {t.dtype}") from None


def _ptr(t: Optional[Tensor]):
    return None if t is None else t.data_ptr()


def _stream(dev) -> int:
    return torch.cuda.current_stream(dev).cuda_stream


def _need_cuda(*ts):
    dev = None
    for t in ts:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError("KDA CUDA operators cannot run on CPU tensors (there is no CPU fallback)")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise RuntimeError("all KDA tensors must be on the same CUDA device")
    return dev


def _bytes(n: int, dev) -> Tensor:
    return torch.empty(max(int(n), 256), dtype=torch.uint8, device=dev)


# --------------------------------------------------------------------------------------------
# torch.jit traces
# --------------------------------------------------------------------------------------------

@contextlib.contextmanager
def _untraced():
    state = torch._C._get_tracing_state()
    torch._C._set_tracing_state(None)
    try:
        yield
    finally:
        torch._C._set_tracing_state(state)


class _TracedCall(torch.autograd.Function):
    """A native call as one node of a trace: the tracer records Python autograd functions, and the C++ graph that the call
    builds is kept inside and differentiated by the backward."""

    @staticmethod
    def forward(ctx, call, *tensors):
        with _untraced(), torch.enable_grad():
            leaves = [t.detach().requires_grad_(wanted) for t, wanted in zip(tensors, ctx.needs_input_grad[1:])]
            outs = call(*leaves)
            like = [(tuple(o.shape), o.dtype, o.device) for o in outs]
        ctx.inner = leaves, outs
        results = tuple(torch.empty(shape, dtype=dtype, device=device) for shape, dtype, device in like)      # the tracer has to have seen them
        with _untraced():
            for r, o in zip(results, outs):
                r.copy_(o)
        return results

    @staticmethod
    def backward(ctx, *grads):
        leaves, outs = ctx.inner
        pairs = [(o, g) for o, g in zip(outs, grads) if o.requires_grad]
        wanted = [t for t in leaves if t.requires_grad]
        got = iter(torch.autograd.grad([o for o, _ in pairs], wanted, [g for _, g in pairs], retain_graph=True, allow_unused=True))
        return (None, *[next(got) if t.requires_grad else None for t in leaves])


def traced(call, tensors):
    """call(*tensors) -> tuple of tensors and Nones, as one node of the torch.jit trace in progress.  None outside of a trace,
    and where the call itself declines its inputs (answers None)."""
    if torch._C._get_tracing_state() is None:
        return None
    at = [i for i, t in enumerate(tensors) if t is not None]

    def bound(*given):
        full = [None] * len(tensors)
        for i, t in zip(at, given):
            full[i] = t
        return call(*full)

    given = [tensors[i] for i in at]
    with _untraced(), torch.no_grad():
        first = bound(*given)
    if first is None:
        return None
    outs = iter(_TracedCall.apply(lambda *ts: [o for o in bound(*ts) if o is not None], *given))
    return tuple(None if o is None else next(outs) for o in first)


# --------------------------------------------------------------------------------------------
# chunked KDA on activated inputs
# --------------------------------------------------------------------------------------------

def _shape(q, v, g, n_seq, seq_len, scale, l2norm, lane, forward_only=False) -> "_lib.ChunkShape":
    tokens = q.shape[0] * q.shape[1]
    return _lib.ChunkShape(n_seq, seq_len, tokens, q.shape[2], q.shape[3], v.shape[3], _dt(q), _dt(g), lane,
                           1 if l2norm else 0, float(scale), 1 if forward_only else 0)


def poll_status(dev) -> None:
    """Raise if an earlier chunk call on `dev` left a device status (an expired bounded wait, an inconsistent cu_seqlens).
    The kernels write a page-locked host word when something fails, so this is one read of host memory."""
    _native.load().watch_status(torch.device(dev).index or 0)


def chunk_kda_fwd(q, k, v, g, beta, h0, cu_seqlens, scale, l2norm, want_final, lane=_lib.LANE_FP32, forward_only=False, norm=None):
    """Returns (o, final_state or None, saved) where saved = (shape, workspace) for the backward.
    forward_only: inference / prefill - the panels only a backward reads are neither stored nor allocated.
    norm = (gate, weight float32 [V], eps): also apply the gated RMSNorm in the output kernel's epilogue (tensor-core lane
    only); the return value then is (o, final_state, saved, y, inv_rms)."""
    lib = _lib.load()
    dev = _need_cuda(q, k, v, g, beta, h0, cu_seqlens)
    poll_status(dev)
    B, T, H, K = q.shape
    V = v.shape[-1]
    if cu_seqlens is not None:
        n_seq, seq_len = cu_seqlens.numel() - 1, 0
    else:
        n_seq, seq_len = B, T
    sh = _shape(q, v, g, n_seq, seq_len, scale, l2norm, lane, forward_only)
    o = torch.empty(B, T, H, V, dtype=v.dtype, device=dev)
    fs = torch.empty(n_seq, H, V, K, dtype=torch.float32, device=dev) if want_final else None
    nbytes = lib.kda_chunk_workspace_bytes(sh)
    ws = _bytes(nbytes, dev)
    with torch.cuda.device(dev):
        if norm is None:
            rc = lib.kda_chunk_fwd(sh, _ptr(q), _ptr(k), _ptr(v), _ptr(g), _ptr(beta), _ptr(h0), _ptr(cu_seqlens), _ptr(o),
                                   _ptr(fs), _ptr(ws), ws.numel(), _stream(dev))
            _lib.check(rc, "kda_chunk_fwd")
        else:
            gate, nw, eps = norm
            y = torch.empty_like(o)
            inv = torch.empty(B * T * H, dtype=torch.float32, device=dev)
            rc = lib.kda_chunk_fwd_norm(sh, _ptr(q), _ptr(k), _ptr(v), _ptr(g), _ptr(beta), _ptr(h0), _ptr(cu_seqlens), _ptr(o),
                                        _ptr(fs), _ptr(ws), ws.numel(), _ptr(gate), _ptr(nw), float(eps), _ptr(y), _ptr(inv),
                                        _stream(dev))
            _lib.check(rc, "kda_chunk_fwd_norm")
    if norm is not None:
        return o, fs, (sh, ws), y, inv
    return o, fs, (sh, ws)


def chunk_kda_conv_fwd(xq, xk, xv, wq, wk, wv, g, beta, h0, cu_seqlens, scale, l2norm, want_final):
    """No-grad forward with the three short convolutions (width 4, SiLU, zero padding at every sequence start) folded
    into the intra-chunk kernel: xq, xk, xv [B,T,H,128] bf16 are the convolutions' inputs, wq, wk, wv [H*128,4] their
    weights (float32 or bf16).  Tensor-core lane only.  Returns (o, final_state or None), bit-identical to
    conv_fwd x3 followed by chunk_kda_fwd(forward_only=True)."""
    lib = _lib.load()
    dev = _need_cuda(xq, xk, xv, wq, wk, wv, g, beta, h0, cu_seqlens)
    poll_status(dev)
    B, T, H, K = xq.shape
    if cu_seqlens is not None:
        n_seq, seq_len = cu_seqlens.numel() - 1, 0
    else:
        n_seq, seq_len = B, T
    sh = _shape(xq, xv, g, n_seq, seq_len, scale, l2norm, _lib.LANE_TC, True)
    ws_ = [w.contiguous() for w in (wq, wk, wv)]
    if len({w.dtype for w in ws_}) != 1 or ws_[0].dtype not in (torch.float32, torch.bfloat16) or any(w.shape != (H * K, 4) for w in ws_):
        raise ValueError("convolution weights must share one dtype (float32 or bfloat16) and have shape [H*K, 4]")
    o = torch.empty(B, T, H, K, dtype=xv.dtype, device=dev)
    fs = torch.empty(n_seq, H, K, K, dtype=torch.float32, device=dev) if want_final else None
    ws = _bytes(lib.kda_chunk_workspace_bytes(sh), dev)
    with torch.cuda.device(dev):
        rc = lib.kda_chunk_fwd_conv(sh, _ptr(xq), _ptr(xk), _ptr(xv), _ptr(ws_[0]), _ptr(ws_[1]), _ptr(ws_[2]), 4,
                                    _lib.DTYPE_F32 if ws_[0].dtype == torch.float32 else _lib.DTYPE_BF16, _ptr(g), _ptr(beta),
                                    _ptr(h0), _ptr(cu_seqlens), _ptr(o), _ptr(fs), _ptr(ws), ws.numel(), _stream(dev))
        _lib.check(rc, "kda_chunk_fwd_conv")
    return o, fs


def chunk_kda_bwd(q, k, v, g, beta, cu_seqlens, do, dfs, saved, want_dh0):
    lib = _lib.load()
    sh, ws = saved
    dev = q.device
    poll_status(dev)
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    dg, db = torch.empty_like(g), torch.empty_like(beta)
    n_seq = sh.n_seq
    dh0 = torch.empty(n_seq, sh.heads, sh.value_dim, sh.key_dim, dtype=torch.float32, device=dev) if want_dh0 else None
    scr = _bytes(lib.kda_chunk_bwd_scratch_bytes(sh), dev)
    with torch.cuda.device(dev):
        rc = lib.kda_chunk_bwd(sh, _ptr(q), _ptr(k), _ptr(v), _ptr(g), _ptr(beta), _ptr(cu_seqlens), _ptr(do), _ptr(dfs),
                               _ptr(ws), ws.numel(), _ptr(scr), scr.numel(), _ptr(dq), _ptr(dk), _ptr(dv), _ptr(dg),
                               _ptr(db), _ptr(dh0), _stream(dev))
        _lib.check(rc, "kda_chunk_bwd")
    return dq, dk, dv, dg, db, dh0


def chunk_status(saved, dev) -> None:
    """Raise if a bounded device-side wait expired in the kernels that used this workspace (synchronises the stream)."""
    sh, ws = saved
    with torch.cuda.device(dev):
        rc = _lib.load().kda_chunk_status(sh, _ptr(ws), _stream(dev))
    _lib.check(rc, "kda_chunk_status")


# --------------------------------------------------------------------------------------------
# gate activations
# --------------------------------------------------------------------------------------------

class GateFunction:
    """(raw_gate, beta_logits, A_log, dt_bias) -> (g, beta) in float32, differentiable, with the parameter gradients
    reduced deterministically (reference chunk_wy_backward.cu:3881-3987)."""

    @staticmethod
    def apply(raw_gate, beta_logits, A_log, dt_bias, lower_bound):
        out = _native.load().gate(raw_gate, beta_logits, A_log, dt_bias, lower_bound)
        if out is None:
            out = traced(lambda *ts: _native.load().gate(*ts, lower_bound), (raw_gate, beta_logits, A_log, dt_bias))
        if out is None:
            _need_cuda(raw_gate, beta_logits, A_log, dt_bias)
            _dt(raw_gate)
            raise RuntimeError("kda_gate_fwd takes raw_gate [B,T,H,K], beta_logits [B,T,H], A_log [H] and dt_bias with H*K values")
        return out


# --------------------------------------------------------------------------------------------
# decode
# --------------------------------------------------------------------------------------------

def decode_step(q, k, v, g, beta, state, scale, l2norm=True, out_state: Optional[Tensor] = None):
    """One token per sequence.  q,k,g [B,1,H,K] (or [B,H,K]); state [B,H,V,K] float32.
    Returns (o shaped like v, new state).  The input state is left untouched unless
    out_state aliases it."""
    if q.is_cuda:
        out = _native.load().decode_step(q, k, v, g, beta, state, scale, bool(l2norm), out_state)
        if out is not None:
            return out
    lib = _lib.load()
    dev = _need_cuda(q, k, v, g, beta, state)
    q, k, v, g, beta = (t.contiguous() for t in (q, k, v, g, beta))
    if g.dtype != beta.dtype:
        beta = beta.to(g.dtype)
    H, K = q.shape[-2], q.shape[-1]
    V = v.shape[-1]
    n = q.numel() // (H * K)
    if state.dtype != torch.float32 or not state.is_contiguous() or tuple(state.shape) != (n, H, V, K):
        raise ValueError(f"state must be contiguous float32 V-first [B, H, V, K] with shape {(n, H, V, K)}")
    new_state = torch.empty_like(state) if out_state is None else out_state
    o = torch.empty_like(v)
    with torch.cuda.device(dev):
        rc = lib.kda_decode_step(n, H, K, V, _dt(q), _dt(g), 1 if l2norm else 0, float(scale), _ptr(q), _ptr(k), _ptr(v),
                                 _ptr(g), _ptr(beta), _ptr(state), _ptr(new_state), _ptr(o), _stream(dev))
    _lib.check(rc, "kda_decode_step")
    return o, new_state


def decode_step_raw(q, k, v, raw_gate, beta_logits, A_log, dt_bias, lower_bound, state, scale, out_state: Optional[Tensor] = None):
    """One decode token on RAW inputs (gate and beta activations fused into the kernel, q and k L2-normalised): the
    signature of the reference's recurrent_decode operator in a single launch.  `out_state` may be `state` itself."""
    lib = _lib.load()
    dev = _need_cuda(q, k, v, raw_gate, beta_logits, A_log, dt_bias, state)
    q, k, v, raw_gate, beta_logits = (t.contiguous() for t in (q, k, v, raw_gate, beta_logits))
    if not (q.dtype == k.dtype == v.dtype == raw_gate.dtype == beta_logits.dtype):
        raise RuntimeError("decode_step_raw takes q, k, v, raw_gate and beta_logits in one dtype")
    H, K = q.shape[-2], q.shape[-1]
    V = v.shape[-1]
    n = q.numel() // (H * K)
    if state.dtype != torch.float32 or not state.is_contiguous() or tuple(state.shape) != (n, H, V, K):
        raise ValueError(f"state must be contiguous float32 V-first [B, H, V, K] with shape {(n, H, V, K)}")
    if A_log.dtype != torch.float32 or dt_bias.dtype != torch.float32 or A_log.numel() != H or dt_bias.numel() != H * K:
        raise ValueError("A_log [H] and dt_bias [H*K] must be float32")
    new_state = torch.empty_like(state) if out_state is None else out_state
    o = torch.empty_like(v)
    with torch.cuda.device(dev):
        rc = lib.kda_decode_step_raw(n, H, K, V, _dt(q), float(scale), _ptr(q), _ptr(k), _ptr(v), _ptr(raw_gate), _ptr(beta_logits),
                                     _ptr(A_log.contiguous()), _ptr(dt_bias.contiguous()), float(lower_bound), _ptr(state),
                                     _ptr(new_state), _ptr(o), _stream(dev))
    _lib.check(rc, "kda_decode_step_raw")
    return o, new_state


def conv_step_multi(xs, weights, caches, silu=True):
    """One decode token through several same-shaped convolutions in one launch; `caches` ([B,C,W] each) are updated IN
    PLACE.  xs: [B,C] (or [B,1,C]) tensors.  Returns the outputs, shaped like xs."""
    import ctypes as C
    lib = _lib.load()
    xs = [x.contiguous() for x in xs]
    ws = [w.contiguous() for w in weights]
    dev = _need_cuda(*xs, *ws, *caches)
    Bn, Cc, W = caches[0].shape
    for x, w, c in zip(xs, ws, caches):
        if x.numel() != Bn * Cc or tuple(c.shape) != (Bn, Cc, W) or tuple(w.shape) != (Cc, W) or not c.is_contiguous() or c.dtype != x.dtype:
            raise ValueError("conv_step_multi needs x [B,C], weight [C,W] and a contiguous cache [B,C,W] of the activation dtype per branch")
    ys = [torch.empty_like(x) for x in xs]
    with torch.cuda.device(dev):
        rc = lib.kda_conv_step_multi(len(xs), Bn, Cc, W, _dt(xs[0]) | _wflag(xs[0], ws[0]), 1 if silu else 0,
                                     C.cast(_ptr_array(xs), C.c_void_p), C.cast(_ptr_array(ws), C.c_void_p),
                                     C.cast(_ptr_array(caches), C.c_void_p), C.cast(_ptr_array(ys), C.c_void_p), _stream(dev))
    _lib.check(rc, "kda_conv_step_multi")
    return ys


def decode_steps(q, k, v, g, beta, state, scale, l2norm=True):
    """n consecutive decode steps in one library call.  q,k,g [n,B,H,K]; v [n,B,H,V]; beta [n,B,H]; `state` [B,H,V,K]
    float32 is UPDATED IN PLACE.  Returns o [n,B,H,V].  One kernel launch per step, issued from C without a host round
    trip per token (the serving loop of the reference makes one operator call per token: nanochat/engine.py:83-226)."""
    lib = _lib.load()
    dev = _need_cuda(q, k, v, g, beta, state)
    q, k, v, g, beta = (t.contiguous() for t in (q, k, v, g, beta))
    if g.dtype != beta.dtype:
        beta = beta.to(g.dtype)
    n, B, H, K = q.shape
    V = v.shape[-1]
    if state.dtype != torch.float32 or not state.is_contiguous() or tuple(state.shape) != (B, H, V, K):
        raise ValueError(f"state must be contiguous float32 V-first [B, H, V, K] with shape {(B, H, V, K)}")
    o = torch.empty_like(v)
    with torch.cuda.device(dev):
        rc = lib.kda_decode_steps(n, B, H, K, V, _dt(q), _dt(g), 1 if l2norm else 0, float(scale), _ptr(q), _ptr(k), _ptr(v),
                                  _ptr(g), _ptr(beta), _ptr(state), _ptr(o), _stream(dev))
    _lib.check(rc, "kda_decode_steps")
    return o


# --------------------------------------------------------------------------------------------
# short convolution
# --------------------------------------------------------------------------------------------

KDA_WEIGHT_F32 = 0x100


def _wflag(x, weight):
    """float32 weights next to lower-precision activations are read as they are (rounded on load by the kernel)."""
    return KDA_WEIGHT_F32 if (weight.dtype == torch.float32 and x.dtype != torch.float32) else 0


def conv_fwd(x, weight, initial_state, want_final, silu=True):
    lib = _lib.load()
    dev = _need_cuda(x, weight, initial_state)
    B, T, Cc = x.shape
    W = weight.shape[-1]
    y = torch.empty_like(x)
    fin = torch.empty(B, Cc, W, dtype=x.dtype, device=dev) if want_final else None
    with torch.cuda.device(dev):
        rc = lib.kda_conv_fwd(B, T, Cc, W, _dt(x) | _wflag(x, weight), 1 if silu else 0, _ptr(x), _ptr(weight), _ptr(initial_state), _ptr(y),
                              _ptr(fin), _stream(dev))
    _lib.check(rc, "kda_conv_fwd")
    return y, fin


def conv_bwd(x, weight, initial_state, dy, dfin, silu=True):
    lib = _lib.load()
    dev = x.device
    B, T, Cc = x.shape
    W = weight.shape[-1]
    dx = torch.empty_like(x)
    dw = torch.empty(Cc, W, dtype=torch.float32, device=dev)
    dinit = torch.empty_like(initial_state) if initial_state is not None else None
    scr = _bytes(lib.kda_conv_bwd_scratch_bytes(B, T, Cc, W), dev)
    with torch.cuda.device(dev):
        rc = lib.kda_conv_bwd(B, T, Cc, W, _dt(x) | _wflag(x, weight), 1 if silu else 0, _ptr(x), _ptr(weight), _ptr(initial_state), _ptr(dy),
                              _ptr(dfin), _ptr(dx), _ptr(dw), _ptr(dinit), _ptr(scr), scr.numel(), _stream(dev))
    _lib.check(rc, "kda_conv_bwd")
    return dx, dw, dinit


def _ptr_array(ts):
    import ctypes as C
    arr = (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])
    return arr


class ConvMultiFunction:
    """n same-shaped causal convolutions + SiLU (the q, k and v branches of a layer) in one launch each way, differentiable.
    Training path only (no cache, no final state); runs the tensors one by one when the library declines."""

    @staticmethod
    def apply(silu, n, *tensors):
        xs, ws = list(tensors[:n]), list(tensors[n:])
        ys = _native.load().conv_multi(xs, ws, bool(silu))
        if ys is None:
            ys = traced(lambda *ts: _native.load().conv_multi(list(ts[:n]), list(ts[n:]), bool(silu)), tensors)
        return tuple(ys) if ys is not None else tuple(conv(x, w, None, False, silu)[0] for x, w in zip(xs, ws))


def conv(x, weight, initial_state, output_final_state, silu=True):
    """Causal depthwise convolution (+ SiLU) with an explicit cache, differentiable (role of the reference's
    _ProjectConvolutionAutograd, nanochat/mixers/kda.py:439-466).  weight [C,W] or [C,1,W]."""
    out = _native.load().conv(x, weight, initial_state, bool(output_final_state), bool(silu))
    if out is None:
        out = traced(lambda *ts: _native.load().conv(*ts, bool(output_final_state), bool(silu)), (x, weight, initial_state))
    if out is None:
        _need_cuda(x, weight, initial_state)
        _dt(x)
        raise RuntimeError("the convolution takes x [B,T,C], weight [C,W] and a state [B,C,W], none of them empty")
    return out


# --------------------------------------------------------------------------------------------
# gated RMSNorm
# --------------------------------------------------------------------------------------------

def rmsnorm_gate_fwd(x, gate, weight, eps):
    lib = _lib.load()
    dev = _need_cuda(x, gate, weight)
    D = x.shape[-1]
    rows = x.numel() // D
    y = torch.empty_like(x)
    inv = torch.empty(rows, dtype=torch.float32, device=dev)
    with torch.cuda.device(dev):
        rc = lib.kda_rmsnorm_gate_fwd(rows, D, _dt(x), float(eps), _ptr(x), _ptr(gate), _ptr(weight), _ptr(y), _ptr(inv),
                                      _stream(dev))
    _lib.check(rc, "kda_rmsnorm_gate_fwd")
    return y, inv


def rmsnorm_gate_bwd(x, gate, weight, inv, dy):
    lib = _lib.load()
    dev = x.device
    D = x.shape[-1]
    rows = x.numel() // D
    dx, dgate = torch.empty_like(x), torch.empty_like(gate)
    dw = torch.empty(D, dtype=torch.float32, device=dev)
    scr = _bytes(lib.kda_rmsnorm_gate_bwd_scratch_bytes(rows, D), dev)
    with torch.cuda.device(dev):
        rc = lib.kda_rmsnorm_gate_bwd(rows, D, _dt(x), _ptr(x), _ptr(gate), _ptr(weight), _ptr(inv), _ptr(dy), _ptr(dx),
                                      _ptr(dgate), _ptr(dw), _ptr(scr), scr.numel(), _stream(dev))
    _lib.check(rc, "kda_rmsnorm_gate_bwd")
    return dx, dgate, dw


def rmsnorm_gated(x, gate, weight, eps):
    """y = rms_norm(x; w, eps) * sigmoid(gate), differentiable
    (role of the reference's _ProjectRMSNormGateAutograd, nanochat/mixers/kda.py:418-436)."""
    y = _native.load().rmsnorm(x, gate, weight, eps)
    if y is None:
        y, = traced(lambda *ts: None if (out := _native.load().rmsnorm(*ts, eps)) is None else (out,), (x, gate, weight)) or (None,)
    if y is None:
        _need_cuda(x, gate, weight)
        _dt(x)
        if x.numel() == 0 and gate.shape == x.shape:
            return x * gate * weight.to(x.dtype)      # nothing to normalise; keeps the graph
        raise RuntimeError("the gated RMSNorm takes x and gate of one shape and a weight of their last dimension")
    return y
