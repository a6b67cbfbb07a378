"""Thin torch-tensor front end of the C ABI: pointer plumbing and output allocation.

Every function here enqueues CUDA work on torch's current stream through
``libzmoe.so`` and returns torch tensors.  Tensors must live on a CUDA device;
there is no CPU path.
"""

from __future__ import annotations

import contextlib
import ctypes
import math

import torch

from . import _lib

_U32_LIKE = (torch.int32, torch.uint32)


def _ptr(t: torch.Tensor | None):
    return None if t is None else t.data_ptr()


# handle of the current stream of a device, without building a Stream object on every call
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (
    lambda index: torch.cuda.current_stream(index).cuda_stream)


def _stream():
    return _raw_stream(torch.cuda.current_device())


_HERE = contextlib.nullcontext()


def _on(dev: torch.device):
    """``dev`` as the current device; nothing to switch where it is that already (some microseconds a call)."""
    return _HERE if torch.cuda.current_device() == dev.index else torch.cuda.device(dev)


def _need_cuda(*tensors: torch.Tensor | None) -> torch.device:
    dev = None
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError(
                "zmlx_b200 kernels run on CUDA tensors only (no CPU fallback); got a tensor on " + str(t.device)
            )
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise RuntimeError(f"tensors on different devices: {dev} and {t.device}")
    assert dev is not None
    return dev


def _dtype_code(t: torch.Tensor) -> int:
    if t.dtype == torch.float32:
        return _lib.F32
    if t.dtype == torch.bfloat16:
        return _lib.BF16
    raise TypeError(f"unsupported dtype {t.dtype}: this build computes in bfloat16 / float32")


def qmode_code(mode: str) -> int:
    if mode == "affine":
        return _lib.Q_AFFINE4
    if mode == "mxfp4":
        return _lib.Q_MXFP4
    raise ValueError(f"unknown quantisation mode {mode!r}")


def plan_bytes(rows: int, E: int) -> int:
    return int(_lib.load().zmoe_plan_bytes(int(rows), int(E)))


def _int32(idx: torch.Tensor) -> torch.Tensor:
    """Flat int32 indices; the uint32 ones that the routers return are taken as they are."""
    idx = idx.reshape(-1).contiguous()
    return idx.view(torch.int32) if idx.dtype == torch.uint32 else idx.to(torch.int32)


def build_plan(rhs: torch.Tensor, E: int, *, M: int = 1, lhs: torch.Tensor | None = None, lhs_div: int = 1,
               out: torch.Tensor | None = None) -> torch.Tensor:
    """Group (lhs, rhs) gather pairs by expert; returns the int32 plan buffer."""
    dev = _need_cuda(rhs, lhs)
    rhs = _int32(rhs)
    if lhs is not None:
        lhs = _int32(lhs)
        if lhs.numel() != rhs.numel():
            raise ValueError("lhs and rhs index counts differ")
    P = rhs.numel()
    nbytes = plan_bytes(P * M, E)
    if out is None:
        out = torch.empty(nbytes // 4, dtype=torch.int32, device=dev)
    with _on(dev):
        _lib.check(_lib.load().zmoe_build_plan(_ptr(lhs), int(lhs_div), _ptr(rhs), P, int(M), int(E), _ptr(out),
                                               out.numel() * 4, _stream()))
    return out


def check_plan(plan: torch.Tensor) -> None:
    """Raise ``ZmoeError(ERR_TIMEOUT)`` if a bounded wait ran out in a grouped matmul on this plan since the last check.
    Synchronises the current stream."""
    with torch.cuda.device(plan.device):
        _lib.check(_lib.load().zmoe_plan_status(_ptr(plan), 1, _stream()))


def qmm_workspace_bytes(rows: int, E: int, K: int, *, rows_hint: int, mode: str) -> int:
    """Size of the workspace of one grouped matmul call; 0 where the call gains nothing from one."""
    return int(_lib.load().zmoe_qmm_workspace_bytes(int(rows), int(E), int(K), int(rows_hint), qmode_code(mode)))


def qmm_workspace(rows: int, E: int, K: int, *, rows_hint: int, mode: str, device) -> torch.Tensor | None:
    """Workspace of one grouped matmul call, from torch's allocator (so it belongs to the current stream and goes back
    to the pool when the call's reference is dropped), or None where the call gains nothing from one."""
    n = qmm_workspace_bytes(rows, E, K, rows_hint=rows_hint, mode=mode)
    if n == 0:
        return None
    try:
        return torch.empty(n, dtype=torch.uint8, device=device)
    except torch.OutOfMemoryError:
        return None  # the kernels that need none still serve the call


def _ws_args(ws: torch.Tensor | None):
    return (None, 0) if ws is None else (_ptr(ws), ws.numel())


def _check_packed(w: torch.Tensor, name: str) -> None:
    if w.dtype not in _U32_LIKE:
        raise TypeError(f"{name} must be uint32-packed (torch.uint32 or torch.int32), got {w.dtype}")
    if not w.is_contiguous():
        raise ValueError(f"{name} must be contiguous")


def gather_qmm_swiglu_rows(x2: torch.Tensor, gate_w, gate_s, gate_b, up_w, up_s, up_b, plan: torch.Tensor, rows: int,
                           *, rows_hint: int, group_size: int = 64, mode: str = "affine",
                           swiglu: int = _lib.SWIGLU_CPU, out: torch.Tensor | None = None) -> torch.Tensor:
    dev = _need_cuda(x2, gate_w, gate_s, gate_b, up_w, up_s, up_b, plan)
    if x2.dtype != torch.bfloat16:
        raise TypeError(f"activations must be bfloat16, got {x2.dtype}")
    _check_packed(gate_w, "gate_w")
    _check_packed(up_w, "up_w")
    E, N, K8 = gate_w.shape
    K = K8 * 8
    if x2.shape[-1] != K or x2.stride(-1) != 1:
        raise ValueError(f"x has inner dimension {x2.shape[-1]}, weights expect {K}")
    if out is None:
        out = torch.empty((rows, N), dtype=torch.bfloat16, device=dev)
    with _on(dev):
        ws = qmm_workspace(rows, E, K, rows_hint=rows_hint, mode=mode, device=dev)
        _lib.check(_lib.load().zmoe_gather_qmm_swiglu_ws(
            _ptr(x2), x2.shape[0], x2.stride(0), _ptr(gate_w), _ptr(gate_s), _ptr(gate_b), _ptr(up_w), _ptr(up_s),
            _ptr(up_b), E, N, K, int(group_size), qmode_code(mode), _ptr(plan), int(rows), int(rows_hint), _ptr(out),
            int(swiglu), *_ws_args(ws), _stream()))
    return out


def gather_qmm_rows(x2: torch.Tensor, w, s, b, plan: torch.Tensor, rows: int, *, rows_hint: int,
                    group_size: int = 64, mode: str = "affine", x_by_output_row: bool = False,
                    out: torch.Tensor | None = None) -> torch.Tensor:
    dev = _need_cuda(x2, w, s, b, plan)
    if x2.dtype != torch.bfloat16:
        raise TypeError(f"activations must be bfloat16, got {x2.dtype}")
    _check_packed(w, "w")
    E, N, K8 = w.shape
    K = K8 * 8
    if x2.shape[-1] != K or x2.stride(-1) != 1:
        raise ValueError(f"x has inner dimension {x2.shape[-1]}, weights expect {K}")
    if out is None:
        out = torch.empty((rows, N), dtype=torch.bfloat16, device=dev)
    with _on(dev):
        ws = qmm_workspace(rows, E, K, rows_hint=rows_hint, mode=mode, device=dev)
        _lib.check(_lib.load().zmoe_gather_qmm_ws(
            _ptr(x2), x2.shape[0], x2.stride(0), _ptr(w), _ptr(s), _ptr(b), E, N, K, int(group_size),
            qmode_code(mode), _ptr(plan), int(rows), int(rows_hint), int(bool(x_by_output_row)), _ptr(out),
            *_ws_args(ws), _stream()))
    return out


def combine(y: torch.Tensor, w: torch.Tensor, mode: int, *, out_t: bool = False,
            residual: torch.Tensor | None = None) -> torch.Tensor:
    """out[t, d] = sum_i w[t, i] * y[t, i, d]; y (T, K, D), w (T, K)."""
    dev = _need_cuda(y, w, residual)
    T, K, D = y.shape
    y = y.contiguous()
    w = w.contiguous()
    fp32_mode = mode in (_lib.COMBINE_FP32, _lib.COMBINE_FP32_NO_FMA)
    out_dtype = torch.float32 if (fp32_mode and not out_t) else torch.bfloat16
    out = torch.empty((T, D), dtype=out_dtype, device=dev)
    if residual is not None:
        residual = residual.contiguous()
        if residual.dtype != torch.bfloat16 or residual.shape != (T, D):
            raise ValueError("residual must be bfloat16 of shape (T, D)")
    if T == 0:
        return out
    with _on(dev):
        for t0 in range(0, T, 65535):
            n = min(T - t0, 65535)
            _lib.check(_lib.load().zmoe_moe_combine(
                _ptr(y[t0:]), _dtype_code(y), _ptr(w[t0:]), _dtype_code(w), n, K, D, int(mode), _ptr(out[t0:]),
                int(out_t), _ptr(residual[t0:]) if residual is not None else None, _stream()))
    return out


def swiglu(gate: torch.Tensor, up: torch.Tensor, *, mode: int = _lib.SWIGLU_PER_OP) -> torch.Tensor:
    """Elementwise silu(gate) * up on bfloat16 tensors of the same shape (``zmoe_swiglu``)."""
    dev = _need_cuda(gate, up)
    if gate.shape != up.shape:
        raise ValueError("swiglu2: gate and up must have the same shape")
    if gate.dtype != torch.bfloat16 or up.dtype != torch.bfloat16:
        raise TypeError(f"swiglu: gate and up must be bfloat16, got {gate.dtype} and {up.dtype}")
    g, u = gate.contiguous(), up.contiguous()
    out = torch.empty_like(g)
    if g.numel() == 0:
        return out
    with _on(dev):
        _lib.check(_lib.load().zmoe_swiglu(_ptr(g), _ptr(u), g.numel(), int(mode), _ptr(out), _stream()))
    return out


def router_softmax_topk(logits: torch.Tensor, k: int, *, flavour: int, bias: torch.Tensor | None = None,
                        renorm: int = 0):
    dev = _need_cuda(logits, bias)
    E = logits.shape[-1]
    l2 = logits.reshape(-1, E).contiguous()
    T = l2.shape[0]
    if bias is not None:
        bias = bias.reshape(-1).to(torch.float32).contiguous()
    w = torch.empty((T, k), dtype=torch.float32, device=dev)
    idx = torch.empty((T, k), dtype=torch.int32, device=dev)
    with _on(dev):
        if T > 0:
            _lib.check(_lib.load().zmoe_router_softmax_topk(_ptr(l2), _dtype_code(l2), T, E, int(k), int(flavour),
                                                            _ptr(bias), int(renorm), _ptr(w), _ptr(idx), _stream()))
    shape = logits.shape[:-1] + (k,)
    return w.reshape(shape), idx.view(torch.uint32).reshape(shape)


def router_sigmoid_topk(logits: torch.Tensor, bias: torch.Tensor, k: int, *, n_group: int = 1, topk_group: int = 1,
                        scale: float = 1.0):
    dev = _need_cuda(logits, bias)
    E = logits.shape[-1]
    l2 = logits.reshape(-1, E).contiguous()
    T = l2.shape[0]
    bias = bias.reshape(-1).to(torch.float32).contiguous()
    w = torch.empty((T, k), dtype=torch.float32, device=dev)
    idx = torch.empty((T, k), dtype=torch.int32, device=dev)
    with _on(dev):
        if T > 0:
            _lib.check(_lib.load().zmoe_router_sigmoid_bias_topk(_ptr(l2), _dtype_code(l2), T, E, int(k), _ptr(bias),
                                                                 int(n_group), int(topk_group),
                                                                 ctypes.c_float(float(scale)), _ptr(w), _ptr(idx),
                                                                 _stream()))
    shape = logits.shape[:-1] + (k,)
    return w.reshape(shape), idx.view(torch.uint32).reshape(shape)


def router_logits(x: torch.Tensor, wr: torch.Tensor, *, out_dtype: torch.dtype = torch.bfloat16) -> torch.Tensor:
    dev = _need_cuda(x, wr)
    if x.dtype != torch.bfloat16 or wr.dtype != torch.bfloat16:
        raise TypeError("router_logits expects bfloat16 activations and weights")
    d = x.shape[-1]
    x2 = x.reshape(-1, d).contiguous()
    wr = wr.contiguous()
    T, E = x2.shape[0], wr.shape[0]
    out = torch.empty((T, E), dtype=out_dtype, device=dev)
    with _on(dev):
        if T > 0:
            _lib.check(_lib.load().zmoe_router_logits(_ptr(x2), _ptr(wr), T, E, d, _ptr(out), _dtype_code(out),
                                                      _stream()))
    return out.reshape(x.shape[:-1] + (E,))


# ------------------------------------------------------------------ the attention side of the decoder


def _dense_bf16(name: str, t: torch.Tensor, numel: int) -> None:
    """The decoder's kernels take pointers only: what they assume about the tensors is checked here."""
    if t.dtype != torch.bfloat16 or not t.is_contiguous() or t.numel() != numel:
        raise ValueError(f"{name}: expected {numel} contiguous bfloat16 values, got {tuple(t.shape)} {t.dtype} with "
                         f"strides {t.stride()}")


def add_rms_norm(h: torch.Tensor, delta: torch.Tensor | None, w: torch.Tensor, eps: float) -> torch.Tensor:
    """``h += delta`` in place (when given), then the RMS norm of the rows of h (R, d) with weight w (d)."""
    dev = _need_cuda(h, delta, w)
    _dense_bf16("h", h, h.numel())
    if delta is not None:
        _dense_bf16("delta", delta, h.numel())
    _dense_bf16("w", w, h.shape[1])
    x = torch.empty_like(h)
    with _on(dev):
        _lib.check(_lib.load().zmoe_add_rms_norm(_ptr(h), _ptr(delta), _ptr(w), ctypes.c_float(eps), h.shape[0],
                                                 h.shape[1], _ptr(x), _stream()))
    return x


def qkv_post(q, k, v, q_norm, k_norm, cos, sin, eps: float, B: int, S: int, pos, k_cache, v_cache) -> torch.Tensor:
    """Normalise and rotate the q and k heads of B*S projected tokens, append k and v to one layer's caches
    (>= B, Hk, max_seq, hd); returns q (B, Hq, S, hd).  ``pos``: position of the first token, or an int64 device scalar."""
    dev = _need_cuda(q, k, v, k_cache, v_cache)
    hk, max_seq, hd = k_cache.shape[-3:]
    hq = q.shape[-1] // hd
    for name, t, heads in (("q", q, hq), ("k", k, hk), ("v", v, hk)):
        _dense_bf16(name, t, B * S * heads * hd)
    out = torch.empty((B, hq, S, hd), dtype=torch.bfloat16, device=dev)
    on_dev = isinstance(pos, torch.Tensor)
    with _on(dev):
        _lib.check(_lib.load().zmoe_qkv_post(
            _ptr(q), _ptr(k), _ptr(v), _ptr(q_norm), _ptr(k_norm), _ptr(cos), _ptr(sin), ctypes.c_float(eps), B, S, hq,
            hk, hd, _ptr(pos) if on_dev else None, 0 if on_dev else int(pos), max_seq, _ptr(out), _ptr(k_cache),
            _ptr(v_cache), _stream()))
    return out


def decode_attention(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, *, npos: int | None = None,
                     pos: torch.Tensor | None = None) -> torch.Tensor | None:
    """Attention of one token per sequence, q (B, Hq, 1, hd), over the first ``npos`` positions of the caches (or up to
    and including the int64 device scalar ``pos``): (B, Hq * hd) bfloat16, or None for head shapes without a kernel."""
    dev = _need_cuda(q, k_cache, v_cache, pos)
    B, hq, _, hd = q.shape
    _dense_bf16("q", q, B * hq * hd)
    hk, max_seq = k_cache.shape[-3], k_cache.shape[-2]
    lib = _lib.load()
    n = int(lib.zmoe_decode_attention_workspace_bytes(B, hq, hk, hd, max_seq if npos is None else npos))
    if n == 0:
        return None
    ws = torch.empty(n, dtype=torch.uint8, device=dev)
    out = torch.empty((B, hq * hd), dtype=torch.bfloat16, device=dev)
    with _on(dev):
        _lib.check(lib.zmoe_decode_attention(_ptr(q), _ptr(k_cache), _ptr(v_cache), B, hq, hk, hd, _ptr(pos),
                                             0 if npos is None else int(npos), max_seq,
                                             ctypes.c_float(1.0 / math.sqrt(hd)), _ptr(ws), n, _ptr(out), _stream()))
    return out
