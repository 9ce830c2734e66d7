"""One call per layer: the argument structures of ``kch_csa_layer``, ``kch_hca_layer`` and ``kch_kda_layer``.

Each function takes a call whose shapes are the ordinary ones of its layer and returns ``None`` for any other, which the
caller then runs step by step (and which names what is wrong with it, where something is).  The same results to the bit either
way: the operators are the same kernels with the same operands, and what Python leaves to torch between them (weights laid one
after the other, a slice widened to fp32) is exact.  Here the launches are issued by the library instead of by Python.
"""
from __future__ import annotations

import torch

from . import _lib


# Bytes of intermediate results up to which a call is issued as one.  They come as one block that lives as long as the call; step
# by step each is freed as soon as it has been read, and the host work that one call saves (0.2 ms a layer) hides behind the
# kernels long before: writing this much takes longer.
WORKSPACE_LIMIT = 1 << 30


def _tag(dt):
    return _lib.KCH_BF16 if dt == torch.bfloat16 else _lib.KCH_F32 if dt == torch.float32 else None


def _dense(x):
    """A [B, T, d] tensor of an ordinary type on the GPU whose rows are dense and one after the other."""
    return x.is_cuda and x.dim() == 3 and x.is_contiguous() and x.numel() > 0 and type(x) in (torch.Tensor, torch.nn.Parameter)


def _weight(w, rows, cols, x):
    return w.dtype == x.dtype and w.device == x.device and w.dim() == 2 and w.shape[1] == cols and (rows is None or w.shape[0] == rows) \
        and w.stride(1) == 1 and w.stride(0) >= cols


def _biases(shape, x, *biases):
    b0 = biases[0]
    return all(b.device == x.device and b.dtype == b0.dtype and b.is_contiguous() and b.numel() >= s for b, s in zip(biases, shape)) \
        and _tag(b0.dtype) is not None


def _sink_ok(sink, nh, x):
    return sink is None or (sink.device == x.device and sink.numel() == nh and sink.is_contiguous() and _tag(sink.dtype) is not None)


def _parts(dst, weights, K):
    """Weights that the call fuses itself; False where 16-byte copies cannot read one."""
    es = weights[0].element_size()
    if K * es % 16:
        return False
    for i, w in enumerate(weights):
        if w.stride(0) * es % 16 or w.data_ptr() % 16:
            return False
        dst[i].w, dst[i].ld, dst[i].rows = w.data_ptr(), w.stride(0), w.shape[0]
    return True


def _common(l, x, out, norm, W_o, residual):
    B, T, d = x.shape
    l.B, l.T, l.d, l.dtype, l.x, l.ld_x = B, T, d, _tag(x.dtype), x.data_ptr(), d
    l.out = out.data_ptr()
    if norm is not None:
        l.norm_w, l.norm_b, l.norm_dtype, l.eps = norm.weight.data_ptr(), norm.bias.data_ptr(), _tag(norm.weight.dtype), norm.eps
    if W_o is not None:
        l.W_o, l.ld_wo, l.d_out = W_o.data_ptr(), W_o.stride(0), W_o.shape[0]
        if residual is not None:
            l.residual, l.ld_res = residual.data_ptr(), W_o.shape[0]


def _norm_ok(norm, x):
    w, b = norm.weight, norm.bias
    return (w is not None and b is not None and w.dtype == b.dtype and _tag(w.dtype) is not None and w.device == b.device == x.device
            and w.numel() == b.numel() == x.shape[-1] and w.is_contiguous() and b.is_contiguous())


def _out_ok(W_o, width, residual, x):
    return _weight(W_o, None, width, x) and (residual is None or (
        _dense(residual) and residual.dtype == x.dtype and residual.device == x.device
        and residual.shape[:2] == x.shape[:2] and residual.shape[2] == W_o.shape[0]))


def _run(a, size_fn, call_fn, x):
    with _lib.device(x.device):
        need = size_fn(a)
        if need > WORKSPACE_LIMIT:
            return False
        ws = torch.empty(need, dtype=torch.uint8, device=x.device)       # (the caching allocator's blocks start on 512 bytes)
        a.l.workspace, a.l.workspace_bytes = ws.data_ptr(), need
        _lib.check(call_fn(a, _lib.stream()))
    return True


def csa_layer(x, weights, Ba, Bb, B_idx, sink, *, m, topk, nh, nIh, c, c_I, dc, scale, sliding_window, W=None, Wq=None, norm=None,
              W_o=None, residual=None, want_proj=False, want_rows=False):
    """``(out, proj or None, rows or None)``, ``rows``: the compressed rows and indexer keys in fp32; ``weights``: the ten matrices
    in the order a | b keys, a | b gates, indexer key | gate, query down, indexer weights, queries, indexer queries, or None
    where ``W`` and ``Wq`` are given."""
    d = x.shape[-1]
    if not _dense(x) or _tag(x.dtype) is None or x.shape[1] < m:
        return None
    if not _biases((m * c, m * c, m * c_I), x, Ba, Bb, B_idx) or not _sink_ok(sink, nh, x):
        return None
    used, used_q = 4 * c + 2 * c_I + dc + nIh, nh * c + nIh * c_I
    a = _lib.CsaLayerArgs()
    if W is not None and Wq is not None:
        if not _weight(W, None, d, x) or not _weight(Wq, None, dc, x) or W.shape[0] < used or Wq.shape[0] < used_q:
            return None
        a.W, a.ld_w, a.n_w, a.Wq, a.ld_wq, a.n_q = W.data_ptr(), W.stride(0), W.shape[0], Wq.data_ptr(), Wq.stride(0), Wq.shape[0]
    else:
        rows = (c, c, c, c, c_I, c_I, dc, nIh, nh * c, nIh * c_I)
        if not all(_weight(w, r, d if i < 8 else dc, x) for i, (w, r) in enumerate(zip(weights, rows))):
            return None
        if not _parts(a.parts, weights[:8], d) or weights[8].element_size() * dc % 16:
            return None
        for i in (8, 9):
            w = weights[i]
            if w.stride(0) * w.element_size() % 16 or w.data_ptr() % 16:
                return None
            a.parts[i].w, a.parts[i].ld, a.parts[i].rows = w.data_ptr(), w.stride(0), w.shape[0]
        a.n_w, a.n_q = used + (-used) % 8, used_q
    if norm is not None and not _norm_ok(norm, x):
        return None
    if W_o is not None and not _out_ok(W_o, nh * c, residual, x):
        return None
    B, T = x.shape[:2]
    out = torch.empty(B, T, W_o.shape[0] if W_o is not None else nh * c, dtype=x.dtype, device=x.device)
    proj = rows = None
    if want_proj:
        proj = torch.empty(B, T, a.n_w, dtype=x.dtype, device=x.device)
        a.proj = proj.data_ptr()
    if want_rows:
        rows = (torch.empty(B, T // m, c, dtype=torch.float32, device=x.device),
                torch.empty(B, T // m, c_I, dtype=torch.float32, device=x.device))
        a.comp, a.kcomp = rows[0].data_ptr(), rows[1].data_ptr()
    _common(a.l, x, out, norm, W_o, residual)
    a.c, a.c_I, a.dc, a.nh, a.nIh, a.m, a.topk, a.sliding_window, a.T_blocks, a.scale = \
        c, c_I, dc, nh, nIh, m, topk, sliding_window, T // m, scale
    a.Ba, a.Bb, a.B_idx, a.bias_dtype = Ba.data_ptr(), Bb.data_ptr(), B_idx.data_ptr(), _tag(Ba.dtype)
    if sink is not None:
        a.sink, a.sink_dtype = sink.data_ptr(), _tag(sink.dtype)
    lib = _lib.load()
    if not _run(a, lib.kch_csa_layer_workspace_bytes, lib.kch_csa_layer, x):
        return None
    return out, proj, rows


def hca_layer(x, weights, B_pos, sink, *, m2, nh, c, dc, scale, sliding_window, W=None, Wq=None, norm=None, W_o=None, residual=None,
              want_proj=False, want_rows=False):
    """``(out, proj or None, rows or None)``; ``weights``: keys, gates and query down-projection, or None where ``W`` is given."""
    d = x.shape[-1]
    if not _dense(x) or _tag(x.dtype) is None or x.shape[1] < m2:
        return None
    if not _biases((m2 * c,), x, B_pos) or not _sink_ok(sink, nh, x) or not _weight(Wq, nh * c, dc, x):
        return None
    used = 2 * c + dc
    a = _lib.HcaLayerArgs()
    if W is not None:
        if not _weight(W, None, d, x) or W.shape[0] < used:
            return None
        a.W, a.ld_w, a.n_w = W.data_ptr(), W.stride(0), W.shape[0]
    else:
        if not all(_weight(w, r, d, x) for w, r in zip(weights, (c, c, dc))) or not _parts(a.parts, weights, d):
            return None
        a.n_w = used + (-used) % 8
    if norm is not None and not _norm_ok(norm, x):
        return None
    if W_o is not None and not _out_ok(W_o, nh * c, residual, x):
        return None
    B, T = x.shape[:2]
    out = torch.empty(B, T, W_o.shape[0] if W_o is not None else nh * c, dtype=x.dtype, device=x.device)
    proj = rows = None
    if want_proj:
        proj = torch.empty(B, T, a.n_w, dtype=x.dtype, device=x.device)
        a.proj = proj.data_ptr()
    if want_rows:
        rows = (torch.empty(B, T // m2, c, dtype=torch.float32, device=x.device), None)
        a.comp = rows[0].data_ptr()
    _common(a.l, x, out, norm, W_o, residual)
    a.c, a.dc, a.nh, a.m2, a.sliding_window, a.T_blocks, a.scale = c, dc, nh, m2, sliding_window, T // m2, scale
    a.Wq, a.ld_wq = Wq.data_ptr(), Wq.stride(0)
    a.B_pos, a.bias_dtype = B_pos.data_ptr(), _tag(B_pos.dtype)
    if sink is not None:
        a.sink, a.sink_dtype = sink.data_ptr(), _tag(sink.dtype)
    lib = _lib.load()
    if not _run(a, lib.kch_hca_layer_workspace_bytes, lib.kch_hca_layer, x):
        return None
    return out, proj, rows


def kda_layer(x, cfg, W, W_gup, W_o, conv_w, conv_b, state, lookback, *, scale, norm=None, residual=None, state_out=None):
    """``(out, state, lookback)`` of a call over T >= 2 tokens; ``state_out`` (fp32, dense, not ``state``) receives the state."""
    if not _dense(x) or _tag(x.dtype) is None or x.shape[1] < 2 or (norm is not None and not _norm_ok(norm, x)):
        return None
    B, T, d = x.shape
    H, HV, K, V = cfg.n_heads_qk, cfg.n_heads_v, cfg.head_dim_k, cfg.head_dim_v
    if K > 128 or cfg.kda_chunk_size < 1:
        return None
    if not _weight(W, None, d, x) or W.shape[0] % 8 or not _weight(W_gup, HV * K, K, x) or not _out_ok(W_o, HV * V, residual, x):
        return None
    if not (conv_w.dtype == conv_b.dtype == x.dtype and conv_w.is_contiguous() and conv_b.is_contiguous() and conv_w.device == x.device
            and conv_w.numel() == 3 * d and conv_b.numel() == d):
        return None
    if (H * K) % 8 or (HV * V) % 8 or K % 8:         # slices of the projection that the operator reads in place
        return None
    if lookback is not None and not (lookback.dtype == x.dtype and lookback.device == x.device and lookback.is_contiguous()
                                     and lookback.shape == (B, 2, d)):
        return None
    if state is not None and not (state.dtype == torch.float32 and state.device == x.device and state.is_contiguous()
                                  and state.shape == (B, HV, K, V)):
        return None
    a = _lib.KdaLayerArgs()
    out = torch.empty(B, T, W_o.shape[0], dtype=x.dtype, device=x.device)
    new_state = torch.empty(B, HV, K, V, dtype=torch.float32, device=x.device) if state_out is None else state_out
    new_lookback = torch.empty(B, 2, d, dtype=x.dtype, device=x.device)
    _common(a.l, x, out, norm, W_o, residual)
    a.H, a.HV, a.K, a.V, a.chunk_size = H, HV, K, V, cfg.kda_chunk_size
    a.scale, a.decay_scale, a.g_clamp_min = scale, cfg.kda_decay_scale, -10.0
    a.lookback, a.lookback_out = _lib.ptr(lookback), new_lookback.data_ptr()
    a.conv_w, a.conv_b = conv_w.data_ptr(), conv_b.data_ptr()
    a.W, a.ld_w, a.n_w, a.W_gup, a.ld_wg = W.data_ptr(), W.stride(0), W.shape[0], W_gup.data_ptr(), W_gup.stride(0)
    a.state, a.state_out = _lib.ptr(state), new_state.data_ptr()
    lib = _lib.load()
    if not _run(a, lib.kch_kda_layer_workspace_bytes, lib.kch_kda_layer, x):
        return None
    return out, new_state, new_lookback
