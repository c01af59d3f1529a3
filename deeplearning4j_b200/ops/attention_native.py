"""Scaled dot-product attention on the native kernels.

Reference formulation: ``libnd4j/include/helpers/impl/AttentionHelper.cpp:189-470`` (matmul,
scale, mask add, softmax over the full score matrix, matmul) and the ``dot_product_attention``
/ ``multi_head_dot_product_attention`` ops.  Here every matmul is one launch of the batched
tcgen05 GEMM over strided views of the packed projection buffer (no transposes, no per-head
copies), the scale is folded into the GEMM epilogue, masking + softmax is one in-place fused
kernel, and the backward pass is four batched GEMMs plus one fused softmax-gradient kernel.
The output is produced directly in ``[B, Tq, H, D]`` memory order so the following
``[B*Tq, H*D]`` reshape for the output projection is free.
"""
from __future__ import annotations

import ctypes

import torch

from . import native

_LONG2 = ctypes.c_long * 2


def _ok_view(t):
    """[B, H, T, D] view usable by a rank-4 tensor map: unit inner stride, 16-byte aligned strides, none of them 0 (an expanded axis)."""
    s = t.stride()
    return len(s) == 4 and s[3] == 1 and not (s[0] | s[1] | s[2]) & 7 and s[0] and s[1] and s[2] and t.data_ptr() % 16 == 0 and t.size(3) % 8 == 0


def _prep(t):
    # a copy also where the tensor counts as contiguous: an extent of one leaves its stride open, and the map wants all of them aligned
    return t if _ok_view(t) else t.clone(memory_format=torch.contiguous_format)


def _bgemm(l, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, alpha, H, Bn, a_bs, b_bs, c_bs, dtype, out_fp32=0):
    if not hasattr(l.dl4j_gemm_batched, "_typed"):
        vp, i32, lng, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_long, ctypes.c_float
        l.dl4j_gemm_batched.argtypes = [vp, vp, vp, i32, i32, i32, lng, lng, lng, i32, i32, i32, i32, f32, i32, i32, i32, i32,
                                        ctypes.POINTER(ctypes.c_long), ctypes.POINTER(ctypes.c_long),
                                        ctypes.POINTER(ctypes.c_long), vp]
        l.dl4j_gemm_batched.restype = ctypes.c_int
        l.dl4j_gemm_batched._typed = True
    bn = 256 if N > 128 else 128
    rc = l.dl4j_gemm_batched(ctypes.c_void_p(A), ctypes.c_void_p(B), ctypes.c_void_p(C), M, N, K, lda, ldb, ldc, a_mn, b_mn,
                             native._DT[dtype], out_fp32, float(alpha), bn, native.num_sms(), H, Bn, _LONG2(*a_bs),
                             _LONG2(*b_bs), _LONG2(*c_bs), native._stream())
    native._check(rc, "dl4j_gemm_batched")


def _typed_softmax(l):
    if not hasattr(l.dl4j_attn_softmax_fwd, "_typed"):
        vp, i32, i64, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
        l.dl4j_attn_softmax_fwd.argtypes = [vp, vp, i64, i32, i32, i32, vp]
        l.dl4j_attn_softmax_fwd.restype = ctypes.c_int
        l.dl4j_attn_softmax_bwd.argtypes = [vp, vp, i64, i32, f32, i32, vp]
        l.dl4j_attn_softmax_bwd.restype = ctypes.c_int
        l.dl4j_attn_softmax_fwd._typed = True


class _AttentionFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, key_mask, scale, dropout_p=0.0, flags=0):
        l = native.require()
        _typed_softmax(l)
        q, k, v = _prep(q), _prep(k), _prep(v)
        Bn, H, Tq, D = q.shape
        Tk = k.shape[2]
        dt = q.dtype
        ctx.flash = (USE_FLASH or dropout_p > 0.0 or flags) and scale >= 0.0 and flash_supported(q, k, v)
        if ctx.flash:
            # fused kernel: the score matrix stays in tensor memory; only O and the row log-sum-exp are written
            seed = _next_dropout_seed(q.device) if dropout_p > 0.0 else None
            mk = key_mask.to(torch.float32).contiguous() if key_mask is not None else None
            O, lse = flash_forward(q, k, v, mk, scale, dropout_p, seed, flags)
            ctx.save_for_backward(q, k, v, O, lse, mk, seed)
            ctx.scale, ctx.dropout_p, ctx.flags = scale, float(dropout_p), flags
            return O.permute(0, 2, 1, 3)
        if dropout_p > 0.0:
            raise RuntimeError("attention dropout needs the fused kernels (head size up to 64, key length a multiple of 128)")
        P = torch.empty((Bn, H, Tq, Tk), dtype=dt, device=q.device)
        # S = scale * Q K^T
        _bgemm(l, q.data_ptr(), k.data_ptr(), P.data_ptr(), Tq, Tk, D, q.stride(2), k.stride(2), Tk, 0, 0, scale, H, Bn,
               (q.stride(1), q.stride(0)), (k.stride(1), k.stride(0)), (Tq * Tk, H * Tq * Tk), dt)
        mk = None
        if key_mask is not None:
            mk = key_mask.to(torch.float32).contiguous()
        rc = l.dl4j_attn_softmax_fwd(native._ptr(P), native._ptr(mk), Bn * H * Tq, Tk, H * Tq, native._DT[dt], native._stream())
        native._check(rc, "dl4j_attn_softmax_fwd")
        # O = P V, written as [B, Tq, H, D]
        O = torch.empty((Bn, Tq, H, D), dtype=dt, device=q.device)
        _bgemm(l, P.data_ptr(), v.data_ptr(), O.data_ptr(), Tq, D, Tk, Tk, v.stride(2), H * D, 0, 1, 1.0, H, Bn,
               (Tq * Tk, H * Tq * Tk), (v.stride(1), v.stride(0)), (D, Tq * H * D), dt)
        ctx.save_for_backward(q, k, v, P)
        ctx.scale = scale
        return O.permute(0, 2, 1, 3)

    @staticmethod
    def backward(ctx, dO):
        l = native.require()
        if ctx.flash:
            q, k, v, O, lse, mk, seed = ctx.saved_tensors
            if torch.is_grad_enabled() and seed is None:     # create_graph: the gradient has to be differentiable itself
                return (*_grad_in_ops(q, k, v, dO, mk, ctx.scale, ctx.flags), None, None, None, None)
            dO = _prep(dO)
            dvec = torch.empty_like(lse)             # D_r = sum_d dO * O per query row, laid out like the log-sum-exp
            Bn, H, Tq, D = q.shape
            rc = _flash_lib().dl4j_attn_dvec(native._ptr(dO), _LONG3(*dO.stride()[:3]), native._ptr(O), native._ptr(dvec), Bn, H, Tq, D,
                                             native._stream())
            native._check(rc, "dl4j_attn_dvec")
            return (*_flash_backward(q, k, v, dO, lse, dvec, mk, ctx.scale, ctx.flags, ctx.dropout_p, seed), None, None, None, None)
        q, k, v, P = ctx.saved_tensors
        Bn, H, Tq, D = q.shape
        Tk = k.shape[2]
        dt = q.dtype
        dO = _prep(dO)
        same_len = Tq == Tk
        # packed gradient buffer [B, T, 3, H, D] when possible so the three results share one allocation
        if same_len:
            dqkv = torch.empty((Bn, Tq, 3, H, D), dtype=dt, device=q.device)
            dq_t, dk_t, dv_t = dqkv[:, :, 0], dqkv[:, :, 1], dqkv[:, :, 2]          # [B, T, H, D] views
        else:
            dq_t = torch.empty((Bn, Tq, H, D), dtype=dt, device=q.device)
            dk_t = torch.empty((Bn, Tk, H, D), dtype=dt, device=q.device)
            dv_t = torch.empty((Bn, Tk, H, D), dtype=dt, device=q.device)
        pbs = (Tq * Tk, H * Tq * Tk)

        def obs(t):   # batch strides (head, example) and row stride of a [B, T, H, D] output view
            return (t.stride(2), t.stride(0)), t.stride(1)
        # dV = P^T dO
        cbs, ldc = obs(dv_t)
        _bgemm(l, P.data_ptr(), dO.data_ptr(), dv_t.data_ptr(), Tk, D, Tq, Tk, dO.stride(2), ldc, 1, 1, 1.0, H, Bn,
               pbs, (dO.stride(1), dO.stride(0)), cbs, dt)
        # dP = dO V^T
        dP = torch.empty_like(P)
        _bgemm(l, dO.data_ptr(), v.data_ptr(), dP.data_ptr(), Tq, Tk, D, dO.stride(2), v.stride(2), Tk, 0, 0, 1.0, H, Bn,
               (dO.stride(1), dO.stride(0)), (v.stride(1), v.stride(0)), pbs, dt)
        rc = l.dl4j_attn_softmax_bwd(native._ptr(P), native._ptr(dP), Bn * H * Tq, Tk, float(ctx.scale), native._DT[dt],
                                     native._stream())
        native._check(rc, "dl4j_attn_softmax_bwd")
        # dQ = dS K
        cbs, ldc = obs(dq_t)
        _bgemm(l, dP.data_ptr(), k.data_ptr(), dq_t.data_ptr(), Tq, D, Tk, Tk, k.stride(2), ldc, 0, 1, 1.0, H, Bn,
               pbs, (k.stride(1), k.stride(0)), cbs, dt)
        # dK = dS^T Q
        cbs, ldc = obs(dk_t)
        _bgemm(l, dP.data_ptr(), q.data_ptr(), dk_t.data_ptr(), Tk, D, Tq, Tk, q.stride(2), ldc, 1, 1, 1.0, H, Bn,
               pbs, (q.stride(1), q.stride(0)), cbs, dt)
        return dq_t.permute(0, 2, 1, 3), dk_t.permute(0, 2, 1, 3), dv_t.permute(0, 2, 1, 3), None, None, None, None


def _grad_in_ops(q, k, v, dO, mask, scale, flags):
    """(dq, dk, dv) in differentiable torch operators, for second derivatives; the fused kernels' rules for hidden keys and empty rows."""
    s = torch.matmul(q, k.transpose(-1, -2)).float() * scale
    hidden = None
    if flags & 1:
        hidden = torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1)
    if mask is not None:
        m = (mask == 0)[:, None, None, :]
        hidden = m if hidden is None else hidden | m
    if hidden is not None:
        s = s.masked_fill(hidden, float("-inf"))
        if not flags & 2:
            s = s.masked_fill(hidden.expand(s.shape).all(-1, keepdim=True), 0.0)
    p = torch.softmax(s, -1)
    if hidden is not None and not flags & 2:
        p = p.masked_fill(hidden, 0.0)
    dv = torch.matmul(p.to(dO.dtype).transpose(-1, -2), dO)
    dp = torch.matmul(dO, v.transpose(-1, -2)).float()
    ds = p * (dp - (dp * p).sum(-1, keepdim=True)) * scale
    if hidden is not None:
        ds = ds.masked_fill(hidden, 0.0)
    ds = ds.to(q.dtype)
    return torch.matmul(ds, k), torch.matmul(ds.transpose(-1, -2), q), dv


def _bad_mask(q, k, mask):
    return mask is not None and (mask.dim() != 2 or mask.shape[0] != q.shape[0] or mask.shape[1] != k.shape[2])


def _empty_rows_are_zero(D, Tq, Tk):
    """What a query whose keys are all masked gets.  The lengths that have always run on these kernels give 0; on the others, which
    the softmax over -inf served before, and with a causal mask it is NaN, and stays so."""
    return Tk % 128 == 0 or (D % 8 == 0 and Tk % 8 == 0 and Tq % 8 == 0 and Tk <= 1024)


def attention(q, k, v, mask, scale, dropout_p=0.0, causal=False):
    """q, k, v: [B, H, T, D]; ``mask``: None or a [B, Tk] key mask (non-zero = attend); ``dropout_p``: probability of dropping an
    attention weight (training); ``causal``: query i sees the keys 0 .. i.  Returns None when the case is not covered by the native
    kernels.

    bf16 with head sizes up to 64 runs on the fused kernels for any number of queries and keys (the copy engine zero-fills narrower
    heads and the last key block); other head sizes and fp16 on batched GEMMs with a materialised score matrix."""
    if not native.available() or q.dim() != 4 or q.dtype not in (torch.bfloat16, torch.float16):
        return None
    if _bad_mask(q, k, mask) or not native.on_current_device(q, k, v, mask) or not native._plain_autograd():
        return None
    _, _, Tq, D = q.shape
    Tk = k.size(2)
    scale = float(scale) if scale is not None else D ** -0.5
    # the fused kernels take a row's maximum over raw scores: with a negative scale that is the smallest exponent, and exp overflows
    fused = scale >= 0.0 and flash_supported(q, k, v)
    if dropout_p > 0.0 and (not fused or Tk % 128 or causal):
        return None
    if fused and (USE_FLASH or dropout_p > 0.0):
        flags = (1 if causal else 0) | (0 if _empty_rows_are_zero(D, Tq, Tk) and not causal else 2)
        if dropout_p == 0.0 and not (torch.is_grad_enabled() and (q.requires_grad or k.requires_grad or v.requires_grad)):
            return flash_forward(q, k, v, mask, scale, flags=flags)[0].permute(0, 2, 1, 3)       # nothing to differentiate
        # laid out here and not in forward(): second derivatives go through the saved operands
        return _AttentionFn.apply(_prep(q), _prep(k), _prep(v), mask, scale, float(dropout_p), flags)
    if causal or D % 8 or Tk % 8 or Tq % 8 or Tk > 1024 or k.shape != v.shape or q.shape[:2] != k.shape[:2] or D != k.shape[3] \
            or not q.dtype == k.dtype == v.dtype:
        return None
    return _AttentionFn.apply(q, k, v, mask, scale, float(dropout_p))


def attention_grad(q, k, v, mask, scale, dout, causal=False):
    """(dq, dk, dv) without materialising the output: the forward kernel hands the row sums of dO * O straight to the backward kernel.
    None when the fused kernels do not cover the case."""
    if not USE_FLASH or not native.available() or not flash_supported(q, k, v) or _bad_mask(q, k, mask) or dout.dim() != 4 \
            or not native.on_current_device(q, k, v, mask, dout) or not native._plain_autograd() or dout.shape != (*q.shape[:3], v.shape[3]):
        return None
    scale = float(scale) if scale is not None else q.shape[3] ** -0.5
    if not scale >= 0.0:
        return None
    q, k, v, dout = _prep(q.detach()), _prep(k.detach()), _prep(v.detach()), _prep(dout.detach().to(q.dtype))
    Bn, H, Tq, D = q.shape
    flags = (1 if causal else 0) | (0 if _empty_rows_are_zero(D, Tq, k.shape[2]) and not causal else 2)
    mk = mask.detach().to(torch.float32).contiguous() if mask is not None else None
    stats = q.new_empty((2, Bn, H, Tq), dtype=torch.float32)
    lse, dvec = stats[0], stats[1]
    rc = _flash_lib().dl4j_flash_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), None, lse.data_ptr(), native._ptr(mk), Bn, H, Tq,
                                          k.size(2), D, _LONG3(*q.stride()[:3]), _LONG3(*k.stride()[:3]), _LONG3(*v.stride()[:3]), scale,
                                          flags, dout.data_ptr(), _LONG3(*dout.stride()[:3]), dvec.data_ptr(), 0.0, None,
                                          native._stream())
    native._check(rc, "dl4j_flash_attn_fwd")
    return _flash_backward(q, k, v, dout, lse, dvec, mk, scale, flags, 0.0, None)


# Dropout seeds live on the device: every fused forward call with dropout takes a private copy of the running seed and
# advances it, both with device-side operations, so a captured CUDA graph draws a new mask at every replay; the backward pass
# reads the forward's copy.
_DROPOUT_SEED = {}


def set_dropout_seed(seed, device=None):
    """(Re)starts the attention-dropout seed sequence of ``device`` (default: the current CUDA device)."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    _DROPOUT_SEED[device] = torch.tensor([int(seed) & 0x7fffffffffffffff], dtype=torch.int64, device=device)


def _next_dropout_seed(device):
    state = _DROPOUT_SEED.get(device)
    if state is None:
        set_dropout_seed(torch.initial_seed(), device)
        state = _DROPOUT_SEED[device]
    mine = state.clone()
    state.add_(0x9E3779B97F4A7C15 & 0x3fffffffffffffff)      # any odd stride: consecutive calls never share a Philox key
    return mine


_LONG3 = ctypes.c_long * 3
USE_FLASH = True      # False: batched GEMMs + separate softmax kernels with a materialised score matrix (cross-check path)


def _flash_lib():
    l = native.require()
    if not hasattr(l.dl4j_flash_attn_bwd, "_typed"):
        vp, i32, f32, lng = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_long
        lp = ctypes.POINTER(ctypes.c_long)
        l.dl4j_flash_attn_fwd.argtypes = [vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, lp, lp, lp, f32, i32, vp, lp, vp, f32, vp, vp]
        l.dl4j_flash_attn_fwd.restype = ctypes.c_int
        l.dl4j_flash_attn_bwd.argtypes = [vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, lp, lp, lp, lp, lng, lng, lng,
                                          lng, f32, i32, f32, vp, vp]
        l.dl4j_flash_attn_bwd.restype = ctypes.c_int
        l.dl4j_attn_dvec.argtypes = [vp, lp, vp, vp, i32, i32, i32, i32, vp]
        l.dl4j_attn_dvec.restype = ctypes.c_int
        l.dl4j_attn_dq_finish.argtypes = [vp, vp, lng, lng, i32, i32, i32, i32, i32, i32, vp]
        l.dl4j_attn_dq_finish.restype = ctypes.c_int
        l.dl4j_flash_attn_bwd._typed = True
    return l


def _flash_backward(q, k, v, dO, lse, dvec, mk, scale, flags, dropout_p, seed):
    l = _flash_lib()
    Bn, H, Tq, D = q.shape
    Tk = k.shape[2]
    if Tq == Tk:
        # one packed [B, T, 3, H, D] gradient buffer, so the gradient of the fused q/k/v projection is a plain view
        dqkv = q.new_empty((Bn, Tq, 3, H, D))
        dq_t, dk_t, dv_t = dqkv[:, :, 0], dqkv[:, :, 1], dqkv[:, :, 2]
    else:
        dq_t, dk_t, dv_t = q.new_empty((Bn, Tq, H, D)), q.new_empty((Bn, Tk, H, D)), q.new_empty((Bn, Tk, H, D))
    # more than one key block contributes to a query's gradient: an fp32 buffer, its own for every call (streams and threads may run the
    # same shape at the same time).  The lengths that the batched products and the operators served before repeat bit for bit: their key
    # blocks store slabs that are added in order.  The others always added in arrival order and keep the smaller buffer.
    blocks = (Tk + 127) // 128
    acc, slabs = None, 1
    if blocks > 1 and (Tk % 128 or flags & 1):
        slabs = blocks
        acc = q.new_empty((blocks, Bn, H, Tq, D), dtype=torch.float32)
        flags |= 4
    elif blocks > 1:
        acc = torch.zeros((Bn, H, Tq, D), dtype=torch.float32, device=q.device)
    stream = native._stream()
    rc = l.dl4j_flash_attn_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), dO.data_ptr(), lse.data_ptr(), dvec.data_ptr(),
                               native._ptr(mk), native._ptr(acc), dq_t.data_ptr(), dk_t.data_ptr(), dv_t.data_ptr(), Bn, H, Tq, Tk, D,
                               _LONG3(*q.stride()[:3]), _LONG3(*k.stride()[:3]), _LONG3(*v.stride()[:3]), _LONG3(*dO.stride()[:3]),
                               dq_t.stride(0), dq_t.stride(1), dk_t.stride(0), dk_t.stride(1), scale, flags, dropout_p, native._ptr(seed),
                               stream)
    native._check(rc, "dl4j_flash_attn_bwd")
    if acc is not None:
        rc = l.dl4j_attn_dq_finish(native._ptr(acc), native._ptr(dq_t), dq_t.stride(0), dq_t.stride(1), Bn, H, Tq, D, slabs,
                                   flags & 1, stream)
        native._check(rc, "dl4j_attn_dq_finish")
    return dq_t.permute(0, 2, 1, 3), dk_t.permute(0, 2, 1, 3), dv_t.permute(0, 2, 1, 3)


def flash_supported(q, k, v):
    if not native.available() or not q.is_cuda or not q.dtype == k.dtype == v.dtype == torch.bfloat16:
        return False
    qs, ks = q.shape, k.shape
    return (len(qs) == 4 and ks == v.shape and len(ks) == 4 and qs[3] <= 64 and qs[3] % 8 == 0 and qs[3] == ks[3] and qs[:2] == ks[:2]
            and min(qs) > 0 and min(ks) > 0)


def flash_forward(q, k, v, key_mask, scale, dropout_p=0.0, seed=None, flags=0):
    """Fused attention forward: returns (out [B, Tq, H, D] bf16, lse [B, H, Tq] fp32).  q, k, v: [B, H, T, D] views."""
    l = _flash_lib()
    q, k, v = _prep(q), _prep(k), _prep(v)
    Bn, H, Tq, D = q.shape
    out = q.new_empty((Bn, Tq, H, D))
    lse = q.new_empty((Bn, H, Tq), dtype=torch.float32)
    mk = key_mask.to(torch.float32).contiguous() if key_mask is not None else None
    rc = l.dl4j_flash_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), native._ptr(mk), Bn, H, Tq,
                               k.size(2), D, _LONG3(*q.stride()[:3]), _LONG3(*k.stride()[:3]), _LONG3(*v.stride()[:3]), float(scale), flags,
                               None, None, None, float(dropout_p), native._ptr(seed), native._stream())
    native._check(rc, "dl4j_flash_attn_fwd")
    return out, lse
