"""ctypes bindings to the in-tree sm_100a library (``csrc/libdl4j_b200.so``) and the autograd
functions that put its kernels on the training path.

The library exports a plain C ABI over raw device pointers + a CUDA stream, so loading it does
not depend on torch's C++ ABI and building it takes seconds.  On a machine with a GPU the
library is mandatory: ``require()`` raises if it cannot be loaded, so a silent torch fallback
cannot masquerade as the native path.
"""
from __future__ import annotations

import ctypes
import functools
import os
import struct
import threading

import numpy as np
import torch
from torch.autograd import forward_ad

_LIB = None
_LIB_ERR = None
_LOCK = threading.Lock()
# DL4J_DEBUG_BOUNDS=1 loads the build whose kernels check their element offsets (``csrc/build.py --debug-bounds``), DL4J_ASAN=1 the
# build whose host code runs under AddressSanitizer / UBSan (``--asan``; the process needs libasan preloaded).
_LIB_FLAVOUR = "dbg" if os.environ.get("DL4J_DEBUG_BOUNDS", "0") == "1" else "asan" if os.environ.get("DL4J_ASAN", "0") == "1" else ""
_LIB_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "csrc",
                         "libdl4j_b200" + ("_" + _LIB_FLAVOUR if _LIB_FLAVOUR else "") + ".so")

LAUNCHES = 0     # number of native kernel launches issued by this process (bench.py reports it)

_ACT_IDS = {"ActivationIdentity": 0, "ActivationReLU": 1, "ActivationGELU": 6, "ActivationSigmoid": 4, "ActivationTanH": 5}


def _load():
    global _LIB, _LIB_ERR
    with _LOCK:
        if _LIB is not None or _LIB_ERR is not None:
            return _LIB
        path = os.path.abspath(_LIB_PATH)
        if not os.path.exists(path):
            _LIB_ERR = f"{path} not built (run python -m deeplearning4j_b200.csrc.build)"
            return None
        try:
            lib = ctypes.CDLL(path)
        except OSError as e:
            _LIB_ERR = str(e)
            return None
        vp, i32, i64, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
        lng = ctypes.c_long
        sig = {
            "dl4j_gemm": [vp, vp, vp, vp, vp, vp, i32, i32, i32, lng, lng, lng, lng, lng, i32, i32, i32, i32, i32, i32,
                          i32, i32, f32, i32, i32, vp],
            "dl4j_fused_update": [vp, vp, vp, vp, vp, vp, i32, vp, vp, i32, f32, i32, vp],
            "dl4j_cast_f32_bf16": [vp, vp, i64, vp],
            "dl4j_threshold_encode_to": [vp, vp, i64, f32, vp, i32, vp],
            "dl4j_threshold_encode": [vp, i64, f32, vp, i32, vp],
            "dl4j_threshold_decode": [vp, i32, vp, i64, f32, i32, vp],
            "dl4j_bitmap_encode_to": [vp, vp, i64, f32, vp, vp],
            "dl4j_bitmap_decode_to": [vp, vp, vp, i64, f32, vp],
            "dl4j_layer_norm_fwd": [vp, vp, vp, vp, vp, vp, vp, vp, i32, i32, f32, i32, vp],
            "dl4j_layer_norm_grad": [vp, vp, vp, vp, vp, vp, vp, vp, vp, i64, i32, f32, i32, i32, i32, vp],
            "dl4j_softmax_xent": [vp, vp, vp, vp, vp, i32, i32, i64, i32, i32, vp],
            "dl4j_scatter_add_rows": [vp, vp, vp, i64, i32, i64, i64, i32, vp],
            "dl4j_softmax_xent_fwd": [vp, vp, vp, vp, vp, vp, i32, i32, i64, i32, i32, vp],
            "dl4j_softmax_xent_bwd": [vp, vp, vp, vp, vp, vp, vp, i32, i32, i64, i64, i32, i32, vp],
            "dl4j_lstm_cell_fwd": [vp, vp, vp, vp, vp, i32, i32, i32, vp],
            "dl4j_lstm_cell_bwd": [vp, vp, vp, vp, vp, vp, vp, i32, i32, i32, vp],
            "dl4j_lstm_seq_fwd": [vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, vp, vp],
            "dl4j_lstm_seq_bwd": [vp, vp, vp, vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, vp, vp],
            "dl4j_transpose16": [vp, vp, i32, i32, vp],
            "dl4j_bias_act_bwd": [vp, vp, vp, vp, i32, i32, i32, i32, vp],
            "dl4j_bn_fwd_train": [vp, vp, vp, vp, vp, vp, i32, f32, f32, i32, vp, vp, vp, vp, vp, i64, i32, vp],
            "dl4j_bn_apply": [vp, vp, vp, vp, i32, vp, i64, i32, vp],
            "dl4j_bn_bwd": [vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i64, i32, i32, vp],
            "dl4j_add_relu": [vp, vp, vp, i64, vp],
            "dl4j_maxpool_fwd": [vp, vp, vp, vp, vp],
            "dl4j_maxpool_bwd": [vp, vp, vp, vp, vp],
            "dl4j_subsample": [vp, vp, vp, i32, vp],
            "dl4j_conv_weight_to_cl": [vp, vp, i32, i32, i32, vp],
            "dl4j_conv_wgrad_from_cl": [vp, vp, i32, i32, i32, vp],
            "dl4j_read_status": [i32],
            "dl4j_num_sms": [],
            "dl4j_bind_device": [i32],
            "dl4j_abi_version": [],
        }
        for name, args in sig.items():
            fn = getattr(lib, name, None)
            if fn is not None:
                fn.argtypes = args
                fn.restype = ctypes.c_int
        for name in dir(lib):
            pass
        _LIB = lib
        return lib


def lib():
    return _load()


def available() -> bool:
    # asked before every launch: once torch has initialised CUDA there is a device, and is_available() (environment look-ups on
    # each call, 2 us) need not be asked again
    if _LIB is not None and torch.cuda.is_initialized():
        return True
    return torch.cuda.is_available() and _load() is not None


def require():
    """Fail loudly when a GPU is present but the native library is not."""
    if _LIB is None and torch.cuda.is_available() and _load() is None:
        raise RuntimeError(f"deeplearning4j_b200 native library unavailable on a GPU machine: {_LIB_ERR}")
    return _LIB


def load_error():
    _load()
    return _LIB_ERR


# without the "is CUDA initialised" question of torch.cuda.current_device: asked where there are CUDA tensors
_current_device = getattr(torch._C, "_cuda_getDevice", torch.cuda.current_device)


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _stream():
    """Current torch stream handle; also binds the current device's context to this thread for the
    library's own CUDA runtime instance (autograd worker threads may not have one bound yet)."""
    dev = _current_device()
    rc = _LIB.dl4j_bind_device(dev)
    if rc != 0:
        raise RuntimeError(f"dl4j_bind_device failed with CUDA error {rc}")
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(dev))       # the raw handle: a Stream object costs 10 us a launch


def on_current_device(*ts):
    """Whether every given tensor (or None) lives on the current device, where ``_stream`` launches."""
    dev = _current_device()
    for t in ts:
        if t is not None and t.get_device() != dev:          # -1: host memory
            return False
    return True


def _check(rc, what):
    global LAUNCHES
    LAUNCHES += 1
    if rc != 0:
        raise RuntimeError(f"{what} failed with code {rc}")


def check_status(reset=True):
    """Raise if any bounded device-side wait expired since the last check (synchronises)."""
    l = require()
    if l is None:
        return 0
    v = l.dl4j_read_status(1 if reset else 0)
    if _LIB_FLAVOUR == "dbg":
        rec = debug_bounds(reset)
        if rec["failures"]:
            raise RuntimeError(f"debug bounds check failed {rec['failures']} time(s); first: source line {rec['line']}, "
                               f"offset {rec['offset']}, extent {rec['extent']}")
    if v != 0:
        names = {1: "TMA producer wait", 2: "MMA wait", 3: "epilogue wait", 4: "peer wait", 5: "index out of bounds"}
        raise RuntimeError(f"device-side bounded wait/ check failed: {names.get(v, v)}")
    return v


def debug_bounds(reset=True):
    """The debug-bounds build's record: number of out-of-range offsets the kernels skipped since the last reset, and the source
    line, offset and extent of the first (synchronises).  ``None`` in the normal build."""
    l = require()
    if l is None:
        return None
    out = (ctypes.c_ulonglong * 4)()
    l.dl4j_debug_bounds.argtypes = [ctypes.c_void_p, ctypes.c_int]
    l.dl4j_debug_bounds.restype = ctypes.c_int
    if l.dl4j_debug_bounds(out, 1 if reset else 0) != 0:
        return None
    off = out[2] - (1 << 64) if out[2] >= (1 << 63) else out[2]
    return {"failures": int(out[0]), "line": int(out[1]), "offset": int(off), "extent": int(out[3])}


_DT = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}
_NUM_SMS = None


def num_sms():
    global _NUM_SMS
    if _NUM_SMS is None:
        _NUM_SMS = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    return _NUM_SMS


# =========================================================================== GEMM
def _operand_a(a):
    """logical [M, K] -> (tensor, mn_major flag, leading dim) or None."""
    if a.stride(1) == 1 and a.stride(0) % 8 == 0 and a.stride(0) >= a.shape[1] and a.data_ptr() % 16 == 0:
        return a, 0, a.stride(0)
    if a.stride(0) == 1 and a.stride(1) % 8 == 0 and a.stride(1) >= a.shape[0] and a.data_ptr() % 16 == 0:
        return a, 1, a.stride(1)
    return None


def _operand_b(b):
    """logical [K, N] -> (tensor, mn_major flag, leading dim) or None."""
    if b.stride(0) == 1 and b.stride(1) % 8 == 0 and b.stride(1) >= b.shape[0] and b.data_ptr() % 16 == 0:
        return b, 0, b.stride(1)       # stored [N, K]
    if b.stride(1) == 1 and b.stride(0) % 8 == 0 and b.stride(0) >= b.shape[1] and b.data_ptr() % 16 == 0:
        return b, 1, b.stride(0)       # stored [K, N]
    return None


def gemm_supported(a, b) -> bool:
    if not available() or a.dim() != 2 or b.dim() != 2 or a.dtype != b.dtype or a.dtype not in (torch.bfloat16, torch.float16):
        return False
    if a.shape[1] != b.shape[0] or min(a.shape[0], a.shape[1], b.shape[1]) == 0:
        return False
    return _operand_a(a) is not None and _operand_b(b) is not None


_PAIR_TILE = 512          # `block_n` code of the 256 x 256 tiles on pairs of CTAs


def _pair_rows(M):
    """Whether 256-row tiles cover M rows with at most a quarter more padding than 128-row tiles."""
    return (M + 255) // 256 * 8 <= (M + 127) // 128 * 5


@functools.lru_cache(maxsize=4096)      # of sizes alone; small networks ask for it as often as they launch
def _pick_block_n(M, N, splits=1, K=0):
    """Tile of a GEMM by waves x columns: 128 x 256, 128 x 128 (pays 4 - 14 % more per column: 16384 rows, N and K 768 - 3072) or, with K
    given, 256 x 256 on a pair of CTAs.  A pair needs a third fewer bytes from L2 per step of K and about 1 us more to start and end, so it
    takes problems with at least 36 steps of 64 per CTA.  256 wide / pair, us: 16384 x 3072 x 768 67 / 58, 16384 x 768 x 3072 62 / 57,
    16384 x 768 x 768 (36 steps) 21.3 / 19.8, 3200 x 4096 x 1024 (48) 24.6 / 22.9, 2456 x 30520 x 768 150 / 122; with fewer steps 32768 x 512 x
    512 (32) 20.2 / 19.1, but its GELU form 30.9 / 31.3, 4096 x 1024 x 1024 (16) 11.6 / 12.4, 25088 x 512 x 128 (6) 11.6 / 12.6."""
    sms = num_sms()
    best, best_cost = 256, None
    for bn, rows, units, f in ((256, 128, sms, 1.0), (128, 128, sms, 1.08), (_PAIR_TILE, 256, sms // 2, 0.9)):
        cols = min(bn, 256)
        tiles = ((M + rows - 1) // rows) * ((N + cols - 1) // cols) * splits
        waves = (tiles + units - 1) // units
        if bn == _PAIR_TILE and (waves * (((K + 63) // 64 + splits - 1) // splits) < 36 or not _pair_rows(M)):
            continue
        cost = waves * cols * f
        if best_cost is None or cost < best_cost:
            best, best_cost = bn, cost
    return best


def gemm_raw(a, b, out=None, bias=None, act=0, aux=None, residual=None, out_dtype=None, atomic=False, splits=1,
             alpha=1.0, block_n=None, pair=None, res_act=0):
    """out[M,N] = act(alpha * a @ b + bias) + residual with a logical [M,K], b logical [K,N].  With ``res_act`` (an activation id)
    ``residual`` holds pre-activations z and the result is multiplied by act'(z) instead: a data-gradient GEMM that writes dz."""
    l = require()
    if res_act:
        if residual is None or act:
            raise ValueError("res_act needs the pre-activations as `residual` and no forward activation")
        act = int(res_act) << 8
    oa, ob = _operand_a(a), _operand_b(b)
    if oa is None or ob is None:
        raise ValueError("operand layout not addressable by TMA (need unit stride in one dim, 16-byte alignment)")
    M, K = a.shape
    N = b.shape[1]
    if out is None:
        out_dtype = out_dtype or a.dtype
        out = (torch.zeros if atomic else torch.empty)((M, N), dtype=out_dtype, device=a.device)
    if out.stride(1) != 1:
        raise ValueError("output must be row-major")
    out_fp32 = 1 if out.dtype == torch.float32 else 0
    if not out_fp32 and out.dtype != a.dtype:
        raise ValueError("output dtype must be the input dtype or float32")
    kb = (K + 63) // 64
    splits = max(1, min(int(splits), kb))
    if splits > 1 and not (atomic and out_fp32):
        splits = 1
    bn = block_n or (_PAIR_TILE if pair else _pick_block_n(M, N, splits, K if pair is None else 0))
    bias_fp32 = 1 if (bias is not None and bias.dtype == torch.float32) else 0
    if bias is not None and not bias_fp32 and bias.dtype != a.dtype:
        bias = bias.to(a.dtype)
    if bias is not None and not bias.is_contiguous():
        bias = bias.contiguous()
    rc = l.dl4j_gemm(_ptr(oa[0]), _ptr(ob[0]), _ptr(out), _ptr(aux), _ptr(bias), _ptr(residual), M, N, K, oa[2], ob[2],
                     out.stride(0), 0 if aux is None else aux.stride(0), 0 if residual is None else residual.stride(0),
                     oa[1], ob[1], _DT[a.dtype], bias_fp32, out_fp32, int(act), 1 if atomic else 0, splits, float(alpha),
                     bn, num_sms(), _stream())
    _check(rc, "dl4j_gemm")
    return out


@functools.lru_cache(maxsize=4096)
def _long_k_splits(M, N, K):
    """Split-K factor for a 16-bit-output GEMM with few output tiles and a long reduction (the data gradient of a wide output layer).
    The estimate, fitted to the measurements below (us): a k-block of 64 takes 0.36 in a tile of 128 x 256, 0.24 in one of 128 x 128 and 0.30
    in one of 256 x 256 on a pair of CTAs, a product 11, 7 and 12 besides; the partial results of a split cost 6 for a second launch and 2
    per million of their elements.  Measured unsplit / best split (factor): 128 x 768 x 30522 73 / 23 (16), 1000 x 768 x 30522 95 / 44 (6),
    256 x 512 x 10001 63 / 19 (16), 1500 x 768 x 20000 75 / 43 (4), 2456 x 512 x 8192 28 / 29 (3), 2456 x 768 x 30522 106 / 97 (2),
    3000 x 512 x 30000 131 / 76 (3), 4000 x 768 x 16000 87 / 83 (3), 1024 x 1024 x 4096 15 / 19 (4), 300 x 768 x 2048 9 / 15.  A gain of
    less than a tenth by the estimate is not worth the partial results."""
    sms, kb = num_sms(), (K + 63) // 64
    rows, cols = (M + 127) // 128, (N + 255) // 256
    tiles, pair_tiles = rows * cols, ((M + 255) // 256) * cols
    if tiles >= sms or kb < 32:
        return 1

    def wide(s):                # k-block time of the 256-wide tiles that `s` parts run on
        steps, pair_waves = (kb + s - 1) // s, -(-pair_tiles * s // (sms // 2))
        if pair_waves * steps >= 36 and _pair_rows(M):
            return pair_waves * steps * 0.30
        return -(-tiles * s // sms) * steps * 0.36
    best, best_cost = 1, 0.9 * min(7 + -(-rows * ((N + 127) // 128) // sms) * kb * 0.24, 12 + wide(1))
    for s in range(2, 17):
        if kb // s < 8:
            break
        c = 17 + wide(s) + s * M * N * 2e-6
        if c < best_cost:
            best, best_cost = s, c
    return best


def _dgrad_gemm(a, b, out=None):
    """``a @ b`` in a's type; a long reduction over few output tiles is split and summed in fp32, in order, before the one rounding."""
    M, N = a.shape[0], b.shape[1]
    s = _long_k_splits(M, N, a.shape[1])
    if s == 1 or N % 4:
        return gemm_raw(a, b, out=out)
    return _split_gemm(a, b, s, out)


def _split_gemm(a, b, s, out=None):
    """``a @ b`` with the reduction in ``s`` parts, added in order: repeats bit for bit."""
    l = require()
    M, N = a.shape[0], b.shape[1]
    if out is None:
        out = torch.empty((M, N), dtype=a.dtype, device=a.device)
    if not hasattr(l.dl4j_gemm_split, "_typed"):
        vp, i32, lng = ctypes.c_void_p, ctypes.c_int, ctypes.c_long
        l.dl4j_gemm_split.argtypes = [vp, vp, vp, vp, i32, i32, i32, lng, lng, lng, i32, i32, i32, i32, i32, vp]
        l.dl4j_gemm_split.restype = i32
        l.dl4j_gemm_split._typed = True
    oa, ob = _operand_a(a), _operand_b(b)
    if oa is None or ob is None:
        raise ValueError("operand layout not addressable by TMA (need unit stride in one dim, 16-byte alignment)")
    part = torch.empty((s, M, N), dtype=torch.float32, device=a.device)
    rc = l.dl4j_gemm_split(_ptr(oa[0]), _ptr(ob[0]), _ptr(part), _ptr(out), M, N, a.shape[1], oa[2], ob[2], out.stride(0), oa[1], ob[1],
                           _DT[a.dtype], s, num_sms(), _stream())
    global LAUNCHES
    LAUNCHES += 1
    _check(rc, "dl4j_gemm_split")
    return out


class _MatmulFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, a, b):
        ctx.save_for_backward(a, b)
        return gemm_raw(a, b)

    @staticmethod
    def backward(ctx, dy):
        a, b = ctx.saved_tensors
        dy = dy if dy.stride(1) == 1 or dy.stride(0) == 1 else dy.contiguous()
        da = db = None
        if ctx.needs_input_grad[0]:
            da = gemm(dy, b.t())
        if ctx.needs_input_grad[1]:
            db = gemm(a.t(), dy)
        return da, db


def gemm(a, b):
    """Differentiable 2-D matmul on the tcgen05 kernel (falls back to torch for odd layouts)."""
    if not gemm_supported(a, b):
        return torch.matmul(a, b)
    if torch.is_grad_enabled() and (a.requires_grad or b.requires_grad):
        return _MatmulFn.apply(a, b)
    return gemm_raw(a, b)


# =========================================================================== Linear (+bias +activation)
def _act_id(activation):
    if activation is None:
        return 0
    name = type(activation).__name__
    if name == "ActivationGELU":
        return 3 if getattr(activation, "precise", False) else 6      # tanh form / x * sigmoid(1.702 x)
    if name == "ActivationReLU":
        if getattr(activation, "max", None) is not None or getattr(activation, "threshold", None) or getattr(activation, "negativeSlope", None):
            return None
        return 1
    return _ACT_IDS.get(name)


def _wgrad_splits(n_out_tiles, K):
    """Split-K factor of a weight gradient (``n_out_tiles`` tiles of 128 x 256, reduction over ``K`` rows): two waves of tiles, at most 32 parts
    or, over up to four tiles, one wave of at most 64.  256 x 64 over 200704 rows with 32 / 64 parts 27.4 / 23.6 us, over 100352 12.6 / 10.4;
    512 x 128 over 25088 (four tiles) 9.0 / 10.4.  A part's accumulator is truncated once per 16 rows: longer parts would be less exact."""
    sms = num_sms()
    if n_out_tiles >= sms:
        return 1
    t = max(n_out_tiles, 1)
    return max(1, min((K + 63) // 64, 2 * sms // t, max(32, min(sms // t, 64))))


def _bias_grad_buffer(b, needed, N, device):
    """(accumulator, returned gradient): the bias' own fp32 ``.grad`` when the kernels may add into it, else a fresh buffer."""
    if b is None or not needed:
        return None, None
    if b.is_leaf and b.grad is not None and b.grad.dtype == torch.float32 and b.grad.is_contiguous():
        return b.grad, None
    acc = torch.zeros(N, dtype=torch.float32, device=device)
    return acc, acc


def _weight_grad(W, x, dz):
    """dW of ``y = x @ W`` accumulated into ``W.grad`` when its layout allows (returns None), else returned in W's layout."""
    M, N = dz.shape
    nIn = x.shape[1]
    tiles = ((N + 127) // 128) * ((nIn + 255) // 256)
    splits = _wgrad_splits(tiles, M)
    g = W.grad if (W.is_leaf and W.grad is not None) else None
    if g is not None and g.dim() == 4 and g.shape[2] == 1 and g.shape[3] == 1 and g.is_contiguous():
        g = g.view(g.shape[0], g.shape[1]).t()      # 1x1 convolution kernel [nOut, nIn, 1, 1]: same memory as an 'f' dense weight
    if g is not None and g.dtype == torch.float32 and g.dim() == 2 and g.stride(0) == 1 and g.stride(1) == nIn \
            and g.data_ptr() % 16 == 0 and nIn % 4 == 0:
        gemm_raw(dz.t(), x, out=g.t(), atomic=True, splits=splits)
        return None
    if g is not None and g.dtype == torch.float32 and g.dim() == 2 and g.is_contiguous() and g.data_ptr() % 16 == 0 and N % 4 == 0:
        # row-major [nIn, nOut] master (SameDiff variables): dW = x^T dz accumulated in place
        tiles2 = ((nIn + 127) // 128) * ((N + 255) // 256)
        gemm_raw(x.t(), dz, out=g, atomic=True, splits=_wgrad_splits(tiles2, M))
        return None
    dWt = gemm_raw(dz.t(), x, out_dtype=torch.float32, atomic=True, splits=splits)
    return dWt.reshape(W.shape).to(W.dtype) if W.dim() == 4 else dWt.t().to(W.dtype)


def _fwd_bias(b, dtype):
    """(bias operand for the forward GEMM, master the gradient goes to)."""
    if b is None:
        return None, None
    b_fwd = b if b.dtype == dtype else getattr(b, "_lp", None)
    if b_fwd is not None:
        b_fwd = b_fwd.detach()
    master = getattr(b, "_master", b)
    if b_fwd is None:
        b_fwd = master
    return b_fwd.reshape(-1), master


class _MlpFn(torch.autograd.Function):
    """y = act(x @ W1 + b1) @ W2 + b2 as one autograd node.  Forward: two GEMMs (the first saves its pre-activation z1 from the
    epilogue).  Backward: the data-gradient GEMM of the second layer multiplies by act'(z1) in its epilogue and writes dz1
    directly, so the separate pass that read dy1 and z1 and wrote dz1 disappears; the bias gradient of the first layer is a
    column sum over dz1 alone."""

    @staticmethod
    def forward(ctx, x, W1, b1, W2, b2, act, W1_lp, W2_lp):
        z1 = torch.empty((x.shape[0], W1_lp.shape[1]), dtype=x.dtype, device=x.device)
        b1_fwd, b1_m = _fwd_bias(b1, x.dtype)
        b2_fwd, b2_m = _fwd_bias(b2, x.dtype)
        y1 = gemm_raw(x, W1_lp, bias=b1_fwd, act=act, aux=z1)
        y2 = gemm_raw(y1, W2_lp, bias=b2_fwd)
        ctx.act = act
        ctx.refs = (getattr(W1, "_master", W1), b1_m, getattr(W2, "_master", W2), b2_m)
        ctx.save_for_backward(x, W1_lp, W2_lp, z1, y1)
        return y2

    @staticmethod
    def backward(ctx, dy2):
        x, W1_lp, W2_lp, z1, y1 = ctx.saved_tensors
        W1, b1, W2, b2 = ctx.refs
        l = require()
        dy2 = _dense16(dy2)
        M, N2 = dy2.shape
        N1 = z1.shape[1]
        need = ctx.needs_input_grad
        acc2, db2 = _bias_grad_buffer(b2, need[4], N2, dy2.device)
        if acc2 is not None:
            _check(l.dl4j_bias_act_bwd(_ptr(dy2), None, None, _ptr(acc2), M, N2, 0, _DT[dy2.dtype], _stream()), "dl4j_bias_act_bwd")
        dW2 = _weight_grad(W2, y1, dy2) if need[3] else None
        # dz1 = (dy2 @ W2^T) * act'(z1): one GEMM
        dz1 = gemm_raw(dy2, W2_lp.t(), residual=z1, res_act=ctx.act)
        acc1, db1 = _bias_grad_buffer(b1, need[2], N1, dy2.device)
        if acc1 is not None:
            _check(l.dl4j_bias_act_bwd(_ptr(dz1), None, None, _ptr(acc1), M, N1, 0, _DT[dz1.dtype], _stream()), "dl4j_bias_act_bwd")
        dW1 = _weight_grad(W1, x, dz1) if need[1] else None
        dx = gemm_raw(dz1, W1_lp.t()) if need[0] else None
        if db1 is not None:
            db1 = db1.reshape(b1.shape).to(b1.dtype)
        if db2 is not None:
            db2 = db2.reshape(b2.shape).to(b2.dtype)
        return dx, dW1, db1, dW2, db2, None, None, None


def _lp_weight(W, dtype):
    W_lp = getattr(W, "_lp", None)
    if W_lp is None:
        if W.stride(0) != 1 and W.stride(1) != 1:
            return None
        W_lp = W.detach() if W.dtype == dtype else W.detach().to(dtype)
    return W_lp if W_lp.dtype == dtype else None


def mlp(x, W1, b1, W2, b2, activation):
    """``act(x @ W1 + b1) @ W2 + b2`` with the activation gradient folded into the second layer's data-gradient GEMM; returns None
    when the case is not covered (then the two layers run separately)."""
    if not available() or x.dim() != 2 or x.dtype not in (torch.bfloat16, torch.float16):
        return None
    act = _act_id(activation)
    if act not in (1, 2, 3, 4, 5, 6):
        return None
    W1_lp, W2_lp = _lp_weight(W1, x.dtype), _lp_weight(W2, x.dtype)
    if W1_lp is None or W2_lp is None or W1_lp.shape[1] != W2_lp.shape[0]:
        return None
    if not x.is_contiguous():
        x = x.contiguous()
    for w in (W1_lp, W2_lp):
        if _operand_b(w) is None or _operand_b(w.t()) is None or w.shape[0] % 8 or w.shape[1] % 8:
            return None
    if _operand_a(x) is None:
        return None
    return _MlpFn.apply(x, W1, b1, W2, b2, act, W1_lp, W2_lp)


class _LinearFn(torch.autograd.Function):
    """y = act(x @ W + b).  ``W`` is the fp32 (or bf16) leaf, ``W_lp`` its low-precision shadow used
    by the GEMMs.  When ``W`` is a leaf with a preallocated row-major-transposed ``.grad`` view (the
    DL4J 'f' layout inside the flat gradient buffer), the weight gradient is accumulated straight
    into it by the GEMM epilogue (split-K vector reductions) and ``None`` is returned for it."""

    @staticmethod
    def forward(ctx, x, W, b, act, W_lp):
        need_z = act in (2, 3, 4, 5, 6)
        z = torch.empty((x.shape[0], W_lp.shape[1]), dtype=x.dtype, device=x.device) if need_z and any(ctx.needs_input_grad) else None
        W = getattr(W, "_master", W)          # accumulate weight/bias gradients straight into the fp32 masters
        # the forward GEMM takes the bias in the operand format when there is one (shadow of the master): it is then added
        # by one extra tensor-core step instead of a per-element broadcast in the epilogue
        b_fwd = None
        if b is not None:
            b_fwd = b if b.dtype == x.dtype else getattr(b, "_lp", None)
            if b_fwd is not None:
                b_fwd = b_fwd.detach()
        b = getattr(b, "_master", b) if b is not None else None
        if b_fwd is None:
            b_fwd = b
        y = gemm_raw(x, W_lp, bias=None if b_fwd is None else b_fwd.reshape(-1), act=act, aux=z)
        ctx.act = act
        ctx.has_bias = b is not None
        ctx.W_ref = W
        ctx.b_ref = b
        ctx.save_for_backward(x, W_lp, z if z is not None else (y if act == 1 else None))
        return y

    @staticmethod
    def backward(ctx, dy):
        x, W_lp, saved = ctx.saved_tensors
        act = ctx.act
        l = require()
        dy = _dense16(dy)
        M, N = dy.shape
        W, b = ctx.W_ref, ctx.b_ref
        # ---- dz and bias gradient
        db = None
        b_acc = None
        if ctx.has_bias and ctx.needs_input_grad[2]:
            if b.is_leaf and b.grad is not None and b.grad.dtype == torch.float32 and b.grad.is_contiguous():
                b_acc = b.grad
            else:
                b_acc = torch.zeros(N, dtype=torch.float32, device=dy.device)
                db = b_acc
        if act != 0:
            dz = torch.empty_like(dy)
            zz = saved
            if zz is None:
                raise RuntimeError("linear backward: activation input was not saved")
            rc = l.dl4j_bias_act_bwd(_ptr(dy), _ptr(zz), _ptr(dz), _ptr(b_acc), M, N, 1 if act == 1 else act, _DT[dy.dtype], _stream())
            _check(rc, "dl4j_bias_act_bwd")
        else:
            dz = dy
            if b_acc is not None:
                rc = l.dl4j_bias_act_bwd(_ptr(dy), None, None, _ptr(b_acc), M, N, 0, _DT[dy.dtype], _stream())
                _check(rc, "dl4j_bias_act_bwd")
        if db is not None:
            db = db.reshape(b.shape).to(b.dtype)
        # ---- data gradient: dx = dz @ W^T
        dx = None
        if ctx.needs_input_grad[0]:
            dx = _dgrad_gemm(dz, W_lp.t())
        # ---- weight gradient: dW^T [nOut, nIn] = dz^T @ x
        dW = None
        if ctx.needs_input_grad[1]:
            nIn = x.shape[1]
            tiles = ((N + 127) // 128) * ((nIn + 255) // 256)
            splits = _wgrad_splits(tiles, M)
            g = W.grad if (W.is_leaf and W.grad is not None) else None
            if g is not None and g.dim() == 4 and g.shape[2] == 1 and g.shape[3] == 1 and g.is_contiguous():
                g = g.view(g.shape[0], g.shape[1]).t()      # 1x1 convolution kernel [nOut, nIn, 1, 1]: same memory as an 'f' dense weight
            if g is not None and g.dtype == torch.float32 and g.dim() == 2 and g.stride(0) == 1 and g.stride(1) == nIn \
                    and g.data_ptr() % 16 == 0 and nIn % 4 == 0:
                gemm_raw(dz.t(), x, out=g.t(), atomic=True, splits=splits)
            elif g is not None and g.dtype == torch.float32 and g.dim() == 2 and g.is_contiguous() and g.data_ptr() % 16 == 0 \
                    and N % 4 == 0:
                # row-major [nIn, nOut] master (SameDiff variables): dW = x^T dz accumulated in place
                tiles2 = ((nIn + 127) // 128) * ((N + 255) // 256)
                gemm_raw(x.t(), dz, out=g, atomic=True, splits=_wgrad_splits(tiles2, M))
            else:
                dWt = gemm_raw(dz.t(), x, out_dtype=torch.float32, atomic=True, splits=splits)
                dW = dWt.reshape(W.shape).to(W.dtype) if W.dim() == 4 else dWt.t().to(W.dtype)
        return dx, dW, db, None, None


def linear(x, W, b, activation):
    """Fused linear on the tcgen05 GEMM; returns None when the case is not covered."""
    if not available() or x.dim() != 2:
        return None
    act = _act_id(activation)
    if act is None:
        return None
    W_lp = getattr(W, "_lp", None)
    if W_lp is None:
        W_lp = W.detach() if W.dtype == x.dtype else W.detach().to(x.dtype)
        if W.stride(0) != 1 and W.stride(1) != 1:
            return None
    if W_lp.dtype != x.dtype:
        return None
    if not x.is_contiguous():
        x = x.contiguous()
    # fewer rows stay with the library: forward + backward of 128 x 512 x 10001 takes 60 us of device time here against 107 there, but
    # its two autograd products cost the caller 118 us where this function costs 296
    if ((W.shape[1] % 8) or (x.shape[1] % 8)) and _PAD_ODD_WIDTHS and x.shape[0] >= 256:
        return _linear_padded(x, W, b, act)
    if _operand_a(x) is None or _operand_b(W_lp) is None or _operand_b(W_lp.t()) is None:
        return None
    # wgrad needs x as an MN-major operand: row stride multiple of 8 elements, and dz^T likewise
    if (W_lp.shape[1] % 8) or (x.shape[1] % 8):
        return None
    return _LinearFn.apply(x, W, b, act, W_lp)


def pitch_copy(src, dst):
    """dst <- src (2-D, unit column stride, any row pitch; fp32 -> 16-bit converts)."""
    l = require()
    if not hasattr(l.dl4j_pitch_copy, "_typed"):
        vp, i32, lng = ctypes.c_void_p, ctypes.c_int, ctypes.c_long
        l.dl4j_pitch_copy.argtypes = [vp, i32, vp, i32, lng, i32, lng, lng, vp]
        l.dl4j_pitch_copy.restype = i32
        l.dl4j_pitch_copy._typed = True
    rc = l.dl4j_pitch_copy(_ptr(src), _DT[src.dtype], _ptr(dst), _DT[dst.dtype], src.shape[0], src.shape[1], src.stride(0), dst.stride(0), _stream())
    _check(rc, "dl4j_pitch_copy")
    return dst


def _pitched(rows, cols, dtype, device):
    """Uninitialised [rows, cols] matrix whose rows start on 16-byte boundaries (and whose padding belongs to its storage)."""
    return torch.empty((rows, (cols + 7) // 8 * 8), dtype=dtype, device=device)[:, :cols]


def _on_pitch(t, dtype):
    """``t`` in ``dtype`` with unit column stride and rows on 16-byte boundaries, padding included in the storage; copied if need be."""
    P = (t.shape[1] + 7) // 8 * 8
    if t.dtype == dtype and t.stride(1) == 1 and t.stride(0) == P and t.data_ptr() % 16 == 0 \
            and (t.storage_offset() + t.shape[0] * P) * t.element_size() <= t.untyped_storage().nbytes():
        return t
    if t.stride(1) != 1 or (t.dtype != dtype and t.dtype != torch.float32):
        t = t.to(dtype).contiguous()
    return pitch_copy(t, _pitched(t.shape[0], t.shape[1], dtype, t.device))


class _OddLinearFn(torch.autograd.Function):
    """``act(x @ W + b)`` for layer widths off the 8-element grid (a 77-symbol alphabet, a 30522-word vocabulary, ten classes).  TMA asks
    for 16-byte row pitches, not for widths: the weights are copied once to such a pitch, results and their gradients live on it as
    strided views, and the tiles' edges are clipped by the tensor maps."""

    @staticmethod
    def forward(ctx, x, W, b, act):
        dt = x.dtype
        M, K = x.shape
        N = W.shape[1]
        xp = _on_pitch(x.detach(), dt)
        Wd = W.detach()
        rows = Wd.stride(1) == 1 or Wd.stride(0) != 1          # row-major [K, N]; else 'f' order, stored as [N, K]
        Wp = _on_pitch(Wd, dt) if rows else _on_pitch(Wd.t(), dt).t()
        y = _pitched(M, N, dt, x.device)
        z = _pitched(M, N, dt, x.device) if act in (2, 3, 4, 5, 6) and any(ctx.needs_input_grad) else None
        # the parameter itself, like the weights: in its own precision and as it is now (its 16-bit shadow is neither)
        b_fwd = None if b is None else _dense16(b.detach().reshape(-1))
        gemm_raw(xp, Wp, out=y, bias=b_fwd, act=act, aux=z)
        ctx.act, ctx.rows, ctx.w_dtype, ctx.b_like = act, rows, W.dtype, None if b is None else (b.shape, b.dtype)
        ctx.save_for_backward(xp, Wp, z if z is not None else (y if act == 1 else None))
        return y

    @staticmethod
    def backward(ctx, dy):
        l = require()
        xp, Wp, saved = ctx.saved_tensors
        M, K = xp.shape
        N = Wp.shape[1]
        dt = xp.dtype
        dz = _on_pitch(dy, dt)
        P = dz.stride(0)
        acc = torch.zeros(P, dtype=torch.float32, device=dy.device) if ctx.b_like is not None and ctx.needs_input_grad[2] else None
        if ctx.act:
            out = _pitched(M, N, dt, dy.device)
            rc = l.dl4j_bias_act_bwd(_ptr(dz), _ptr(saved), _ptr(out), _ptr(acc), M, P, ctx.act, _DT[dt], _stream())
            _check(rc, "dl4j_bias_act_bwd")
            dz = out
        elif acc is not None:
            _check(l.dl4j_bias_act_bwd(_ptr(dz), None, None, _ptr(acc), M, P, 0, _DT[dt], _stream()), "dl4j_bias_act_bwd")
        db = None if acc is None else acc[:N].reshape(ctx.b_like[0]).to(ctx.b_like[1])
        dx = None
        if ctx.needs_input_grad[0]:
            dx = _dgrad_gemm(dz, Wp.t(), out=None if K % 8 == 0 else _pitched(M, K, dt, dy.device))
        dW = None
        if ctx.needs_input_grad[1]:
            a, c = (xp.t(), dz) if ctx.rows else (dz.t(), xp)
            R, C = a.shape[0], c.shape[1]
            splits = _wgrad_splits(((R + 127) // 128) * ((C + 255) // 256), M)
            wide = ctx.w_dtype == torch.float32 or splits > 1       # partial sums and fp32 gradients stay in fp32
            buf = torch.zeros((R, (C + 7) // 8 * 8), dtype=torch.float32, device=dy.device)[:, :C] if wide else _pitched(R, C, dt, dy.device)
            gemm_raw(a, c, out=buf, atomic=wide, splits=splits)
            if not buf.is_contiguous() or buf.dtype != ctx.w_dtype:
                same = ctx.w_dtype in (buf.dtype, torch.float16, torch.bfloat16) and (buf.dtype == torch.float32 or buf.dtype == ctx.w_dtype)
                buf = pitch_copy(buf, torch.empty((R, C), dtype=ctx.w_dtype, device=dy.device)) if same else buf.to(ctx.w_dtype).contiguous()
            dW = buf if ctx.rows else buf.t()
        return dx, dW, db, None


def _linear_padded(x, W, b, act):
    """Layer widths that are not multiples of 8, see ``_OddLinearFn``; None when the case is not covered."""
    if W.dim() != 2 or min(x.shape[0], W.shape[0], W.shape[1]) == 0 or W.dtype not in (x.dtype, torch.float32) or not on_current_device(x, W, b) \
            or (b is not None and b.numel() != W.shape[1]):
        return None
    return _OddLinearFn.apply(x, W, b, act)


_PAD_ODD_WIDTHS = os.environ.get("DL4J_PAD_ODD_WIDTHS", "1") != "0"


# =========================================================================== small fp32 layers
def _sgemm(a, b, out, bias=None, act=0):
    """out [M, N] (unit column stride) = act(a @ b + bias) in fp32, for operands with a unit stride in one dimension."""
    l = require()
    if not hasattr(l.dl4j_sgemm_small, "_typed"):
        vp, i32, lng = ctypes.c_void_p, ctypes.c_int, ctypes.c_long
        l.dl4j_sgemm_small.argtypes = [vp, lng, i32, vp, lng, i32, vp, vp, lng, i32, i32, i32, i32, i32, vp]
        l.dl4j_sgemm_small.restype = i32
        l.dl4j_sgemm_small._typed = True
    a_kc, b_kc = a.stride(1) == 1, b.stride(0) == 1
    rc = l.dl4j_sgemm_small(_ptr(a), a.stride(0) if a_kc else a.stride(1), int(a_kc), _ptr(b), b.stride(1) if b_kc else b.stride(0), int(b_kc),
                            _ptr(bias), _ptr(out), out.stride(0), a.shape[0], b.shape[1], a.shape[1], act, num_sms(), _stream())
    _check(rc, "dl4j_sgemm_small")
    return out


def _unit(t):
    return t.dim() == 2 and 1 in t.stride()


def _sgemm_wins(M, N, K, relu, grad):
    """Whether an fp32 layer (M rows, N units, a sum of K terms) leaves a library kernel short of tiles.  A tile of
    64 x 64 has at most eight CTAs, so the time grows with K.  us of device time, here / library product [+ ReLU launch]:
        M, N          K = 256    1024      2048      4096      8192      25088
        64, 64        13 / 22    16 / 28   25 / 30   39 / 42   72 / 61   199 / 104
        128, 512      12 / 22    19 / 38   29 / 41   49 / 56   90 / 88   254 / 150
        512, 512      14 / 22    31 / 40   51 / 65   90 / 114  169 / 149 496 / 332
        64, 4096      15 / 22    33 / 42   55 / 67   100 / 118 188 / 148 548 / 331
        16, 512       12 / 22    16 / 17   25 / 23   41 / 30   72 / 34   203 / 75
        32, 4096      15 / 22    33 / 40   55 / 47   98 / 74   186 / 111 543 / 319
        1, 4096       14 / 13    31 / 17   53 / 22
    Below 16 rows the library has matrix-vector kernels: 12 / 11 at K = 128, 12 / 13 at 256, 14 / 13 - 21 / 13 at 512.  Without a ReLU launch
    to save: 128 x 512 x 10 6 / 9, 16 rows 12 / 8 at K = 128, 12 / 10 at 256, 12 / 12 at 512.
    With a gradient to come the layer's backward saves what its product loses: replayed steps of 784-512-512-10 took 76 us here and 94 with
    library products at 8 rows, 68 and 72 at one."""
    if ((M + 63) // 64) * ((N + 63) // 64) > 64:
        return False
    if not grad and (M < 16 and not (relu and K <= 256) or not relu and K < 256):
        return False
    return K <= (4096 if M >= 64 else 1024)


def _sgemm_wins_dgrad(M, N, nIn):
    """The same for the bare data gradient dz [M, N] @ W^T, up to 16 tiles; its sum has N terms.  here / library:
        M, nIn        N = 256    512       1024      4096      8192
        64, 64        12 / 12    12 / 18   16 / 21   39 / 40   71 / 57
        128, 512      12 / 12    14 / 18   19 / 31   49 / 52   88 / 82
        32, 1024                 14 / 15   20 / 19   51 / 44 - 53
        16, 512       12 / 13    12 / 13   16 / 13   39 / 23
        1, any        10 / 7     12 / 8
    The weight gradient stays a library product that adds into its target: 7 us against 8 - 12 here."""
    if ((M + 63) // 64) * ((nIn + 63) // 64) > 16 or M < 2:
        return False
    return N <= (4096 if M >= 64 else 512)


_transforms, _tracing, _compiling = torch._C._functorch.peek_interpreter_stack, torch._C._is_tracing, torch.compiler.is_compiling


def _plain_autograd():
    """No forward-mode level, functorch transform or tracer is active: the cases that differentiate or record through torch operators
    and that a custom autograd function does not serve."""
    return forward_ad._current_level < 0 and _transforms() is None and not _tracing() and not _compiling()


_STEP = threading.local()


class TrainingStep:
    """A trainer's forward and backward pass:

        with TrainingStep() as step:
            step.backward(loss_of(inputs))

    While ``step.backward`` runs, the fp32 layers of that forward pass add their weight and bias gradients straight into the parameters'
    preallocated ``.grad``.  Anywhere else (``torch.autograd.grad``, a user's own ``backward``) they return them to autograd, which
    knows what was asked for."""
    __slots__ = ("live", "outer")

    def __enter__(self):
        self.live, self.outer = False, getattr(_STEP, "current", None)
        _STEP.current = self
        return self

    def __exit__(self, *exc):
        _STEP.current = self.outer
        return False

    def backward(self, loss):
        self.live = True
        try:
            loss.backward()
        finally:
            self.live = False


def _own_grad(p, step):
    """The parameter's preallocated fp32 gradient when the kernels may add to it in autograd's place (the trainer's own backward pass is
    running and nobody hooked the leaf)."""
    g = p.grad if step is not None and step.live and p.is_leaf else None
    if g is None or g.dtype != torch.float32 or p._backward_hooks or getattr(p, "_post_accumulate_grad_hooks", None) \
            or getattr(p, "_grad_ready", None) is not None:
        return None
    return g


class _Linear32Fn(torch.autograd.Function):
    """``act(x @ W + b)`` in fp32 for small layers: bias and ReLU in the product's epilogue, the bias gradient in the pass that applies
    the activation's, the weight gradient added straight into the parameter's."""

    @staticmethod
    def forward(ctx, x, W, b, relu):
        y = torch.empty((x.shape[0], W.shape[1]), dtype=torch.float32, device=x.device)
        _sgemm(x, W, y, bias=None if b is None else b.detach().reshape(-1), act=1 if relu else 0)
        ctx.relu, ctx.refs, ctx.step = relu, (W, b), getattr(_STEP, "current", None)
        ctx.save_for_backward(x, W, b, y if relu else None)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, W, b, y = ctx.saved_tensors
        need = ctx.needs_input_grad
        if torch.is_grad_enabled():                    # create_graph: the gradient has to be differentiable itself
            dz = dy.masked_fill(y <= 0, 0.0) if ctx.relu else dy
            return (dz @ W.t() if need[0] else None, x.t() @ dz if need[1] else None,
                    dz.sum(0).reshape(b.shape) if b is not None and need[2] else None, None)
        l = require()
        dy = _dense16(dy)
        M, N = dy.shape
        Wl, bl = ctx.refs
        db = acc = None
        if b is not None and need[2]:
            acc = _own_grad(bl, ctx.step)
            if acc is None or not acc.is_contiguous():
                acc = db = torch.zeros(N, dtype=torch.float32, device=dy.device)
        dz = dy
        if ctx.relu or acc is not None:
            dz = torch.empty_like(dy) if ctx.relu else dy
            rc = l.dl4j_bias_act_bwd(_ptr(dy), _ptr(y), _ptr(dz) if ctx.relu else None, _ptr(acc), M, N, 1 if ctx.relu else 0, 2, _stream())
            _check(rc, "dl4j_bias_act_bwd")
        dx = dW = None
        if need[0]:
            dx = _sgemm(dz, W.t(), torch.empty_like(x, memory_format=torch.contiguous_format)) if _sgemm_wins_dgrad(M, N, x.shape[1]) else dz @ W.t()
        if need[1]:
            g = _own_grad(Wl, ctx.step)
            if g is not None and _unit(g):
                g.addmm_(x.t(), dz)
            elif W.stride(0) == 1 and W.shape[0] > 1:           # 'f' order
                dW = (dz.t() @ x).t()
            else:
                dW = x.t() @ dz
        return dx, dW, None if db is None else db.reshape(b.shape), None


def linear32(x, W, b, relu):
    """fp32 dense layer on the small-problem kernel, or None when the case is not covered or the library does it better."""
    if not available() or x.dim() != 2 or x.dtype != torch.float32 or W.dtype != torch.float32 or W.dim() != 2 \
            or W.shape[0] != x.shape[1] or min(x.shape[0], *W.shape) == 0:
        return None
    grad = torch.is_grad_enabled() and (x.requires_grad or W.requires_grad or (b is not None and b.requires_grad))
    if not _sgemm_wins(x.shape[0], W.shape[1], x.shape[1], relu, grad) \
            or torch.backends.cuda.matmul.allow_tf32 or torch.is_autocast_enabled() or not _unit(x) or not on_current_device(x, W, b):
        return None
    if not ((W.stride(0) == 1 and W.stride(1) >= W.shape[0]) or (W.stride(1) == 1 and W.stride(0) >= W.shape[1])):
        return None
    if b is not None and (b.dtype != torch.float32 or b.numel() != W.shape[1] or not b.is_contiguous()):
        return None
    if not _plain_autograd():
        return None
    if x.stride(1) != 1:
        x = x.contiguous()
    if not grad:
        return _sgemm(x, W, torch.empty((x.shape[0], W.shape[1]), dtype=torch.float32, device=x.device), bias=b, act=1 if relu else 0)
    return _Linear32Fn.apply(x, W, b, bool(relu))


# =========================================================================== layer norm
_LN_ONE_PASS = os.environ.get("DL4J_LN_BWD_ONEPASS", "0") == "1"


def _dense16(t):
    """Contiguous, with the strides of its shape and on a 16-byte boundary (the vector kernels' requirement): a view off the grid is
    copied.  An extent of one leaves its stride open, and a slice keeps the pitch it was cut from there."""
    t = t.contiguous()
    if t.data_ptr() % 16:
        return t.clone(memory_format=torch.contiguous_format)
    return t.view(-1).view(t.shape) if 1 in t.shape else t


class _LayerNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gain, bias, eps, res=None):
        l = require()
        shp = x.shape
        C = shp[-1]
        x2 = _dense16(x.reshape(-1, C))
        rows = x2.shape[0]
        y = torch.empty_like(x2)
        mean = torch.empty(rows, dtype=torch.float32, device=x.device)
        rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
        gain = getattr(gain, "_master", gain)
        bias = getattr(bias, "_master", bias) if bias is not None else None
        g32 = _dense16(gain.detach().float().reshape(-1))
        b32 = _dense16(bias.detach().float().reshape(-1)) if bias is not None else None
        r2 = s2 = None
        if res is not None:
            # y = LN(x + res): the kernel adds the residual while loading and writes the sum once (kept for the backward)
            r2 = _dense16(res.reshape(-1, C))
            s2 = torch.empty_like(x2)
        rc = l.dl4j_layer_norm_fwd(_ptr(x2), _ptr(r2), _ptr(g32), _ptr(b32), _ptr(y), _ptr(s2), _ptr(mean), _ptr(rstd), rows, C,
                                   float(eps), _DT[x.dtype], _stream())
        _check(rc, "dl4j_layer_norm_fwd")
        ctx.has_res = res is not None
        ctx.save_for_backward(x2 if s2 is None else s2, g32, mean, rstd)
        ctx.refs = (gain, bias)
        ctx.shape = shp
        return y.reshape(shp)

    @staticmethod
    def backward(ctx, dy):
        l = require()
        x2, g32, mean, rstd = ctx.saved_tensors
        gain, bias = ctx.refs
        rows, C = x2.shape
        dy2 = dy.reshape(rows, C)
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dx = torch.empty_like(x2)

        def acc_for(p):
            if p is None:
                return None, None
            if p.is_leaf and p.grad is not None and p.grad.dtype == torch.float32 and p.grad.is_contiguous():
                return p.grad, None
            t = torch.zeros(C, dtype=torch.float32, device=dy.device)
            return t, t
        gacc, gret = acc_for(gain)
        bacc, bret = acc_for(bias)
        if _LN_ONE_PASS and C <= 1024 and C % 8 == 0 and all(t is None or t.data_ptr() % 16 == 0 for t in (dy2, x2, dx, g32)):
            # one kernel: dx and the per-block partial sums of dgain / dbias from a single read of dy and x, summed in block order
            if not hasattr(l.dl4j_layer_norm_bwd_noalloc, "_typed"):
                vp = ctypes.c_void_p
                l.dl4j_layer_norm_bwd_noalloc.argtypes = [vp, vp, vp, vp, vp, vp, vp, vp, ctypes.c_longlong, ctypes.c_int, ctypes.c_int,
                                                          ctypes.c_int, vp]
                l.dl4j_layer_norm_bwd_noalloc.restype = ctypes.c_int
                l.dl4j_layer_norm_bwd_noalloc._typed = True
            rc = l.dl4j_layer_norm_bwd_noalloc(_ptr(dy2), _ptr(x2), _ptr(g32), _ptr(mean), _ptr(rstd), _ptr(dx), _ptr(gacc), _ptr(bacc),
                                               rows, C, _DT[x2.dtype], 1, _stream())
            _check(rc, "dl4j_layer_norm_bwd_noalloc")
        else:
            partial = torch.empty(4 * num_sms() * C, dtype=torch.float32, device=dy.device)
            rc = l.dl4j_layer_norm_grad(_ptr(dy2), _ptr(x2), _ptr(g32), _ptr(mean), _ptr(rstd), _ptr(dx), _ptr(gacc), _ptr(bacc),
                                        _ptr(partial), rows, C, 0.0, _DT[x2.dtype], 1, num_sms(), _stream())
            _check(rc, "dl4j_layer_norm_grad")
        if gret is not None:
            gret = gret.reshape(gain.shape).to(gain.dtype)
        if bret is not None:
            bret = bret.reshape(bias.shape).to(bias.dtype)
        dx = dx.reshape(ctx.shape)
        return dx, gret, bret, None, (dx if ctx.has_res else None)


def layer_norm_grad(x, gain, bias, dy, eps):
    """(dx, dgain, dbias) of LN(x) over the last axis without running the forward (``dbias`` None without ``bias``): one sweep that
    takes the row statistics on the way.  None when the case is not covered."""
    if not available() or not x.is_cuda or x.dtype not in _DT or x.dim() < 1 or not 1 <= x.shape[-1] <= 8192 or x.numel() == 0:
        return None
    C = x.shape[-1]
    for p in (gain, bias):
        if p is not None and (p.numel() != C or not p.is_floating_point() or p.dtype == torch.float64):
            return None
    if dy.numel() != x.numel() or not on_current_device(x, gain, bias, dy) or not _plain_autograd():
        return None
    l = _LIB
    x2 = x if x.is_contiguous() else x.contiguous()
    dy2 = dy if dy.dtype == x.dtype and dy.is_contiguous() else dy.to(x.dtype).contiguous()
    g32 = gain if gain.dtype == torch.float32 and gain.is_contiguous() else gain.float().contiguous()
    rows = x2.numel() // C
    sms = num_sms()
    dx, dg = torch.empty_like(x2), torch.empty_like(g32)             # a third of the time of an empty() with its type and device
    db = None if bias is None else g32.new_empty(bias.shape)
    partial = g32.new_empty(4 * sms * C)
    rc = l.dl4j_layer_norm_grad(dy2.data_ptr(), x2.data_ptr(), g32.data_ptr(), None, None, dx.data_ptr(), dg.data_ptr(), _ptr(db),
                                partial.data_ptr(), rows, C, float(eps), _DT[x.dtype], 0, sms, _stream())
    _check(rc, "dl4j_layer_norm_grad")
    return dx, dg if gain.dtype == torch.float32 else dg.to(gain.dtype), db if bias is None or bias.dtype == torch.float32 else db.to(bias.dtype)


def layer_norm(x, gain, bias, eps, residual=None):
    """LN(x) or, with ``residual`` (same shape and dtype as x), LN(x + residual) in one pass."""
    C = x.shape[-1]
    if not available() or C % 8 != 0 or C > 1024 or x.dtype not in _DT:
        return None
    if residual is not None and (residual.shape != x.shape or residual.dtype != x.dtype):
        return None
    return _LayerNormFn.apply(x, gain, bias, eps, residual)


# =========================================================================== softmax cross entropy
class _SoftmaxXentFn(torch.autograd.Function):
    """Per-row loss; the forward stores only (loss, log-sum-exp, label mass) and the backward writes the gradient already
    multiplied by the upstream per-row scale, so neither pass materialises an unscaled gradient."""

    @staticmethod
    def forward(ctx, logits, labels, sparse):
        l = require()
        if logits.stride(1) != 1:
            logits = logits.contiguous()
        rows, C = logits.shape
        loss = torch.empty(rows, dtype=torch.float32, device=logits.device)
        stats = torch.empty((2, rows), dtype=torch.float32, device=logits.device)
        if sparse:
            idx, lab = labels.reshape(-1).to(torch.int64).contiguous(), None
        else:
            idx, lab = None, labels.to(logits.dtype).contiguous()
        rc = l.dl4j_softmax_xent_fwd(_ptr(logits), _ptr(lab), _ptr(idx), _ptr(loss), _ptr(stats[0]), _ptr(stats[1]), rows, C,
                                     logits.stride(0), -100, _DT[logits.dtype], _stream())
        _check(rc, "dl4j_softmax_xent_fwd")
        ctx.save_for_backward(logits, stats, *([idx] if sparse else [lab]))
        ctx.sparse = sparse
        return loss

    @staticmethod
    def backward(ctx, dloss):
        l = require()
        logits, stats, lab_or_idx = ctx.saved_tensors
        rows, C = logits.shape
        # logits on a 16-byte row pitch (a layer of odd width) get a gradient on the same pitch: vector stores here, no copy there
        pitched = C % 8 and logits.stride(0) == (C + 7) // 8 * 8
        grad = _pitched(rows, C, logits.dtype, logits.device) if pitched else torch.empty((rows, C), dtype=logits.dtype, device=logits.device)
        d = dloss.reshape(-1).float().contiguous()
        idx, lab = (lab_or_idx, None) if ctx.sparse else (None, lab_or_idx)
        rc = l.dl4j_softmax_xent_bwd(_ptr(logits), _ptr(lab), _ptr(idx), _ptr(stats[0]), _ptr(stats[1]), _ptr(d), _ptr(grad), rows, C,
                                     logits.stride(0), grad.stride(0), -100, _DT[logits.dtype], _stream())
        _check(rc, "dl4j_softmax_xent_bwd")
        return grad, None, None


def softmax_xent(logits, labels, sparse):
    if not available() or logits.dim() != 2 or logits.dtype not in _DT:
        return None
    return _SoftmaxXentFn.apply(logits, labels, bool(sparse))


# =========================================================================== row gather (embedding lookup)
class _GatherRowsFn(torch.autograd.Function):
    """``table[idx]`` along dim 0.  The gradient is scattered with fp32 vector reductions: straight into the table's
    preallocated fp32 gradient when it has one (nothing is returned for the table then), else into a fresh fp32 buffer."""

    @staticmethod
    def forward(ctx, table, idx):
        ctx.table_ref = getattr(table, "_master", table)
        ctx.table_dtype, ctx.V = table.dtype, table.shape[0]
        ctx.save_for_backward(idx)
        return torch.index_select(table.detach(), 0, idx)

    @staticmethod
    def backward(ctx, dy):
        (idx,) = ctx.saved_tensors
        l = require()
        tbl = ctx.table_ref
        if dy.stride(1) != 1 or dy.stride(0) % 8 or dy.data_ptr() % 16:
            dy = dy.contiguous()
        C = dy.shape[1]
        g = tbl.grad if (tbl.is_leaf and tbl.grad is not None) else None
        direct = g is not None and g.dtype == torch.float32 and g.is_contiguous() and g.data_ptr() % 16 == 0
        out = g if direct else torch.zeros((ctx.V, C), dtype=torch.float32, device=dy.device)
        rc = l.dl4j_scatter_add_rows(_ptr(dy), _ptr(idx), _ptr(out), idx.numel(), C, dy.stride(0), ctx.V, _DT[dy.dtype], _stream())
        _check(rc, "dl4j_scatter_add_rows")
        return (None if direct else out.to(ctx.table_dtype)), None


def gather_rows(table, idx):
    """Differentiable ``table[idx]`` (2-D table, 1-D int64 indices) or None when the case is not covered."""
    if not available() or table.dim() != 2 or table.dtype not in _DT or table.shape[1] % 8 or not table.is_contiguous():
        return None
    if not (torch.is_grad_enabled() and table.requires_grad):
        return None
    return _GatherRowsFn.apply(table, idx.reshape(-1).to(torch.int64).contiguous())


# =========================================================================== LSTM cell
class _LstmCellFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, z, c_prev):
        l = require()
        mb, n4 = z.shape
        n = n4 // 4
        z = z.contiguous()
        c_prev = c_prev.contiguous()
        h = torch.empty((mb, n), dtype=z.dtype, device=z.device)
        c = torch.empty((mb, n), dtype=torch.float32, device=z.device)
        need = any(ctx.needs_input_grad)
        gates = torch.empty_like(z) if need else None
        rc = l.dl4j_lstm_cell_fwd(_ptr(z), _ptr(c_prev), _ptr(h), _ptr(c), _ptr(gates), mb, n, _DT[z.dtype], _stream())
        _check(rc, "dl4j_lstm_cell_fwd")
        ctx.save_for_backward(gates, c, c_prev)
        return h, c

    @staticmethod
    def backward(ctx, dh, dc):
        l = require()
        gates, c, c_prev = ctx.saved_tensors
        mb, n = c.shape
        dz = torch.empty_like(gates)
        dc_prev = torch.empty_like(c)
        dh = dh.contiguous() if dh is not None else None
        dc = dc.contiguous().float() if dc is not None else None
        rc = l.dl4j_lstm_cell_bwd(_ptr(dh), _ptr(dc), _ptr(gates), _ptr(c), _ptr(c_prev), _ptr(dz), _ptr(dc_prev), mb, n,
                                  _DT[gates.dtype], _stream())
        _check(rc, "dl4j_lstm_cell_bwd")
        return dz, dc_prev


def lstm_cell(z, c_prev):
    if not available() or z.dtype not in _DT or c_prev.dtype != torch.float32:
        return None
    return _LstmCellFn.apply(z, c_prev)


class _LstmSeqFn(torch.autograd.Function):
    """Whole-sequence LSTM layer: forward is one persistent cooperative kernel (recurrent weights resident in
    shared memory, tcgen05 MMAs per step, grid-wide step barrier); backward walks the steps with the fused
    cell-gradient kernel plus one small GEMM per step and finishes with a single large weight-gradient GEMM.
    Gate order and math: libnd4j ops/declarable/helpers/impl/lstmLayer.cpp, LSTMHelpers.java."""

    PERSISTENT_BACKWARD = True       # False: per-step cell-gradient kernel + GEMM (kept as the cross-check path)

    @staticmethod
    def forward(ctx, zx, rw, h0, c0, reverse, rw_lp):
        l = require()
        T, mb, n4 = zx.shape
        n = n4 // 4
        zx = zx.contiguous()
        rw_t = rw_lp.t().contiguous()              # [4n, n]; a no-op for the 'f'-ordered parameter view
        ctx.rw_dtype = rw.dtype
        dev = zx.device
        h_all = torch.empty((T + 1, mb, n), dtype=torch.bfloat16, device=dev)
        h_all[0].copy_(h0)
        cs = torch.empty((T, mb, n), dtype=torch.float32, device=dev)
        gates = torch.empty((T, mb, n4), dtype=torch.bfloat16, device=dev)
        counter = torch.empty(1, dtype=torch.int32, device=dev)       # of this launch alone: two streams may run the kernel at once
        c0 = c0.contiguous()
        rc = l.dl4j_lstm_seq_fwd(_ptr(zx), _ptr(rw_t), _ptr(h_all), _ptr(c0), _ptr(cs), _ptr(gates), T, mb, n, int(bool(reverse)),
                                 _ptr(counter), _stream())
        _check(rc, "dl4j_lstm_seq_fwd")
        ctx.reverse = bool(reverse)
        ctx.save_for_backward(rw_t, h_all, cs, gates, c0)
        out = h_all[1:].flip(0) if reverse else h_all[1:]
        t_last = 0 if reverse else T - 1
        return out, h_all[T], cs[t_last]

    @staticmethod
    def backward(ctx, dout, dh_last, dc_last):
        l = require()
        rw_t, h_all, cs, gates, c0 = ctx.saved_tensors
        T, mb, n = cs.shape
        rev = ctx.reverse
        dout = dout.contiguous() if dout is not None else torch.zeros((T, mb, n), dtype=torch.bfloat16, device=cs.device)
        dzx = torch.empty_like(gates)
        dc = dc_last.contiguous().float() if dc_last is not None else None
        dh_rec = dh_last.to(torch.bfloat16) if dh_last is not None else None
        dt = _DT[gates.dtype]
        stream = _stream()
        persistent = _LstmSeqFn.PERSISTENT_BACKWARD and dout.dtype == torch.bfloat16
        if persistent:
            # every step of the gradient recursion in one cooperative kernel; weights as [n, 4n] row-major
            if dh_rec is not None:
                dout = dout.clone()
                dout[0 if rev else T - 1] += dh_rec
            rwt = transpose16(rw_t)
            need_h0, need_c0 = ctx.needs_input_grad[2], ctx.needs_input_grad[3]
            dh0 = torch.empty((mb, n), dtype=torch.bfloat16, device=cs.device) if need_h0 else None
            dc0 = torch.empty_like(c0) if need_c0 else None
            counter = torch.empty(1, dtype=torch.int32, device=cs.device)
            rc = l.dl4j_lstm_seq_bwd(_ptr(dout), _ptr(gates), _ptr(cs), _ptr(c0), _ptr(rwt), _ptr(dzx), _ptr(dc), _ptr(dh0), _ptr(dc0),
                                     T, mb, n, int(rev), _ptr(counter), stream)
            _check(rc, "dl4j_lstm_seq_bwd")
            dh_rec, dc = dh0, dc0
        dc_bufs = (torch.empty_like(c0), torch.empty_like(c0))
        for s in (range(T - 1, -1, -1) if not persistent else ()):
            t = T - 1 - s if rev else s
            if s == T - 1:
                dh = dout[t] if dh_rec is None else dout[t] + dh_rec
            else:
                dh = dh_rec
            if s > 0:
                tp = t + 1 if rev else t - 1
                c_prev = cs[tp]
            else:
                c_prev = c0
            dc_new = dc_bufs[s & 1]
            rc = l.dl4j_lstm_cell_bwd(_ptr(dh), _ptr(dc), _ptr(gates[t]), _ptr(cs[t]), _ptr(c_prev), _ptr(dzx[t]), _ptr(dc_new), mb, n,
                                      dt, stream)
            _check(rc, "dl4j_lstm_cell_bwd")
            dc = dc_new
            if s > 0:
                tn = t + 1 if rev else t - 1           # time index processed by step s - 1
                dh_rec = torch.addmm(dout[tn], dzx[t], rw_t)
            else:
                dh_rec = torch.mm(dzx[t], rw_t) if ctx.needs_input_grad[2] else None
        drw = None
        if ctx.needs_input_grad[1]:
            h_prev = h_all[:T].flip(0) if rev else h_all[:T]      # hidden state entering each time index
            a, b = dzx.reshape(T * mb, 4 * n).t(), h_prev.reshape(T * mb, n)
            if ctx.rw_dtype == torch.float32 and _operand_a(a) is not None and _operand_b(b) is not None:
                drw_t = gemm_raw(a, b, out_dtype=torch.float32)
            else:
                drw_t = torch.mm(a, b).to(ctx.rw_dtype)
            drw = drw_t.t()
        return dzx, drw, dh_rec, (dc if ctx.needs_input_grad[3] else None), None, None


def transpose16(m):
    """Dense 2-D bf16 / fp16 matrix -> its transpose as a new dense matrix (tiled kernel; falls back to the strided copy)."""
    if m.dim() == 2 and m.is_contiguous() and m.is_cuda and m.element_size() == 2 and m.shape[0] % 2 == 0 and m.shape[1] % 2 == 0:
        out = torch.empty((m.shape[1], m.shape[0]), dtype=m.dtype, device=m.device)
        rc = require().dl4j_transpose16(_ptr(m), _ptr(out), m.shape[0], m.shape[1], _stream())
        _check(rc, "dl4j_transpose16")
        return out
    return m.t().contiguous()


def lstm_seq_supported(zx, n, mb):
    """Hidden sizes off the 64 grid run zero-padded (``lstm_seq``) from two steps on; for a single one the padding costs more than the
    general step (two layers of 500 units, 100 rows: inference 595 against 457 us, training 1934 against 1535; at two steps 594 against
    620 and 1958 against 1982)."""
    return (available() and zx.is_cuda and zx.dtype == torch.bfloat16 and 1 <= n <= 1280 and 1 <= mb <= 128 and (n % 64 == 0 or zx.shape[0] > 1))


def lstm_seq(zx, rw, h0, c0, reverse=False):
    """``zx`` [T, mb, 4n] bf16 input pre-activations, ``rw`` [n, 4n] recurrent weights.  Returns (h for every
    time index [T, mb, n], last h, last c).

    The kernels work on 64 hidden units at a time; other sizes are padded with units whose pre-activations and weights are zero: such a
    unit stays at c = 0, h = 0 and contributes exactly nothing to the others.  Two layers of 200 units, 50 steps, 32 sequences: the
    step-by-step path took 1355 launches and 4.3 ms per training step."""
    rw_lp = getattr(rw, "_lp", None)
    if rw_lp is None or rw_lp.dtype != zx.dtype:
        rw_lp = rw.detach() if rw.dtype == zx.dtype else rw.detach().to(zx.dtype)
    n = h0.shape[1]
    pad = -n % 64
    if pad == 0:
        return _LstmSeqFn.apply(zx, rw, h0, c0, reverse, rw_lp)
    import torch.nn.functional as F
    T, mb = zx.shape[0], zx.shape[1]

    def wide(w):        # [n, 4n] -> [n + pad, 4 (n + pad)], column-major like the parameter
        return F.pad(w.t().reshape(4, n, n), (0, pad, 0, pad)).reshape(4 * (n + pad), n + pad).t()
    zx_w = F.pad(zx.reshape(T, mb, 4, n), (0, pad)).reshape(T, mb, 4 * (n + pad))
    rw_m = getattr(rw, "_master", rw)
    hs, h, c = _LstmSeqFn.apply(zx_w, wide(rw_m), F.pad(h0, (0, pad)), F.pad(c0, (0, pad)), reverse, wide(rw_lp))
    return hs[..., :n], h[:, :n].contiguous(), c[:, :n].contiguous()


def _f_ordered(w, *types):
    """A weight of one of the given types whose columns are contiguous (the 'f'-ordered parameter views)."""
    return w.dim() == 2 and w.is_cuda and w.dtype in types and w.stride(0) == 1 and w.stride(1) == w.shape[0]


def lstm_step_supported(x, W, RW, n, mb, *rest):
    """One inference step as one launch (``csrc/lstm_step.cu``) for mb * n up to LSTM_STEP_MAX; ``rest``: its other operands."""
    return (available() and x.is_cuda and x.dtype == torch.bfloat16 and not torch.is_grad_enabled() and mb * n <= LSTM_STEP_MAX
            and _f_ordered(W, torch.float32) and _f_ordered(RW, torch.float32) and on_current_device(x, W, RW, *rest)
            and _plain_autograd())


# Measured per call for two layers (whole rnnTimeStep, device / wall us; step kernel against sequence kernel): 256 x 1: 17.7 / 195 against
# 40 / 352; 1024 x 8: 42 / 195 against 56 / 328; 1024 x 32: 114 / 166 against 56 / 328; 1024 x 64: 210 / 222 against 57 / 328.  Up to
# here the launches saved are worth more than the device time lost; past it a caller that queues steps would be slowed down.
LSTM_STEP_MAX = 32768


def _small_sigs(l):
    if not hasattr(l.dl4j_lstm_step, "_typed"):
        vp, i32, lng = ctypes.c_void_p, ctypes.c_int, ctypes.c_long
        l.dl4j_lstm_step.argtypes = [vp, lng, vp, vp, vp, vp, vp, vp, vp, i32, i32, i32, vp]
        l.dl4j_lstm_step.restype = i32
        l.dl4j_linear_small.argtypes = [vp, lng, vp, i32, vp, vp, i32, i32, i32, vp]
        l.dl4j_linear_small.restype = i32
        l.dl4j_lstm_step._typed = True
    return l


def lstm_step(x, W, RW, b, h, c):
    """(h', c') of one LSTM step: x [mb, nIn] bf16, W [nIn, 4n] / RW [n, 4n] fp32 column-major, b fp32, h [mb, n] bf16, c [mb, n] fp32."""
    l = _small_sigs(require())
    mb, nIn = x.shape
    x = x if x.stride(1) == 1 else x.contiguous()
    h, c = h.contiguous(), c.contiguous()
    h_out, c_out = torch.empty_like(h), torch.empty_like(c)
    rc = l.dl4j_lstm_step(_ptr(x), x.stride(0), _ptr(W), _ptr(RW), _ptr(b), _ptr(h), _ptr(c), _ptr(h_out),
                          _ptr(c_out), mb, nIn, h.shape[1], _stream())
    _check(rc, "dl4j_lstm_step")
    return h_out, c_out


def linear_small(x, W, b):
    """``x @ W + b`` without a gradient for up to 32 rows of bf16 activations on the parameters themselves, or None when not covered."""
    if torch.is_grad_enabled() or not available() or not x.is_cuda or x.dim() != 2 or x.dtype != torch.bfloat16 or not 1 <= x.shape[0] <= 32 \
            or not _f_ordered(W, torch.float32, torch.bfloat16) or W.shape[0] != x.shape[1] or W.numel() == 0 or (b is not None and (b.dtype != torch.float32 or b.numel() != W.shape[1])) \
            or not on_current_device(x, W, b) or not _plain_autograd():
        return None
    l = _small_sigs(require())
    x = x if x.stride(1) == 1 else x.contiguous()
    b = None if b is None else b.detach().reshape(-1).contiguous()
    y = torch.empty((x.shape[0], W.shape[1]), dtype=x.dtype, device=x.device)
    rc = l.dl4j_linear_small(_ptr(x), x.stride(0), _ptr(W), int(W.dtype == torch.float32), _ptr(b), _ptr(y), x.shape[0], x.shape[1], W.shape[1],
                             _stream())
    _check(rc, "dl4j_linear_small")
    return y


class _ConvWeightFn(torch.autograd.Function):
    """fp32 [O, I, kH, kW] convolution kernel -> bf16 channels-last view for the tensor-core convolution kernels (one cast +
    relayout pass); the channels-last weight gradient is added straight into the fp32 gradient buffer of the parameter."""

    @staticmethod
    def forward(ctx, W):
        l = require()
        O, I, kH, kW = W.shape
        buf = torch.empty((O, kH, kW, I), dtype=torch.bfloat16, device=W.device)
        Wm = getattr(W, "_master", W)
        rc = l.dl4j_conv_weight_to_cl(_ptr(Wm.detach().contiguous()), _ptr(buf), O, I, kH * kW, _stream())
        _check(rc, "dl4j_conv_weight_to_cl")
        ctx.W_ref = Wm
        return buf.permute(0, 3, 1, 2)

    @staticmethod
    def backward(ctx, dW):
        l = require()
        W = ctx.W_ref
        O, I, kH, kW = W.shape
        g_cl = dW.to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
        tgt = W.grad if (W.is_leaf and W.grad is not None and W.grad.dtype == torch.float32 and W.grad.is_contiguous()) else None
        out = tgt if tgt is not None else torch.zeros(W.shape, dtype=torch.float32, device=W.device)
        rc = l.dl4j_conv_wgrad_from_cl(_ptr(g_cl), _ptr(out), O, I, kH * kW, _stream())
        _check(rc, "dl4j_conv_wgrad_from_cl")
        return None if tgt is not None else out.to(W.dtype)


def _conv_sigs(l):
    if getattr(l, "_conv_typed", False):
        return
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    l.dl4j_conv2d.argtypes = [i32, vp, vp, vp, vp] + [i32] * 17 + [vp]
    l.dl4j_conv2d.restype = i32
    l.dl4j_conv2d_wgrad.argtypes = [vp, vp, vp] + [i32] * 15 + [vp]
    l.dl4j_conv2d_wgrad.restype = i32
    l.dl4j_conv_wgrad_f32_from_cl.argtypes = [vp, vp, i32, i32, i32, vp]
    l.dl4j_conv_wgrad_f32_from_cl.restype = i32
    l._conv_typed = True


class _Conv2dFn(torch.autograd.Function):
    """Stride-1 2-D convolution on the tcgen05 implicit-GEMM kernels (``csrc/conv_tcgen05.cu``): forward, data gradient
    and weight gradient.  ``x`` is a channels-last 16-bit activation [N, Cin, H, W].  ``W`` is either the fp32 parameter
    [Cout, Cin, kH, kW] (it is cast and laid out channels-last here, and its gradient is added straight into the
    parameter's fp32 gradient buffer when it has one) or an already channels-last 16-bit kernel (its gradient is returned).
    ``fuse_w``: few-channel stem form, see ``dl4j_conv2d``."""

    @staticmethod
    def forward(ctx, x, W, bias, pad, dil, fuse_w, path=0):
        l = require()
        _conv_sigs(l)
        x = _dense_cl(x)
        N, Cin, H, Wd = x.shape
        Wm = getattr(W, "_master", W)
        Cout, _, kH, kW = Wm.shape
        if Wm.dtype == torch.float32:
            w_cl = torch.empty((Cout, kH, kW, Cin), dtype=x.dtype, device=x.device)
            if x.dtype == torch.bfloat16 and Wm.is_contiguous():
                rc = l.dl4j_conv_weight_to_cl(_ptr(Wm.detach()), _ptr(w_cl), Cout, Cin, kH * kW, _stream())
                _check(rc, "dl4j_conv_weight_to_cl")
            else:
                w_cl.copy_(Wm.detach().permute(0, 2, 3, 1))
            ctx.master = Wm
        else:
            w_cl = W.detach().permute(0, 2, 3, 1).contiguous()
            ctx.master = None
        OH = H + 2 * pad[0] - (kH - 1) * dil[0]
        OW = Wd + 2 * pad[1] - (kW - 1) * dil[1]
        y = torch.empty((N, OH, OW, Cout), dtype=x.dtype, device=x.device)
        b = None
        if bias is not None:
            b = bias.detach().reshape(-1)
            b = b if b.dtype in (torch.float32, x.dtype) else b.float()
            b = b.contiguous()
        ctx.geom = (N, H, Wd, Cin, OH, OW, Cout, kH, kW, int(pad[0]), int(pad[1]), int(dil[0]), int(dil[1]))
        ctx.fuse_w = int(bool(fuse_w))
        ctx.path = int(path)          # 0 automatic, 2 per-tap kernel, 4 halo kernel (tests)
        rc = l.dl4j_conv2d(0, _ptr(x), _ptr(w_cl), _ptr(y), _ptr(b), *ctx.geom, _DT[x.dtype],
                           1 if (b is not None and b.dtype == torch.float32) else 0, 0, ctx.fuse_w | ctx.path, _stream())
        _check(rc, "dl4j_conv2d")
        ctx.has_bias = bias is not None
        ctx.bias_dtype = bias.dtype if bias is not None else None
        ctx.bias_shape = tuple(bias.shape) if bias is not None else None
        ctx.w_dtype = W.dtype
        ctx.save_for_backward(x, w_cl)
        return y.permute(0, 3, 1, 2)

    @staticmethod
    def backward(ctx, dy):
        l = require()
        x, w_cl = ctx.saved_tensors
        N, H, Wd, Cin, OH, OW, Cout, kH, kW, ph, pw, dh, dw_ = ctx.geom
        dy = _dense_cl(dy)
        if dy.dtype != x.dtype:
            dy = dy.to(x.dtype)
        dx = dW = db = None
        if ctx.needs_input_grad[0]:
            dxb = torch.empty((N, H, Wd, Cin), dtype=x.dtype, device=x.device)
            rc = l.dl4j_conv2d(1, _ptr(dy), _ptr(w_cl), _ptr(dxb), None, *ctx.geom, _DT[x.dtype], 0, 0, ctx.path, _stream())
            _check(rc, "dl4j_conv2d")
            dx = dxb.permute(0, 3, 1, 2)
        if ctx.needs_input_grad[1] or ctx.master is not None:
            g_cl = torch.zeros((Cout, kH, kW, Cin), dtype=torch.float32, device=x.device)
            rc = l.dl4j_conv2d_wgrad(_ptr(dy), _ptr(x), _ptr(g_cl), *ctx.geom, _DT[x.dtype], ctx.fuse_w, _stream())
            _check(rc, "dl4j_conv2d_wgrad")
            Wm = ctx.master
            if Wm is not None:
                tgt = Wm.grad if (Wm.is_leaf and Wm.grad is not None and Wm.grad.dtype == torch.float32 and Wm.grad.is_contiguous()) else None
                out = tgt if tgt is not None else torch.zeros(Wm.shape, dtype=torch.float32, device=x.device)
                rc = l.dl4j_conv_wgrad_f32_from_cl(_ptr(g_cl), _ptr(out), Cout, Cin, kH * kW, _stream())
                _check(rc, "dl4j_conv_wgrad_f32_from_cl")
                dW = None if tgt is not None else out.to(ctx.w_dtype)
            else:
                dW = g_cl.permute(0, 3, 1, 2).to(ctx.w_dtype)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = dy.float().sum((0, 2, 3)).reshape(ctx.bias_shape).to(ctx.bias_dtype)
        return dx, dW, db, None, None, None, None


def conv2d(x, W, bias, pad, dil, fuse_w=False, path=None, relu=False):
    """Stride-1 convolution on the native implicit-GEMM kernels, or None when the case is not covered (the caller then
    uses the library path): 16-bit CUDA activation, channel counts multiples of 8, non-negative output size.  ``relu`` (inference
    only: no gradient) applies ReLU in the epilogue."""
    if not (available() and x.is_cuda and x.dim() == 4 and x.dtype in (torch.bfloat16, torch.float16)):
        return None
    Wm = getattr(W, "_master", W)
    if Wm.dim() != 4 or Wm.shape[1] != x.shape[1] or x.shape[1] % 8 or Wm.shape[0] % 8:
        return None
    if Wm.dtype != torch.float32 and Wm.dtype != x.dtype:
        return None
    kH, kW = Wm.shape[2], Wm.shape[3]
    if kH * kW > 64:
        return None
    if x.shape[2] + 2 * pad[0] - (kH - 1) * dil[0] < 1 or x.shape[3] + 2 * pad[1] - (kW - 1) * dil[1] < 1:
        return None
    if pad[0] < 0 or pad[1] < 0 or pad[0] > 255 or pad[1] > 255:
        return None
    if fuse_w and (pad[1] != 0 or dil[1] != 1 or kW * x.shape[1] > 64):
        fuse_w = False
    if relu:
        assert not (torch.is_grad_enabled() and (x.requires_grad or W.requires_grad)) and Wm.dtype == x.dtype and bias.dtype == torch.float32
        x = _dense_cl(x)
        return conv_infer_kxk(x, _dense16(W.permute(0, 2, 3, 1)), bias.contiguous(), kH, kW, pad, dil, True, fuse_w)
    return _Conv2dFn.apply(x, W, bias, (int(pad[0]), int(pad[1])), (int(dil[0]), int(dil[1])), bool(fuse_w),
                           {None: 0, "tap": 2, "halo": 4}[path])


# --------------------------------------------------------------------------- inference convolutions with batch norm folded in
def bn_fold(table, block_entry, params, w_out, b_out):
    """Folded weights (bf16, channels-last) and biases (fp32) of every convolution in ``table`` (``csrc/bn_fold.cu``), one launch."""
    l = require()
    if not hasattr(l.dl4j_bn_fold, "_typed"):
        vp, i32 = ctypes.c_void_p, ctypes.c_int
        l.dl4j_bn_fold.argtypes = [vp, vp, i32, vp, vp, vp, vp]
        l.dl4j_bn_fold.restype = i32
        l.dl4j_bn_fold._typed = True
    _check(l.dl4j_bn_fold(_ptr(table), _ptr(block_entry), block_entry.numel(), _ptr(params), _ptr(w_out), _ptr(b_out), _stream()),
           "dl4j_bn_fold")


def conv_infer_1x1(x, w, b, relu, residual=None):
    """relu?(x * w + b [+ residual]) for a dense channels-last x [N, Cin, H, W] and w [Cout, Cin] bf16, b fp32; one GEMM."""
    l = require()
    N, C, H, W = x.shape
    O = w.shape[0]
    M = N * H * W
    y = torch.empty((N, H, W, O), dtype=x.dtype, device=x.device)
    act = (1 << 16 if residual is not None else 1) if relu else 0
    rc = l.dl4j_gemm(x.data_ptr(), w.data_ptr(), y.data_ptr(), None, b.data_ptr(), None if residual is None else residual.data_ptr(), M, O, C,
                     C, C, O, 0, O, 0, 0, _DT[x.dtype], 1, 0, act, 0, 1, 1.0, _pick_block_n(M, O), num_sms(), _stream())
    _check(rc, "dl4j_gemm")
    return y.permute(0, 3, 1, 2)


def conv_infer_kxk(x, w, b, kH, kW, pad, dil, relu, fuse_w=False):
    """relu?(conv(x, w) + b), stride 1, for a dense channels-last x and w [Cout, kH * kW * Cin] bf16 (channels-last), b fp32."""
    l = require()
    _conv_sigs(l)
    N, C, H, W = x.shape
    O = w.shape[0]
    OH, OW = H + 2 * pad[0] - (kH - 1) * dil[0], W + 2 * pad[1] - (kW - 1) * dil[1]
    y = torch.empty((N, OH, OW, O), dtype=x.dtype, device=x.device)
    rc = l.dl4j_conv2d(0, x.data_ptr(), w.data_ptr(), y.data_ptr(), b.data_ptr(), N, H, W, C, OH, OW, O, kH, kW, pad[0], pad[1], dil[0], dil[1],
                       _DT[x.dtype], 1, int(bool(relu)), int(bool(fuse_w)), _stream())
    _check(rc, "dl4j_conv2d")
    return y.permute(0, 3, 1, 2)


def infer_program(steps, n, workspace, inputs, w, b):
    """Issues the ``n`` steps of a planned run of folded convolutions (``csrc/infer_program.cu``)."""
    global LAUNCHES
    l = require()
    if not hasattr(l.dl4j_infer_program, "_typed"):
        vp, i32 = ctypes.c_void_p, ctypes.c_int
        l.dl4j_infer_program.argtypes = [ctypes.c_char_p, i32, vp, vp, vp, vp, i32, i32, vp]
        l.dl4j_infer_program.restype = i32
        l.dl4j_infer_program._typed = True
    ext = (ctypes.c_void_p * len(inputs))(*[t.data_ptr() for t in inputs])
    rc = l.dl4j_infer_program(steps, n, _ptr(workspace), ext, _ptr(w), _ptr(b), _DT[workspace.dtype], num_sms(), _stream())
    LAUNCHES += n - 1
    _check(rc, "dl4j_infer_program")


def conv_weight_cl(W):
    """bf16 channels-last version of an fp32 convolution kernel parameter, or None when not applicable."""
    if not (available() and W.is_cuda and W.dim() == 4 and W.dtype == torch.float32 and W.is_contiguous()):
        return None
    return _ConvWeightFn.apply(W)


class _SubsampleFn(torch.autograd.Function):
    """x[:, :, ::sH, ::sW] of a channels-last bf16 activation as one gather kernel; the gradient is one scatter-with-zeros."""

    @staticmethod
    def forward(ctx, x, sH, sW):
        l = require()
        x = _dense_cl(x)
        N, C, H, W = x.shape
        OH, OW = (H + sH - 1) // sH, (W + sW - 1) // sW
        y = torch.empty((N, C, OH, OW), dtype=x.dtype, device=x.device, memory_format=torch.channels_last)
        ctx.shape = (N, H, W, C, OH, OW, 1, 1, sH, sW, 0, 0)
        rc = l.dl4j_subsample(_ptr(x), _ptr(y), (ctypes.c_int * 12)(*ctx.shape), 0, _stream())
        _check(rc, "dl4j_subsample")
        return y

    @staticmethod
    def backward(ctx, dy):
        l = require()
        N, H, W, C = ctx.shape[:4]
        dy = _dense_cl(dy)
        dx = torch.empty((N, C, H, W), dtype=dy.dtype, device=dy.device, memory_format=torch.channels_last)
        rc = l.dl4j_subsample(_ptr(dy), _ptr(dx), (ctypes.c_int * 12)(*ctx.shape), 1, _stream())
        _check(rc, "dl4j_subsample")
        return dx, None, None


def stem_space_to_depth(x, pad, Hs, Ws, CP):
    """2x2 space-to-depth view of the zero-padded input ``x`` [N, C, H, W] (16-bit, any strides, no gradient) as a channels-last
    tensor [N, CP, Hs, Ws] with channel (bh * 2 + bw) * C + c; one pass instead of pad / reshape / permute / pad / contiguous.
    Returns None when the case is not covered."""
    if not available() or x.requires_grad or x.dtype not in (torch.bfloat16, torch.float16) or CP not in (8, 16, 32):
        return None
    N, C, H, W = x.shape
    if 4 * C > CP:
        return None
    l = require()
    if not hasattr(l.dl4j_stem_space_to_depth, "_typed"):
        vp, i32 = ctypes.c_void_p, ctypes.c_int
        l.dl4j_stem_space_to_depth.argtypes = [vp, vp, i32, i32, i32, i32, ctypes.POINTER(ctypes.c_longlong), i32, i32, i32, i32, i32, vp]
        l.dl4j_stem_space_to_depth.restype = ctypes.c_int
        l.dl4j_stem_space_to_depth._typed = True
    out = torch.empty((N, Hs, Ws, CP), dtype=x.dtype, device=x.device)
    st = (ctypes.c_longlong * 4)(*x.stride())
    rc = l.dl4j_stem_space_to_depth(_ptr(x), _ptr(out), N, C, H, W, st, int(pad[0]), int(pad[1]), Hs, Ws, CP, _stream())
    _check(rc, "dl4j_stem_space_to_depth")
    return out.permute(0, 3, 1, 2)


def conv_few_channels(x, W, b, stride, pad, dil):
    """Convolution over an image of a few channels (an RGB stem; no gradient into it) as a GEMM over its patches, or None when not covered:
    16-bit image of any strides, ``W`` [Cout, C, kH, kW], C kH kW <= 64 and patches no larger than the output.  64 x 3 x 56 x 56 -> 256
    channels, 3 x 3, bf16: patches 11 us, products 41 us forward and 32 us for the weights; the library's zero-padded convolution took 52 and 63 us and 11 us of copies."""
    if not (available() and x.is_cuda and x.dim() == 4 and x.dtype in (torch.bfloat16, torch.float16)) or x.requires_grad or W.dim() != 4 \
            or W.shape[1] != x.shape[1] or min(*pad) < 0 or min(*stride, *dil) < 1 or not on_current_device(x, W, b) or not _plain_autograd():
        return None
    N, C, H, Wd = x.shape
    Cout, _, kH, kW = W.shape
    K = C * kH * kW
    KP = K + -K % 8
    OH, OW = (H + 2 * pad[0] - (kH - 1) * dil[0] - 1) // stride[0] + 1, (Wd + 2 * pad[1] - (kW - 1) * dil[1] - 1) // stride[1] + 1
    if KP > 64 or KP > Cout or Cout % 8 or N < 1 or OH < 1 or OW < 1 or N * OH * OW * KP // 8 >= 1 << 31:
        return None
    l = require()
    if not hasattr(l.dl4j_stem_patches, "_typed"):
        vp = ctypes.c_void_p
        l.dl4j_stem_patches.argtypes = [vp, vp, vp, ctypes.POINTER(ctypes.c_longlong), vp]
        l.dl4j_stem_patches.restype = ctypes.c_int
        l.dl4j_stem_patches._typed = True
    patches = torch.empty((N, OH, OW, KP), dtype=x.dtype, device=x.device)
    geom = (ctypes.c_int * 15)(N, C, H, Wd, OH, OW, kH, kW, *map(int, stride), *map(int, pad), *map(int, dil), KP)
    _check(l.dl4j_stem_patches(_ptr(x), _ptr(patches), geom, (ctypes.c_longlong * 4)(*x.stride()), _stream()), "dl4j_stem_patches")
    W2 = W.reshape(Cout, K, 1, 1)
    if KP != K:
        W2 = torch.nn.functional.pad(W2, (0, 0, 0, 0, 0, KP - K))
    return conv1x1(patches.permute(0, 3, 1, 2), W2, b)


def conv1x1(x, W, b, stride=(1, 1)):
    """1x1 convolution over a channels-last activation as one tcgen05 GEMM: [N*H*W, Cin] x [Cin, Cout] (forward, data
    gradient and weight gradient all run on the hand-written kernel).  ``W`` is the [Cout, Cin, 1, 1] parameter; returns
    None when the case is not covered."""
    if not available() or not x.is_cuda or x.dim() != 4 or x.dtype not in (torch.bfloat16, torch.float16):
        return None
    Cout, Cin = W.shape[0], W.shape[1]
    if W.dim() != 4 or W.shape[2] != 1 or W.shape[3] != 1 or Cin % 8 or Cout % 8 or x.shape[1] != Cin:
        return None
    W_lp = getattr(W, "_lp", None)
    if W_lp is None or W_lp.dtype != x.dtype:
        W_lp = W.detach() if W.dtype == x.dtype else W.detach().to(x.dtype)
    if not W_lp.is_contiguous() or W_lp.data_ptr() % 16:
        return None
    if stride[0] != 1 or stride[1] != 1:
        x = _SubsampleFn.apply(x, int(stride[0]), int(stride[1])) if x.dtype == torch.bfloat16 else x[:, :, ::stride[0], ::stride[1]]
    x = _dense_cl(x)
    N, _, H, Wd = x.shape
    x2 = x.permute(0, 2, 3, 1).reshape(N * H * Wd, Cin)
    if _operand_a(x2) is None:
        return None
    y2 = _LinearFn.apply(x2, W, b, 0, W_lp.view(Cout, Cin).t())
    return y2.view(N, H, Wd, Cout).permute(0, 3, 1, 2)


class _MaxPoolFn(torch.autograd.Function):
    """Channels-last max pooling; forward keeps one byte per output element (winning window position), backward gathers."""

    @staticmethod
    def forward(ctx, x, k, s, p):
        l = require()
        x = _dense_cl(x)
        N, C, H, W = x.shape
        OH = (H + 2 * p[0] - k[0]) // s[0] + 1
        OW = (W + 2 * p[1] - k[1]) // s[1] + 1
        y = torch.empty((N, C, OH, OW), dtype=x.dtype, device=x.device, memory_format=torch.channels_last)
        need = ctx.needs_input_grad[0]
        idx = torch.empty(N * OH * OW * C, dtype=torch.uint8, device=x.device) if need else None
        shape = (ctypes.c_int * 12)(N, H, W, C, OH, OW, k[0], k[1], s[0], s[1], p[0], p[1])
        rc = l.dl4j_maxpool_fwd(_ptr(x), _ptr(y), _ptr(idx), shape, _stream())
        _check(rc, "dl4j_maxpool_fwd")
        ctx.shape = (N, H, W, C, OH, OW, k[0], k[1], s[0], s[1], p[0], p[1])
        ctx.save_for_backward(idx)
        return y

    @staticmethod
    def backward(ctx, dy):
        l = require()
        (idx,) = ctx.saved_tensors
        N, H, W, C = ctx.shape[:4]
        dy = _dense_cl(dy)
        dx = torch.empty((N, C, H, W), dtype=dy.dtype, device=dy.device, memory_format=torch.channels_last)
        shape = (ctypes.c_int * 12)(*ctx.shape)
        rc = l.dl4j_maxpool_bwd(_ptr(dy), _ptr(idx), _ptr(dx), shape, _stream())
        _check(rc, "dl4j_maxpool_bwd")
        return dx, None, None, None


class _GlobalAvgPoolFn(torch.autograd.Function):
    """Mean over H and W of a channels-last activation; the gradient is written channels-last, as the layers in front of it want it."""

    @staticmethod
    def forward(ctx, x):
        l = _avgpool_lib()
        N, C, H, W = x.shape
        y = torch.empty((N, C), dtype=x.dtype, device=x.device)
        _check(l.dl4j_global_avgpool(0, _ptr(x), _ptr(y), N, H * W, C, _DT[x.dtype], _stream()), "dl4j_global_avgpool")
        ctx.shape = (N, C, H, W)
        return y

    @staticmethod
    def backward(ctx, dy):
        N, C, H, W = ctx.shape
        if torch.is_grad_enabled():                    # create_graph
            return (dy / (H * W)).reshape(N, C, 1, 1).expand(N, C, H, W)
        dy = _dense16(dy)
        dx = torch.empty((N, C, H, W), dtype=dy.dtype, device=dy.device, memory_format=torch.channels_last)
        _check(_avgpool_lib().dl4j_global_avgpool(1, _ptr(dy), _ptr(dx), N, H * W, C, _DT[dy.dtype], _stream()), "dl4j_global_avgpool")
        return dx


def _avgpool_lib():
    l = require()
    if not hasattr(l.dl4j_global_avgpool, "_typed"):
        vp, i32 = ctypes.c_void_p, ctypes.c_int
        l.dl4j_global_avgpool.argtypes = [i32, vp, vp, i32, i32, i32, i32, vp]
        l.dl4j_global_avgpool.restype = i32
        l.dl4j_global_avgpool._typed = True
    return l


def global_avgpool(x):
    """[N, C, H, W] 16-bit channels-last -> [N, C], or None when the case is not covered."""
    if not available() or x.dim() != 4 or x.dtype not in (torch.bfloat16, torch.float16) or x.numel() == 0 or x.shape[1] % 8 \
            or not on_current_device(x) or x.shape[0] > 65535 or not x.is_contiguous(memory_format=torch.channels_last) or x.data_ptr() % 16 or not _plain_autograd():
        return None
    return _GlobalAvgPoolFn.apply(x)


def maxpool2d(x, k, s, p):
    if not (available() and x.is_cuda and x.dim() == 4 and x.dtype == torch.bfloat16 and x.shape[1] % 8 == 0):
        return None
    if k[0] * k[1] > 255 or p[0] >= k[0] or p[1] >= k[1] or min(x.shape) == 0:
        return None
    if (x.shape[2] + 2 * p[0] - k[0]) < 0 or (x.shape[3] + 2 * p[1] - k[1]) < 0:
        return None
    return _MaxPoolFn.apply(x, tuple(int(v) for v in k), tuple(int(v) for v in s), tuple(int(v) for v in p))


# =========================================================================== batch norm (+ residual) (+ ReLU)
def _rows_c(x):
    """(rows, C) of a channels-last 4-D or a plain 2-D activation."""
    if x.dim() == 4:
        return x.shape[0] * x.shape[2] * x.shape[3], x.shape[1]
    return x.shape[0], x.shape[1]


def _dense_cl(x):
    """Channels-last dense layout for 4-D tensors, row-major for 2-D ones (copies only when needed)."""
    if x.dim() == 4:
        return x if x.is_contiguous(memory_format=torch.channels_last) else x.contiguous(memory_format=torch.channels_last)
    return x.contiguous()


def _dense_cl16(x):
    """``_dense_cl`` on a 16-byte boundary: a view off the grid is copied."""
    x = _dense_cl(x)
    return x if x.data_ptr() % 16 == 0 else x.clone()


class _BnActFn(torch.autograd.Function):
    """y = act(batchnorm_train(x) [+ res]) over channels-last bf16 activations; running statistics are updated in place by
    the kernel (``nn/layers/normalization/BatchNormalization.java`` semantics: biased batch variance, decay rule)."""

    @staticmethod
    def forward(ctx, x, res, gamma, beta, run_mean, run_stat, use_log_std, decay, eps, relu, pre_bias=None):
        l = require()
        x = _dense_cl16(x)
        res = _dense_cl16(res) if res is not None else None
        rows, C = _rows_c(x)
        y = torch.empty_like(x)
        save = torch.empty(2 * C, dtype=torch.float32, device=x.device)
        work = torch.empty(4 * C + 8, dtype=torch.float32, device=x.device)      # [sums | ticket | scale | shift]
        g = gamma.detach().float().contiguous() if gamma is not None else None
        b = beta.detach().float().contiguous() if beta is not None else None
        rc = l.dl4j_bn_fwd_train(_ptr(x), _ptr(res), _ptr(g), _ptr(b), _ptr(run_mean), _ptr(run_stat), int(bool(use_log_std)),
                                 float(decay), float(eps), int(bool(relu)), _ptr(y), _ptr(save), _ptr(save[C:]), _ptr(work),
                                 _ptr(pre_bias), rows, C, _stream())
        _check(rc, "dl4j_bn_fwd_train")
        global LAUNCHES
        LAUNCHES += 2
        ctx.relu, ctx.has_res, ctx.has_affine = bool(relu), res is not None, gamma is not None
        ctx.gb_refs = (gamma, beta)
        ctx.save_for_backward(x, y if (res is not None and relu) else None, save, work)
        return y

    @staticmethod
    def backward(ctx, dy):
        l = require()
        x, y, save, work = ctx.saved_tensors
        rows, C = _rows_c(x)
        dy = _dense_cl16(dy)
        dx = torch.empty_like(x)
        dres = torch.empty_like(x) if ctx.has_res else None
        # the kernel adds dgamma / dbeta to what its targets hold: the parameters' preallocated fp32 gradients when they have
        # them (nothing is returned then, so autograd launches no accumulation), else a zeroed scratch that is returned
        def target(p_):
            if p_ is not None and p_.is_leaf and p_.grad is not None and p_.grad.dtype == torch.float32 and p_.grad.is_contiguous() \
                    and p_.grad.numel() == C:
                return p_.grad
            return None
        gamma, beta = ctx.gb_refs
        tg, tb = (target(gamma), target(beta)) if ctx.has_affine else (None, None)
        dgb = None
        if ctx.has_affine and (tg is None or tb is None):
            dgb = torch.zeros(2 * C, dtype=torch.float32, device=x.device)
        pg = tg if tg is not None else (dgb[:C] if dgb is not None else None)
        pb = tb if tb is not None else (dgb[C:] if dgb is not None else None)
        rc = l.dl4j_bn_bwd(_ptr(dy), _ptr(x), _ptr(y), _ptr(save), _ptr(save[C:]), _ptr(work), _ptr(dx), _ptr(dres),
                           _ptr(pg), _ptr(pb), rows, C, int(ctx.relu), _stream())
        _check(rc, "dl4j_bn_bwd")
        global LAUNCHES
        LAUNCHES += 1
        dg = pg.reshape(gamma.shape) if (ctx.has_affine and tg is None and ctx.needs_input_grad[2]) else None
        db = pb.reshape(beta.shape) if (ctx.has_affine and tb is None and ctx.needs_input_grad[3]) else None
        return dx, dres, dg, db, None, None, None, None, None, None, None


def bn_supported(x):
    if not (available() and x.is_cuda and x.dtype == torch.bfloat16 and x.dim() in (2, 4)):
        return False
    rows, C = _rows_c(x)
    return rows > 0 and 8 <= C <= 2048 and (C & (C - 1)) == 0


def bn_act_train(x, res, gamma, beta, run_mean, run_stat, use_log_std, decay, eps, relu, pre_bias=None):
    """Fused training-mode batch norm; ``gamma`` / ``beta`` fp32 [C] (or None), running buffers fp32 [C] updated in place.
    ``pre_bias`` (fp32 [C]) is a bias that the producer left out of ``x``: it only enters the running mean."""
    pb = pre_bias.detach().float().reshape(-1).contiguous() if pre_bias is not None else None
    # gamma / beta go in as they are (any shape with C elements): a reshape would hide a parameter leaf and its gradient slice
    return _BnActFn.apply(x, res, gamma, beta, run_mean, run_stat, use_log_std, decay, eps, relu, pb)


def bn_act_eval(x, res, scale, shift, relu):
    """y = act(x * scale + shift [+ res]) with fp32 per-channel scale / shift (inference statistics folded in)."""
    l = require()
    x = _dense_cl16(x)
    res = _dense_cl16(res) if res is not None else None
    rows, C = _rows_c(x)
    y = torch.empty_like(x)
    rc = l.dl4j_bn_apply(_ptr(x), _ptr(res), _ptr(scale.float().contiguous()), _ptr(shift.float().contiguous()), int(bool(relu)), _ptr(y),
                         rows, C, _stream())
    _check(rc, "dl4j_bn_apply")
    return y


class _AddReluFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, a, b):
        l = require()
        a = _dense_cl16(a)
        b = _dense_cl16(b)
        if b.stride() != a.stride():
            b = b.contiguous(memory_format=torch.channels_last) if a.dim() == 4 else b.contiguous()
        y = torch.empty_like(a)
        rc = l.dl4j_add_relu(_ptr(a), _ptr(b), _ptr(y), a.numel(), _stream())
        _check(rc, "dl4j_add_relu")
        ctx.save_for_backward(y)
        return y

    @staticmethod
    def backward(ctx, dy):
        (y,) = ctx.saved_tensors
        g = dy * (y > 0).to(dy.dtype)
        return g, g


def add_relu(a, b):
    if not (available() and a.is_cuda and a.dtype == b.dtype == torch.bfloat16 and a.device == b.device and a.shape == b.shape and a.numel() % 8 == 0 and a.dim() in (2, 4)):
        return None
    return _AddReluFn.apply(a, b)


def attention(q, k, v, mask, scale, dropout_p=0.0, causal=False):
    return attention_native.attention(q, k, v, mask, scale, dropout_p, causal)


def attention_grad(q, k, v, mask, scale, dout, causal=False):
    return attention_native.attention_grad(q, k, v, mask, scale, dout, causal)


# =========================================================================== fused updater
_SEG_FMT = "<qqqqqfffiii"     # offset, block_start, block_numel, state_off, shadow_off, l1, l2, wd, kernel_id, hyper, pad
_CHUNK_FMT = "<qii"
_CHUNK = int(os.environ.get("DL4J_UPDATER_CHUNK", "16384"))     # most elements per block of the multi-segment updater launch


def _cfg_index(known, cfg):
    """Index of ``cfg`` among the distinct updater configurations seen so far (hyper-parameter sets are per
    configuration, not per state block)."""
    for i, c in enumerate(known):
        if c is cfg or c == cfg:
            return i
    known.append(cfg)
    return len(known) - 1


def _chunk_size(numel):
    """Elements per block of the updater launch: enough blocks for eight per SM, between one pass of a block's 256 threads (1024) and
    the measured best of large networks.  0.67 M parameters in 16384-element chunks were 41 blocks on 148 SMs: 34 us, now 7.7.
    The exchange kernels of a parallel group, which walk their chunks persistently, keep the large ones."""
    return max(1024, min(_CHUNK, numel // (8 * num_sms()) // 1024 * 1024))


def _build_tables(upd, shadow_offsets):
    """Static part of the segment / chunk tables for a MultiLayerUpdater; the chunk table for the exchange kernels and the one for the
    single-process launch."""
    segs = upd.segments(0, 0)
    block_ids = []
    seg_rows, chunks, small = [], [], []
    upd._seg_chunk0 = []                 # first chunk of every segment (bucketed gradient exchange addresses chunk ranges)
    size = _chunk_size(sum(sg[1] for sg in segs))
    for si, (off, numel, st_off, bn, bs, kid, lr, l1, l2, wd, cfg) in enumerate(segs):
        upd._seg_chunk0.append(len(chunks))
        hid = _cfg_index(block_ids, cfg)
        seg_rows.append([off, bs, bn, st_off, shadow_offsets[si] if shadow_offsets is not None else 0, l1, l2, wd, kid, hid, 0])
        for table, step in ((chunks, _CHUNK), (small, size)):
            for o in range(0, numel, step):
                table.append(struct.pack(_CHUNK_FMT, off + o, min(step, numel - o), si))
    upd._seg_chunk0.append(len(chunks))
    return seg_rows, b"".join(chunks), len(chunks), b"".join(small), len(small), len(block_ids)


def update_tables(upd, iteration, epoch, shadow_offsets=None):
    """Device chunk/segment tables + this iteration's hyper-parameter table for ``upd``; None if unsupported."""
    cache = getattr(upd, "_native_tables", None)
    if cache is None or cache["shadow"] is not shadow_offsets:
        seg_rows, chunk_bytes, n_chunks, small_bytes, n_small, n_hyper = _build_tables(upd, shadow_offsets)
        if n_hyper > 8:
            upd._native_tables = {"unsupported": True, "shadow": shadow_offsets}
            return None
        dev = upd.params.device
        chunks_t = torch.frombuffer(bytearray(chunk_bytes), dtype=torch.uint8).to(dev)
        small_t = torch.frombuffer(bytearray(small_bytes), dtype=torch.uint8).to(dev)
        cache = {"seg_rows": seg_rows, "chunks": chunks_t, "n_chunks": n_chunks, "small": small_t, "n_small": n_small, "n_hyper": n_hyper, "shadow": shadow_offsets,
                 "segs_dev": None, "segs_key": None}
        upd._native_tables = cache
    if cache.get("unsupported"):
        return None
    # dynamic part: per-block hyper-parameters and any scheduled regularisation coefficients
    segs = upd.segments(iteration, epoch)
    hyper = np.zeros((8, 8), dtype=np.float32)
    key = []
    seen = []
    for si, (off, numel, st_off, bn, bs, kid, lr, l1, l2, wd, cfg) in enumerate(segs):
        key.append((l1, l2, wd))
        hid = _cfg_index(seen, cfg)
        b1 = getattr(cfg, "beta1", 0.0); b2 = getattr(cfg, "beta2", 0.0); eps = getattr(cfg, "epsilon", 0.0)
        from ..nn.updaters import _eps_t, Nesterovs, AdaMax
        eps_t = 0.0
        if hasattr(cfg, "beta1"):
            eps_t = _eps_t(lr, b1, b2, iteration, eps, with_sqrt=not isinstance(cfg, AdaMax))
        mu = cfg.currentMomentum(iteration, epoch) if isinstance(cfg, Nesterovs) else 0.0
        rho = getattr(cfg, "rmsDecay", getattr(cfg, "rho", 0.0))
        mb1t = 1.0 - b1 ** (iteration + 1) if b1 else 1.0
        hyper[hid] = (lr, b1, b2, eps, eps_t, mb1t, mu, rho)
    key = tuple(key)
    if cache["segs_key"] != key:
        rows = cache["seg_rows"]
        buf = bytearray()
        for r, (l1, l2, wd) in zip(rows, key):
            buf += struct.pack(_SEG_FMT, r[0], r[1], r[2], r[3], r[4], l1, l2, wd, r[8], r[9], 0)
        cache["segs_dev"] = torch.frombuffer(buf, dtype=torch.uint8).to(upd.params.device)
        cache["segs_key"] = key
    cache["hyper"] = hyper
    return cache


def fused_update(upd, iteration, epoch, shadow=None, shadow_offsets=None, grad_scale=1.0, zero_grads=True, residual=None) -> bool:
    """One launch: regularisation + updater + params -= update (+ bf16 shadow refresh, + grad zeroing); with
    ``residual`` the update is accumulated into it instead and the parameters are left untouched."""
    l = require()
    if l is None:
        return False
    cache = update_tables(upd, iteration, epoch, shadow_offsets)
    if cache is None:
        return False
    hyper = cache["hyper"]
    state = upd.state
    hp = hyper.ctypes.data_as(ctypes.c_void_p)
    rc = l.dl4j_fused_update(_ptr(upd.params), _ptr(upd.grads), _ptr(state) if state.numel() else None, _ptr(shadow),
                             _ptr(residual), _ptr(cache["small"]), cache["n_small"], _ptr(cache["segs_dev"]), hp, cache["n_hyper"],
                             float(grad_scale), 1 if zero_grads else 0, _stream())
    _check(rc, "dl4j_fused_update")
    upd._fused_zeroes_grads = bool(zero_grads)
    return True


def cast_to_bf16(src_f32, dst_bf16):
    l = require()
    rc = l.dl4j_cast_f32_bf16(_ptr(src_f32), _ptr(dst_bf16), src_f32.numel(), _stream())
    _check(rc, "dl4j_cast_f32_bf16")


# =========================================================================== gradient codecs
def threshold_encode(x, tau, capacity=None, msg=None, residual=None):
    """Sparse threshold encode of fp32 ``x``; returns the int32 message.  The residual goes to ``residual`` (same size), or stays in
    ``x`` without one."""
    l = require()
    n = x.numel()
    capacity = int(capacity if capacity is not None else n)
    if msg is None:
        msg = torch.empty(4 + capacity, dtype=torch.int32, device=x.device)
    if residual is None:
        rc = l.dl4j_threshold_encode(_ptr(x), n, float(tau), _ptr(msg), capacity, _stream())
    else:
        rc = l.dl4j_threshold_encode_to(_ptr(x), _ptr(residual), n, float(tau), _ptr(msg), capacity, _stream())
    _check(rc, "dl4j_threshold_encode")
    return msg


def threshold_decode(msg, target, scale=1.0, atomics=False, capacity=None):
    l = require()
    capacity = int(capacity if capacity is not None else msg.numel() - 4)
    rc = l.dl4j_threshold_decode(_ptr(msg), capacity, _ptr(target), target.numel(), float(scale), 1 if atomics else 0, _stream())
    _check(rc, "dl4j_threshold_decode")
    return target


def bitmap_encode(x, tau, msg=None, residual=None):
    l = require()
    n = x.numel()
    if msg is None:
        msg = torch.empty(4 + (n + 15) // 16, dtype=torch.int32, device=x.device)
    rc = l.dl4j_bitmap_encode_to(_ptr(x), _ptr(x if residual is None else residual), n, float(tau), _ptr(msg), _stream())
    _check(rc, "dl4j_bitmap_encode")
    return msg


def bitmap_decode(msg, target, scale=1.0, out=None):
    """Adds the decoded steps to ``target`` in place, or writes the sum to ``out``."""
    l = require()
    out = target if out is None else out
    rc = l.dl4j_bitmap_decode_to(_ptr(msg), _ptr(target), _ptr(out), target.numel(), float(scale), _stream())
    _check(rc, "dl4j_bitmap_decode")
    return out


# =========================================================================== word2vec / t-SNE
def w2v_batch(syn0, syn1, syn1neg, neg_table, target, ng_starter, points, codes, context, alpha, random, ns_rounds, train_words=True):
    """One launch of the skip-gram (``context`` None) or CBOW output-layer update for a batch of examples, in place on the fp32
    tables.  ``target`` / ``ng_starter`` [B], ``points`` / ``codes`` [B, L] (-1 padded) or None, ``context`` [B, W] (-1 padded) or
    None, ``alpha`` fp32 [B] or [1], ``random`` int64 [B] or [1].  Returns False when the case is not covered."""
    l = lib()
    if l is None or not syn0.is_cuda or syn0.dtype != torch.float32 or not syn0.is_contiguous() or syn0.dim() != 2:
        return False
    for t in (syn1, syn1neg):
        if t is not None and (t.dtype != torch.float32 or not t.is_contiguous() or t.shape[1] != syn0.shape[1]):
            return False
    dev = syn0.device
    V, D = int(syn0.shape[0]), int(syn0.shape[1])
    if D > 4096:
        return False

    def i32(t):
        return None if t is None else t.to(device=dev, dtype=torch.int32).contiguous()
    target = i32(target.reshape(-1))
    B = int(target.numel())
    if B == 0:
        return True
    ng_starter = i32(ng_starter.reshape(-1)) if ng_starter is not None else None
    L = W = 0
    if points is not None and syn1 is not None:
        points = i32(points.reshape(B, -1))
        codes = codes.reshape(B, -1).to(device=dev, dtype=torch.int8).contiguous()
        L = int(points.shape[1])
    else:
        points = codes = None
    if context is not None:
        context = i32(context.reshape(B, -1))
        W = int(context.shape[1])
    neg_table = i32(neg_table.reshape(-1)) if neg_table is not None and neg_table.numel() else None
    alpha = alpha.to(device=dev, dtype=torch.float32).reshape(-1).contiguous()
    random = random.to(device=dev, dtype=torch.int64).reshape(-1).contiguous()
    if not hasattr(l.dl4j_w2v_batch, "_typed"):
        vp, i32c, i64c = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
        l.dl4j_w2v_batch.argtypes = [vp, vp, vp, vp, i64c, vp, vp, vp, vp, vp, vp, i32c, vp, i32c, i32c, i32c, i32c, i32c, i32c, i32c, i32c, vp]
        l.dl4j_w2v_batch.restype = ctypes.c_int
        l.dl4j_w2v_batch._typed = True
    rc = l.dl4j_w2v_batch(_ptr(syn0), _ptr(syn1), _ptr(syn1neg), _ptr(neg_table), 0 if neg_table is None else int(neg_table.numel()),
                          _ptr(target), _ptr(ng_starter), _ptr(points), _ptr(codes), _ptr(context), _ptr(alpha), int(alpha.numel()),
                          _ptr(random), int(random.numel()), B, L, W, D, V, int(ns_rounds), 1 if train_words else 0, _stream())
    _check(rc, "dl4j_w2v_batch")
    return True


def barnes_edge_forces(row_p, col_p, val_p, y):
    """Attractive t-SNE forces over a CSR matrix; ``y`` fp32 [N, D <= 8].  None when the case is not covered."""
    l = lib()
    if l is None or not y.is_cuda or y.dtype != torch.float32 or y.dim() != 2 or y.shape[1] > 8:
        return None
    N, D = int(y.shape[0]), int(y.shape[1])
    row_p = row_p.to(device=y.device, dtype=torch.int32).contiguous()
    col_p = col_p.to(device=y.device, dtype=torch.int32).contiguous()
    val_p = val_p.to(device=y.device, dtype=torch.float32).contiguous()
    y = y.contiguous()
    out = torch.empty_like(y)
    if not hasattr(l.dl4j_barnes_edge_forces, "_typed"):
        vp, i32c = ctypes.c_void_p, ctypes.c_int
        l.dl4j_barnes_edge_forces.argtypes = [vp, vp, vp, vp, vp, i32c, i32c, vp]
        l.dl4j_barnes_edge_forces.restype = ctypes.c_int
        l.dl4j_barnes_edge_forces._typed = True
    rc = l.dl4j_barnes_edge_forces(_ptr(row_p), _ptr(col_p), _ptr(val_p), _ptr(y), _ptr(out), N, D, _stream())
    _check(rc, "dl4j_barnes_edge_forces")
    return out


from . import attention_native  # noqa: E402  (it imports this module; a relative import inside the two calls above costs 1 us each time)
