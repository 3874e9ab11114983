"""ctypes binding of libflashfwd_b200.so, the B200 (sm_100a) attention-forward library.

The shared library is the product; this module only loads it and mirrors the reference's host
entry point for Python callers (tests, the benchmark). There is no fallback of any kind: if the
library is missing or fails to load, importing `lib()` raises, and every call goes to the CUDA
kernels.

The directory name contains a hyphen, so the package is imported by path (see `load_package`
in `__graft_entry__.py`) under the module name `flash_attn_rtx5060_b200`.

Reference interface mirrored here: run_flash_attention (src/flash_forward.h:593-612 of the
reference) and its call site (src/main.cu:99).
"""
import ctypes
import os
import sys
import threading
import warnings

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "libflashfwd_b200.so")

FA_OK, FA_INVALID_ARG, FA_UNSUPPORTED, FA_CUDA_ERROR, FA_DEVICE_TIMEOUT = range(5)
STATUS_NAMES = {0: "FA_OK", 1: "FA_INVALID_ARG", 2: "FA_UNSUPPORTED", 3: "FA_CUDA_ERROR", 4: "FA_DEVICE_TIMEOUT"}

# every symbol include/flash_forward_b200.h declares
EXPORTS = (
    "flash_forward",
    "flash_forward_ex",
    "flash_forward_alibi",
    "flash_forward_lse",
    "flash_forward_dropout",
    "flash_forward_dropout_keep_probability",
    "flash_forward_multi_gpu",
    "flash_forward_host",
    "flash_forward_host_workspace_bytes",
    "flash_forward_check",
    "flash_forward_noalloc",
    "flash_forward_noalloc_check",
    "run_flash_attention_c",
    "flash_forward_last_error",
    "flash_forward_flops",
    "flash_forward_kv_range",
    "flash_forward_head_group",
    "flash_forward_shutdown",
)

_lock = threading.RLock()  # around the first load of either
_lib = None
_native = None  # forward() of _torch_binding once looked for; answers NotImplemented where there is none


class FlashForwardError(RuntimeError):
    def __init__(self, code, message):
        super().__init__(f"{STATUS_NAMES.get(code, code)}: {message}")
        self.code = code


def lib():
    """Loads the shared library once. Raises OSError when it has not been built."""
    global _lib
    if _lib is None:
        with _lock:
            if _lib is None:
                _lib = _open()
        if "torch" in sys.modules:
            _load_native()
    return _lib


def _open():
    if not os.path.exists(LIB_PATH):
        raise OSError(f"{LIB_PATH} not found: build it with `make -C {os.path.join(_HERE, 'csrc')}`")
    L = ctypes.CDLL(LIB_PATH)
    vp, i, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    L.flash_forward.argtypes = [vp, vp, vp, vp, i, i, i, i, f, i, i, i, vp]
    L.flash_forward.restype = i
    L.flash_forward_alibi.argtypes = [vp, vp, vp, vp, i, i, i, i, f, i, i, i, vp, vp]
    L.flash_forward_alibi.restype = i
    L.flash_forward_lse.argtypes = [vp, vp, vp, vp, vp, i, i, i, i, f, i, i, i, vp, vp]
    L.flash_forward_lse.restype = i
    L.flash_forward_dropout.argtypes = [vp, vp, vp, vp, i, i, i, i, f, i, i, i, vp, f, ctypes.c_ulonglong, vp]
    L.flash_forward_dropout.restype = i
    L.flash_forward_dropout_keep_probability.argtypes = [f]
    L.flash_forward_dropout_keep_probability.restype = ctypes.c_double
    pp = ctypes.POINTER(vp)
    L.flash_forward_multi_gpu.argtypes = [i, ctypes.POINTER(i), pp, pp, pp, pp, ctypes.POINTER(i), i, i, f, i, i, i, pp, i]
    L.flash_forward_multi_gpu.restype = i
    L.flash_forward_ex.argtypes = [vp, vp, vp, vp, i, i, i, i, f, i, i, i, vp, i, i, vp]
    L.flash_forward_ex.restype = i
    L.flash_forward_host.argtypes = [vp, vp, vp, vp, i, i, i, i, f, i, i, i, vp, ctypes.c_size_t, i]
    L.flash_forward_host.restype = i
    L.flash_forward_host_workspace_bytes.argtypes = [i, i, i]
    L.flash_forward_host_workspace_bytes.restype = ctypes.c_size_t
    L.flash_forward_noalloc.argtypes = [vp, vp, vp, vp, i, i, i, i, f, i, i, i, vp, i, i]
    L.flash_forward_noalloc.restype = i
    L.flash_forward_noalloc_check.argtypes = [vp, i]
    L.flash_forward_noalloc_check.restype = i
    L.flash_forward_check.argtypes = [vp]
    L.flash_forward_check.restype = i
    L.run_flash_attention_c.argtypes = [i, i, i, i, vp, vp, vp, vp, vp, vp, i, i, i, i, i, vp, f, vp]
    L.run_flash_attention_c.restype = i
    L.flash_forward_last_error.argtypes = []
    L.flash_forward_last_error.restype = ctypes.c_char_p
    L.flash_forward_flops.argtypes = [i, i, i, i, i, i, i]
    L.flash_forward_flops.restype = ctypes.c_double
    ip = ctypes.POINTER(ctypes.c_int)
    L.flash_forward_kv_range.argtypes = [i, i, i, i, i, i, ip, ip, ip]
    L.flash_forward_kv_range.restype = i
    L.flash_forward_head_group.argtypes = [i, i, i, i, i, i, i]
    L.flash_forward_head_group.restype = i
    L.flash_forward_shutdown.argtypes = []
    L.flash_forward_shutdown.restype = i
    return L


def _load_native():
    """The native form of attention_forward (host/torch_binding.cpp), if it was built against the torch it is used with.
    Without it everything runs through ctypes, with the same results. With it the loaded library's flash_forward_noalloc is
    called without ctypes as well, where the arguments are plain numbers."""
    global _native
    L = lib()
    with _lock:
        if _native is not None:
            return _native
        try:
            import torch  # noqa: F401  (its libraries have to be loaded first)

            from . import _torch_binding
            built_against = getattr(_torch_binding, "torch_version", None)
            usable = built_against == str(torch.__version__)
            if not usable:
                warnings.warn(f"{_torch_binding.__file__} was built against torch {built_against}, not {torch.__version__}: "
                              "calls go through ctypes, 5 us slower, until `make` has built it again")
        except ImportError:
            usable = False
        if not usable:
            _native = lambda *args: NotImplemented  # noqa: E731
            return _native
        entry_points = (L.flash_forward, L.flash_forward_alibi, L.flash_forward_lse, L.flash_forward_dropout,
                        L.flash_forward_noalloc)
        _native, noalloc = _torch_binding.bind(*(ctypes.cast(fn, ctypes.c_void_p).value for fn in entry_points),
                                               L.flash_forward_noalloc)
        L.flash_forward_noalloc = _called_natively(L, L.flash_forward_noalloc, noalloc)
        return _native


def _called_natively(L, fn, native):
    """The ctypes function `fn` of L, except that `native` answers its calls, until its argtypes, restype or errcheck are set:
    from then on ctypes does, by what was set. A call costs 0.05 us more than `native` itself (0.21 -> 0.26 us for one that is
    refused; through ctypes 2.1)."""
    class NativelyCalled(type(fn)):
        _flags_, _restype_ = type(fn)._flags_, type(fn)._restype_

        def __setattr__(self, name, value):
            super().__setattr__(name, value)
            if name in ("argtypes", "restype", "errcheck") and "__call__" in vars(NativelyCalled):
                del NativelyCalled.__call__

    same = NativelyCalled((fn.__name__, L))
    same.__name__, same.argtypes, same.restype = fn.__name__, fn.argtypes, fn.restype
    NativelyCalled.__call__ = native
    return same


def _raise(code):
    raise FlashForwardError(code, lib().flash_forward_last_error().decode())


def flash_forward(q, k, v, o, batch, heads, seqlen, head_dim, softmax_scale=0.0, is_causal=False, window_left=-1,
                  window_right=-1, stream=None, kernel=0, variant=0, dbg=None):
    """Enqueues the attention forward on raw device pointers (ints). Asynchronous."""
    rc = lib().flash_forward_ex(q, k, v, o, batch, heads, seqlen, head_dim, softmax_scale, int(bool(is_causal)),
                                window_left, window_right, stream, kernel, variant, dbg)
    if rc != FA_OK:
        _raise(rc)


def flash_forward_multi_gpu(devices, q, k, v, o, slab_heads, seqlen, head_dim, softmax_scale=0.0, is_causal=False,
                            window_left=-1, window_right=-1, streams=None, wait=True):
    """One slab of heads per entry of `devices`; q, k, v, o are lists of raw device pointers (ints)."""
    n = len(devices)
    assert len(q) == len(k) == len(v) == len(o) == len(slab_heads) == n
    ints = lambda xs: (ctypes.c_int * n)(*xs)  # noqa: E731
    ptrs = lambda xs: (ctypes.c_void_p * n)(*xs)  # noqa: E731
    rc = lib().flash_forward_multi_gpu(n, ints(devices), ptrs(q), ptrs(k), ptrs(v), ptrs(o), ints(slab_heads), seqlen,
                                       head_dim, softmax_scale, int(bool(is_causal)), window_left, window_right,
                                       None if streams is None else ptrs(streams), int(bool(wait)))
    if rc != FA_OK:
        _raise(rc)


def flash_forward_host(q_host, k_host, v_host, o_host, batch, heads, seqlen, head_dim, workspace, workspace_bytes,
                       chunk_heads, softmax_scale=0.0, is_causal=False, window_left=-1, window_right=-1):
    """Forward on HOST buffers (raw pointers): chunked upload / kernel / download pipeline. Blocking."""
    rc = lib().flash_forward_host(q_host, k_host, v_host, o_host, batch, heads, seqlen, head_dim, softmax_scale,
                                  int(bool(is_causal)), window_left, window_right, workspace, workspace_bytes,
                                  chunk_heads)
    if rc != FA_OK:
        _raise(rc)


def host_workspace_bytes(seqlen, head_dim, chunk_heads):
    return lib().flash_forward_host_workspace_bytes(seqlen, head_dim, chunk_heads)


def check(stream=None):
    """Waits for the stream and raises if a device-side wait gave up."""
    rc = lib().flash_forward_check(stream)
    if rc != FA_OK:
        _raise(rc)


def flops(batch, heads, seqlen, head_dim, is_causal=False, window_left=-1, window_right=-1):
    return lib().flash_forward_flops(batch, heads, seqlen, head_dim, int(bool(is_causal)), window_left, window_right)


def kv_range(seqlen, is_causal, window_left, window_right, row_begin, row_end):
    """(tile_begin, tile_end, masked_tiles) of the kv tiles a block of query rows reads."""
    a, b, c = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    rc = lib().flash_forward_kv_range(seqlen, int(bool(is_causal)), window_left, window_right, row_begin, row_end,
                                      ctypes.byref(a), ctypes.byref(b), ctypes.byref(c))
    if rc != FA_OK:
        _raise(rc)
    return a.value, b.value, c.value


def head_group(batch_heads, seqlen, head_dim, is_causal=False, window_left=-1, window_right=-1, num_sms=148):
    """Heads per scheduling group the default kernel uses for this shape (host logic)."""
    return lib().flash_forward_head_group(batch_heads, seqlen, head_dim, int(bool(is_causal)), window_left, window_right,
                                          num_sms)


def run_flash_attention(B, N, S, d, Q, K, V, O, L=None, M=None, Is_dropout=False, Is_causal=False, Is_local=False,
                        Has_alibi=False, window_size=0, alibi_slopes=None, dropout_prob=0.0, states=None):
    """The reference's entry point, argument for argument (N = heads, S = sequence length there).

    Q, K, V, O are raw device pointers. Blocks until the result is ready and prints `TIME: <ms>`
    as the reference does. Raises FlashForwardError where the reference would exit or abort.
    """
    rc = lib().run_flash_attention_c(B, N, S, d, Q, K, V, O, L, M, int(bool(Is_dropout)), int(bool(Is_causal)),
                                     int(bool(Is_local)), int(bool(Has_alibi)), window_size, alibi_slopes,
                                     dropout_prob, states)
    if rc != FA_OK:
        _raise(rc)


def attention_forward(q, k, v, causal=False, window_left=-1, window_right=-1, softmax_scale=0.0, out=None, kernel=0,
                      variant=0, alibi_slopes=None, return_lse=False, dropout_p=0.0, seed=0):
    """Convenience wrapper for torch CUDA tensors of shape [B, H, N, d], fp16, contiguous, on one device.

    `out`, if given, is written as [B, H, N, d] from its beginning, so its own shape does not matter as long as it is
    contiguous and large enough. alibi_slopes: float32, one per head. Other operands raise an AssertionError.
    torch is used for device memory and the current stream only; the computation is the library's.
    With return_lse the result is (out, lse), lse a float32 [B, H, N] tensor (flash_forward_lse).
    With dropout_p > 0 the call is flash_forward_dropout(dropout_p, seed).
    """
    if kernel == 0 and variant == 0:
        r = (_native or _load_native())(q, k, v, causal, window_left, window_right, softmax_scale, out, alibi_slopes,
                                        return_lse, dropout_p, seed)
        if r is not NotImplemented:
            if type(r) is int:
                _raise(r)
            return r
    import torch

    _check_operands(torch, q, k, v, out, alibi_slopes)
    if out is None:
        out = torch.empty_like(q)
    args = (torch, q, k, v, out, causal, window_left, window_right, softmax_scale, kernel, variant, alibi_slopes,
            return_lse, dropout_p, seed)
    device = q.get_device()
    if device == torch.cuda.current_device():
        return _enqueue_forward(device, *args)
    with torch.cuda.device(device):
        return _enqueue_forward(device, *args)


def _check_operands(torch, q, k, v, out, alibi_slopes):
    """The kernels get bare addresses: a tensor elsewhere, smaller or laid out otherwise would be read or written out of
    bounds. Raised here and not asserted, so that it holds under `python -O` too."""
    def fits(t, dtype):
        return t.is_cuda and t.get_device() == q.get_device() and t.dtype == dtype and t.is_contiguous()
    half = torch.float16
    if not (q.is_cuda and q.dim() == 4 and fits(q, half)):
        raise AssertionError("q: a contiguous fp16 CUDA tensor [B, H, N, d] is needed")
    if not (k.shape == q.shape and v.shape == q.shape and fits(k, half) and fits(v, half)):
        raise AssertionError("k and v have to be like q, on its device")
    if out is not None and not (fits(out, half) and out.numel() >= q.numel()):
        raise AssertionError("out: a contiguous fp16 tensor on q's device with room for the result is needed")
    if alibi_slopes is not None and not (fits(alibi_slopes, torch.float32) and alibi_slopes.numel() == q.shape[1]):
        raise AssertionError("alibi_slopes: a contiguous float32 tensor on q's device, one slope per head, is needed")


def _current_raw_stream(torch, device):
    """Handle of the current stream. Building a torch.cuda.Stream object and entering a device context for every call
    cost 5 us of the 14 us a call took on the host, more than the kernel of a small call (B1 H4 N512 d64), so the handle
    comes from the accessor that torch's own generated code uses; it is not public API, hence the second way."""
    raw = getattr(torch._C, "_cuda_getCurrentRawStream", None)
    return raw(device) if raw is not None else torch.cuda.current_stream(device).cuda_stream


def _enqueue_forward(device, torch, q, k, v, out, causal, window_left, window_right, softmax_scale, kernel, variant,
                     alibi_slopes, return_lse, dropout_p, seed):
    stream = _current_raw_stream(torch, device)
    B, H, N, d = q.shape
    L = lib()
    lse = None
    if dropout_p > 0.0:
        assert kernel == 0 and variant == 0 and not return_lse
        rc = L.flash_forward_dropout(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), B, H, N, d, softmax_scale,
                                     int(bool(causal)), window_left, window_right,
                                     None if alibi_slopes is None else alibi_slopes.data_ptr(), dropout_p, seed, stream)
    elif return_lse:
        assert kernel == 0 and variant == 0
        lse = torch.empty((B, H, N), device=q.device, dtype=torch.float32)
        rc = L.flash_forward_lse(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), B, H, N, d,
                                 softmax_scale, int(bool(causal)), window_left, window_right,
                                 None if alibi_slopes is None else alibi_slopes.data_ptr(), stream)
    elif alibi_slopes is not None:
        rc = L.flash_forward_alibi(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), B, H, N, d, softmax_scale,
                                   int(bool(causal)), window_left, window_right, alibi_slopes.data_ptr(), stream)
    else:
        rc = L.flash_forward_ex(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), B, H, N, d, softmax_scale,
                                int(bool(causal)), window_left, window_right, stream, kernel, variant, None)
    if rc != FA_OK:
        _raise(rc)
    return (out, lse) if return_lse else out
