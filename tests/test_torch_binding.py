"""The native form of the Python entry points (host/torch_binding.cpp) against the Python code that it stands in for: the
same results bit for bit, the same errors, and whatever it does not know is left to the Python code."""
import builtins
import ctypes
import importlib.util
import math
import os
import shutil
import sys
import threading

import pytest

from conftest import ROOT

torch = pytest.importorskip("torch")


@pytest.fixture
def native(pkg):
    pkg.lib()
    fn = pkg._load_native()
    assert type(fn).__name__ == "builtin_function_or_method", "the binding was not built"
    return fn


PKG_DIR = os.path.join(ROOT, "flash-attn-rtx5060_b200")


@pytest.fixture
def load_as(monkeypatch):
    """Imports the package a second time, under a name of its own."""
    def load(name, directory=PKG_DIR):
        spec = importlib.util.spec_from_file_location(name, os.path.join(directory, "__init__.py"),
                                                      submodule_search_locations=[directory])
        module = importlib.util.module_from_spec(spec)
        monkeypatch.setitem(sys.modules, name, module)
        spec.loader.exec_module(module)
        return module
    return load


def test_first_calls_of_two_threads(load_as, monkeypatch):
    """Two threads that load the native part at once, the second of them as late as it can be."""
    pkg = load_as("flash_attn_of_two_threads")
    both_here, first_done, arrivals = threading.Barrier(2), threading.Event(), []
    plain_import = builtins.__import__

    def slow_import(name, globals=None, locals=None, fromlist=(), level=0):
        module = plain_import(name, globals, locals, fromlist, level)
        if fromlist and "_torch_binding" in fromlist:
            arrivals.append(None)
            second = len(arrivals) == 2
            try:
                both_here.wait(timeout=1.0)
            except threading.BrokenBarrierError:
                pass  # the other thread is kept out meanwhile
            if second:
                first_done.wait(timeout=10.0)
        return module

    def load():
        pkg._load_native()
        first_done.set()
    monkeypatch.setattr(builtins, "__import__", slow_import)
    threads = [threading.Thread(target=load) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    with pytest.raises(ctypes.ArgumentError):  # (once loaded twice, it passed such arguments on to itself)
        pkg.lib().flash_forward_noalloc(object(), 16, 16, 16, 1, 1, 1, 63, 0.0, 0, -1, -1, None, 0, 0)


@pytest.fixture
def copies(load_as, native, tmp_path):
    """The package, a copy of it, and the package with another build of the library, in one process."""
    second = str(tmp_path / "second")
    shutil.copytree(PKG_DIR, second)
    other_build = str(tmp_path / "another_build.so")
    shutil.copy(os.path.join(PKG_DIR, "libflashfwd_b200.so"), other_build)
    packages = [load_as("flash_attn_first"), load_as("flash_attn_second", second), load_as("flash_attn_other_build")]
    packages[2].LIB_PATH = other_build
    for p in packages:
        p.lib()
    return packages


def test_noalloc_calls_the_library_that_its_package_loaded(copies):
    """(A failing call leaves its text in the library that ran.)"""
    faults = [(dict(q=None), b"null tensor"), (dict(head_dim=63), b"head_dim"), (dict(scale=math.nan), b"NaN")]
    for p, (fault, _) in zip(copies, faults):
        a = dict(q=16, k=16, v=16, o=16, batch=1, heads=1, seqlen=1, head_dim=64, scale=0.0) | fault
        assert p.lib().flash_forward_noalloc(*a.values(), 0, -1, -1, None, 0, 0) != p.FA_OK
    for p, (_, text) in zip(copies, faults):
        assert text in p.lib().flash_forward_last_error()


@pytest.mark.gpu
def test_attention_forward_calls_the_library_that_its_package_loaded(copies):
    x = torch.zeros(1, 1, 8, 64, device="cuda", dtype=torch.float16)
    y = torch.zeros(1, 1, 8, 32, device="cuda", dtype=torch.float16)
    faults = [(y, 0.0, "head_dim"), (x, math.nan, "NaN"), (x, 1e-35, "finite")]
    for p, (t, scale, text) in zip(copies, faults):
        with pytest.raises(p.FlashForwardError, match=text):
            p.attention_forward(t, t, t, softmax_scale=scale)
    for p, (_, _, text) in zip(copies, faults):
        assert text.encode() in p.lib().flash_forward_last_error()


def test_arguments_that_are_not_plain_go_to_ctypes(pkg, native):
    fn = pkg.lib().flash_forward_noalloc
    assert fn(0, None, 0, 0, 1, 1, 1, 64, 0.0, 0, -1, -1, None, 0, 0) == pkg.FA_INVALID_ARG
    assert b"null tensor" in pkg.lib().flash_forward_last_error()
    assert fn(ctypes.c_void_p(16), 16, 16, 16, 1, 1, 1, 63, 0, 0, -1, -1, None, 0, False) == pkg.FA_UNSUPPORTED
    assert fn(16, 16, 16, 16, 1, 1, 1, 64, 0.0, 0, -1, -1, None, 99, 0) == pkg.FA_INVALID_ARG
    with pytest.raises(TypeError):
        fn(1, 2, 3)
    with pytest.raises(ctypes.ArgumentError):
        fn(object(), 16, 16, 16, 1, 1, 1, 63, 0.0, 0, -1, -1, None, 0, 0)
    with pytest.raises(ctypes.ArgumentError):
        fn(16, 16, 16, 16, 1, 1, 1, 63.0, 0.0, 0, -1, -1, None, 0, 0)


def test_a_binding_built_against_another_torch_is_not_used(load_as, native, monkeypatch):
    p = load_as("flash_attn_another_torch")
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    with pytest.warns(UserWarning, match="0.0.1"):
        p.lib()
    assert p._load_native()(None) is NotImplemented
    assert type(p.lib().flash_forward_noalloc) is type(p.lib().flash_forward)


def test_noalloc_is_still_a_ctypes_function(load_as, native):
    p = load_as("flash_attn_ctypes_function")
    p.lib()
    p._load_native()
    fn, plain = p.lib().flash_forward_noalloc, p.lib().flash_forward
    bad = (None, 16, 16, 16, 1, 1, 1, 64, 0.0, 0, -1, -1, None, 0, 0)
    assert fn.argtypes == [*plain.argtypes, ctypes.c_int, ctypes.c_int] and fn.restype is ctypes.c_int
    assert fn.errcheck is None and fn.__name__ == "flash_forward_noalloc"
    assert ctypes.cast(fn, ctypes.c_void_p).value and isinstance(fn, ctypes._CFuncPtr)
    assert fn(*bad) == p.FA_INVALID_ARG
    fn.errcheck = lambda result, func, args: ("checked", result, func is fn, args[0])
    assert fn(*bad) == ("checked", p.FA_INVALID_ARG, True, None)
    del fn.errcheck
    fn.restype = lambda rc: -rc
    assert fn(*bad) == -p.FA_INVALID_ARG


def test_tensors_that_are_refused_stay_refused(pkg, native):
    q = torch.zeros(1, 2, 64, 64, dtype=torch.float16)
    with pytest.raises(AssertionError):
        pkg.attention_forward(q, q, q)
    assert native(q, q, q, False, -1, -1, 0.0, None, None, False, 0.0, 0) is NotImplemented
    assert native(q, q, q) is NotImplemented
    with pytest.raises(AttributeError):
        pkg.attention_forward(None, q, q)


class Tensor:
    """What the Python code asks of a tensor."""
    def __init__(self, shape=(1, 2, 64, 64), dtype=torch.float16, device=0, contiguous=True):
        self.shape, self.dtype, self.device, self.contiguous = shape, dtype, device, contiguous
        self.is_cuda = device >= 0
    dim = lambda self: len(self.shape)  # noqa: E731
    numel = lambda self: math.prod(self.shape)  # noqa: E731
    get_device = lambda self: self.device  # noqa: E731
    is_contiguous = lambda self: self.contiguous  # noqa: E731


ROOMY = (1, 2, 65, 64)
REFUSED = [dict(k=dict(device=-1)), dict(v=dict(device=-1)), dict(k=dict(device=1)), dict(v=dict(device=1)),
           dict(k=dict(dtype=torch.float32)), dict(v=dict(dtype=torch.bfloat16)), dict(v=dict(contiguous=False)),
           dict(out=dict(device=-1)), dict(out=dict(device=1)), dict(out=dict(shape=(1, 2, 63, 64))),
           dict(out=dict(contiguous=False)), dict(out=dict(dtype=torch.float32)), dict(out=dict(dtype=torch.bfloat16)),
           dict(alibi_slopes=dict(shape=(2,), dtype=torch.float32, contiguous=False)),
           dict(alibi_slopes=dict(shape=(2,), dtype=torch.float32, device=1)),
           dict(alibi_slopes=dict(shape=(2,), dtype=torch.float32, device=-1)),
           dict(alibi_slopes=dict(shape=(3,), dtype=torch.float32)), dict(alibi_slopes=dict(shape=(2,)))]
ACCEPTED = [dict(), dict(out=dict()), dict(out=dict(shape=(2, 64, 64))), dict(out=dict(shape=ROOMY)),
            dict(alibi_slopes=dict(shape=(2,), dtype=torch.float32)), dict(alibi_slopes=dict(shape=(2, 1), dtype=torch.float32))]


@pytest.mark.parametrize("operands,accepted", [(o, False) for o in REFUSED] + [(o, True) for o in ACCEPTED], ids=str)
def test_operands_that_the_kernel_could_not_take_are_refused(pkg, monkeypatch, operands, accepted):
    enqueued = []
    monkeypatch.setattr(pkg, "_native", lambda *a: NotImplemented)
    monkeypatch.setattr(pkg, "_enqueue_forward", lambda *a: enqueued.append(a))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch, "empty_like", lambda t: t)
    a = {n: Tensor(**operands.get(n, {})) for n in "qkv"}
    a |= {n: Tensor(**operands[n]) for n in ("out", "alibi_slopes") if n in operands}
    if accepted:
        pkg.attention_forward(**a)
    else:
        with pytest.raises(AssertionError):
            pkg.attention_forward(**a)
    assert len(enqueued) == accepted


def bind_to_counters():
    """The native part bound to entry points that only note their calls, so that nothing is launched: (forward, calls)."""
    from flash_attn_rtx5060_b200 import _torch_binding

    vp, i, f, u = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_ulonglong
    tensors, shape = [vp, vp, vp, vp], [i, i, i, i, f, i, i, i]
    signatures = dict(plain=tensors + shape + [vp], alibi=tensors + shape + [vp, vp], lse=tensors + [vp] + shape + [vp, vp],
                      dropout=tensors + shape + [vp, f, u, vp], noalloc=tensors + shape + [vp, i, i])
    calls = []
    note = [ctypes.CFUNCTYPE(i, *s)(lambda *a, n=n: calls.append((n, *a)) or 0) for n, s in signatures.items()]
    native, _ = _torch_binding.bind(*(ctypes.cast(f, vp).value for f in note), note[-1])
    return lambda *a, keep=note: native(*a), calls


@pytest.mark.gpu
@pytest.mark.parametrize("operands,accepted", [(o, False) for o in REFUSED] + [(o, True) for o in ACCEPTED], ids=str)
def test_the_native_part_leaves_such_operands_to_the_python_code(pkg, native, monkeypatch, operands, accepted):
    def tensor(shape=(1, 2, 64, 64), dtype=torch.float16, device=0, contiguous=True):
        if device >= torch.cuda.device_count():
            pytest.skip("one GPU")
        t = torch.zeros(*shape, 1 if contiguous else 2, dtype=dtype, device="cpu" if device < 0 else f"cuda:{device}")
        return t[..., 0]
    forward, calls = bind_to_counters()
    a = {n: tensor(**operands.get(n, {})) for n in "qkv"}
    a |= {n: tensor(**operands[n]) for n in ("out", "alibi_slopes") if n in operands}
    r = forward(a["q"], a["k"], a["v"], False, -1, -1, 0.0, a.get("out"), a.get("alibi_slopes"), False, 0.0, 0)
    assert (r is not NotImplemented) == accepted and len(calls) == accepted
    if accepted:
        assert calls[0][1:5] == (a["q"].data_ptr(), a["k"].data_ptr(), a["v"].data_ptr(), r.data_ptr())
    else:
        monkeypatch.setattr(pkg, "_native", forward)
        monkeypatch.setattr(pkg, "_enqueue_forward", None)
        with pytest.raises(AssertionError):
            pkg.attention_forward(**a)


@pytest.mark.gpu
def test_a_dropout_probability_below_the_range_of_a_float(pkg, native):
    """1e-50 is 0 as a float and still a probability: with the log-sum-exp refused, else the dropout entry point's."""
    forward, calls = bind_to_counters()
    q = torch.zeros(1, 2, 64, 64, device="cuda", dtype=torch.float16)
    assert forward(q, q, q, False, -1, -1, 0.0, None, None, True, 1e-50, 0) is NotImplemented
    assert forward(q, q, q, False, -1, -1, 0.0, None, None, False, 1e-50, 7) is not NotImplemented
    assert [c[0] for c in calls] == ["dropout"] and calls[0][14:16] == (0.0, 7)
    with pytest.raises(AssertionError):
        pkg.attention_forward(q, q, q, return_lse=True, dropout_p=1e-50)


FORMS = [dict(), dict(causal=True), dict(causal=1), dict(causal=True, window_left=40), dict(window_left=64, window_right=10),
         dict(softmax_scale=0.25), dict(softmax_scale=1), dict(alibi=True, causal=True), dict(return_lse=True),
         dict(return_lse=True, alibi=True), dict(dropout_p=0.3, seed=7), dict(dropout_p=0.3, seed=-1),
         dict(dropout_p=0.5, alibi=True, seed=1 << 63), dict(out=True), dict(out=True, return_lse=True)]


@pytest.mark.gpu
@pytest.mark.parametrize("d,n", [(64, 200), (128, 77)])
@pytest.mark.parametrize("form", FORMS, ids=str)
def test_same_bits_as_the_python_code(pkg, native, monkeypatch, d, n, form):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    q, k, v = (torch.randn(2, 3, n, d, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))

    def call():
        kw = dict(form)
        if kw.pop("alibi", False):
            kw["alibi_slopes"] = torch.tensor([0.5, 0.25, 0.125], device="cuda")
        given = torch.empty_like(q) if kw.pop("out", False) else None
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
            r = pkg.attention_forward(q, k, v, out=given, **kw)
            torch.cuda.current_stream().synchronize()
        r = r if isinstance(r, tuple) else (r,)
        assert given is None or r[0] is given
        return r
    fast = call()
    monkeypatch.setattr(pkg, "_native", lambda *a: NotImplemented)
    slow = call()
    assert len(fast) == len(slow)
    for a, b in zip(fast, slow):
        assert a.dtype == b.dtype and a.shape == b.shape and a.device == b.device and not a.requires_grad
        assert torch.equal(a.view(torch.int16 if a.dtype == torch.float16 else torch.int32),
                           b.view(torch.int16 if b.dtype == torch.float16 else torch.int32))


@pytest.mark.gpu
def test_errors_and_special_tensors(pkg, native):
    q = torch.randn(1, 2, 96, 64, device="cuda", dtype=torch.float16)
    for bad in (q.float(), q[0], q.transpose(1, 2), q[:, :, ::2]):
        with pytest.raises(AssertionError):
            pkg.attention_forward(bad, bad, bad)
    with pytest.raises(AssertionError):
        pkg.attention_forward(q, q[:, :1].contiguous(), q)
    with pytest.raises(AssertionError):
        pkg.attention_forward(q, q, q, alibi_slopes=torch.zeros(3, device="cuda"))
    with pytest.raises(AssertionError):
        pkg.attention_forward(q, q, q, dropout_p=0.1, return_lse=True)
    x = torch.randn(1, 2, 96, 32, device="cuda", dtype=torch.float16)
    with pytest.raises(pkg.FlashForwardError) as e:
        pkg.attention_forward(x, x, x)
    assert e.value.code == pkg.FA_UNSUPPORTED and "head_dim" in str(e.value)
    with pytest.raises(pkg.FlashForwardError):
        pkg.attention_forward(q, q, q, softmax_scale=float("nan"))
    want = pkg.attention_forward(q, q, q)
    # a parameter that requires a gradient, and a subclass
    p = torch.nn.Parameter(q.clone())
    assert torch.equal(pkg.attention_forward(p, p, p), want)

    class Sub(torch.Tensor):
        pass
    s = q.clone().as_subclass(Sub)
    assert torch.equal(pkg.attention_forward(s, s, s).as_subclass(torch.Tensor), want)
