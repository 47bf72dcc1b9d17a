"""The operators' native host side (csrc/host_calls.cc) against the Python wrappers' own path: the same bits, the same refusals,
on any stream and from several threads."""
import glob
import importlib.util
import os
import shutil
import subprocess
import sys
import threading

import pytest
import torch

from tests.helpers import gaussian

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ac4k_kernel_b200")
MODULES = ("quant", "linear", "attention", "rope_3d")


@pytest.fixture
def both_paths(monkeypatch):
    """run(fn): the results of fn() through the native host side and through the wrappers' own path, each a value or the
    type of what it raised"""
    import ac4k_kernel_b200.ops  # noqa: F401
    from ac4k_kernel_b200.native import host_calls
    if host_calls is None:
        pytest.skip("the native host side is not built")

    def run(fn):
        res = []
        for calls in (host_calls, None):
            for m in MODULES:
                monkeypatch.setattr(sys.modules[f"ac4k_kernel_b200.ops.{m}"], "host_calls", calls)
            try:
                res.append(fn())
            except Exception as e:
                res.append(type(e))
        return res
    return run


@pytest.mark.parametrize("path", glob.glob(os.path.join(PKG, "native", "*.so")), ids=os.path.basename)
def test_modules_use_the_shared_libstdcxx(path):
    """A module with a libstdc++ of its own ends the process when an error message with a number in it is formatted."""
    if shutil.which("readelf") is None:
        pytest.skip("no readelf")
    needed = subprocess.run(["readelf", "-d", path], capture_output=True, text=True, check=True).stdout
    assert "libstdc++.so.6" in needed


def test_the_library_builds_without_torch(monkeypatch, capsys):
    spec = importlib.util.spec_from_file_location("build_without_torch", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    monkeypatch.setattr(build, "build", lambda **_: "the library")
    monkeypatch.setitem(sys.modules, "torch", None)
    build.main([])
    printed = capsys.readouterr()
    assert printed.out == "the library\n" and "torch is not installed" in printed.err


@pytest.mark.parametrize("error,said", [(ModuleNotFoundError("none"), "is not built"), (ImportError("undefined symbol: x"), "does not load")])
def test_a_missing_module_is_said(monkeypatch, error, said):
    """Everything works without it, at several times the host time: not silently"""
    import ac4k_kernel_b200.native as native

    class Finder:
        @staticmethod
        def find_spec(name, path=None, target=None):
            if name.endswith("_host_calls"):
                raise error
    spec = importlib.util.spec_from_file_location("without_host_calls", native.__file__, submodule_search_locations=[])
    module = importlib.util.module_from_spec(spec)
    monkeypatch.setitem(sys.modules, "without_host_calls", module)
    monkeypatch.setattr(sys, "meta_path", [Finder, *sys.meta_path])
    with pytest.warns(RuntimeWarning, match=said):
        spec.loader.exec_module(module)
    assert module.host_calls is None


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(max_scale=-1.0), dict(max_scale=0), dict(max_scale=-5)])
def test_refused_by_the_library(both_paths, kw):
    from ac4k_kernel_b200 import ops
    x = gaussian((64, 128), seed=1).cuda()
    assert both_paths(lambda: ops.quantize(x, 0, 1, **kw)) == [RuntimeError, RuntimeError]
    with pytest.raises(RuntimeError, match=r"code -2\): max_scale must be positive"):
        ops.quantize(x, 0, 1, **kw)


@pytest.mark.gpu
def test_options_are_left_to_the_wrappers(both_paths):
    """What the wrappers accept or refuse with an error of their own: options of other types than the usual ones"""
    from ac4k_kernel_b200 import ops
    x, q = gaussian((64, 128), seed=1).cuda(), gaussian((1, 20, 2, 64), seed=2).cuda()
    w = ops.quantize(x, 0, 1)

    def same(fn):
        native, python = both_paths(fn)
        assert isinstance(native, tuple) and len(native) == len(python)
        assert all(torch.equal(a.view(torch.uint8) if a.dtype == torch.float8_e4m3fn else a,
                               b.view(torch.uint8) if b.dtype == torch.float8_e4m3fn else b) for a, b in zip(native, python))
    for precision in ("int8", "fp8e4m3"):
        same(lambda: ops.quantize(x, 0, 1, precision=precision, sf_layout=None))
    same(lambda: ops.quantize(x, 0, 1, swizzle=1))
    same(lambda: ops.quantize(x, True, False, precision="int8"))
    same(lambda: ops.quantize(x, 0, 1, max_scale=torch.tensor(100.0)))
    for fn, error in ((lambda: ops.quantize(x, 0, 1, precision=None), AssertionError),
                      (lambda: ops.quantize(x, 0, 1, sf_layout=None), AssertionError),
                      (lambda: ops.quantize(x, None, 1), TypeError),
                      (lambda: ops.quantize(x, 2 ** 70, 1), None),
                      (lambda: ops.quantize(x, 0, 1, precision="fp8e4m3", swizzle=None), TypeError),
                      (lambda: ops.attention(q, q, q, layout=None), AssertionError),
                      (lambda: ops.attention(q, q, q, precision=1), AssertionError),
                      (lambda: ops.linear_requant(*w, *w, w[2], sf_layout=None), ValueError)):
        native, python = both_paths(fn)
        assert native is python and issubclass(native, Exception) and error in (None, native)


def _bytes(v):
    """results as a list of byte tensors"""
    out = []
    for t in v if isinstance(v, tuple) else (v,):
        assert isinstance(t, torch.Tensor), t
        out.append((t.shape, t.stride(), t.dtype, t.contiguous().reshape(-1).view(torch.uint8)))
    return out


def _same(a, b):
    a, b = _bytes(a), _bytes(b)
    return len(a) == len(b) and all(x[:3] == y[:3] and torch.equal(x[3], y[3]) for x, y in zip(a, b))


def _offset(t):
    """the same values one element behind a 256-byte boundary"""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,cross,reduce", [((20, 256), 0, 1), ((300, 4104), 0, 1), ((3, 70, 1000), 1, 2), ((2, 130, 3, 80), 3, 1), ((2, 33, 3, 65), -1, -3),
                                                ((2, 2, 50, 64), -2, -1), ((64, 96), 1, 0), ((1, 1024, 1, 130), 3, 1)])
def test_quantize_same_bits(both_paths, shape, cross, reduce):
    """every precision and option; also on a tensor that is not 16-byte aligned"""
    from ac4k_kernel_b200 import ops
    x = gaussian(shape, seed=sum(shape)).cuda()
    for kw in (dict(), dict(sf_layout="128x4"), dict(swizzle=True), dict(max_scale=1000), dict(max_scale=0.1), dict(precision="fp8e4m3"),
               dict(precision="fp8e4m3", swizzle=True, max_scale=2.25), dict(precision="fp8e4m3", max_scale=100), dict(precision="int8"),
               dict(precision="int8", max_scale=100), dict(precision="int8", max_scale=-5), dict(precision="int8", max_scale=12.0)):
        native, python = both_paths(lambda: ops.quantize(x, cross, reduce, **kw))
        assert _same(native, python), kw
        assert all(_same(v, python) for v in both_paths(lambda: ops.quantize(_offset(x), cross, reduce, **kw))), kw


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["ac4k", "128x4"])
@pytest.mark.parametrize("m", [1, 37, 100, 300])
def test_linear_same_bits(both_paths, m, layout):
    from ac4k_kernel_b200 import ops
    n, k = 192, 528
    a, w = ops.quantize(gaussian((m, k), seed=m).cuda(), 0, 1, sf_layout=layout), ops.quantize(gaussian((n, k), seed=1).cuda(), 0, 1, sf_layout=layout)
    gs = torch.tensor(0.01, device="cuda")
    for dtype in (torch.bfloat16, torch.float16, torch.float32):
        bias = gaussian((n,), seed=2).to(dtype).cuda()
        for b in (None, bias, bias.view(1, n)):
            assert _same(*both_paths(lambda: ops.linear(*a, *w, bias=b)))
            out = torch.empty((m, n), dtype=dtype, device="cuda")

            def given():
                out.fill_(float("nan"))
                assert ops.linear(*a, *w, b, out) is out
                return out.clone()
            assert _same(*both_paths(given))
            for out_layout in ("ac4k", "128x4"):
                assert _same(*both_paths(lambda: ops.linear_requant(*a, *w, gs, bias=b, sf_layout=out_layout)))


@pytest.mark.gpu
@pytest.mark.parametrize("n,d", [(3, 128), (2, 20), (1, 1032)])
def test_rope_same_bits(both_paths, n, d):
    from ac4k_kernel_b200 import ops
    from oracle import emulation as E
    x, freqs = gaussian((2, 24, n, d), seed=d).cuda(), E.rope_params_ref(8, d).cuda()
    grid = torch.tensor([[2, 3, 4], [1, 2, 3]], dtype=torch.int32, device="cuda")
    out = torch.empty_like(x)

    def given():
        out.zero_()
        assert ops.rope3d(x, grid, freqs, out) is out
        return out.clone()
    results = [*both_paths(lambda: ops.rope3d(x, grid, freqs)), *both_paths(given), *both_paths(lambda: ops.rope3d(_offset(x), grid, freqs))]
    assert all(_same(results[0], r) for r in results)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["nvfp4", "int8+fp8e4m3"])
@pytest.mark.parametrize("nq,nkv,d,dv", [(70, 70, 80, 80), (1, 200, 128, 64), (130, 515, 65, 33)])
def test_attention_same_bits(both_paths, nq, nkv, d, dv, precision):
    """head dimensions that differ, rows that are not 16-byte aligned; the INT8 path also takes q and k that are not contiguous"""
    from ac4k_kernel_b200 import ops
    q, k, v = gaussian((2, nq, 3, d), seed=1).cuda(), gaussian((2, nkv, 3, d), seed=2).cuda(), gaussian((2, nkv, 3, dv), seed=3).cuda()
    native, python = both_paths(lambda: ops.attention(q, k, v, precision=precision))
    assert _same(native, python) and not bool(torch.isnan(native.float()).any())
    assert all(_same(r, python) for r in both_paths(lambda: ops.attention(_offset(q), _offset(k), _offset(v), precision=precision)))
    t = [x.transpose(1, 2).contiguous() for x in (q, k, v)]
    buf = torch.empty((2, 3, nq + 1, dv + 3), dtype=torch.bfloat16, device="cuda")[:, :, 1:, 3:]      # rows at odd offsets

    def given():
        buf.zero_()
        assert ops.attention(*t, layout="BHND", precision=precision, out=buf) is buf
        return buf.clone()
    for r in (*both_paths(lambda: ops.attention(*t, layout="BHND", precision=precision)), *both_paths(given)):
        assert torch.equal(r, python.transpose(1, 2))
    strided = [x.transpose(1, 2) for x in t[:2]]
    results = both_paths(lambda: ops.attention(*strided, v, precision=precision))
    assert results == [RuntimeError, RuntimeError] if precision == "nvfp4" else all(torch.equal(r, python) for r in results)
    if precision != "nvfp4":
        shared = k[:, :, :1].expand(-1, -1, 3, -1)                       # one key head for three query heads: a stride of 0
        native, python = both_paths(lambda: ops.attention(q, shared, v, precision=precision))
        assert _same(native, python) and _same(native, ops.attention(q, shared.contiguous(), v, precision=precision))


@pytest.mark.gpu
@pytest.mark.parametrize("n,d", [(1024, 128), (1000, 65), (515, 96), (100, 128)])
def test_attention_takes_one_mean(both_paths, n, d):
    """The keys' mean is a sum in fp32 that is rounded to bf16: of this many means, sums in two orders round some differently"""
    from ac4k_kernel_b200 import ops
    for seed in range(4):
        k = (gaussian((4, n, 40, d), seed=seed).float() * 2 + 3).bfloat16().cuda()
        q, v = gaussian((4, 64, 40, d), seed=seed + 10).cuda(), gaussian((4, n, 40, d), seed=seed + 20).cuda()
        assert _same(*both_paths(lambda: ops.attention(q, k, v)))
        turned = [t.transpose(1, 2).contiguous() for t in (q, k, v)]
        assert _same(*both_paths(lambda: ops.attention(*turned, layout="BHND")))
        assert _same(*both_paths(lambda: ops.attention(q[:, :, :1].expand(-1, -1, 40, -1), k[..., :1].expand(-1, -1, -1, d), v)))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,cross,reduce,swizzle", [((50, 8192), 0, 1, False), ((666, 4096), 0, 1, False), ((2049, 4096), 0, 1, False), ((16, 8192), 0, 1, False),
                                                        ((2, 100, 3, 128), 3, 1, True), ((2, 33, 3, 65), 3, 1, True), ((4100, 4096), 0, 1, False)])
def test_dynamic_entry_with_and_without_scratch(shape, cross, reduce, swizzle):
    """ac4k_quantize_nvfp4_dynamic called as from C: scratch may be NULL at any size"""
    from ac4k_kernel_b200 import _cuda_ops as ct
    from ac4k_kernel_b200 import ops
    x = gaussian(shape, seed=4).cuda()
    want = ops.quant.Ac4kQuantizeOp()(x, cross, reduce, swizzle=swizzle)
    size, stride, _ = ct._view4(x, cross, reduce)
    scratch = torch.full((1024,), -1, dtype=torch.int32, device="cuda")
    for s in (None, scratch.data_ptr()):
        q, sf, g = torch.empty_like(want[0]), torch.empty_like(want[1]), torch.empty((), device="cuda")
        rc = ct.LIB.ac4k_quantize_nvfp4_dynamic(q.data_ptr(), sf.data_ptr(), g.data_ptr(), s, x.data_ptr(), 2688.0, ct._I64x4(*size),
                                                ct._I64x4(*stride), int(swizzle), 0, torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and _same((q, sf, g), want)


def _every_operator(i):
    """a call of every operator on inputs of its own; returns the results in one tuple"""
    from ac4k_kernel_b200 import ops
    from oracle import emulation as E
    x, w = gaussian((50 + 300 * (i % 2), 1024), seed=i).cuda(), gaussian((512, 1024), seed=i + 50).cuda()
    q, k, v = (gaussian((1, 200 + 30 * i, 2, 64), seed=i + j).cuda() for j in (100, 200, 300))
    grid, freqs = torch.tensor([[q.shape[1], 1, 1]], dtype=torch.int32, device="cuda"), E.rope_params_ref(512, 64).cuda()
    torch.cuda.synchronize()

    def run():
        a, b = ops.quantize(x * 1.5, 0, 1), ops.quantize(w, 0, 1)          # (the inputs are made on the stream as well)
        y = ops.linear(*a, *b)
        turned = ops.rope3d(q + k, grid, freqs)
        return (*a, *b, y, *ops.quantize(y, 0, 1, precision="int8"), *ops.quantize(y, 0, 1, precision="fp8e4m3"), turned,
                ops.attention(turned, k, v), ops.attention(turned, k, v, precision="nvfp4"))
    return run


@pytest.mark.gpu
def test_side_streams():
    """Operators on two streams at once, behind work of those streams: as on the default stream"""
    from ac4k_kernel_b200 import _lib
    runs = [_every_operator(i) for i in range(4)]
    want = [r() for r in runs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = {}
    busy = torch.randn((4096, 4096), device="cuda")
    for _ in range(5):
        for i, r in enumerate(runs):
            with torch.cuda.stream(streams[i % 2]):
                torch.mm(busy, busy)                                     # the host is ahead of the stream
                got[i] = r()
        torch.cuda.synchronize()
        assert all(_same(got[i], want[i]) for i in range(4))
    assert _lib.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("i", [0, 1])
def test_captured_operators(i):
    """every operator in one graph, replayed over results of its own that are cleared in between"""
    run = _every_operator(i)
    want = run()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = run()
    for _ in range(3):
        for r in got:
            r.view(torch.uint8).fill_(0x55) if r.dim() else r.fill_(7.0)
        g.replay()
        torch.cuda.synchronize()
        assert _same(got, want)


@pytest.mark.gpu
def test_several_threads():
    """Three host threads, each with a stream of its own (the native calls run without the interpreter lock)"""
    from ac4k_kernel_b200 import _lib
    runs = [_every_operator(i) for i in range(3)]
    want = [r() for r in runs]
    torch.cuda.synchronize()
    failed = []

    def thread(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(30):
                    got = runs[i]()
                    torch.cuda.current_stream().synchronize()
                    assert _same(got, want[i])
        except BaseException as e:
            failed.append((i, repr(e)))
    threads = [threading.Thread(target=thread, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not failed and not any(t.is_alive() for t in threads), failed
    assert _lib.device_status() == 0


class Sub(torch.Tensor):
    pass


@pytest.mark.gpu
def test_subclasses_are_left_to_the_wrappers(both_paths):
    """A subclass without a dispatch of its own: results are of the type that the wrappers make them (empty_like for RoPE)"""
    from ac4k_kernel_b200 import ops
    x, q = gaussian((64, 128), seed=1).cuda(), gaussian((1, 24, 2, 64), seed=2).cuda()
    w, bias = ops.quantize(x, 0, 1), gaussian((64,), seed=3).cuda()
    grid, freqs = torch.tensor([[2, 3, 4]], dtype=torch.int32, device="cuda"), torch.zeros((8, 32), dtype=torch.complex128, device="cuda")

    def sub(t):
        return t.as_subclass(Sub)
    for fn in (lambda: ops.rope3d(sub(q), grid, freqs), lambda: ops.rope3d(q, sub(grid), freqs), lambda: ops.rope3d(q, grid, freqs, sub(q.clone())),
               lambda: ops.attention(sub(q), q, q), lambda: ops.attention(q, q, sub(q), precision="nvfp4"),
               lambda: ops.quantize(sub(x), 0, 1)[0], lambda: ops.quantize(sub(x), 0, 1, precision="int8")[0],
               lambda: ops.linear(*w, *w, bias=sub(bias)), lambda: ops.linear(*w, *w, out=sub(torch.empty((64, 64), device="cuda"))),
               lambda: ops.linear_requant(*w, *w, sub(w[2]))[2]):
        native, python = both_paths(fn)
        assert type(native) is type(python) and torch.equal(native.as_subclass(torch.Tensor), python.as_subclass(torch.Tensor))
    assert type(ops.quantize(torch.nn.Parameter(x), 0, 1)[0]) is torch.Tensor


def _empties(fn, listener):
    """how many uninitialised tensors the listener saw fn() make"""
    if listener == "dispatch mode":
        from torch.utils._python_dispatch import TorchDispatchMode
        seen = []

        class Mode(TorchDispatchMode):
            def __torch_dispatch__(self, func, types, args=(), kwargs=None):
                seen.append(str(func))
                return func(*args, **(kwargs or {}))
        with Mode():
            fn()
        return sum(name.startswith("aten.empty") for name in seen)
    if listener == "profiler":
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as p:
            fn()
        return sum(e.count for e in p.key_averages() if e.key == "aten::empty")
    x = torch.zeros(4, device="cuda")
    if listener == "tracer":
        graph = torch.jit.trace(lambda t: (fn()[0], t), x, check_trace=False).graph
        return str(graph).count("aten::empty")
    from torch.fx.experimental.proxy_tensor import make_fx
    return make_fx(lambda t: (fn()[0], t))(x).code.count("aten.empty")


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("listener,least", [("dispatch mode", 3), ("profiler", 3), ("tracer", 1), ("make_fx", 1)])
def test_outputs_are_made_where_listeners_see_them(listener, least):
    """The native host side takes its outputs straight from the allocator's factory only where nothing listens to operator calls"""
    from ac4k_kernel_b200 import ops
    from ac4k_kernel_b200.native import host_calls
    assert host_calls is not None
    x = gaussian((20, 256), seed=1).cuda()
    assert _empties(lambda: ops.quantize(x, 0, 1), listener) >= least


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore")
def test_under_modes_and_transforms_as_the_wrappers(both_paths):
    """the same results, the same kind of tensor, or an error on both paths"""
    from ac4k_kernel_b200 import ops
    x = gaussian((20, 256), seed=1).cuda()
    q = gaussian((1, 70, 2, 64), seed=2).cuda()
    ones = torch.ones(3, device="cuda")

    def all_ops():
        return (*ops.quantize(x, 0, 1), *ops.quantize(x, 0, 1, precision="int8"), ops.attention(q, q, q), ops.attention(q, q, q, precision="nvfp4"))
    want = all_ops()

    def inference():
        with torch.inference_mode():
            return all_ops()
    native, python = both_paths(inference)
    assert _same(native, want) and _same(python, want) and all(a.is_inference() and b.is_inference() for a, b in zip(native, python))

    def deterministic():
        before = torch.are_deterministic_algorithms_enabled()
        torch.use_deterministic_algorithms(True, warn_only=True)
        try:
            return all_ops()
        finally:
            torch.use_deterministic_algorithms(before)
    assert all(_same(r, want) for r in both_paths(deterministic))
    for transform in (lambda: torch.func.vmap(lambda y: ops.quantize(x, 0, 1)[2] * y)(ones),
                      lambda: torch.func.functionalize(lambda y: ops.quantize(x, 0, 1)[2] * y)(ones),
                      lambda: torch.func.jvp(lambda y: ops.quantize(x, 0, 1)[2] * y, (ones,), (ones,))[0],
                      lambda: torch.func.grad(lambda y: (ops.quantize(x, 0, 1)[2] * y).sum())(ones),
                      lambda: torch.func.vmap(lambda y: ops.quantize(y, 0, 1)[2])(torch.stack([x, x]))):
        native, python = both_paths(transform)
        assert (isinstance(native, type) and isinstance(python, type)) or torch.equal(native, python), (native, python)
