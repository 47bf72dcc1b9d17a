"""The operators' native host side (csrc/host_calls.cc) against the Python wrappers' own path: what it refuses."""
import glob
import importlib.util
import os
import shutil
import subprocess
import sys

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
