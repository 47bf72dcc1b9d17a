"""The operators' native host side (csrc/host_calls.cc) against the Python wrappers' own path: what it refuses."""
import glob
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


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(max_scale=-1.0), dict(max_scale=0), dict(max_scale=-5)])
def test_refused_by_the_library(both_paths, kw):
    from ac4k_kernel_b200 import ops
    x = gaussian((64, 128), seed=1).cuda()
    assert both_paths(lambda: ops.quantize(x, 0, 1, **kw)) == [RuntimeError, RuntimeError]
    with pytest.raises(RuntimeError, match=r"code -2\): max_scale must be positive"):
        ops.quantize(x, 0, 1, **kw)
