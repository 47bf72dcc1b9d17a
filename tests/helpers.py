"""Seeded synthetic inputs shared by the CPU and GPU tests."""
import ctypes
import os

import numpy as np
import pytest
import torch

HOOKS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ac4k_kernel_b200", "build_hooks", "libac4k_b200_hooks.so")


def hooks_library():
    """The debug-hook build of the library (`build.py --hooks`), with its switches; skips the test where it is not built."""
    from ac4k_kernel_b200 import _lib
    if not os.path.exists(HOOKS):
        pytest.skip("debug-hook build not present (python ac4k_kernel_b200/build.py --hooks)")
    lib = ctypes.CDLL(HOOKS)
    for name, (res, args) in _lib.SIGNATURES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    lib.ac4k_debug_set_wait_ns.argtypes = [ctypes.c_uint64]
    lib.ac4k_debug_set_flags.argtypes = [ctypes.c_int]
    return lib


def takes_one_launch(shape, cross, reduce, swizzle=False, sms=148):
    """The library's own rule, for a contiguous 16-byte aligned tensor: whether the call is sent to the one-launch kernel (no GPU needed)"""
    lib = hooks_library()
    stride, n = [0] * len(shape), 1
    for i in reversed(range(len(shape))):
        stride[i], n = n, n * shape[i]
    order = [i for i in range(len(shape)) if i not in (cross, reduce)] + [cross, reduce]
    pad, c = 4 - len(shape), ctypes.c_int64 * 4
    return bool(lib.ac4k_debug_takes_one_launch(c(*[1] * pad, *[shape[i] for i in order]), c(*[0] * pad, *[stride[i] for i in order]), int(swizzle), sms))


def dynamic_nvfp4(lib, x, cross, reduce, swizzle=False, layout="ac4k", scratch=None):
    """ac4k_quantize_nvfp4_dynamic of `lib` on the current stream; scratch: None for one of its own, or a device address"""
    from ac4k_kernel_b200 import _cuda_ops as ct
    size, stride, others = ct._view4(x, cross, reduce)
    lead, m, kt = [x.shape[i] for i in others], x.shape[cross], (x.shape[reduce] + 63) // 64
    q = torch.empty(lead + [m, kt * 32], dtype=torch.uint8, device=x.device)
    shape = lead + ([kt, (m + 15) // 16 * 16, 4] if layout == "ac4k" else [(m + 127) // 128, kt, 32, 4, 4])
    sf, g = torch.empty(shape, dtype=torch.float8_e4m3fn, device=x.device), torch.empty((), device=x.device)
    own = torch.empty(1024, dtype=torch.int32, device=x.device) if scratch is None else None
    rc = lib.ac4k_quantize_nvfp4_dynamic(q.data_ptr(), sf.data_ptr(), g.data_ptr(), own.data_ptr() if scratch is None else scratch, x.data_ptr(),
                                         2688.0, ct._I64x4(*size), ct._I64x4(*stride), int(swizzle), int(layout != "ac4k"),
                                         torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.ac4k_last_error()
    return q, sf, g


def bf16_from_bits(arr: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(arr.view(np.int16).copy()).view(torch.bfloat16)


def gaussian(shape, seed=0, std=1.0, outlier_frac=0.0, outlier_mul=1.0):
    """CPU-generated so that CPU and GPU runs see identical bits."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(shape, generator=g) * std
    if outlier_frac > 0:
        mask = torch.rand(shape, generator=g) < outlier_frac
        x = torch.where(mask, x * outlier_mul, x)
    return x.bfloat16()


def bf16_ulp(ref: torch.Tensor) -> torch.Tensor:
    """Size of one bf16 ulp at |ref| (fp32 tensor), 2^(floor(log2|ref|) - 7); bf16 min normal floor."""
    a = ref.abs().float().clamp(min=2.0 ** -126)
    e = torch.frexp(a)[1] - 1
    return torch.ldexp(torch.ones_like(a), e - 7)
