"""The compiled pybind11 form of the operator module (`_cuda_ops`, built from csrc/bindings_pybind.cc by
`python ac4k_kernel_b200/build.py --pybind`): the same names and positional signatures as the reference's
`ac4k_kernel._cuda_ops` (lib/cuda_bindings.cc:37-97).  `ac4k_kernel_b200._cuda_ops` is the ctypes form of the
same interface; both call the same C ABI."""

import warnings

try:
    from . import _host_calls as host_calls      # the operators in one native call each (csrc/host_calls.cc)
except ImportError as e:
    # The Python wrappers give the same results in more launches and several times the host time, so this is said once.
    host_calls = None
    warnings.warn("ac4k_kernel_b200: the operators' native host side (native/_host_calls) "
                  + ("is not built" if isinstance(e, ModuleNotFoundError) else f"does not load ({e})")
                  + "; small calls take several times longer without it.  Build it with `python ac4k_kernel_b200/build.py`.",
                  RuntimeWarning, stacklevel=2)


def load():
    """Import and return the compiled module; raises ImportError with the build command if it is not built."""
    try:
        from . import _cuda_ops
    except ImportError as e:
        raise ImportError("the pybind module is not built: run `python ac4k_kernel_b200/build.py --pybind`") from e
    return _cuda_ops
