"""Numeric mode switch for fp32 inputs.

``allow_tf32 = True``  : fp32 features/weights are multiplied as TF32 on the
                         tensor cores (fp32 accumulate) -- the reference default
                         on CUDA (flex_gemm/kernels/triton/spconv/config.py:6).
``allow_tf32 = False`` : fp32-accurate products (split-TF32 on the tensor cores).
16-bit inputs are unaffected.  A pass, forward or backward, takes the setting of
the time it runs.
"""
import ctypes
import sys
import types

_native_tf32 = ctypes.c_bool(True)  # what native backward passes read: they run without the interpreter


class _Config(types.ModuleType):
    def __setattr__(self, name, value):
        if name == "allow_tf32":
            _native_tf32.value = bool(value)
        super().__setattr__(name, value)


allow_tf32 = True
sys.modules[__name__].__class__ = _Config
