"""The torch host module (``csrc/host/fgb_torch.cpp``): whole forward and backward
passes in one native call.  There is no fallback for a missing file: loading
raises and every op fails, as with the CUDA library it drives."""
import ctypes
import importlib.machinery
import importlib.util
import os

import torch  # noqa: F401  (the module needs torch's libraries in the process)

from . import _build, _cabi

_mod = None


def ext():
    global _mod
    if _mod is None:
        path = _build.host_path()
        if not os.path.exists(path):
            raise RuntimeError(f"{path} not found: build it with `python -m flexgemm_b200._build`")
        spec = importlib.util.spec_from_file_location("_fgb_torch", path, loader=importlib.machinery.ExtensionFileLoader("_fgb_torch", path))
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        from .kernels import config
        mod.init(_cabi.lib()._handle, ctypes.addressof(config._native_tf32))
        _mod = mod
    return _mod
