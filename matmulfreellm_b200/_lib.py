"""ctypes binding of libmmfree_b200.so (the C ABI declared in include/mmfree_b200.h).

There is no CPU or PyTorch fallback behind these bindings: if the shared library is
missing, or the device is not a B200-class GPU, the calls raise.
"""
from __future__ import annotations

import ctypes
from ctypes import c_char_p, c_double, c_float, c_int, c_int64, c_void_p
from pathlib import Path

LIB_PATH = Path(__file__).resolve().parent / "libmmfree_b200.so"

F32, BF16, F16 = 0, 1, 2
KERNEL_AUTO, KERNEL_GEMV, KERNEL_MMA = 0, 1, 2
KERNEL_STREAM = 3   # Python-level selector: the mma.sync decode experiment (mmf_bitlinear_decode, experiments build only)
STREAM_MAX_M = 64
TILE_ROWS, TILE_K = 128, 64
ABSMEAN_PARTIALS = 1024
ABI_VERSION = 3

ERR_CUDA, ERR_TIMEOUT = -4, -7
_ERR_NAMES = {
    -1: "MMF_ERR_BAD_ARG", -2: "MMF_ERR_BAD_SHAPE", -3: "MMF_ERR_ALIGN", -4: "MMF_ERR_CUDA",
    -5: "MMF_ERR_ARCH", -6: "MMF_ERR_WORKSPACE", -7: "MMF_ERR_TIMEOUT",
    -8: "MMF_ERR_NOT_RESIDENT",
}

class DecodeLinearArgs(ctypes.Structure):
    """mmf_decode_linear_args of the header, field by field."""
    _fields_ = [("prologue", c_int), ("epilogue", c_int), ("dtype", c_int), ("round_sum_first", c_int), ("M", c_int64),
                ("N", c_int64), ("K", c_int64), ("packed", c_void_p), ("w_scale", c_void_p), ("x", c_void_p),
                ("residual", c_void_p), ("ld_x", c_int64), ("ld_residual", c_int64), ("row_ids", c_void_p), ("x_rows", c_int64),
                ("norm_w", c_void_p), ("eps_norm", c_float), ("eps_bl", c_float), ("bl_norm_w", c_void_p * 3),
                ("residual_out", c_void_p), ("codes", c_void_p), ("dq", c_void_p), ("rowsum", c_void_p), ("out", c_void_p),
                ("ld_out", c_int64), ("g_out", c_void_p), ("lower_bound", c_void_p), ("mask", c_void_p), ("state", c_void_p)]


class DecodeStepLayer(ctypes.Structure):
    """mmf_decode_step_layer of the header."""
    _fields_ = [("weights", c_void_p), ("lower_bound", c_void_p), ("state", c_void_p), ("eps_gate", c_float), ("eps_bl", c_float)]


class DecodeStepArgs(ctypes.Structure):
    """mmf_decode_step_args of the header, field by field."""
    _fields_ = [("dtype", c_int), ("M", c_int64), ("hidden", c_int64), ("inner", c_int64), ("layers", c_int64),
                ("layer", ctypes.POINTER(DecodeStepLayer)), ("x", c_void_p), ("ld_x", c_int64), ("row_ids", c_void_p), ("x_rows", c_int64),
                ("mask", c_void_p), ("eps_norm", c_float), ("out", c_void_p), ("residual_out", c_void_p), ("workspace", c_void_p),
                ("workspace_bytes", c_int64), ("status", c_void_p), ("gave_up_host", c_void_p)]


PRO_QUANT, PRO_PRENORM, PRO_GATENORM = 1, 2, 3
EPI_STORE, EPI_GATES, EPI_SWIGLU = 0, 1, 2

# name -> (restype, argtypes); must list every symbol include/mmfree_b200.h declares
PROTOTYPES = {
    "mmf_last_error": (c_char_p, []),
    "mmf_abi_version": (c_int, []),
    "mmf_check_device": (c_int, []),
    "mmf_absmean_f32": (c_int, [c_void_p, c_int64, c_void_p, c_void_p, c_void_p]),
    "mmf_packed_bytes": (c_int64, [c_int64, c_int64]),
    "mmf_pack_ternary": (c_int, [c_void_p, c_int64, c_int64, c_void_p, c_void_p, c_void_p]),
    "mmf_unpack_ternary": (c_int, [c_void_p, c_int64, c_int64, c_void_p, c_void_p]),
    "mmf_act_quant": (c_int, [c_void_p, c_int, c_int64, c_void_p, c_int, c_float, c_void_p, c_void_p, c_void_p,
                              c_int64, c_int64, c_void_p]),
    "mmf_bitlinear_workspace_bytes": (c_int64, [c_int64, c_int64, c_int64]),
    "mmf_bitlinear": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_int, c_int64,
                              c_void_p, c_int64, c_int64, c_int64, c_void_p, c_int64, c_int, c_void_p]),
    "mmf_bitlinear_gemv_static": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_int, c_int64,
                                          c_int64, c_int64, c_int64, c_void_p]),
    "mmf_int8_mma_peak": (c_int, [c_int, c_int, c_void_p, c_void_p]),
    "mmf_sync_probe": (c_int, [c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p]),
    "mmf_hgrn_workspace_bytes": (c_int64, [c_int64, c_int64, c_int64]),
    "mmf_hgrn_scan": (c_int, [c_void_p, c_int, c_void_p, c_int, c_void_p, c_void_p, c_int, c_void_p, c_int64,
                              c_int64, c_int64, c_int, c_void_p, c_int64, c_void_p]),
    "mmf_hgrn_status": (c_int, [c_void_p]),
    "mmf_hgrn_gated": (c_int, [c_void_p, c_void_p, c_int64, c_int, c_void_p, c_void_p, c_void_p, c_int64, c_int64,
                               c_int64, c_void_p, c_int64, c_void_p]),
    "mmf_hgrn_gated_masked": (c_int, [c_void_p, c_void_p, c_int64, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_int64,
                                      c_int64, c_int64, c_void_p, c_int64, c_void_p]),
    "mmf_prenorm_quant": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_int, c_int, c_void_p, c_float, c_void_p,
                                  c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_float, c_void_p, c_void_p, c_void_p,
                                  c_int64, c_int64, c_void_p]),
    "mmf_gatenorm_quant": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_int, c_void_p, c_float, c_void_p, c_float,
                                   c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_void_p]),
    "mmf_decode_mix": (c_int, [c_void_p, c_int64, c_int, c_void_p, c_void_p, c_void_p, c_float, c_void_p, c_float, c_void_p,
                               c_void_p, c_void_p, c_int64, c_int64, c_void_p]),
    "mmf_decode_mix_masked": (c_int, [c_void_p, c_int64, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_float, c_void_p, c_float,
                                      c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_void_p]),
    "mmf_swiglu_quant": (c_int, [c_void_p, c_void_p, c_int64, c_int, c_void_p, c_float, c_void_p, c_void_p, c_void_p,
                                 c_int64, c_int64, c_void_p]),
    "mmf_decode_linear": (c_int, [c_void_p, c_void_p]),
    "mmf_decode_step_layer_bytes": (c_int64, [c_int64, c_int64]),
    "mmf_decode_step_pack": (c_int, [c_void_p, c_int64, c_int64, c_void_p, c_void_p]),
    "mmf_decode_step_workspace_bytes": (c_int64, [c_int64, c_int64, c_int64, c_int64]),
    "mmf_decode_step": (c_int, [c_void_p, c_void_p]),
    "mmf_rmsnorm": (c_int, [c_void_p, c_int, c_void_p, c_int, c_void_p, c_float, c_void_p, c_void_p, c_int64,
                            c_int64, c_void_p]),
    "mmf_rmsnorm_swishgate": (c_int, [c_void_p, c_void_p, c_int, c_void_p, c_float, c_void_p, c_int64, c_int64,
                                      c_void_p]),
    "mmf_swiglu": (c_int, [c_void_p, c_int64, c_void_p, c_int64, c_void_p, c_int64, c_int, c_int64, c_int64,
                           c_void_p]),
    "mmf_argmax_rows": (c_int, [c_void_p, c_int, c_int64, c_int64, c_int64, c_void_p, c_void_p]),
    "mmf_sample_top_p": (c_int, [c_void_p, c_int, c_int64, c_float, c_float, c_void_p, c_void_p, c_int64, c_int64, c_void_p]),
    "mmf_embedding": (c_int, [c_void_p, c_int, c_int64, c_int64, c_void_p, c_void_p, c_int64, c_void_p]),
}


class MMFreeError(RuntimeError):
    """A C-ABI call returned a negative status."""

    def __init__(self, fn: str, code: int, text: str):
        self.code = code
        super().__init__(f"{fn} failed with {_ERR_NAMES.get(code, code)}: {text}")


_lib = None
EXPERIMENTS_LIB_PATH = LIB_PATH.with_name("libmmfree_b200_experiments.so")
_EXPERIMENT_PROTOTYPES = {
    "mmf_tuning": (c_int, [c_int, c_int]), "mmf_row_trace": (c_int, [c_void_p]),
    "mmf_rounding_check": (c_int, [c_void_p, c_void_p]),
    "mmf_repack_slabs": (c_int, [c_void_p, c_int64, c_int64, c_void_p, c_void_p]),
    "mmf_bitlinear_decode_fits": (c_int, [c_int64, c_int64]),
    "mmf_bitlinear_decode": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_int, c_int64,
                                     c_void_p, c_int64, c_int64, c_int64, c_void_p, c_void_p]),
}


def _open(path: Path, prototypes) -> ctypes.CDLL:
    lib = ctypes.CDLL(str(path))
    for name, (res, args) in prototypes.items():
        fn = getattr(lib, name)  # AttributeError here = header and library out of sync
        fn.restype = res
        fn.argtypes = args
    if lib.mmf_abi_version() != ABI_VERSION:
        raise RuntimeError(f"{path.name} ABI {lib.mmf_abi_version()} != binding ABI {ABI_VERSION}")
    return lib


def load() -> ctypes.CDLL:
    """Load the shared library (once) and attach prototypes. Raises if it has not been built."""
    global _lib
    if _lib is not None:
        return _lib
    if not LIB_PATH.exists():
        raise RuntimeError(
            f"{LIB_PATH} is missing. Build it with `python -m matmulfreellm_b200._build` "
            "(needs nvcc); there is no fallback implementation.")
    _lib = _open(LIB_PATH, PROTOTYPES)
    return _lib


class experiments_library:
    """Context manager for kernel experiments and the configuration-sweep tests: inside it every call of this module
    goes to libmmfree_b200_experiments.so (the same sources built with -DMMF_EXPERIMENTS), which also exports
    mmf_tuning; on exit all overrides are reset and the product library is current again."""

    KNOBS = 15
    _handle = None

    def __enter__(self):
        global _lib
        cls = experiments_library
        if cls._handle is None:
            if not EXPERIMENTS_LIB_PATH.exists():
                raise RuntimeError(f"{EXPERIMENTS_LIB_PATH} is missing: python -m matmulfreellm_b200._build")
            cls._handle = _open(EXPERIMENTS_LIB_PATH, {**PROTOTYPES, **_EXPERIMENT_PROTOTYPES})
        self._saved = load()
        _lib = cls._handle
        if _native is not None:
            _native.use_library(str(EXPERIMENTS_LIB_PATH))
        return cls._handle

    def __exit__(self, *exc):
        global _lib
        for k in range(self.KNOBS):
            experiments_library._handle.mmf_tuning(k, 0)
        _lib = self._saved
        if _native is not None:
            _native.use_library(str(LIB_PATH))
        return False


NATIVE_PATH = LIB_PATH.with_name("_native.so")
_native = None


def native():
    """The native host path (csrc/binding.cpp), loaded once; it calls whichever library is current (see
    experiments_library).  Raises if it has not been built."""
    global _native
    if _native is None:
        import importlib.machinery
        import importlib.util

        import torch  # noqa: F401 - its libraries must be loaded before the module that links against them

        from . import kernels
        load()
        if not NATIVE_PATH.exists():
            raise RuntimeError(f"{NATIVE_PATH} is missing. Build it with `python -m matmulfreellm_b200._build`; there is no "
                               "fallback implementation.")
        name = __package__ + "._native"
        spec = importlib.util.spec_from_loader(name, importlib.machinery.ExtensionFileLoader(name, str(NATIVE_PATH)))
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        mod.set_hooks(MMFreeError, kernels.stream_workspace, require_device)
        mod.use_library(str(EXPERIMENTS_LIB_PATH if _lib is experiments_library._handle else LIB_PATH))
        _native = mod
    return _native


# kernels each entry point launches per successful call (for launch accounting in benchmarks)
_LAUNCHES = {"mmf_absmean_f32": 2}
launch_count = 0


def call(name: str, *args) -> None:
    """Invoke an int-returning entry point and raise MMFreeError on a negative status."""
    global launch_count
    lib = load()
    rc = getattr(lib, name)(*args)
    if rc != 0:
        raise MMFreeError(name, rc, lib.mmf_last_error().decode(errors="replace"))
    launch_count += _LAUNCHES.get(name, 1)


_device_checked = set()


def require_device(index: int) -> None:
    """Fail loudly (once per device) unless `index` is a compute-capability-10.x GPU."""
    if index in _device_checked:
        return
    import torch
    if not torch.cuda.is_available():
        raise RuntimeError("matmulfreellm_b200 needs a CUDA device (B200, sm_100a); none is available")
    with torch.cuda.device(index):
        call("mmf_check_device")
    _device_checked.add(index)
