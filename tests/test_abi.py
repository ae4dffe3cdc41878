"""CPU-side checks of the C-ABI shared library: it builds, loads, exports every symbol the header declares,
and validates its arguments before touching a device.  No GPU needed (nvcc cross-compiles)."""
import ctypes
import re
from pathlib import Path

import pytest

from matmulfreellm_b200 import _build, _lib

HEADER = Path(__file__).resolve().parent.parent / "include" / "mmfree_b200.h"


@pytest.fixture(scope="module")
def lib():
    _build.build_library()
    return _lib.load()


def declared_symbols():
    text = HEADER.read_text()
    return sorted(set(re.findall(r"\b(mmf_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported_and_bound(lib):
    names = declared_symbols()
    assert len(names) >= 15
    for name in names:
        assert hasattr(lib, name), f"{name} declared in the header but not exported"
        assert name in _lib.PROTOTYPES, f"{name} has no ctypes prototype"
    assert sorted(_lib.PROTOTYPES) == names


def test_abi_version_and_constants(lib):
    assert lib.mmf_abi_version() == _lib.ABI_VERSION
    text = HEADER.read_text()
    assert f"#define MMF_ABI_VERSION {_lib.ABI_VERSION}" in text
    assert f"#define MMF_TILE_ROWS {_lib.TILE_ROWS}" in text and f"#define MMF_TILE_K {_lib.TILE_K}" in text
    assert lib.mmf_packed_bytes(128, 64) == 128 * 16
    assert lib.mmf_packed_bytes(200, 192) == 2 * 3 * 128 * 16
    assert lib.mmf_packed_bytes(128, 100) == 0          # K must be a multiple of 64
    assert lib.mmf_hgrn_workspace_bytes(8, 2048, 2048) == 0
    assert lib.mmf_hgrn_workspace_bytes(1, 8192, 128) > 0
    assert lib.mmf_bitlinear_workspace_bytes(1, 2048, 2048) % 256 == 0


def test_argument_validation_needs_no_device(lib):
    """Bad arguments are rejected on the host with a status code and a message (no CUDA call is made)."""
    with pytest.raises(_lib.MMFreeError) as e:
        _lib.call("mmf_act_quant", None, 1, 64, None, 1, 1e-6, None, None, None, 1, 64, None)
    assert e.value.code == -1 and "null" in str(e.value)
    buf = (ctypes.c_char * 4096)()
    p = (ctypes.addressof(buf) + 15) & ~15
    with pytest.raises(_lib.MMFreeError) as e:   # K not a multiple of 16
        _lib.call("mmf_act_quant", p, 1, 40, None, 1, 1e-6, p, p, p, 1, 40, None)
    assert e.value.code == -2
    with pytest.raises(_lib.MMFreeError) as e:   # misaligned x
        _lib.call("mmf_act_quant", p + 2, 1, 64, None, 1, 1e-6, p, p, p, 1, 64, None)
    assert e.value.code == -3
    with pytest.raises(_lib.MMFreeError) as e:   # unknown dtype
        _lib.call("mmf_rmsnorm", p, 7, None, 7, None, 1e-6, p, None, 1, 64, None)
    assert e.value.code == -1
    with pytest.raises(_lib.MMFreeError) as e:   # K % 64 != 0
        _lib.call("mmf_pack_ternary", p, 128, 96, p, p, None)
    assert e.value.code == -2
    with pytest.raises(_lib.MMFreeError) as e:   # groups must split N into multiples of 128
        _lib.call("mmf_bitlinear", p, p, p, p, p, 3, p, 1, 300, None, 1, 300, 64, None, 0, 0, None)
    assert e.value.code == -2
    with pytest.raises(_lib.MMFreeError) as e:   # D % 8
        _lib.call("mmf_hgrn_scan", p, 1, p, 1, None, None, 0, p, 1, 4, 12, 0, None, 0, None)
    assert e.value.code == -2
    # empty problems are accepted without a launch
    _lib.call("mmf_act_quant", p, 1, 64, None, 1, 1e-6, p, p, p, 0, 64, None)
    _lib.call("mmf_hgrn_scan", p, 1, p, 1, None, None, 0, p, 0, 4, 16, 0, None, 0, None)


def test_decode_linear_refuses_bad_arguments(lib):
    """Every refusal of mmf_decode_linear comes from the host, before any CUDA call."""
    buf = (ctypes.c_char * 4096)()
    p = (ctypes.addressof(buf) + 15) & ~15
    L = _lib

    def rc(**change):
        args = dict(prologue=L.PRO_PRENORM, epilogue=L.EPI_STORE, dtype=L.BF16, M=2, N=64, K=128, packed=p, w_scale=p, x=p, ld_x=128,
                    out=p, ld_out=64)
        args.update(change)
        bl = args.pop("bl_norm_w", (None, None, None))
        return lib.mmf_decode_linear(ctypes.byref(L.DecodeLinearArgs(bl_norm_w=(ctypes.c_void_p * 3)(*bl), **args)), None)

    BAD_ARG, BAD_SHAPE, ALIGN = -1, -2, -3
    assert lib.mmf_decode_linear(None, None) == BAD_ARG
    ws = dict(codes=p, dq=p, rowsum=p)
    gates = dict(epilogue=L.EPI_GATES, N=384, state=p, g_out=p)
    gatenorm = dict(prologue=L.PRO_GATENORM, residual=p, ld_residual=128)
    for want, cases in {
        BAD_ARG: [dict(dtype=L.F32), dict(dtype=7), dict(packed=None), dict(w_scale=None), dict(out=None), dict(x=None), dict(prologue=0),
                  dict(prologue=9), dict(epilogue=9), dict(gatenorm, residual=None), dict(ws, dq=None), dict(ws, rowsum=None),
                  dict(ws, codes=p + 8), dict(gates, state=None), dict(gates, g_out=None), dict(gates, state=p + 4),
                  dict(gates, g_out=p + 2), dict(gates, lower_bound=p + 2), dict(ld_out=63), dict(row_ids=p, x_rows=0),
                  dict(row_ids=p, x_rows=5, residual=p, ld_residual=128), dict(row_ids=p, x_rows=5, prologue=L.PRO_QUANT)],
        BAD_SHAPE: [dict(ws, M=16, N=(1 << 24) - 128, ld_out=1 << 24),       # partial sums do not fit; the row kernel has not run either
                    dict(M=-1), dict(M=3), dict(ws, M=17), dict(N=0), dict(N=1 << 24), dict(K=0), dict(K=96), dict(K=4160, ld_x=4160),
                    dict(K=8256, ld_x=8256, prologue=L.PRO_QUANT), dict(gatenorm, K=4160, ld_x=4160, ld_residual=4160),
                    dict(gates, N=256), dict(gates, K=192, N=576, ld_x=192), dict(epilogue=L.EPI_SWIGLU, N=66, ld_out=34),
                    dict(epilogue=L.EPI_SWIGLU, ld_out=33), dict(epilogue=L.EPI_SWIGLU, ld_out=30), dict(ld_x=120), dict(ld_x=0),
                    dict(gatenorm, ld_residual=120), dict(row_ids=p, x_rows=5, M=1, ld_x=64)],
        ALIGN: [dict(packed=p + 8), dict(x=p + 2), dict(out=p + 8), dict(ld_x=129), dict(residual=p + 8, ld_residual=128),
                dict(residual=p, ld_residual=132), dict(residual_out=p + 8), dict(norm_w=p + 4), dict(bl_norm_w=(p + 4, None, None)),
                dict(gates, bl_norm_w=(p, p, p + 8))],
    }.items():
        for change in cases:
            assert rc(**change) == want, (change, lib.mmf_last_error())
    for change in (dict(), ws, gates, gatenorm, dict(epilogue=L.EPI_SWIGLU, ld_out=32)):
        assert rc(**change, M=0) == 0           # an empty problem is accepted without a launch


def test_decode_step_refuses_bad_arguments(lib):
    """What mmf_decode_step refuses on the host, before any CUDA call."""
    from matmulfreellm_b200 import _lib as L
    BAD_ARG, BAD_SHAPE, ALIGN = -1, -2, -3
    p = 4096

    def rc(layer=None, **change):
        args = dict(dtype=L.BF16, M=2, hidden=256, inner=512, layers=1, x=p, ld_x=256, out=p, residual_out=p, workspace=p, workspace_bytes=1 << 30, status=p)
        args.update(change)
        y = L.DecodeStepLayer(**{**dict(weights=p, state=p), **(layer or {})})
        return lib.mmf_decode_step(ctypes.byref(L.DecodeStepArgs(layer=ctypes.pointer(y), **args)), None)

    assert lib.mmf_decode_step(None, None) == BAD_ARG and lib.mmf_decode_step_pack(None, 256, 512, p, None) == BAD_ARG
    for want, cases in {
        BAD_ARG: [dict(dtype=L.F32), dict(x=None), dict(out=None), dict(residual_out=None), dict(workspace=None), dict(status=None),
                  dict(layer=dict(weights=None)), dict(layer=dict(state=None)), dict(row_ids=p)],
        BAD_SHAPE: [dict(M=0), dict(layers=0), dict(layers=97), dict(ld_x=248), dict(M=1, row_ids=p, x_rows=5, ld_x=128)],
        ALIGN: [dict(x=p + 8), dict(ld_x=260), dict(out=p + 8), dict(residual_out=p + 8), dict(workspace=p + 128), dict(layer=dict(weights=p + 8)),
                dict(layer=dict(state=p + 4)), dict(layer=dict(lower_bound=p + 2))],
    }.items():
        for change in cases:
            assert rc(**change) == want, (change, lib.mmf_last_error())


def test_cpu_tensors_are_refused():
    import torch
    from matmulfreellm_b200 import kernels
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        kernels.rmsnorm(torch.zeros(2, 64), torch.ones(64), 1e-6)


def test_kernels_refuse_tensors_of_another_device(monkeypatch):
    """The C entry points launch on the current CUDA device; tensors that live on another GPU must be refused before
    anything is launched (checked with stand-in tensor objects: no GPU needed)."""
    import types

    import pytest
    import torch

    from matmulfreellm_b200 import _lib, kernels
    monkeypatch.setattr(kernels, "_raw_device", lambda: 0)
    monkeypatch.setattr(_lib, "require_device", lambda idx: None)
    t0 = types.SimpleNamespace(is_cuda=True, device=torch.device("cuda", 0))
    t1 = types.SimpleNamespace(is_cuda=True, device=torch.device("cuda", 1))
    cpu = types.SimpleNamespace(is_cuda=False, device=torch.device("cpu"))
    assert kernels._need_cuda(t0, None, t0) == torch.device("cuda", 0)
    with pytest.raises(RuntimeError, match="current device is cuda:0"):
        kernels._need_cuda(t1)
    with pytest.raises(RuntimeError, match="different devices"):
        kernels._need_cuda(t0, t1)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        kernels._need_cuda(cpu)
