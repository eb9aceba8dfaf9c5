"""The C-ABI library loads and exports every symbol include/leviathan_cuda.h
declares (no compute calls: this runs without a GPU)."""
import ctypes
import os
import re

import pytest

from leviathan_b200 import _lib as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "leviathan_cuda.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(lev_[a-z0-9_]+)\s*\(", text)))


@pytest.fixture(scope="module")
def lib():
    if not os.path.exists(L.LIB_PATH):
        from leviathan_b200.build import build_library

        build_library()
    return ctypes.CDLL(L.LIB_PATH)


def test_every_declared_symbol_is_exported(lib):
    names = _declared_symbols()
    assert len(names) >= 30
    for n in names:
        assert hasattr(lib, n), f"{n} is declared but not exported"


def test_binding_table_matches_header():
    assert sorted(L.SIGNATURES) == _declared_symbols()


def test_version_and_status_names(lib):
    lib.lev_cuda_abi_version.restype = ctypes.c_int
    assert lib.lev_cuda_abi_version() == 1
    lib.lev_status_name.restype = ctypes.c_char_p
    for code, name in L.STATUS.items():
        assert lib.lev_status_name(code).decode() == name


def test_init_without_a_gpu_fails_with_a_status_not_a_crash(lib):
    import torch

    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    h = ctypes.c_void_p()
    lib.lev_cuda_init.restype = ctypes.c_int
    st = lib.lev_cuda_init(0, ctypes.byref(h))
    assert st == 8 and not h.value  # LEV_DEVICE_UNAVAILABLE


def test_package_fails_loudly_when_library_is_missing(monkeypatch):
    monkeypatch.setattr(L, "_lib", None)
    monkeypatch.setattr(L, "LIB_PATH", "/nonexistent/libleviathan_cuda.so")
    with pytest.raises(RuntimeError, match="no fallback"):
        L.load()


# the arguments each native call takes (csrc/lev_pyhost.c), handles NULL
HOST_CALLS = {
    "matvec": (None, None, 0, 16, None, 32, 1, None, 16, -1, 0),
    "matvec_fused": (None, None, 0, 16, None, 32, 1, 1, None, 1e-6, None, 1.0, None, 16),
    "matvec_chain": (None, 1, None, 0),
    "rmsnorm": (None, None, 1, 32, None, 1e-6, None, None),
    "axpy": (None, 1.0, None, None, 32, None),
    "act_bf16": (None, None, 32, None),
    "gemm_prefill": (None, None, None, 16, None, 0),
    "moe_layer": (None, None, None, 1, 8, None, None, None, 0),
    "moe_layer_residual": (None, None, None, 1, 8, None, 1.0, None, 0),
    "kv_append": (None, None, None, None, None, None, None, 1, None, None),
    "attn_decode": (None, None, None, None, None, None, None, 1, 8, None, 0, 1.0, None),
}


def test_host_layer_native_and_through_ctypes(lib, monkeypatch, tmp_path):
    """Both forms of the per-token calls take the same arguments; without a file for this interpreter, ctypes serves."""
    native = L.host()
    assert os.path.exists(L.HOST_PATH) and sorted(n for n in dir(native) if not n.startswith("_")) == sorted(HOST_CALLS)
    monkeypatch.setattr(L, "_host", None)
    monkeypatch.setattr(L, "HOST_PATH", str(tmp_path / "missing.so"))
    through_ctypes = L.host()
    for name, args in HOST_CALLS.items():
        a, b = getattr(native, name)(*args), getattr(through_ctypes, name)(*args)
        assert a == b and L.STATUS[a] == "badArgument", name
        for form in (native, through_ctypes):
            with pytest.raises(TypeError):
                getattr(form, name)(*args[:-1])


def test_build_without_a_compiler_leaves_ctypes(lib, monkeypatch, tmp_path):
    from leviathan_b200 import build

    path = tmp_path / "_pyhost.so"
    monkeypatch.setattr(build, "HOST_PATH", str(path))
    monkeypatch.setenv("CC", str(tmp_path / "no-such-compiler"))
    assert build.build_library() == build.LIB_PATH and not path.exists()
    path.write_bytes(b"of another library")
    os.utime(path, (0, 0))
    assert build.build_library() == build.LIB_PATH and not path.exists()
