"""CPU checks of the boundary: the library loads and exports exactly what include/vinf_b200.h declares."""
from __future__ import annotations

import ctypes
import re
from pathlib import Path

import numpy as np
import pytest

from vinf_3080ti_b200 import _capi
from vinf_3080ti_b200.gguf_types import TRAITS, GGUFTensorType, row_bytes

REPO = Path(__file__).resolve().parent.parent


def declared_functions() -> set[str]:
    text = (REPO / "include" / "vinf_b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return set(re.findall(r"\b(vqm_\w+)\s*\(", text))


@pytest.fixture(scope="module")
def lib():
    from vinf_3080ti_b200 import build

    build.build()
    return _capi.load()


def test_every_declared_entry_point_is_exported_and_bound(lib):
    declared = declared_functions()
    assert declared, "header parse found nothing"
    for name in declared:
        assert hasattr(lib, name), f"{name} is declared in include/vinf_b200.h but not exported"
    assert declared == set(_capi.SIGNATURES), declared ^ set(_capi.SIGNATURES)


def test_header_type_ids_match_the_python_table():
    text = (REPO / "include" / "vinf_b200.h").read_text()
    ids = {name: int(val) for name, val in re.findall(r"VQM_(\w+) = (\d+)", text) if name in GGUFTensorType.__members__}
    assert ids == {t.name: int(t) for t in TRAITS}


def test_status_codes_map_to_the_reference_exceptions():
    assert _capi._EXC == {1: KeyError, 2: ValueError, 3: TypeError, 4: MemoryError, 5: RuntimeError}


def test_row_bytes_of_the_benchmark_shapes():
    assert row_bytes(GGUFTensorType.Q4_K, 5120) == 2880
    assert row_bytes(GGUFTensorType.Q3_K, 5120) == 2200
    assert row_bytes(GGUFTensorType.Q6_K, 5120) == 4200
    assert row_bytes(GGUFTensorType.Q4_K, 17408) == 9792
    with pytest.raises(ValueError):
        row_bytes(GGUFTensorType.Q4_K, 100)


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_capi, "_lib", None)
    monkeypatch.setattr(_capi, "LIB_PATH", tmp_path / "libvinf_b200.so")
    with pytest.raises(_capi.ExtensionMissingError):
        _capi.load()


@pytest.mark.parametrize("ntok,seen", [(3, 3), (np.int64(7), 7), (2.9, 2), ("5", 5), (True, 1), (-1, -1), (2**32 + 9, 9)])
def test_pycall_hands_its_arguments_on_as_ctypes_does(ntok, seen):
    got = []

    @ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_char_p, ctypes.c_char_p, ctypes.c_char_p, ctypes.c_int)
    def fn(*args):
        got.append(args)
        return 4

    address = ctypes.cast(fn, ctypes.c_void_p).value
    assert _capi.pycall().qmv(address, 123, "w", "größe", "y\0z", ntok) == 4
    assert got == [(123, b"w", "größe".encode(), b"y", seen)]
    for bad in ((b"w", "x", "y", 1), ("w", None, "y", 1)):
        with pytest.raises(AttributeError):
            _capi.pycall().qmv(address, 123, *bad)
    with pytest.raises(UnicodeEncodeError):
        _capi.pycall().qmv(address, 123, "w", "\udc80", "y", 1)
    with pytest.raises((TypeError, ValueError)):
        _capi.pycall().qmv(address, 123, "w", "x", "y", None)
    with pytest.raises((TypeError, ValueError)):  # a closed runtime
        _capi.pycall().qmv(address, None, "w", "x", "y", 1)
    assert len(got) == 1


def test_the_call_without_ctypes_is_optional(monkeypatch, tmp_path):
    import sys

    from vinf_3080ti_b200 import build

    seen = []
    monkeypatch.setattr(_capi, "load", lambda: type("Lib", (), {"vqm_qmv": staticmethod(lambda *a: seen.append(a) or 4)}))
    monkeypatch.setitem(sys.modules, "vinf_3080ti_b200._vqm_pycall", None)  # as if this interpreter could not load it
    monkeypatch.delattr("vinf_3080ti_b200._vqm_pycall", raising=False)
    assert _capi.pycall() is None
    call, address = _capi.qmv_caller()
    assert call(address, 123, "w", "größe", "y", np.int64(7)) == 4
    assert seen == [(123, b"w", "größe".encode(), b"y", 7)]
    # a box without a C compiler gets the library all the same, and no stale module
    stale = tmp_path / build.PYCALL.name
    stale.write_bytes(b"")
    monkeypatch.setattr(build, "PYCALL", stale)
    monkeypatch.setattr(build, "up_to_date", lambda: True)
    monkeypatch.setenv("PATH", str(tmp_path))
    assert build.build_pycall(force=True) is None and not stale.exists()
    assert build.build() == build.LIB


@pytest.mark.parametrize("call", ["qmv('w', 'x', 'y')", "matvec('w', bytes(4))", "has('w')", "qmv_argmax('w', 'x', None)", "argmax('x', 1)",
                                  "write('x', bytes(4))", "synchronize()", "stream()", "capture_begin()", "graph_launch(0)",
                                  "exchange_create(8)", "qmv_group(['w'], 'x', ['y'], 1)"])
def test_calls_on_a_closed_runtime_are_errors(call):
    from vinf_3080ti_b200.runtime import Runtime

    rt = Runtime.__new__(Runtime)  # (a real one needs a GPU)
    rt._lib = _capi.load()
    rt._qmv, rt._qmv_fn = _capi.qmv_caller()
    rt._h = ctypes.c_void_p()
    rt.close()
    rt.close()
    with pytest.raises(ValueError, match="closed"):
        eval(f"rt.{call}", {"rt": rt})
