"""The C-ABI library loads on a CPU-only host and exports what include/mie_b200.h declares."""

from __future__ import annotations

import ctypes
import re
from pathlib import Path

import pytest

from mini_inference_engine_b200 import _lib, build

HEADER = Path(__file__).resolve().parents[1] / "include" / "mie_b200.h"


def declared_functions() -> set[str]:
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return set(re.findall(r"\b(mie_[a-z0-9_]+)\s*\(", text))


@pytest.fixture(scope="module")
def library():
    build.build_library()
    return ctypes.CDLL(str(build.LIB_PATH))


def test_header_and_binding_agree():
    assert declared_functions() == set(_lib.exported_symbols())


def test_every_declared_symbol_is_exported(library):
    for name in declared_functions():
        assert hasattr(library, name), name


def test_host_only_calls_work_without_a_gpu(library):
    lib = _lib.load()
    assert lib.mie_version() >= 1
    assert lib.mie_decode_scratch_bytes(4, 32, 8, 128, 4 * 2048) > 0
    assert lib.mie_decode_scratch_bytes(-1, 32, 8, 128, 0) == 0


def test_argument_errors_are_reported_on_the_host(library):
    lib = _lib.load()
    empty_view = _lib.View4T(None, (ctypes.c_int64 * 4)(0, 0, 0, 0))
    empty_index = _lib.IndexT(None, 0, 0, 0)
    code = lib.mie_write_decode_kv(empty_view, empty_view, empty_index, empty_index, empty_index, empty_view,
                                   empty_view, 1, 1, 128, 16, 4, 1, 3, None, None)
    assert code == -1
    assert b"elem_bytes" in lib.mie_last_error()
    with pytest.raises(ValueError):
        _lib.check(code)


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "libmie_b200.so")
    with pytest.raises(_lib.MieLibraryError, match="no CPU or PyTorch fallback"):
        _lib.load()


def test_library_path_override(monkeypatch, tmp_path):
    """``MIE_LIBRARY_PATH`` points the binding at a build kept elsewhere; a wrong path fails as loudly."""

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setenv("MIE_LIBRARY_PATH", str(build.LIB_PATH))
    assert _lib.library_path() == build.LIB_PATH and _lib.load().mie_version() >= 1
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setenv("MIE_LIBRARY_PATH", str(tmp_path / "elsewhere.so"))
    with pytest.raises(_lib.MieLibraryError, match="elsewhere.so is missing"):
        _lib.load()


def test_weights_are_requested_early_only_on_request(library):
    """``MIE_GEMM_STATIC_WEIGHTS`` is a promise of the caller, not the default (an empty product returns before any
    launch, after its flags were looked at)."""

    lib = _lib.load()
    aligned = ctypes.c_void_p(4096)

    def gemm(flags):
        return lib.mie_fp8_gemm(aligned, 128, aligned, 1, aligned, 128, aligned, 1, aligned, 128, 1, 0, 128, 128, 0, flags,
                                None, None)

    assert "MIE_GEMM_STATIC_WEIGHTS 2" in HEADER.read_text() and _lib.GEMM_STATIC_WEIGHTS == 2
    assert [gemm(flags) for flags in (0, 1, 2, 3, 4)] == [0, 0, 0, 0, -1]


def test_misaligned_cache_writes_are_refused(library):
    """The q/k/v rows are read and written eight bytes at a time; every operand is checked on the host (no rows here)."""

    lib = _lib.load()
    index = _lib.IndexT(4096, 0, 1, 1)

    def view(address):
        return _lib.View4T(address, (ctypes.c_int64 * 4)(2048, 2048, 128, 1))

    def calls(norms=4096, rope=4096, queries=4096, pages=4096, pool=4096, scales=4096):
        shared = (norms, norms, rope, 64, index, index, index, queries)
        yield lib.mie_qkv_norm_rope_write(4096, 384, *shared, view(pages), view(4096), 0, 1, 1, 16, 1, 1, 1, 1e-6, None, None)
        yield lib.mie_qkv_norm_rope_write_kv8(4096, 384, *shared, pool, 4096, scales, 0, 1, 1, 1, 1, 1, 1e-6, None, None)
        product = (4096, 128, 4096, 1, 4096, 128, 4096, 1)
        sizes = (0, 128, 1, 1, 16, 1, 1, 1, 1e-6, 0, 0, None, None)
        yield lib.mie_fp8_gemm_qkv(*product, *shared, view(pages), view(4096), None, 0, None, *sizes)
        yield lib.mie_fp8_gemm_qkv(*product, *shared, view(4096), view(4096), pool, 4096, scales, *sizes)

    assert list(calls()) == [0, 0, 0, 0]
    for name in ("norms", "rope", "queries"):
        assert list(calls(**{name: 4096 + 2})) == [-1, -1, -1, -1], name
    assert list(calls(pages=4096 + 4)) == [-1, 0, -1, 0]
    for name in ("pool", "scales"):
        assert list(calls(**{name: 4096 + 2})) == [0, -1, 0, -1], name


@pytest.mark.parametrize("gated,n,k,tokens", [
    # (weight, token counts at which the finished projection measured faster by more than 2 %, and where slower)
    (0, 6144, 2560, {1: 1, 32: 1, 48: 1, 128: 0}), (0, 6144, 512, {1: 1, 32: 1, 64: 0, 65: 0}),
    (0, 1536, 2560, {17: 1, 64: 1, 96: 1}), (0, 10240, 4096, {1: 1, 33: 0, 128: 0}), (0, 4096, 1024, {1: 1, 64: 1, 128: 1}),
    (1, 19456, 2560, {1: 1, 32: 1, 33: 0, 128: 0}), (1, 18688, 4096, {1: 0, 32: 0, 64: 1}),
    (1, 1024, 8192, {1: 0, 32: 0, 64: 0, 128: 0}), (1, 6144, 4096, {1: 1, 64: 1, 128: 1}),
    (1, 1536, 1024, {1: 1, 64: 1, 65: 0, 128: 0}), (1, 2048, 4096, {1: 1, 32: 1, 48: 0, 96: 0}),
    (1, 4864, 2560, {1: 1, 33: 1, 128: 1})])
def test_where_finished_projections_pay(library, gated, n, k, tokens):
    lib = _lib.load()
    for m, pays in tokens.items():
        assert lib.mie_fp8_gemm_finish_pays(m, n, k, gated, 0) == pays, (m, n, k)
    assert lib.mie_fp8_gemm_finish_pays(129, n, k, gated, 0) == 0 and lib.mie_fp8_gemm_finish_pays(0, n, k, gated, 0) == 0
