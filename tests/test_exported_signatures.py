"""The types that the kernel libraries' functions are called with, read from their declarations (no GPU needed)."""
import ctypes
import re

import pytest

from cisr_b200.ops import build


def test_every_exported_function_of_every_source_has_its_types():
    for source in sorted(build.CSRC.glob("*.cu")):
        declared = sum(len(re.findall(r"^CISR_EXPORT", p.read_text(), re.MULTILINE)) for p in build.source_closure(source))
        assert declared == len(build.exported_signatures(source)) > 0, source.name


def test_kinds_of_parameters(tmp_path, monkeypatch):
    monkeypatch.setattr(build, "CSRC", tmp_path)
    (tmp_path / "a.cu").write_text('#include "b.cuh"\nCISR_EXPORT int f(const void* a, float* b, int c, float d,\n  double e, long long g, void* s) {\n}\n')
    (tmp_path / "b.cuh").write_text("CISR_EXPORT void g() { }\nCISR_EXPORT long long h(int n) { return n; }\n")
    p = ctypes.c_void_p
    assert build.exported_signatures(tmp_path / "a.cu") == {
        "f": (ctypes.c_int, [p, p, ctypes.c_int, ctypes.c_float, ctypes.c_double, ctypes.c_longlong, p]), "g": (None, []), "h": (ctypes.c_longlong, [ctypes.c_int])}
    (tmp_path / "a.cu").write_text("CISR_EXPORT int f(unsigned n) {\n}\n")
    with pytest.raises(build.BuildError):
        build.exported_signatures(tmp_path / "a.cu")


def test_an_address_is_passed_whole_and_undeclared_functions_are_refused():
    lib = build.load_library("gemm_tcgen05.cu")
    assert lib.cisr_gemm_tcgen05.argtypes[0] is ctypes.c_void_p and lib.cisr_gemm_tcgen05(1 << 47, 1 << 47, 1 << 47, 0, 8, 8, 0, 1.0, 0) == 0      # no rows: nothing is done
    with pytest.raises(AttributeError):
        lib.cisr_not_there
    with pytest.raises(ctypes.ArgumentError):
        lib.cisr_gemm_tcgen05(0.5, 0, 0, 0, 8, 8, 0, 1.0, 0)


def test_other_threads_find_a_function_only_with_its_types():
    path = build.load_library("gemm_tcgen05.cu")._name
    found = []

    class Watched(dict):
        def __getitem__(self, name):                     # what another thread would find while this one looks the types up
            found.append(vars(lib).get(name))
            return dict.__getitem__(self, name)

    lib = build.KernelLibrary(path, Watched(build.exported_signatures(build.CSRC / "gemm_tcgen05.cu")))
    fn = lib.cisr_gemm_tcgen05
    assert found == [None] and vars(lib)["cisr_gemm_tcgen05"] is fn and fn.argtypes[0] is ctypes.c_void_p and lib.cisr_gemm_tcgen05 is fn
