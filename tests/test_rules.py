"""The library's decisions that need no device (csrc/rules.h), compiled for the host."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vfs-wind_gb300", "csrc")
SHIM = """
#include "rules.h"
extern "C" {
int t_in_place(int type, int memory_device, int device, uintptr_t address) {
  return vfs::in_place((vfs::MemoryType)type, memory_device, device, address);
}
int t_overlap(size_t a, size_t na, size_t b, size_t nb, size_t c, size_t nc) {
  return vfs::overlap({{(void *)a, na}, {(void *)b, nb}, {(void *)c, nc}});
}
int t_line_columns(int P, int fp64, int cap, int max_threads) { return vfs::line_columns(P, fp64, cap, max_threads); }
}
"""
HOST, DEVICE, MANAGED = 0, 1, 2


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, str(d / "shim.cpp"),
                    "-o", str(d / "shim.so")], check=True)
    L = C.CDLL(str(d / "shim.so"))
    L.t_in_place.argtypes = [C.c_int, C.c_int, C.c_int, C.c_size_t]
    L.t_overlap.argtypes = [C.c_size_t] * 6
    return L


def test_only_reachable_arrays_are_used_in_place(rules):
    """An array of another GPU, of the host or at an address that no FP64 load takes is
    staged, as every array was that a caller could pass before kernels took any in place."""
    at = 0x7f0000001000
    for device in (0, 3):
        for other in (0, 1, 2, 3):
            assert rules.t_in_place(DEVICE, other, device, at) == (other == device)
            assert rules.t_in_place(MANAGED, other, device, at) == 1
            assert rules.t_in_place(HOST, other, device, at) == 0
        for off in range(1, 8):
            assert rules.t_in_place(DEVICE, device, device, at + off) == 0
            assert rules.t_in_place(MANAGED, device, device, at + off) == 0
        assert rules.t_in_place(DEVICE, device, device, at + 8) == 1


def test_the_library_asks_the_rule():
    """No entry point that staged its arrays once decides by the kind of memory alone."""
    src = open(os.path.join(CSRC, "poisson.cu")).read()
    for entry in ("set_nvert", "rhs", "volume_flux", "volume_flux0", "contra2cart", "ib_bc", "solve", "update_pressure",
                  "projection", "divergence", "get_rhs", "apply"):
        start = src.index(f"\nint vfs_poisson_{entry}(")
        body = src[start:src.index("\n}\n", start)]
        assert "in_place(h," in body or "device_view(h," in body or "device_inout(h," in body, entry
        assert "= is_device_ptr(" not in body and "!is_device_ptr(" not in body, entry
    start = src.index("int device_view(")
    assert "is_device_ptr" not in src[start:src.index("int download(", start)]


def test_overlapping_arrays(rules):
    a, n, none = 0x10000, 240, (0, 240)
    for b, nb, want in ((a, n, 1), (a + n, n, 0), (a - 80, 80, 0), (a + n - 8, 80, 1), (a - 80, 88, 1), (a + 8, 16, 1),
                        (a - 8, 400, 1), (0, n, 0)):
        assert rules.t_overlap(a, n, b, nb, *none) == want
        assert rules.t_overlap(b, nb, *none, a, n) == want


def test_line_columns(rules):
    """FP64 blocks stay within the limit without giving up the lanes that four columns
    use; FP32 halves sixteen; a cap holds."""
    limit = 384

    def used(P, c):
        return P * c / ((P * c + 31) // 32 * 32)

    for P in range(1, limit + 1):
        c = rules.t_line_columns(P, 1, 0, limit)
        four = next(t for t in (4, 2, 1) if t * P <= limit or t == 1)
        assert 1 <= c <= 8 and c * P <= limit
        assert used(P, c) >= used(P, four) and c >= four
        assert rules.t_line_columns(P, 0, 0, limit) == next(t for t in (16, 8, 4, 2, 1) if t * P <= limit or t == 1)
        for cap in (1, 2, 3, 4, 6):
            assert rules.t_line_columns(P, 1, cap, limit) <= cap
            assert rules.t_line_columns(P, 0, cap, limit) <= cap
    assert rules.t_line_columns(5, 1, 0, limit) == 6
    assert rules.t_line_columns(77, 1, 0, limit) == 4
