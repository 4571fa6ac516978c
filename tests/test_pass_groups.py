"""The rule that sizes a frame's pass groups (csrc/pass_groups.hpp): whole
groups by film size, and never more state than a quarter of the free memory."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "pass_groups.hpp"
extern "C" {
unsigned by_size(unsigned long long pixels, unsigned spp, int spectral) { return wpbr::group_passes(pixels, spp, spectral); }
unsigned within(unsigned k, unsigned long long bytes, unsigned long long room) {
  return wpbr::group_passes_within(k, bytes, room);
}
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("pass_groups")
    (d / "p.cpp").write_text(SRC)
    so = str(d / "p.so")
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "woodenpbrengine_gb300", "csrc"), str(d / "p.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    lib.by_size.argtypes = [C.c_ulonglong, C.c_uint, C.c_int]
    lib.within.argtypes = [C.c_uint, C.c_ulonglong, C.c_ulonglong]
    return lib


@pytest.mark.parametrize("pixels,spp,spectral,want", [
    (1, 1, 0, 1), (1, 100, 0, 8), (1, 100, 1, 4), (1920 * 1080, 16, 0, 8), (1 << 21, 16, 0, 8), ((1 << 21) + 1, 16, 0, 7),
    (3840 * 2160, 3, 0, 2), (1 << 24, 16, 0, 1), ((1 << 24) + 1, 16, 0, 1), (2 ** 32 - 1, 16, 1, 1)])
def test_groups_by_film_size(rule, pixels, spp, spectral, want):
    assert rule.by_size(pixels, spp, spectral) == want


@pytest.mark.parametrize("room", [0, 1, 3 << 20, 1 << 32, 280 << 30])
@pytest.mark.parametrize("pixels,per_pixel", [(64, 240), (1920 * 1080, 240), (1001 * 563, 508)])
def test_groups_leave_three_quarters_of_the_memory(rule, room, pixels, per_pixel):
    k = rule.within(8, pixels * per_pixel, room)
    assert 1 <= k <= 8 and (k - 1) * pixels * per_pixel <= room // 4
    assert k == 8 or k * pixels * per_pixel > room // 4
