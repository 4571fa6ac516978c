"""The sample streams with precomputed reciprocals (csrc/sampler.cuh) against
wpbr_sampling.h: equal bits over pass counts that are powers of two, primes,
squares, one and large, and both sampler modes; and the division they rest on
at the edges of its range."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "sampler.cuh"
using namespace wpbr;
extern "C" {
void divs(long n, unsigned d, const unsigned* x, unsigned* q, unsigned* r) {
  const FastDiv f = fast_div(d);
  for (long i = 0; i < n; ++i) q[i] = div_mod(x[i], f, r + i);
}
int samples(unsigned seed, unsigned stream, unsigned spp, unsigned arrays, long n, const unsigned* pix, const unsigned* pass) {
  const wpbr_rng::Stream s{seed, stream, spp, arrays};
  const Sampler S = make_sampler(s);
  int bad = 0;
  for (long i = 0; i < n; ++i)
    for (unsigned dim = 0; dim < 4; ++dim) {
      float a, b, c, d;
      sample2d(S, pix[i], pass[i], dim, &a, &b);
      wpbr_rng::sample2d(s, pix[i], pass[i], dim, &c, &d);
      const float e = sample1d(S, pix[i], pass[i], dim), f = wpbr_rng::sample1d(s, pix[i], pass[i], dim);
      bad += memcmp(&a, &c, 4) || memcmp(&b, &d, 4) || memcmp(&e, &f, 4);
    }
  return bad;
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sampler")
    (d / "s.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "woodenpbrengine_gb300", "csrc"), str(d / "s.cpp"), "-o", str(d / "s.so")],
                   check=True)
    return C.CDLL(str(d / "s.so"))


def up(a):
    return a.ctypes.data_as(C.POINTER(C.c_uint))


@pytest.mark.parametrize("d", [1, 2, 3, 7, 16, 255, 1920, 65535, 65536, 65537, 10 ** 9 + 7, 2 ** 31 - 1, 2 ** 31, 2 ** 32 - 1])
def test_division(lib, d):
    rng = np.random.default_rng(d)
    near = np.arange(-3, 4, dtype=np.int64)
    mult = (rng.integers(0, max(1, (1 << 32) // d), 2000).astype(np.int64) * d)[:, None] + near
    x = np.concatenate([rng.integers(0, 1 << 32, 100000), mult.ravel(), (1 << 32) - 1 - np.arange(5)])
    x = x[(x >= 0) & (x < 1 << 32)].astype(np.uint32)
    q, r = np.empty_like(x), np.empty_like(x)
    lib.divs(C.c_long(x.size), C.c_uint(d), up(x), up(q), up(r))
    assert np.array_equal(q, x // np.uint32(d)) and np.array_equal(r, x % np.uint32(d))


@pytest.mark.parametrize("spp", [1, 2, 3, 4, 5, 12, 16, 17, 36, 64, 97, 1000, 4096, 99991])
@pytest.mark.parametrize("arrays", [0, 1])
def test_samples(lib, spp, arrays):
    rng = np.random.default_rng(spp)
    n = 3000
    pix = rng.integers(0, 1 << 32, n).astype(np.uint32)
    pix[: n // 2] %= 1 << 21
    passes = rng.integers(0, spp, n).astype(np.uint32)
    assert lib.samples(C.c_uint(5), C.c_uint(9), C.c_uint(spp), C.c_uint(arrays), C.c_long(n), up(pix), up(passes)) == 0
