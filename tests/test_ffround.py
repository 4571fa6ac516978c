"""The float-pair forms of the reference's double expressions (csrc/ffround.cuh)
against those expressions: equal bits for every operand, over ordinary values,
the edges of the fast paths' ranges and special values, with the approximate
reciprocals exact and moved two units in the last place either way (the
device's are within one or two)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "geom.cuh"
using namespace wpbr;
#define EACH for (long i = 0; i < n; ++i)
extern "C" {
void f_mul(long n, const float* x, float* a, float* b) { EACH { a[i] = mul_const(x[i], kTwoPiMul); b[i] = mul_const_d(x[i], 2.0 * kPI); } }
void f_log2(long n, const float* x, float* a, float* b) { EACH { a[i] = mul_const(x[i], kLog2eMul); b[i] = mul_const_d(x[i], 1.4426950408889634); } }
void f_div(long n, const float* x, float* a, float* b) { EACH { a[i] = div_const(x[i], kPiDiv); b[i] = div_const_d(x[i], kPI); } }
void f_div2(long n, const float* x, float* a, float* b) { EACH { a[i] = div_const(x[i], kTwoPiDiv); b[i] = div_const_d(x[i], 2.0 * kPI); } }
void f_sqrt1m(long n, const float* x, float* a, float* b) { EACH { a[i] = sqrt_one_minus(x[i]); b[i] = sqrt_one_minus_d(x[i]); } }
void f_sub1(long n, const float* x, float* a, float* b) { EACH { a[i] = 1.0f - x[i]; b[i] = (float)(1.0 - (double)x[i]); } }
void f_rcp(long n, const float* x, float* a, float* b) { EACH { a[i] = 1.0f / x[i]; b[i] = (float)(1.0 / (double)x[i]); } }
void f_lerp(long n, const float* x, const float* y, float* a, float* b) { EACH { a[i] = lerp_to_one(x[i], y[i]); b[i] = lerp_to_one_d(x[i], y[i]); } }
void f_dbs(long n, const float* x, const float* y, float* a, float* b) { EACH { a[i] = div_by_scaled(x[i], kTwoPiSqMul, y[i]); b[i] = div_by_scaled_d(x[i], (2.0 * kPI) * kPI, y[i]); } }
void f_tr(long n, const float* ax, const float* ay, const float* c4, const float* g, float* a, float* b) {
  EACH { a[i] = tr_rcp(kPiMul, ax[i], ay[i], c4[i], g[i]); b[i] = tr_rcp_d(kPI, ax[i], ay[i], c4[i], g[i]); } }
void f_quad(long n, const float* qa, const float* qb, const float* qc, float* a, float* b) {
  EACH {
    float *u = a + 3 * i, *v = b + 3 * i;
    u[1] = u[2] = v[1] = v[2] = 0.0f;
    u[0] = quadratic(qa[i], qb[i], qc[i], u + 1, u + 2);
    const Roots r = quadratic_d(qa[i], qb[i], qc[i]);
    v[0] = r.real;
    v[1] = r.t0;
    v[2] = r.t1;
  } }
}
"""


@pytest.fixture(scope="module", params=["", "-DWPBR_FF_PERTURB=2u", "-DWPBR_FF_PERTURB=-2u"])
def lib(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("ff")
    (d / "ff.cpp").write_text(SRC)
    flags = [f for f in (request.param,) if f]
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-DWPBR_FF_HOST", *flags,
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "woodenpbrengine_gb300", "csrc"),
                    str(d / "ff.cpp"), "-o", str(d / "ff.so")], check=True)
    return C.CDLL(str(d / "ff.so"))


N = 400_000
EDGES = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 1e-45, -1e-45, 1.2e-38, 3.4e38, 0.5, 2.0,
                  1 - 2.0 ** -24, 1 + 2.0 ** -23, 2.0 ** -40, 2.0 ** 40, 2.0 ** -41, 2.0 ** 41, 2.0 ** -24, 2.0 ** 24,
                  2.0 ** -25, 2.0 ** -30, 2.0 ** -29, 2.0 ** -16, 2.0 ** 36, 2.0 ** 60, 2.0 ** -60], np.float32)


def uni(rng, lo, hi):
    return rng.uniform(lo, hi, N).astype(np.float32)


def logu(rng, lo, hi):
    return np.exp2(rng.uniform(lo, hi, N)).astype(np.float32)


def any_bits(rng):
    return rng.integers(0, 1 << 32, N, dtype=np.uint32).view(np.float32)


def edges(*cols):
    """Operands with the special values in every combination at the front."""
    grid = np.meshgrid(*[EDGES] * len(cols), indexing="ij")
    return [np.ascontiguousarray(np.concatenate([g.ravel(), c])) for g, c in zip(grid, cols)]


def same(lib, name, cols, width=1):
    n = cols[0].size
    a, b = np.empty(n * width, np.float32), np.empty(n * width, np.float32)
    p = lambda v: v.ctypes.data_as(C.POINTER(C.c_float))  # noqa: E731
    getattr(lib, name)(C.c_long(n), *[p(c) for c in cols], p(a), p(b))
    ok = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
    bad = np.flatnonzero(~ok)[:3] // width
    assert ok.all(), (name, [[float(c[i]).hex() for c in cols] for i in bad])


@pytest.mark.parametrize("name", ["f_mul", "f_log2", "f_div", "f_div2", "f_sub1", "f_rcp"])
def test_one_operand(lib, name):
    rng = np.random.default_rng(1)
    for x in (uni(rng, -7, 7), logu(rng, -60, 60), -logu(rng, -45, 45), any_bits(rng)):
        if name == "f_rcp":  # a root that is neither denormal nor so large that its reciprocal is
            x = np.clip(np.abs(np.nan_to_num(x)), 2.0 ** -76, 2.0 ** 64).astype(np.float32)
            same(lib, name, [x])
        else:
            same(lib, name, edges(x))


def test_sqrt_one_minus(lib):
    rng = np.random.default_rng(2)
    near = np.float32(1) - logu(rng, -24, -1)
    for x in (uni(rng, 0, 1), logu(rng, -60, 0), near, uni(rng, -1, 2), any_bits(rng)):
        same(lib, "f_sqrt1m", edges(x))


def test_two_operands(lib):
    rng = np.random.default_rng(3)
    for u, c in ((uni(rng, 0, 1), uni(rng, 0, 1)), (logu(rng, -40, 0), logu(rng, -40, 0)),
                 (uni(rng, 0, 1), np.float32(1) - logu(rng, -24, -1)), (any_bits(rng), any_bits(rng))):
        same(lib, "f_lerp", edges(u, c))
    for n, s in ((uni(rng, 0, 9), uni(rng, 0, 1)), (logu(rng, -45, 45), -logu(rng, -45, 45)),
                 (-logu(rng, -60, 60), logu(rng, -60, 60)), (any_bits(rng), any_bits(rng))):
        same(lib, "f_dbs", edges(n, s))


def test_trowbridge_reitz(lib):
    rng = np.random.default_rng(4)
    alpha = uni(rng, 0.04, 1.6)
    for ax, ay, c4, g in ((alpha, alpha, uni(rng, 0, 1), np.float32(1) + logu(rng, -20, 20)),
                          (logu(rng, -20, 12), logu(rng, -20, 12), logu(rng, -35, 6), logu(rng, -6, 40)),
                          (any_bits(rng), any_bits(rng), any_bits(rng), any_bits(rng))):
        same(lib, "f_tr", [ax, ay, c4, g])
    k = EDGES[:19]
    same(lib, "f_tr", [np.ascontiguousarray(g.ravel()) for g in np.meshgrid(k, k, k, k, indexing="ij")])


def test_quadratic(lib):
    rng = np.random.default_rng(5)
    one = np.float32(1) + uni(rng, -1e-6, 1e-6)
    # unit directions at spheres of radius 0.02 .. 3, hit and missed
    o, d = rng.normal(size=(N, 3)) * 6, rng.normal(size=(N, 3))
    r = rng.uniform(0.02, 3, N)
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    near = (-o + rng.normal(size=(N, 3)) * r[:, None] * 0.7)
    aim = (near / np.linalg.norm(near, axis=1, keepdims=True)).astype(np.float32)
    o = o.astype(np.float32)
    for v in (d, aim):
        same(lib, "f_quad", [np.ascontiguousarray((v * v).sum(1)), np.ascontiguousarray(2 * (v * o).sum(1)),
                             np.ascontiguousarray((o * o).sum(1) - (r * r).astype(np.float32))], 3)
    # near-tangent: c within 2^-10 .. 2^-50 of b^2 / 4a, either side
    b = uni(rng, -20, 20)
    c = (b.astype(np.float64) ** 2 / (4 * one.astype(np.float64)) * (1 + rng.choice([-1, 1], N) * np.exp2(rng.uniform(-50, -1, N))))
    same(lib, "f_quad", [one, b, c.astype(np.float32)], 3)
    same(lib, "f_quad", [one, b, (b * b / (4 * one)).astype(np.float32)], 3)
    # scaled objects, tiny and huge coefficients, and any bits
    same(lib, "f_quad", [logu(rng, -26, 26), logu(rng, -26, 26) * rng.choice(np.float32([-1, 1]), N),
                         logu(rng, -26, 26) * rng.choice(np.float32([-1, 1]), N)], 3)
    same(lib, "f_quad", edges(any_bits(rng), any_bits(rng), any_bits(rng)), 3)
