"""CPU: accuracy of the arithmetic that the kernels build on (common.cuh, fft_reg.cuh), compiled for
the host with nvcc and run on random values against long double.

The bounds compare a formula with the plain one it stands for, evaluated beside it on the same
values, so they hold for any correct rounding of either:

* pspec_product in FP32 against complex coefficients rounded once: its phases carry two more
  roundings of a cross coefficient, so with the coefficient's own rounding and those of the product
  and the sum at least as many, the variance at most doubles: sqrt(2).
"""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "solver_gb300" / "csrc"

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <cuda_runtime.h>
#include "fft_reg.cuh"
namespace peec { int fail_cuda(cudaError_t, const char*, const char*, int) { return 0; } }
using namespace peec;

static std::mt19937_64 gen(7);
static double normal() { static std::normal_distribution<double> n; return n(gen); }
static double angle() { static std::uniform_real_distribution<double> u(0, 6.283185307179586); return u(gen); }
static c64 unit() { const double t = angle(); return mk<double>(cos(t), sin(t)); }

static void product() {
  double e[2] = {0, 0};
  auto f32 = [](c64 z) { return mk<float>((float)z.x, (float)z.y); };
  for (int i = 0; i < 300000; ++i) {
    const c64 E[3] = {unit(), unit(), unit()};
    float r[6];
    c32 a[3];
    for (float& v : r) v = (float)normal();
    for (c32& v : a) v = f32(mk<double>(normal(), normal()));
    const int at[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
    c32 c[3][3], b[3] = {a[0], a[1], a[2]};
    c64 S[3][3], ex[3];
    for (int f = 0; f < 3; ++f) {
      ex[f] = mk<double>(0, 0);
      for (int g = 0; g < 3; ++g) {
        S[f][g] = f == g ? mk<double>(r[f], 0) : cscale(cmulc(E[f], E[g]), (double)r[at[f][g]]);
        c[f][g] = f32(S[f][g]);
        ex[f] = ex[f] + S[f][g] * mk<double>(a[g].x, a[g].y);
      }
    }
    const c32 ey = f32(E[0]), exx = f32(E[1]), ez = f32(E[2]);
    pspec_product<float>(r, cmulc(ey, exx), cmulc(ey, ez), cmulc(exx, ez), b[0], b[1], b[2]);
    for (int f = 0; f < 3; ++f) {
      const c32 t = c[f][0] * a[0] + c[f][1] * a[1] + c[f][2] * a[2];
      e[0] += pow(t.x - ex[f].x, 2) + pow(t.y - ex[f].y, 2);
      e[1] += pow(b[f].x - ex[f].x, 2) + pow(b[f].y - ex[f].y, 2);
    }
  }
  printf("product %.17g\n", sqrt(e[1] / e[0]));
}

static long double value(ff a) { return (long double)a.hi + (long double)a.lo; }

static void complex_products() {
  double e[2] = {0, 0};
  for (int i = 0; i < 500000; ++i) {
    const c64 w = unit();
    const cff a = mk<ff>(ff(normal()), ff(normal())), b = mk<ff>(ff(w.x), ff(w.y));
    const cff p[2] = {a * b, cmulc(a, b)};
    for (int conj = 0; conj < 2; ++conj) {
      const ff by = conj ? -b.y : b.y;
      const ff plain[2] = {a.x * b.x - a.y * by, a.x * by + a.y * b.x};
      const ff got[2] = {p[conj].x, p[conj].y};
      const long double ex[2] = {value(a.x) * value(b.x) - value(a.y) * value(by),
                                 value(a.x) * value(by) + value(a.y) * value(b.x)};
      for (int k = 0; k < 2; ++k) {
        e[0] += powl(value(plain[k]) - ex[k], 2);
        e[1] += powl(value(got[k]) - ex[k], 2);
      }
    }
  }
  printf("ff_product %.17g\n", sqrt(e[1] / e[0]));
}

static void sums(int terms) {
  double e[2] = {0, 0};
  for (int i = 0; i < 400000 / terms; ++i) {
    const cff zero = mk<ff>(ff(0.f, 0.f), ff(0.f, 0.f));
    cff got[2] = {zero, zero}, plain[2] = {zero, zero};
    long double ex[2][2] = {{0, 0}, {0, 0}};
    for (int t = 0; t < terms; ++t) {
      const cff u = mk<ff>(ff(normal()), ff(normal())), x = mk<ff>(ff(normal()), ff(normal()));
      cmac(got[0], u, x);
      cmac_conj(got[1], u, x);
      for (int conj = 0; conj < 2; ++conj) {
        const ff uy = conj ? -u.y : u.y;
        plain[conj].x = plain[conj].x + (u.x * x.x - uy * x.y);
        plain[conj].y = plain[conj].y + (u.x * x.y + uy * x.x);
        ex[conj][0] += value(u.x) * value(x.x) - value(uy) * value(x.y);
        ex[conj][1] += value(u.x) * value(x.y) + value(uy) * value(x.x);
      }
    }
    for (int c = 0; c < 2; ++c) {
      e[0] += powl(value(plain[c].x) - ex[c][0], 2) + powl(value(plain[c].y) - ex[c][1], 2);
      e[1] += powl(value(got[c].x) - ex[c][0], 2) + powl(value(got[c].y) - ex[c][1], 2);
    }
  }
  printf("ff_sums_%d %.17g\n", terms, sqrt(e[1] / e[0]));
}

static void lanes() {
  double e[2] = {0, 0};
  for (int i = 0; i < 100000; ++i) {
    ffsum f[32];
    double d[32];
    long double ex = 0;
    for (int l = 0; l < 32; ++l) {
      const ff v(normal() * pow(2.0, 8 * normal()));
      f[l] = ffsum_of(v);
      d[l] = (double)v;
      ex += value(v);
    }
    for (int s = 16; s >= 1; s >>= 1)
      for (int l = 0; l < s; ++l) {
        f[l] = f[l] + f[l + s];
        d[l] = d[l] + d[l + s];
      }
    const double scale = fabs((double)ex);
    e[0] += powl((d[0] - ex) / scale, 2);
    e[1] += powl((ffsum_double(f[0]) - ex) / scale, 2);
  }
  printf("lanes %.17g\n", sqrt(e[1] / e[0]));
}

int main() {
  product();
  lanes();
  sums(8);
  sums(64);
  complex_products();
  return 0;
}
"""


@pytest.fixture(scope="module")
def measured(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc is not installed")
    d = tmp_path_factory.mktemp("arith")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-Xcompiler", "-ffp-contract=off", "-I", str(CSRC), "-o", str(d / "t"),
                    str(d / "t.cu")], check=True, capture_output=True, text=True)
    out = subprocess.run([str(d / "t")], check=True, capture_output=True, text=True).stdout
    return {k: float(v) for k, v in (line.split() for line in out.splitlines())}


def test_block_product(measured):
    assert measured["product"] <= 2 ** 0.5, measured


def test_float_float_complex_product(measured):
    assert measured["ff_product"] <= 1.05, measured


@pytest.mark.parametrize("terms", [8, 64])
def test_float_float_sums_of_products(measured, terms):
    assert measured[f"ff_sums_{terms}"] <= 1.05, measured


def test_lane_sums(measured):
    assert measured["lanes"] <= 1.05, measured
