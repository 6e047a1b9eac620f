"""Accuracy of the double-float arithmetic of df64.cuh, compiled for the host,
against extended precision.

Reciprocal and square root, arguments: 400,000 log-uniform values in 1/7 .. 7.  The root starts from an FP32
reciprocal root up to 2 units in the last place off, CUDA's documented bound
for rsqrtf.  Bars: what the IEEE-rounded forms give on the same arguments, the
division operator (x.hi / y.hi and its remainder over y.hi: at most 2^-46.2,
root mean square 2^-49.05) and the root by __fsqrt_rn and a division (2^-46.4,
2^-49.5).

Face values of the reconstruction, cell value of 0.5 to 1.5 plus a step of at most
a few tenths: kappa 0 limited, kappa 1/3 limited and unlimited.  Bars: what
products and accurate sums of the same terms give (2^-47.2, 2^-49.68)."""
import subprocess

from fvs2d_gb300 import _build

HEAD = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include "df64.cuh"
using fvs::df64;
typedef long double X;
static X val(df64 a) { return X(a.hi) + X(a.lo); }
struct Err {
  double max = 0, sum = 0;
  long n = 0;
  void add(df64 z, X exact) {
    const double d = double(fabsl((val(z) - exact) / exact));
    max = std::max(max, d);
    sum += d * d;
    n++;
  }
  void print(const char* what) const { std::printf("%s %.3f %.3f\n", what, std::log2(max), 0.5 * std::log2(sum / n)); }
};
"""

ROOTS = HEAD + r"""
int main() {
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> u(-std::log(7.0), std::log(7.0));
  Err rcp, root;
  for (int i = 0; i < 400000; i++) {
    const df64 x(std::exp(u(g)));
    rcp.add(fvs::drcp_(x), 1 / val(x));
    float y = float(1 / sqrtl(X(x.hi)));
    for (int k = int(g() % 5) - 2; k; k += k < 0 ? 1 : -1) y = std::nextafter(y, k < 0 ? 0.0f : 4.0f);
    root.add(fvs::dsqrt_from(x, y), sqrtl(val(x)));
  }
  rcp.print("rcp");
  root.print("root");
}
"""

FACES = HEAD + r"""
int main() {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  Err e[3];
  for (int i = 0; i < 300000; i++) {
    const double eps = i % 2 ? 1e-1 : 1e-3, p = 1 + 0.5 * u(g);
    const df64 P(p), Q(p * (1 + eps * u(g))), gx(30 * eps * u(g)), gy(30 * eps * u(g)), dx(0.01 * u(g)), dy(0.01 * u(g));
    const df64 phi(0.5 + 0.495 * u(g)), kh(1.0 / 6.0), omk(2.0 / 3.0);
    const df64 diff(double(Q) - double(P));
    const df64 grad = fvs::dfma(dx, gx, dy * gy), step = fvs::dfma(kh, diff, omk * grad);
    const X xg = val(dx) * val(gx) + val(dy) * val(gy), xs = val(kh) * val(diff) + val(omk) * xg;
    e[0].add(fvs::dfma_big(phi, grad, P), val(P) + val(phi) * xg);
    e[1].add(fvs::dfma_big(phi, step, P), val(P) + val(phi) * xs);
    e[2].add(fvs::dadd_big(P, step), val(P) + xs);
  }
  e[0].print("kappa0");
  e[1].print("limited");
  e[2].print("unlimited");
}
"""


def run(tmp_path, src):
    """{name: (log2 of the largest error, log2 of its root mean square)}"""
    f, exe = tmp_path / "t.cu", str(tmp_path / "t")
    f.write_text(src)
    # (two_prod and two_sum rest on unfused products and sums)
    subprocess.run([_build.nvcc(), "-O2", "-std=c++17", *_build.ARCH, "-Xcompiler", "-ffp-contract=off", "-I", _build.CSRC,
                    str(f), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {p[0]: (float(p[1]), float(p[2])) for p in (line.split() for line in out.splitlines())}


def test_reciprocal_and_root(tmp_path):
    e = run(tmp_path, ROOTS)
    assert e["rcp"][0] <= -46.15 and e["rcp"][1] <= -49.0, e
    assert e["root"][0] <= -46.35 and e["root"][1] <= -49.45, e


def test_face_values(tmp_path):
    for name, (big, rms) in run(tmp_path, FACES).items():
        assert big <= -47.2 and rms <= -49.68, (name, big, rms)
