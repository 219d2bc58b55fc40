"""sinh and cosh as sums of two floats (csrc/sinhcosh.cuh), compiled for the host
against long double: the stated error bound over the whole range, and the rescaled
mean and variance of the screen, which must be the correctly rounded floats
wherever they are not left to FP64, and left to it rarely."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include "sinhcosh.cuh"
using namespace abc;
int main() {
  std::mt19937_64 gen(1);
  std::uniform_real_distribution<double> U(0, 1);
  long double worst = 0;
  long wrong = 0, left = 0;
  const long n = 4000000;
  for (long it = 0; it < n; ++it) {
    const int kind = it & 3;
    double a = kind == 0 ? std::exp(-20 + 19 * U(gen)) : kind == 1 ? 0.35 * U(gen) + 1e-8 : 0.35 + (kind == 2 ? 3 : 29.64) * U(gen);
    if (U(gen) < 0.5) a = -a;
    const FF u = {(float)a, (float)(a - (double)(float)a)};
    FF s, c;
    if (!sinh_cosh(u, s, c)) return 1;
    const long double x = (long double)u.h + u.l;
    worst = fmaxl(worst, fabsl(((long double)s.h + s.l) / sinhl(x) - 1));
    worst = fmaxl(worst, fabsl(((long double)c.h + c.l) / coshl(x) - 1));
    if (s.h != (float)((double)s.h + s.l) || c.h != (float)((double)c.h + c.l)) return 2;
    // standardised outputs, scales and means of a surrogate's statistics
    const float mu = (float)(8 * U(gen) - 4), var = (float)std::exp(-9 + 11 * U(gen)), sd = (float)(0.01 + 3 * U(gen));
    const float mean = (float)(6 * U(gen) - 2), sc = (it & 7) ? (float)std::exp(-5 + 10 * U(gen)) : 0.0f;
    float m, v;
    if (!unscale32(mu, var, sd, mean, sc, m, v)) {
      ++left;
      continue;
    }
    const long double y = (long double)mu * sd + mean, vu = (long double)var * sd * sd, ch = (long double)sc * coshl(y);
    if (m != (float)(sc > 0 ? sc * sinhl(y) : y) || v != (float)(sc > 0 ? ch * ch * vu : vu)) ++wrong;
  }
  std::printf("worst 2^%.2Lf, wrong %ld, left to FP64 %ld of %ld\n", log2l(worst), wrong, left, n);
  const float inf = INFINITY;  // refused, not rounded
  float m, v;
  const float bad[][5] = {{NAN, 1, 1, 0, 1}, {1, NAN, 1, 0, 1}, {inf, 1, 1, 0, 1}, {0, 1, 1, 0, 1}, {40, 1, 1, 0, 1},
                          {1, 1, 1e-30f, 0, 1}, {1, 1, 1, 0, 1e-30f}, {1, 1e30f, 1, 0, 1}, {0, 1, 1, 0, 0}, {1, 1, 1, inf, 0}};
  for (const auto& b : bad)
    if (unscale32(b[0], b[1], b[2], b[3], b[4], m, v)) return 3;
  return worst < kSinhCoshErr / 4 && wrong == 0 && left < n / 1000 ? 0 : 4;
}
"""


def test_two_float_sinh_cosh_and_rescaling(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "abc_inference_transcription_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
