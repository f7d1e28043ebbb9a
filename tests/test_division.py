"""The softmax's division (``DivideBy`` in csrc/sbb_math.cuh) against ``/``, bit by bit, on the CPU: the method is IEEE
operations alone, so the header itself is compiled for the host.  Where such a method fails it fails on quotients next to
the middle between two neighbouring numbers, so these are what is tried: for a divisor with significand D the dividends V
with V 2^s = K D + e, K odd, |e| small (K from the inverse of D modulo 2^s)."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

PROGRAM = r"""
#include <cuda_runtime.h>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
template <class To, class From> static To bits(From f) { To t; static_assert(sizeof(t) == sizeof(f), ""); std::memcpy(&t, &f, sizeof t); return t; }
static inline unsigned __float_as_uint(float f) { return bits<unsigned>(f); }
static inline float __uint_as_float(unsigned u) { return bits<float>(u); }
static inline long long __double_as_longlong(double d) { return bits<long long>(d); }
static inline float __frcp_rn(float f) { return 1.f / f; }
static inline double __drcp_rn(double d) { return 1.0 / d; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
#define __log2f std::log2
#include "sbb_math.cuh"

static unsigned long long tried = 0, wrong = 0;
template <class T> void check(T v, T d) {
  const sbb::DivideBy<T> by(d);
  const T want = v / d;
  ++tried;
  if (by(v) != want && wrong++ < 10)
    std::printf("%a / %a: %a, not %a\n", (double)v, (double)d, (double)by(v), (double)want);
}
template <class T, int P> struct Hard {   // P significand bits
  // scale: v = V 2^vs, d = D 2^(1 - P) 2^ds
  static void divisor(uint64_t D, int span, int vs, int ds) {
    if (D % 2 == 0) return;   // (an even one is an odd one with fewer bits: its quotients stay further from the middle)
    const T d = std::ldexp((T)D, 1 - P + ds);
    unsigned __int128 inv = D;
    for (int k = 0; k < 6; ++k) inv *= 2 - D * inv;
    for (int s = P; s <= P + 1; ++s) {
      const unsigned __int128 mod = (unsigned __int128)1 << s;
      for (int e = -span; e <= span; ++e) {
        uint64_t K = (uint64_t)((unsigned __int128)(__int128)-e * inv & (mod - 1));
        if (K < (1ull << P)) K += (uint64_t)mod;
        if (K % 2 == 0 || K >= (1ull << (P + 1))) continue;
        const __int128 num = (__int128)K * D + e;
        const uint64_t V = (uint64_t)(num >> s);
        if (V >> (P - 1) != 1) continue;
        check<T>(std::ldexp((T)V, 1 - P + vs), d);
      }
    }
  }
  static void run(uint64_t divisors, int span) {
    std::mt19937_64 rng(P);
    const uint64_t lo = 1ull << (P - 1), n = lo;
    const int least = sizeof(T) == 4 ? -100 : -900;
    for (uint64_t k = 0; k < divisors; ++k) {
      const uint64_t D = k < divisors / 4 ? lo + n - 1 - k : k < divisors / 2 ? lo + (k - divisors / 4) : lo + rng() % n;
      divisor(D, span, -1, 0);
      divisor(D, span, least, (int)(rng() % 21));   // the smallest dividends that the method takes, larger divisors
    }
    for (uint64_t k = 0; k < divisors; ++k) {
      const T d = std::ldexp((T)(lo + rng() % n), 1 - P + (int)(rng() % 9));
      check<T>(std::ldexp((T)(lo + rng() % n), -P - (int)(rng() % (sizeof(T) == 4 ? 148 : 1073))), d);
      const T all_ones = std::ldexp((T)(2 * lo - 1), 1 - P + (int)(rng() % 9));
      check<T>(std::ldexp((T)(lo + rng() % n), -P), all_ones);
      check<T>((T)0, d);
    }
    check<T>((T)1, (T)1);
  }
};
int main() {
  Hard<float, 24>::run(1 << 19, 24);
  Hard<double, 53>::run(1 << 17, 24);
  std::printf("%llu tried, %llu wrong\n", tried, wrong);
  return wrong != 0;
}
"""


def test_division_by_the_reciprocal_is_the_division(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("needs a host compiler and the CUDA headers")
    src, exe = str(tmp_path / "division.cpp"), str(tmp_path / "division")
    with open(src, "w") as f:
        f.write(PROGRAM)
    # -ffp-contract=off: what is written is what is rounded; -march=native: fma as one instruction where the host has it
    subprocess.run(["g++", "-O2", "-std=c++17", "-march=native", "-ffp-contract=off", "-w", "-I" + os.path.join(cuda, "include"),
                    "-I" + os.path.join(REPO, "streambrain_b200", "csrc"), src, "-o", exe], check=True, timeout=300)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout
    assert int(run.stdout.split()[-4]) > 10_000_000, run.stdout
