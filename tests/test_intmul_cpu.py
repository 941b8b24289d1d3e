"""The integer FP64 multiplication (mfe_intmul.cuh), compiled for the host,
against the processor's: random mantissas, few-bit mantissas (exact products
and ties) and runs of ones (carries into the next binade)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#define __host__
#define __device__
#define __forceinline__ inline
#include "mfe_intmul.cuh"
#include <cstdio>
#include <cstring>
#include <random>
static std::mt19937_64 gen(1);
static double make(uint64_t frac)
{
  const uint64_t bits = (gen() & 1) << 63 | (uint64_t)(1023 - 300 + gen() % 600) << 52 | (frac & ((1ull << 52) - 1));
  double d;
  memcpy(&d, &bits, 8);
  return d;
}
static long bad = 0;
static void check(double a, double b)
{
  uint64_t x, y, z;
  memcpy(&x, &a, 8);
  memcpy(&y, &b, 8);
  uint32_t hi, lo;
  mfe::intmul(mfe::intmul_split(x >> 32, x), mfe::intmul_split(y >> 32, y), hi, lo);
  const volatile double p = a * b;
  const double q = p;
  memcpy(&z, &q, 8);
  if (z != ((uint64_t)hi << 32 | lo) && bad++ < 5) printf("%a * %a = %a, got %08x%08x\n", a, b, q, hi, lo);
}
int main()
{
  for (int i = 0; i < 5000000; ++i) check(make(gen()), make(gen()));
  for (int n = 0; n <= 52; ++n)
    for (int m = 0; m <= 52; ++m)
      for (int i = 0; i < 500; ++i) check(make(gen() << (52 - n)), make(gen() << (52 - m)));
  for (int i = 0; i < 2000000; ++i) {
    auto run = [] { return gen() % 2 ? (1ull << 52) - (1ull << (gen() % 52)) : (1ull << (gen() % 52)) - gen() % 3; };
    check(make(run()), make(run()));
  }
  return bad != 0;
}
'''


def test_integer_product_is_the_rounded_product(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "intmul.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "intmul"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "minife_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
