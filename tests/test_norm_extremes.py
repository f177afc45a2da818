"""The extremes by which the viscosity norms' maximum pass skips blocks (order keys and extreme_abs,
meshfreetrixi.jl_gb300/csrc/mft_fpbits.h), compiled for the host: the keys order like the values
and convert back; the largest |x - m| over several sets found through their extremes is that over
all elements bit for bit, with empty sets among them (which must not take part), infinities, both
zeros and all elements equal to m."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include "mft_fpbits.h"
using namespace mft::fpbits;
static uint64_t rng = 0x9E3779B97F4A7C15ull;
static uint64_t next() { rng ^= rng >> 12; rng ^= rng << 25; rng ^= rng >> 27; return rng * 2685821657736338717ull; }
static uint64_t bits(double x) { uint64_t b; memcpy(&b, &x, 8); return b; }
static double val(uint64_t b) { double x; memcpy(&x, &b, 8); return x; }
int main() {
  long bad = 0;
  const double special[] = {0.0, -0.0, INFINITY, -INFINITY, 1.0, -1.0, 4.9e-324, 1.7976931348623157e308};
  for (int t = 0; t < 200000; ++t) {
    double x = val(next()), y = val(next());
    if (t < 64) { x = special[t / 8]; y = special[t % 8]; }
    if (isnan(x) || isnan(y)) continue;
    if (order_back(order_bits(bits(x))) != bits(x)) ++bad;
    if (x < y && !(order_bits(bits(x)) < order_bits(bits(y)))) ++bad;
  }
  for (int t = 0; t < 20000; ++t) {
    const int sets = 1 + (int)(next() % 6);
    const bool flat = t % 7 == 0, inf = t % 5 == 0;
    const double m = inf ? 1.0 : (double)(int64_t)next() * 1e-18;
    uint64_t want = 0, got = 0;
    for (int q = 0; q < sets; ++q) {
      uint64_t lo = kLowest, hi = 0;
      const int len = (int)(next() % 4);  // every fourth set empty
      for (int k = 0; k < len; ++k) {
        double x = (double)(int64_t)next() * 1e-18;
        if (flat) x = m;
        if (inf && next() % 3 == 0) x = next() % 2 ? INFINITY : -INFINITY;
        const uint64_t key = order_bits(bits(x)), d = abs_bits(bits(x - m));
        lo = key < lo ? key : lo;
        hi = key > hi ? key : hi;
        want = d > want ? d : want;
      }
      const uint64_t e = extreme_abs(lo, hi, [&](uint64_t b) { return bits(val(b) - m); });
      got = e > got ? e : got;
    }
    if (got != want) ++bad;
  }
  printf("%ld bad\n", bad);
  return bad != 0;
}
"""


def test_extremes(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "ext.cpp", tmp_path / "ext"
    src.write_text(SRC)
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "meshfreetrixi.jl_gb300" / "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
