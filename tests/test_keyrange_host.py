"""Host-side check of the LTS threshold's key ranges (mirorr_b200/csrc/keyrange.cuh
compiled as plain C++, no GPU).

The radix select narrows a key range pass by pass until few keys, or equal ones,
are left.  Restated here with the same functions, it has to keep the key of the
wanted rank in the range at every pass and end with a range that holds it, for
residuals over all magnitudes, zeros, infinities and NaN of either sign (whose
bit patterns lie where a bin's width reaches beyond 64 bits).
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "keyrange.cuh"

using u64 = unsigned long long;
static const size_t kFew = 512;

static bool select(const std::vector<u64> &keys, size_t rank) {
  std::vector<u64> sorted(keys);
  std::sort(sorted.begin(), sorted.end());
  const u64 want = sorted[rank];
  u64 lo = 0, hi = 0;
  size_t k = rank;
  int shift = 0;
  for (int pass = 0; pass < 8; ++pass) {
    std::vector<size_t> h(mb2::kKeyBins, 0);
    for (u64 q : keys) {
      if (pass == 0) ++h.at(mb2::first_bin(q));
      else if (q >= lo && q <= hi) ++h.at((q - lo) >> shift);
    }
    size_t cum = 0;
    int d = 0;
    while (d < mb2::kKeyBins && cum + h[d] <= k) cum += h[d++];
    if (d == mb2::kKeyBins) return false;  // the rank is not in the range
    k -= cum;
    if (pass == 0) mb2::first_range(d, lo, hi);
    else mb2::range_step(lo, hi, shift, d);
    if (lo > hi || want < lo || want > hi) return false;
    size_t in = 0;
    for (u64 q : keys) in += q >= lo && q <= hi;
    if (in != h[d]) return false;
    if (h[d] <= kFew || lo == hi) return true;
    shift = mb2::range_shift(lo, hi);
  }
  return false;
}

static u64 bits(double v) { u64 b; std::memcpy(&b, &v, 8); return b; }

int main() {
  std::mt19937_64 rng(5);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  int bad = 0, runs = 0;
  for (int kind = 0; kind < 9; ++kind)
    for (int n : {1, 7, 600, 4000, 9000})
      for (int rep = 0; rep < 4; ++rep) {
        std::vector<u64> keys(n);
        for (u64 &q : keys) {
          const double m = std::ldexp(u(rng), (int)(rng() % 80) - 40);
          const u64 pos = 0x7ff8000000000000ULL + rng() % 3, neg = 0xfff8000000000000ULL + rng() % 3;
          switch (kind) {
            case 0: q = bits(m); break;
            case 1: q = bits(u(rng) < 0.7 ? 4.0 : m); break;
            case 2: q = bits(u(rng) < 0.5 ? 0.0 : m); break;
            case 3: q = u(rng) < 0.6 ? 0x7ff0000000000000ULL : bits(m); break;
            case 4: q = u(rng) < 0.6 ? pos : bits(m); break;
            case 5: q = u(rng) < 0.6 ? neg : bits(m); break;
            case 6: q = neg; break;
            case 7: q = u(rng) < 0.5 ? ~0ULL : neg; break;
            default: q = rng(); break;  // any bit pattern
          }
        }
        for (size_t rank : {(size_t)0, (size_t)n / 2, (size_t)(0.9 * n), (size_t)n - 1}) {
          ++runs;
          if (!select(keys, rank)) {
            if (bad++ < 10) std::printf("kind %d n %d rank %zu\n", kind, n, rank);
          }
        }
      }
  std::printf("%d of %d\n", bad, runs);
  return bad ? 1 : 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_rank_stays_in_the_range(tmp_path):
    src = tmp_path / "keyrange.cpp"
    src.write_text(SRC)
    exe = tmp_path / "keyrange"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-x", "c++",
                           "-I", os.path.join(ROOT, "mirorr_b200", "csrc"), str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
