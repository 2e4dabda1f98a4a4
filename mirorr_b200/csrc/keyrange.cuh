// keyrange.cuh -- the key ranges of the LTS threshold's radix select (lts.cu).
//
// A key is the bit pattern of a non-negative FP64 residual (NaN included, with
// either sign).  Each pass counts the keys of a range [lo, hi] in kKeyBins bins
// and goes on with the bin that holds the rank.  Host and device code.
#pragma once

#include "tfm.cuh"  // MB2_HD

namespace mb2 {

constexpr int kKeyBins = 2048;
// The first histogram's keys: 64 bins per octave over [2^-12, 2^20) mm^2 (a
// residual's bit pattern above kKeyLo in steps of 2^46), one bin below and one
// above.
constexpr unsigned long long kKeyLo = (1023ULL - 12ULL) << 52;
constexpr int kKeyShift = 46;

// Bin of a key in the first histogram, and the keys [lo, hi] of a bin.
MB2_HD unsigned int first_bin(unsigned long long key) {
  if (key < kKeyLo) return 0;
  const unsigned long long b = (key - kKeyLo) >> kKeyShift;
  return b < (unsigned long long)(kKeyBins - 2) ? (unsigned int)b + 1u : (unsigned int)(kKeyBins - 1);
}
MB2_HD void first_range(int bin, unsigned long long &lo, unsigned long long &hi) {
  if (bin == 0) {
    lo = 0;
    hi = kKeyLo - 1;
  } else {
    lo = kKeyLo + ((unsigned long long)(bin - 1) << kKeyShift);
    hi = bin == kKeyBins - 1 ? ~0ULL : lo + ((1ULL << kKeyShift) - 1);
  }
}

// Width 2^shift of the bins that [lo, hi] is counted in next.
MB2_HD int range_shift(unsigned long long lo, unsigned long long hi) {
  int shift = 0;
  while (((hi - lo) >> shift) >= (unsigned long long)kKeyBins) ++shift;
  return shift;
}
// [lo, hi] becomes its bin d of width 2^shift, cut at hi: the last bin's width
// may reach beyond it, and beyond the largest 64-bit number.
MB2_HD void range_step(unsigned long long &lo, unsigned long long &hi, int shift, int d) {
  const unsigned long long width = (1ULL << shift) - 1ULL;
  lo += (unsigned long long)d << shift;
  if (hi - lo > width) hi = lo + width;
}

}  // namespace mb2
