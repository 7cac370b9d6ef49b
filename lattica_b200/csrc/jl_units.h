// Work split of the JL kernels (jl.cu), on the host alone: units of 32 columns over
// persistent CTAs of some producer warps, one CTA per SM at a time.
#pragma once
#include <stdint.h>

namespace grid {

constexpr uint32_t kUnitCols = 32;  // columns per unit (K of one MMA)
// Units one CTA may accumulate: a packed byte is at most 2 (1 + 4 + 16 + 64) = 170, a byte
// of a word 255, and 170 * 255 * 2^16 stays below 2^32, the accumulators' wrap.
constexpr unsigned long long kMaxUnitsPerCta = (1ull << 16) / kUnitCols;

// CTAs for nunits units: one per SM (or per unit, if fewer), and where those would
// accumulate past their bound as many more as fill every SM again. The units are shared
// out evenly, so a few CTAs in a wave of their own would take as long as all of the first
// (projection of r = 64, n = 2304, 148 CTAs: 0.46 ms; of n = 2400 0.93 on 151, 0.49 on 296).
// nunits at most 2^31 (parts_per_launch), so that unit indices fit 32 bits past the last turn.
inline unsigned unit_grid(unsigned long long nunits, int warps, int num_sms) {
  const unsigned long long sms = (unsigned long long)num_sms;
  const unsigned long long per_cta = kMaxUnitsPerCta / warps * warps;
  const unsigned long long need = (nunits + per_cta - 1) / per_cta;
  const unsigned long long all = (need + sms - 1) / sms * sms;
  return (unsigned)(all < nunits ? all : nunits);
}

// Parts of per_part units that one launch takes (billions of short parts take several);
// 0 if a single part is too long.
inline unsigned long long parts_per_launch(unsigned long long per_part,
                                           unsigned long long num_parts) {
  const unsigned long long fit = (1ull << 31) / per_part;
  return fit < num_parts ? fit : num_parts;
}

}  // namespace grid
