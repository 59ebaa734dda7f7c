// How the step kernels split a grid among CTAs: z planes per CTA.  Plain functions
// of the grid and of how many CTAs the GPU holds at once (slots).
#pragma once

#include <algorithm>
#include <cmath>

namespace kh {

inline long long plan_tiles(int nx, int ny, int tile_x, int tile_y) {
  return (long long)((nx + tile_x - 1) / tile_x) * ((ny + tile_y - 1) / tile_y);
}

// General TMA-staged kernel (kh_tma.cu), which reads one curl-source plane more than
// it updates: 10 planes (a measured optimum on 128- and 256-plane grids: that halo
// plane against enough CTAs to balance the SMs), fewer when the launch would not fill
// two rounds of resident CTAs.  At the reduced-state kernel's depths, µs a step: FP32
// 160×160×96 with the CPU-path semantics 93.8, 89.5 at these; FP64 256×256×128 with σ 656
// and 634, 160×160×96 periodic with χ3 383 and 363.
inline int general_zplanes(int nz, long long tiles, int slots) {
  const long long fill = tiles * nz / (2LL * std::max(1, slots));
  return int(std::min<long long>(nz, std::max(2LL, std::min<long long>(10, fill))));
}

// CTAs that a launch can have along z.
constexpr int kMaxGridZ = 65535;

// Time of a launch of FP64 chunks of z planes, in planes of a full SM: bound by
// arithmetic, so a round of resident CTAs takes its planes times its CTAs per SM, a
// CTA alone on its SM 1.4 times its share; a CTA's start costs 0.3 planes.
inline double reduced_cost_f64(int nz, long long tiles, int slots, int sms, int z) {
  const long long ctas = tiles * ((nz + z - 1) / z), rounds = ctas / slots;
  const int per_sm = std::max(1, slots / sms), last = int((ctas % slots + sms - 1) / sms);
  return (z + 0.3) * (double(rounds * per_sm) + (last == 0 ? 0.0 : std::max(1.4, double(last))));
}

inline int reduced_zplanes_f64(int nz, long long tiles, int slots, int sms, bool cpml) {
  // Without CPML all planes cost the same and deeper chunks save starts and halo
  // planes.  With it, chunks of two balance the planes inside and outside best, unless
  // their last round of CTAs is nearly empty.  Another depth than two has to promise
  // more than the estimate is off by.  µs a step at 2 / 3 / 4 / 5 / 6 planes, without
  // CPML: 64³ 35.7 / 36.7 / 32.3 / 37.2 / 41.5, 100³ 104 / 100 / 98 / 119 / 97, 181×97×75 113 /
  // 119 / 116 / 122 / 115, 240×144×96 265 / 257 / 259 / 248 / 267, 320×192×128 561 / 541 /
  // 539 / 532 / 523; with: 64³ 54.5 / 56.1 / 52.9 / 62.1 / 75.0, 100³ 155 / 160 / 166 / 178 /
  // 166, 181×97×75 157 / 164 / 165 / 180 / 182, 240×144×96 333 / 334 / 336 / 338 / 348,
  // 320×192×128 655 / 645 / 652 / 644 / 650.
  int best = std::min(2, nz);
  const double two = reduced_cost_f64(nz, tiles, slots, sms, best);
  double least = (cpml ? 0.9 : 0.95) * two;
  for (int z = 3; z <= std::min(6, nz); ++z) {
    const double c = reduced_cost_f64(nz, tiles, slots, sms, z);
    if (c < least) {
      least = c;
      best = z;
    }
  }
  return best;
}

inline int reduced_zplanes_f32(int nz, long long tiles, int slots) {
  // A plane costs a CTA about 1.4 µs whatever else runs, its start about three
  // planes; more rounds of CTAs cost less than their number (the SMs overlap them).
  // The optimum of that grows with the square root of the rounds at one plane per
  // CTA (320×192×128, 96 steps: 15.66 / 15.35 / 15.04 / 15.04 / 15.12 / 15.36 ms at 3 /
  // 4 / 5 / 6 / 7 / 10 planes; 200×200×64: 23.97 / 23.58 / 22.96 / 23.07 / 23.40 at 3 - 7).
  const double rounds = double(tiles) * nz / double(slots);
  auto ctas = [&](int z) { return tiles * ((nz + z - 1) / z); };
  const int best = int(std::max(2.0, std::min(7.0, std::floor(1.25 * std::sqrt(rounds) + 0.5))));
  const double many = (best + 3) * (1.15 + 0.3 * double(ctas(best)) / double(slots));
  // … unless all CTAs (but a few of the last, shorter ones) are resident at once at
  // a depth that costs clearly less (96³, 64 steps: 3.87 ms at 5 planes, 4.05 at 2;
  // 181×97×75, where it does not: 6.09 ms at 3 planes, 6.72 at 7).
  for (int z = 1; z <= 10; ++z) {
    const double r = double(ctas(z)) / double(slots);
    if (r > 1.06) continue;
    if ((z + 3) * (r > 1.0 ? 1.1 : 1.0) < 0.925 * many) return std::min(z, nz);
    break;
  }
  return std::min(best, nz);
}

// Reduced-state kernel (kh_lean.cu).
inline int reduced_zplanes(int nz, long long tiles, int slots, int sms, bool fp64, bool cpml) {
  const int z = fp64 ? reduced_zplanes_f64(nz, tiles, slots, sms, cpml) : reduced_zplanes_f32(nz, tiles, slots);
  return std::max(z, (nz + kMaxGridZ - 1) / kMaxGridZ);
}

}  // namespace kh
