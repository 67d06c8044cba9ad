// ytf_radii.h -- the distinct radii of a pixel set (host).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

namespace ytf {

// every bit of the pattern into the low bits: radii of round coordinates (whole and half units, powers of two)
// differ in the high bits of their patterns alone
inline uint64_t radius_hash(double r) {
  uint64_t h;
  std::memcpy(&h, &r, 8);
  h ^= h >> 32;
  h *= 0x9E3779B97F4A7C15ull;
  h ^= h >> 29;
  h *= 0x9E3779B97F4A7C15ull;
  return h ^ h >> 32;
}

// distinct radii hypot(x_i, y_j) in first-occurrence order over (i fastest, j), as the
// reference, and each pixel's index into them (open addressing by the radius' bits: no allocation per
// radius, as a node-based map makes). A NaN is a radius of its own. Returns the slots looked at.
inline long radii_map(int nx, const double* xs, int ny, const double* ys, std::vector<double>& ur, std::vector<int>& rmap) {
  const long npix = (long)nx * ny;
  long probes = 0;
  ur.clear();
  rmap.assign(npix, 0);
  size_t cap = 16;
  while (cap < 2 * (size_t)npix) cap *= 2;
  std::vector<int> slot(cap, -1);
  for (int j = 0; j < ny; ++j)
    for (int i = 0; i < nx; ++i) {
      const double r = std::hypot(xs[i], ys[j]);
      int& at = rmap[i + (long)nx * j];
      if (std::isnan(r)) {
        at = (int)ur.size();
        ur.push_back(r);
        continue;
      }
      size_t q = (size_t)radius_hash(r) & (cap - 1);
      for (++probes; slot[q] >= 0 && ur[slot[q]] != r; ++probes) q = (q + 1) & (cap - 1);
      if (slot[q] < 0) {
        slot[q] = (int)ur.size();
        ur.push_back(r);
      }
      at = slot[q];
    }
  return probes;
}

}  // namespace ytf
