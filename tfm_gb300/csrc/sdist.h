// How k_sdist shares the pairs of a chain out over CTAs; plain C++, so that
// the host can check it at chain lengths that no test would step.
#pragma once

#ifdef __CUDACC__
#define CCPGPU_HD __host__ __device__
#else
#define CCPGPU_HD
#endif

namespace ccpgpu {

constexpr int SDIST_PCHUNK = 256;  // first beads of a CTA's pairs
constexpr int SDIST_SEPS = 128;    // separations

CCPGPU_HD inline long long sdist_tiles(int len, int smax) {
  return (long long)((smax + SDIST_SEPS - 1) / SDIST_SEPS) * ((len + SDIST_PCHUNK - 1) / SDIST_PCHUNK);
}

// First separation and first bead of tile k of a chain. A chain has (len /
// 256)^2 tiles, more than 32 bits hold from 11.9 million beads on.
CCPGPU_HD inline void sdist_tile(long long k, int smax, int &s0, int &p0) {
  const int nsep = (smax + SDIST_SEPS - 1) / SDIST_SEPS;
  const int row = (int)(k / nsep);
  s0 = (int)(k - (long long)row * nsep) * SDIST_SEPS + 1;
  p0 = row * SDIST_PCHUNK;
}

}  // namespace ccpgpu
