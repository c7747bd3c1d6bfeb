// Device functions that the tile sweeps (kernels.cu) and the marching kernels
// (march.cu) share: the staggered differences, the boundary ring, receivers.
#pragma once

#include "fwigb_kernels.h"
#include "quotient.h"

namespace fwigb {

constexpr float C1 = 1.125f;          // 9/8  (el_stress.cu:42)
constexpr float C2 = 1.0f / 24.0f;    // 1/24 (el_stress.cu:43)
constexpr float kMega = 1.0e6f;       // MEGA (utilities.h:16)

// Bounded waits: a kernel that has waited this long (global timer) gives up,
// raises its error word and returns instead of hanging.
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Staggered 4th-order differences. Dm uses (i-2, i-1, i, i+1), Dp
// (i-1, i, i+1, i+2); `s` is the stride of the direction and r the
// reciprocal spacing.
__device__ __forceinline__ float sdm(const float* a, int i, int s, float r) {
  return (C1 * (a[i] - a[i - s]) - C2 * (a[i + s] - a[i - 2 * s])) * r;
}
__device__ __forceinline__ float sdp(const float* a, int i, int s, float r) {
  return (C1 * (a[i + s] - a[i]) - C2 * (a[i + 2 * s] - a[i - s])) * r;
}

// Index of cell (z, x) in the per-step boundary ring, or -1. Top and bottom
// bands are stored column by column (5 depths each), left and right bands
// column by column over their height, so a warp of consecutive depths writes
// consecutive words.
__device__ __forceinline__ int ring_index(const Geo& g, int z, int x) {
  if (z < g.rz0 || z > g.rz1 || x < g.rx0 || x > g.rx1) return -1;
  if (z <= g.rz0 + 4) return (x - g.rx0) * 5 + (z - g.rz0);
  if (z >= g.rz1 - 4) return 5 * g.ringW + (x - g.rx0) * 5 + (z - (g.rz1 - 4));
  if (x <= g.rx0 + 4) return 10 * g.ringW + (x - g.rx0) * g.ringH + (z - (g.rz0 + 5));
  if (x >= g.rx1 - 4) return 10 * g.ringW + 5 * g.ringH + (x - (g.rx1 - 4)) * g.ringH + (z - (g.rz0 + 5));
  return -1;
}

// from_bnd of step it for cell (z, x) when it lies in the ring: the stresses
// before the step's update and the velocities of the staged tile
// (Boundary.cu:55-76).
__device__ __forceinline__ void ring_save(const Geo& g, const StoreD& st, int it, int z, int x, float szz, float sxz,
                                          float sxx, float vz, float vx) {
  const int k = ring_index(g, z, x);
  if (k < 0) return;
  float* p = st.base + static_cast<size_t>(it) * 5 * g.ring_len + k;
  p[0] = szz;
  p[g.ring_len] = sxz;
  p[2 * g.ring_len] = sxx;
  p[3 * g.ring_len] = vz;
  p[4 * g.ring_len] = vx;
}

__device__ __forceinline__ bool in_box(int z, int x, int z0, int z1, int x0, int x1) {
  return z >= z0 && z <= z1 && x >= x0 && x <= x1;
}

// Receiver list of the 32 x 8 bin holding (z, x).
__device__ __forceinline__ int2 bin_range(const ShotD& sh, int z, int x) {
  const int b = (z / kBinZ) + (x / kBinX) * sh.nbin_z;
  return make_int2(sh.blk_off[b], sh.blk_off[b + 1]);
}

// First receiver of cell (z, x), as rec_map holds it: -1 for none. (Without a
// map, which costs a dependent load per receiver of the bin.)
__device__ __forceinline__ int first_receiver(const ShotD& sh, int z, int x) {
  if (!in_box(z, x, sh.rbz0, sh.rbz1, sh.rbx0, sh.rbx1)) return -1;
  if (sh.rec_map) return sh.rec_map[(x - sh.rbx0) * (sh.rbz1 - sh.rbz0 + 1) + (z - sh.rbz0)];
  const int2 rr = bin_range(sh, z, x);
  for (int k = rr.x; k < rr.y; ++k) {
    const int r = sh.blk_rec[k];
    if (sh.rec_z[r] == z && sh.rec_x[r] == x) return r | kRecMore;
  }
  return -1;
}

// The receiver after r (a value of first_receiver or of this) on cell (z, x).
__device__ __forceinline__ int next_receiver(const ShotD& sh, int r, int z, int x) {
  if (!(r & kRecMore)) return -1;
  r &= kRecMore - 1;
  if (sh.rec_map) return sh.rec_next[r];
  const int2 rr = bin_range(sh, z, x);  // the bin lists its receivers in ascending order
  for (int k = rr.x; k < rr.y; ++k) {
    const int q = sh.blk_rec[k];
    if (q > r && sh.rec_z[q] == z && sh.rec_x[q] == x) return q | kRecMore;
  }
  return -1;
}

// The recorded sample (utilities.cu:557-567) of cell (z, x) at step it + 1; r
// is the cell's first_receiver.
__device__ __forceinline__ void record(const ShotD& sh, int it, int r, int z, int x, float szz, float sxx) {
  for (; r >= 0; r = next_receiver(sh, r, z, x))
    sh.data[static_cast<size_t>(r & (kRecMore - 1)) * sh.nSteps + it + 1] = szz + 3.0f * sxx;
}

// res_injection (utilities.cu:569-580) of step it at cell (z, x).
__device__ __forceinline__ void inject_res(const ShotD& sh, int it, int r, int z, int x, float& sa, float& xa) {
  for (; r >= 0; r = next_receiver(sh, r, z, x)) {
    const float rv = sh.res[static_cast<size_t>(r & (kRecMore - 1)) * sh.nSteps + it];
    sa += rv;
    xa += 3.0f * rv;
  }
}

}  // namespace fwigb
