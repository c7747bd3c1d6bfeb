// Marching kernels: a whole pass over time in one launch, for calls whose
// grids are too small to fill the GPU in every sweep.
//
// A sweep of a small grid is all latency: 5-6 us a launch on a 96 x 84 grid as
// on a 192 x 264 one (launch, cold parameter block, barrier set-up, staging
// copy, one wave of tiles), four launches a step. Here each shot's columns are
// cut into strips, one block each, and a block carries its strip through every
// sweep of every step. A strip's stencils reach two columns into the strips beside it, so
// between two sweeps a block waits only for its two neighbours: each block
// publishes the number of sweeps it has finished in a flag word, and starts
// the next sweep when both neighbours have reached its own count (which
// orders their writes before its reads, and their reads before its writes).
// All blocks of a launch are resident together (a cooperative launch). The
// hand-over costs 1.1 us of a sweep, the sweep itself 1-1.5 us at the smallest
// sizes: a step of a 96 x 84 grid takes 9.1 us (21.1 with a launch per sweep),
// of two 192 x 264 grids 15.1 us (23.8), of one 192 x 448 grid 13.0 us (22.7).
//
// A warp takes 32 depths of one column at a time and reads its stencil samples
// from the fields themselves (L1 / L2): at these sizes the fields live in L2,
// and staging would add its own latency.
#include <algorithm>

#include "fwigb_kernels.h"
#include "sweep_cells.cuh"

namespace fwigb {
namespace {

constexpr unsigned kFlagStride = 32;  // words between flags: one 128-byte line each

__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits until a neighbour's flag reaches `count`: bounded by kWaitLimitNs, and
// given up as soon as another block has raised the error word.
__device__ __forceinline__ bool wait_flag(const unsigned* flag, unsigned count, unsigned* err) {
  unsigned long long t0 = 0;
  for (unsigned n = 0;; ++n) {
    if (ld_acquire(flag) >= count) return true;
    if ((n & 63) == 63) {
      if (ld_relaxed(err) != 0) return false;
      const unsigned long long t = global_timer_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > kWaitLimitNs) {
        atomicOr(err, 1u);
        return false;
      }
    }
  }
}

// A block's strip of a shot and its place among the strips.
struct Strip {
  int shot, xa, xb;        // columns [xa, xb) of the shot's sub-grid
  bool left, right;        // has a neighbour
  unsigned* flag;          // its own flag
  int nch;                 // 32-depth chunks down to the last row a sweep touches
};

__device__ __forceinline__ Strip strip_of(const MarchPack& P, unsigned* flags) {
  Strip s;
  s.shot = 0;
  while (s.shot + 1 < P.nshots && static_cast<int>(blockIdx.x) >= P.first[s.shot + 1]) ++s.shot;
  const int j = blockIdx.x - P.first[s.shot], nb = P.first[s.shot + 1] - P.first[s.shot];
  const Geo& g = P.slots[s.shot].g;
  s.xa = static_cast<int>(static_cast<long long>(j) * g.nx / nb);
  s.xb = static_cast<int>(static_cast<long long>(j + 1) * g.nx / nb);
  s.left = j > 0;
  s.right = j + 1 < nb;
  s.flag = flags + static_cast<size_t>(blockIdx.x) * kFlagStride;
  s.nch = (min(g.nz, max(g.zact1, P.slots[s.shot].sh.rbz1) + 1) + 31) / 32;
  return s;
}

// Ends a sweep: publishes `count`, waits for the neighbours. False: give up.
__device__ __forceinline__ bool strip_sync(const Strip& s, unsigned count, unsigned* err) {
  __syncthreads();
  bool ok = true;
  if (threadIdx.x == 0) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(s.flag), "r"(count) : "memory");
    if (s.left) ok = wait_flag(s.flag - kFlagStride, count, err);
  } else if (threadIdx.x == 32) {  // (at least four warps)
    if (s.right) ok = wait_flag(s.flag + kFlagStride, count, err);
  }
  return __syncthreads_and(ok);
}

// A warp's place in its block's list of work: part, then column, then 32-depth
// chunk (chunks fastest), every warp taking every blockDim.x / 32-th item.
struct Item {
  int part, x, ch;
};
__device__ __forceinline__ void step_item(const Strip& s, Item& t, int n) {
  t.ch += n;
  while (t.ch >= s.nch) {
    t.ch -= s.nch;
    if (++t.x >= s.xb) {
      t.x = s.xa;
      ++t.part;
    }
  }
}
// Calls fn(part, z0, x) for the warp's items of `parts` parts, from its first item on.
template <class F>
__device__ __forceinline__ void for_items(const Strip& s, Item t, int parts, F fn) {
  while (t.part < parts) {
    fn(t.part, t.ch * 32, t.x);
    step_item(s, t, blockDim.x >> 5);
  }
}

// What does not change over time, per cell of the strip: the row of the
// boundary ring plus one (0: none) and where the cell lies. In shared memory:
// working it out in every part took a third of its instructions.
constexpr unsigned kRing = (1u << 21) - 1, kDom = 1u << 21, kZp = 1u << 22, kXp = 1u << 23, kXpV = 1u << 24,
                   kInner = 1u << 25, kRec = 1u << 26, kSrc = 1u << 27, kXb = 1u << 28, kZb = 1u << 29;

__device__ unsigned cell_info(const ShotSlot& S, int z, int x) {
  const Geo& g = S.g;
  const ShotD& sh = S.sh;
  if (z >= g.nz) return 0;
  unsigned v = static_cast<unsigned>(ring_index(g, z, x) + 1);
  if (in_box(z, x, g.zi0, g.zi1, g.xi0, g.xi1)) v |= kInner;
  if (z == sh.src_z && x == sh.src_x) v |= kSrc;
  if (first_receiver(sh, z, x) >= 0) v |= kRec;
  if (in_box(z, x, g.zs0, g.zs1, g.xs0, g.xs1)) {
    v |= kDom;
    if (z < g.nPml || z > g.zpml_hi) v |= kZp;
    if (x < g.nPml || x > g.xpml_hi_s) v |= kXp;
    if (x < g.nPml || x > g.xpml_hi_v) v |= kXpV;
    if (x <= g.xband_lo || x >= g.xband_hi) v |= kXb;
    if (z <= g.zband_lo || z >= g.zband_hi) v |= kZb;
  }
  return v;
}

// The shot's arrays as offsets from three bases (the engine lays its 18 fields,
// the media and the sums out one after the other), so that an address takes
// one integer multiply-add instead of a load of its pointer.
enum Field {
  VZ, VX, SZZ, SXX, SXZ, VZ_A, VX_A, SZZ_A, SXX_A, SXZ_A,
  M_VZ_Z, M_VZ_X, M_VX_Z, M_VX_X, M_SZZ_Z, M_SXX_X, M_SXZ_Z, M_SXZ_X
};
enum Medium { LAM = 0, L2M = 3, AMU = 4, BYA = 5, BYB = 6 };
enum Sum { G_LAM, G_MU, G_TAU, G_VA, G_VB, G_ILLUM };
enum Profile { K_, A_, B_, KH, AH, BH, RK, RKH };  // (the last two: 1 / K, 1 / K_half)
constexpr int kProfiles = 8;

struct March {
  const ShotSlot* S;
  float* f;            // fields, n floats apart
  const float* m;      // media, mn floats apart
  float* g;            // sums, n floats apart
  int n, mn, ldz;
  float dt, rdz, rdx;
  const float* prof;   // shared: kProfiles z profiles of nz values, then as many x profiles of w columns
  const unsigned* info;  // shared: nch * 32 depths of each column
  int nz, w, xa, depth;
};

// The thread's cell of an item: its index, its depth, its column in the strip.
struct Cell {
  int i, z, xl;
  unsigned v;
};
__device__ __forceinline__ Cell cell_at(const March& M, int z0, int x) {
  Cell c;
  c.z = z0 + (threadIdx.x & 31);
  c.xl = x - M.xa;
  c.i = x * M.ldz + c.z;
  c.v = M.info[c.xl * M.depth + c.z];
  return c;
}
__device__ __forceinline__ float& fld(const March& M, const Cell& c, int q) { return M.f[c.i + q * M.n]; }
__device__ __forceinline__ float med(const March& M, const Cell& c, int q) { return M.m[c.i + q * M.mn]; }
__device__ __forceinline__ float& sum(const March& M, const Cell& c, int q) { return M.g[c.i + q * M.n]; }
__device__ __forceinline__ float pz(const March& M, const Cell& c, int q) { return M.prof[q * M.nz + c.z]; }
__device__ __forceinline__ float px(const March& M, const Cell& c, int q) { return M.prof[kProfiles * M.nz + q * M.w + c.xl]; }
// a / K with r = 1 / K rounded: the quotient estimate a r corrected by its
// residual, correctly rounded by Markstein's theorem (IBM J. Res. Dev. 34,
// 1990) as the division is, without its range checks (K is in [1, 2]).
__device__ __forceinline__ float over(float a, float K, float r) {
  const float q = a * r;
  return fmaf(fmaf(-K, q, a), r, q);
}
__device__ __forceinline__ float over_z(const March& M, const Cell& c, float a, int h) {
  return over(a, pz(M, c, h ? KH : K_), pz(M, c, h ? RKH : RK));
}
__device__ __forceinline__ float over_x(const March& M, const Cell& c, float a, int h) {
  return over(a, px(M, c, h ? KH : K_), px(M, c, h ? RKH : RK));
}
__device__ __forceinline__ float dmz(const March& M, const Cell& c, int q) { return sdm(M.f, c.i + q * M.n, 1, M.rdz); }
__device__ __forceinline__ float dpz(const March& M, const Cell& c, int q) { return sdp(M.f, c.i + q * M.n, 1, M.rdz); }
__device__ __forceinline__ float dmx(const March& M, const Cell& c, int q) { return sdm(M.f, c.i + q * M.n, M.ldz, M.rdx); }
__device__ __forceinline__ float dpx(const March& M, const Cell& c, int q) { return sdp(M.f, c.i + q * M.n, M.ldz, M.rdx); }
// The five saved values of ring row v & kRing of a step (szz, sxz, sxx, vz, vx).
__device__ __forceinline__ float* ring_at(const March& M, const Cell& c, int it) {
  return M.S->st.base + static_cast<size_t>(it) * 5 * M.S->g.ring_len + ((c.v & kRing) - 1);
}

// Each sweep is two or three independent parts (fields that no other part of
// the sweep reads or writes), which different warps take: at these sizes a
// sweep lasts as long as one warp's chain of dependent instructions. A part
// loads everything it may need before it stores anything: the arrays do not
// alias, which the compiler cannot know, and a load behind a store would cost
// another L2 round trip.

// F1, normal stresses: szz, sxx, the source, recording, their ring samples and the velocities'.
__device__ __forceinline__ void f1_normal(const March& M, int it, int save, int z0, int x) {
  const Cell c = cell_at(M, z0, x);
  if (!(c.v & (kDom | kRing | kSrc | kRec))) return;
  const ShotD& sh = M.S->sh;
  const bool dom = c.v & kDom, zp = c.v & kZp, xp = c.v & kXp, src = c.v & kSrc;
  const int rec = c.v & kRec ? first_receiver(sh, c.z, x) : -1;
  const float s1 = src ? sh.src_szz[it] : 0.0f, s2 = src ? sh.src_sxx[it] : 0.0f;
  float szz = fld(M, c, SZZ), sxx = fld(M, c, SXX);
  const float lam = med(M, c, LAM), l2m = med(M, c, L2M);
  float mz = zp ? fld(M, c, M_VZ_Z) : 0.0f, mx = xp ? fld(M, c, M_VX_X) : 0.0f;
  float dvz_dz = 0.0f, dvx_dx = 0.0f;
  if (dom) {
    dvz_dz = dmz(M, c, VZ);
    dvx_dx = dmx(M, c, VX);
  }
  if (save && (c.v & kRing)) {
    const float vz = fld(M, c, VZ), vx = fld(M, c, VX);
    float* p = ring_at(M, c, it);
    const int len = M.S->g.ring_len;
    p[0] = szz;
    p[2 * len] = sxx;
    p[3 * len] = vz;
    p[4 * len] = vx;
  }
  if (zp) {
    mz = pz(M, c, B_) * mz + pz(M, c, A_) * dvz_dz;
    dvz_dz = over_z(M, c, dvz_dz, 0) + mz;
    fld(M, c, M_VZ_Z) = mz;
  }
  if (xp) {
    mx = px(M, c, B_) * mx + px(M, c, A_) * dvx_dx;
    dvx_dx = over_x(M, c, dvx_dx, 0) + mx;
    fld(M, c, M_VX_X) = mx;
  }
  if (dom) {
    szz += (l2m * dvz_dz + lam * dvx_dx) * M.dt;
    sxx += (lam * dvz_dz + l2m * dvx_dx) * M.dt;
  }
  if (src) {
    szz += s1;
    sxx += s2;
  }
  if (dom || src) {
    fld(M, c, SZZ) = szz;
    fld(M, c, SXX) = sxx;
  }
  record(sh, it, rec, c.z, x, szz, sxx);
}

// F1, shear stress.
__device__ __forceinline__ void f1_shear(const March& M, int it, int save, int z0, int x) {
  const Cell c = cell_at(M, z0, x);
  if (!(c.v & (kDom | kRing))) return;
  const bool dom = c.v & kDom, zp = c.v & kZp, xp = c.v & kXp;
  const float sxz = fld(M, c, SXZ), amu = med(M, c, AMU);
  float mz = zp ? fld(M, c, M_VX_Z) : 0.0f, mx = xp ? fld(M, c, M_VZ_X) : 0.0f;
  if (save && (c.v & kRing)) ring_at(M, c, it)[M.S->g.ring_len] = sxz;
  if (!dom) return;
  float dvx_dz = dpz(M, c, VX), dvz_dx = dpx(M, c, VZ);
  if (zp) {
    mz = pz(M, c, BH) * mz + pz(M, c, AH) * dvx_dz;
    dvx_dz = over_z(M, c, dvx_dz, 1) + mz;
    fld(M, c, M_VX_Z) = mz;
  }
  if (xp) {
    mx = px(M, c, BH) * mx + px(M, c, AH) * dvz_dx;
    dvz_dx = over_x(M, c, dvz_dx, 1) + mx;
    fld(M, c, M_VZ_X) = mx;
  }
  fld(M, c, SXZ) = sxz + amu * (dvx_dz + dvz_dx) * M.dt;
}

// F2, one velocity component (0 outside the stencil domain): vz from dszz/dz (half-point profile) and dsxz/dx, or
// vx from dsxz/dz and dsxx/dx (half-point profile).
template <bool Z>
__device__ __forceinline__ float f2_velocity(const March& M, const Cell& c) {
  if (!(c.v & kDom)) return 0.0f;
  const bool zp = c.v & kZp, xp = c.v & kXpV;
  constexpr int V = Z ? VZ : VX, MZ = Z ? M_SZZ_Z : M_SXZ_Z, MX = Z ? M_SXZ_X : M_SXX_X;
  constexpr int hz = Z ? 3 : 0, hx = Z ? 0 : 3;  // half-point profiles
  const float old = fld(M, c, V), by = med(M, c, Z ? BYA : BYB);
  float mz = zp ? fld(M, c, MZ) : 0.0f, mx = xp ? fld(M, c, MX) : 0.0f;
  float dz = Z ? dpz(M, c, SZZ) : dmz(M, c, SXZ);
  float dx = Z ? dmx(M, c, SXZ) : dpx(M, c, SXX);
  if (zp) {
    mz = pz(M, c, B_ + hz) * mz + pz(M, c, A_ + hz) * dz;
    dz = over_z(M, c, dz, hz) + mz;
    fld(M, c, MZ) = mz;
  }
  if (xp) {
    mx = px(M, c, B_ + hx) * mx + px(M, c, A_ + hx) * dx;
    dx = over_x(M, c, dx, hx) + mx;
    fld(M, c, MX) = mx;
  }
  const float v = old + (dz + dx) * by * M.dt;
  fld(M, c, V) = v;
  return v;
}

// F2 with the illumination, which takes both components.
__device__ __forceinline__ void f2_illum(const March& M, const Cell& c) {
  if (!(c.v & kDom)) return;
  const float e = sum(M, c, G_ILLUM);
  const float nvz = f2_velocity<true>(M, c), nvx = f2_velocity<false>(M, c);
  sum(M, c, G_ILLUM) = e + (nvz * nvz + nvx * nvx);
}

// B, forward fields: source removal, reverse stresses, the sums of the lambda and mu kernels, the ring's stresses.
__device__ __forceinline__ void b_stress(const March& M, int it, int z0, int x) {
  const Cell c = cell_at(M, z0, x);
  if (!(c.v & (kInner | kSrc | kRing))) return;
  const ShotD& sh = M.S->sh;
  const bool src = c.v & kSrc, ring = c.v & kRing;
  const float s1 = src ? sh.src_szz_r[it] : 0.0f, s2 = src ? sh.src_sxx_r[it] : 0.0f;
  float szz = fld(M, c, SZZ), sxx = fld(M, c, SXX), sxz = fld(M, c, SXZ), r0 = 0.0f, r1 = 0.0f, r2 = 0.0f;
  if (ring) {
    const float* p = ring_at(M, c, it);
    const int len = M.S->g.ring_len;
    r0 = p[0];
    r1 = p[len];
    r2 = p[2 * len];
  }
  if (src) {
    szz -= s1;
    sxx -= s2;
  }
  if (c.v & kInner) {
    const float lam = med(M, c, LAM), l2m = med(M, c, L2M), amu = med(M, c, AMU), dt = M.dt;
    const float gl = sum(M, c, G_LAM), gm = sum(M, c, G_MU), gt = sum(M, c, G_TAU);
    const float sa = fld(M, c, SZZ_A), xa = fld(M, c, SXX_A), za = fld(M, c, SXZ_A);
    const float dvz_dz = dmz(M, c, VZ), dvx_dx = dmx(M, c, VX), e = dpz(M, c, VX) + dpx(M, c, VZ);
    szz -= (l2m * dvz_dz + lam * dvx_dx) * dt;
    sxx -= (lam * dvz_dz + l2m * dvx_dx) * dt;
    sxz -= amu * e * dt;
    sum(M, c, G_LAM) = gl + (sa + xa) * (dvz_dz + dvx_dx);
    sum(M, c, G_MU) = gm + (sa * dvz_dz + xa * dvx_dx);
    sum(M, c, G_TAU) = gt + za * e;
  }
  fld(M, c, SZZ) = ring ? r0 : szz;
  fld(M, c, SXZ) = ring ? r1 : sxz;
  fld(M, c, SXX) = ring ? r2 : sxx;
}

// B, one adjoint velocity component (el_velocity_adj.cu:57-102) with the memory arrays it feeds; the psi memory terms
// are read only where their CPML coefficient is non-zero. vx_a: normal stresses differ along x (a_x, K_x), the shear
// stress along z (a_zh, K_zh); vz_a: along z (a_z, K_z) and x (a_xh, K_xh).
template <bool X>
__device__ __forceinline__ void b_velocity(const March& M, int z0, int x) {
  const Cell c = cell_at(M, z0, x);
  if (!(c.v & kDom)) return;
  const bool zp = c.v & kZp, xp = c.v & kXp;
  constexpr int V = X ? VX_A : VZ_A, MX = X ? M_SXX_X : M_SXZ_X, MZ = X ? M_SXZ_Z : M_SZZ_Z;
  const float dt = M.dt, lam = med(M, c, LAM), l2m = med(M, c, L2M), amu = med(M, c, AMU);
  const float mx = xp ? fld(M, c, MX) : 0.0f, mz = zp ? fld(M, c, MZ) : 0.0f;
  const float by = xp || zp ? med(M, c, X ? BYB : BYA) : 0.0f;
  float v = fld(M, c, V), q1 = 0.0f, q2 = 0.0f;
  const bool band = c.v & (kXb | kZb);  // (a = 0 and K = 1 outside the bands)
  if (c.v & (X ? kXb : kZb)) q1 = X ? dpx(M, c, M_VX_X) : dpz(M, c, M_VZ_Z);
  if (c.v & (X ? kZb : kXb)) q2 = X ? dmz(M, c, M_VX_Z) : dmx(M, c, M_VZ_X);
  const float dzz = X ? dpx(M, c, SZZ_A) : dpz(M, c, SZZ_A);
  const float dxx = X ? dpx(M, c, SXX_A) : dpz(M, c, SXX_A);
  const float dxz = X ? dmz(M, c, SXZ_A) : dmx(M, c, SXZ_A);
  float tn = (X ? lam * dzz + l2m * dxx : l2m * dzz + lam * dxx), ts = amu * dxz, t = 0.0f;
  if (band) {
    const float an = X ? px(M, c, A_) : pz(M, c, A_), as = X ? pz(M, c, AH) : px(M, c, AH);
    t = (an != 0.0f ? an * q1 : 0.0f) + (as != 0.0f ? as * q2 : 0.0f);
    tn = X ? over_x(M, c, tn, 0) : over_z(M, c, tn, 0);
    ts = X ? over_z(M, c, ts, 1) : over_x(M, c, ts, 1);
  }
  v -= (tn + ts) * dt + t;
  fld(M, c, V) = v;
  if (xp) fld(M, c, MX) = px(M, c, X ? BH : B_) * mx + by * v * dt;
  if (zp) fld(M, c, MZ) = pz(M, c, X ? B_ : BH) * mz + by * v * dt;
}

// C, adjoint stresses: residual injection, el_stress_adj.cu:53-97 with the memory arrays in their bands (within two
// cells of the CPML), and the source gradient.
__device__ __forceinline__ void c_stress(const March& M, int it, int z0, int x) {
  const Cell c = cell_at(M, z0, x);
  if (!(c.v & (kDom | kRec))) return;
  const ShotD& sh = M.S->sh;
  const bool dom = c.v & kDom, xb = c.v & kXb, zb = c.v & kZb;
  const int rec = c.v & kRec ? first_receiver(sh, c.z, x) : -1;
  float sa = fld(M, c, SZZ_A), xa = fld(M, c, SXX_A), za = fld(M, c, SXZ_A);
  const float bA = med(M, c, BYA), bB = med(M, c, BYB), dt = M.dt;
  float m1 = 0.0f, m2 = 0.0f, m3 = 0.0f, m4 = 0.0f, amu = 0.0f, lam = 0.0f, l2m = 0.0f;
  if (xb) {
    m1 = fld(M, c, M_VZ_X);
    m2 = fld(M, c, M_VX_X);
  }
  if (zb) {
    m3 = fld(M, c, M_VX_Z);
    m4 = fld(M, c, M_VZ_Z);
  }
  if (xb || zb) {
    amu = med(M, c, AMU);
    lam = med(M, c, LAM);
    l2m = med(M, c, L2M);
  }
  if (dom) {
    float q1 = 0.0f, q2 = 0.0f, q3 = 0.0f, q4 = 0.0f;
    if (xb) {
      q1 = dpx(M, c, M_SXZ_X);
      q3 = dmx(M, c, M_SXX_X);
    }
    if (zb) {
      q2 = dpz(M, c, M_SXZ_Z);
      q4 = dmz(M, c, M_SZZ_Z);
    }
    float d1 = dpx(M, c, VZ_A), d2 = dpz(M, c, VX_A), d3 = dmx(M, c, VX_A), d4 = dmz(M, c, VZ_A);
    float t1 = 0.0f, t2 = 0.0f, t3 = 0.0f;
    if (xb || zb) {
      const float ax = px(M, c, A_), az = pz(M, c, A_), axh = px(M, c, AH), azh = pz(M, c, AH);
      t1 = (ax != 0.0f ? ax * q1 : 0.0f) + (az != 0.0f ? az * q2 : 0.0f);
      t2 = axh != 0.0f ? axh * q3 : 0.0f;
      t3 = azh != 0.0f ? azh * q4 : 0.0f;
      d1 = over_x(M, c, d1, 0);
      d2 = over_z(M, c, d2, 0);
      d3 = over_x(M, c, d3, 1);
      d4 = over_z(M, c, d4, 1);
    }
    inject_res(sh, it, rec, c.z, x, sa, xa);
    za -= (d1 * bA + d2 * bB) * dt + t1;
    xa -= bB * d3 * dt + t2;
    sa -= bA * d4 * dt + t3;
    if (xb) {
      fld(M, c, M_VZ_X) = px(M, c, BH) * m1 + za * amu * dt;
      fld(M, c, M_VX_X) = px(M, c, B_) * m2 + (lam * sa + l2m * xa) * dt;
    }
    if (zb) {
      fld(M, c, M_VX_Z) = pz(M, c, BH) * m3 + za * amu * dt;
      fld(M, c, M_VZ_Z) = pz(M, c, B_) * m4 + (l2m * sa + lam * xa) * dt;
    }
    fld(M, c, SXZ_A) = za;
  } else {
    inject_res(sh, it, rec, c.z, x, sa, xa);
  }
  fld(M, c, SZZ_A) = sa;
  fld(M, c, SXX_A) = xa;
  if (it >= 1 && (c.v & kSrc)) sh.gstf[it - 1] = -(sa + 3.0f * xa) * dt;
}

// C, one forward velocity component taken back to step it - 1 (it >= 1) with its sum of the rho kernel and the ring.
template <bool Z>
__device__ __forceinline__ void c_velocity(const March& M, int it, int z0, int x) {
  const Cell c = cell_at(M, z0, x);
  if (!(c.v & (kInner | kRing))) return;
  const bool ring = c.v & kRing;
  constexpr int V = Z ? VZ : VX;
  float v = fld(M, c, V), r = 0.0f;
  if (ring) r = ring_at(M, c, it - 1)[(Z ? 3 : 4) * M.S->g.ring_len];
  if (c.v & kInner) {
    const float by = med(M, c, Z ? BYA : BYB), w = fld(M, c, Z ? VZ_A : VX_A), a = sum(M, c, Z ? G_VA : G_VB);
    const float e = Z ? dpz(M, c, SZZ) + dmx(M, c, SXZ) : dmz(M, c, SXZ) + dpx(M, c, SXX);
    v -= e * by * M.dt;
    sum(M, c, Z ? G_VA : G_VB) = a + w * e;
  }
  fld(M, c, V) = ring ? r : v;
}

// Sets a block up: its strip's CPML profiles (which would otherwise come from
// L2 in every sweep) and cell_info in shared memory, the bases in registers.
__device__ __forceinline__ March set_up(const ShotSlot& S, const Strip& s, float* sm) {
  March M;
  M.S = &S;
  M.f = S.f.vz;
  M.n = static_cast<int>(S.f.vx - S.f.vz);
  M.m = S.m.lam;
  M.mn = static_cast<int>(S.m.aveMu - S.m.l2m);
  M.g = S.gr.lam;
  M.ldz = S.g.ldz;
  M.dt = S.g.dt;
  M.rdz = S.g.rdz;
  M.rdx = S.g.rdx;
  M.nz = S.g.nz;
  M.w = s.xb - s.xa;
  M.xa = s.xa;
  M.depth = s.nch * 32;
  const float* gz[6] = {S.c.K_z, S.c.a_z, S.c.b_z, S.c.K_zh, S.c.a_zh, S.c.b_zh};
  const float* gx[6] = {S.c.K_x, S.c.a_x, S.c.b_x, S.c.K_xh, S.c.a_xh, S.c.b_xh};
  float* sx = sm + kProfiles * M.nz;
  unsigned* info = reinterpret_cast<unsigned*>(sx + kProfiles * M.w);
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    for (int i = threadIdx.x; i < M.nz; i += blockDim.x) sm[q * M.nz + i] = gz[q][i];
    for (int i = threadIdx.x; i < M.w; i += blockDim.x) sx[q * M.w + i] = gx[q][s.xa + i];
  }
  for (int h = 0; h < 2; ++h) {
    for (int i = threadIdx.x; i < M.nz; i += blockDim.x) sm[(RK + h) * M.nz + i] = 1.0f / gz[3 * h][i];
    for (int i = threadIdx.x; i < M.w; i += blockDim.x) sx[(RK + h) * M.w + i] = 1.0f / gx[3 * h][s.xa + i];
  }
  for (int i = threadIdx.x; i < M.w * M.depth; i += blockDim.x)
    info[i] = cell_info(S, i % M.depth, s.xa + i / M.depth);
  M.prof = sm;
  M.info = info;
  __syncthreads();
  return M;
}

// One forward pass of every shot of the pack over its own record. flags: bit 0
// saves the boundary ring, bit 1 is the timeout test hook (the first block
// gives up its first wait and raises err; the others follow).
__global__ void __launch_bounds__(kMarchThreads, 1)
    k_march_fwd(const __grid_constant__ MarchPack P, int flags, unsigned* done, unsigned* err) {
  const Strip s = strip_of(P, done);
  const ShotSlot& S = P.slots[s.shot];
  extern __shared__ float sm[];
  const March M = set_up(S, s, sm);
  const int n = S.nSteps;
  Item first{0, s.xa, 0};
  step_item(s, first, threadIdx.x >> 5);
  for (int it = 0; it <= n - 2; ++it) {
    for_items(s, first, 2, [&](int part, int z0, int x) {
      if (part == 0)
        f1_normal(M, it, flags & 1, z0, x);
      else
        f1_shear(M, it, flags & 1, z0, x);
    });
    if ((flags & 2) && it == 0 && blockIdx.x == 0) {
      if (threadIdx.x == 0) atomicOr(err, 1u);
      return;
    }
    if (!strip_sync(s, 2 * it + 1, err)) return;
    if (S.gr.illum)
      for_items(s, first, 1, [&](int, int z0, int x) { f2_illum(M, cell_at(M, z0, x)); });
    else
      for_items(s, first, 2, [&](int part, int z0, int x) {
        if (part == 0)
          f2_velocity<true>(M, cell_at(M, z0, x));
        else
          f2_velocity<false>(M, cell_at(M, z0, x));
      });
    if (!strip_sync(s, 2 * it + 2, err)) return;
  }
}

// The adjoint pass: sweep C of the last step, then B and C of every step back
// to the first (backward iteration j: step nSteps - 2 - j).
__global__ void __launch_bounds__(kMarchThreads, 1)
    k_march_bwd(const __grid_constant__ MarchPack P, unsigned* done, unsigned* err) {
  const Strip s = strip_of(P, done);
  const ShotSlot& S = P.slots[s.shot];
  extern __shared__ float sm[];
  const March M = set_up(S, s, sm);
  const int n = S.nSteps;
  Item first{0, s.xa, 0};
  step_item(s, first, threadIdx.x >> 5);
  auto sweep_C = [&](int it) {
    for_items(s, first, it >= 1 ? 3 : 1, [&](int part, int z0, int x) {
      if (part == 0)
        c_stress(M, it, z0, x);
      else if (part == 1)
        c_velocity<true>(M, it, z0, x);
      else
        c_velocity<false>(M, it, z0, x);
    });
  };
  unsigned count = 0;
  sweep_C(n - 1);
  if (!strip_sync(s, ++count, err)) return;
  for (int it = n - 2; it >= 0; --it) {
    for_items(s, first, 3, [&](int part, int z0, int x) {
      if (part == 0)
        b_stress(M, it, z0, x);
      else if (part == 1)
        b_velocity<true>(M, z0, x);
      else
        b_velocity<false>(M, z0, x);
    });
    if (!strip_sync(s, ++count, err)) return;
    sweep_C(it);
    if (!strip_sync(s, ++count, err)) return;
  }
}

}  // namespace

size_t march_flag_bytes(const MarchPack& p) {
  return static_cast<size_t>(p.first[p.nshots]) * kFlagStride * sizeof(unsigned);
}

bool march_plan(MarchPack& p, int sms) {
  // The narrowest strips that are all resident with one block per SM; at least
  // 2 columns, because a stencil reaches two into the next strip. (A 96 x 84
  // grid takes 9.1 / 9.8 / 10.5 / 13.7 us a step with strips of 2 / 3 / 4 / 6.)
  int total = 0, chunks = 1;
  for (int k = 0; k < p.nshots; ++k) {
    const Geo& g = p.slots[k].g;
    total += g.nx;
    chunks = std::max(chunks, (std::min(g.nz, std::max(g.zact1, p.slots[k].sh.rbz1) + 1) + 31) / 32);
    // Ring rows and offsets from the bases fit their 21 and 31 bits.
    const long long media = p.slots[k].m.aveMu - p.slots[k].m.l2m;
    if (g.ring_len >= 1 << 21 || 18ll * g.ldz * g.nx >= 1ll << 31 || 8 * media >= 1ll << 31) return false;
  }
  for (int w = 2; w <= total; ++w) {
    int n = 0;
    for (int k = 0; k < p.nshots; ++k) {
      p.first[k] = n;
      n += std::max(1, p.slots[k].g.nx / w);  // (widths w or more)
    }
    p.first[p.nshots] = n;
    if (n > sms) continue;
    int widest = 0;
    for (int k = 0; k < p.nshots; ++k) {
      const int nb = p.first[k + 1] - p.first[k];
      widest = std::max(widest, (p.slots[k].g.nx + nb - 1) / nb);
    }
    p.threads = 32 * std::max(4, std::min(kMarchThreads / 32, 3 * widest * chunks));
    p.smem = static_cast<int>((kProfiles * (p.slots[0].g.nz + widest) + widest * chunks * 32) * sizeof(float));
    return p.smem <= 48 * 1024;
  }
  return false;
}

cudaError_t launch_march(cudaStream_t s, const MarchPack& p, bool backward, int flags, unsigned* done, unsigned* err) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.first[p.nshots]);
  cfg.blockDim = dim3(p.threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return backward ? cudaLaunchKernelEx(&cfg, k_march_bwd, p, done, err)
                  : cudaLaunchKernelEx(&cfg, k_march_fwd, p, flags, done, err);
}

}  // namespace fwigb
