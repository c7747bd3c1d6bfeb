// Marching kernels: a whole pass over time in one launch, for calls whose
// grids are too small to fill the GPU in every sweep.
//
// A sweep of a small grid is all latency: 4 us a launch on a 96 x 84 grid as
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
// sizes; marches() in engine.cu has the times against a launch per sweep.
//
// A warp takes 64 depths of one column at a time, two adjacent ones a thread,
// and reads its stencil samples from the fields themselves (L1 / L2): at these
// sizes the fields live in L2, and staging would add its own latency. Where a
// block's work takes several rounds of its warps it is bound by the instructions
// of its loads and their addresses (about 150 loads a cell of a step), which
// paired loads halve.
// With several rounds the forward pass runs two blocks of 512 threads on each
// SM, so that one works while the other waits for its neighbours. us a step, two
// blocks / one: two 192 x 264 grids 4.96 / 6.03, three 160 x 190 4.99 / 6.08, one
// 224 x 448 4.88 / 5.65, sixteen 96 x 88 7.69 / 8.77; but one 320 x 324 6.52 /
// 5.98 and one 352 x 334 6.65 / 5.99. The backward pass has more operands in
// flight: one block with 128 registers a thread, against two of 64: the same
// grids 8.82 / 9.42, 8.67 / 10.0, 7.24 / 9.76, 14.3 / 14.8, 8.53 / 9.30 and 8.65 /
// 10.2, and two 96 x 84 ones 5.48 / 7.05.
#include <algorithm>

#include "fwigb_kernels.h"
#include "sweep_cells.cuh"

namespace fwigb {
namespace {

constexpr int R = 2;  // depths per thread
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

// The limit of the timeout test hook's wait (k_march_fwd).
constexpr unsigned long long kInjectWaitNs = 20000000ull;

// Waits until a neighbour's flag reaches `count`: at most `limit`, and given up
// as soon as another block has raised the error word.
__device__ __forceinline__ bool wait_flag(const unsigned* flag, unsigned count, unsigned* err,
                                          unsigned long long limit = kWaitLimitNs) {
  unsigned long long t0 = 0;
  for (unsigned n = 0;; ++n) {
    if (ld_acquire(flag) >= count) return true;
    if ((n & 63) == 63) {
      if (ld_relaxed(err) != 0) return false;
      const unsigned long long t = global_timer_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > limit) {
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
  int nch;                 // 64-depth chunks down to the last row a sweep touches
};

__device__ __forceinline__ Strip strip_of(const MarchPack& P, const MarchSplit& split, unsigned* flags) {
  Strip s;
  s.shot = 0;
  while (s.shot + 1 < P.nshots && static_cast<int>(blockIdx.x) >= split.first[s.shot + 1]) ++s.shot;
  const int j = blockIdx.x - split.first[s.shot], nb = split.first[s.shot + 1] - split.first[s.shot];
  const Geo& g = P.slots[s.shot].g;
  s.xa = static_cast<int>(static_cast<long long>(j) * g.nx / nb);
  s.xb = static_cast<int>(static_cast<long long>(j + 1) * g.nx / nb);
  s.left = j > 0;
  s.right = j + 1 < nb;
  s.flag = flags + static_cast<size_t>(blockIdx.x) * kFlagStride;
  s.nch = (min(g.nz, max(g.zact1, P.slots[s.shot].sh.rbz1) + 1) + 32 * R - 1) / (32 * R);
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

// A warp's place in its block's list of work: part, then column, then 64-depth
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
    fn(t.part, t.ch * 32 * R, t.x);
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
enum Profile { K_, A_, B_, KH, AH, BH, RK, RKH };  // (the last two: 1 / K, 1 / K_half; K and 1 / K scaled, over())
constexpr int kProfiles = 8;

struct March {
  const ShotSlot* S;
  float* f;            // fields, n floats apart
  const float* m;      // media, mn floats apart
  float* g;            // sums, n floats apart
  int n, mn, ldz;
  float dt, rdz, rdx;
  const float* prof;   // shared: kProfiles z profiles of nz values, then as many x profiles of w columns
  const unsigned* info;  // shared: the strip's cells, `depth` of each column
  int nz, w, xa, depth;
};

// The thread's cells of an item (adjacent depths; the first one's index, depth
// and column in the strip), what each of them is and what any of them is.
struct Cells {
  int i, z, xl;
  unsigned v[R], any;
};
__device__ __forceinline__ Cells cells_at(const March& M, int z0, int x) {
  Cells c;
  c.z = z0 + R * (threadIdx.x & 31);
  c.xl = x - M.xa;
  c.i = x * M.ldz + c.z;
  const unsigned* p = M.info + c.xl * M.depth + c.z;
  const uint2 t = *reinterpret_cast<const uint2*>(p);
  c.v[0] = t.x;
  c.v[1] = t.y;
  c.any = t.x | t.y;
  return c;
}

// Values at the thread's cells: one paired access (even depths, columns a
// multiple of 32 floats apart).
struct Vals {
  float v[R];
  __device__ __forceinline__ float& operator[](int r) { return v[r]; }
  __device__ __forceinline__ float operator[](int r) const { return v[r]; }
};
__device__ __forceinline__ Vals load(const float* p) {
  const float2 t = *reinterpret_cast<const float2*>(p);
  return {{t.x, t.y}};
}
__device__ __forceinline__ Vals load_if(bool on, const float* p) {
  Vals a{};
  if (on) a = load(p);
  return a;
}
__device__ __forceinline__ void store(float* p, const Vals& a) {
  *reinterpret_cast<float2*>(p) = make_float2(a.v[0], a.v[1]);
}
__device__ __forceinline__ float* fld(const March& M, const Cells& c, int q) { return M.f + (c.i + q * M.n); }
__device__ __forceinline__ const float* med(const March& M, const Cells& c, int q) { return M.m + (c.i + q * M.mn); }
__device__ __forceinline__ float* sum(const March& M, const Cells& c, int q) { return M.g + (c.i + q * M.n); }
__device__ __forceinline__ float pz(const March& M, const Cells& c, int r, int q) { return M.prof[q * M.nz + c.z + r]; }
__device__ __forceinline__ float px(const March& M, const Cells& c, int q) {
  return M.prof[kProfiles * M.nz + q * M.w + c.xl];
}
__device__ __forceinline__ float over_z(const March& M, const Cells& c, int r, float a, int h) {
  return over<false>(a, pz(M, c, r, h ? KH : K_), pz(M, c, r, h ? RKH : RK));
}
__device__ __forceinline__ float over_x(const March& M, const Cells& c, float a, int h) {
  return over<false>(a, px(M, c, h ? KH : K_), px(M, c, h ? RKH : RK));
}
// Differences at the cells. Only where one of them is in the stencil domain:
// the pair's samples then lie in the array (two columns follow the domain's last).
__device__ __forceinline__ float diff(float p, float q, float s, float t, float r) {
  return (C1 * (p - q) - C2 * (s - t)) * r;
}
__device__ __forceinline__ Vals dmz(const March& M, const Cells& c, int q) {
  const float* a = fld(M, c, q);
  const Vals m = load(a - 2), e = load(a), p = load(a + 2);
  return {{diff(e[0], m[1], e[1], m[0], M.rdz), diff(e[1], e[0], p[0], m[1], M.rdz)}};
}
__device__ __forceinline__ Vals dpz(const March& M, const Cells& c, int q) {
  const float* a = fld(M, c, q);
  const Vals m = load(a - 2), e = load(a), p = load(a + 2);
  return {{diff(e[1], e[0], p[0], m[1], M.rdz), diff(p[0], e[1], p[1], e[0], M.rdz)}};
}
__device__ __forceinline__ Vals dmx(const March& M, const Cells& c, int q) {
  const float* a = fld(M, c, q);
  const Vals e = load(a), m = load(a - M.ldz), p = load(a + M.ldz), n = load(a - 2 * M.ldz);
  Vals o;
#pragma unroll
  for (int r = 0; r < R; ++r) o.v[r] = diff(e[r], m[r], p[r], n[r], M.rdx);
  return o;
}
__device__ __forceinline__ Vals dpx(const March& M, const Cells& c, int q) {
  const float* a = fld(M, c, q);
  const Vals e = load(a), p = load(a + M.ldz), n = load(a + 2 * M.ldz), m = load(a - M.ldz);
  Vals o;
#pragma unroll
  for (int r = 0; r < R; ++r) o.v[r] = diff(p[r], e[r], n[r], m[r], M.rdx);
  return o;
}
// The five saved values of a cell in ring row v & kRing of a step (szz, sxz, sxx, vz, vx).
__device__ __forceinline__ float* ring_at(const March& M, unsigned v, int it) {
  return M.S->st.base + static_cast<size_t>(it) * 5 * M.S->g.ring_len + ((v & kRing) - 1);
}

// Each sweep is two or three independent parts (fields that no other part of
// the sweep reads or writes), which different warps take: at the smallest sizes
// a sweep lasts as long as one warp's chain of dependent instructions. A part
// loads everything it may need before it stores anything: the arrays do not
// alias, which the compiler cannot know, and a load behind a store would cost
// another L2 round trip. A pair is loaded and stored whole when either cell
// needs it; the other one's values go back as they came.

// F1, normal stresses: szz, sxx, the source, recording, their ring samples and the velocities'.
__device__ __forceinline__ void f1_normal(const March& M, int it, int save, int z0, int x) {
  const Cells c = cells_at(M, z0, x);
  if (!(c.any & (kDom | kRing | kSrc | kRec))) return;
  const ShotD& sh = M.S->sh;
  const bool zp = c.any & kZp, xp = c.any & kXp;
  int rec[R];
  float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
  for (int r = 0; r < R; ++r) rec[r] = c.v[r] & kRec ? first_receiver(sh, c.z + r, x) : -1;
  if (c.any & kSrc) {
    s1 = sh.src_szz[it];
    s2 = sh.src_sxx[it];
  }
  Vals szz = load(fld(M, c, SZZ)), sxx = load(fld(M, c, SXX));
  const Vals lam = load(med(M, c, LAM)), l2m = load(med(M, c, L2M));
  Vals mz = load_if(zp, fld(M, c, M_VZ_Z)), mx = load_if(xp, fld(M, c, M_VX_X));
  Vals dz{}, dx{};
  if (c.any & kDom) {
    dz = dmz(M, c, VZ);
    dx = dmx(M, c, VX);
  }
  if (save && (c.any & kRing)) {
    const Vals vz = load(fld(M, c, VZ)), vx = load(fld(M, c, VX));
    const int len = M.S->g.ring_len;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (c.v[r] & kRing) {
        float* p = ring_at(M, c.v[r], it);
        p[0] = szz[r];
        p[2 * len] = sxx[r];
        p[3 * len] = vz[r];
        p[4 * len] = vx[r];
      }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (c.v[r] & kZp) {
      mz[r] = pz(M, c, r, B_) * mz[r] + pz(M, c, r, A_) * dz[r];
      dz[r] = over_z(M, c, r, dz[r], 0) + mz[r];
    }
    if (c.v[r] & kXp) {
      mx[r] = px(M, c, B_) * mx[r] + px(M, c, A_) * dx[r];
      dx[r] = over_x(M, c, dx[r], 0) + mx[r];
    }
    if (c.v[r] & kDom) {
      szz[r] += (l2m[r] * dz[r] + lam[r] * dx[r]) * M.dt;
      sxx[r] += (lam[r] * dz[r] + l2m[r] * dx[r]) * M.dt;
    }
    if (c.v[r] & kSrc) {
      szz[r] += s1;
      sxx[r] += s2;
    }
  }
  if (zp) store(fld(M, c, M_VZ_Z), mz);
  if (xp) store(fld(M, c, M_VX_X), mx);
  if (c.any & (kDom | kSrc)) {
    store(fld(M, c, SZZ), szz);
    store(fld(M, c, SXX), sxx);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) record(sh, it, rec[r], c.z + r, x, szz[r], sxx[r]);
}

// F1, shear stress.
__device__ __forceinline__ void f1_shear(const March& M, int it, int save, int z0, int x) {
  const Cells c = cells_at(M, z0, x);
  if (!(c.any & (kDom | kRing))) return;
  const bool zp = c.any & kZp, xp = c.any & kXp;
  Vals sxz = load(fld(M, c, SXZ));
  const Vals amu = load(med(M, c, AMU));
  Vals mz = load_if(zp, fld(M, c, M_VX_Z)), mx = load_if(xp, fld(M, c, M_VZ_X));
  if (save) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (c.v[r] & kRing) ring_at(M, c.v[r], it)[M.S->g.ring_len] = sxz[r];
  }
  if (!(c.any & kDom)) return;
  Vals dz = dpz(M, c, VX), dx = dpx(M, c, VZ);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (c.v[r] & kZp) {
      mz[r] = pz(M, c, r, BH) * mz[r] + pz(M, c, r, AH) * dz[r];
      dz[r] = over_z(M, c, r, dz[r], 1) + mz[r];
    }
    if (c.v[r] & kXp) {
      mx[r] = px(M, c, BH) * mx[r] + px(M, c, AH) * dx[r];
      dx[r] = over_x(M, c, dx[r], 1) + mx[r];
    }
    if (c.v[r] & kDom) sxz[r] = sxz[r] + amu[r] * (dz[r] + dx[r]) * M.dt;
  }
  if (zp) store(fld(M, c, M_VX_Z), mz);
  if (xp) store(fld(M, c, M_VZ_X), mx);
  store(fld(M, c, SXZ), sxz);
}

// F2, one velocity component: vz from dszz/dz (half-point profile) and dsxz/dx, or vx from dsxz/dz and dsxx/dx
// (half-point profile). Only cells with one of the pair in the stencil domain.
template <bool Z>
__device__ __forceinline__ Vals f2_velocity(const March& M, const Cells& c) {
  const bool zp = c.any & kZp, xp = c.any & kXpV;
  constexpr int V = Z ? VZ : VX, MZ = Z ? M_SZZ_Z : M_SXZ_Z, MX = Z ? M_SXZ_X : M_SXX_X;
  constexpr int hz = Z ? 3 : 0, hx = Z ? 0 : 3;  // half-point profiles
  Vals v = load(fld(M, c, V));
  const Vals by = load(med(M, c, Z ? BYA : BYB));
  Vals mz = load_if(zp, fld(M, c, MZ)), mx = load_if(xp, fld(M, c, MX));
  Vals dz = Z ? dpz(M, c, SZZ) : dmz(M, c, SXZ);
  Vals dx = Z ? dmx(M, c, SXZ) : dpx(M, c, SXX);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (c.v[r] & kZp) {
      mz[r] = pz(M, c, r, B_ + hz) * mz[r] + pz(M, c, r, A_ + hz) * dz[r];
      dz[r] = over_z(M, c, r, dz[r], hz) + mz[r];
    }
    if (c.v[r] & kXpV) {
      mx[r] = px(M, c, B_ + hx) * mx[r] + px(M, c, A_ + hx) * dx[r];
      dx[r] = over_x(M, c, dx[r], hx) + mx[r];
    }
    if (c.v[r] & kDom) v[r] = v[r] + (dz[r] + dx[r]) * by[r] * M.dt;
  }
  if (zp) store(fld(M, c, MZ), mz);
  if (xp) store(fld(M, c, MX), mx);
  store(fld(M, c, V), v);
  return v;
}
template <bool Z>
__device__ __forceinline__ void f2_part(const March& M, int z0, int x) {
  const Cells c = cells_at(M, z0, x);
  if (c.any & kDom) f2_velocity<Z>(M, c);
}

// F2 with the illumination, which takes both components.
__device__ __forceinline__ void f2_illum(const March& M, int z0, int x) {
  const Cells c = cells_at(M, z0, x);
  if (!(c.any & kDom)) return;
  Vals e = load(sum(M, c, G_ILLUM));
  const Vals vz = f2_velocity<true>(M, c), vx = f2_velocity<false>(M, c);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (c.v[r] & kDom) e[r] = e[r] + (vz[r] * vz[r] + vx[r] * vx[r]);
  store(sum(M, c, G_ILLUM), e);
}

// B, forward fields: source removal, reverse stresses, the sums of the lambda and mu kernels, the ring's stresses.
__device__ __forceinline__ void b_stress(const March& M, int it, int z0, int x) {
  const Cells c = cells_at(M, z0, x);
  if (!(c.any & (kInner | kSrc | kRing))) return;
  const ShotD& sh = M.S->sh;
  float s1 = 0.0f, s2 = 0.0f, ring[3][R];
  if (c.any & kSrc) {
    s1 = sh.src_szz_r[it];
    s2 = sh.src_sxx_r[it];
  }
  Vals szz = load(fld(M, c, SZZ)), sxx = load(fld(M, c, SXX)), sxz = load(fld(M, c, SXZ));
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (c.v[r] & kRing) {
      const float* p = ring_at(M, c.v[r], it);
      const int len = M.S->g.ring_len;
      ring[0][r] = p[0];
      ring[1][r] = p[len];
      ring[2][r] = p[2 * len];
    }
  if (c.any & kInner) {
    const float dt = M.dt;
    const Vals lam = load(med(M, c, LAM)), l2m = load(med(M, c, L2M)), amu = load(med(M, c, AMU));
    Vals gl = load(sum(M, c, G_LAM)), gm = load(sum(M, c, G_MU)), gt = load(sum(M, c, G_TAU));
    const Vals sa = load(fld(M, c, SZZ_A)), xa = load(fld(M, c, SXX_A)), za = load(fld(M, c, SXZ_A));
    const Vals a = dmz(M, c, VZ), b = dmx(M, c, VX), e1 = dpz(M, c, VX), e2 = dpx(M, c, VZ);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (c.v[r] & kSrc) {
        szz[r] -= s1;
        sxx[r] -= s2;
      }
      if (c.v[r] & kInner) {
        const float e = e1[r] + e2[r];  // dvx_dz + dvz_dx
        szz[r] -= (l2m[r] * a[r] + lam[r] * b[r]) * dt;
        sxx[r] -= (lam[r] * a[r] + l2m[r] * b[r]) * dt;
        sxz[r] -= amu[r] * e * dt;
        gl[r] += (sa[r] + xa[r]) * (a[r] + b[r]);
        gm[r] += sa[r] * a[r] + xa[r] * b[r];
        gt[r] += za[r] * e;
      }
    }
    store(sum(M, c, G_LAM), gl);
    store(sum(M, c, G_MU), gm);
    store(sum(M, c, G_TAU), gt);
  } else if (c.any & kSrc) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (c.v[r] & kSrc) {
        szz[r] -= s1;
        sxx[r] -= s2;
      }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (c.v[r] & kRing) {
      szz[r] = ring[0][r];
      sxz[r] = ring[1][r];
      sxx[r] = ring[2][r];
    }
  store(fld(M, c, SZZ), szz);
  store(fld(M, c, SXZ), sxz);
  store(fld(M, c, SXX), sxx);
}

// B, one adjoint velocity component (el_velocity_adj.cu:57-102) with the memory arrays it feeds; the psi memory terms
// are read only where their CPML coefficient may be non-zero. vx_a: normal stresses differ along x (a_x, K_x), the
// shear stress along z (a_zh, K_zh); vz_a: along z (a_z, K_z) and x (a_xh, K_xh).
template <bool X>
__device__ __forceinline__ void b_velocity(const March& M, int z0, int x) {
  const Cells c = cells_at(M, z0, x);
  if (!(c.any & kDom)) return;
  const bool zp = c.any & kZp, xp = c.any & kXp;
  constexpr int V = X ? VX_A : VZ_A, MX = X ? M_SXX_X : M_SXZ_X, MZ = X ? M_SXZ_Z : M_SZZ_Z;
  const float dt = M.dt;
  const Vals lam = load(med(M, c, LAM)), l2m = load(med(M, c, L2M)), amu = load(med(M, c, AMU));
  Vals mx = load_if(xp, fld(M, c, MX)), mz = load_if(zp, fld(M, c, MZ));
  const Vals by = load_if(xp || zp, med(M, c, X ? BYB : BYA));
  Vals v = load(fld(M, c, V)), q1{}, q2{};
  if (c.any & (X ? kXb : kZb)) q1 = X ? dpx(M, c, M_VX_X) : dpz(M, c, M_VZ_Z);
  if (c.any & (X ? kZb : kXb)) q2 = X ? dmz(M, c, M_VX_Z) : dmx(M, c, M_VZ_X);
  const Vals dzz = X ? dpx(M, c, SZZ_A) : dpz(M, c, SZZ_A);
  const Vals dxx = X ? dpx(M, c, SXX_A) : dpz(M, c, SXX_A);
  const Vals dxz = X ? dmz(M, c, SXZ_A) : dmx(M, c, SXZ_A);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (!(c.v[r] & kDom)) continue;
    float tn = X ? lam[r] * dzz[r] + l2m[r] * dxx[r] : l2m[r] * dzz[r] + lam[r] * dxx[r];
    float ts = amu[r] * dxz[r], t = 0.0f;
    if (c.v[r] & (kXb | kZb)) {  // (a = 0 and K = 1 outside the bands)
      const float an = X ? px(M, c, A_) : pz(M, c, r, A_), as = X ? pz(M, c, r, AH) : px(M, c, AH);
      t = (an != 0.0f ? an * q1[r] : 0.0f) + (as != 0.0f ? as * q2[r] : 0.0f);
      tn = X ? over_x(M, c, tn, 0) : over_z(M, c, r, tn, 0);
      ts = X ? over_z(M, c, r, ts, 1) : over_x(M, c, ts, 1);
    }
    v[r] -= (tn + ts) * dt + t;
    if (c.v[r] & kXp) mx[r] = px(M, c, X ? BH : B_) * mx[r] + by[r] * v[r] * dt;
    if (c.v[r] & kZp) mz[r] = pz(M, c, r, X ? B_ : BH) * mz[r] + by[r] * v[r] * dt;
  }
  store(fld(M, c, V), v);
  if (xp) store(fld(M, c, MX), mx);
  if (zp) store(fld(M, c, MZ), mz);
}

// C, adjoint stresses: residual injection, el_stress_adj.cu:53-97 with the memory arrays in their bands (within two
// cells of the CPML), and the source gradient.
__device__ __forceinline__ void c_stress(const March& M, int it, int z0, int x) {
  const Cells c = cells_at(M, z0, x);
  if (!(c.any & (kDom | kRec))) return;
  const ShotD& sh = M.S->sh;
  const bool xb = c.any & kXb, zb = c.any & kZb;
  int rec[R];
#pragma unroll
  for (int r = 0; r < R; ++r) rec[r] = c.v[r] & kRec ? first_receiver(sh, c.z + r, x) : -1;
  Vals sa = load(fld(M, c, SZZ_A)), xa = load(fld(M, c, SXX_A)), za = load(fld(M, c, SXZ_A));
  const Vals bA = load(med(M, c, BYA)), bB = load(med(M, c, BYB));
  const float dt = M.dt;
  Vals m1 = load_if(xb, fld(M, c, M_VZ_X)), m2 = load_if(xb, fld(M, c, M_VX_X));
  Vals m3 = load_if(zb, fld(M, c, M_VX_Z)), m4 = load_if(zb, fld(M, c, M_VZ_Z));
  const Vals amu = load_if(xb || zb, med(M, c, AMU)), lam = load_if(xb || zb, med(M, c, LAM)),
                l2m = load_if(xb || zb, med(M, c, L2M));
  Vals d1{}, d2{}, d3{}, d4{}, q1{}, q2{}, q3{}, q4{};
  if (c.any & kDom) {
    if (xb) {
      q1 = dpx(M, c, M_SXZ_X);
      q3 = dmx(M, c, M_SXX_X);
    }
    if (zb) {
      q2 = dpz(M, c, M_SXZ_Z);
      q4 = dmz(M, c, M_SZZ_Z);
    }
    d1 = dpx(M, c, VZ_A);
    d2 = dpz(M, c, VX_A);
    d3 = dmx(M, c, VX_A);
    d4 = dmz(M, c, VZ_A);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    inject_res(sh, it, rec[r], c.z + r, x, sa[r], xa[r]);
    if (!(c.v[r] & kDom)) continue;
    float t1 = 0.0f, t2 = 0.0f, t3 = 0.0f;
    if (c.v[r] & (kXb | kZb)) {
      const float ax = px(M, c, A_), az = pz(M, c, r, A_), axh = px(M, c, AH), azh = pz(M, c, r, AH);
      t1 = (ax != 0.0f ? ax * q1[r] : 0.0f) + (az != 0.0f ? az * q2[r] : 0.0f);
      t2 = axh != 0.0f ? axh * q3[r] : 0.0f;
      t3 = azh != 0.0f ? azh * q4[r] : 0.0f;
      d1[r] = over_x(M, c, d1[r], 0);
      d2[r] = over_z(M, c, r, d2[r], 0);
      d3[r] = over_x(M, c, d3[r], 1);
      d4[r] = over_z(M, c, r, d4[r], 1);
    }
    za[r] -= (d1[r] * bA[r] + d2[r] * bB[r]) * dt + t1;
    xa[r] -= bB[r] * d3[r] * dt + t2;
    sa[r] -= bA[r] * d4[r] * dt + t3;
    if (c.v[r] & kXb) {
      m1[r] = px(M, c, BH) * m1[r] + za[r] * amu[r] * dt;
      m2[r] = px(M, c, B_) * m2[r] + (lam[r] * sa[r] + l2m[r] * xa[r]) * dt;
    }
    if (c.v[r] & kZb) {
      m3[r] = pz(M, c, r, BH) * m3[r] + za[r] * amu[r] * dt;
      m4[r] = pz(M, c, r, B_) * m4[r] + (l2m[r] * sa[r] + lam[r] * xa[r]) * dt;
    }
  }
  if (xb) {
    store(fld(M, c, M_VZ_X), m1);
    store(fld(M, c, M_VX_X), m2);
  }
  if (zb) {
    store(fld(M, c, M_VX_Z), m3);
    store(fld(M, c, M_VZ_Z), m4);
  }
  if (c.any & kDom) store(fld(M, c, SXZ_A), za);
  store(fld(M, c, SZZ_A), sa);
  store(fld(M, c, SXX_A), xa);
  if (it >= 1 && (c.any & kSrc)) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (c.v[r] & kSrc) sh.gstf[it - 1] = -(sa[r] + 3.0f * xa[r]) * dt;
  }
}

// C, one forward velocity component taken back to step it - 1 (it >= 1) with its sum of the rho kernel and the ring.
template <bool Z>
__device__ __forceinline__ void c_velocity(const March& M, int it, int z0, int x) {
  const Cells c = cells_at(M, z0, x);
  if (!(c.any & (kInner | kRing))) return;
  constexpr int V = Z ? VZ : VX, G = Z ? G_VA : G_VB;
  Vals v = load(fld(M, c, V));
  float ring[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (c.v[r] & kRing) ring[r] = ring_at(M, c.v[r], it - 1)[(Z ? 3 : 4) * M.S->g.ring_len];
  if (c.any & kInner) {
    const Vals by = load(med(M, c, Z ? BYA : BYB)), w = load(fld(M, c, Z ? VZ_A : VX_A));
    Vals a = load(sum(M, c, G));
    const Vals e1 = Z ? dpz(M, c, SZZ) : dmz(M, c, SXZ), e2 = Z ? dmx(M, c, SXZ) : dpx(M, c, SXX);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (c.v[r] & kInner) {
        const float e = e1[r] + e2[r];
        v[r] -= e * by[r] * M.dt;
        a[r] += w[r] * e;
      }
    store(sum(M, c, G), a);
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (c.v[r] & kRing) v[r] = ring[r];
  store(fld(M, c, V), v);
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
  M.depth = s.nch * 32 * R;
  const float* gz[6] = {S.c.K_z, S.c.a_z, S.c.b_z, S.c.K_zh, S.c.a_zh, S.c.b_zh};
  const float* gx[6] = {S.c.K_x, S.c.a_x, S.c.b_x, S.c.K_xh, S.c.a_xh, S.c.b_xh};
  float* sx = sm + kProfiles * M.nz;
  unsigned* info = reinterpret_cast<unsigned*>(sm + (kProfiles * (M.nz + M.w) + 1) / 2 * 2);  // (8-byte aligned)
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const float scale = q % 3 == 0 ? kQuotientScale : 1.0f;
    for (int i = threadIdx.x; i < M.nz; i += blockDim.x) sm[q * M.nz + i] = gz[q][i] * scale;
    for (int i = threadIdx.x; i < M.w; i += blockDim.x) sx[q * M.w + i] = gx[q][s.xa + i] * scale;
  }
  for (int h = 0; h < 2; ++h) {
    for (int i = threadIdx.x; i < M.nz; i += blockDim.x) sm[(RK + h) * M.nz + i] = 1.0f / gz[3 * h][i] / kQuotientScale;
    for (int i = threadIdx.x; i < M.w; i += blockDim.x) sx[(RK + h) * M.w + i] = 1.0f / gx[3 * h][s.xa + i] / kQuotientScale;
  }
  for (int i = threadIdx.x; i < M.w * M.depth; i += blockDim.x)
    info[i] = cell_info(S, i % M.depth, s.xa + i / M.depth);
  M.prof = sm;
  M.info = info;
  __syncthreads();
  return M;
}

// One forward pass of every shot of the pack over its own record. flags: bit 0
// saves the boundary ring, bit 1 is the timeout test hook (the first block ends
// its first sweep with a wait for a count that nothing publishes, which runs out
// after kInjectWaitNs and raises err; the others follow). B: blocks per SM.
template <int B>
__global__ void __launch_bounds__(kMarchThreads, B)
    k_march_fwd(const __grid_constant__ MarchPack P, int flags, unsigned* done, unsigned* err) {
  const Strip s = strip_of(P, P.fwd, done);
  const ShotSlot& S = P.slots[s.shot];
  extern __shared__ __align__(16) float sm[];
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
      if (threadIdx.x == 0) wait_flag(s.flag, ~0u, err, kInjectWaitNs);
      return;
    }
    if (!strip_sync(s, 2 * it + 1, err)) return;
    if (S.gr.illum)
      for_items(s, first, 1, [&](int, int z0, int x) { f2_illum(M, z0, x); });
    else
      for_items(s, first, 2, [&](int part, int z0, int x) {
        if (part == 0)
          f2_part<true>(M, z0, x);
        else
          f2_part<false>(M, z0, x);
      });
    if (!strip_sync(s, 2 * it + 2, err)) return;
  }
}

// The adjoint pass: sweep C of the last step, then B and C of every step back
// to the first (backward iteration j: step nSteps - 2 - j).
__global__ void __launch_bounds__(kMarchThreads, 1)
    k_march_bwd(const __grid_constant__ MarchPack P, unsigned* done, unsigned* err) {
  const Strip s = strip_of(P, P.bwd, done);
  const ShotSlot& S = P.slots[s.shot];
  extern __shared__ __align__(16) float sm[];
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
  return static_cast<size_t>(std::max(p.fwd.first[p.nshots], p.bwd.first[p.nshots])) * kFlagStride * sizeof(unsigned);
}

namespace {
// Cuts the shots into at most `blocks` strips, the narrowest such ones; at
// least 2 columns, because a stencil reaches two into the next strip. (A
// 96 x 84 grid takes 9.1 / 9.8 / 10.5 / 13.7 us a step with strips of
// 2 / 3 / 4 / 6.) Returns the rounds of a block's warps in a sweep; 0 when
// there are more shots than that or a strip's flags and profiles do not fit
// its shared memory.
int split_shots(const MarchPack& p, int blocks, int parts, MarchSplit& split) {
  int total = 0, rows = 1;
  for (int k = 0; k < p.nshots; ++k) {
    const Geo& g = p.slots[k].g;
    total += g.nx;
    rows = std::max(rows, std::min(g.nz, std::max(g.zact1, p.slots[k].sh.rbz1) + 1));
  }
  for (int w = 2; w <= total; ++w) {
    int n = 0, widest = 0;
    for (int k = 0; k < p.nshots; ++k) {
      const int nx = p.slots[k].g.nx, nb = std::max(1, nx / w);  // (widths w or more)
      split.first[k] = n;
      n += nb;
      widest = std::max(widest, (nx + nb - 1) / nb);
    }
    split.first[p.nshots] = n;
    if (n > blocks) continue;
    const int chunks = (rows + 32 * R - 1) / (32 * R);
    const int items = parts * widest * chunks, warps = std::max(4, std::min(kMarchThreads / 32, items));
    split.threads = 32 * warps;
    split.smem = static_cast<int>((kProfiles * (p.slots[0].g.nz + widest) + 1 + widest * chunks * 32 * R) *
                                  sizeof(float));
    return split.smem <= 48 * 1024 ? (items + warps - 1) / warps : 0;
  }
  return 0;
}
}  // namespace

bool march_plan(MarchPack& p, int sms) {
  for (int k = 0; k < p.nshots; ++k) {
    // Ring rows and offsets from the bases fit their 21 and 31 bits.
    const Geo& g = p.slots[k].g;
    const long long media = p.slots[k].m.aveMu - p.slots[k].m.l2m;
    if (g.ring_len >= 1 << 21 || 18ll * g.ldz * g.nx >= 1ll << 31 || 8 * media >= 1ll << 31) return false;
  }
  // Two blocks per SM in the forward pass (the figures above), unless one of more
  // registers has a single round (a sweep of two 96 x 84 grids: 1.02 us; 1.05 with
  // 64 registers).
  p.fwd_blocks = split_shots(p, sms, 2, p.fwd) == 1 ? 1 : 2;
  return (p.fwd_blocks == 1 || split_shots(p, 2 * sms, 2, p.fwd)) && split_shots(p, sms, 3, p.bwd);
}

cudaError_t launch_march(cudaStream_t s, const MarchPack& p, bool backward, int flags, unsigned* done, unsigned* err) {
  const MarchSplit& split = backward ? p.bwd : p.fwd;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(split.first[p.nshots]);
  cfg.blockDim = dim3(split.threads);
  cfg.dynamicSmemBytes = split.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (backward) return cudaLaunchKernelEx(&cfg, k_march_bwd, p, done, err);
  return p.fwd_blocks == 1 ? cudaLaunchKernelEx(&cfg, k_march_fwd<1>, p, flags, done, err)
                           : cudaLaunchKernelEx(&cfg, k_march_fwd<2>, p, flags, done, err);
}

}  // namespace fwigb
