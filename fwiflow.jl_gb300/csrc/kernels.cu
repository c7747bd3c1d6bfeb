// GB300 (sm_103a) kernels of the elastic FWI operator: 4th-order staggered
// velocity-stress sweeps with CPML, the fused reverse-time / adjoint / imaging
// sweeps, the residual / misfit reduction and the model set-up.
//
// Per time step the reference launches el_stress, add_source, el_velocity,
// recording and five from_bnd kernels forward (libCUFD.cu:202-240) and twelve
// kernels backward (libCUFD.cu:374-445). Here a forward step is two sweeps and
// a backward step is two sweeps:
//   forward  F1: boundary-ring save + stress update + source + recording
//            F2: velocity update
//   backward B : source removal + reverse stress + lambda/mu imaging + stress
//                ring restore + velocity adjoint                 (step it)
//            C : residual injection + stress adjoint + source gradient (it-1)
//                + reverse velocity + rho imaging + velocity ring restore
// The reference scatters the mu and rho kernels with atomicAdd in every step
// (el_stress.cu:113-124, el_velocity.cu:101-110); here the sweeps sum each
// cell's own time-dependent factor and one kernel per call gathers them (see
// "Imaging" below), so there are no atomics and the sums are deterministic.
#include "fwigb_kernels.h"
#include "sweep_cells.cuh"

#include <cudaTypedefs.h>

#include <cstdint>
#include <utility>

namespace fwigb {
namespace {

// Bounded waits (kWaitLimitNs) for the staged tiles: each poll asks the
// hardware to suspend the thread until the barrier phase completes or
// kWaitHintNs pass, so a waiting warp issues a few instructions instead of
// spinning.
constexpr unsigned kWaitHintNs = 1000000u;
// Polls (without a suspend hint) of the injected wait of the timeout test
// hook (stage_wait).
constexpr unsigned kInjectPolls = 256;

// ---- mbarrier / TMA (sm_90+ PTX; issued by one thread per block) ----
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_try_wait_hint(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(kWaitHintNs)
      : "memory");
  return ok != 0;
}
// Waits for phase `parity` of the barrier, at most kWaitLimitNs.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity) {
  if (mbar_try_wait_hint(bar, parity)) return true;
  const unsigned long long t0 = global_timer_ns();
  for (;;) {
    if (mbar_try_wait_hint(bar, parity)) return true;
    if (global_timer_ns() - t0 > kWaitLimitNs) return false;
  }
}
// Polls phase `parity` of the barrier `polls` times without a suspend hint.
__device__ __forceinline__ bool mbar_poll(uint64_t* bar, unsigned parity, unsigned polls) {
  for (unsigned n = 0; n < polls; ++n)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_load_2d(float* dst, const CUtensorMap* tm, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}

// Stages NA arrays of the tile at (z0, x0) into shared memory: one 2-D TMA
// copy each of the box [z0-4, z0-4+BOXZ) x [x0-2, x0+TX+2), zero filled
// outside the grid. The leader initialises the mbarrier (fenced so the copies
// see it) and issues the copies after the block has met the barrier's
// initialisation; the caller then loads its own-cell operands (which overlap
// with the copies) and calls stage_wait.
template <int NA, int TX, int BOXZ, int FIRST = 0>
__device__ __forceinline__ void stage_issue(const TileMaps& mp, float* sm, uint64_t* bar, int z0, int x0) {
  constexpr int N = BOXZ * (TX + 4);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    mbar_expect_tx(bar, NA * N * static_cast<unsigned>(sizeof(float)));
#pragma unroll
    for (int a = 0; a < NA; ++a) tma_load_2d(sm + a * N, &mp.t[FIRST + a], z0 - 4, x0 - 2, bar);
  }
}
__device__ __forceinline__ void stage_init(uint64_t* bar) {
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
}

// Waits (bounded) for the staged tiles. On a timeout the error word is raised
// and the thread waits once more so that copies still in flight land before
// the block exits; the caller then returns without computing. Should that
// second wait run out too, copies may still land after the block has left:
// the host then reports FWIGB_ERR_TIMEOUT for the whole call and its outputs
// are undefined (the next run re-zeroes every field it uses).
// `inject` (the timeout test hook): once the tiles have landed, the thread
// also waits for the barrier's next phase, which nothing completes, so the
// bounded wait runs out with no copy in flight and the error word is raised.
__device__ __forceinline__ bool stage_wait(uint64_t* bar, unsigned* err, bool inject = false) {
  if (!mbar_wait_bounded(bar, 0)) {
    atomicOr(err, 1u);
    mbar_wait_bounded(bar, 0);
    return false;
  }
  if (inject && !mbar_poll(bar, 1, kInjectPolls)) {
    atomicOr(err, 1u);
    return false;
  }
  return true;
}

// sdm / sdp on global memory.
__device__ __forceinline__ float gdm(const float* __restrict__ a, size_t i, size_t s, float r) {
  return (C1 * (a[i] - a[i - s]) - C2 * (a[i + s] - a[i - 2 * s])) * r;
}
__device__ __forceinline__ float gdp(const float* __restrict__ a, size_t i, size_t s, float r) {
  return (C1 * (a[i + s] - a[i]) - C2 * (a[i + 2 * s] - a[i - s])) * r;
}

// Whether the tile of tz depths x tx columns at (z0, x0) meets the bounding
// box of the shot's receivers and source.
__device__ __forceinline__ bool tile_meets_shot_box(const ShotD& sh, int z0, int x0, int tz, int tx) {
  return !(z0 + tz - 1 < sh.rbz0 || z0 > sh.rbz1 || x0 + tx - 1 < sh.rbx0 || x0 > sh.rbx1);
}

// An edge tile without a cell of the reverse-time interior, the source or a receiver.
__device__ __forceinline__ bool outer_tile(const ShotSlot& S, int z0, int x0, int tz, int tx) {
  const Geo& g = S.g;
  const bool inner = z0 + tz > g.zi0 && z0 <= g.zi1 && x0 + tx > g.xi0 && x0 <= g.xi1;
  return !inner && !tile_meets_shot_box(S.sh, z0, x0, tz, tx);
}

// Every sweep is one launch per time step for a pack of shots: a block takes a
// tile of TZ depths x TX columns of one shot (whose slot holds its sub-grid,
// fields, source, receivers and TMA maps), in the order that the host picks
// (TileSplit::order). A tile inside the shot's fast rectangle runs the sweep's
// fast body (the interior form of the reference kernels); a tile inside the mid
// rectangle (no CPML cell) runs the fast body with per-cell ring, band and guard
// handling; any other tile runs its edge body (the full CPML / boundary-ring /
// band logic), in the backward sweeps the shorter body of an outer tile where it
// can. The choice is uniform per block. Blocks past a narrower shot's grid leave
// before staging anything, and so do blocks whose tile lies wholly below row
// zact1 (the nPad rows, where no sweep reads or writes a cell of its own) unless
// it holds the shot's source or a receiver.
//
// Work split. Block (32, TX): lane threadIdx.x covers R adjacent depths
// (R = TZ / 32), threadIdx.y the column. Index arithmetic takes about as many
// instructions as the floating-point work (a cell of F1 on one 1120 x 3152 shot:
// 26 integer and 29 FP32 of 148; 57 and 27 of 164 when a block worked its tile
// split out and every address was 64 bits wide), so the tile split comes with the
// parameters, and a thread's addresses are pointers plus a byte offset in 32 bits
// (SWEEP_ADDRESS). The split and the shifted 64-row tiles together: a gradient's
// sweeps on 608 x 1600 (500 steps) 24.4 -> 23.1 ms, two shots of 352 x 832 (400
// steps) 15.9 -> 15.1 ms, four of 1120 x 3152 (60 steps) 35.4 -> 34.5 ms, 16 of
// 352 x 832 unchanged.
//
// Programmatic dependent launch: a sweep lets the next sweep's blocks be
// scheduled as soon as all of its own blocks have started, and waits
// (pdl_wait) for the previous sweep to complete, and its writes to be
// visible, before it touches any field. The parameter reads, the tile
// classification, the staging-barrier set-up and the loads of the media (which
// no sweep writes) come before the wait and overlap the previous sweep's last
// blocks.
#define SWEEP_KERNEL_TILE(TZ_, BACK_)                                          \
  const int order = P.tiles[0].order;                                          \
  const bool by_tile = K > 1 && (order & kByTile);                             \
  const bool back = order & (BACK_);                                           \
  const int ntx = by_tile ? gridDim.z : gridDim.y, q = by_tile ? blockIdx.z : blockIdx.y; \
  const int tz = by_tile ? blockIdx.y : blockIdx.x, tx = back ? ntx - 1 - q : q; \
  const int shot = K == 1 ? 0 : by_tile ? blockIdx.x : back ? gridDim.z - 1 - blockIdx.z : blockIdx.z; \
  const Geo& g0 = P.slots[shot].g;                                             \
  const TileSplit& ts = P.tiles[shot];                                         \
  const int z0 = tz * (TZ_) + ts.zoff, x0 = tx * TX;                           \
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");              \
  if (z0 >= g0.nz || x0 >= g0.nx) return;                                      \
  if (z0 > g0.zact1 && !tile_meets_shot_box(P.slots[shot].sh, z0, x0, (TZ_), TX)) return; \
  const bool fast = tz >= ts.ftz0 && tz < ts.ftz1 && tx >= ts.ftx0 && tx < ts.ftx1; \
  const bool mid = !fast && tz >= ts.mtz0 && tz < ts.mtz1 && tx >= ts.mtx0 && tx < ts.mtx1;

#define SWEEP_BODY_SLOT()                                                      \
  const ShotSlot& S = P.slots[shot];                                           \
  const Geo& g = S.g;                                                          \
  const Fields& f = S.f;                                                       \
  const MediaD& m = S.m;                                                       \
  const ShotD& sh = S.sh;

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A thread's own cells are at `base` + `off` bytes from an array's start: with
// WIDE the tile's 64-bit offset (block-uniform) and the thread's from there, else
// a 32-bit offset alone, for arrays of less than 4 GB. Without the additions to
// every pointer F2 needs no spills: 16 shots of 352 x 832 27.0 -> 24.5 us, 608-row
// windows of 24 shots 89.8 -> 84.8, four 1120 x 3152 shots 73.4 -> 68.2; F1 and C
// 1 % less. B, whose offset then costs a spilled register, keeps the uniform base
// (206.6 us on those windows; 213.0 without).
#define SWEEP_ADDRESS(R_, WIDE_)                                               \
  const size_t base =                                                          \
      (WIDE_) ? static_cast<size_t>((static_cast<long long>(x0) * g.ldz + z0) * static_cast<long long>(sizeof(float))) \
              : 0;                                                             \
  const unsigned off =                                                         \
      (((WIDE_) ? threadIdx.y : x0 + threadIdx.y) * static_cast<unsigned>(g.ldz) + ((WIDE_) ? 0 : z0) + \
       (R_) * threadIdx.x) *                                                   \
      static_cast<unsigned>(sizeof(float));

// Fast and mid tiles lie wholly inside the grid; b is the index of the thread's
// first cell in a staged box. `special` marks the tiles that meet the bounding
// box of the shot's receivers and source.
#define SWEEP_FAST(TZ_, BOXZ_, R_, WIDE_)                                      \
  SWEEP_BODY_SLOT()                                                            \
  const bool special = tile_meets_shot_box(sh, z0, x0, (TZ_), TX);             \
  constexpr int N = (BOXZ_) * (TX + 4);                                        \
  SWEEP_ADDRESS(R_, WIDE_)                                                     \
  const int b = (threadIdx.y + 2) * (BOXZ_) + (R_) * threadIdx.x + 4;          \
  const int z = z0 + (R_) * static_cast<int>(threadIdx.x), x = x0 + threadIdx.y; \
  SWEEP_SMEM()

#define SWEEP_SMEM()                                                           \
  extern __shared__ __align__(128) float sm[];                                 \
  __shared__ __align__(8) uint64_t bar;                                        \
  stage_init(&bar);
#define SWEEP_TMA(NA, BOXZ_) stage_issue<NA, TX, (BOXZ_)>(P.maps[shot], sm, &bar, z0, x0);

// Edge tiles: the thread's first cell (z, x), its global index i, its box index
// b, whether it lies in the grid (`live`: depths may also lie above it, in a
// shifted tile grid) and how many of its R depths do (rows_in). A thread with no
// cell in the grid takes part in the staging set-up only.
#define SWEEP_EDGE(BOXZ_, R_)                                                  \
  SWEEP_BODY_SLOT()                                                            \
  const CpmlD& c = S.c;                                                        \
  constexpr int N = (BOXZ_) * (TX + 4);                                        \
  const size_t ldz = static_cast<size_t>(g.ldz);                               \
  const int z = z0 + (R_) * static_cast<int>(threadIdx.x), x = x0 + threadIdx.y; \
  const bool live = z >= 0 && z < g.nz && x < g.nx;                            \
  const int rows_in = live ? g.nz - z : 0;                                     \
  const size_t i = static_cast<size_t>(x) * ldz + z;                           \
  const int b = (threadIdx.y + 2) * (BOXZ_) + (R_) * threadIdx.x + 4;          \
  (void)rows_in;                                                               \
  SWEEP_SMEM()

// Which of an edge thread's cells are in the stencil domain
// (dom) and in the CPML along z (zc), and their address as in fast tiles (live
// threads: even depths, so a pair lies in the padded column).
#define SWEEP_EDGE_CELLS(R_, WIDE_)                                            \
  SWEEP_ADDRESS(R_, WIDE_)                                                     \
  bool dom[R_], zc[R_], any_dom = false, any_z = false;                        \
  _Pragma("unroll") for (int r = 0; r < (R_); ++r) {                           \
    dom[r] = in_box(z + r, x, g.zs0, g.zs1, g.xs0, g.xs1);                     \
    zc[r] = dom[r] && (z + r < g.nPml || z + r > g.zpml_hi);                   \
    any_dom |= dom[r];                                                         \
    any_z |= zc[r];                                                            \
  }                                                                            \
  (void)i;

// Values of the thread's R depths that lie in the grid (rows_in of them);
// the others are left 0.
template <int R>
__device__ __forceinline__ void ldrows(const float* p, int rows_in, float (&v)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = r < rows_in ? p[r] : 0.0f;
}

// Own-cell values of a thread's R adjacent depths at a byte offset from a
// block-uniform pointer (8-byte paired when R == 2: even depth, ldz a
// multiple of 32).
template <int R>
__device__ __forceinline__ void ldo(const float* p, size_t base, unsigned off, float (&v)[R]) {
  const char* q = reinterpret_cast<const char*>(p) + base + off;
  if constexpr (R == 2) {
    const float2 t = *reinterpret_cast<const float2*>(q);
    v[0] = t.x;
    v[1] = t.y;
  } else {
    v[0] = *reinterpret_cast<const float*>(q);
  }
}
template <int R>
__device__ __forceinline__ void sto(float* p, size_t base, unsigned off, const float (&v)[R]) {
  char* q = reinterpret_cast<char*>(p) + base + off;
  if constexpr (R == 2)
    *reinterpret_cast<float2*>(q) = make_float2(v[0], v[1]);
  else
    *reinterpret_cast<float*>(q) = v[0];
}

// Asynchronous copy of a thread's own values into its place in shared memory,
// and the wait for the thread's own copies (each thread reads only what it
// copied, so there is no barrier).
template <int R>
__device__ __forceinline__ void ldasync(float* dst, const float* p, size_t base, unsigned off) {
  const char* q = reinterpret_cast<const char*>(p) + base + off;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(q), "n"(4 * R) : "memory");
}
__device__ __forceinline__ void ldasync_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The media arrays are read by every sweep and, in a batched launch, by every
// shot of the pack (their sub-grids are windows of the same model): their
// loads carry an L2 evict-last policy so that the streamed fields do not push
// them out of L2 (createpolicy / ld.global.L2::cache_hint).
__device__ __forceinline__ uint64_t media_policy() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
template <int R>
__device__ __forceinline__ void ldm(const float* a, size_t base, unsigned off, float (&v)[R], uint64_t pol) {
  const char* q = reinterpret_cast<const char*>(a) + base + off;
  if constexpr (R == 2)
    asm("ld.global.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(v[0]), "=f"(v[1]) : "l"(q), "l"(pol));
  else
    asm("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v[0]) : "l"(q), "l"(pol));
}

// Paired shared-memory loads of two adjacent depths (even box index).
__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }

// 4th-order staggered difference from its four samples: (C1 (p - q) -
// C2 (s - t)) r, the expression of sdm / sdp.
__device__ __forceinline__ float dd(float p, float q, float s, float t, float r) {
  return (C1 * (p - q) - C2 * (s - t)) * r;
}

// The differences of a staged array at the thread's R depths: along z (Dm, Dp)
// and along x. With two depths (b even) the float2 at b + o (o even) holds
// both depths' samples at offset o, so a z stencil of both takes the pairs at
// b - 2, b, b + 2 and an x stencil those at b + k BOXZ.
template <int R>
__device__ __forceinline__ void dmz(const float* a, int b, float r, float (&o)[R]) {
  if constexpr (R == 1) {
    o[0] = sdm(a, b, 1, r);
  } else {
    const float2 m = ld2(a + b - 2), c = ld2(a + b), p = ld2(a + b + 2);
    o[0] = dd(c.x, m.y, c.y, m.x, r);
    o[1] = dd(c.y, c.x, p.x, m.y, r);
  }
}
template <int R>
__device__ __forceinline__ void dpz(const float* a, int b, float r, float (&o)[R]) {
  if constexpr (R == 1) {
    o[0] = sdp(a, b, 1, r);
  } else {
    const float2 m = ld2(a + b - 2), c = ld2(a + b), p = ld2(a + b + 2);
    o[0] = dd(c.y, c.x, p.x, m.y, r);
    o[1] = dd(p.x, c.y, p.y, c.x, r);
  }
}
template <int R, int BOXZ>
__device__ __forceinline__ void dmx(const float* a, int b, float r, float (&o)[R]) {
  if constexpr (R == 1) {
    o[0] = sdm(a, b, BOXZ, r);
  } else {
    const float2 c = ld2(a + b), m = ld2(a + b - BOXZ), p = ld2(a + b + BOXZ), m2 = ld2(a + b - 2 * BOXZ);
    o[0] = dd(c.x, m.x, p.x, m2.x, r);
    o[1] = dd(c.y, m.y, p.y, m2.y, r);
  }
}
template <int R, int BOXZ>
__device__ __forceinline__ void dpx(const float* a, int b, float r, float (&o)[R]) {
  if constexpr (R == 1) {
    o[0] = sdp(a, b, BOXZ, r);
  } else {
    const float2 c = ld2(a + b), p = ld2(a + b + BOXZ), p2 = ld2(a + b + 2 * BOXZ), m = ld2(a + b - BOXZ);
    o[0] = dd(p.x, c.x, p2.x, m.x, r);
    o[1] = dd(p.y, c.y, p2.y, m.y, r);
  }
}
template <int R>
__device__ __forceinline__ void own(const float* a, int b, float (&o)[R]) {
  if constexpr (R == 1) {
    o[0] = a[b];
  } else {
    const float2 c = ld2(a + b);
    o[0] = c.x;
    o[1] = c.y;
  }
}

// Register budgets (measured on GB300 over the tile widths; the sweeps wait
// on memory latency, so resident warps count for more than the bytes
// spilled): forward sweeps 32 registers (64 warps per SM). Backward sweeps:
// NT resident threads per SM, so 65536 / NT registers: with one cell per
// thread 2048 (32 registers) or 1536 (40 registers), picked by the autotuner;
// with two cells 1024 (64 registers).
#define FWD_BOUNDS __launch_bounds__(32 * TX, 2048 / (32 * TX))
#define BWD_BOUNDS __launch_bounds__(32 * TX, (NT / (32 * TX)) > 0 ? (NT / (32 * TX)) : 1)

// psi differences of two memory arrays at the thread's cells in the stencil domain: Dm of the first and Dp of the
// second along z; Dp of the first and Dm of the second along x.
template <int R>
__device__ __forceinline__ void psi_z(const float* a, const float* d, const bool (&dom)[R], size_t i, float r,
                                      float (&pa)[R], float (&pd)[R]) {
#pragma unroll
  for (int k = 0; k < R; ++k) {
    pa[k] = dom[k] ? gdm(a, i + k, 1, r) : 0.0f;
    pd[k] = dom[k] ? gdp(d, i + k, 1, r) : 0.0f;
  }
}
template <int R>
__device__ __forceinline__ void psi_x(const float* a, const float* d, const bool (&dom)[R], size_t i, size_t ldz,
                                      float r, float (&pa)[R], float (&pd)[R]) {
#pragma unroll
  for (int k = 0; k < R; ++k) {
    pa[k] = dom[k] ? gdp(a, i + k, ldz, r) : 0.0f;
    pd[k] = dom[k] ? gdm(d, i + k, ldz, r) : 0.0f;
  }
}

// One CPML convolution (el_stress.cu:64-85): the memory value and the derivative. CALL as in over().
template <bool CALL = true>
__device__ __forceinline__ void cpml_fwd(const float4& q, float& mm, float& d) {
  mm = q.z * mm + q.y * d;
  d = over<CALL>(d, q.x, q.w) + mm;
}

// ---------------------------------------------------------------------------
// F1: el_stress (el_stress.cu:50-88) + add_source (utilities.cu:521-541) +
// recording (utilities.cu:557-567) + from_bnd of the 5 fields (Boundary.cu:55-76).
// Staged: vz, vx.
//
// Forward edge bodies. A load behind a store cannot be moved ahead of it (the
// arrays might alias), so a body of one cell after the other makes up to ten
// dependent trips to memory. Here a thread asks for the own values and the CPML
// memory values of its R depths, as pairs, before it waits for the staged
// tiles; a cell with CPML along both directions reads the x values when it is
// done with those along z. F2 keeps the memory values in flight by cp.async
// into shared memory, which holds no register. F1, which takes more registers
// a cell, loads them into registers, the shear stress first: the shared memory
// would come out of its L1 (on 1120 x 3152 grids 101 us; 97 this way).
// us a sweep, one cell after the other / this: 16 shots of 352 x 832 F1 40.8 /
// 38.2, F2 32.0 / 29.0; 608-row windows of 24 shots F1 116.3 / 111.0, F2 102.9
// / 94.8; one 608 x 1600 shot F1 8.7 / 8.4, F2 7.6 / 7.1; four 1120 x 3152
// shots F1 96.9 / 97.1, F2 80.7 / 78.1. (F2 with registers: 30.0, 97.6, 7.4,
// 78.4.) F2 works the z terms off before it forms the x ones, and has large
// quotients in place, or it spills: 16 shots of 352 x 832 26.2 us (27.8), eight
// of 608 x 1600 41.7 (44.4), four of 1120 x 3152 71.2 (75.5).
template <int TX, int K, int R, bool WIDE>
__device__ __forceinline__ void fwd_stress_edge(const SweepPack<K>& P, int shot, int z0, int x0, int it, int save,
                                                bool inject, unsigned* err) {
  constexpr int BOXZ = 32 * R + 8;
  SWEEP_EDGE(BOXZ, R)
  SWEEP_EDGE_CELLS(R, WIDE)
  const bool xc = any_dom && (x < g.nPml || x > g.xpml_hi_s);
  float lam[R], l2m[R], amu[R], szz[R], sxx[R], sxz[R], m1[R], m2[R];
  if (live) {
    ldo<R>(m.lam, base, off, lam);
    ldo<R>(m.l2m, base, off, l2m);
    ldo<R>(m.aveMu, base, off, amu);
  }
  pdl_wait();
  SWEEP_TMA(2, BOXZ)
  if (!live) return;
  ldo<R>(f.szz, base, off, szz);
  ldo<R>(f.sxx, base, off, sxx);
  ldo<R>(f.sxz, base, off, sxz);
  if (any_z) {
    ldo<R>(f.m_dvz_dz, base, off, m1);
    ldo<R>(f.m_dvx_dz, base, off, m2);
  } else if (xc) {
    ldo<R>(f.m_dvx_dx, base, off, m1);
    ldo<R>(f.m_dvz_dx, base, off, m2);
  }
  const bool special = tile_meets_shot_box(sh, z0, x0, 32 * R, TX);
  if (!stage_wait(&bar, err, inject)) return;
  const float* s_vz = sm;
  const float* s_vx = sm + N;
  if (save) {
#pragma unroll
    for (int r = 0; r < R; ++r) ring_save(g, S.st, it, z + r, x, szz[r], sxz[r], sxx[r], s_vz[b + r], s_vx[b + r]);
  }
  if (any_dom) {
    {
      float dz[R], dx[R];
      dpz<R>(s_vx, b, g.rdz, dz);
      dpx<R, BOXZ>(s_vz, b, g.rdx, dx);
      if (any_z) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (zc[r]) cpml_fwd(__ldg(c.q_zh + z + r), m2[r], dz[r]);
        sto<R>(f.m_dvx_dz, base, off, m2);
        if (xc) ldo<R>(f.m_dvz_dx, base, off, m2);
      }
      if (xc) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (dom[r]) cpml_fwd(__ldg(c.q_xh + x), m2[r], dx[r]);
        sto<R>(f.m_dvz_dx, base, off, m2);
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (dom[r]) sxz[r] = sxz[r] + amu[r] * (dz[r] + dx[r]) * g.dt;
      sto<R>(f.sxz, base, off, sxz);
    }
    float dz[R], dx[R];
    dmz<R>(s_vz, b, g.rdz, dz);
    dmx<R, BOXZ>(s_vx, b, g.rdx, dx);
    if (any_z) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (zc[r]) cpml_fwd(__ldg(c.q_z + z + r), m1[r], dz[r]);
      sto<R>(f.m_dvz_dz, base, off, m1);
      if (xc) ldo<R>(f.m_dvx_dx, base, off, m1);
    }
    if (xc) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (dom[r]) cpml_fwd(__ldg(c.q_x + x), m1[r], dx[r]);
      sto<R>(f.m_dvx_dx, base, off, m1);
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (dom[r]) {
        szz[r] += (l2m[r] * dz[r] + lam[r] * dx[r]) * g.dt;
        sxx[r] += (lam[r] * dz[r] + l2m[r] * dx[r]) * g.dt;
      }
  }
  if (special) {
    // The velocity sweep that follows does not change the stresses, so the
    // sample of step it+1 is taken here.
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (z + r == sh.src_z && x == sh.src_x) {
        szz[r] += sh.src_szz[it];
        sxx[r] += sh.src_sxx[it];
      }
      record(sh, it, first_receiver(sh, z + r, x), z + r, x, szz[r], sxx[r]);
    }
  }
  if (any_dom || special) {
    sto<R>(f.szz, base, off, szz);
    sto<R>(f.sxx, base, off, sxx);
  }
}

// F2: el_velocity, isFor = true (el_velocity.cu:45-82). Staged: szz, sxx, sxz.
template <int TX, int K, int R, bool WIDE>
__device__ __forceinline__ void fwd_velocity_edge(const SweepPack<K>& P, int shot, int z0, int x0, unsigned* err) {
  constexpr int BOXZ = 32 * R + 8;
  SWEEP_EDGE(BOXZ, R)
  SWEEP_EDGE_CELLS(R, WIDE)
  constexpr int M = 32 * TX * R;  // floats between the thread's places in the shared arrays behind the staged ones
  float* mem = sm + 3 * N + R * (threadIdx.y * 32 + threadIdx.x);
  (void)sh;
  const bool xc = any_dom && (x < g.nPml || x > g.xpml_hi_v);
  float bA[R], bB[R], vz[R], vx[R];
  if (any_dom) {
    ldo<R>(m.bycA, base, off, bA);
    ldo<R>(m.bycB, base, off, bB);
  }
  pdl_wait();
  SWEEP_TMA(3, BOXZ)
  if (!live) return;
  if (any_z) {
    ldasync<R>(mem, f.m_dszz_dz, base, off);
    ldasync<R>(mem + M, f.m_dsxz_dz, base, off);
  }
  if (xc) {
    ldasync<R>(mem + 2 * M, f.m_dsxz_dx, base, off);
    ldasync<R>(mem + 3 * M, f.m_dsxx_dx, base, off);
  }
  if (any_dom) {
    ldo<R>(f.vz, base, off, vz);
    ldo<R>(f.vx, base, off, vx);
  }
  ldasync_wait();
  if (!stage_wait(&bar, err) || !any_dom) return;
  const float* s_szz = sm;
  const float* s_sxx = sm + N;
  const float* s_sxz = sm + 2 * N;
  float dszz_dz[R], dsxz_dz[R];
  dpz<R>(s_szz, b, g.rdz, dszz_dz);
  dmz<R>(s_sxz, b, g.rdz, dsxz_dz);
  if (any_z) {
    float m1[R], m2[R];
    own<R>(mem, 0, m1);
    own<R>(mem + M, 0, m2);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (zc[r]) {
        cpml_fwd<false>(__ldg(c.q_zh + z + r), m1[r], dszz_dz[r]);
        cpml_fwd<false>(__ldg(c.q_z + z + r), m2[r], dsxz_dz[r]);
      }
    sto<R>(f.m_dszz_dz, base, off, m1);
    sto<R>(f.m_dsxz_dz, base, off, m2);
  }
  float dsxz_dx[R], dsxx_dx[R];
  dmx<R, BOXZ>(s_sxz, b, g.rdx, dsxz_dx);
  dpx<R, BOXZ>(s_sxx, b, g.rdx, dsxx_dx);
  if (xc) {
    float m1[R], m2[R];
    own<R>(mem + 2 * M, 0, m1);
    own<R>(mem + 3 * M, 0, m2);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (dom[r]) {
        cpml_fwd<false>(__ldg(c.q_x + x), m1[r], dsxz_dx[r]);
        cpml_fwd<false>(__ldg(c.q_xh + x), m2[r], dsxx_dx[r]);
      }
    sto<R>(f.m_dsxz_dx, base, off, m1);
    sto<R>(f.m_dsxx_dx, base, off, m2);
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (dom[r]) {
      vz[r] = vz[r] + (dszz_dz[r] + dsxz_dx[r]) * bA[r] * g.dt;
      vx[r] = vx[r] + (dsxz_dz[r] + dsxx_dx[r]) * bB[r] * g.dt;
    }
  sto<R>(f.vz, base, off, vz);
  sto<R>(f.vx, base, off, vx);
  if (S.gr.illum) {
    float e[R];
    ldo<R>(S.gr.illum, base, off, e);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (dom[r]) e[r] += vz[r] * vz[r] + vx[r] * vx[r];
    sto<R>(S.gr.illum, base, off, e);
  }
}

// ---------------------------------------------------------------------------
// Imaging. The reference adds to the lambda, mu and rho kernels at every step
// (el_stress.cu:110-124, el_velocity.cu:98-110), the mu kernel through the
// chain rule of the 2x2 harmonic average and the rho kernel through that of
// the two buoyancies. The chain rules do not depend on time, so the sweeps
// sum over time only what does, at the cell itself,
//   gr.lam += (szz_a + sxx_a)(dvz/dz + dvx/dx)     gr.tau += sxz_a (dvx/dz + dvz/dx)
//   gr.mu  += szz_a dvz/dz + sxx_a dvx/dx          gr.va += vz_a (dszz/dz + dsxz/dx)
//                                                  gr.vb += vx_a (dsxz/dz + dsxx/dx)
// and k_reduce_grads applies them once per call. Gathering them in every step
// took the neighbours' strains and divergences again, and the media values of
// the chain rules; summing two values more per cell instead takes less: B 254
// -> 234 us and C 257 -> 246 us a step of 24 aperture-windowed 608-row shots,
// 16.5 -> 14.3 us and 15.4 -> 14.0 us on one 608 x 1600 shot.

// B: add_source(-) + el_stress(isFor=false) with the sums of the lambda / mu
// kernels + to_bnd(stress) + el_velocity_adj. Staged: vz, vx, szz_a, sxx_a, sxz_a.
template <int TX, int K, int R>
__device__ __forceinline__ void bwd_B_edge(const SweepPack<K>& P, int shot, int z0, int x0, int j, unsigned* err) {
  constexpr int BOXZ = 32 * R + 8;
  SWEEP_EDGE(BOXZ, R)
  const Grads& gr = S.gr;
  float p_lam[R], p_l2m[R], p_amu[R];
  float p_szz[R], p_sxx[R], p_sxz[R], p_vza[R], p_vxa[R];
  ldrows<R>(m.lam + i, rows_in, p_lam);
  ldrows<R>(m.l2m + i, rows_in, p_l2m);
  ldrows<R>(m.aveMu + i, rows_in, p_amu);
  pdl_wait();
  SWEEP_TMA(5, BOXZ)
  ldrows<R>(f.szz + i, rows_in, p_szz);
  ldrows<R>(f.sxx + i, rows_in, p_sxx);
  ldrows<R>(f.sxz + i, rows_in, p_sxz);
  ldrows<R>(f.vz_a + i, rows_in, p_vza);
  ldrows<R>(f.vx_a + i, rows_in, p_vxa);
  if (!live) return;
  const StoreD& st = S.st;
  const int it = S.nSteps - 2 - j;  // this shot's time step at backward iteration j
  const float dt = g.dt;
  if (!stage_wait(&bar, err)) return;
  const float* s_vz = sm;
  const float* s_vx = sm + N;
  const float* s_szz_a = sm + 2 * N;
  const float* s_sxx_a = sm + 3 * N;
  const float* s_sxz_a = sm + 4 * N;
  auto cell = [&](const int r, const int z, const size_t i, const int b) {
  float szz = p_szz[r], sxx = p_sxx[r], sxz = p_sxz[r];
  const float lam = p_lam[r], l2m = p_l2m[r], amu = p_amu[r];
  const float va_z = p_vza[r], va_x = p_vxa[r];
  const bool interior = in_box(z, x, g.zi0, g.zi1, g.xi0, g.xi1);
  const bool src = (z == sh.src_z && x == sh.src_x);
  const int k = ring_index(g, z, x);
  if (interior || src || k >= 0) {
    if (src) {
      szz -= sh.src_szz_r[it];
      sxx -= sh.src_sxx_r[it];
    }
    if (interior) {
      const float dvz_dz = sdm(s_vz, b, 1, g.rdz);
      const float dvx_dx = sdm(s_vx, b, BOXZ, g.rdx);
      const float e = sdp(s_vx, b, 1, g.rdz) + sdp(s_vz, b, BOXZ, g.rdx);  // dvx_dz + dvz_dx
      szz -= (l2m * dvz_dz + lam * dvx_dx) * dt;
      sxx -= (lam * dvz_dz + l2m * dvx_dx) * dt;
      sxz -= amu * e * dt;
      const float sa = s_szz_a[b], xa = s_sxx_a[b];
      gr.lam[i] += (sa + xa) * (dvz_dz + dvx_dx);
      gr.mu[i] += sa * dvz_dz + xa * dvx_dx;
      gr.tau[i] += s_sxz_a[b] * e;
    }
    if (k >= 0) {
      const float* p = st.base + static_cast<size_t>(it) * 5 * g.ring_len + k;
      szz = p[0];
      sxz = p[g.ring_len];
      sxx = p[2 * g.ring_len];
    }
    f.szz[i] = szz;
    f.sxx[i] = sxx;
    f.sxz[i] = sxz;
  }
  // el_velocity_adj (el_velocity_adj.cu:57-102); the psi memory terms are
  // read only where their CPML coefficient is non-zero.
  if (!in_box(z, x, g.zs0, g.zs1, g.xs0, g.xs1)) return;
  const bool zp = (z < g.nPml) || (z > g.zpml_hi);
  const bool xp = (x < g.nPml) || (x > g.xpml_hi_s);
  {
    const float4 cx = __ldg(c.q_x + x), czh = __ldg(c.q_zh + z);  // {K, a, b, 1 / K}, scaled for over()
    const float dszz_dx = -sdp(s_szz_a, b, BOXZ, g.rdx);
    const float dsxx_dx = -sdp(s_sxx_a, b, BOXZ, g.rdx);
    const float dsxz_dz = -sdm(s_sxz_a, b, 1, g.rdz);
    float t = over(lam * dszz_dx, cx.x, cx.w) * dt + over(l2m * dsxx_dx, cx.x, cx.w) * dt +
              over(amu, czh.x, czh.w) * dsxz_dz * dt;
    if (cx.y != 0.0f) t += cx.y * (-gdp(f.m_dvx_dx, i, ldz, g.rdx));
    if (czh.y != 0.0f) t += czh.y * (-gdm(f.m_dvx_dz, i, 1, g.rdz));
    const float v = va_x + t;
    f.vx_a[i] = v;
    if (xp || zp) {
      const float bB = m.bycB[i];
      if (xp) f.m_dsxx_dx[i] = c.b_xh[x] * f.m_dsxx_dx[i] + bB * v * dt;
      if (zp) f.m_dsxz_dz[i] = c.b_z[z] * f.m_dsxz_dz[i] + bB * v * dt;
    }
  }
  {
    const float4 cz = __ldg(c.q_z + z), cxh = __ldg(c.q_xh + x);
    const float dszz_dz = -sdp(s_szz_a, b, 1, g.rdz);
    const float dsxx_dz = -sdp(s_sxx_a, b, 1, g.rdz);
    const float dsxz_dx = -sdm(s_sxz_a, b, BOXZ, g.rdx);
    float t = over(l2m * dszz_dz, cz.x, cz.w) * dt + over(lam * dsxx_dz, cz.x, cz.w) * dt +
              over(amu, cxh.x, cxh.w) * dsxz_dx * dt;
    if (cz.y != 0.0f) t += cz.y * (-gdp(f.m_dvz_dz, i, 1, g.rdz));
    if (cxh.y != 0.0f) t += cxh.y * (-gdm(f.m_dvz_dx, i, ldz, g.rdx));
    const float v = va_z + t;
    f.vz_a[i] = v;
    if (xp || zp) {
      const float bA = m.bycA[i];
      if (xp) f.m_dsxz_dx[i] = c.b_x[x] * f.m_dsxz_dx[i] + bA * v * dt;
      if (zp) f.m_dszz_dz[i] = c.b_zh[z] * f.m_dszz_dz[i] + bA * v * dt;
    }
  }
  };
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (z + r < g.nz) cell(r, z + r, i + r, b + r);
}

// B of an outer tile: an edge tile without a cell of the reverse-time interior,
// the source or a receiver, so that of the forward fields only the ring's
// stresses are restored and only the adjoint stresses are staged. With an absorbing
// layer as thick as a tile these are all tiles of the CPML but the few around
// the source and receivers. They are bound by their memory trips as the forward
// edge tiles are: all values but the x ones of the corners are asked for before
// the staged tiles are waited for, which this body's fewer operands leave
// registers for. us a sweep, edge body / this: 16 shots of 352 x 832 B 68.8 /
// 66.1, C 71.5 / 67.9; 608-row windows of 24 shots B 224.1 / 220.2, C 226.1 /
// 219.7; one 608 x 1600 shot B 13.5 / 13.1, C 13.8 / 12.6; four 1120 x 3152
// shots B 202.4 / 203.8, C 185.9 / 183.9.
template <int TX, int K, int R>
__device__ __forceinline__ void bwd_B_outer(const SweepPack<K>& P, int shot, int z0, int x0, int j, unsigned* err) {
  constexpr int BOXZ = 32 * R + 8;
  SWEEP_EDGE(BOXZ, R)
  SWEEP_EDGE_CELLS(R, true)
  (void)sh;
  const bool xc = any_dom && (x < g.nPml || x > g.xpml_hi_s);
  // Where there is something to read along x and z: in the CPML, and where a psi coefficient may not be zero.
  const bool xq = xc || (any_dom && (x <= g.xband_lo || x >= g.xband_hi));
  const bool zq = any_z || (any_dom && (z <= g.zband_lo || z + R - 1 >= g.zband_hi));
  float lam[R], l2m[R], amu[R], bA[R], bB[R], va_x[R], va_z[R], p1[R], p2[R], m1[R], m2[R];
  if (any_dom) {
    ldo<R>(m.lam, base, off, lam);
    ldo<R>(m.l2m, base, off, l2m);
    ldo<R>(m.aveMu, base, off, amu);
    ldo<R>(m.bycA, base, off, bA);
    ldo<R>(m.bycB, base, off, bB);
  }
  pdl_wait();
  stage_issue<3, TX, BOXZ, 2>(P.maps[shot], sm, &bar, z0, x0);
  if (!live) return;
  // The psi terms' differences and the memory values, along z, or along x where there are none along z.
  if (zq) {
    psi_z<R>(f.m_dvx_dz, f.m_dvz_dz, dom, i, g.rdz, p1, p2);
    ldo<R>(f.m_dsxz_dz, base, off, m1);
    ldo<R>(f.m_dszz_dz, base, off, m2);
  } else if (xq) {
    psi_x<R>(f.m_dvx_dx, f.m_dvz_dx, dom, i, ldz, g.rdx, p1, p2);
    ldo<R>(f.m_dsxx_dx, base, off, m1);
    ldo<R>(f.m_dsxz_dx, base, off, m2);
  }
  if (any_dom) {
    ldo<R>(f.vx_a, base, off, va_x);
    ldo<R>(f.vz_a, base, off, va_z);
  }
  const float* ring = S.st.base + static_cast<size_t>(S.nSteps - 2 - j) * 5 * g.ring_len;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int k = ring_index(g, z + r, x);
    if (k >= 0) {
      const float s1 = ring[k], s2 = ring[k + g.ring_len], s3 = ring[k + 2 * g.ring_len];
      f.szz[i + r] = s1;
      f.sxz[i + r] = s2;
      f.sxx[i + r] = s3;
    }
  }
  if (!stage_wait(&bar, err) || !any_dom) return;
  const float* s_szz_a = sm;
  const float* s_sxx_a = sm + N;
  const float* s_sxz_a = sm + 2 * N;
  const float dt = g.dt;
  // el_velocity_adj (el_velocity_adj.cu:57-102); a psi term counts only where its CPML coefficient is not zero.
  {
    float d1[R], d2[R], d3[R], q1[R], n1[R];
    dpx<R, BOXZ>(s_szz_a, b, g.rdx, d1);
    dpx<R, BOXZ>(s_sxx_a, b, g.rdx, d2);
    dmz<R>(s_sxz_a, b, g.rdz, d3);
    if (xq && zq) {
      ldo<R>(f.m_dsxx_dx, base, off, n1);
#pragma unroll
      for (int r = 0; r < R; ++r) q1[r] = dom[r] ? gdp(f.m_dvx_dx, i + r, ldz, g.rdx) : 0.0f;
    }
    const float4 cx = __ldg(c.q_x + x);  // {K, a, b, 1 / K}, scaled for over()
    const float bxh = xc ? __ldg(c.b_xh + x) : 0.0f;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (dom[r]) {
        float t = 0.0f;
        const float4 czh = __ldg(c.q_zh + z + r);
        if (xq && cx.y != 0.0f) t += cx.y * (zq ? q1[r] : p1[r]);
        if (zq && czh.y != 0.0f) t += czh.y * p1[r];
        va_x[r] -= (over(lam[r] * d1[r] + l2m[r] * d2[r], cx.x, cx.w) + over(amu[r] * d3[r], czh.x, czh.w)) * dt + t;
        const float add = bB[r] * va_x[r] * dt;
        if (xc && !zq) m1[r] = bxh * m1[r] + add;
        if (xc && zq) n1[r] = bxh * n1[r] + add;
        if (zc[r]) m1[r] = __ldg(c.b_z + z + r) * m1[r] + add;
      }
    sto<R>(f.vx_a, base, off, va_x);
    if (any_z) sto<R>(f.m_dsxz_dz, base, off, m1);
    if (xc && !zq) sto<R>(f.m_dsxx_dx, base, off, m1);
    if (xc && zq) sto<R>(f.m_dsxx_dx, base, off, n1);
  }
  {
    float d1[R], d2[R], d3[R], q2[R], n2[R];
    dpz<R>(s_szz_a, b, g.rdz, d1);
    dpz<R>(s_sxx_a, b, g.rdz, d2);
    dmx<R, BOXZ>(s_sxz_a, b, g.rdx, d3);
    if (xq && zq) {
      ldo<R>(f.m_dsxz_dx, base, off, n2);
#pragma unroll
      for (int r = 0; r < R; ++r) q2[r] = dom[r] ? gdm(f.m_dvz_dx, i + r, ldz, g.rdx) : 0.0f;
    }
    const float4 cxh = __ldg(c.q_xh + x);
    const float bx = xc ? __ldg(c.b_x + x) : 0.0f;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (dom[r]) {
        float t = 0.0f;
        const float4 cz = __ldg(c.q_z + z + r);
        if (zq && cz.y != 0.0f) t += cz.y * p2[r];
        if (xq && cxh.y != 0.0f) t += cxh.y * (zq ? q2[r] : p2[r]);
        va_z[r] -= (over(l2m[r] * d1[r] + lam[r] * d2[r], cz.x, cz.w) + over(amu[r] * d3[r], cxh.x, cxh.w)) * dt + t;
        const float add = bA[r] * va_z[r] * dt;
        if (xc && !zq) m2[r] = bx * m2[r] + add;
        if (xc && zq) n2[r] = bx * n2[r] + add;
        if (zc[r]) m2[r] = __ldg(c.b_zh + z + r) * m2[r] + add;
      }
    sto<R>(f.vz_a, base, off, va_z);
    if (any_z) sto<R>(f.m_dszz_dz, base, off, m2);
    if (xc && !zq) sto<R>(f.m_dsxz_dx, base, off, m2);
    if (xc && zq) sto<R>(f.m_dsxz_dx, base, off, n2);
  }
}

// C: res_injection (utilities.cu:569-580) + el_stress_adj (el_stress_adj.cu:53-97)
//    + source_grad (utilities.cu:582-593) + el_velocity(isFor=false) with the
//    sums of the density kernel (el_velocity.cu:84-117) + to_bnd(velocity).
//    Staged: vz_a, vx_a, szz, sxx, sxz.
template <int TX, int K, int R>
__device__ __forceinline__ void bwd_C_edge(const SweepPack<K>& P, int shot, int z0, int x0, int j, unsigned* err) {
  constexpr int BOXZ = 32 * R + 8;
  SWEEP_EDGE(BOXZ, R)
  const Grads& gr = S.gr;
  const int rev = S.nSteps - 2 - j >= 1;
  float p_bA[R], p_bB[R], p_amu[R], p_lam[R], p_l2m[R], p_sa[R], p_xa[R], p_za[R], p_vz[R], p_vx[R];
  ldrows<R>(m.bycA + i, rows_in, p_bA);
  ldrows<R>(m.bycB + i, rows_in, p_bB);
  ldrows<R>(m.aveMu + i, rows_in, p_amu);
  ldrows<R>(m.lam + i, rows_in, p_lam);
  ldrows<R>(m.l2m + i, rows_in, p_l2m);
  pdl_wait();
  SWEEP_TMA(5, BOXZ)
  ldrows<R>(f.szz_a + i, rows_in, p_sa);
  ldrows<R>(f.sxx_a + i, rows_in, p_xa);
  ldrows<R>(f.sxz_a + i, rows_in, p_za);
  ldrows<R>(f.vz + i, rev ? rows_in : 0, p_vz);
  ldrows<R>(f.vx + i, rev ? rows_in : 0, p_vx);
  if (!live) return;
  const StoreD& st = S.st;
  const bool rec_tile = tile_meets_shot_box(sh, z0, x0, 32 * R, TX);
  // Backward iteration j handles res_injection + el_stress_adj of step
  // it = nSteps - 2 - j (j = -1: the shot's last step) and the reverse
  // velocity of step it - 1.
  const int it = S.nSteps - 2 - j;
  const float dt = g.dt;
  if (!stage_wait(&bar, err)) return;
  const float* s_vz_a = sm;
  const float* s_vx_a = sm + N;
  const float* s_szz = sm + 2 * N;
  const float* s_sxx = sm + 3 * N;
  const float* s_sxz = sm + 4 * N;
  auto cell = [&](const int r, const int z, const size_t i, const int b) {
  float sa = p_sa[r], xa = p_xa[r], za = p_za[r];
  const float bA = p_bA[r], bB = p_bB[r], amu = p_amu[r], lam = p_lam[r], l2m = p_l2m[r];
  float vz = p_vz[r], vx = p_vx[r];
  const bool dom = in_box(z, x, g.zs0, g.zs1, g.xs0, g.xs1);
  const int rec = rec_tile ? first_receiver(sh, z, x) : -1;
  inject_res(sh, it, rec, z, x, sa, xa);
  if (dom) {
    {
      const float dvz_dx = -sdp(s_vz_a, b, BOXZ, g.rdx);
      const float dvx_dz = -sdp(s_vx_a, b, 1, g.rdz);
      const float4 cx = __ldg(c.q_x + x), cz = __ldg(c.q_z + z);
      float t = over(dvz_dx, cx.x, cx.w) * bA * dt + over(dvx_dz, cz.x, cz.w) * bB * dt;
      if (cx.y != 0.0f) t += cx.y * (-gdp(f.m_dsxz_dx, i, ldz, g.rdx));
      if (cz.y != 0.0f) t += cz.y * (-gdp(f.m_dsxz_dz, i, 1, g.rdz));
      za += t;
      f.sxz_a[i] = za;
    }
    const bool xb = (x <= g.xband_lo) || (x >= g.xband_hi);
    const bool zb = (z <= g.zband_lo) || (z >= g.zband_hi);
    if (xb) f.m_dvz_dx[i] = c.b_xh[x] * f.m_dvz_dx[i] + za * amu * dt;
    if (zb) f.m_dvx_dz[i] = c.b_zh[z] * f.m_dvx_dz[i] + za * amu * dt;
    {
      const float dvx_dx = -sdm(s_vx_a, b, BOXZ, g.rdx);
      const float dvz_dz = -sdm(s_vz_a, b, 1, g.rdz);
      const float4 cxh = __ldg(c.q_xh + x), czh = __ldg(c.q_zh + z);
      float tx = over(bB * dvx_dx, cxh.x, cxh.w) * dt;
      float tz = over(bA * dvz_dz, czh.x, czh.w) * dt;
      if (cxh.y != 0.0f) tx += cxh.y * (-gdm(f.m_dsxx_dx, i, ldz, g.rdx));
      if (czh.y != 0.0f) tz += czh.y * (-gdm(f.m_dszz_dz, i, 1, g.rdz));
      xa += tx;
      sa += tz;
    }
    if (xb) f.m_dvx_dx[i] = c.b_x[x] * f.m_dvx_dx[i] + lam * sa * dt + l2m * xa * dt;
    if (zb) f.m_dvz_dz[i] = c.b_z[z] * f.m_dvz_dz[i] + l2m * sa * dt + lam * xa * dt;
  }
  if (dom || rec >= 0) {
    f.szz_a[i] = sa;
    f.sxx_a[i] = xa;
  }
  if (!rev) return;
  if (z == sh.src_z && x == sh.src_x) sh.gstf[it - 1] = -(sa + 3.0f * xa) * dt;
  const bool interior = in_box(z, x, g.zi0, g.zi1, g.xi0, g.xi1);
  const int k = ring_index(g, z, x);
  if (interior) {
    const float ea = sdp(s_szz, b, 1, g.rdz) + sdm(s_sxz, b, BOXZ, g.rdx);  // dszz_dz + dsxz_dx
    const float eb = sdm(s_sxz, b, 1, g.rdz) + sdp(s_sxx, b, BOXZ, g.rdx);  // dsxz_dz + dsxx_dx
    vz -= ea * bA * dt;
    vx -= eb * bB * dt;
    gr.va[i] += s_vz_a[b] * ea;
    gr.vb[i] += s_vx_a[b] * eb;
  }
  if (k >= 0) {
    const float* p = st.base + static_cast<size_t>(it - 1) * 5 * g.ring_len + k;
    vz = p[3 * g.ring_len];
    vx = p[4 * g.ring_len];
  }
  if (interior || k >= 0) {
    f.vz[i] = vz;
    f.vx[i] = vx;
  }
  };
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (z + r < g.nz) cell(r, z + r, i + r, b + r);
}

// C of an outer tile (bwd_B_outer): of the forward fields only the ring's
// velocities of step it - 1 are restored; only the adjoint velocities are staged.
template <int TX, int K, int R, bool WIDE>
__device__ __forceinline__ void bwd_C_outer(const SweepPack<K>& P, int shot, int z0, int x0, int j, unsigned* err) {
  constexpr int BOXZ = 32 * R + 8;
  SWEEP_EDGE(BOXZ, R)
  SWEEP_EDGE_CELLS(R, WIDE)
  (void)sh;
  (void)zc;
  (void)any_z;
  const bool xq = any_dom && (x <= g.xband_lo || x >= g.xband_hi);
  const bool zq = any_dom && (z <= g.zband_lo || z + R - 1 >= g.zband_hi);
  float bA[R], bB[R], lam[R], l2m[R], amu[R], sa[R], xa[R], za[R], p1[R], p2[R], m1[R], m2[R];
  if (any_dom) {
    ldo<R>(m.bycA, base, off, bA);
    ldo<R>(m.bycB, base, off, bB);
    ldo<R>(m.aveMu, base, off, amu);
    ldo<R>(m.lam, base, off, lam);
    ldo<R>(m.l2m, base, off, l2m);
  }
  pdl_wait();
  stage_issue<2, TX, BOXZ>(P.maps[shot], sm, &bar, z0, x0);
  if (!live) return;
  if (zq) {
    psi_z<R>(f.m_dszz_dz, f.m_dsxz_dz, dom, i, g.rdz, p1, p2);
    ldo<R>(f.m_dvz_dz, base, off, m1);
    ldo<R>(f.m_dvx_dz, base, off, m2);
  } else if (xq) {
    psi_x<R>(f.m_dsxz_dx, f.m_dsxx_dx, dom, i, ldz, g.rdx, p2, p1);
    ldo<R>(f.m_dvx_dx, base, off, m1);
    ldo<R>(f.m_dvz_dx, base, off, m2);
  }
  if (any_dom) {
    ldo<R>(f.szz_a, base, off, sa);
    ldo<R>(f.sxx_a, base, off, xa);
    ldo<R>(f.sxz_a, base, off, za);
  }
  const int it = S.nSteps - 2 - j;
  if (it >= 1) {
    const float* ring = S.st.base + static_cast<size_t>(it - 1) * 5 * g.ring_len + 3 * g.ring_len;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = ring_index(g, z + r, x);
      if (k >= 0) {
        const float v1 = ring[k], v2 = ring[k + g.ring_len];
        f.vz[i + r] = v1;
        f.vx[i + r] = v2;
      }
    }
  }
  if (!stage_wait(&bar, err) || !any_dom) return;
  const float* s_vz_a = sm;
  const float* s_vx_a = sm + N;
  const float dt = g.dt;
  {  // shear stress: psi terms p2 (along z, else x), memory values m2
    float d1[R], d2[R], q[R], n[R];
    dpx<R, BOXZ>(s_vz_a, b, g.rdx, d1);
    dpz<R>(s_vx_a, b, g.rdz, d2);
    if (xq && zq) {
      ldo<R>(f.m_dvz_dx, base, off, n);
#pragma unroll
      for (int r = 0; r < R; ++r) q[r] = dom[r] ? gdp(f.m_dsxz_dx, i + r, ldz, g.rdx) : 0.0f;
    }
    const float4 cx = __ldg(c.q_x + x);
    const float bxh = __ldg(c.b_xh + x);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (dom[r]) {
        float t = 0.0f;
        const float4 cz = __ldg(c.q_z + z + r);
        if (xq && cx.y != 0.0f) t += cx.y * (zq ? q[r] : p2[r]);
        if (zq && cz.y != 0.0f) t += cz.y * p2[r];
        za[r] -= (over(d1[r], cx.x, cx.w) * bA[r] + over(d2[r], cz.x, cz.w) * bB[r]) * dt + t;
        const float add = za[r] * amu[r] * dt;
        if (xq && !zq) m2[r] = bxh * m2[r] + add;
        if (xq && zq) n[r] = bxh * n[r] + add;
        if (zq && (z + r <= g.zband_lo || z + r >= g.zband_hi)) m2[r] = __ldg(c.b_zh + z + r) * m2[r] + add;
      }
    sto<R>(f.sxz_a, base, off, za);
    if (zq) sto<R>(f.m_dvx_dz, base, off, m2);
    if (xq && !zq) sto<R>(f.m_dvz_dx, base, off, m2);
    if (xq && zq) sto<R>(f.m_dvz_dx, base, off, n);
  }
  {  // normal stresses
    float d3[R], d4[R], q[R], n[R];
    dmx<R, BOXZ>(s_vx_a, b, g.rdx, d3);
    dmz<R>(s_vz_a, b, g.rdz, d4);
    if (xq && zq) {
      ldo<R>(f.m_dvx_dx, base, off, n);
#pragma unroll
      for (int r = 0; r < R; ++r) q[r] = dom[r] ? gdm(f.m_dsxx_dx, i + r, ldz, g.rdx) : 0.0f;
    }
    const float4 cxh = __ldg(c.q_xh + x);
    const float bx = __ldg(c.b_x + x);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (dom[r]) {
        const float4 czh = __ldg(c.q_zh + z + r);
        float tx = over(bB[r] * d3[r], cxh.x, cxh.w) * dt, tz = over(bA[r] * d4[r], czh.x, czh.w) * dt;
        if (xq && cxh.y != 0.0f) tx += cxh.y * (zq ? q[r] : p1[r]);
        if (zq && czh.y != 0.0f) tz += czh.y * p1[r];
        xa[r] -= tx;
        sa[r] -= tz;
        const float ex = (lam[r] * sa[r] + l2m[r] * xa[r]) * dt;
        if (xq && !zq) m1[r] = bx * m1[r] + ex;
        if (xq && zq) n[r] = bx * n[r] + ex;
        if (zq && (z + r <= g.zband_lo || z + r >= g.zband_hi))
          m1[r] = __ldg(c.b_z + z + r) * m1[r] + (l2m[r] * sa[r] + lam[r] * xa[r]) * dt;
      }
    sto<R>(f.szz_a, base, off, sa);
    sto<R>(f.sxx_a, base, off, xa);
    if (zq) sto<R>(f.m_dvz_dz, base, off, m1);
    if (xq && !zq) sto<R>(f.m_dvx_dx, base, off, m1);
    if (xq && zq) sto<R>(f.m_dvx_dx, base, off, n);
  }
}

// ---------------------------------------------------------------------------
// Fast-tile forms of the four sweeps. Every cell of a fast tile is in the
// stencil domain and the reverse-time interior, outside the CPML, the
// adjoint memory bands and the boundary ring, with K = 1 and a = 0: the
// reference's CPML divisions by K are exact there (x / 1 = x) and are left
// out, the memory-array updates and the ring are never reached, and the
// source / receiver terms are evaluated only in tiles that meet the bounding
// box of the shot's receivers and source. Operation order of the fields'
// updates otherwise follows the edge bodies.
// MID: the tile is a mid tile (no CPML cell; it may hold ring cells).
// Own-cell operands and results move as float2 with two depths per thread.

template <int TX, int K, int R, bool MID, bool WIDE>
__device__ __forceinline__ void fwd_stress_fast(const SweepPack<K>& P, int shot, int z0, int x0, int it, int save,
                                                bool inject, unsigned* err) {
  constexpr int TZ = 32 * R, BOXZ = TZ + 8;
  SWEEP_FAST(TZ, BOXZ, R, WIDE)
  const uint64_t pol = media_policy();
  float lam[R], l2m[R], amu[R], szz[R], sxx[R], sxz[R];
  ldm<R>(m.lam, base, off, lam, pol);
  ldm<R>(m.l2m, base, off, l2m, pol);
  ldm<R>(m.aveMu, base, off, amu, pol);
  pdl_wait();
  SWEEP_TMA(2, BOXZ)
  ldo<R>(f.szz, base, off, szz);
  ldo<R>(f.sxx, base, off, sxx);
  ldo<R>(f.sxz, base, off, sxz);
  if (!stage_wait(&bar, err, inject)) return;
  const float* s_vz = sm;
  const float* s_vx = sm + N;
  const float rdz = g.rdz, rdx = g.rdx, dt = g.dt;
  if constexpr (MID) {
    if (save) {
#pragma unroll
      for (int r = 0; r < R; ++r) ring_save(g, S.st, it, z + r, x, szz[r], sxz[r], sxx[r], s_vz[b + r], s_vx[b + r]);
    }
  } else {
    (void)save;
  }
  float dvz_dz[R], dvx_dx[R], dvx_dz[R], dvz_dx[R];
  dmz<R>(s_vz, b, rdz, dvz_dz);
  dmx<R, BOXZ>(s_vx, b, rdx, dvx_dx);
  dpz<R>(s_vx, b, rdz, dvx_dz);
  dpx<R, BOXZ>(s_vz, b, rdx, dvz_dx);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    szz[r] += (l2m[r] * dvz_dz[r] + lam[r] * dvx_dx[r]) * dt;
    sxx[r] += (lam[r] * dvz_dz[r] + l2m[r] * dvx_dx[r]) * dt;
    sxz[r] = sxz[r] + amu[r] * (dvx_dz[r] + dvz_dx[r]) * dt;
  }
  sto<R>(f.sxz, base, off, sxz);
  if (special) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (z + r == sh.src_z && x == sh.src_x) {
        szz[r] += sh.src_szz[it];
        sxx[r] += sh.src_sxx[it];
      }
      record(sh, it, first_receiver(sh, z + r, x), z + r, x, szz[r], sxx[r]);
    }
  }
  sto<R>(f.szz, base, off, szz);
  sto<R>(f.sxx, base, off, sxx);
}

template <int TX, int K, int R, bool WIDE>
__device__ __forceinline__ void fwd_velocity_fast(const SweepPack<K>& P, int shot, int z0, int x0, unsigned* err) {
  constexpr int TZ = 32 * R, BOXZ = TZ + 8;
  SWEEP_FAST(TZ, BOXZ, R, WIDE)
  (void)special;
  (void)z;
  (void)x;
  const uint64_t pol = media_policy();
  float bA[R], bB[R], vz[R], vx[R];
  ldm<R>(m.bycA, base, off, bA, pol);
  ldm<R>(m.bycB, base, off, bB, pol);
  pdl_wait();
  SWEEP_TMA(3, BOXZ)
  ldo<R>(f.vz, base, off, vz);
  ldo<R>(f.vx, base, off, vx);
  if (!stage_wait(&bar, err)) return;
  const float* s_szz = sm;
  const float* s_sxx = sm + N;
  const float* s_sxz = sm + 2 * N;
  const float rdz = g.rdz, rdx = g.rdx, dt = g.dt;
  float dszz_dz[R], dsxz_dx[R], dsxz_dz[R], dsxx_dx[R];
  dpz<R>(s_szz, b, rdz, dszz_dz);
  dmx<R, BOXZ>(s_sxz, b, rdx, dsxz_dx);
  dmz<R>(s_sxz, b, rdz, dsxz_dz);
  dpx<R, BOXZ>(s_sxx, b, rdx, dsxx_dx);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    vz[r] = vz[r] + (dszz_dz[r] + dsxz_dx[r]) * bA[r] * dt;
    vx[r] = vx[r] + (dsxz_dz[r] + dsxx_dx[r]) * bB[r] * dt;
  }
  sto<R>(f.vz, base, off, vz);
  sto<R>(f.vx, base, off, vx);
  if (S.gr.illum) {
    float e[R];
    ldo<R>(S.gr.illum, base, off, e);
#pragma unroll
    for (int r = 0; r < R; ++r) e[r] += vz[r] * vz[r] + vx[r] * vx[r];
    sto<R>(S.gr.illum, base, off, e);
  }
}

// MID: the reverse stress update and the imaging sums only at cells of the
// reverse-time interior, and the ring's stresses of step it restored.
template <int TX, int K, int R, bool MID>
__device__ __forceinline__ void bwd_B_fast(const SweepPack<K>& P, int shot, int z0, int x0, int j, unsigned* err) {
  constexpr int TZ = 32 * R, BOXZ = TZ + 8;
  SWEEP_FAST(TZ, BOXZ, R, true)
  const Grads& gr = S.gr;
  const int it = S.nSteps - 2 - j;
  const uint64_t pol = media_policy();
  float lam[R], l2m[R], amu[R], szz[R], sxx[R], sxz[R], gl[R], gm[R], gt[R], va_z[R], va_x[R];
  ldm<R>(m.lam, base, off, lam, pol);
  ldm<R>(m.l2m, base, off, l2m, pol);
  ldm<R>(m.aveMu, base, off, amu, pol);
  pdl_wait();
  SWEEP_TMA(5, BOXZ)
  ldo<R>(f.szz, base, off, szz);
  ldo<R>(f.sxx, base, off, sxx);
  ldo<R>(f.sxz, base, off, sxz);
  ldo<R>(gr.lam, base, off, gl);
  ldo<R>(gr.mu, base, off, gm);
  ldo<R>(gr.tau, base, off, gt);
  ldo<R>(f.vz_a, base, off, va_z);
  ldo<R>(f.vx_a, base, off, va_x);
  if (!stage_wait(&bar, err)) return;
  const float* s_vz = sm;
  const float* s_vx = sm + N;
  const float* s_szz_a = sm + 2 * N;
  const float* s_sxx_a = sm + 3 * N;
  const float* s_sxz_a = sm + 4 * N;
  const float rdz = g.rdz, rdx = g.rdx, dt = g.dt;
  {
    float dvz_dz[R], dvx_dx[R], e[R], t[R], sa[R], xa[R], za[R];
    dmz<R>(s_vz, b, rdz, dvz_dz);
    dmx<R, BOXZ>(s_vx, b, rdx, dvx_dx);
    dpz<R>(s_vx, b, rdz, e);
    dpx<R, BOXZ>(s_vz, b, rdx, t);
    own<R>(s_szz_a, b, sa);
    own<R>(s_sxx_a, b, xa);
    own<R>(s_sxz_a, b, za);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      e[r] += t[r];  // dvx_dz + dvz_dx
      if (special && z + r == sh.src_z && x == sh.src_x) {
        szz[r] -= sh.src_szz_r[it];
        sxx[r] -= sh.src_sxx_r[it];
      }
      if (!MID || in_box(z + r, x, g.zi0, g.zi1, g.xi0, g.xi1)) {
        szz[r] -= (l2m[r] * dvz_dz[r] + lam[r] * dvx_dx[r]) * dt;
        sxx[r] -= (lam[r] * dvz_dz[r] + l2m[r] * dvx_dx[r]) * dt;
        sxz[r] -= amu[r] * e[r] * dt;
        gl[r] += (sa[r] + xa[r]) * (dvz_dz[r] + dvx_dx[r]);
        gm[r] += sa[r] * dvz_dz[r] + xa[r] * dvx_dx[r];
        gt[r] += za[r] * e[r];
      }
      if constexpr (MID) {  // to_bnd of the stresses (the ring's values replace the update)
        const int q = ring_index(g, z + r, x);
        if (q >= 0) {
          const float* p = S.st.base + static_cast<size_t>(it) * 5 * g.ring_len + q;
          szz[r] = p[0];
          sxz[r] = p[g.ring_len];
          sxx[r] = p[2 * g.ring_len];
        }
      }
    }
  }
  sto<R>(f.szz, base, off, szz);
  sto<R>(f.sxx, base, off, sxx);
  sto<R>(f.sxz, base, off, sxz);
  sto<R>(gr.lam, base, off, gl);
  sto<R>(gr.mu, base, off, gm);
  sto<R>(gr.tau, base, off, gt);
  // el_velocity_adj without the psi memory terms.
  {
    float d1[R], d2[R], d3[R];
    dpx<R, BOXZ>(s_szz_a, b, rdx, d1);
    dpx<R, BOXZ>(s_sxx_a, b, rdx, d2);
    dmz<R>(s_sxz_a, b, rdz, d3);
#pragma unroll
    for (int r = 0; r < R; ++r) va_x[r] -= (lam[r] * d1[r] + l2m[r] * d2[r] + amu[r] * d3[r]) * dt;
    sto<R>(f.vx_a, base, off, va_x);
  }
  {
    float d1[R], d2[R], d3[R];
    dpz<R>(s_szz_a, b, rdz, d1);
    dpz<R>(s_sxx_a, b, rdz, d2);
    dmx<R, BOXZ>(s_sxz_a, b, rdx, d3);
#pragma unroll
    for (int r = 0; r < R; ++r) va_z[r] -= (l2m[r] * d1[r] + lam[r] * d2[r] + amu[r] * d3[r]) * dt;
    sto<R>(f.vz_a, base, off, va_z);
  }
}

// MID: the adjoint memory arrays updated in their bands (el_stress_adj.cu:68-94,
// within 2 cells of the CPML), the reverse velocity update and its imaging
// sums only at cells of the reverse-time interior, and the ring's velocities
// of step it-1 restored.
template <int TX, int K, int R, bool MID, bool WIDE>
__device__ __forceinline__ void bwd_C_fast(const SweepPack<K>& P, int shot, int z0, int x0, int j, unsigned* err) {
  constexpr int TZ = 32 * R, BOXZ = TZ + 8;
  SWEEP_FAST(TZ, BOXZ, R, WIDE)
  const Grads& gr = S.gr;
  const int it = S.nSteps - 2 - j;
  const bool rev = it >= 1;
  const uint64_t pol = media_policy();
  float bA[R], bB[R], sa[R], xa[R], za[R], vz[R], vx[R], ga[R], gb[R];
  ldm<R>(m.bycA, base, off, bA, pol);
  ldm<R>(m.bycB, base, off, bB, pol);
  pdl_wait();
  SWEEP_TMA(5, BOXZ)
  ldo<R>(f.szz_a, base, off, sa);
  ldo<R>(f.sxx_a, base, off, xa);
  ldo<R>(f.sxz_a, base, off, za);
  ldo<R>(f.vz, base, off, vz);
  ldo<R>(f.vx, base, off, vx);
  ldo<R>(gr.va, base, off, ga);
  ldo<R>(gr.vb, base, off, gb);
  if (!stage_wait(&bar, err)) return;
  const float* s_vz_a = sm;
  const float* s_vx_a = sm + N;
  const float* s_szz = sm + 2 * N;
  const float* s_sxx = sm + 3 * N;
  const float* s_sxz = sm + 4 * N;
  const float rdz = g.rdz, rdx = g.rdx, dt = g.dt;
  if (special) {
#pragma unroll
    for (int r = 0; r < R; ++r) inject_res(sh, it, first_receiver(sh, z + r, x), z + r, x, sa[r], xa[r]);
  }
  {
    float d1[R], d2[R], d3[R], d4[R];
    dpx<R, BOXZ>(s_vz_a, b, rdx, d1);
    dpz<R>(s_vx_a, b, rdz, d2);
    dmx<R, BOXZ>(s_vx_a, b, rdx, d3);
    dmz<R>(s_vz_a, b, rdz, d4);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      za[r] -= (d1[r] * bA[r] + d2[r] * bB[r]) * dt;
      xa[r] -= bB[r] * d3[r] * dt;
      sa[r] -= bA[r] * d4[r] * dt;
    }
  }
  if constexpr (MID) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int zr = z + r;
      const bool xb = (x <= g.xband_lo) || (x >= g.xband_hi);
      const bool zb = (zr <= g.zband_lo) || (zr >= g.zband_hi);
      if (xb || zb) {
        const CpmlD& c = S.c;
        const size_t ir = static_cast<size_t>(x) * g.ldz + zr;
        const float amu = m.aveMu[ir], lam = m.lam[ir], l2m = m.l2m[ir];
        if (xb) f.m_dvz_dx[ir] = c.b_xh[x] * f.m_dvz_dx[ir] + za[r] * amu * dt;
        if (zb) f.m_dvx_dz[ir] = c.b_zh[zr] * f.m_dvx_dz[ir] + za[r] * amu * dt;
        if (xb) f.m_dvx_dx[ir] = c.b_x[x] * f.m_dvx_dx[ir] + lam * sa[r] * dt + l2m * xa[r] * dt;
        if (zb) f.m_dvz_dz[ir] = c.b_z[zr] * f.m_dvz_dz[ir] + l2m * sa[r] * dt + lam * xa[r] * dt;
      }
    }
  }
  sto<R>(f.sxz_a, base, off, za);
  sto<R>(f.szz_a, base, off, sa);
  sto<R>(f.sxx_a, base, off, xa);
  if (!rev) return;
  float ea[R], eb[R], t[R], wa[R], wb[R];
  dpz<R>(s_szz, b, rdz, ea);
  dmx<R, BOXZ>(s_sxz, b, rdx, t);
#pragma unroll
  for (int r = 0; r < R; ++r) ea[r] += t[r];  // dszz_dz + dsxz_dx
  dmz<R>(s_sxz, b, rdz, eb);
  dpx<R, BOXZ>(s_sxx, b, rdx, t);
  own<R>(s_vz_a, b, wa);
  own<R>(s_vx_a, b, wb);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    eb[r] += t[r];  // dsxz_dz + dsxx_dx
    if (special && z + r == sh.src_z && x == sh.src_x) sh.gstf[it - 1] = -(sa[r] + 3.0f * xa[r]) * dt;
    if (!MID || in_box(z + r, x, g.zi0, g.zi1, g.xi0, g.xi1)) {
      vz[r] -= ea[r] * bA[r] * dt;
      vx[r] -= eb[r] * bB[r] * dt;
      ga[r] += wa[r] * ea[r];
      gb[r] += wb[r] * eb[r];
    }
    if constexpr (MID) {  // to_bnd of the velocities of step it - 1
      const int q = ring_index(g, z + r, x);
      if (q >= 0) {
        const float* p = S.st.base + static_cast<size_t>(it - 1) * 5 * g.ring_len + q;
        vz[r] = p[3 * g.ring_len];
        vx[r] = p[4 * g.ring_len];
      }
    }
  }
  sto<R>(f.vz, base, off, vz);
  sto<R>(f.vx, base, off, vx);
  sto<R>(gr.va, base, off, ga);
  sto<R>(gr.vb, base, off, gb);
}

// ---------------------------------------------------------------------------
// The sweep kernels: one launch per sweep and time step.

// Forward sweeps: R depths per thread (tiles of 32 R rows), R in {1, 2}
// picked per workload by the autotuner.
// flags: bit 0 saves the boundary ring, bit 1 is the timeout test hook
// (stage_wait's `inject`).
template <int TX, int K, int R, bool WIDE>
__global__ void FWD_BOUNDS k_fwd_stress(const __grid_constant__ SweepPack<K> P, int it, int flags, unsigned* err) {
  SWEEP_KERNEL_TILE(32 * R, 0)
  const bool inject = (flags & 2) != 0;
  if (fast)
    fwd_stress_fast<TX, K, R, false, WIDE>(P, shot, z0, x0, it, 0, inject, err);
  else if (mid)
    fwd_stress_fast<TX, K, R, true, WIDE>(P, shot, z0, x0, it, flags & 1, inject, err);
  else
    fwd_stress_edge<TX, K, R, WIDE>(P, shot, z0, x0, it, flags & 1, inject, err);
}

template <int TX, int K, int R, bool WIDE>
__global__ void FWD_BOUNDS k_fwd_velocity(const __grid_constant__ SweepPack<K> P, unsigned* err) {
  SWEEP_KERNEL_TILE(32 * R, kBackF2)
  // A mid tile of this sweep has nothing beyond the fast form: no CPML cell,
  // every cell in the stencil domain, and no ring or band work.
  if (fast || mid)
    fwd_velocity_fast<TX, K, R, WIDE>(P, shot, z0, x0, err);
  else
    fwd_velocity_edge<TX, K, R, WIDE>(P, shot, z0, x0, err);
}

// Backward sweeps: R depths per thread (tiles of 32 R rows), R in {1, 2};
// NT resident threads per SM (the register budget, BWD_BOUNDS).
template <int TX, int K, int R, int NT>
__global__ void BWD_BOUNDS k_bwd_B(const __grid_constant__ SweepPack<K> P, int j, unsigned* err) {
  SWEEP_KERNEL_TILE(32 * R, 0)
  if (fast)
    bwd_B_fast<TX, K, R, false>(P, shot, z0, x0, j, err);
  else if (mid)
    bwd_B_fast<TX, K, R, true>(P, shot, z0, x0, j, err);
  else if (outer_tile(P.slots[shot], z0, x0, 32 * R, TX))
    bwd_B_outer<TX, K, R>(P, shot, z0, x0, j, err);
  else
    bwd_B_edge<TX, K, R>(P, shot, z0, x0, j, err);
}

template <int TX, int K, int R, int NT, bool WIDE>
__global__ void BWD_BOUNDS k_bwd_C(const __grid_constant__ SweepPack<K> P, int j, unsigned* err) {
  SWEEP_KERNEL_TILE(32 * R, kBackC)
  if (fast)
    bwd_C_fast<TX, K, R, false, WIDE>(P, shot, z0, x0, j, err);
  else if (mid)
    bwd_C_fast<TX, K, R, true, WIDE>(P, shot, z0, x0, j, err);
  else if (outer_tile(P.slots[shot], z0, x0, 32 * R, TX))
    bwd_C_outer<TX, K, R, WIDE>(P, shot, z0, x0, j, err);
  else
    bwd_C_edge<TX, K, R>(P, shot, z0, x0, j, err);
}

// ---------------------------------------------------------------------------
// Model set-up.
constexpr int kT = 32;

// Row-major double [nz][nx] (MPa) -> column-major float (Pa), through a
// shared-memory tile so both sides are coalesced (libCUFD.cu:67-78).
__global__ void k_media_from_rowmajor(int nz, int nx, int ldz, const double* __restrict__ L,
                                      const double* __restrict__ M, const double* __restrict__ D, float* lam,
                                      float* mu, float* den, unsigned* cpmax_bits) {
  __shared__ double tl[kT][kT + 1], tm[kT][kT + 1], td[kT][kT + 1];
  const int x0 = blockIdx.x * kT, z0 = blockIdx.y * kT;
  for (int r = threadIdx.y; r < kT; r += blockDim.y) {
    const int z = z0 + r, x = x0 + threadIdx.x;
    if (z < nz && x < nx) {
      const size_t s = static_cast<size_t>(z) * nx + x;
      tl[r][threadIdx.x] = L[s];
      tm[r][threadIdx.x] = M[s];
      td[r][threadIdx.x] = D[s];
    }
  }
  __syncthreads();
  float cpmax = 0.0f;
  for (int r = threadIdx.y; r < kT; r += blockDim.y) {
    const int x = x0 + r, z = z0 + threadIdx.x;
    if (z < nz && x < nx) {
      const size_t d = static_cast<size_t>(x) * ldz + z;
      const float l = static_cast<float>(tl[threadIdx.x][r] * 1e6);
      const float u = static_cast<float>(tm[threadIdx.x][r] * 1e6);
      const float rho = static_cast<float>(td[threadIdx.x][r]);
      lam[d] = l;
      mu[d] = u;
      den[d] = rho;
      const float cp = static_cast<float>(sqrt((l + 2.0 * u) / rho));  // velInit (utilities.cu:119-121)
      cpmax = fmaxf(cpmax, cp);
    }
  }
  // cp >= 0 (or NaN), so its bit pattern orders like an unsigned integer.
  atomicMax(cpmax_bits, __float_as_uint(cpmax));
}

// The media of a Vp model with Vs = Vp / sqrt(3) and Gardner's density
// rho = 310 Vp^(1/4), formed in double as velocity_to_moduli does
// (src/Utils.jl:221-227): Vp = vp0 (1 - mask) + vp mask within [vmin, vmax] (vp
// itself when vp0 is null), row-major, kept in v. On the host these were a
// dozen passes and two pow per cell, half the time of a gradient call on the
// largest grid: 57 of 284 ms on 1120 x 3152 cells. Bound by the uploads of its
// three inputs, as k_media_from_rowmajor.
__global__ void k_media_from_vp(int nz, int nx, int ldz, const double* __restrict__ vp, const double* __restrict__ vp0,
                                const double* __restrict__ mask, double vmin, double vmax, double* __restrict__ v,
                                float* lam, float* mu, float* den, unsigned* cpmax_bits) {
  __shared__ float tl[kT][kT + 1], tm[kT][kT + 1], td[kT][kT + 1];
  const int x0 = blockIdx.x * kT, z0 = blockIdx.y * kT;
  for (int r = threadIdx.y; r < kT; r += blockDim.y) {
    const int z = z0 + r, x = x0 + threadIdx.x;
    if (z < nz && x < nx) {
      const size_t s = static_cast<size_t>(z) * nx + x;
      double c = vp[s];
      if (vp0) {
        c = __dadd_rn(__dmul_rn(vp0[s], 1.0 - mask[s]), __dmul_rn(c, mask[s]));
        c = c < vmin ? vmin : (c > vmax ? vmax : c);  // (a NaN stays one)
      }
      v[s] = c;
      const double cs = c / 1.7320508075688772, rho = 310.0 * sqrt(sqrt(c));
      const double cs2 = __dmul_rn(cs, cs);
      const double l = __dadd_rn(__dmul_rn(c, c), -2.0 * cs2) * rho / 1e6, u = cs2 * rho / 1e6;
      tl[r][threadIdx.x] = static_cast<float>(l * 1e6);
      tm[r][threadIdx.x] = static_cast<float>(u * 1e6);
      td[r][threadIdx.x] = static_cast<float>(rho);
    }
  }
  __syncthreads();
  float cpmax = 0.0f;
  for (int r = threadIdx.y; r < kT; r += blockDim.y) {
    const int x = x0 + r, z = z0 + threadIdx.x;
    if (z < nz && x < nx) {
      const size_t d = static_cast<size_t>(x) * ldz + z;
      const float l = tl[threadIdx.x][r], u = tm[threadIdx.x][r], rho = td[threadIdx.x][r];
      lam[d] = l;
      mu[d] = u;
      den[d] = rho;
      const float cp = static_cast<float>(sqrt((l + 2.0 * u) / rho));  // velInit (utilities.cu:119-121)
      cpmax = fmaxf(cpmax, cp);
    }
  }
  atomicMax(cpmax_bits, __float_as_uint(cpmax));  // (see k_media_from_rowmajor)
}

// dJ/dVp of that model, row-major: the chain rule of lambda = mu = rho Vp^2 /
// 3e6 MPa and rho = 310 Vp^(1/4) on the column-major gradients, times mask
// (when not null). The host's form took 95 of 284 ms on 1120 x 3152 cells.
__global__ void k_vp_gradient(int nz, int nx, int ldz, const double* __restrict__ v, const double* __restrict__ mask,
                              const float* __restrict__ g_lam, const float* __restrict__ g_mu,
                              const float* __restrict__ g_den, double* __restrict__ out) {
  __shared__ double tm[kT][kT + 1];
  __shared__ float td[kT][kT + 1];
  const int z0 = blockIdx.x * kT, x0 = blockIdx.y * kT;
  for (int r = threadIdx.y; r < kT; r += blockDim.y) {
    const int x = x0 + r, z = z0 + threadIdx.x;
    if (z < nz && x < nx) {
      const size_t i = static_cast<size_t>(x) * ldz + z;
      tm[r][threadIdx.x] = static_cast<double>(g_lam[i]) + static_cast<double>(g_mu[i]);
      td[r][threadIdx.x] = g_den[i];
    }
  }
  __syncthreads();
  for (int r = threadIdx.y; r < kT; r += blockDim.y) {
    const int z = z0 + r, x = x0 + threadIdx.x;
    if (z < nz && x < nx) {
      const size_t i = static_cast<size_t>(z) * nx + x;
      const double c = v[i], q = sqrt(sqrt(c)), rho = 310.0 * q, drho = 77.5 / (q * q * q);
      const double dmod = (drho * c * c + 2.0 * rho * c) / 3e6;
      const double g = tm[threadIdx.x][r] * dmod + static_cast<double>(td[threadIdx.x][r]) * drho;
      out[i] = mask ? g * mask[i] : g;
    }
  }
}

// aveMuInit / aveBycInit (utilities.cu:125-152) plus the terms of the fused
// imaging sweeps.
__global__ void k_media_derived(int nz, int nx, int ldz, const float* __restrict__ lam,
                                const float* __restrict__ mu, const float* __restrict__ den, float* l2m,
                                float* aveMu, float* bycA, float* bycB, float* hs, float* muw) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  if (z >= nz || x >= nx) return;
  const size_t i = static_cast<size_t>(x) * ldz + z;
  const float u = mu[i];
  l2m[i] = lam[i] + 2.0f * u;
  muw[i] = (u != 0.0f) ? static_cast<float>(1.0 / (static_cast<double>(u) * u)) : 0.0f;
  float am = 0.0f, ha = 0.0f, ba = 1.0f / 1000.0f, bb = 1.0f / 1000.0f;
  if (z >= 2 && z <= nz - 3 && x >= 2 && x <= nx - 3) {
    const float a = u, b = mu[i + 1], c = mu[i + ldz], d = mu[i + ldz + 1];
    if (!(a == 0.0f || b == 0.0f || c == 0.0f || d == 0.0f)) {
      const double s = 1.0 / a + 1.0 / b + 1.0 / c + 1.0 / d;
      am = static_cast<float>(4.0 / s);
      ha = static_cast<float>(am / s * 1e6);
    }
    ba = static_cast<float>(2.0 / (den[i + 1] + den[i]));
    bb = static_cast<float>(2.0 / (den[i + ldz] + den[i]));
  }
  aveMu[i] = am;
  hs[i] = ha;
  bycA[i] = ba;
  bycB[i] = bb;
}

// Column-major float -> row-major double (libCUFD.cu:480-486).
__global__ void k_to_rowmajor(int nz, int nx, int ldz, const float* __restrict__ src, double* dst, double scale) {
  __shared__ float t[kT][kT + 1];
  const int z0 = blockIdx.x * kT, x0 = blockIdx.y * kT;
  for (int r = threadIdx.y; r < kT; r += blockDim.y) {
    const int x = x0 + r, z = z0 + threadIdx.x;
    if (z < nz && x < nx) t[r][threadIdx.x] = src[static_cast<size_t>(x) * ldz + z];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < kT; r += blockDim.y) {
    const int z = z0 + r, x = x0 + threadIdx.x;
    if (z < nz && x < nx) dst[static_cast<size_t>(z) * nx + x] = t[threadIdx.x][r] * scale;
  }
}

// ---------------------------------------------------------------------------
// Residual (libCUFD.cu:257-313): taper obs and syn, res = obs - syn with
// sample 0 zeroed (gpuMinus, utilities.cu:154-167), partial sums of res^2 in
// double, then the adjoint taper.
constexpr int kResThreads = 256;
constexpr int kResBlocks = 304;  // 2 x 152 SMs

__global__ void __launch_bounds__(kResThreads)
    k_residual(int nrec, int nSteps, const float* __restrict__ obs, float* syn, float* res,
               const float* __restrict__ taper_o, const float* __restrict__ taper_r, int per_trace,
               double* partials) {
  const size_t n = static_cast<size_t>(nrec) * nSteps;
  double acc = 0.0;
  for (size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; k < n;
       k += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(k % nSteps);
    const float wo = taper_o ? (per_trace ? taper_o[k] : taper_o[t]) : 1.0f;
    const float wr = taper_r ? (per_trace ? taper_r[k] : taper_r[t]) : 1.0f;
    const float s = syn[k] * wo;
    const float o = obs[k] * wo;
    syn[k] = s;
    const float d = (t == 0) ? 0.0f : o - s;
    acc += static_cast<double>(d) * d;
    res[k] = d * wr;
  }
  __shared__ double sh[kResThreads / 32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = (threadIdx.x < kResThreads / 32) ? sh[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) partials[blockIdx.x] = v;
  }
}

// out = in * taper (taper [nrec][nSteps] when per_trace, else [nSteps]); in
// may be out.
__global__ void k_apply_taper(int nrec, int nSteps, const float* in, float* out, const float* __restrict__ taper,
                              int per_trace) {
  const size_t n = static_cast<size_t>(nrec) * nSteps;
  for (size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; k < n;
       k += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[k] = in[k] * (per_trace ? taper[k] : taper[k % nSteps]);
}

// Band-pass of every trace as a circular convolution with the filter's
// impulse response h (length 2 nt, see the engine): y[r][t] =
// sum_{s < nt} x[r][s] h[(t - s) mod 2 nt]. Block: trace blockIdx.y, outputs
// t0 .. t0 + 255; the samples and the 511 taps a chunk of 256 samples needs
// are staged in shared memory. x and y are distinct.
constexpr int kFilt = 256;
__global__ void __launch_bounds__(kFilt) k_trace_filter(int nt, const float* __restrict__ x, float* __restrict__ y,
                                                        const float* __restrict__ h) {
  __shared__ float xs[kFilt];
  __shared__ float hs[2 * kFilt];
  const int r = blockIdx.y, t0 = blockIdx.x * kFilt, tid = threadIdx.x, t = t0 + tid;
  const int n2 = 2 * nt;
  const float* xr = x + static_cast<size_t>(r) * nt;
  float acc = 0.0f;
  for (int s0 = 0; s0 < nt; s0 += kFilt) {
    xs[tid] = (s0 + tid < nt) ? xr[s0 + tid] : 0.0f;
    for (int j = tid; j < 2 * kFilt - 1; j += kFilt) {
      int m = (t0 - s0 - (kFilt - 1) + j) % n2;
      if (m < 0) m += n2;
      hs[j] = h[m];
    }
    __syncthreads();
#pragma unroll 8
    for (int u = 0; u < kFilt; ++u) acc += xs[u] * hs[tid - u + kFilt - 1];
    __syncthreads();
  }
  if (t < nt) y[static_cast<size_t>(r) * nt + t] = acc;
}

// Source-wavelet update (source_update, utilities.cu:927-1035). Traces are
// zero-padded to M = 2 nt and tapered by w2 (cuda_window over M, ratio 0.01;
// only its first nt values meet data); the spectra O_r(f), C_r(f) of observed
// and synthetic traces, f = 0 .. nt, are direct DFTs
//   X(f) = sum_{t < nt} w2[t] x[t] e^{-2 pi i f t / M},
// an FP32 GEMM of the twiddle table (cos, sin)(2 pi k / M), k = f t mod M,
// against the traces. Block: 64 frequencies x 32 traces, samples in chunks of
// 32 staged in shared memory; thread (fg, rg) = (tid & 15, tid >> 4) holds the
// four spectra (O, C; re, im) of frequencies f0 + fg + 16 i (i < 4) for traces
// r0 + rg + 16 j (j < 2). Each block writes its traces' partial sums of
//   num(f) = sum_r conj(C_r) O_r,  den(f) = sum_r |C_r|^2
// to part[(blockIdx.y * 3 + {0: Re num, 1: Im num, 2: den}) * (nt + 1) + f].
constexpr int kSpF = 64, kSpR = 32, kSpT = 32, kSpPad = kSpT + 4;
__global__ void __launch_bounds__(256) k_src_spectra(int nt, int nrec, const float* __restrict__ obs,
                                                     const float* __restrict__ syn, const float* __restrict__ w2,
                                                     const float2* __restrict__ tw, float* __restrict__ part) {
  __shared__ __align__(16) float sc[kSpF][kSpPad];
  __shared__ __align__(16) float ss[kSpF][kSpPad];
  __shared__ __align__(16) float so[kSpR][kSpPad];
  __shared__ __align__(16) float sd[kSpR][kSpPad];
  __shared__ float red[3][16][kSpF];
  const int tid = threadIdx.x, fg = tid & 15, rg = tid >> 4;
  const int f0 = blockIdx.x * kSpF, r0 = blockIdx.y * kSpR;
  const int nf = nt + 1;
  const unsigned M = 2u * static_cast<unsigned>(nt);
  float acc[4][2][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0f;
  for (int t0 = 0; t0 < nt; t0 += kSpT) {
    for (int e = tid; e < kSpF * kSpT; e += 256) {
      const int fl = e / kSpT, tl = e % kSpT, f = f0 + fl, t = t0 + tl;
      float2 v = make_float2(0.0f, 0.0f);
      if (f < nf && t < nt) v = tw[(static_cast<unsigned>(f) * static_cast<unsigned>(t)) % M];
      sc[fl][tl] = v.x;
      ss[fl][tl] = v.y;
    }
    for (int e = tid; e < kSpR * kSpT; e += 256) {
      const int rl = e / kSpT, tl = e % kSpT, r = r0 + rl, t = t0 + tl;
      float o = 0.0f, d = 0.0f;
      if (r < nrec && t < nt) {
        const size_t q = static_cast<size_t>(r) * nt + t;
        const float w = w2[t];
        o = obs[q] * w;
        d = syn[q] * w;
      }
      so[rl][tl] = o;
      sd[rl][tl] = d;
    }
    __syncthreads();
#pragma unroll 2
    for (int tl = 0; tl < kSpT; tl += 4) {
      float4 c[4], sn[4], o[2], d[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        c[i] = *reinterpret_cast<const float4*>(&sc[fg + 16 * i][tl]);
        sn[i] = *reinterpret_cast<const float4*>(&ss[fg + 16 * i][tl]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        o[j] = *reinterpret_cast<const float4*>(&so[rg + 16 * j][tl]);
        d[j] = *reinterpret_cast<const float4*>(&sd[rg + 16 * j][tl]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float* a = acc[i][j];
          a[0] = fmaf(o[j].x, c[i].x, a[0]);
          a[1] = fmaf(-o[j].x, sn[i].x, a[1]);
          a[2] = fmaf(d[j].x, c[i].x, a[2]);
          a[3] = fmaf(-d[j].x, sn[i].x, a[3]);
          a[0] = fmaf(o[j].y, c[i].y, a[0]);
          a[1] = fmaf(-o[j].y, sn[i].y, a[1]);
          a[2] = fmaf(d[j].y, c[i].y, a[2]);
          a[3] = fmaf(-d[j].y, sn[i].y, a[3]);
          a[0] = fmaf(o[j].z, c[i].z, a[0]);
          a[1] = fmaf(-o[j].z, sn[i].z, a[1]);
          a[2] = fmaf(d[j].z, c[i].z, a[2]);
          a[3] = fmaf(-d[j].z, sn[i].z, a[3]);
          a[0] = fmaf(o[j].w, c[i].w, a[0]);
          a[1] = fmaf(-o[j].w, sn[i].w, a[1]);
          a[2] = fmaf(d[j].w, c[i].w, a[2]);
          a[3] = fmaf(-d[j].w, sn[i].w, a[3]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float nre = 0.0f, nim = 0.0f, den = 0.0f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float Or = acc[i][j][0], Oi = acc[i][j][1], Cr = acc[i][j][2], Ci = acc[i][j][3];
      nre += Cr * Or + Ci * Oi;
      nim += Cr * Oi - Ci * Or;
      den += Cr * Cr + Ci * Ci;
    }
    red[0][rg][fg + 16 * i] = nre;
    red[1][rg][fg + 16 * i] = nim;
    red[2][rg][fg + 16 * i] = den;
  }
  __syncthreads();
  if (tid < 3 * kSpF) {
    const int q = tid / kSpF, fl = tid % kSpF, f = f0 + fl;
    float v = 0.0f;
    for (int u = 0; u < 16; ++u) v += red[q][u][fl];
    if (f < nf) part[(static_cast<size_t>(blockIdx.y) * 3 + q) * nf + f] = v;
  }
}

// coef(f) = num(f) / (den(f) + 1e-6) over the trace blocks' partial sums,
// added in block order (cuda_spectrum_update, utilities.cu:768-826).
__global__ void k_src_coef(int nf, int nblk, const float* __restrict__ part, float2* __restrict__ coef) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  float nre = 0.0f, nim = 0.0f, den = 0.0f;
  for (int b = 0; b < nblk; ++b) {
    nre += part[(static_cast<size_t>(b) * 3 + 0) * nf + f];
    nim += part[(static_cast<size_t>(b) * 3 + 1) * nf + f];
    den += part[(static_cast<size_t>(b) * 3 + 2) * nf + f];
  }
  den += 1e-6f;
  coef[f] = make_float2(nre / den, nim / den);
}

// Impulse response of the update, the length-M inverse transform of the
// Hermitian spectrum coef(0 .. nt) divided by M (the C2R + cuda_normalize
// pair): k[n] = (coef_0 + coef_nt (-1)^n + 2 sum_{f=1}^{nt-1} Re(coef_f
// e^{2 pi i f n / M})) / M, accumulated in double. Multiplying a padded
// trace's spectrum by coef and cropping is then y[t] = sum_{m < nt} x[m]
// k[(t - m) mod M] (k_trace_filter).
__global__ void k_src_response(int nt, const float2* __restrict__ coef, const float2* __restrict__ tw,
                               float* __restrict__ kresp) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int M = 2 * nt;
  if (n >= M) return;
  double acc = static_cast<double>(coef[0].x) + static_cast<double>(coef[nt].x) * ((n & 1) ? -1.0 : 1.0);
  int k = 0;
  for (int f = 1; f < nt; ++f) {
    k += n;
    if (k >= M) k -= M;
    const float2 c = coef[f], w = tw[k];
    acc += 2.0 * (static_cast<double>(c.x) * w.x - static_cast<double>(c.y) * w.y);
  }
  kresp[n] = static_cast<float>(acc / M);
}

// The updated wavelet's source terms for the reverse reconstruction, as the
// add_source arithmetic forms them (utilities.cu:528-555): 1500^2 amp dt in
// float, and 3 * 1500^2 * amp * dt in double rounded once.
__global__ void k_src_terms(int nt, float dt, const float* __restrict__ amp, float* __restrict__ szz,
                            float* __restrict__ sxx) {
  const int it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= nt) return;
  const float scale = 2250000.0f;
  const float a = amp[it];
  szz[it] = __fmul_rn(__fmul_rn(scale, a), dt);
  sxx[it] = static_cast<float>(__dmul_rn(__dmul_rn(__dmul_rn(3.0, static_cast<double>(scale)), static_cast<double>(a)),
                                         static_cast<double>(dt)));
}

// Adds the per-shot gradients and / or illuminations of a shot group into
// the global ones, in group order (deterministic): shot k's sub-grid column j
// is global padded column x_off[k] + j. The gradients come out of the sweeps'
// sums over time through the imaging chain rules: lambda and mu directly, mu
// through the 2x2 harmonic averages whose top-left corner is (z, x), (z-1, x),
// (z, x-1), (z-1, x-1) (hs = aveMu / sum(1/mu) 1e6, muw = 1 / mu^2), with the
// guards of el_stress.cu:118-123 (the x guard of :120 is always true), and rho
// through the buoyancies of (z, x), (z-1, x) and (z, x-1)
// (el_velocity.cu:101-110; the x guard of :109 is always true). The sums are
// zero outside a shot's reverse-time interior.
__global__ void k_reduce_grads(int nz, int nx, int ldz, int nshots, const ShotSlot* __restrict__ slots, float* g_lam,
                               float* g_mu, float* g_den, float* g_illum) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  if (z >= nz || x >= nx) return;
  const size_t i = static_cast<size_t>(x) * ldz + z;
  if (g_lam) {
    float a = g_lam[i], b = g_mu[i], c = g_den[i];
    for (int k = 0; k < nshots; ++k) {
      const ShotSlot& S = slots[k];
      const Geo& g = S.g;
      const int xs = x - S.x_off;
      if (!in_box(z, xs, g.zi0, g.zi1, g.xi0, g.xi1 + 1)) continue;
      const size_t j = static_cast<size_t>(xs) * ldz + z, l = j - ldz;
      const float* __restrict__ hs = S.m.hs;
      const float* __restrict__ tau = S.gr.tau;
      const float dt = g.dt;
      a -= S.gr.lam[j] * dt * kMega;
      auto block = [&](size_t q) { return hs[q] != 0.0f ? hs[q] * tau[q] : 0.0f; };  // hs = 0: fluid, no shear term
      float t = block(l);
      if (xs <= g.xi1) t += block(j) + block(j - 1) + block(l - 1);
      b -= 2.0f * S.gr.mu[j] * dt * kMega + S.m.muw[j] * (t * dt);
      const float bA = S.m.bycA[j], bAu = S.m.bycA[j - 1], bB = S.m.bycB[j], bBl = S.m.bycB[l];
      c += 0.5f * dt *
           (bA * bA * S.gr.va[j] + bB * bB * S.gr.vb[j] + bAu * bAu * S.gr.va[j - 1] + bBl * bBl * S.gr.vb[l]);
    }
    g_lam[i] = a;
    g_mu[i] = b;
    g_den[i] = c;
  }
  if (g_illum) {
    float e = g_illum[i];
    for (int k = 0; k < nshots; ++k) {
      const int xs = x - slots[k].x_off;
      if (xs < 0 || xs >= slots[k].g.nx) continue;
      e += slots[k].gr.illum[static_cast<size_t>(xs) * ldz + z];
    }
    g_illum[i] = e;
  }
}

// Fixed-order sum of the block partials into *acc (one warp).
__global__ void k_sum_partials(const double* __restrict__ partials, int n, double* acc) {
  double v = 0.0;
  for (int k = threadIdx.x; k < n; k += 32) v += partials[k];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (threadIdx.x == 0) *acc += v;
}

}  // namespace

// ---------------------------------------------------------------------------
namespace {

template <int TX, int BOXZ>
constexpr size_t smem_bytes(int na) {
  return static_cast<size_t>(na) * BOXZ * (TX + 4) * sizeof(float);
}
// Sweep F2: na staged arrays and the edge body's four arrays of memory values.
template <int TX, int R>
constexpr size_t smem_f2(int na) {
  return smem_bytes<TX, 32 * R + 8>(na) + 4 * 32 * TX * R * sizeof(float);
}
}  // namespace

#define FWIGB_DISPATCH_TX(tx, ...) \
  switch (tx) {                    \
    case 4: {                      \
      constexpr int TX = 4;        \
      __VA_ARGS__;                 \
      break;                       \
    }                              \
    case 8: {                      \
      constexpr int TX = 8;        \
      __VA_ARGS__;                 \
      break;                       \
    }                              \
    default: {                     \
      constexpr int TX = 16;       \
      __VA_ARGS__;                 \
      break;                       \
    }                              \
  }

// Launches a sweep with programmatic stream serialisation (see
// SWEEP_KERNEL_TILE); inside a stream capture this becomes a programmatic
// dependency edge of the graph.
template <typename... KArgs, typename... Args>
void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

dim3 sweep_grid(int tx, int tz, const SweepGrid& gr, int nshots) {
  const int ntz = (gr.nz - (tz == kTileZFwd ? gr.zoff : 0) + tz - 1) / tz, ntx = (gr.nx + tx - 1) / tx;
  return gr.order & kByTile ? dim3(nshots, ntz, ntx) : dim3(ntz, ntx, nshots);
}

template <int K>
int launch_fwd_stress(cudaStream_t s, int tx, int rows, const SweepPack<K>& p, int nshots, const SweepGrid& gr, int it,
                      int flags, unsigned* err) {
  const int sv = flags & 3;
  if (gr.wide)
    launch_pdl(k_fwd_stress<kWideTx, K, 1, true>, sweep_grid(kWideTx, kTileZ, gr, nshots), dim3(32, kWideTx),
               smem_bytes<kWideTx, kBoxZ>(2), s, p, it, sv, err);
  else if (rows == 2)
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_fwd_stress<TX, K, 2, false>, sweep_grid(TX, kTileZFwd, gr, nshots), dim3(32, TX),
                                     smem_bytes<TX, kBoxZFwd>(2), s, p, it, sv, err))
  else
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_fwd_stress<TX, K, 1, false>, sweep_grid(TX, kTileZ, gr, nshots), dim3(32, TX),
                                     smem_bytes<TX, kBoxZ>(2), s, p, it, sv, err))
  return 1;
}

template <int K>
int launch_fwd_velocity(cudaStream_t s, int tx, int rows, const SweepPack<K>& p, int nshots, const SweepGrid& gr,
                        unsigned* err) {
  if (gr.wide)
    launch_pdl(k_fwd_velocity<kWideTx, K, 1, true>, sweep_grid(kWideTx, kTileZ, gr, nshots), dim3(32, kWideTx),
               smem_f2<kWideTx, 1>(3), s, p, err);
  else if (rows == 2)
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_fwd_velocity<TX, K, 2, false>, sweep_grid(TX, kTileZFwd, gr, nshots), dim3(32, TX),
                                     smem_f2<TX, 2>(3), s, p, err))
  else
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_fwd_velocity<TX, K, 1, false>, sweep_grid(TX, kTileZ, gr, nshots), dim3(32, TX),
                                     smem_f2<TX, 1>(3), s, p, err))
  return 1;
}

template <int K>
int launch_bwd_B(cudaStream_t s, int tx, int rows, int regs, const SweepPack<K>& p, int nshots,
                 const SweepGrid& gr, int j, unsigned* err) {
  if (rows == 2)
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_bwd_B<TX, K, 2, 1024>, sweep_grid(TX, kTileZFwd, gr, nshots), dim3(32, TX),
                                     smem_bytes<TX, kBoxZFwd>(5), s, p, j, err))
  else if (regs > 32)
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_bwd_B<TX, K, 1, 1536>, sweep_grid(TX, kTileZ, gr, nshots), dim3(32, TX),
                                     smem_bytes<TX, kBoxZ>(5), s, p, j, err))
  else
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_bwd_B<TX, K, 1, 2048>, sweep_grid(TX, kTileZ, gr, nshots), dim3(32, TX),
                                     smem_bytes<TX, kBoxZ>(5), s, p, j, err))
  return 1;
}

template <int K>
int launch_bwd_C(cudaStream_t s, int tx, int rows, int regs, const SweepPack<K>& p, int nshots,
                 const SweepGrid& gr, int j, unsigned* err) {
  if (gr.wide)
    launch_pdl(k_bwd_C<kWideTx, K, 1, 2048, true>, sweep_grid(kWideTx, kTileZ, gr, nshots), dim3(32, kWideTx),
               smem_bytes<kWideTx, kBoxZ>(5), s, p, j, err);
  else if (rows == 2)
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_bwd_C<TX, K, 2, 1024, false>, sweep_grid(TX, kTileZFwd, gr, nshots), dim3(32, TX),
                                     smem_bytes<TX, kBoxZFwd>(5), s, p, j, err))
  else if (regs > 32)
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_bwd_C<TX, K, 1, 1536, false>, sweep_grid(TX, kTileZ, gr, nshots), dim3(32, TX),
                                     smem_bytes<TX, kBoxZ>(5), s, p, j, err))
  else
    FWIGB_DISPATCH_TX(tx, launch_pdl(k_bwd_C<TX, K, 1, 2048, false>, sweep_grid(TX, kTileZ, gr, nshots), dim3(32, TX),
                                     smem_bytes<TX, kBoxZ>(5), s, p, j, err))
  return 1;
}

#define FWIGB_INSTANTIATE(K)                                                                                    \
  template int launch_fwd_stress<K>(cudaStream_t, int, int, const SweepPack<K>&, int, const SweepGrid&, int, int,  \
                                    unsigned*);                                                                  \
  template int launch_fwd_velocity<K>(cudaStream_t, int, int, const SweepPack<K>&, int, const SweepGrid&,        \
                                      unsigned*);                                                                \
  template int launch_bwd_B<K>(cudaStream_t, int, int, int, const SweepPack<K>&, int, const SweepGrid&, int,      \
                               unsigned*);                                                                       \
  template int launch_bwd_C<K>(cudaStream_t, int, int, int, const SweepPack<K>&, int, const SweepGrid&, int,      \
                               unsigned*);
FWIGB_INSTANTIATE(1)
FWIGB_INSTANTIATE(kPackShots)
#undef FWIGB_INSTANTIATE

// Tensor maps: one per staged array, a 2-D view (z inner, x outer; row stride
// ldz floats) with the box kBoxZ x (TX + 4), and kBoxZFwd x (TX + 4) for
// the two-row sweeps. cuTensorMapEncodeTiled checks the
// base (16-byte aligned: every array starts a multiple of ldz*nx floats into
// a 256-byte aligned allocation) and the stride (ldz*4, a multiple of 128);
// the x coordinate of every copy, z0 - 4 with z0 a multiple of 32, is a
// multiple of 4 floats.
bool encode_sweep_maps(const Geo& g, const Fields& f, int tx, SweepMaps& out, const char** err) {
  // g is the shot's sub-grid; f its fields.
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
      *err = "cuTensorMapEncodeTiled unavailable";
      return false;
    }
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  if (g.ldz % 32 != 0) {
    *err = "column stride is not a multiple of 32 floats";
    return false;
  }
  auto one = [&](CUtensorMap* m, float* base, int boxz) {
    if (reinterpret_cast<uintptr_t>(base) % 16 != 0) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(g.nz), static_cast<cuuint64_t>(g.nx)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(g.ldz) * sizeof(float)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(boxz), static_cast<cuuint32_t>(tx + 4)};
    const cuuint32_t estr[2] = {1, 1};
    return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  bool ok = true;
  const int F = kBoxZFwd, B = kBoxZ;
  ok = ok && one(&out.f1.t[0], f.vz, B) && one(&out.f1.t[1], f.vx, B);
  ok = ok && one(&out.f2.t[0], f.szz, B) && one(&out.f2.t[1], f.sxx, B) && one(&out.f2.t[2], f.sxz, B);
  ok = ok && one(&out.f1w.t[0], f.vz, F) && one(&out.f1w.t[1], f.vx, F);
  ok = ok && one(&out.f2w.t[0], f.szz, F) && one(&out.f2w.t[1], f.sxx, F) && one(&out.f2w.t[2], f.sxz, F);
  ok = ok && one(&out.b.t[0], f.vz, B) && one(&out.b.t[1], f.vx, B) && one(&out.b.t[2], f.szz_a, B) &&
       one(&out.b.t[3], f.sxx_a, B) && one(&out.b.t[4], f.sxz_a, B);
  ok = ok && one(&out.c.t[0], f.vz_a, B) && one(&out.c.t[1], f.vx_a, B) && one(&out.c.t[2], f.szz, B) &&
       one(&out.c.t[3], f.sxx, B) && one(&out.c.t[4], f.sxz, B);
  ok = ok && one(&out.bw.t[0], f.vz, F) && one(&out.bw.t[1], f.vx, F) && one(&out.bw.t[2], f.szz_a, F) &&
       one(&out.bw.t[3], f.sxx_a, F) && one(&out.bw.t[4], f.sxz_a, F);
  ok = ok && one(&out.cw.t[0], f.vz_a, F) && one(&out.cw.t[1], f.vx_a, F) && one(&out.cw.t[2], f.szz, F) &&
       one(&out.cw.t[3], f.sxx, F) && one(&out.cw.t[4], f.sxz, F);
  if (!ok) *err = "cuTensorMapEncodeTiled rejected a sweep tile";
  return ok;
}

void launch_media_from_rowmajor(cudaStream_t s, int nz, int nx, int ldz, const double* lam_mpa, const double* mu_mpa,
                                const double* den, float* lam, float* mu, float* den_f, unsigned* cpmax_bits) {
  dim3 grid((nx + kT - 1) / kT, (nz + kT - 1) / kT);
  k_media_from_rowmajor<<<grid, dim3(kT, 8), 0, s>>>(nz, nx, ldz, lam_mpa, mu_mpa, den, lam, mu, den_f, cpmax_bits);
}

void launch_media_from_vp(cudaStream_t s, int nz, int nx, int ldz, const double* vp, const double* vp0,
                          const double* mask, double vmin, double vmax, double* v, float* lam, float* mu, float* den,
                          unsigned* cpmax_bits) {
  dim3 grid((nx + kT - 1) / kT, (nz + kT - 1) / kT);
  k_media_from_vp<<<grid, dim3(kT, 8), 0, s>>>(nz, nx, ldz, vp, vp0, mask, vmin, vmax, v, lam, mu, den, cpmax_bits);
}

void launch_vp_gradient(cudaStream_t s, int nz, int nx, int ldz, const double* v, const double* mask,
                        const float* g_lam, const float* g_mu, const float* g_den, double* out) {
  dim3 grid((nz + kT - 1) / kT, (nx + kT - 1) / kT);
  k_vp_gradient<<<grid, dim3(kT, 8), 0, s>>>(nz, nx, ldz, v, mask, g_lam, g_mu, g_den, out);
}

void launch_media_derived(cudaStream_t s, int nz, int nx, int ldz, const float* lam, const float* mu,
                          const float* den, float* l2m, float* aveMu, float* bycA, float* bycB, float* hs,
                          float* muw) {
  dim3 grid((nz + 31) / 32, (nx + 7) / 8);
  k_media_derived<<<grid, dim3(32, 8), 0, s>>>(nz, nx, ldz, lam, mu, den, l2m, aveMu, bycA, bycB, hs, muw);
}

int residual_blocks(int n) {
  int b = (n + kResThreads - 1) / kResThreads;
  return b < kResBlocks ? (b < 1 ? 1 : b) : kResBlocks;
}

void launch_residual(cudaStream_t s, int nrec, int nSteps, const float* obs, float* syn, float* res,
                     const float* taper_o, const float* taper_r, int per_trace, double* partials) {
  const int nb = residual_blocks(nrec * nSteps);
  k_residual<<<nb, kResThreads, 0, s>>>(nrec, nSteps, obs, syn, res, taper_o, taper_r, per_trace, partials);
}

void launch_apply_taper(cudaStream_t s, int nrec, int nSteps, const float* in, float* out, const float* taper,
                        int per_trace) {
  k_apply_taper<<<residual_blocks(nrec * nSteps), kResThreads, 0, s>>>(nrec, nSteps, in, out, taper, per_trace);
}

int src_spectra_blocks(int nrec) { return (nrec + kSpR - 1) / kSpR; }

void launch_src_update_coef(cudaStream_t s, int nrec, int nt, const float* obs, const float* syn, const float* w2,
                            const float2* tw, float* part, float2* coef, float* kresp) {
  const int nf = nt + 1, nblk = src_spectra_blocks(nrec);
  k_src_spectra<<<dim3((nf + kSpF - 1) / kSpF, nblk), 256, 0, s>>>(nt, nrec, obs, syn, w2, tw, part);
  k_src_coef<<<(nf + 255) / 256, 256, 0, s>>>(nf, nblk, part, coef);
  k_src_response<<<(2 * nt + 63) / 64, 64, 0, s>>>(nt, coef, tw, kresp);
}

void launch_src_terms(cudaStream_t s, int nt, float dt, const float* amp, float* szz, float* sxx) {
  k_src_terms<<<(nt + 255) / 256, 256, 0, s>>>(nt, dt, amp, szz, sxx);
}

void launch_trace_filter(cudaStream_t s, int nrec, int nt, const float* x, float* y, const float* h) {
  k_trace_filter<<<dim3((nt + kFilt - 1) / kFilt, nrec), kFilt, 0, s>>>(nt, x, y, h);
}

void launch_sum_partials(cudaStream_t s, const double* partials, int n, double* acc) {
  k_sum_partials<<<1, 32, 0, s>>>(partials, n, acc);
}

void launch_reduce_grads(cudaStream_t s, int nz, int nx, int ldz, int nshots, const ShotSlot* slots, float* g_lam,
                         float* g_mu, float* g_den, float* g_illum) {
  dim3 grid((nz + 31) / 32, (nx + 7) / 8);
  k_reduce_grads<<<grid, dim3(32, 8), 0, s>>>(nz, nx, ldz, nshots, slots, g_lam, g_mu, g_den, g_illum);
}

void launch_to_rowmajor(cudaStream_t s, int nz, int nx, int ldz, const float* src, double* dst, double scale) {
  dim3 grid((nz + kT - 1) / kT, (nx + kT - 1) / kT);
  k_to_rowmajor<<<grid, dim3(kT, 8), 0, s>>>(nz, nx, ldz, src, dst, scale);
}

}  // namespace fwigb
