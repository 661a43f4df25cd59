// Per-extent dispatch of the pass kernels (host side).
#pragma once

#include <cuda_runtime.h>

#include <atomic>

#include "passes.cuh"

namespace ns3d {

// Extents with compiled plans.
#ifndef NS3D_FOR_EACH_EXTENT
#define NS3D_FOR_EACH_EXTENT(X) \
  X(8) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(384) X(512)
#endif

// Points per thread of power-of-two extents, per pass family.
#ifndef NS3D_PXY
#define NS3D_PXY 16
#endif
#ifndef NS3D_PFX
#define NS3D_PFX 16
#endif

// Points per thread: x/y passes that hold one or two lines per thread, and
// the z / fwd_x passes that hold several fields per thread at once.
constexpr int p_pow2(int n, int p) { return p > n ? n : p; }
constexpr int p_xy(int n) { return n % 3 == 0 ? 12 : p_pow2(n, NS3D_PXY); }
constexpr int p_fx(int n) { return n % 3 == 0 ? 12 : p_pow2(n, NS3D_PFX); }
// The nonlinear term's z pass: 16 points per thread for powers of two (one
// Stockham exchange per 256-point transform instead of two), 12 for multiples
// of 3; the tangent form, six velocities and three products in registers: 4 (6).
#ifndef NS3D_PZST
#define NS3D_PZST 16
#endif
constexpr int p_z(int n) { return n % 3 == 0 ? 12 : p_pow2(n, NS3D_PZST); }
constexpr int p_zuv(int n) { return n % 3 == 0 ? 6 : 4; }
// points per thread of the plain line passes (8 measured slower than 16 at 256^3 and 512^3)
#ifndef NS3D_PLINE
#define NS3D_PLINE 16
#endif
constexpr int p_line(int n) { return n % 3 == 0 ? 12 : p_pow2(n, NS3D_PLINE); }
// points per thread of the plain transforms' z passes (pairs of real lines)
#ifndef NS3D_PZPLAIN
#define NS3D_PZPLAIN 8
#endif
constexpr int p_zplain(int n) { return n % 3 == 0 ? 12 : p_pow2(n, NS3D_PZPLAIN); }
// The autotuner's alternative tile of the pipelined x / y passes: 8 points
// per thread for powers of two from 32, 6 for multiples of 3 from 48 (twice
// the lines per CTA, half the registers and prefetch buffers); 0: none.
constexpr int p_alt(int n) {
  return n % 3 == 0 ? (n >= 48 ? 6 : 0) : (n >= 32 ? 8 : 0);
}
inline bool has_alt_tile(int n) {
  switch (n) {
#define NS3D_CASE(N) \
  case N:            \
    return p_alt(N) > 0;
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return false;
  }
}

// The bulk-copy (TMA) form of inv_y (inv_y_tma_kernel): FP64 lines spread
// over the CTA (y extents from 48).  It is tile 2 of the inv_y family, at p_tma(n) points per
// thread (the default or the alternative points per thread, whichever
// spreads its lines over the CTA; 0: no such form for this extent), and runs
// where the handle built tensor maps for its scratch; the tangent form and
// the FP32 mode run the cp.async form at p_tma(n) points per thread instead.
// NS3D_Y_TMA 0 compiles no bulk-copy form.
#ifndef NS3D_Y_TMA
#define NS3D_Y_TMA 1
#endif
// 1: the TMA form runs persistent CTAs (resident CTAs, groups dealt round
// robin), so each CTA's copy ring runs across many groups; 0: NS3D_SCHED.
#ifndef NS3D_Y_TMA_PERSIST
#define NS3D_Y_TMA_PERSIST 0
#endif
constexpr int p_tma(int n) {
  return NS3D_Y_TMA == 0                              ? 0
         : n / p_xy(n) >= NS3D_SPREAD_T                          ? p_xy(n)
         : (p_alt(n) > 0 && n / p_alt(n) >= NS3D_SPREAD_T) ? p_alt(n)
                                                      : 0;
}

// Lines per CTA of the TMA form of inv_y for extent n, 0 when it has none.
inline int inv_y_tma_lpc_inline(int n) {
  switch (n) {
#define NS3D_CASE(N) \
  case N:            \
    return p_tma(N) > 0 ? LaneMap<N / (p_tma(N) > 0 ? p_tma(N) : 1)>::LPC : 0;
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return 0;
  }
}

inline bool extent_supported_inline(int n) {
  switch (n) {
#define NS3D_CASE(N) case N:
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    return true;
    default:
      return false;
  }
}

template <int N, int P>
constexpr int lines_per_cta_xy() {
  return LaneMap<N / P>::LPC;
}
template <int N, int P>
constexpr int lines_per_cta_z() {
  return ZLaneMap<N / P>::LPC;
}

inline unsigned blocks_for(long long lines, int lpc) { return (unsigned)((lines + lpc - 1) / lpc); }

constexpr long long kSms = 148;  // of a B200: the unit of the rules on group counts below

// Persistent grid for a pipelined pass: set the dynamic shared-memory
// attribute and query the resident CTAs per SM once per kernel instantiation
// (Tag) and device; grid = min(groups, SMs x resident CTAs).
template <int KIND, int N, int P, int X>
struct KTag {};

// Passes that run resident CTAs, the groups of lines dealt round robin, so that
// a CTA reads its twiddles once and its copy pipeline runs on from group to
// group: the FP32 lines and the plain transforms' passes, whose groups are
// short (FP32) or a single unit (plain).  FP64 lines keep one CTA per group:
// their neighbouring groups then run side by side.  Per launch on a B200 at
// 256^3, one CTA per group / resident CTAs: FP32 inv_x 134 / 125 us, inv_y 149 /
// 141, fwd_y 102 / 95, fwd_x 278 / 260; FP64 170 / 175, 265 / 268, 150 / 165,
// 248 / 249; a plain R2C and C2R 359 / 297 us.  FP32 lines of 512 points, four
// to a CTA, lose: inv_x 1.39 / 1.52 ms, fwd_x 2.76 / 3.16.
template <typename C, int N>
constexpr bool cap_grid() { return NS3D_SCHED != 0 || (sizeof(C) == 8 && N < 512); }

// The caches are atomics: host threads that launch on the same device may
// race to fill them, and each writes the same values.
// kCap: cap the grid at the resident CTAs whatever NS3D_SCHED says (kernels
// whose CTAs keep a copy pipeline running across their groups).
template <typename Tag, bool kCap = (NS3D_SCHED != 0), typename Kern>
inline unsigned persistent_grid(Kern kern, size_t smem, long long groups) {
  static std::atomic<int> per_sm[64] = {};
  static std::atomic<int> sms[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (per_sm[dev].load(std::memory_order_acquire) == 0) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreads, smem);
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    sms[dev].store(n > 0 ? n : 1, std::memory_order_relaxed);
    per_sm[dev].store(occ > 0 ? occ : 1, std::memory_order_release);
  }
  const long long cap = !kCap ? groups : (long long)sms[dev].load() * per_sm[dev].load();
  return (unsigned)(groups < cap ? (groups > 0 ? groups : 1) : cap);
}

// Whether the inv_x, inv_y and fwd_y passes give each CTA one field instead of
// all of them: where the groups of lines alone leave SMs idle, the chain of
// transforms a CTA runs one after the other is then a third (sixth) as long.
// With more groups than SMs the CTAs' start (twiddles, tables) costs more than
// the shorter chain gives.  The RK3 step on a B200, all fields / one per CTA:
// 32^3 (16 to 18 groups) 144 / 109 us, 64^3 (48 to 66) 149 / 116; 96^3 (192 to
// 294) 350 / 372.
inline bool one_field_per_cta(long long groups) { return groups < kSms; }
// Whether larger grids too run one field per CTA, with one prefetch buffer and
// three CTAs per SM instead of two: then 12 warps per SM hide what 8 with a
// deeper pipeline cannot.  FP64 lines of 12 and 16 points only (the others have
// three CTAs already, or live on L1); lines of 32 threads, four to a CTA, and
// inv_x's plain form from 16 threads a line keep two.  Per launch on a B200, two /
// three CTAs: inv_y 96^3 26.6 / 23.3 us, 128^3 44 / 37, 256^3 265 / 218, 512^3
// 2274 / 2454; inv_x 96^3 22.8 / 22.4, 128^3 36 / 31, 256^3 170 / 178; the tangent
// step (six fields) at 128^3 1205 / 1074.  FP32 lines: inv_x so at four CTAs,
// 128^3 28.7 / 25.1 us, 256^3 127 / 120; their inv_y does not (142 / 155-167).
template <int P, typename C>
constexpr bool dense_ctas(bool wide) { return sizeof(C) == 16 && P > 8 && !wide; }

// KTag's last argument separates the FP64 and FP32 instantiations.
template <typename C>
constexpr int prec_tag() { return sizeof(C) == 16 ? 0 : 100; }

template <int N, int P, int NF, typename C, int V = 0>
cudaError_t launch_inv_x_p(const InvXArgs<NF, C>& a, const PassGeom& g, cudaStream_t st,
                           bool prepare_only) {
  const long long lines = ((long long)g.nlive * nbatch(g)) << g.lw;
  using S = PassSmem<N, P, C, double2, V>;
  const long long groups = (lines + S::LPC - 1) / S::LPC;
  const unsigned grid1 = persistent_grid<KTag<60, N, P, NF + prec_tag<C>() + 1000 * V>, cap_grid<C, N>()>(
      inv_x_kernel<N, P, NF, C, V, 1>, S::BYTES, groups);
  constexpr bool DENSE = sizeof(C) == 8 ? P > 8 && N / P < 32
                                        : dense_ctas<P, C>(NF == 3 && N / P >= 16);
  if constexpr (DENSE) {
    using S1 = PassSmem<N, P, C, double2, V, 1>;
    const unsigned gridd = persistent_grid<KTag<70, N, P, NF + prec_tag<C>() + 1000 * V>, cap_grid<C, N>()>(
        inv_x_kernel<N, P, NF, C, V, 1, 1>, S1::BYTES, groups);
    if (prepare_only) return cudaGetLastError();
    if (!one_field_per_cta(groups)) {
      inv_x_kernel<N, P, NF, C, V, 1, 1><<<dim3(gridd, NF), kThreads, S1::BYTES, st>>>(a, g);
      return cudaGetLastError();
    }
  } else {
    const unsigned grid = persistent_grid<KTag<0, N, P, NF + prec_tag<C>() + 1000 * V>, cap_grid<C, N>()>(
        inv_x_kernel<N, P, NF, C, V>, S::BYTES, groups);
    if (prepare_only) return cudaGetLastError();
    if (!one_field_per_cta(groups)) {
      inv_x_kernel<N, P, NF, C, V><<<grid, kThreads, S::BYTES, st>>>(a, g);
      return cudaGetLastError();
    }
  }
  inv_x_kernel<N, P, NF, C, V, 1><<<dim3(grid1, NF), kThreads, S::BYTES, st>>>(a, g);
  return cudaGetLastError();
}

// The x / y families' tiles 3 and 4: the default and the alternative points
// per thread with the reversed radix schedule, where it differs.
template <int N>
constexpr bool rev_tile_default() {
  return plan_reversible<N, p_xy(N)>();
}
template <int N>
constexpr bool rev_tile_alt() {
  if constexpr (p_alt(N) > 0) {
    return plan_reversible<N, p_alt(N)>();
  } else {
    return false;
  }
}
inline bool rev_tile_exists_inline(int n, int tile) {
  switch (n) {
#define NS3D_CASE(N) \
  case N:            \
    return tile == 3 ? rev_tile_default<N>() : (tile == 4 ? rev_tile_alt<N>() : false);
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return false;
  }
}

// V = 0: tiles 0 and 1; V = 1: tiles 3 and 4 (the reversed schedules)
template <int NF, typename C, int V = 0>
cudaError_t launch_inv_x(const InvXArgs<NF, C>& a, const PassGeom& g, cudaStream_t st,
                         bool prepare_only = false) {
  const int tile = g.tile[kTileInvX];
  switch (g.Nx) {
#define NS3D_CASE(N)                                                                \
  case N:                                                                           \
    if constexpr (V == 0) {                                                         \
      if constexpr (p_alt(N) > 0) {                                                 \
        if (tile == 1) return launch_inv_x_p<N, p_alt(N), NF, C>(a, g, st, prepare_only); \
      }                                                                             \
      return launch_inv_x_p<N, p_xy(N), NF, C>(a, g, st, prepare_only);             \
    } else {                                                                        \
      if constexpr (rev_tile_alt<N>()) {                                            \
        if (tile == 4)                                                              \
          return launch_inv_x_p<N, p_alt(N), NF, C, 1>(a, g, st, prepare_only);     \
      }                                                                             \
      if constexpr (rev_tile_default<N>()) {                                        \
        if (tile == 3)                                                              \
          return launch_inv_x_p<N, p_xy(N), NF, C, 1>(a, g, st, prepare_only);      \
      }                                                                             \
      return cudaErrorInvalidValue;                                                 \
    }
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <int N, int P>
cudaError_t launch_inv_y_tma(const InvYArgs<3, double2>& a, const PassGeom& g, cudaStream_t st,
                             bool prepare_only) {
  using S = InvYTmaSmem<N, P>;
  const long long groups = (long long)g.Nx * ((g.Zp + S::LPC - 1) / S::LPC);
  const unsigned grid = persistent_grid<KTag<90, N, P, 3>, NS3D_Y_TMA_PERSIST != 0>(
      inv_y_tma_kernel<N, P, 3>, S::BYTES, groups);
  if (prepare_only) return cudaGetLastError();
  InvYTmaArgs<3> t;
  t.m = *a.maps;
  for (int f = 0; f < 3; ++f) {
    t.C[f] = a.C[f];
    t.D[f] = a.D[f];
    t.E[f] = a.E[f];
  }
  t.tw = a.tw;
  t.err = a.err;
  inv_y_tma_kernel<N, P, 3><<<grid, kThreads, S::BYTES, st>>>(t, g);
  return cudaGetLastError();
}

template <int N, int P, int NF, typename C, int V = 0>
cudaError_t launch_inv_y_p(const InvYArgs<NF, C>& a, const PassGeom& g, cudaStream_t st,
                           bool prepare_only, bool bulk = false) {
  if constexpr (V == 0 && NF == 3 && sizeof(C) == 16 && P == p_tma(N)) {
    if (bulk && (a.maps || prepare_only)) {
      const cudaError_t e = launch_inv_y_tma<N, P>(a, g, st, prepare_only);
      if (!prepare_only || e != cudaSuccess) return e;
    }
  }
  const long long lines = (long long)g.Nx * g.Zp;
  using S = PassSmem<N, P, C, C, V>;
  const long long groups = (lines + S::LPC - 1) / S::LPC;
  const unsigned grid1 = persistent_grid<KTag<61, N, P, NF + prec_tag<C>() + 1000 * V>, cap_grid<C, N>()>(
      inv_y_kernel<N, P, NF, C, V, 1>, S::BYTES, groups);
  constexpr bool DENSE = dense_ctas<P, C>(N / P >= 32);
  if constexpr (DENSE) {
    using S1 = PassSmem<N, P, C, C, V, 1>;
    const unsigned gridd = persistent_grid<KTag<71, N, P, NF + prec_tag<C>() + 1000 * V>>(
        inv_y_kernel<N, P, NF, C, V, 1, 1>, S1::BYTES, groups);
    if (prepare_only) return cudaGetLastError();
    if (!one_field_per_cta(groups)) {
      inv_y_kernel<N, P, NF, C, V, 1, 1><<<dim3(gridd, NF), kThreads, S1::BYTES, st>>>(a, g);
      return cudaGetLastError();
    }
  } else {
    const unsigned grid = persistent_grid<KTag<1, N, P, NF + prec_tag<C>() + 1000 * V>, cap_grid<C, N>()>(
        inv_y_kernel<N, P, NF, C, V>, S::BYTES, groups);
    if (prepare_only) return cudaGetLastError();
    if (!one_field_per_cta(groups)) {
      inv_y_kernel<N, P, NF, C, V><<<grid, kThreads, S::BYTES, st>>>(a, g);
      return cudaGetLastError();
    }
  }
  inv_y_kernel<N, P, NF, C, V, 1><<<dim3(grid1, NF), kThreads, S::BYTES, st>>>(a, g);
  return cudaGetLastError();
}

template <int NF, typename C, int V = 0>
cudaError_t launch_inv_y(const InvYArgs<NF, C>& a, const PassGeom& gi, cudaStream_t st,
                         bool prepare_only = false) {
  const PassGeom g = planes_geom(gi);
  const int tile = g.tile[kTileInvY];
  switch (g.Ny) {
#define NS3D_CASE(N)                                                                \
  case N:                                                                           \
    if constexpr (V == 0) {                                                         \
      if constexpr (p_tma(N) > 0) {                                                 \
        if (tile == 2)                                                              \
          return launch_inv_y_p<N, p_tma(N), NF, C>(a, g, st, prepare_only, true);  \
      }                                                                             \
      if constexpr (p_alt(N) > 0) {                                                 \
        if (tile == 1) return launch_inv_y_p<N, p_alt(N), NF, C>(a, g, st, prepare_only); \
      }                                                                             \
      return launch_inv_y_p<N, p_xy(N), NF, C>(a, g, st, prepare_only);             \
    } else {                                                                        \
      if constexpr (rev_tile_alt<N>()) {                                            \
        if (tile == 4)                                                              \
          return launch_inv_y_p<N, p_alt(N), NF, C, 1>(a, g, st, prepare_only);     \
      }                                                                             \
      if constexpr (rev_tile_default<N>()) {                                        \
        if (tile == 3)                                                              \
          return launch_inv_y_p<N, p_xy(N), NF, C, 1>(a, g, st, prepare_only);      \
      }                                                                             \
      return cudaErrorInvalidValue;                                                 \
    }
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

// STAGED: as z_kernel (the tangent form stages nothing)
template <typename C, int NF, bool STAGED = true>
cudaError_t launch_z(const ZArgs<NF, C>& a, const PassGeom& gi, cudaStream_t st) {
  const PassGeom g = planes_geom(gi);
  const long long lines = (long long)g.Nx * g.Ny;
  switch (g.Nz) {
#define NS3D_CASE(N)                                                                  \
  case N: {                                                                           \
    constexpr bool UV = NF == 6;                                                      \
    constexpr int P = UV ? p_zuv(N) : p_z(N);                                         \
    if constexpr (UV) {                                                               \
      z_uv_kernel<N, P, C>                                                            \
          <<<blocks_for(lines, lines_per_cta_z<N, P>()), kThreads, 0, st>>>(a, g);    \
    } else {                                                                          \
      constexpr bool ST = STAGED || N <= 64; /* short lines: one form */              \
      using S = ZSmem<N, P, C, ST>;                                                   \
      const unsigned groups = blocks_for(lines, S::LM::LPC);                          \
      const unsigned grid = persistent_grid<KTag<ST ? 40 : 41, N, P, prec_tag<C>()>>( \
          z_kernel<N, P, C, ST>, S::BYTES, groups);                                   \
      z_kernel<N, P, C, ST><<<grid, kThreads, S::BYTES, st>>>(a, g);                  \
    }                                                                                 \
    return cudaGetLastError();                                                        \
  }
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <int N, int P, int MODE, bool COMBINE, typename C>
cudaError_t launch_fwd_x_p(const FwdXArgs<C>& a, const PassGeom& g, cudaStream_t st,
                           bool prepare_only) {
  const long long lines = (long long)g.Ny * g.Mz * nbatch(g);
  using S = PassSmem<N, P, C, C>;
  const unsigned grid =
      persistent_grid<KTag<2 + 2 * MODE + (COMBINE ? 1 : 0), N, P, prec_tag<C>()>, cap_grid<C, N>()>(
          fwd_x_kernel<N, P, MODE, COMBINE, C>, S::BYTES, (lines + S::LPC - 1) / S::LPC);
  if (prepare_only) return cudaGetLastError();
  fwd_x_kernel<N, P, MODE, COMBINE, C><<<grid, kThreads, S::BYTES, st>>>(a, g);
  return cudaGetLastError();
}

// fwd_x with the update operands in the prefetch ring (fwd_x_ring_kernel), at
// 8 points per thread where a line then fills a warp (256) or its wider tile
// would stay inside a warp (to 64), 16 at 128 and 512, whose lines interleaved
// over the CTA read wider rows that way (per plain launch at 512^3: 16 points
// 3.42 ms, 8 points 4.69), 12 for multiples of 3.  The 12-point lines spread
// over the CTA (96, 192) keep fwd_x_kernel: 25.8 against 26.7 us at 96^3 (FP32
// lines 22.5 against 25.8).
#ifndef NS3D_PFXR
#define NS3D_PFXR 8
#endif
constexpr int p_fxr(int n) {
  return n % 3 == 0 ? 12 : (n == 128 || n == 512) ? 16 : p_pow2(n, NS3D_PFXR);
}
constexpr int nslot_fxr(int p) { return p > 12 ? 2 : (p > 8 ? 3 : NS3D_FX_SLOTS); }
constexpr bool fx_use_ring(int n) { return n % 3 != 0 || n / 12 < NS3D_SPREAD_T || n / 12 >= 32; }
// The 16-point ring keeps fwd_x_kernel's results bit for bit, and loses to it
// while an SM has one CTA of it, or not even that: its update then waits for one
// unit after the other with no other CTA's transforms to cover them.  FP64 lines,
// whose fwd_x_kernel is slower, cross over at two thirds of the SMs; the implicit
// update (two divisions a point, and fwd_x_kernel spills) stays with the ring, and
// so does the plain convolution, which has no update.
// The RK3 step on a B200, fwd_x_kernel / ring: 128 x 32 x 64 (66 groups) 120 / 135
// us, FP32 lines 109 / 123; 128 x 64 x 64 (132 groups) 188 / 180, FP32 129 / 141;
// 512 x 8 x 8 (10 groups) 98 / 113.  Implicit step at 128 x 64 x 64 134 / 118 us.
template <typename C>
inline bool fx_few_groups(long long groups) {
  return groups <= (sizeof(C) == 8 ? kSms : 2 * kSms / 3);
}

template <int N, int P, int MODE, bool COMBINE, typename C>
cudaError_t launch_fwd_x_ring(const FwdXArgs<C>& a, const PassGeom& g, cudaStream_t st,
                              bool prepare_only) {
  constexpr int NSLOT = nslot_fxr(P);
  const long long lines = (long long)g.Ny * g.Mz * nbatch(g);
  using S = FxRingSmem<N, P, NSLOT, C>;
  const unsigned grid =
      persistent_grid<KTag<50 + 2 * MODE + (COMBINE ? 1 : 0), N, P, prec_tag<C>()>, cap_grid<C, N>()>(
          fwd_x_ring_kernel<N, P, MODE, COMBINE, NSLOT, C>, S::BYTES,
          (lines + S::LPC - 1) / S::LPC);
  if (prepare_only) return cudaGetLastError();
  fwd_x_ring_kernel<N, P, MODE, COMBINE, NSLOT, C><<<grid, kThreads, S::BYTES, st>>>(a, g);
  return cudaGetLastError();
}

template <int N, int MODE, bool COMBINE, typename C>
cudaError_t launch_fwd_x_n(const FwdXArgs<C>& a, const PassGeom& g, cudaStream_t st,
                           bool prepare_only) {
  if constexpr (!fx_use_ring(N)) {
    return launch_fwd_x_p<N, p_fx(N), MODE, COMBINE, C>(a, g, st, prepare_only);
  } else if constexpr (p_fxr(N) != 16 || MODE == kImplicit || MODE == kConvOut) {
    return launch_fwd_x_ring<N, p_fxr(N), MODE, COMBINE, C>(a, g, st, prepare_only);
  } else {
    static_assert(p_fx(N) == p_fxr(N), "the same transform in both kernels");
    const long long lines = (long long)g.Ny * g.Mz * nbatch(g);
    constexpr int LPC = LaneMap<N / p_fx(N)>::LPC;
    if (prepare_only || !fx_few_groups<C>((lines + LPC - 1) / LPC)) {
      const cudaError_t e =
          launch_fwd_x_ring<N, p_fxr(N), MODE, COMBINE, C>(a, g, st, prepare_only);
      if (!prepare_only || e != cudaSuccess) return e;
    }
    return launch_fwd_x_p<N, p_fx(N), MODE, COMBINE, C>(a, g, st, prepare_only);
  }
}

template <int MODE, bool COMBINE, typename C>
cudaError_t launch_fwd_x(const FwdXArgs<C>& a, const PassGeom& g, cudaStream_t st,
                         bool prepare_only = false) {
  switch (g.Nx) {
#define NS3D_CASE(N)                                                                  \
  case N:                                                                             \
    if constexpr (p_alt(N) > 0) {                                                     \
      if (g.tile[kTileFwdX])                                                          \
        return launch_fwd_x_p<N, p_alt(N), MODE, COMBINE, C>(a, g, st, prepare_only); \
    }                                                                                 \
    return launch_fwd_x_n<N, MODE, COMBINE, C>(a, g, st, prepare_only);
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <int N, int P, typename C, int V = 0>
cudaError_t launch_fwd_y_p(const FwdYArgs<C>& a, const PassGeom& g, cudaStream_t st,
                           bool prepare_only) {
  const long long lines = (long long)g.Nx * g.Mz;
  using S = PassSmem<N, P, C, C, V>;
  const long long groups = (lines + S::LPC - 1) / S::LPC;
  const unsigned grid = persistent_grid<KTag<20, N, P, prec_tag<C>() + 1000 * V>, cap_grid<C, N>()>(
      fwd_y_kernel<N, P, C, V>, S::BYTES, groups);
  const unsigned grid1 = persistent_grid<KTag<62, N, P, prec_tag<C>() + 1000 * V>, cap_grid<C, N>()>(
      fwd_y_kernel<N, P, C, V, 1>, S::BYTES, groups);
  if (prepare_only) return cudaGetLastError();
  if (one_field_per_cta(groups))
    fwd_y_kernel<N, P, C, V, 1><<<dim3(grid1, 3), kThreads, S::BYTES, st>>>(a, g);
  else
    fwd_y_kernel<N, P, C, V><<<grid, kThreads, S::BYTES, st>>>(a, g);
  return cudaGetLastError();
}

template <typename C, int V = 0>
cudaError_t launch_fwd_y(const FwdYArgs<C>& a, const PassGeom& gi, cudaStream_t st,
                         bool prepare_only = false) {
  const PassGeom g = planes_geom(gi);
  const int tile = g.tile[kTileFwdY];
  switch (g.Ny) {
#define NS3D_CASE(N)                                                                \
  case N:                                                                           \
    if constexpr (V == 0) {                                                         \
      if constexpr (p_alt(N) > 0) {                                                 \
        if (tile == 1) return launch_fwd_y_p<N, p_alt(N), C>(a, g, st, prepare_only); \
      }                                                                             \
      return launch_fwd_y_p<N, p_xy(N), C>(a, g, st, prepare_only);                 \
    } else {                                                                        \
      if constexpr (rev_tile_alt<N>()) {                                            \
        if (tile == 4) return launch_fwd_y_p<N, p_alt(N), C, 1>(a, g, st, prepare_only); \
      }                                                                             \
      if constexpr (rev_tile_default<N>()) {                                        \
        if (tile == 3) return launch_fwd_y_p<N, p_xy(N), C, 1>(a, g, st, prepare_only); \
      }                                                                             \
      return cudaErrorInvalidValue;                                                 \
    }
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <int AXIS, int DIR>
cudaError_t launch_line(const LineArgs& a, const PassGeom& g, cudaStream_t st,
                        bool prepare_only = false) {
  const long long lines = AXIS == 0 ? (long long)g.Ny * g.Mz : (long long)g.Nx * g.Mz;
  const PlainGeom pg{g.Nx, g.Ny, g.Mz};
  switch (AXIS == 0 ? g.Nx : g.Ny) {
#define NS3D_CASE(N)                                                                    \
  case N: {                                                                             \
    constexpr int P = p_line(N);                                                           \
    using S = PassSmem<N, P>;                                                           \
    const unsigned grid = persistent_grid<KTag<30 + 2 * AXIS + (DIR > 0 ? 1 : 0), N, P, 0>, true>( \
        line_kernel<N, P, AXIS, DIR>, S::BYTES, (lines + S::LPC - 1) / S::LPC);         \
    if (prepare_only) return cudaGetLastError();                                        \
    line_kernel<N, P, AXIS, DIR><<<grid, kThreads, S::BYTES, st>>>(a, pg);               \
    return cudaGetLastError();                                                          \
  }
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

template <bool C2R>
cudaError_t launch_z_plain(const ZPlainArgs& a, const PassGeom& g, cudaStream_t st) {
  const long long pairs = ((long long)g.Nx * g.Ny) / 2;
  const PlainGeom pg{g.Nx, g.Ny, g.Mz};
  switch (g.Nz) {
#define NS3D_CASE(N)                                                                  \
  case N: {                                                                           \
    constexpr int P = p_zplain(N);                                                    \
    const unsigned grid = blocks_for(pairs, lines_per_cta_z<N, P>());                 \
    if (C2R)                                                                          \
      z_c2r_kernel<N, P><<<grid, kWarpsPerCta * 32, 0, st>>>(a, pg);                  \
    else                                                                              \
      z_r2c_kernel<N, P><<<grid, kWarpsPerCta * 32, 0, st>>>(a, pg);                  \
    return cudaGetLastError();                                                        \
  }
    NS3D_FOR_EACH_EXTENT(NS3D_CASE)
#undef NS3D_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace ns3d
