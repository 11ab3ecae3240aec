// seq_i64.cuh -- the FP64 velocity sums (sphere BVE and plane) with their products and divisions
// on the integer pipes (fp64_int.cuh), bit-identical to the reference's FP64 loops.
//
// The FP64 pipe (2 lanes per clock per SM) bounds these sums: a BVE pair is 13 products, 9
// additions and one division in the reference's association.  Here the ten products of
// coordinates, the division and the three final products run as integers, beside the FP64 pipe,
// which keeps the additions (in the plane also the two final products).  Source records hold the mantissas and exponents taken apart
// once, by the prep kernel; a target's are taken apart once per thread.
//
// A pair whose factors lie outside the exponent ranges below takes the plain FP64 instructions,
// so every input gives what the reference gives: coordinates with 2^-120 <= |x| < 2^61 (or 0), a
// radius (or delta) within 2^+-30, and the strengths' ranges.  Then every product is normal:
// |x_i x_j| >= 2^-240, sums of such products are 0 or >= 2^-292, the denominator is in
// 2^-354 .. 2^189, and with strengths in 2^-540 .. 2^541 (sphere, where the terms are integer
// products too) or 2^-820 .. 2^601 (plane) so are the quotients and terms.  A term with a zero
// strength or factor is +-0, and adding either zero to a sum that started at +0 leaves it as it
// is, so the zeros' signs need no care.
#pragma once

#include "engine.cuh"
#include "fp64_int.cuh"
#include "ops.cuh"

namespace lpm {

constexpr int kI64CoordLo = -120, kI64CoordHi = 60;
constexpr int kI64BveStrength = 540, kI64PlaneStrengthLo = -820, kI64PlaneStrengthHi = 600;
constexpr int kI64ScaleLo = -30, kI64ScaleHi = 29;

// Flags of a record and of a target: the pair in plain FP64 (a coordinate or the strength out of
// range); a strength of zero; a coordinate x, y, z of zero, which has no parts; a factor whose
// mantissa ends in many zeros, so that a product may be a tie.
enum : uint32_t {
  kI64Plain = 1u,
  kI64ZeroQ = 2u,
  kI64ZeroX = 4u,
  kI64ZeroY = 8u,
  kI64ZeroZ = 16u,
  kI64Short = 32u
};
constexpr uint32_t kI64Care = kI64ZeroQ | kI64ZeroX | kI64ZeroY | kI64ZeroZ | kI64Short;

__device__ __forceinline__ uint32_t i64_coord_flags(double v, uint32_t zero) {
  if (f64_is_zero(v)) return zero;
  return (f64_in_range(v, kI64CoordLo, kI64CoordHi) ? 0u : static_cast<uint32_t>(kI64Plain)) |
         (f64_short(v) ? static_cast<uint32_t>(kI64Short) : 0u);
}

__device__ __forceinline__ uint32_t i64_strength_flags(double q, int lo, int hi) {
  return f64_is_zero(q) ? static_cast<uint32_t>(kI64ZeroQ)
                        : (f64_in_range(q, lo, hi) ? 0u : static_cast<uint32_t>(kI64Plain));
}

// A product, zero where `zero` says that a factor is (CARE: it may be zero, or a tie).
template <bool CARE>
__device__ __forceinline__ double i64_mul(const F64Parts& a, const F64Factor& b, bool zero) {
  const double v = mul_rn_int<CARE>(a, b);
  return CARE && zero ? 0.0 : v;
}

// ------------------------------------------------------------------ sphere BVE
// BVESphereVelocity, src/SphereBVESolver.f90:395-420 (ASSOC 0: ((a^2 - xi xj) - yi yj) - zi zj,
// :403-404) and setVelocityFromVorticity, src/SphereBVE.f90:489-531 (ASSOC 1:
// a^2 - ((xi xj + yi yj) + zi zj), :509).
template <int ASSOC>
struct BveI64 {
  static constexpr int kMinLanes = 4;  // i64_lanes
  struct __align__(16) Rec {
    F64Factor x, y, z;
    F64Parts q;  // of -zeta_j A_j: the reference negates the quotient
    int32_t idx;
    uint32_t flags;
    uint32_t pad[2];
  };
  struct Tgt {
    F64Parts x, y, z;
    F64Factor k;  // 4 pi a
    uint32_t flags;
  };
  using Params = BveF64Params;
  static constexpr int NA = 3;
  __device__ static Tgt load(const Params& p, int64_t i) {
    Tgt t;
    const double x = p.x[i], y = p.y[i], z = p.z[i];
    t.flags = i64_coord_flags(x, kI64ZeroX) | i64_coord_flags(y, kI64ZeroY) | i64_coord_flags(z, kI64ZeroZ) |
              (f64_in_range(p.a2, 2 * kI64ScaleLo, 2 * kI64ScaleHi + 1) ? 0u : static_cast<uint32_t>(kI64Plain)) |
              ((__double2loint(p.kden) & 0x7ffff) == 0 ? static_cast<uint32_t>(kI64Short) : 0u);
    t.x = f64_parts(x);
    t.y = f64_parts(y);
    t.z = f64_parts(z);
    t.k = f64_factor(f64_parts(p.kden));
    return t;
  }
  // The three terms of a pair, to be added to u, v, w.  False when they are not what the pair
  // gives: CARE = true (zeros and ties in any product) then leaves it to plain_terms, CARE = false
  // to CARE = true.
  template <bool CARE>
  __device__ static __forceinline__ bool terms(const Params& p, const Tgt& t, const Rec& r, double (&out)[NA]) {
    const uint32_t f = t.flags | r.flags;
    const bool tx = t.flags & kI64ZeroX, ty = t.flags & kI64ZeroY, tz = t.flags & kI64ZeroZ;
    const bool rx = r.flags & kI64ZeroX, ry = r.flags & kI64ZeroY, rz = r.flags & kI64ZeroZ;
    const double m1 = i64_mul<CARE>(t.x, r.x, tx || rx), m2 = i64_mul<CARE>(t.y, r.y, ty || ry),
                 m3 = i64_mul<CARE>(t.z, r.z, tz || rz);
    const double den = ASSOC == 0 ? __dsub_rn(__dsub_rn(__dsub_rn(p.a2, m1), m2), m3)
                                  : __dsub_rn(p.a2, __dadd_rn(__dadd_rn(m1, m2), m3));
    const F64Parts sp = div_parts(r.q, mul_words<CARE>(f64_parts(den), t.k));
    const F64Factor s = f64_factor(sp);
    const double c0 = __dsub_rn(i64_mul<CARE>(t.y, r.z, ty || rz), i64_mul<CARE>(t.z, r.y, tz || ry));
    const double c1 = __dsub_rn(i64_mul<CARE>(t.z, r.x, tz || rx), i64_mul<CARE>(t.x, r.z, tx || rz));
    const double c2 = __dsub_rn(i64_mul<CARE>(t.x, r.y, tx || ry), i64_mul<CARE>(t.y, r.x, ty || rx));
    if (CARE) {
      const double v = r.flags & kI64ZeroQ ? 0.0 : f64_whole(sp);
      out[0] = __dmul_rn(c0, v);
      out[1] = __dmul_rn(c1, v);
      out[2] = __dmul_rn(c2, v);
      return !(f & kI64Plain) && !f64_tiny(den);
    }
    out[0] = mul_rn_int<false>(f64_parts(c0), s);
    out[1] = mul_rn_int<false>(f64_parts(c1), s);
    out[2] = mul_rn_int<false>(f64_parts(c2), s);
    // A low word of zero: a zero, or 32 and more trailing zeros.  With at most 18 in the other
    // factor (the target's flags vouch for 4 pi a) no product is a tie.  The cross product of a
    // mesh's mirror points often has a zero component.
    if (__double2loint(c0) == 0 || __double2loint(c1) == 0 || __double2loint(c2) == 0 || (sp.lo & 0x7ffffu) == 0) {
      const double v = f64_whole(sp);
      out[0] = __dmul_rn(c0, v);
      out[1] = __dmul_rn(c1, v);
      out[2] = __dmul_rn(c2, v);
    }
    return __double2loint(den) != 0;
  }
  // The same in plain FP64, from the particle arrays.
  __device__ static __forceinline__ void plain_terms(const Params& p, const Tgt&, int64_t i, const Rec& r,
                                                     double (&out)[NA]) {
    const int64_t j = r.idx;
    const double tx = p.x[i], ty = p.y[i], tz = p.z[i], sx = p.x[j], sy = p.y[j], sz = p.z[j];
    const double q = -__dmul_rn(p.q[j], p.area[j]);
    const double m1 = __dmul_rn(tx, sx), m2 = __dmul_rn(ty, sy), m3 = __dmul_rn(tz, sz);
    const double den = ASSOC == 0 ? __dsub_rn(__dsub_rn(__dsub_rn(p.a2, m1), m2), m3)
                                  : __dsub_rn(p.a2, __dadd_rn(__dadd_rn(m1, m2), m3));
    const double s = __ddiv_rn(q, __dmul_rn(p.kden, den));
    out[0] = __dmul_rn(__dsub_rn(__dmul_rn(ty, sz), __dmul_rn(tz, sy)), s);
    out[1] = __dmul_rn(__dsub_rn(__dmul_rn(tz, sx), __dmul_rn(tx, sz)), s);
    out[2] = __dmul_rn(__dsub_rn(__dmul_rn(tx, sy), __dmul_rn(ty, sx)), s);
  }
  __device__ static void store(const Params& p, int64_t il, const double (&a)[NA]) {
    p.u[il] = a[0];
    p.v[il] = a[1];
    p.w[il] = a[2];
  }
};

template <int ASSOC>
__global__ void prep_bve_i64_kernel(const double* x, const double* y, const double* z, const double* zeta,
                                    const double* area, const int32_t* idx, int64_t ns,
                                    typename BveI64<ASSOC>::Rec* out) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= ns) return;
  const int32_t j = idx[k];
  typename BveI64<ASSOC>::Rec r;
  const double px = x[j], py = y[j], pz = z[j];
  const double q = -__dmul_rn(zeta[j], area[j]);
  r.flags = i64_coord_flags(px, kI64ZeroX) | i64_coord_flags(py, kI64ZeroY) | i64_coord_flags(pz, kI64ZeroZ) |
            i64_strength_flags(q, -kI64BveStrength, kI64BveStrength);
  r.x = f64_factor(f64_parts(px));
  r.y = f64_factor(f64_parts(py));
  r.z = f64_factor(f64_parts(pz));
  r.q = f64_parts(q);
  r.idx = j;
  r.pad[0] = r.pad[1] = 0u;
  out[k] = r;
}

// ------------------------------------------------------------------ plane
// planarIncompressibleVelocity, src/PlaneIncompressibleSolver.f90:291-308
struct PlaneI64 {
  static constexpr int kMinLanes = 2;  // i64_lanes
  struct __align__(16) Rec {
    double x, y;
    F64Parts q;
    int32_t idx;
    uint32_t flags;
    uint32_t pad[3];
  };
  struct Tgt {
    double x, y;
    F64Factor k;  // 2 pi
    uint32_t flags;
  };
  using Params = PlaneF64Params;
  static constexpr int NA = 2;
  __device__ static Tgt load(const Params& p, int64_t i) {
    Tgt t;
    t.x = p.x[i];
    t.y = p.y[i];
    t.flags = (i64_coord_flags(t.x, 0u) & kI64Plain) | (i64_coord_flags(t.y, 0u) & kI64Plain) |
              (f64_is_zero(p.d2) || f64_in_range(p.d2, 2 * kI64ScaleLo, 2 * kI64ScaleHi + 1)
                   ? 0u
                   : static_cast<uint32_t>(kI64Plain));
    t.k = f64_factor(f64_parts(p.two_pi));
    return t;
  }
  template <bool CARE>
  __device__ static __forceinline__ bool terms(const Params& p, const Tgt& t, const Rec& r, double (&out)[NA]) {
    const double dx = __dsub_rn(t.x, r.x), dy = __dsub_rn(t.y, r.y);
    const F64Parts px = f64_parts(dx), py = f64_parts(dy);
    // particles of a mesh often share a coordinate: these zeros are always handled here
    const double xx = mul_rn_int<CARE>(px, f64_factor(px)), yy = mul_rn_int<CARE>(py, f64_factor(py));
    const double r2 = __dadd_rn(__dadd_rn(f64_tiny(dx) ? 0.0 : xx, f64_tiny(dy) ? 0.0 : yy), p.d2);
    const double s = f64_whole(div_parts(r.q, mul_words<CARE>(f64_parts(r2), t.k)));
    const bool zq = CARE && r.flags & kI64ZeroQ;
    out[0] = zq ? 0.0 : -__dmul_rn(dy, s);
    out[1] = zq ? 0.0 : __dmul_rn(dx, s);
    if (CARE) return !((t.flags | r.flags) & kI64Plain) && !f64_tiny(r2);
    // a square is a tie only for exactly 26 trailing zeros, the product with 2 pi (3 of them)
    // only for 48 or 49 (a zero r2 has more)
    return (__double2loint(dx) & 0x7ffffff) != 0x4000000 && (__double2loint(dy) & 0x7ffffff) != 0x4000000 &&
           (__double2loint(r2) | (__double2hiint(r2) << 16)) != 0;
  }
  __device__ static __forceinline__ void plain_terms(const Params& p, const Tgt& t, int64_t, const Rec& r,
                                                     double (&out)[NA]) {
    const double dx = __dsub_rn(t.x, r.x), dy = __dsub_rn(t.y, r.y);
    const double q = __dmul_rn(p.q[r.idx], p.area[r.idx]);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), p.d2);
    const double s = __ddiv_rn(q, __dmul_rn(p.two_pi, r2));
    out[0] = -__dmul_rn(dy, s);
    out[1] = __dmul_rn(dx, s);
  }
  __device__ static void store(const Params& p, int64_t il, const double (&a)[NA]) {
    p.u[il] = a[0];
    p.v[il] = a[1];
  }
};

__global__ void prep_plane_i64_kernel(const double* x, const double* y, const double* omega, const double* area,
                                      const int32_t* idx, int64_t ns, PlaneI64::Rec* out) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= ns) return;
  const int32_t j = idx[k];
  PlaneI64::Rec r;
  r.x = x[j];
  r.y = y[j];
  const double q = __dmul_rn(omega[j], area[j]);
  r.flags = (i64_coord_flags(r.x, 0u) & kI64Plain) | (i64_coord_flags(r.y, 0u) & kI64Plain) |
            i64_strength_flags(q, kI64PlaneStrengthLo, kI64PlaneStrengthHi);
  r.q = f64_parts(q);
  r.idx = j;
  r.pad[0] = r.pad[1] = r.pad[2] = 0u;
  out[k] = r;
}

// ------------------------------------------------------------------ sweep
// S lanes per target.  Lane k of a target's group evaluates the terms of source j = j0 + k of
// each run of S; the S terms of a run are then added in ascending j, each accumulator component by
// one lane of the group (lane k keeps components k, k + S, ...), with the rounding of the
// sequential loop.  More lanes give a small target set more warps, for S ceil(NA / S) additions
// per pair instead of NA (i64_lanes picks S).
//
// Bound by the FP64 pipe and the integer pipes together (BVE at icos nest 6, S = 4: 10.7 FP64
// instructions a pair, where the plain loop has 31, are 83 % of the pipe at 49 Ginteractions/s; counters at nest
// 4, 27 Ginteractions/s: FP64 47 %, ALU 36 % busy; plane at quad nest 6: FP64 78 %, ALU 33 %); a small set by
// the latency of a pair's chain.  Host calls on GB300,
// Ginteractions/s, against the same loop in FP64 instructions only: BVE icos nest 3, 4, 5, 6
// 3.9, 13.1, 15.6, 15.7 -> 6.5, 27.4, 43.7, 49.1; plane quad nest 4, 5, 6 6.8, 21.0, 27.7 ->
// 10.0, 34.2, 53.6.  Two sources per lane in flight (the same rates) and the final products on
// the FP64 pipe (35 at nest 5) were no better.
template <class Op, int S, int TILE, int THREADS>
__global__ void __launch_bounds__(THREADS) seq_i64_kernel(typename Op::Params p,
                                                          const typename Op::Rec* __restrict__ src, int64_t ns,
                                                          int64_t ib, int64_t nt, int* status) {
  static_assert(32 % S == 0 && TILE % S == 0, "a target's lanes stay in one warp; whole runs per tile");
  using Rec = typename Op::Rec;
  constexpr int NA = Op::NA;
  constexpr int NSLOT = (NA + S - 1) / S;  // components per lane
  __shared__ __align__(128) Rec stage[2][TILE];
  __shared__ __align__(8) uint64_t bars[2];
  const int k = static_cast<int>(threadIdx.x) % S;
  const int lane0 = static_cast<int>(threadIdx.x & 31u) - k;  // the group's first lane in the warp
  const int64_t il = static_cast<int64_t>(blockIdx.x) * (THREADS / S) + threadIdx.x / S;
  const bool valid = il < nt;
  const int64_t i = ib + (valid ? il : nt - 1);
  const typename Op::Tgt t = Op::load(p, i);
  double slot[NSLOT];  // slot m: component k + m S of the target's sum
#pragma unroll
  for (int m = 0; m < NSLOT; ++m) slot[m] = 0.0;
  // The terms of the last run: their additions, a chain of S, wait for the next run's products to
  // run beside.
  double run[S][NSLOT];
#pragma unroll
  for (int q = 0; q < S; ++q)
#pragma unroll
    for (int m = 0; m < NSLOT; ++m) run[q][m] = 0.0;
  auto add_run = [&]() {
#pragma unroll
    for (int q = 0; q < S; ++q)
#pragma unroll
      for (int m = 0; m < NSLOT; ++m) slot[m] = __dadd_rn(slot[m], run[q][m]);
  };
  const int64_t n_tiles = ceil_div(ns, TILE);
  int64_t tile = 0;
  pipe_init(bars);
  uint32_t g = 0;
  staged_sweep<Rec, TILE>(src, 0, n_tiles, stage[0], stage[1], bars, g, status, [&](const Rec* tl) {
    const int64_t j0 = tile * TILE;
    const int cnt = static_cast<int>(ns - j0 < TILE ? ns - j0 : TILE);
    for (int jb = 0; jb < cnt; jb += S) {
      const Rec& r = tl[jb + k < cnt ? jb + k : 0];
      const bool has = jb + k < cnt && r.idx != i;
      double x[NA];
      // the warp's targets or sources ask for care, or a pair turns out to need it
      bool care = __any_sync(0xffffffffu, (t.flags | r.flags) != 0);
      if (!care) {
        add_run();
        const bool ok = Op::template terms<false>(p, t, r, x) || !has;
        care = __any_sync(0xffffffffu, !ok);
      } else {
        add_run();
      }
      if (care) {
        const bool ok = Op::template terms<true>(p, t, r, x);
        if (has && !ok) Op::plain_terms(p, t, i, r, x);
      }
      // a pair left out adds +0, which leaves the sum as it is
#pragma unroll
      for (int c = 0; c < NA; ++c) x[c] = has ? x[c] : 0.0;
#pragma unroll
      for (int q = 0; q < S; ++q) {
        double y[NA];
#pragma unroll
        for (int c = 0; c < NA; ++c) y[c] = __shfl_sync(0xffffffffu, x[c], lane0 + q);
#pragma unroll
        for (int m = 0; m < NSLOT; ++m) {
          run[q][m] = y[m * S];
#pragma unroll
          for (int c = m * S + 1; c < NA && c < (m + 1) * S; ++c) run[q][m] = k == c - m * S ? y[c] : run[q][m];
        }
      }
    }
    ++tile;
  });
  add_run();
  double acc[NA];
#pragma unroll
  for (int c = 0; c < NA; ++c) acc[c] = __shfl_sync(0xffffffffu, slot[c / S], lane0 + c % S);
  if (valid && k == 0) Op::store(p, il, acc);
}

}  // namespace lpm
