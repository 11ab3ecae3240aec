// pse64.cuh -- the FP64 PSE sums: every target over the sources within r = 7, each pair in a form
// without square root, arctangent or division.
//
// Every PSE kernel is E(q) (k0 + k1 q + k2 q^2 + k3 q^3) with q = r^2 = (distance / eps)^2 and
// E = exp(-q), so a pair needs q, not r:
//  - chord distances: q = |d|^2 / eps^2;
//  - great-circle distances: q = theta^2 (a / eps)^2, with theta^2 = 4 asin^2(c / 2) a polynomial
//    in the squared chord c^2 of the unit directions (Chebyshev interpolation of the function,
//    within 2^-57 of it; for c up to 0.45, 1.14 and, with the supplement beyond 90 degrees, 2).
//    c^2 comes from the positions: |d|^2 / r^2 for particles as far from the centre as each other to their
//    rounding, (|d|^2 - (r - r')^2) / (r r') for others;
//  - pi and the powers of eps divide the sum once at the end;
//  - E by table and polynomial (P. T. P. Tang, Table-driven implementation of the exponential
//    function, ACM TOMS 15, 1989): with s = 256 q / ln 2 and i = round(s),
//    E = 2^-(i / 256) 2^-((s - i) / 256), a table of 256 powers and a polynomial of degree 4
//    (remainder 4e-17).
// That is about 32 FP64 instructions a pair for K8 of the great-circle distance, where the
// reference's expressions take about 150.  The results agree with the reference's to its own rounding
// (1e-15 of the largest; its exp and atan2 are not CUDA's either): root mean square error against the sums in
// extended precision, as a share of the reference expressions' own, at cubed nest 5: K8 0.58, gradient 0.60,
// divergence 0.87; 0.57, 0.66 and 0.98 for particles 1e-7 off the sphere (pairs of rounded unit directions
// and kernel polynomials in s, with rounded coefficients, gave 1.4 to 3 times the reference's error).
// A lane's sum is in the reference's ascending order; a target has 2 to 8 lanes, each summing its part of
// every tile, and adds the parts at the end.  How many follows from the sources alone, so that a target's bits do not depend on
// which other targets a call has.
//
// At r >= 7 each kernel (its polynomial times e^-49) is below 1e-14 of its peak, and the sum
// leaves those pairs out:
//  - a CTA is one warp of 32 targets (in curve order, so close together).  It lists the source
//    tiles whose ball is within reach of its targets' ball, in ascending order;
//  - each lane tests its own distance to the 64 sources of each listed tile in FP32 (offsets from
//    the tile's centre, so that the test is tight wherever the set lies; the limit is widened by
//    the roundings) and keeps a bit per source;
//  - then each lane walks its own bits through up to 48 tiles, two pairs at a time: the lanes of a
//    warp work on different sources, and take about as many each.  At cubed nest 6 a warp takes
//    1.02 x the mean number of pairs in reach of a target; tile by tile it would take 1.31 x, whole
//    tiles 1.9 x.  Two pairs, because a warp alone waits about 80 clocks for each FP64 result.
// A pair with a particle that has no direction (at the origin of a sphere) or no finite position, or
// whose particles differ by more than a quarter in their distance from the centre, takes the reference's
// expressions as they stand (Op::Plain), as do all pairs of a reach beyond the polynomials' range.
//
// Bound by the FP64 pipe (2 lanes per clock per SM): 74 % busy for K8 and 71 % for the
// gradient at cubed nest 6, the rest being the last warps of an SM.  Host calls on GB300, ms, before (the reference's expressions over whole
// tiles) and after: cubed nest 4 K8 7.1 -> 0.38, gradient 7.5 -> 0.43, double dot 13.5 -> 0.48; nest 6
// K8 37 -> 4.40, Gaussian 12.7 -> 1.64, gradient 40 -> 5.1, divergence 49 -> 6.3, double dot 67 -> 6.8,
// interpolation 37 -> 4.6; quad nest 6 K8 7.3 -> 1.2, gradient 8.4 -> 1.3, second partials 11.5 -> 1.5.
#pragma once

#include "engine.cuh"
#include "ops.cuh"

namespace lpm {

constexpr int kPse64Tile = 64;
constexpr int kPse64Stages = 2;
constexpr int kPse64List = 64;  // tiles listed before they are tested
constexpr int kPse64Mine = 48;  // tiles with sources of its own that a lane holds before they are evaluated
constexpr double kPse64Reach = 7.0;
// A set of up to this many sources (a few tiles) leaves nothing out: particles may then be so far
// apart, against eps, that what lies beyond r = 7 is all there is.
constexpr int64_t kPse64AllPairs = 4 * kPse64Tile;

// How q comes from the squared distance in the test space.
enum { kAngNone = 0, kAngNear = 1, kAngFar = 2, kAngWide = 3 };
constexpr double kAngNearMax = 0.45, kAngFarMax = 1.13, kAngWideMax = 3.15;  // the largest reach (radians)

// (theta / c)^2 as polynomials in c^2.  The first two reach the kernel multiplied by the q of a squared
// angle (Pse64Args::ang).
constexpr int kAngNearN = 9, kAngFarN = 16;
constexpr double kAngleNear[9] = {
    1.0, 0x1.5555555555528p-4, 0x1.6c16c16c21e06p-7, 0x1.d41d41c32ba47p-10,
    0x1.4ce1a15af67f7p-12, 0x1.f85ad3dada806p-15, 0x1.8f6711cda66fbp-17, 0x1.3f8984fdb3592p-19,
    0x1.4ec6f7c8931fap-21};
constexpr double kAngleFar[16] = {
    1.0, 0x1.555555555557dp-4, 0x1.6c16c16c11ab3p-7, 0x1.d41d41d8335acp-10,
    0x1.4ce19a0a71d18p-12, 0x1.f85dcd29033f7p-15, 0x1.8f0a574238fa0p-17, 0x1.46295d746cb2fp-19,
    0x1.0de9a232ae937p-21, 0x1.f9dd6ab3b186cp-24, 0x1.678acc7911957p-27, 0x1.3377469b31787p-26,
    -0x1.0ae9181a54911p-27, 0x1.33d9687615ab8p-28, -0x1.473d3bf6189d6p-30, 0x1.b0132cb15d416p-33};
__device__ constexpr double kAngleWide[21] = {
    1.0, 0x1.5555555555539p-4, 0x1.6c16c16c1ad97p-7, 0x1.d41d41d067cd5p-10,
    0x1.4ce19bc9b7a71p-12, 0x1.f85d52f2033f3p-15, 0x1.8f156d8a2a07fp-17, 0x1.45748f36e7d1bp-19,
    0x1.16520badb72a2p-21, 0x1.63956078e7873p-24, 0x1.2e4682196d94dp-24, -0x1.0a0a04610a73dp-24,
    0x1.46010a5d2b1e0p-24, -0x1.169cae1127812p-24, 0x1.7be9e29dcebbcp-25, -0x1.8c9704395f2ddp-26,
    0x1.3a3073c170e3dp-27, -0x1.6c742eaa3376ap-29, 0x1.2590182d74208p-31, -0x1.2625ff01947f3p-34,
    0x1.187c20d375371p-38};

// ------------------------------------------------------------------ inputs
struct __align__(32) TileBall {
  double x, y, z, r;  // centre and radius in the test space
};

// The source side of a sum: positions, up to three fields, areas.
struct Pse64Src {
  const double *x, *y, *z, *s1, *s2, *s3, *area;
};

struct Pse64Args {
  double c;               // q per squared distance (chord) or squared angle
  double ang[kAngFarN];   // c times the near or the far angle polynomial
  double scale, unscale;  // what divides the kernel's polynomial (pi, powers of eps), and its inverse
  double reach;           // of the cutoff, in the test space
  int unit;               // 1: the test space is unit directions
  int all_plain;          // 1: every pair in the reference's expressions
  const double *x, *y, *z;  // target positions (z may be null)
  Pse64Src src;
  const TileBall* bounds;
  const float4* side;
  const double* powers;   // 2^-(i / 256)
  const int32_t* tperm;   // the targets in curve order, or null: index order
  int64_t ns, n_tiles, ib, nt;
  int* status;
};

constexpr double kPse64PerQ = 369.32993046757463228;  // 256 / ln 2

// The point of particle i in the test space.  A point at the origin of a sphere has no direction
// (and atan2(0, 0) puts it at distance 0 from everything); it becomes NaN, which every test reads
// as "in reach".
struct CutPoint {
  double3 raw, q;  // the position, and the point in the test space
  double r;        // |raw| (test space of unit directions)
};

__device__ __forceinline__ CutPoint cut_point(const double* x, const double* y, const double* z, int64_t i, int unit) {
  CutPoint p;
  p.raw = make_double3(x[i], y[i], z ? z[i] : 0.0);
  p.q = p.raw;
  p.r = 1.0;
  if (unit) {
    // (explicit operations: the targets' and the sources' |p| have to round alike)
    p.r = sqrt(fma(p.raw.x, p.raw.x, fma(p.raw.y, p.raw.y, __dmul_rn(p.raw.z, p.raw.z))));
    const double inv = p.r > 0.0 ? 1.0 / p.r : __longlong_as_double(0x7ff8000000000000LL);
    p.q = make_double3(p.raw.x * inv, p.raw.y * inv, p.raw.z * inv);
  }
  return p;
}

// Whether a point's pairs take the reference's expressions: NaN or infinite in some component of the
// test space, or (unit directions) at a distance whose square would leave the exponent's range.
__device__ __forceinline__ bool odd_point(const CutPoint& p) {
  const double v = (p.q.x - p.q.x) + (p.q.y - p.q.y) + (p.q.z - p.q.z);
  return !(v == 0.0) || !(p.r >= 0x1p-450 && p.r <= 0x1p450);
}

// Whether two particles' distances from the sphere's centre are the same to their rounding (within 8
// units in the last place: turned, scaled and renormalised meshes differ by up to 6, and a pair that is not the same
// takes its warp through the general path); a particle that is odd has one that is no other's.
__device__ __forceinline__ bool same_radius(long long a, double b) {
  return static_cast<unsigned long long>(__double_as_longlong(b)) - static_cast<unsigned long long>(a) + 8ull <= 16ull;
}

// ------------------------------------------------------------------ a pair's kernel value
template <int N>
__device__ __forceinline__ double horner(const double (&c)[N], double v) {
  double p = c[N - 1];
#pragma unroll
  for (int k = N - 2; k >= 0; --k) p = fma(p, v, c[k]);
  return p;
}

// q from the squared distance or squared chord v.
template <int ANG>
__device__ __forceinline__ double pse64_q(const Pse64Args& a, double v) {
  if constexpr (ANG == kAngNear || ANG == kAngFar) {
    constexpr int N = ANG == kAngNear ? kAngNearN : kAngFarN;
    double p = a.ang[N - 1];
#pragma unroll
    for (int k = N - 2; k >= 0; --k) p = fma(p, v, a.ang[k]);
    return __dmul_rn(v, p);
  }
  if (ANG == kAngNone) return __dmul_rn(v, a.c);
  if (v <= 2.0) return __dmul_rn(v * horner(kAngleWide, v), a.c);
  // beyond 90 degrees: the supplement's angle (a kernel that reaches there has eps < 0.45, so
  // that near the antipode, where this loses digits, it is below e^-40)
  const double w = fmax(4.0 - v, 0.0);
  const double t = 3.14159265358979323846 - sqrt(w * horner(kAngleWide, w));
  return __dmul_rn(t * t, a.c);
}

// The kernel (without what divides its polynomial) at q.  The polynomial is in q, where its
// coefficients are exact: in s, their roundings were common to all pairs of a sum, whose moments cancel.
template <class Op>
__device__ __forceinline__ double pse64_kernel_value(double q, const double* powers) {
  const double big = 6755399441055744.0;  // 1.5 x 2^52: the sum's low word is round(s)
  const double t = fma(q, kPse64PerQ, big);
  const int i = __double2loint(t);
  const double f = fma(q, kPse64PerQ, __dsub_rn(big, t));
  double p = 0x1.3b2ab6fba4e77p-39;  // (-ln 2 / 256)^n / n!
  p = fma(p, f, -0x1.c6b08d704a0c0p-29);
  p = fma(p, f, 0x1.ebfbdff82c58fp-19);
  p = fma(p, f, -0x1.62e42fefa39efp-9);
  p = fma(p, f, 1.0);
  const double e = __dmul_rn(powers[i & 255], p);
  const double scaled = __hiloint2double(__double2hiint(e) - ((i >> 8) << 20), __double2loint(e));
  const double w = Op::kPoly ? __dmul_rn(scaled, Op::poly(q)) : scaled;
  // at q >= 707 (0x40861800 00000000, where the kernel is below 1e-300) i leaves the exponent's range
  return __double2hiint(q) >= 0x40861800 ? 0.0 : w;
}

// ------------------------------------------------------------------ operators
// An operator's record holds the position (x, y, z), the fields that its pairs need, the particle's
// index and whether it is odd (odd_point); with great-circle distances also |p| and its inverse (r NaN
// if odd).  add() adds the pair's terms, with d the difference of the positions and w the kernel value.
// The accumulators are Plain's, in units of Pse64Args::scale.
struct Pse64Op {
  static constexpr bool kPoly = true;   // false: a plain Gaussian
  static constexpr bool kUnit = false;  // true: great-circle distances
};
// The kernels over pi as polynomials in q = r^2 (times e^-q).
struct Pse64K8 {  // bivariateLaplacianKernel8
  __device__ static __forceinline__ double poly(double q) {
    return fma(fma(fma(-2.0 / 3.0, q, 10.0), q, -40.0), q, 40.0);
  }
};
struct Pse64K1 {  // bivariateFirstDerivativeKernel8
  __device__ static __forceinline__ double poly(double q) {
    return fma(fma(fma(1.0 / 3.0, q, -5.0), q, 20.0), q, -20.0);
  }
};
struct Pse64Delta8 {  // bivariateDeltaKernel8
  __device__ static __forceinline__ double poly(double q) {
    return fma(fma(fma(-1.0 / 6.0, q, 2.0), q, -6.0), q, 4.0);
  }
};

template <bool UNIT>
struct __align__(16) Pse64ScalarRec {
  double x, y, z, f, area;
  int32_t idx, odd;
};
template <>
struct __align__(16) Pse64ScalarRec<true> {
  double x, y, z, f, area, r, inv;
  int32_t idx, odd;
};

template <int KIND>
struct PseLap64 : Pse64Op, Pse64K8 {
  using Plain = PseF64<KIND>;
  using Params = PseF64Params;
  using Acc = typename Plain::Acc;
  static constexpr int kDim = KIND == kPseK8Chord ? 2 : 3;
  static constexpr bool kPoly = KIND != kPseGaussChord;
  static constexpr bool kUnit = KIND == kPseK8Geodesic;
  using Rec = Pse64ScalarRec<kUnit>;
  struct Tgt {
    double f;
  };
  __device__ static void fill(Rec& r, const Pse64Src& s, int64_t j) {
    r.f = s.s1[j];
    r.area = s.area[j];
  }
  __device__ static Tgt load(const Params& p, int64_t i) { return Tgt{p.f[i]}; }
  __device__ static __forceinline__ void add(const Tgt& t, const Rec& r, double, double, double, double w, Acc& a) {
    a.l = fma((r.f - t.f) * r.area, w, a.l);
  }
  __device__ static Rec64 plain_record(const Pse64Src& s, int64_t j) {
    return Rec64{s.x[j], s.y[j], s.z ? s.z[j] : 0.0, s.s1[j], s.area[j], static_cast<long long>(j)};
  }
};

template <bool SPHERE>
struct PseInterp64 : Pse64Op, Pse64Delta8 {
  static constexpr bool kUnit = SPHERE;
  using Plain = PseInterpF64<SPHERE>;
  using Params = PseExtF64Params;
  using Acc = typename Plain::Acc;
  static constexpr int kDim = 3;
  using Rec = Pse64ScalarRec<SPHERE>;  // f: the product f A
  struct Tgt {};
  __device__ static void fill(Rec& r, const Pse64Src& s, int64_t j) {
    r.f = __dmul_rn(s.s1[j], s.area[j]);
    r.area = 0.0;
  }
  __device__ static Tgt load(const Params&, int64_t) { return Tgt{}; }
  __device__ static __forceinline__ void add(const Tgt&, const Rec& r, double, double, double, double w, Acc& a) {
    a.s = fma(r.f, w, a.s);
  }
  __device__ static Rec64 plain_record(const Pse64Src& s, int64_t j) { return PseLap64<0>::plain_record(s, j); }
};

struct PsePlaneGrad64 : Pse64Op, Pse64K1 {
  using Plain = PsePlaneGradF64;
  using Params = PseExtF64Params;
  using Acc = Plain::Acc;
  static constexpr int kDim = 2;
  using Rec = Pse64ScalarRec<false>;
  struct Tgt {
    double f;
  };
  __device__ static void fill(Rec& r, const Pse64Src& s, int64_t j) {
    r.f = s.s1[j];
    r.area = s.area[j];
  }
  __device__ static Tgt load(const Params& p, int64_t i) { return Tgt{p.s1[i]}; }
  __device__ static __forceinline__ void add(const Tgt& t, const Rec& r, double dx, double dy, double, double w,
                                             Acc& a) {
    const double g = (r.f + t.f) * r.area * w;
    a.gx = fma(g, dx, a.gx);
    a.gy = fma(g, dy, a.gy);
  }
  __device__ static Rec64 plain_record(const Pse64Src& s, int64_t j) { return PseLap64<0>::plain_record(s, j); }
};

template <class Base>  // PsePlaneSecondF64 or PsePlaneDdotF64
struct PlaneD464 : Pse64Op, Pse64K1 {
  using Plain = Base;
  using Params = PseExtF64Params;
  using Acc = typename Base::Acc;
  static constexpr int kDim = 2;
  struct __align__(16) Rec {
    double x, y, z, va, vb, area;
    int32_t idx, odd;
    double pad;
  };
  struct Tgt {
    double a, b;
  };
  __device__ static void fill(Rec& r, const Pse64Src& s, int64_t j) {
    r.va = s.s1[j];
    r.vb = s.s2[j];
    r.area = s.area[j];
    r.pad = 0.0;
  }
  __device__ static Tgt load(const Params& p, int64_t i) { return Tgt{p.s1[i], p.s2[i]}; }
  __device__ static __forceinline__ void add(const Tgt& t, const Rec& r, double dx, double dy, double, double w,
                                             Acc& a) {
    const double g = r.area * w, gx = g * dx, gy = g * dy, sa = r.va + t.a, sb = r.vb + t.b;
    a.ax = fma(sa, gx, a.ax);
    a.ay = fma(sa, gy, a.ay);
    a.bx = fma(sb, gx, a.bx);
    a.by = fma(sb, gy, a.by);
  }
  __device__ static RecVec64 plain_record(const Pse64Src& s, int64_t j) {
    return RecVec64{s.x[j], s.y[j], s.z ? s.z[j] : 0.0, s.s1[j], s.s2[j], s.s3 ? s.s3[j] : 0.0, s.area[j],
                    static_cast<long long>(j)};
  }
};

// The sphere's first-derivative operators.
struct __align__(16) PseVecRec64 {
  double x, y, z, a, b, c, area, r, inv;
  int32_t idx, odd;
};

template <class Base>
struct PseSphereVec64 : Pse64Op, Pse64K1 {
  static constexpr bool kUnit = true;
  using Plain = Base;
  using Acc = typename Base::Acc;
  static constexpr int kDim = 3;
  using Rec = PseVecRec64;
  __device__ static void fill(Rec& r, const Pse64Src& s, int64_t j) {
    r.a = s.s1[j];
    r.b = s.s2 ? s.s2[j] : 0.0;
    r.c = s.s3 ? s.s3[j] : 0.0;
    r.area = s.area[j];
  }
};

struct PseGrad64 : PseSphereVec64<PseGradF64> {
  using Params = PseVecF64Params;
  struct Tgt {
    double f;
  };
  __device__ static Tgt load(const Params& p, int64_t i) { return Tgt{p.f[i]}; }
  __device__ static __forceinline__ void add(const Tgt& t, const Rec& r, double dx, double dy, double dz, double w,
                                             Acc& a) {
    const double g = (r.a + t.f) * r.area * w;
    a.g0 = fma(g, dx, a.g0);
    a.g1 = fma(g, dy, a.g1);
    a.g2 = fma(g, dz, a.g2);
  }
  __device__ static Rec64 plain_record(const Pse64Src& s, int64_t j) { return PseLap64<0>::plain_record(s, j); }
};

struct PseDiv64 : PseSphereVec64<PseDivF64> {
  using Params = PseVecF64Params;
  struct Tgt {
    double x, y, z, vx, vy, vz;
  };
  __device__ static Tgt load(const Params& p, int64_t i) {
    return Tgt{p.x[i], p.y[i], p.z[i], p.vx[i], p.vy[i], p.vz[i]};
  }
  // (P d) . V = d . V - (x . d) (x . V)
  __device__ static __forceinline__ void add(const Tgt& t, const Rec& r, double dx, double dy, double dz, double w,
                                             Acc& a) {
    const double vx = r.a + t.vx, vy = r.b + t.vy, vz = r.c + t.vz;
    const double dv = fma(dx, vx, fma(dy, vy, __dmul_rn(dz, vz)));
    const double xd = fma(t.x, dx, fma(t.y, dy, __dmul_rn(t.z, dz))),
                 xv = fma(t.x, vx, fma(t.y, vy, __dmul_rn(t.z, vz)));
    a.d = fma(fma(-xd, xv, dv) * r.area, w, a.d);
  }
  __device__ static RecVec64 plain_record(const Pse64Src& s, int64_t j) {
    return PlaneD464<PsePlaneSecondF64>::plain_record(s, j);
  }
};

struct PseSphereDdot64 : PseSphereVec64<PseSphereDdotF64> {
  using Params = PseExtF64Params;
  struct Tgt {
    double u, v;
  };
  __device__ static Tgt load(const Params& p, int64_t i) { return Tgt{p.s1[i], p.s2[i]}; }
  __device__ static __forceinline__ void add(const Tgt& t, const Rec& r, double dx, double dy, double dz, double w,
                                             Acc& a) {
    const double g = r.area * w;
    const double gx = g * dx, gy = g * dy, gz = g * dz;
    const double su = r.a + t.u, sv = r.b + t.v, sw = r.c + t.v;  // w_j with v_i, as the reference
    a.ux = fma(su, gx, a.ux);
    a.uy = fma(su, gy, a.uy);
    a.uz = fma(su, gz, a.uz);
    a.vx = fma(sv, gx, a.vx);
    a.vy = fma(sv, gy, a.vy);
    a.vz = fma(sv, gz, a.vz);
    a.wx = fma(sw, gx, a.wx);
    a.wy = fma(sw, gy, a.wy);
    a.wz = fma(sw, gz, a.wz);
  }
  __device__ static RecVec64 plain_record(const Pse64Src& s, int64_t j) {
    return PlaneD464<PsePlaneSecondF64>::plain_record(s, j);
  }
};

// A pair in the reference's expressions.
template <class Op>
__device__ __noinline__ typename Op::Acc pse64_plain(const typename Op::Params& p, const Pse64Src& s, int64_t i,
                                                     int64_t j, typename Op::Acc a) {
  Op::Plain::interact(p, Op::Plain::load(p, i), Op::plain_record(s, j), a);
  return a;
}

// ------------------------------------------------------------------ prep
// Records, FP32 offsets from the tile's centre and ball of one tile; one CTA per tile.  The radius
// is widened by 1e-9 of itself and of the centre's size, which covers the rounding of the tests; an
// odd particle leaves the centre alone and makes the radius infinite.  CTA 0 also writes the
// powers.
template <class Op>
__global__ void __launch_bounds__(kPse64Tile) pse64_prep_kernel(Pse64Src s, const int32_t* idx, int64_t ns, int unit,
                                                                typename Op::Rec* out, float4* side, TileBall* bounds,
                                                                double* powers) {
  __shared__ double red[4][kPse64Tile];
  const int tid = threadIdx.x;
  const int64_t k = static_cast<int64_t>(blockIdx.x) * kPse64Tile + tid;
  const bool valid = k < ns;
  const int32_t j = valid ? idx[k] : 0;
  CutPoint p{};
  if (valid) p = cut_point(s.x, s.y, s.z, j, unit);
  const double3 q = p.q;
  const bool odd = valid && odd_point(p);
  red[0][tid] = odd ? 0.0 : q.x;
  red[1][tid] = odd ? 0.0 : q.y;
  red[2][tid] = odd ? 0.0 : q.z;
  red[3][tid] = valid && !odd ? 1.0 : 0.0;
  __syncthreads();
  for (int w = kPse64Tile / 2; w > 0; w >>= 1) {
    if (tid < w) {
#pragma unroll
      for (int c = 0; c < 4; ++c) red[c][tid] += red[c][tid + w];
    }
    __syncthreads();
  }
  const double cnt = red[3][0] > 0.0 ? red[3][0] : 1.0;
  const double cx = red[0][0] / cnt, cy = red[1][0] / cnt, cz = red[2][0] / cnt;
  const double dx = q.x - cx, dy = q.y - cy, dz = q.z - cz;
  __syncthreads();
  red[0][tid] = odd ? __longlong_as_double(0x7ff0000000000000LL)
                    : valid ? sqrt(dx * dx + dy * dy + dz * dz) : 0.0;
  __syncthreads();
  for (int w = kPse64Tile / 2; w > 0; w >>= 1) {
    if (tid < w) red[0][tid] = fmax(red[0][tid], red[0][tid + w]);
    __syncthreads();
  }
  if (tid == 0) {
    const double sz = fabs(cx) + fabs(cy) + fabs(cz);
    bounds[blockIdx.x] = TileBall{cx, cy, cz, red[0][0] * (1.0 + 1e-9) + 1e-9 * sz};
  }
  typename Op::Rec r{};
  if (valid) {
    Op::fill(r, s, j);
    r.x = p.raw.x;
    r.y = p.raw.y;
    r.z = p.raw.z;
    if constexpr (Op::kUnit) {
      r.r = odd ? __longlong_as_double(0x7ff8000000000000LL) : p.r;
      r.inv = 1.0 / p.r;
    }
    r.idx = j;
    r.odd = odd ? 1 : 0;
  }
  out[k] = r;
  const float nan = __int_as_float(0x7fffffff);
  side[k] = odd ? make_float4(nan, nan, nan, 0.f)
                : make_float4(static_cast<float>(dx), static_cast<float>(dy), static_cast<float>(dz), 0.f);
  if (blockIdx.x == 0) {
    for (int e = tid; e < 256; e += kPse64Tile) powers[e] = exp2(-static_cast<double>(e) / 256.0);
  }
}

// ------------------------------------------------------------------ sweep
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// S lanes per target.
template <class Op, int ANG, int S>
__global__ void __launch_bounds__(32) pse64_sweep_kernel(typename Op::Params p, Pse64Args a,
                                                         const typename Op::Rec* __restrict__ src) {
  using Rec = typename Op::Rec;
  using Acc = typename Op::Acc;
  __shared__ TilePipe<float4, kPse64Tile, kPse64Stages> pp;
  __shared__ uint64_t mine[kPse64Mine][32];   // the lanes' sources, a tile's at a time
  __shared__ int32_t tile_of[kPse64Mine][32];  // and of which tile
  __shared__ double powers[256];
  __shared__ int32_t list[kPse64List];
  const int lane = threadIdx.x;
  const int64_t k = static_cast<int64_t>(blockIdx.x) * (32 / S) + lane / S;
  const bool valid = k < a.nt;
  // this lane's sources of a tile: the (lane modulo S)-th of S consecutive parts
  const uint64_t part = (~0ull >> (64 - 64 / S)) << (lane % S * (64 / S));
  const int64_t kk = valid ? k : a.nt - 1;
  const int64_t i = a.tperm ? static_cast<int64_t>(a.tperm[kk]) : a.ib + kk;
  const typename Op::Tgt t = Op::load(p, i);
  const CutPoint cp = cut_point(a.x, a.y, a.z, i, a.unit);
  const double3 tp = cp.q;
  const bool odd = a.all_plain || odd_point(cp);
  const long long rbits = odd ? static_cast<long long>(1ull << 63) : __double_as_longlong(cp.r);
  const double inv = 1.0 / cp.r, inv2 = __dmul_rn(inv, inv);
  for (int e = lane; e < 256; e += 32) powers[e] = a.powers[e];
  tile_pipe_init(pp);  // (synchronises)
  // The ball around the warp's targets (NaN or infinite: in reach of everything).  The lanes' own tests let
  // a source pass at up to 1.00003 reach + 4e-6 of its tile's radius; no tile with such a source is left
  // out, so that a target's sum does not depend on the warp it is in.
  const double wx = warp_sum(tp.x) / 32.0, wy = warp_sum(tp.y) / 32.0, wz = warp_sum(tp.z) / 32.0;
  double far = (tp.x - wx) * (tp.x - wx) + (tp.y - wy) * (tp.y - wy) + (tp.z - wz) * (tp.z - wz);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) far = fmax(far, __shfl_xor_sync(0xffffffffu, far, o));
  const double wr = sqrt(far) * (1.0 + 1e-9) + 1e-9 * (fabs(wx) + fabs(wy) + fabs(wz)) + a.reach * 1.00004;

  Acc acc{};
  // A pair's kernel value and terms.  `same`: both particles are as far from the sphere's centre.  The
  // squared chord comes from the positions, whose differences are exact to 2^-53: rounding the unit
  // directions moved every target by up to 2^-53, which the derivative kernels amplify by 1 / eps.
  auto offset = [&](const Rec& n) {
    return make_double3(__dsub_rn(cp.raw.x, n.x), __dsub_rn(cp.raw.y, n.y),
                        Op::kDim == 3 ? __dsub_rn(cp.raw.z, n.z) : 0.0);
  };
  auto squared = [&](const Rec& n, const double3& d, bool same) {
    double v = Op::kDim == 3 ? fma(d.x, d.x, fma(d.y, d.y, __dmul_rn(d.z, d.z))) : fma(d.x, d.x, __dmul_rn(d.y, d.y));
    if constexpr (Op::kUnit) {
      if (same) {
        v = __dmul_rn(v, inv2);
      } else {  // |p - p'|^2 = (r - r')^2 + r r' chord^2
        const double dr = __dsub_rn(cp.r, n.r);
        v = __dmul_rn(fma(-dr, dr, v), __dmul_rn(inv, n.inv));
      }
    }
    return v;
  };
  auto regular = [&](const Rec& n) {
    if constexpr (Op::kUnit) return same_radius(rbits, n.r);
    return !odd && !n.odd;
  };
  // any pair
  auto one = [&](const Rec& n) {
    bool plain = odd || n.odd;
    if constexpr (Op::kUnit) plain |= !(fabs(cp.r - n.r) <= 0.25 * cp.r);  // (the difference above cancels)
    if (plain) {
      constexpr int NA = static_cast<int>(sizeof(Acc) / sizeof(double));
      const Acc d = pse64_plain<Op>(p, a.src, i, n.idx, odd ? acc : Acc{});
      if (odd) {
        acc = d;  // an odd target's sum is all in Plain's units
      } else {
        double* av = reinterpret_cast<double*>(&acc);
        const double* dv = reinterpret_cast<const double*>(&d);
#pragma unroll
        for (int c = 0; c < NA; ++c) av[c] = fma(dv[c], a.unscale, av[c]);
      }
      return;
    }
    const double3 d = offset(n);
    const double w = pse64_kernel_value<Op>(pse64_q<ANG>(a, squared(n, d, regular(n))), powers);
    Op::add(t, n, d.x, d.y, d.z, w, acc);
  };
  int held = 0;  // entries of mine and tile_of that this lane holds
  // Evaluates the held sources in ascending order.
  auto evaluate = [&]() {
    int e = 0;
    uint64_t bits = 0;
    const Rec* base = src;
    // the lane's next source, or null
    auto next = [&]() -> const Rec* {
      if (bits == 0) {
        if (e == held) return nullptr;
        bits = mine[e][lane];  // never zero
        base = src + static_cast<int64_t>(tile_of[e][lane]) * kPse64Tile;
        ++e;
      }
      const int j = __ffsll(static_cast<long long>(bits)) - 1;
      bits &= bits - 1;
      return base + j;
    };
    const Rec *at0 = next(), *at1 = next();
    Rec r0 = *(at0 ? at0 : src), r1 = *(at1 ? at1 : src);
    while (at0) {
      const Rec n0 = r0, n1 = r1;
      const bool two = at1 != nullptr;
      at0 = next();
      at1 = next();
      r0 = *(at0 ? at0 : src);  // on their way while this pair of pairs is evaluated
      r1 = *(at1 ? at1 : src);
      if (!(regular(n0) && regular(n1))) {
        one(n0);
        if (two) one(n1);
        continue;
      }
      const double3 d0 = offset(n0), d1 = offset(n1);
      const double w0 = pse64_kernel_value<Op>(pse64_q<ANG>(a, squared(n0, d0, true)), powers);
      const double w1 = pse64_kernel_value<Op>(pse64_q<ANG>(a, squared(n1, d1, true)), powers);
      Op::add(t, n0, d0.x, d0.y, d0.z, w0, acc);
      Acc more = acc;
      Op::add(t, n1, d1.x, d1.y, d1.z, w1, more);
      if (two) acc = more;
    }
    held = 0;
    __syncwarp();
  };

  uint32_t g = 0;
  int cnt = 0;
  for (int64_t w0 = 0; w0 < a.n_tiles; w0 += 32) {
    const int64_t tl = w0 + lane;
    bool in = tl < a.n_tiles;
    if (in) {
      const TileBall b = a.bounds[tl];
      const double dx = wx - b.x, dy = wy - b.y, dz = wz - b.z, lim = wr + b.r * 1.00001;
      in = !(dx * dx + dy * dy + dz * dz > lim * lim);
    }
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (in) list[cnt + __popc(m & ((1u << lane) - 1u))] = static_cast<int32_t>(tl);
    cnt += __popc(m);
    if (cnt <= kPse64List - 32 && w0 + 32 < a.n_tiles) continue;
    __syncwarp();
    int q = 0;
    const bool ok = warp_sweep_tiles(
        a.side, [&](int64_t e) { return static_cast<int64_t>(list[e]); }, cnt, pp, g, a.status, default_wait(),
        static_cast<const float4*>(nullptr), [&](const float4* side) {
          const int64_t tile = list[q];
          const TileBall b = a.bounds[tile];
          const float ox = static_cast<float>(tp.x - b.x), oy = static_cast<float>(tp.y - b.y),
                      oz = static_cast<float>(tp.z - b.z);
          // the offsets' and the test's roundings: a few 2^-24 of the offsets, which are at most
          // the target's own and the tile's radius
          const float lim = static_cast<float>(a.reach) * 1.00001f +
                            1e-6f * (fabsf(ox) + fabsf(oy) + fabsf(oz) + static_cast<float>(b.r));
          const float lim2 = lim * lim;
          const int64_t left = a.ns - tile * kPse64Tile;  // sources of the tile
          uint32_t half[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t bits = 0;
#pragma unroll 8
            for (int j = 0; j < 32; ++j) {
              const float4 s = side[h * 32 + j];
              const float dx = ox - s.x, dy = oy - s.y, dz = oz - s.z;
              if (!(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > lim2)) bits |= 1u << j;
            }
            if (odd) bits = 0xffffffffu;
            const int64_t n = left - 32 * h;
            half[h] = n >= 32 ? bits : (n > 0 ? bits & ((1u << n) - 1u) : 0u);
          }
          ++q;
          const uint64_t bits = ((static_cast<uint64_t>(half[1]) << 32) | half[0]) & part;
          if (bits != 0) {
            mine[held][lane] = bits;
            tile_of[held][lane] = static_cast<int32_t>(tile);
            ++held;
          }
          if (__any_sync(0xffffffffu, held == kPse64Mine)) evaluate();
        });
    if (!ok) return;  // a wait gave up: the status word is set and the outputs are not used
    cnt = 0;
    __syncwarp();
  }
  evaluate();
  constexpr int NA = static_cast<int>(sizeof(Acc) / sizeof(double));
  double* av = reinterpret_cast<double*>(&acc);
#pragma unroll
  for (int c = 0; c < NA; ++c) {
#pragma unroll
    for (int o = 1; o < S; o <<= 1) av[c] += __shfl_xor_sync(0xffffffffu, av[c], o);  // the parts' sums
    if (!odd) av[c] = __dmul_rn(av[c], a.scale);
  }
  if (valid && lane % S == 0) Op::Plain::store(p, i, i - a.ib, acc);
}

}  // namespace lpm
