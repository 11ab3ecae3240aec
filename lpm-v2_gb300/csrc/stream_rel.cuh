// stream_rel.cuh -- the stream functions (sphere, plane, beta-plane log) and the sphere SWE velocity in
// FP32C on group-relative layouts (bve_rel.cuh, plane_rel.cuh): curve-sorted sources, offsets from
// each group's centroid, a precision choice per warp and group, and target pairs in packed FP32x2
// arithmetic.
//
// Sphere.  Reference: SetStreamFunctionsOnMesh, src/SphereBVE.f90:445-485:
//   psi_i = -1/(4 pi) sum_{j != i} ln(a^2 - x_i.x_j) zeta_j A_j   (relative and absolute zeta)
// With p = x / a and c = |p|^2 - 1, a^2 - x_i.x_j = (a^2 / 2) q_ij with q_ij = |d|^2 - c_i - c_j
// (exact), so
//   psi_i = sum_{j != i} S_j ln q_ij - ln(a^2 / 2) / (4 pi) sum_{j != i} zeta_j A_j,
// S_j = -zeta_j A_j / (4 pi).  The sweep forms the first sum; the finish adds the second from
// a fixed-order FP64 total minus the target's own term.
//
// A far warp (every target beyond 3R of the group's centroid) takes the expanded form of the BVE sweep
// in the group's basis (bve_rel.cuh), h = q/2 = C - c gamma - a alpha - b beta, C = 1 - p_i.o, and
// measures it against C, the group's own distance:
//   h = C (1 + x),  sum_j S_j ln q_j = ln(2 C) S_g + sum_j S_j log1p(x_j),  S_g = sum_j S_j,
// where x is three packed operations (the target's gamma, alpha and beta are divided by C once per
// group) and |x| <= (|t| max |(a, b)| + |gamma| max |c|) / C is small: about 2 R / |t|.  log1p is a
// polynomial of degree 6, 9 or 12, whichever the warp's bound allows (|x| <= 0.1375, 0.3125, 0.46), and
// ln(2 C) a two-float log per target and group.  So a pair takes 3 + 6 + 2 packed operations at the
// lowest degree, no integer split, no table load and no MUFU, where the log per pair took 4 + 9 + 2,
// eight integer operations and four table loads; and the partial sums hold terms of size |S_j x_j|,
// not |S_j ln q_j|.  Beyond the last bound a far warp forms ln h per pair (ln_q2_shift).  A compact group
// near the warp takes d = t_hi - s_hi with the self-pair select and the clamp to >= 2^-126, any other
// near group the two-float form, both with a log per pair, flushed into the compensated (hi, lo) sums
// every 16 sources (32 gave errors 1.1 to 1.7 times as large below 30,000 points).  C is common to a
// group's pairs, so what its float misses is carried (cosine_rest; without it the error at 122,882
// points is 2.2 times as large, and the sum 3.5 % faster).
// Bound: the FP32 pipe.  At 122,882 points (81,920 sources) the call took 8.24 ms with a log per pair, 5.85
// with log1p (128 x 4 targets and 4 CTAs per SM), 5.27 with 128 x 6 and 3 (128 x 8 and 2: 6.36; groups of 32,
// 64 and 128 within 3 %, the groups of 64 being the best from 7,682 points on).
// The sphere sweep runs on the warp-decoupled pipeline (engine.cuh, the groups copied with each tile):
// warps meet near and far groups at different rates.
#pragma once

#include "bve_rel.cuh"
#include "ln_table.cuh"
#include "ops.cuh"
#include "plane_rel.cuh"

namespace lpm {

struct StreamFn {
  static constexpr int kGroup = 64;
  static constexpr int kFlush = 16;
  // The largest compact group (its near pairs carry an absolute 2^-24 R): of the sets with 128 to a group
  // that were compact up to a/2, those of 64 up to here are.  Beyond it the two-float form costs little,
  // since such sets have a few hundred sources.
  static constexpr float kCompactRadius = 0.35f;
  struct __align__(16) Rec {
    float4 a;  // -a, -a, -b, -b                 (the source in its group's basis)
    float4 b;  // -c, -c, S_rel, S_rel
    float4 c;  // S_abs, S_abs, -c_j, 0
    float4 d;  // -sx_hi, -sy_hi, -sz_hi, 0      (near forms)
    float4 e;  // -sx_lo, -sy_lo, -sz_lo, 0      (near forms)
  };
  struct __align__(16) Group {
    BveRel::Origin o;  // hi: o, R (-R compact, 3e38 no sources); lo: k, |o|^2 + k, max |(a, b)|, max |c|
    float4 e1;         // e1, o.e1
    float4 e2;         // e2, o.e2
    float4 s;          // S_rel and S_abs of the group as hi, lo pairs
  };
};

// The sphere SWE velocity's record.
struct StreamRel {
  struct __align__(16) Rec {
    float4 a;  // -sx_hi, -sx_hi, -sy_hi, -sy_hi
    float4 b;  // -sz_hi, -sz_hi, -c_j, -c_j
    float4 c;  // S_rel, S_rel, S_abs, S_abs
    float4 d;  // -sx_lo, -sx_lo, -sy_lo, -sy_lo
    float4 e;  // -sz_lo, -sz_lo, 0, 0
  };
};

// Natural log of two positive normal floats (the sweeps clamp them): per lane q = 2^k m with
// m in [sqrt(1/2), sqrt(2)) (an integer split; 0x3f3504f3 = fl(sqrt(1/2))).  Bits 19..23 of
// m pick (inv, ln c) from a 32-entry table in shared memory (ln_table.cuh: 1/c for c the
// midpoint of the key's interval, with ln c exact to ~2e-4 ulp in float -- Gal's accurate
// tables).  Then, packed, r = m inv - 1 (one FMA, |r| <= 0.0305, exact to 2^-30),
// ln(1 + r) = r + r^2 (-1/2 + r/3 - r^2/4 + r^3/5) (truncated at r^6/6 < 2e-10), and
// ln q = (k ln 2 + ln c) + ln(1 + r): 9 packed operations and two 8-byte shared loads (keys
// 6 and 22 alone share banks), no MUFU; good to about 1 ulp of the larger part.
// The exponent split of a positive normal float with bits b: q = 2^k m, m in [sqrt(1/2),
// sqrt(2)) (0x3f3504f3 = fl(sqrt(1/2))); returns k and writes the bits of m.  Inline PTX
// keeps the integer sequence as written: the same four operations in C++, fed straight
// from a packed FFMA2 result in the planar stream sweep's far loop, gave (nvcc 13.0,
// sm_103a) logs as if k were b - 0x3f3504f3, unshifted.
__device__ __forceinline__ int exp_split(int b, int& mb) {
  int k;
  asm("{\n\t.reg .s32 t;\n\tsub.s32 t, %2, 0x3f3504f3;\n\tshr.s32 %0, t, 23;\n\tshl.b32 t, %0, 23;\n\t"
      "sub.s32 %1, %2, t;\n\t}"
      : "=r"(k), "=r"(mb)
      : "r"(b));
  return k;
}

// ln_q2_shift(q, shift_bias(s0, s1)) is (ln q.x - s0 ln 2, ln q.y - s1 ln 2) for small
// integers s: the shift only moves the exponent k (the float k - s is exact), so it costs
// nothing -- it replaces the constant of the magic-number conversion of k.
__device__ __forceinline__ float2 shift_bias(int s0, int s1) {
  return make_float2(-12582912.0f - static_cast<float>(s0), -12582912.0f - static_cast<float>(s1));
}

// The table into shared memory (threads 0..31; the caller's next __syncthreads publishes it).
__device__ __forceinline__ void ln_tab_load(float2* tab) {
  if (threadIdx.x < 32) tab[threadIdx.x] = make_float2(kLnTabInv[threadIdx.x], kLnTabLog[threadIdx.x]);
}

__device__ __forceinline__ float2 ln_q2_shift(float2 q, float2 bias, const float2* tab) {
  int m0, m1;
  const int k0 = exp_split(__float_as_int(q.x), m0), k1 = exp_split(__float_as_int(q.y), m1);
  const float2 e0 = tab[(m0 >> 19) & 31], e1 = tab[(m1 >> 19) & 31];
  const float2 m = make_float2(__int_as_float(m0), __int_as_float(m1));
  const float2 kf = __fadd2_rn(make_float2(__int_as_float(k0 + 0x4b400000), __int_as_float(k1 + 0x4b400000)), bias);
  const float2 r = __ffma2_rn(m, make_float2(e0.x, e1.x), make_float2(-1.0f, -1.0f));
  float2 p = __ffma2_rn(make_float2(0.2f, 0.2f), r, make_float2(-0.25f, -0.25f));
  p = __ffma2_rn(p, r, make_float2(0.33333334f, 0.33333334f));
  p = __ffma2_rn(p, r, make_float2(-0.5f, -0.5f));
  const float2 b = __ffma2_rn(__fmul2_rn(r, r), p, r);
  const float2 a = __ffma2_rn(kf, make_float2(0.69314718f, 0.69314718f), make_float2(e0.y, e1.y));
  return __fadd2_rn(a, b);
}

__device__ __forceinline__ float2 ln_q2(float2 q, const float2* tab) { return ln_q2_shift(q, shift_bias(0, 0), tab); }

// The log argument of a pair: q clamped to >= 2^-126, or 1 (a zero term) when d = 0.
__device__ __forceinline__ float2 stream_arg(float2 u, float2 q) {
  return make_float2(u.x != 0.0f ? fmaxf(q.x, kLogFloor) : 1.0f, u.y != 0.0f ? fmaxf(q.y, kLogFloor) : 1.0f);
}

// ln q as a sum hi + lo, good to about 2^-29 (the parts ln_q2_shift rounds away are kept).
__device__ __forceinline__ void ln_q2_parts(float2 q, float2 bias, const float2* tab, float2& hi, float2& lo) {
  int m0, m1;
  const int k0 = exp_split(__float_as_int(q.x), m0), k1 = exp_split(__float_as_int(q.y), m1);
  const float2 e0 = tab[(m0 >> 19) & 31], e1 = tab[(m1 >> 19) & 31];
  const float2 m = make_float2(__int_as_float(m0), __int_as_float(m1)), lc = make_float2(e0.y, e1.y);
  const float2 kf = __fadd2_rn(make_float2(__int_as_float(k0 + 0x4b400000), __int_as_float(k1 + 0x4b400000)), bias);
  const float2 r = __ffma2_rn(m, make_float2(e0.x, e1.x), make_float2(-1.0f, -1.0f));
  float2 p = __ffma2_rn(make_float2(0.2f, 0.2f), r, make_float2(-0.25f, -0.25f));
  p = __ffma2_rn(p, r, make_float2(0.33333334f, 0.33333334f));
  p = __ffma2_rn(p, r, make_float2(-0.5f, -0.5f));
  const float2 b = __ffma2_rn(__fmul2_rn(r, r), p, r);
  // k ln 2 + ln c: |k ln 2| is 0 or the larger, so one subtraction chain gives the sum's rounding
  const float2 l2 = make_float2(0.69314718f, 0.69314718f);
  const float2 kl = __fmul2_rn(kf, l2);
  float2 ke = __ffma2_rn(kf, l2, make_float2(-kl.x, -kl.y));
  ke = __ffma2_rn(kf, make_float2(-1.9046542e-9f, -1.9046542e-9f), ke);  // ln 2 - fl(ln 2)
  hi = __fadd2_rn(kl, lc);
  const float2 d = __fadd2_rn(hi, make_float2(-kl.x, -kl.y));
  lo = __fadd2_rn(__fadd2_rn(__fadd2_rn(lc, make_float2(-d.x, -d.y)), ke), b);
}

// log1p(x) = x + x^2 Q(x): minimax polynomials of degree N (absolute error <= 4.2e-9 with the
// coefficients in float) on |x| <= log1p_limit(N).
template <int N>
__device__ __forceinline__ constexpr float log1p_limit() {
  static_assert(N == 6 || N == 9 || N == 12, "fitted degrees");
  return N == 6 ? 0.1375f : (N == 9 ? 0.3125f : 0.46f);
}

template <int N>
__device__ __forceinline__ float2 log1p_poly(float2 x) {
  constexpr float c6[5] = {-0.500000179f, 0.333306402f, -0.249940857f, 0.204092115f, -0.171654522f};
  constexpr float c9[8] = {-0.499999315f, 0.333331376f, -0.250072867f, 0.200134292f,
                           -0.164394721f, 0.139719114f, -0.151976928f, 0.140937984f};
  constexpr float c12[11] = {-0.499999851f, 0.333336055f, -0.250013113f, 0.199855641f,   -0.166288242f, 0.145503074f,
                             -0.12986657f,  0.0896346495f, -0.0693810582f, 0.167132765f, -0.171647802f};
  auto c = [&](int k) {
    const float v = N == 6 ? c6[k < 5 ? k : 0] : (N == 9 ? c9[k < 8 ? k : 0] : c12[k]);
    return make_float2(v, v);
  };
  float2 p = c(N - 2);
#pragma unroll
  for (int k = N - 3; k >= 0; --k) p = __ffma2_rn(p, x, c(k));
  return __ffma2_rn(__fmul2_rn(x, x), p, x);
}

// (1 - p.o) - c for a pair of targets p = (hi, lo) and a float c near 1 - p.o: the sum's and the
// products' roundings are carried (two-sum and fma), so the result is good to about 2^-46.
__device__ __forceinline__ float2 cosine_rest(const BveX2::Pair& p, float4 o, float2 c) {
  const float2 h[3] = {p.xh, p.yh, p.zh}, l[3] = {p.xl, p.yl, p.zl};
  const float no[3] = {-o.x, -o.y, -o.z};
  float2 s = make_float2(1.0f, 1.0f), e = make_float2(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float2 n2 = make_float2(no[k], no[k]);
    const float2 q = __fmul2_rn(h[k], n2);
    const float2 qe = __ffma2_rn(h[k], n2, make_float2(-q.x, -q.y));
    const float2 t = __fadd2_rn(s, q);
    const float2 b = __fadd2_rn(t, make_float2(-s.x, -s.y));
    const float2 r = __fadd2_rn(t, make_float2(-b.x, -b.y));
    const float2 te = __fadd2_rn(__fadd2_rn(s, make_float2(-r.x, -r.y)), __fadd2_rn(q, make_float2(-b.x, -b.y)));
    s = t;
    e = __ffma2_rn(l[k], n2, __fadd2_rn(e, __fadd2_rn(te, qe)));
  }
  return __fadd2_rn(__fadd2_rn(s, make_float2(-c.x, -c.y)), e);
}

__device__ __forceinline__ float sqrt_approx(float v) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

template <int NP>
__device__ __forceinline__ void stream_flush(float2 (&ar)[NP], float2 (&aa)[NP], float2 (&hr)[NP], float2 (&lr)[NP],
                                             float2 (&ha)[NP], float2 (&la)[NP]) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    comp_add(hr[p].x, lr[p].x, ar[p].x);
    comp_add(hr[p].y, lr[p].y, ar[p].y);
    comp_add(ha[p].x, la[p].x, aa[p].x);
    comp_add(ha[p].y, la[p].y, aa[p].y);
    ar[p] = aa[p] = make_float2(0.f, 0.f);
  }
}

// One far group in the log1p form: (ga, al, be) are the target's coordinates over C, x0 what C's float
// misses of it, over C.
template <int NP, int N>
__device__ __forceinline__ void stream_far_group(const StreamFn::Rec* __restrict__ gr, const float2 (&x0)[NP],
                                                 const float2 (&ga)[NP],
                                                 const float2 (&al)[NP], const float2 (&be)[NP], float2 (&ar)[NP],
                                                 float2 (&aa)[NP]) {
#pragma unroll 2
  for (int j = 0; j < StreamFn::kGroup; ++j) {
    const float4 ra = gr[j].a, rb = gr[j].b;
    const float2 sa = lo2(gr[j].c);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      float2 x = __ffma2_rn(ga[p], lo2(rb), x0[p]);
      x = __ffma2_rn(al[p], lo2(ra), x);
      x = __ffma2_rn(be[p], hi2(ra), x);
      const float2 y = log1p_poly<N>(x);
      ar[p] = __ffma2_rn(hi2(rb), y, ar[p]);
      aa[p] = __ffma2_rn(sa, y, aa[p]);
    }
  }
}

template <int THREADS, int TPT, int TILE, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) stream_rel_sweep_kernel(SweepArgs<BveF32> a,
                                                                         const StreamFn::Rec* __restrict__ src,
                                                                         const StreamFn::Group* __restrict__ org,
                                                                         const BveRel::Tgt* __restrict__ tgt) {
  static_assert(TPT % 2 == 0, "targets come in pairs");
  constexpr int NP = TPT / 2;
  constexpr int G = StreamFn::kGroup;
  constexpr int GPT = TILE / G;
  constexpr int FL = StreamFn::kFlush;
  static_assert(G % FL == 0, "flush interval must divide the group");
  using Rec = StreamFn::Rec;
  __shared__ TilePipe<Rec, TILE, 2, StreamFn::Group, GPT> pipe;
  __shared__ __align__(8) float2 ln_tab[32];

  const int64_t chunk = blockIdx.y;
  const ChunkTiles ct = chunk_tiles(a.n_tiles);

  BveX2::Pair pr[NP];
  float2 hr[NP], lr[NP], ha[NP], la[NP], ar[NP], aa[NP];
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (THREADS * TPT);
  const int64_t count = a.nt - first < THREADS * TPT ? a.nt - first : THREADS * TPT;
  bve_load_pairs<NP>(tgt + first, count, pr);
#pragma unroll
  for (int p = 0; p < NP; ++p) hr[p] = lr[p] = ha[p] = la[p] = ar[p] = aa[p] = make_float2(0.f, 0.f);

  ln_tab_load(ln_tab);
  tile_pipe_init(pipe);
  uint32_t g = 0;
  auto body = [&](const Rec* tl, const StreamFn::Group* og) {
#pragma unroll 1
    for (int g0 = 0; g0 < TILE; g0 += G) {
      const StreamFn::Group& gp = og[g0 / G];
      const BveRel::Origin o = gp.o;
      const Rec* gr = tl + g0;
      const float rg = fabsf(o.hi.w);
      if (rg == 3.0e38f) continue;  // no sources
      float2 tx[NP], ty[NP], tz[NP], n2[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        tx[p] = rel1x2(pr[p].xh, pr[p].xl, o.hi.x);
        ty[p] = rel1x2(pr[p].yh, pr[p].yl, o.hi.y);
        tz[p] = rel1x2(pr[p].zh, pr[p].zl, o.hi.z);
      }
      // far: every target of the warp beyond 3R (and off the centroid of a zero-radius group)
      const float lim = fmaxf((BveRel::kNearFactor * rg) * (BveRel::kNearFactor * rg), 7.888609052210118e-31f);
      bool nearw = false;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        n2[p] = __ffma2_rn(tz[p], tz[p], __ffma2_rn(ty[p], ty[p], __fmul2_rn(tx[p], tx[p])));
        nearw |= !(n2[p].x > lim) | !(n2[p].y > lim);
      }
      if (!__any_sync(0xffffffffu, nearw)) {
        const float4 e1 = gp.e1, e2 = gp.e2;
        float2 al[NP], be[NP], ga[NP], cc[NP], inv[NP];
        float xb = 0.f;  // the largest |x| of the thread's targets in this group
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const float2 nq = __fadd2_rn(n2[p], pr[p].nc);  // |t|^2 - c_i
          cc[p] = __ffma2_rn(nq, make_float2(0.5f, 0.5f), make_float2(o.lo.x, o.lo.x));
          ga[p] = __ffma2_rn(nq, make_float2(-0.5f, -0.5f), make_float2(o.lo.y, o.lo.y));
          al[p] = __ffma2_rn(tx[p], make_float2(e1.x, e1.x), make_float2(e1.w, e1.w));
          al[p] = __ffma2_rn(ty[p], make_float2(e1.y, e1.y), al[p]);
          al[p] = __ffma2_rn(tz[p], make_float2(e1.z, e1.z), al[p]);
          be[p] = __ffma2_rn(tx[p], make_float2(e2.x, e2.x), make_float2(e2.w, e2.w));
          be[p] = __ffma2_rn(ty[p], make_float2(e2.y, e2.y), be[p]);
          be[p] = __ffma2_rn(tz[p], make_float2(e2.z, e2.z), be[p]);
          inv[p] = make_float2(rcp_approx(cc[p].x), rcp_approx(cc[p].y));
          const float b0 = fmaf(sqrt_approx(n2[p].x), o.lo.z, fabsf(ga[p].x) * o.lo.w) * inv[p].x;
          const float b1 = fmaf(sqrt_approx(n2[p].y), o.lo.z, fabsf(ga[p].y) * o.lo.w) * inv[p].y;
          xb = fmaxf(xb, fmaxf(cc[p].x > 0.f ? b0 : 3.0e38f, cc[p].y > 0.f ? b1 : 3.0e38f));
        }
        float2 x0[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) x0[p] = __fmul2_rn(cosine_rest(pr[p], o.hi, cc[p]), inv[p]);
        const float4 s = gp.s;
        const float xw = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(xb)));
        if (xw <= log1p_limit<12>()) {
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            ga[p] = __fmul2_rn(ga[p], inv[p]);
            al[p] = __fmul2_rn(al[p], inv[p]);
            be[p] = __fmul2_rn(be[p], inv[p]);
          }
          if (xw <= log1p_limit<6>()) {
            stream_far_group<NP, 6>(gr, x0, ga, al, be, ar, aa);
          } else if (xw <= log1p_limit<9>()) {
            stream_far_group<NP, 9>(gr, x0, ga, al, be, ar, aa);
          } else {
            stream_far_group<NP, 12>(gr, x0, ga, al, be, ar, aa);
          }
          // ln(2 C) S_g, the leading product with its rounding
          const float2 bias = shift_bias(-1, -1);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            float2 lh, ll;
            ln_q2_parts(cc[p], bias, ln_tab, lh, ll);
            const float2 pr_ = __fmul2_rn(make_float2(s.x, s.x), lh), pa_ = __fmul2_rn(make_float2(s.z, s.z), lh);
            comp_add(hr[p].x, lr[p].x, pr_.x);
            comp_add(hr[p].y, lr[p].y, pr_.y);
            comp_add(ha[p].x, la[p].x, pa_.x);
            comp_add(ha[p].y, la[p].y, pa_.y);
            float2 er = __ffma2_rn(make_float2(s.x, s.x), lh, make_float2(-pr_.x, -pr_.y));
            float2 ea = __ffma2_rn(make_float2(s.z, s.z), lh, make_float2(-pa_.x, -pa_.y));
            er = __ffma2_rn(make_float2(s.y, s.y), lh, __ffma2_rn(make_float2(s.x, s.x), ll, er));
            ea = __ffma2_rn(make_float2(s.w, s.w), lh, __ffma2_rn(make_float2(s.z, s.z), ll, ea));
            // ll holds ln's second part (up to 2^-5), so it joins the group's own partial
            ar[p] = __fadd2_rn(ar[p], er);
            aa[p] = __fadd2_rn(aa[p], ea);
          }
          stream_flush<NP>(ar, aa, hr, lr, ha, la);
        } else {
          // h = C - c gamma - a alpha - b beta > 0, ln q = ln h + ln 2; what C's float misses, common to
          // the group's pairs, to first order at h = C
          const float2 bias = shift_bias(-1, -1);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            ar[p] = __fmul2_rn(x0[p], make_float2(s.x, s.x));
            aa[p] = __fmul2_rn(x0[p], make_float2(s.z, s.z));
          }
#pragma unroll 1
          for (int j0 = 0; j0 < G; j0 += FL) {
            for (int j = j0; j < j0 + FL; ++j) {
              const float4 ra = gr[j].a, rb = gr[j].b;
              const float2 sa = lo2(gr[j].c);
#pragma unroll
              for (int p = 0; p < NP; ++p) {
                float2 h = __ffma2_rn(ga[p], lo2(rb), cc[p]);
                h = __ffma2_rn(al[p], lo2(ra), h);
                h = __ffma2_rn(be[p], hi2(ra), h);
                const float2 lg = ln_q2_shift(h, bias, ln_tab);
                ar[p] = __ffma2_rn(hi2(rb), lg, ar[p]);
                aa[p] = __ffma2_rn(sa, lg, aa[p]);
              }
            }
            stream_flush<NP>(ar, aa, hr, lr, ha, la);
          }
        }
      } else if (o.hi.w < 0.f) {
        // compact group near the warp: d = t_hi - s_hi (rel2_fast records: a self pair gives d = 0)
#pragma unroll 1
        for (int j0 = 0; j0 < G; j0 += FL) {
          for (int j = j0; j < j0 + FL; ++j) {
            const float4 rb = gr[j].b, rc = gr[j].c, rd = gr[j].d;
            const float2 sr = hi2(rb), sa = lo2(rc), ncj = make_float2(rc.z, rc.z);
#pragma unroll
            for (int p = 0; p < NP; ++p) {
              const float2 dx = __fadd2_rn(tx[p], make_float2(rd.x, rd.x));
              const float2 dy = __fadd2_rn(ty[p], make_float2(rd.y, rd.y));
              const float2 dz = __fadd2_rn(tz[p], make_float2(rd.z, rd.z));
              const float2 u = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
              const float2 q = __fadd2_rn(u, __fadd2_rn(pr[p].nc, ncj));
              const float2 lg = ln_q2(stream_arg(u, q), ln_tab);
              ar[p] = __ffma2_rn(sr, lg, ar[p]);
              aa[p] = __ffma2_rn(sa, lg, aa[p]);
            }
          }
          stream_flush<NP>(ar, aa, hr, lr, ha, la);
        }
      } else {
        // near group: d = (t_hi - s_hi) + (t_lo - s_lo)
        float2 txl[NP], tyl[NP], tzl[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          rel2x2(pr[p].xh, pr[p].xl, o.hi.x, tx[p], txl[p]);
          rel2x2(pr[p].yh, pr[p].yl, o.hi.y, ty[p], tyl[p]);
          rel2x2(pr[p].zh, pr[p].zl, o.hi.z, tz[p], tzl[p]);
        }
#pragma unroll 1
        for (int j0 = 0; j0 < G; j0 += FL) {
          for (int j = j0; j < j0 + FL; ++j) {
            const float4 rb = gr[j].b, rc = gr[j].c, rd = gr[j].d, re = gr[j].e;
            const float2 sr = hi2(rb), sa = lo2(rc), ncj = make_float2(rc.z, rc.z);
#pragma unroll
            for (int p = 0; p < NP; ++p) {
              const float2 dx =
                  __fadd2_rn(__fadd2_rn(tx[p], make_float2(rd.x, rd.x)), __fadd2_rn(txl[p], make_float2(re.x, re.x)));
              const float2 dy =
                  __fadd2_rn(__fadd2_rn(ty[p], make_float2(rd.y, rd.y)), __fadd2_rn(tyl[p], make_float2(re.y, re.y)));
              const float2 dz =
                  __fadd2_rn(__fadd2_rn(tz[p], make_float2(rd.z, rd.z)), __fadd2_rn(tzl[p], make_float2(re.z, re.z)));
              const float2 u = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
              const float2 q = __fadd2_rn(u, __fadd2_rn(pr[p].nc, ncj));
              const float2 lg = ln_q2(stream_arg(u, q), ln_tab);
              ar[p] = __ffma2_rn(sr, lg, ar[p]);
              aa[p] = __ffma2_rn(sa, lg, aa[p]);
            }
          }
          stream_flush<NP>(ar, aa, hr, lr, ha, la);
        }
      }
    }
  };
  warp_sweep_tiles(src, [ct](int64_t k) { return ct.first + k * ct.step; }, ct.count, pipe, g, a.status,
                   default_wait(), org, body);

#pragma unroll
  for (int p = 0; p < NP; ++p) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t il = first + bve_target<TPT>(2 * p + h);
      if (il < a.nt) {
        a.partial[(chunk * 2 + 0) * a.nt + il] =
            static_cast<double>(h ? hr[p].y : hr[p].x) + static_cast<double>(h ? lr[p].y : lr[p].x);
        a.partial[(chunk * 2 + 1) * a.nt + il] =
            static_cast<double>(h ? ha[p].y : ha[p].x) + static_cast<double>(h ? la[p].y : la[p].x);
      }
    }
  }
}

// Records and groups of the sorted sources (CTA t < n_tiles: tile t, TILE threads), then the nt
// targets from ib on as floats.  A source that is also a target leaves its zeta A in
// self_w[c * nt + j - ib] (zeroed before) for the finish to take out of the total.
template <int TILE>
__global__ void __launch_bounds__(TILE) stream_prep_kernel(const double* x, const double* y, const double* z,
                                                           const double* qr, const double* qa, const double* area,
                                                           const int32_t* sorted, int64_t ns, int64_t n_tiles,
                                                           double inv_a, int64_t ib, int64_t nt, StreamFn::Rec* out,
                                                           StreamFn::Group* org, BveRel::Tgt* tgt, double* self_w) {
  constexpr int G = StreamFn::kGroup, WPG = G / 32;
  static_assert(WPG == 2, "two warps per group");
  __shared__ float mx[TILE / 32][2];
  __shared__ double sums[TILE / 32][2];
  const int64_t t = blockIdx.x;
  if (t >= n_tiles) {
    const int64_t il = (t - n_tiles) * TILE + threadIdx.x;
    if (il < nt) tgt[il] = bve_split_target(BveF32::Params{x, y, z, inv_a}, ib + il);
    return;
  }
  const int64_t k = t * TILE + threadIdx.x;
  const bool valid = k < ns;
  const int32_t j = valid ? sorted[k] : 0;
  double px = 0.0, py = 0.0, pz = 0.0, cj = 0.0;
  if (valid) {
    px = x[j] * inv_a;
    py = y[j] * inv_a;
    pz = z[j] * inv_a;
    cj = fma(px, px, fma(py, py, fma(pz, pz, -1.0)));
  }
  const SplitPoint sp = split_point(px, py, pz);
  const GroupFrame f = sphere_group_frame<TILE, G>(valid, sp, cj, StreamFn::kCompactRadius);
  const GroupBasis b = group_basis(f);
  StreamFn::Rec r;
  float sr = 0.f, sa = 0.f, ab = 0.f, cm = 0.f;
  if (valid) {
    float hi[3], lo[3];
    group_offsets(f, sp, hi, lo);
    float af, bf, cf;
    basis_coords(b, f, hi, lo, af, bf, cf);
    const double wr = qr[j] * area[j], wa = qa[j] * area[j];
    sr = __double2float_rn(wr * -kInv4Pi);
    sa = __double2float_rn(wa * -kInv4Pi);
    ab = af * af + bf * bf;
    cm = fabsf(cf);
    r.a = make_float4(-af, -af, -bf, -bf);
    r.b = make_float4(-cf, -cf, sr, sr);
    r.c = make_float4(sa, sa, __double2float_rn(-cj), 0.f);
    r.d = make_float4(-hi[0], -hi[1], -hi[2], 0.f);
    r.e = make_float4(-lo[0], -lo[1], -lo[2], 0.f);
    if (j >= ib && j < ib + nt) {
      self_w[j - ib] = wr;
      self_w[nt + j - ib] = wa;
    }
  } else {
    // inert: zero strength at the centroid (q = |t - o|^2 - c_i > 0 unless the target sits
    // on o, where d = 0 gives a zero term)
    r.a = r.b = r.c = r.d = r.e = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  out[k] = r;
  // the group's totals and the bounds of its sources' coordinates
  double tr = sr, ta = sa;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    tr += __shfl_xor_sync(0xffffffffu, tr, o);
    ta += __shfl_xor_sync(0xffffffffu, ta, o);
    ab = fmaxf(ab, __shfl_xor_sync(0xffffffffu, ab, o));
    cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
  }
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    mx[wid][0] = ab;
    mx[wid][1] = cm;
    sums[wid][0] = tr;
    sums[wid][1] = ta;
  }
  __syncthreads();
  if (threadIdx.x % G == 0) {
    StreamFn::Group g;
    g.o = group_origin(f);
    const float rn = near_radius(f.radius, b);
    g.o.hi.w = f.compact ? -rn : rn;
    if (b.singular) g.o.hi.w = 1e15f;  // near every target
    if (k >= ns) g.o.hi.w = 3.0e38f;   // no sources
    g.o.lo = make_float4(b.k, 1.f - b.k, 1.00001f * sqrtf(fmaxf(mx[wid][0], mx[wid + 1][0])),
                         1.00001f * fmaxf(mx[wid][1], mx[wid + 1][1]));
    g.e1 = make_float4(b.e1[0], b.e1[1], b.e1[2], b.k1);
    g.e2 = make_float4(b.e2[0], b.e2[1], b.e2[2], b.k2);
    float rh, rl, ah, al;
    split2(sums[wid][0] + sums[wid + 1][0], rh, rl);
    split2(sums[wid][1] + sums[wid + 1][1], ah, al);
    g.s = make_float4(rh, rl, ah, al);
    org[t * (TILE / G) + threadIdx.x / G] = g;
  }
}

// The sphere SWE velocity's records and group origins (one CTA of TILE threads per tile).
template <int TILE>
__global__ void __launch_bounds__(TILE) stream_rel_prep_kernel(const double* x, const double* y, const double* z,
                                                               const double* qr, const double* qa, const double* area,
                                                               const int32_t* sorted, int64_t ns, double inv_a,
                                                               StreamRel::Rec* out, BveRel::Origin* org,
                                                               double scale_r, double scale_a) {
  const int64_t t = blockIdx.x;
  const int64_t k = t * TILE + threadIdx.x;
  const bool valid = k < ns;
  const int32_t j = valid ? sorted[k] : 0;
  double px = 0.0, py = 0.0, pz = 0.0, cj = 0.0;
  if (valid) {
    px = x[j] * inv_a;
    py = y[j] * inv_a;
    pz = z[j] * inv_a;
    cj = fma(px, px, fma(py, py, fma(pz, pz, -1.0)));
  }
  const SplitPoint sp = split_point(px, py, pz);
  const GroupFrame f = sphere_group_frame<TILE, BveRel::kGroup>(valid, sp, cj);
  StreamRel::Rec r;
  if (valid) {
    float hi[3], lo[3];
    group_offsets(f, sp, hi, lo);
    const float nc = __double2float_rn(-cj);
    const float sr = __double2float_rn(qr[j] * area[j] * scale_r), sa = __double2float_rn(qa[j] * area[j] * scale_a);
    r.a = make_float4(-hi[0], -hi[0], -hi[1], -hi[1]);
    r.b = make_float4(-hi[2], -hi[2], nc, nc);
    r.c = make_float4(sr, sr, sa, sa);
    r.d = make_float4(-lo[0], -lo[0], -lo[1], -lo[1]);
    r.e = make_float4(-lo[2], -lo[2], 0.f, 0.f);
  } else {
    r.a = r.b = r.c = r.d = r.e = make_float4(0.f, 0.f, 0.f, 0.f);  // inert: zero strength at the centroid
  }
  out[k] = r;
  if (threadIdx.x % BveRel::kGroup == 0) {
    BveRel::Origin o = group_origin(f);
    o.hi.w = f.compact ? -f.radius : f.radius;  // the sign marks a compact group
    org[t * (TILE / BveRel::kGroup) + threadIdx.x / BveRel::kGroup] = o;
  }
}

// ====================================================================== planar stream function
// SetStreamFunctionOnMesh, src/PlanarIncompressible.f90:470-505: psi_i = sum_{j != i}
// ln(|x_i - x_j|^2) omega_j A_j / (4 pi), on the planar group-relative layout (plane_rel.cuh;
// plane_rel_prep_kernel writes S_j = omega_j A_j / (4 pi) and each group's total S_g).
//
// The terms are centred per target and group: with a power of two 2^k near
// max(|t - o|^2, R^2) (k from the exponent split of ln_q2),
//   sum_j S_j ln u_j = sum_j S_j (ln u_j - k ln 2) + k ln 2 S_g,
// so the FP32 partials hold terms of size |S_j| (|ln(u_j 2^-k)| <= ~1.2 for a far group)
// instead of |S_j ln u_j|, and the second part is carried exactly: S_g k as a product of
// a (hi, lo) float pair and a small integer into its own compensated pair, times ln 2 in
// FP64 at the end.  ln_q2_shift applies the shift for free.  A far group (every target of the
// warp at |t - o| > 3R, so u_j > 0) needs no select; in a near group the self pair (u = 0,
// the lo parts cancel bit for bit) takes q = 1, whose centred term -k ln 2 cancels the
// target's own share of k ln 2 S_g.  Per target pair and source (far form): d (2 FADD2),
// |d|^2 (2), ln (ln_q2_shift: integer split, a table load per lane, 9 packed) and the
// accumulation (1 FFMA2).  Near partials are flushed every 16 sources, far ones per group.
template <int THREADS, int TPT, int TILE, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) plane_stream_rel_sweep_kernel(PlaneRelArgs<PlaneRel::Rec> a) {
  static_assert(TPT % 2 == 0, "targets come in pairs");
  constexpr int NP = TPT / 2;
  constexpr int G = PlaneRel::kGroup;
  constexpr int GPT = TILE / G;
  constexpr int FLN = 16;
  static_assert(G % FLN == 0, "flush interval must divide the group");
  using Rec = PlaneRel::Rec;
  __shared__ __align__(128) Rec stage[2][TILE];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ __align__(8) float2 ln_tab[32];

  const int64_t chunk = blockIdx.y;
  const ChunkTiles ct = chunk_tiles(a.n_tiles);

  PlaneRel::Pair pr[NP];
  float2 hs[NP], ls[NP], hk[NP], lk[NP];
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (THREADS * TPT);
  const int64_t count = a.nt - first < THREADS * TPT ? a.nt - first : THREADS * TPT;
  plane_load_pairs<NP>(a.tgt + first, count, pr);
#pragma unroll
  for (int p = 0; p < NP; ++p) hs[p] = ls[p] = hk[p] = lk[p] = make_float2(0.f, 0.f);
  constexpr float kTiny = 7.888609052210118e-31f;  // 2^-100: centring and near floor
  constexpr float kHuge = 1.2676506002282294e30f;  // 2^100

  ln_tab_load(ln_tab);
  pipe_init(bars);
  uint32_t g = 0;
  auto body = [&](const Rec* tl, const PlaneRel::Origin* og) {
#pragma unroll 1
    for (int g0 = 0; g0 < TILE; g0 += G) {
      const PlaneRel::Origin o = og[g0 / G];
      const Rec* gr = tl + g0;
      float2 tx[NP], ty[NP];
      float2 bias[NP];
      bool near = false;
      const float r2 = o.f.x * o.f.x;
      const float lim = fmaxf(PlaneRel::kNearFactor * PlaneRel::kNearFactor * r2, kTiny);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        tx[p] = rel1x2(pr[p].xh, pr[p].xl, o.o.x, o.o.z);
        ty[p] = rel1x2(pr[p].yh, pr[p].yl, o.o.y, o.o.w);
        const float2 n2 = __ffma2_rn(ty[p], ty[p], __fmul2_rn(tx[p], tx[p]));
        near |= !(n2.x > lim) | !(n2.y > lim);
        // the centring shift k: the exponent of max(|t - o|^2, R^2) clamped to [2^-100, 2^100]
        const float c0 = fminf(fmaxf(fmaxf(n2.x, r2), kTiny), kHuge);
        const float c1 = fminf(fmaxf(fmaxf(n2.y, r2), kTiny), kHuge);
        int mb;
        const int sh0 = exp_split(__float_as_int(c0), mb);
        const int sh1 = exp_split(__float_as_int(c1), mb);
        bias[p] = shift_bias(sh0, sh1);
        // k S_g into (hk, lk): S_hi k is exact as a product and its error term
        const float2 kf = make_float2(static_cast<float>(sh0), static_cast<float>(sh1));
        const float2 ph = __fmul2_rn(make_float2(o.f.y, o.f.y), kf);
        const float2 pe = __ffma2_rn(make_float2(o.f.y, o.f.y), kf, make_float2(-ph.x, -ph.y));
        comp_add(hk[p].x, lk[p].x, ph.x);
        comp_add(hk[p].y, lk[p].y, ph.y);
        lk[p] = __ffma2_rn(make_float2(o.f.z, o.f.z), kf, __fadd2_rn(lk[p], pe));
      }
      if (!__any_sync(0xffffffffu, near)) {
        // far group: d = t_hi - s_hi, u > 0
        float2 acc[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) acc[p] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int j = 0; j < G; ++j) {
          const float4 ra = gr[j].a, rb = gr[j].b;
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const float2 dx = __fadd2_rn(tx[p], lo2(ra));
            const float2 dy = __fadd2_rn(ty[p], hi2(ra));
            const float2 u = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
            acc[p] = __ffma2_rn(lo2(rb), ln_q2_shift(u, bias[p], ln_tab), acc[p]);
          }
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          comp_add(hs[p].x, ls[p].x, acc[p].x);
          comp_add(hs[p].y, ls[p].y, acc[p].y);
        }
      } else {
        // near group: d = (t_hi - s_hi) + (t_lo - s_lo)
        float2 txh[NP], tyh[NP], txl[NP], tyl[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          rel2x2(pr[p].xh, pr[p].xl, o.o.x, o.o.z, txh[p], txl[p]);
          rel2x2(pr[p].yh, pr[p].yl, o.o.y, o.o.w, tyh[p], tyl[p]);
        }
#pragma unroll 1
        for (int j0 = 0; j0 < G; j0 += FLN) {
          float2 acc[NP];
#pragma unroll
          for (int p = 0; p < NP; ++p) acc[p] = make_float2(0.f, 0.f);
          for (int j = j0; j < j0 + FLN; ++j) {
            const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
              const float2 dx = __fadd2_rn(__fadd2_rn(txh[p], lo2(ra)), __fadd2_rn(txl[p], hi2(rb)));
              const float2 dy = __fadd2_rn(__fadd2_rn(tyh[p], hi2(ra)), __fadd2_rn(tyl[p], lo2(rc)));
              const float2 u = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
              acc[p] = __ffma2_rn(lo2(rb), ln_q2_shift(stream_arg(u, u), bias[p], ln_tab), acc[p]);
            }
          }
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            comp_add(hs[p].x, ls[p].x, acc[p].x);
            comp_add(hs[p].y, ls[p].y, acc[p].y);
          }
        }
      }
    }
  };
  int64_t tile = ct.first;
  staged_sweep<Rec, TILE>(a.src, ct.first, ct.count, stage[0], stage[1], bars, g, a.status, [&](const Rec* tl) {
    body(tl, a.org + tile * GPT);
    tile += ct.step;
  }, ct.step);

  constexpr double kLn2 = 0.69314718055994530942;
#pragma unroll
  for (int p = 0; p < NP; ++p) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t il = first + bve_target<TPT>(2 * p + h);
      if (il < a.nt) {
        const double c = static_cast<double>(h ? hk[p].y : hk[p].x) + static_cast<double>(h ? lk[p].y : lk[p].x);
        a.partial[chunk * a.nt + il] =
            (static_cast<double>(h ? hs[p].y : hs[p].x) + static_cast<double>(h ? ls[p].y : ls[p].x)) + kLn2 * c;
      }
    }
  }
}

// ====================================================================== sphere SWE velocity
// SWESphereRHSIntegrals, src/SphereSWESolver.f90:299-372, velocity part, on the stream
// functions' layout (two strengths per record: S_r = -zeta_j A_j / (2 pi a^2) and
// S_p = div_j A_j / (2 pi a^2), written by stream_rel_prep_kernel).  With p = x/a, d = p_i - p_j
// and a^2 - x_i.x_j = (a^2/2) q, q = |d|^2 - c_i - c_j, the reference's
//   u -= (x_i x x_j) zeta_j A_j / (4 pi a^2 (a^2 - x_i.x_j)) + x_j a div_j A_j / (4 pi a^2 (a^2 - x_i.x_j))
// is u = Dr x p_i + Dp - p_i W with Dr = sum (S_r/q) d, Dp = sum (S_p/q) d, W = sum S_p/q
// (x_i x x_j = a^2 d x p_i and p_j = p_i - d).  The self pair (d = 0 exactly, in a near or a
// compact group) gets 1/q = 0.  Per target pair and source (far form): d (3 FADD2), |d|^2
// (3), q (1), the select and 2 MUFU, two weights (2), 7 accumulations.  Partials:
// [chunk][7][nt] (Dr, Dp, W).
template <int THREADS, int TPT, int TILE, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) sphere_swe_rel_sweep_kernel(SweepArgs<BveF32> a,
                                                                             const StreamRel::Rec* __restrict__ src,
                                                                             const BveRel::Origin* __restrict__ org) {
  static_assert(TPT % 2 == 0, "targets come in pairs");
  constexpr int NP = TPT / 2;
  constexpr int G = BveRel::kGroup;
  constexpr int GPT = TILE / G;
  constexpr int NC = 7;
  using Rec = StreamRel::Rec;
  __shared__ __align__(128) Rec stage[2][TILE];
  __shared__ __align__(8) uint64_t bars[2];

  const int64_t chunk = blockIdx.y;
  const ChunkTiles ct = chunk_tiles(a.n_tiles);

  BveX2::Pair pr[NP];
  float2 hs[NP][NC], ls[NP][NC];
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (THREADS * TPT);
  const int64_t count = a.nt - first < THREADS * TPT ? a.nt - first : THREADS * TPT;
  bve_load_pairs<NP>(a.p, a.ib + first, count, pr);
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int c = 0; c < NC; ++c) hs[p][c] = ls[p][c] = make_float2(0.f, 0.f);

  pipe_init(bars);
  uint32_t g = 0;
  int64_t tile = ct.first;
  staged_sweep<Rec, TILE>(src, ct.first, ct.count, stage[0], stage[1], bars, g, a.status, [&](const Rec* tl) {
    float2 ac[NP][NC];
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int c = 0; c < NC; ++c) ac[p][c] = make_float2(0.f, 0.f);
    auto terms = [&](float2 (&acc)[NC], float2 dx, float2 dy, float2 dz, float2 q, float2 u, float2 sr, float2 sp) {
      const float2 inv = make_float2(u.x != 0.f ? rcp_approx(q.x) : 0.f, u.y != 0.f ? rcp_approx(q.y) : 0.f);
      const float2 wr = __fmul2_rn(sr, inv), wp = __fmul2_rn(sp, inv);
      acc[0] = __ffma2_rn(wr, dx, acc[0]);
      acc[1] = __ffma2_rn(wr, dy, acc[1]);
      acc[2] = __ffma2_rn(wr, dz, acc[2]);
      acc[3] = __ffma2_rn(wp, dx, acc[3]);
      acc[4] = __ffma2_rn(wp, dy, acc[4]);
      acc[5] = __ffma2_rn(wp, dz, acc[5]);
      acc[6] = __fadd2_rn(wp, acc[6]);
    };
    const BveRel::Origin* og = org + tile * GPT;
#pragma unroll 1
    for (int g0 = 0; g0 < TILE; g0 += G) {
      const BveRel::Origin o = og[g0 / G];
      const Rec* gr = tl + g0;
      float2 tx[NP], ty[NP], tz[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        tx[p] = rel1x2(pr[p].xh, pr[p].xl, o.hi.x);
        ty[p] = rel1x2(pr[p].yh, pr[p].yl, o.hi.y);
        tz[p] = rel1x2(pr[p].zh, pr[p].zl, o.hi.z);
      }
      if (o.hi.w <= 0.f || !warp_near<NP>(tx, ty, tz, o.hi.w)) {  // -R: compact, taken as far
        // compact or far group: d = t_hi - s_hi
#pragma unroll 2
        for (int j = 0; j < G; ++j) {
          const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c;
          const float2 nsx = lo2(ra), nsy = hi2(ra), nsz = lo2(rb), ncj = hi2(rb), sr = lo2(rc), sp = hi2(rc);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const float2 dx = __fadd2_rn(tx[p], nsx);
            const float2 dy = __fadd2_rn(ty[p], nsy);
            const float2 dz = __fadd2_rn(tz[p], nsz);
            const float2 u = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
            terms(ac[p], dx, dy, dz, __fadd2_rn(u, __fadd2_rn(pr[p].nc, ncj)), u, sr, sp);
          }
        }
      } else {
        // near group: d = (t_hi - s_hi) + (t_lo - s_lo)
        float2 txh[NP], tyh[NP], tzh[NP], txl[NP], tyl[NP], tzl[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          rel2x2(pr[p].xh, pr[p].xl, o.hi.x, txh[p], txl[p]);
          rel2x2(pr[p].yh, pr[p].yl, o.hi.y, tyh[p], tyl[p]);
          rel2x2(pr[p].zh, pr[p].zl, o.hi.z, tzh[p], tzl[p]);
        }
        for (int j = 0; j < G; ++j) {
          const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c, rd = gr[j].d, re = gr[j].e;
          const float2 nsx = lo2(ra), nsy = hi2(ra), nsz = lo2(rb), ncj = hi2(rb), sr = lo2(rc), sp = hi2(rc);
          const float2 nlx = lo2(rd), nly = hi2(rd), nlz = lo2(re);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const float2 dx = __fadd2_rn(__fadd2_rn(txh[p], nsx), __fadd2_rn(txl[p], nlx));
            const float2 dy = __fadd2_rn(__fadd2_rn(tyh[p], nsy), __fadd2_rn(tyl[p], nly));
            const float2 dz = __fadd2_rn(__fadd2_rn(tzh[p], nsz), __fadd2_rn(tzl[p], nlz));
            const float2 u = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
            terms(ac[p], dx, dy, dz, __fadd2_rn(u, __fadd2_rn(pr[p].nc, ncj)), u, sr, sp);
          }
        }
      }
    }
    tile += ct.step;
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        comp_add(hs[p][c].x, ls[p][c].x, ac[p][c].x);
        comp_add(hs[p][c].y, ls[p][c].y, ac[p][c].y);
      }
  }, ct.step);

#pragma unroll
  for (int p = 0; p < NP; ++p) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t il = first + bve_target<TPT>(2 * p + h);
      if (il < a.nt) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
          a.partial[(chunk * NC + c) * a.nt + il] = static_cast<double>(h ? hs[p][c].y : hs[p][c].x) +
                                                    static_cast<double>(h ? ls[p][c].y : ls[p][c].x);
      }
    }
  }
}

// ====================================================================== beta-plane stream functions
// The beta plane's SetStreamFunctionsOnMesh, src/BetaPlane.f90:399-442, in FP32 for two
// targets at a time (the direct form of beta_stream_rel_sweep_kernel, csrc/beta_rel.cuh):
//   G = log(cosh(2 pi dy) - cos(2 pi dx)) / (4 pi),  psi += G zeta_j A_j  (j != i).
// cosh 2a - cos 2b = 2 (sinh^2 a + sin^2 b) = 2 4^(k-1) (sh'^2 + sn'^2) with a = pi |dy| =
// k ln 2 + r, b = pi dx and the 2^(k-1)-scaled sh', sn' of BetaF32, so
//   4 pi G = (2k - 1) ln 2 + ln(sh'^2 + sn'^2),
// no cancellation for close pairs and no overflow for far ones; the (2k - 1) ln 2 rides on the
// exponent of ln_q2_shift.  S = zeta A / (4 pi); the self pair (sh' = sn' = 0) is a zero term.
// Terms of both signs cancel to psi, so the caller flushes the FP32 partials often.
struct BetaStreamF32 {
  struct __align__(16) Rec {
    float4 a;  // x_hi, y_hi, x_lo, y_lo
    float4 b;  // S_rel, S_abs, 0, 0
  };
  using Tgt = BetaTgt;
  __device__ static __forceinline__ void interact2(const Tgt& t0, const Tgt& t1, const Rec& r, float (&a0)[2],
                                                   float (&a1)[2], const float2* tab) {
    float2 tt, dy;
    beta_deltas2(t0, t1, r.a, tt, dy);
    const float2 sn = sinpi2(tt, __fmul2_rn(tt, tt));
    const float2 a = __fmul2_rn(make_float2(3.1415927f, 3.1415927f), bits_abs(dy));
    float2 shr, chr, kb;
    sinh_cosh_reduced2(a, shr, chr, kb);
    const int k0 = static_cast<int>(__float_as_uint(kb.x) - 0x4b400000u);
    const int k1 = static_cast<int>(__float_as_uint(kb.y) - 0x4b400000u);
    const unsigned c0 = static_cast<unsigned>(k0 < 126 ? k0 : 126), c1 = static_cast<unsigned>(k1 < 126 ? k1 : 126);
    const float2 pk = make_float2(__uint_as_float(0x3f800000u - (c0 << 23)), __uint_as_float(0x3f800000u - (c1 << 23)));
    const float2 sc = __fadd2_rn(pk, pk);
    const float2 q = __fmul2_rn(pk, pk);
    const float2 shp = __ffma2_rn(__fadd2_rn(make_float2(1.0f, 1.0f), make_float2(-q.x, -q.y)), chr,
                                  __fmul2_rn(__fadd2_rn(make_float2(1.0f, 1.0f), q), shr));
    const float2 snp = __fmul2_rn(sn, sc);
    const float2 x = __ffma2_rn(shp, shp, __fmul2_rn(snp, snp));
    const float2 lg = ln_q2_shift(make_float2(x.x > 0.f ? x.x : 1.0f, x.y > 0.f ? x.y : 1.0f),
                                  shift_bias(1 - 2 * k0, 1 - 2 * k1), tab);
    const float2 g = make_float2(x.x > 0.f ? lg.x : 0.f, x.y > 0.f ? lg.y : 0.f);
    const float2 pr = __ffma2_rn(make_float2(r.b.x, r.b.x), g, make_float2(a0[0], a1[0]));
    const float2 pa = __ffma2_rn(make_float2(r.b.y, r.b.y), g, make_float2(a0[1], a1[1]));
    a0[0] = pr.x;
    a1[0] = pr.y;
    a0[1] = pa.x;
    a1[1] = pa.y;
  }
};

}  // namespace lpm
