// bve_rel.cuh -- the sphere-BVE FP32C sweep on spatially sorted sources in group-relative
// coordinates (10-11 packed FP32x2 operations per target pair and source).
//
// Sources are in Hilbert-curve order (sort.cu), so a group of kGroup consecutive sources
// covers one connected patch of the sphere.  Each source is stored relative to the centroid
// o of its group as a two-float offset (s_hi, s_lo) = rel2(p, o) (p - o to ~2^-48), and the
// group record holds o and the group radius R (the largest |p_j - o|).  The precision is
// chosen per warp and group:
//  - far (every target of the warp at |t - o| >= 3R): d = t_hi - s_hi with t_hi = fl(t - o),
//    one subtraction per component.  The roundings of t_hi and s_hi are <= 2^-24 |t - o|
//    and 2^-24 R, and |d| >= |t - o| - R >= 2R, so the relative error of d is at most
//    ~2^-23 whatever the point distribution;
//  - near (some target of the warp inside 3R, which includes the group's own sources and any
//    target at a source's position): the target forms (t_hi, t_lo) = rel2(t, o) with
//    exactly the operations of the sources, and d = (t_hi - s_hi) + (t_lo - s_lo) keeps ~48
//    bits; a self pair cancels bit for bit.
// A compact group (R <= a/2 and R <= 32 x its smallest spacing h, i.e. a patch of a
// quasi-uniform point set) takes one-subtraction differences for every target: its records use
// rel2_fast, the target's far-form operations, so a self pair still cancels bit for bit.
// For a target near such a group the roundings are an absolute 2^-24 R inside the near-field sum
// sum_j S_j / |d_j|^2, which grows only like ln(1/h) on a quasi-uniform set, so the velocity error
// scales with R, not R/h (1.0e-7 relative at icosahedral nest 8).  Groups that fail the test (clustered or sparse points) keep the
// near/far choice, whose error bound holds for any point distribution.
// Particle order along the mesh or the curve keeps a warp's targets close together, so a
// warp meets few near groups (at icosahedral nest 8 three in a thousand).
// A group whose sources all lie on the sphere to within |c_j| <= 2^-30 h^2 (h its smallest
// spacing; always the case once positions are renormalised) drops c_j: q is then
// fma(dz,dz, fma(dy,dy, fma(dx,dx, -c_i))), one operation less per pair.
// Then  q = |d|^2 - c_i - c_j,  w = S_j / q,  D += w d  with c = |p|^2 - 1 and
// S_j = -zeta_j A_j / (2 pi a) as in BveF32; u = D x p_i in FP64.
// A group whose warp is far (every target at |t - o| >= 3R, 1.5R or 1.25R if it is compact) takes the
// expanded form in a basis (o, e1, e2) of the group, e1 and e2 about orthonormal to o: with the
// source p_j = (1 + c) o + a e1 + b e2 and h = q/2 = 1 - p_i.p_j,
//   h = C - c gamma - a alpha - b beta,   alpha = p_i.e1, beta = p_i.e2, gamma = p_i.o, C = 1 - gamma,
//   sum_j S_j p_j / h = o W + e1 A + e2 B,  W = sum S_j (1 + c) / h, A = sum S_j a / h, B = sum S_j b / h,
// and since u = D x p_i takes no multiple of p_i = o + t, D += (t W - e1 A - e2 B) / 2 (once per
// group).  That is 6 packed FP32x2 operations, 2 MUFU and 3 LDS.128 (for two target pairs) per
// target pair and source, where the form with a Cartesian source offset (q/2 = (|t|^2 - c_i)/2 +
// B_j/2 - t.s_j and four sums) took 8, 2 and 4.  Any basis does: the records solve for (a, b, c) in
// the rounded one, alpha = t.e1 + o.e1 carries the group constant o.e1 (about 2^-25), and gamma =
// |o|^2 + k - ct, C = ct + k with ct = (|t|^2 - c_i)/2 and k = (1 - |o|^2)/2, so no term loses
// digits: C and the products are at most a few h at the 3R boundary, and q stays within a few ulps.
// A compact group with a target of the warp near it keeps d = t_hi - s_hi (10-11 operations; it contains the self pairs), any other near group the two-float form (17).
// Forming the targets' offsets, projections and the near test cost about 25 per pair and group.
// Targets keep their original order (only sources are sorted), so no scatter is needed.
#pragma once

#include "bve_x2.cuh"
#include "engine.cuh"
#include "ops.cuh"

namespace lpm {

struct BveRel {
  struct __align__(16) Rec {
    float4 a;  // -a, -a, -b, -b
    float4 b;  // -c, -c, W, W                  W = S_j (1 + c) / 2
    float4 c;  // A, A, B, B                    A = -S_j a / 2, B = -S_j b / 2
    float4 d;  // -sx_hi, -sy_hi, -sz_hi, S_j   (near forms)
    float4 e;  // -sx_lo, -sy_lo, -sz_lo, -c_j  (near forms)
  };
  struct __align__(16) Origin {
    float4 hi;  // o.x, o.y, o.z, R (the group radius about o; -R/2 for a compact group)
    float4 lo;  // 0, 0, 0, 1 if every c_j of the group is negligible
  };
  // The BVE sweep's group record: the origin and the far form's basis.
  struct __align__(16) Group {
    Origin o;   // lo.x = k = (1 - |o|^2) / 2, lo.y = |o|^2 + k
    float4 e1;  // e1, o.e1
    float4 e2;  // e2, o.e2
  };
  // A target as floats.  The prep kernel splits the FP64 positions once per sum: every CTA of a target
  // block needs them, and 20 FP64 instructions a target in each (2 lanes per clock and SM) took 3 % of
  // a sweep at icosahedral nest 5.
  struct __align__(16) Tgt {
    float4 h;  // p_hi, -c_i (BveF32::load_target)
    float4 l;  // p_lo, 0
  };
  // sources per origin: 128 measured 4.4 % faster than 64 for the BVE sweep (half the per-group
  // work per source) at the same accuracy; the stream-function sweeps share the layout
  static constexpr int kGroup = 128;
  static constexpr float kNearFactor = 3.0f;  // near: |t - o| < kNearFactor R
  static constexpr float kCompactRadius = 0.5f;  // compact: R <= kCompactRadius (unit sphere)
  // and R <= kCompactRatio h: refined meshes have R / h of 10-18 (median 12), sets without an even spacing
  // 44 and more (their closest pairs are rarely consecutive, so h alone does not show them)
  static constexpr float kCompactRatio = 32.0f;
  // the far form of a compact group starts at kCompactFar R, of a small one (R <= kCompactSmall; from
  // icosahedral nest 6 on) at kCompactFarSmall R
  static constexpr float kCompactFar = 1.5f, kCompactFarSmall = 1.25f, kCompactSmall = 0.2f;
};

// Offset of a hi/lo value from a float origin, rounded once: fl(p - o) to ~2^-24 relative
// (the far form needs no more).
__device__ __forceinline__ float2 rel1x2(float2 ph, float2 pl, float oh) {
  return __fadd2_rn(__fadd2_rn(ph, make_float2(-oh, -oh)), pl);
}

// The same offset as two floats from single roundings: r_hi = rel1 (the far form's target
// offset), r_lo the rounding of its last addition only.  Records of compact groups use it,
// so that a target at a source's position reproduces that source's r_hi bit for bit.
__device__ __forceinline__ void rel2_fast(float ph, float pl, float oh, float& rh, float& rl) {
  const float a = __fadd_rn(ph, -oh);
  rh = __fadd_rn(a, pl);
  rl = __fadd_rn(__fadd_rn(a, -rh), pl);
}

// Two-float offset (r_hi, r_lo) of a hi/lo value from a float origin, r_hi + r_lo = p - o to
// ~2^-48 relative: the TwoSum of (p_hi, -o) keeps the rounding of the leading difference
// (it is not exact when o is far from p), then the small terms are added and renormalised.
__device__ __forceinline__ void rel2(float ph, float pl, float oh, float& rh, float& rl) {
  const float s = __fadd_rn(ph, -oh);
  const float v = __fadd_rn(s, -ph);
  const float e = __fadd_rn(__fadd_rn(ph, -__fadd_rn(s, -v)), __fadd_rn(-oh, -v));
  const float r = __fadd_rn(e, pl);
  rh = __fadd_rn(s, r);
  rl = __fadd_rn(r, -__fadd_rn(rh, -s));
}

__device__ __forceinline__ void rel2x2(float2 ph, float2 pl, float oh, float2& rh, float2& rl) {
  const float2 noh = make_float2(-oh, -oh);
  const float2 s = __fadd2_rn(ph, noh);
  const float2 v = __fadd2_rn(s, make_float2(-ph.x, -ph.y));
  const float2 sv = __fadd2_rn(s, make_float2(-v.x, -v.y));
  const float2 e = __fadd2_rn(__fadd2_rn(ph, make_float2(-sv.x, -sv.y)), __fadd2_rn(noh, make_float2(-v.x, -v.y)));
  const float2 r = __fadd2_rn(e, pl);
  rh = __fadd2_rn(s, r);
  const float2 d = __fadd2_rn(rh, make_float2(-s.x, -s.y));
  rl = __fadd2_rn(r, make_float2(-d.x, -d.y));
}

// The place in its CTA's block of a thread's m-th target of TPT: a warp holds 32 TPT consecutive
// targets, which are close together in a mesh's order, so that it meets fewer near groups (by count, for
// 6 targets a thread, 17 % of the groups at icosahedral nest 5 and 4.8 % at nest 6, where 32-runs spread over the block
// would meet 24 % and 6.9 %).
template <int TPT>
__device__ __forceinline__ int bve_target(int m) {
  return static_cast<int>(threadIdx.x >> 5) * (32 * TPT) + m * 32 + static_cast<int>(threadIdx.x & 31u);
}

// Target pairs of a sweep: targets first + bve_target(2p + h), clamped to the `count` valid ones
// (duplicates are computed but not stored).
template <int NP>
__device__ __forceinline__ void bve_load_pairs(const BveF32::Params& prm, int64_t first, int64_t count,
                                               BveX2::Pair (&pr)[NP]) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    int64_t i0 = bve_target<2 * NP>(2 * p), i1 = bve_target<2 * NP>(2 * p + 1);
    if (i0 >= count) i0 = count - 1;
    if (i1 >= count) i1 = count - 1;
    const BveF32::Tgt t0 = BveF32::load_target(prm, first + i0);
    const BveF32::Tgt t1 = BveF32::load_target(prm, first + i1);
    pr[p].xh = make_float2(t0.xh, t1.xh);
    pr[p].yh = make_float2(t0.yh, t1.yh);
    pr[p].zh = make_float2(t0.zh, t1.zh);
    pr[p].xl = make_float2(t0.xl, t1.xl);
    pr[p].yl = make_float2(t0.yl, t1.yl);
    pr[p].zl = make_float2(t0.zl, t1.zl);
    pr[p].nc = make_float2(t0.nc, t1.nc);
  }
}

__device__ __forceinline__ BveRel::Tgt bve_split_target(const BveF32::Params& prm, int64_t i) {
  const BveF32::Tgt t = BveF32::load_target(prm, i);
  return BveRel::Tgt{make_float4(t.xh, t.yh, t.zh, t.nc), make_float4(t.xl, t.yl, t.zl, 0.f)};
}

// The same from targets split before (tgt[0] is the first target of the block).
template <int NP>
__device__ __forceinline__ void bve_load_pairs(const BveRel::Tgt* __restrict__ tgt, int64_t count,
                                               BveX2::Pair (&pr)[NP]) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    int64_t i0 = bve_target<2 * NP>(2 * p), i1 = bve_target<2 * NP>(2 * p + 1);
    if (i0 >= count) i0 = count - 1;
    if (i1 >= count) i1 = count - 1;
    const BveRel::Tgt t0 = tgt[i0], t1 = tgt[i1];
    pr[p].xh = make_float2(t0.h.x, t1.h.x);
    pr[p].yh = make_float2(t0.h.y, t1.h.y);
    pr[p].zh = make_float2(t0.h.z, t1.h.z);
    pr[p].xl = make_float2(t0.l.x, t1.l.x);
    pr[p].yl = make_float2(t0.l.y, t1.l.y);
    pr[p].zl = make_float2(t0.l.z, t1.l.z);
    pr[p].nc = make_float2(t0.h.w, t1.h.w);
  }
}

// Whether any target of the warp lies within kNearFactor R of a group origin (t = t_hi,
// the offsets from it); n2 returns |t|^2.  Every lane of the warp must call it.
template <int NP>
__device__ __forceinline__ bool warp_near(const float2 (&tx)[NP], const float2 (&ty)[NP], const float2 (&tz)[NP],
                                          float r, float2 (&n2)[NP]) {
  const float lim = (BveRel::kNearFactor * r) * (BveRel::kNearFactor * r);
  bool near = false;
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    n2[p] = __ffma2_rn(tz[p], tz[p], __ffma2_rn(ty[p], ty[p], __fmul2_rn(tx[p], tx[p])));
    near |= (n2[p].x < lim) | (n2[p].y < lim);
  }
  return __any_sync(0xffffffffu, near);
}

template <int NP>
__device__ __forceinline__ bool warp_near(const float2 (&tx)[NP], const float2 (&ty)[NP], const float2 (&tz)[NP],
                                          float r) {
  float2 n2[NP];
  return warp_near<NP>(tx, ty, tz, r, n2);
}

// One staged tile against NP target pairs: FP32 partials of D added into (ax, ay, az).  The far
// loop is unrolled UNROLL times (4 is 1 to 2 % faster than 2 for the 128 x 6 sweep, 2 keeps the 128 x 4 one from spilling more).
template <int NP, int TILE, int UNROLL = 4>
__device__ __forceinline__ void bve_rel_tile(const BveRel::Rec* __restrict__ tl, const BveRel::Group* __restrict__ og,
                                             const BveX2::Pair (&pr)[NP], float2 (&ax)[NP], float2 (&ay)[NP],
                                             float2 (&az)[NP]) {
  constexpr int G = BveRel::kGroup;
#pragma unroll 1
  for (int g0 = 0; g0 < TILE; g0 += G) {
    const BveRel::Group& gp = og[g0 / G];
    const BveRel::Origin o = gp.o;
    const BveRel::Rec* gr = tl + g0;
    float2 tx[NP], ty[NP], tz[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      tx[p] = rel1x2(pr[p].xh, pr[p].xl, o.hi.x);
      ty[p] = rel1x2(pr[p].yh, pr[p].yl, o.hi.y);
      tz[p] = rel1x2(pr[p].zh, pr[p].zl, o.hi.z);
    }
    float2 n2[NP];
    if (!warp_near<NP>(tx, ty, tz, fabsf(o.hi.w), n2)) {
      // far group: h = C - c gamma - a alpha - b beta, D += t W + e1 A + e2 B
      const float4 e1 = gp.e1, e2 = gp.e2;
      float2 al[NP], be[NP], ga[NP], cc[NP], ww[NP], va[NP], vb[NP];
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
        ww[p] = va[p] = vb[p] = make_float2(0.f, 0.f);
      }
#pragma unroll UNROLL
      for (int j = 0; j < G; ++j) {
        const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          float2 h = __ffma2_rn(ga[p], lo2(rb), cc[p]);
          h = __ffma2_rn(al[p], lo2(ra), h);
          h = __ffma2_rn(be[p], hi2(ra), h);
          const float2 inv = make_float2(rcp_approx(h.x), rcp_approx(h.y));
          ww[p] = __ffma2_rn(hi2(rb), inv, ww[p]);
          va[p] = __ffma2_rn(lo2(rc), inv, va[p]);
          vb[p] = __ffma2_rn(hi2(rc), inv, vb[p]);
        }
      }
#pragma unroll
      for (int p = 0; p < NP; ++p) {  // the offsets again, rather than held through the loop
        const float2 ux = rel1x2(pr[p].xh, pr[p].xl, o.hi.x);
        const float2 uy = rel1x2(pr[p].yh, pr[p].yl, o.hi.y);
        const float2 uz = rel1x2(pr[p].zh, pr[p].zl, o.hi.z);
        ax[p] = __ffma2_rn(make_float2(e1.x, e1.x), va[p], __ffma2_rn(make_float2(e2.x, e2.x), vb[p], __ffma2_rn(ux, ww[p], ax[p])));
        ay[p] = __ffma2_rn(make_float2(e1.y, e1.y), va[p], __ffma2_rn(make_float2(e2.y, e2.y), vb[p], __ffma2_rn(uy, ww[p], ay[p])));
        az[p] = __ffma2_rn(make_float2(e1.z, e1.z), va[p], __ffma2_rn(make_float2(e2.z, e2.z), vb[p], __ffma2_rn(uz, ww[p], az[p])));
      }
    } else if (o.hi.w < 0.f) {
      // compact group near the warp (it may hold the targets themselves): d = t_hi - s_hi with
      // the records' rel2_fast offsets, so a self pair cancels bit for bit
      if (o.lo.w != 0.f) {
        // every source of the group on the sphere: c_j dropped
        for (int j = 0; j < G; ++j) {
          const float4 rd = gr[j].d;
          const float2 nsx = make_float2(rd.x, rd.x), nsy = make_float2(rd.y, rd.y), nsz = make_float2(rd.z, rd.z),
                       s2 = make_float2(rd.w, rd.w);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const float2 dx = __fadd2_rn(tx[p], nsx);
            const float2 dy = __fadd2_rn(ty[p], nsy);
            const float2 dz = __fadd2_rn(tz[p], nsz);
            float2 q = __ffma2_rn(dx, dx, pr[p].nc);
            q = __ffma2_rn(dy, dy, q);
            q = __ffma2_rn(dz, dz, q);
            const float2 inv = make_float2(rcp_approx(q.x), rcp_approx(q.y));
            const float2 wgt = __fmul2_rn(s2, inv);
            ax[p] = __ffma2_rn(wgt, dx, ax[p]);
            ay[p] = __ffma2_rn(wgt, dy, ay[p]);
            az[p] = __ffma2_rn(wgt, dz, az[p]);
          }
        }
      } else {
        for (int j = 0; j < G; ++j) {
          const float4 rd = gr[j].d;
          const float ncj1 = gr[j].e.w;
          const float2 nsx = make_float2(rd.x, rd.x), nsy = make_float2(rd.y, rd.y), nsz = make_float2(rd.z, rd.z),
                       s2 = make_float2(rd.w, rd.w), ncj = make_float2(ncj1, ncj1);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const float2 dx = __fadd2_rn(tx[p], nsx);
            const float2 dy = __fadd2_rn(ty[p], nsy);
            const float2 dz = __fadd2_rn(tz[p], nsz);
            float2 q = __fadd2_rn(pr[p].nc, ncj);
            q = __ffma2_rn(dx, dx, q);
            q = __ffma2_rn(dy, dy, q);
            q = __ffma2_rn(dz, dz, q);
            const float2 inv = make_float2(rcp_approx(q.x), rcp_approx(q.y));
            const float2 wgt = __fmul2_rn(s2, inv);
            ax[p] = __ffma2_rn(wgt, dx, ax[p]);
            ay[p] = __ffma2_rn(wgt, dy, ay[p]);
            az[p] = __ffma2_rn(wgt, dz, az[p]);
          }
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
        const float4 rd = gr[j].d, re = gr[j].e;
        const float2 nsx = make_float2(rd.x, rd.x), nsy = make_float2(rd.y, rd.y), nsz = make_float2(rd.z, rd.z),
                     s2 = make_float2(rd.w, rd.w);
        const float2 nlx = make_float2(re.x, re.x), nly = make_float2(re.y, re.y), nlz = make_float2(re.z, re.z);
        const float2 ncj = make_float2(re.w, re.w);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const float2 dx = __fadd2_rn(__fadd2_rn(txh[p], nsx), __fadd2_rn(txl[p], nlx));
          const float2 dy = __fadd2_rn(__fadd2_rn(tyh[p], nsy), __fadd2_rn(tyl[p], nly));
          const float2 dz = __fadd2_rn(__fadd2_rn(tzh[p], nsz), __fadd2_rn(tzl[p], nlz));
          float2 q = __fadd2_rn(pr[p].nc, ncj);
          q = __ffma2_rn(dx, dx, q);
          q = __ffma2_rn(dy, dy, q);
          q = __ffma2_rn(dz, dz, q);
          const float2 inv = make_float2(rcp_approx(q.x), rcp_approx(q.y));
          const float2 wgt = __fmul2_rn(s2, inv);
          ax[p] = __ffma2_rn(wgt, dx, ax[p]);
          ay[p] = __ffma2_rn(wgt, dy, ay[p]);
          az[p] = __ffma2_rn(wgt, dz, az[p]);
        }
      }
    }
  }
}

// Adds the FP32 tile partials into the compensated (hi, lo) accumulators.
template <int NP>
__device__ __forceinline__ void bve_merge_pairs(const float2 (&ax)[NP], const float2 (&ay)[NP], const float2 (&az)[NP],
                                                float2 (&hx)[NP], float2 (&hy)[NP], float2 (&hz)[NP],
                                                float2 (&lx)[NP], float2 (&ly)[NP], float2 (&lz)[NP]) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    comp_add(hx[p].x, lx[p].x, ax[p].x);
    comp_add(hx[p].y, lx[p].y, ax[p].y);
    comp_add(hy[p].x, ly[p].x, ay[p].x);
    comp_add(hy[p].y, ly[p].y, ay[p].y);
    comp_add(hz[p].x, lz[p].x, az[p].x);
    comp_add(hz[p].y, lz[p].y, az[p].y);
  }
}

template <int THREADS, int TPT, int TILE, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) bve_rel_sweep_kernel(SweepArgs<BveF32> a,
                                                                      const BveRel::Group* __restrict__ org,
                                                                      const BveRel::Tgt* __restrict__ tgt) {
  static_assert(TPT % 2 == 0, "targets come in pairs");
  static_assert(TILE % BveRel::kGroup == 0, "whole origin groups per tile");
  constexpr int NP = TPT / 2;
  constexpr int GPT = TILE / BveRel::kGroup;
  using Rec = BveRel::Rec;
  __shared__ TilePipe<Rec, TILE, 2> pipe;

  const int64_t chunk = blockIdx.y;
  const ChunkTiles ct = chunk_tiles(a.n_tiles);

  BveX2::Pair pr[NP];
  float2 hx[NP], hy[NP], hz[NP], lx[NP], ly[NP], lz[NP];
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (THREADS * TPT);
  const int64_t count = a.nt - first < THREADS * TPT ? a.nt - first : THREADS * TPT;
  bve_load_pairs<NP>(tgt + first, count, pr);
#pragma unroll
  for (int p = 0; p < NP; ++p) hx[p] = hy[p] = hz[p] = lx[p] = ly[p] = lz[p] = make_float2(0.f, 0.f);

  uint32_t g = 0;
  int64_t tile = ct.first;
  const Rec* src = reinterpret_cast<const Rec*>(a.src);
  auto body = [&](const Rec* tl) {
    float2 ax[NP], ay[NP], az[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) ax[p] = ay[p] = az[p] = make_float2(0.f, 0.f);
    bve_rel_tile<NP, TILE, (NP >= 3 ? 4 : 2)>(tl, org + tile * GPT, pr, ax, ay, az);
    tile += ct.step;
    bve_merge_pairs<NP>(ax, ay, az, hx, hy, hz, lx, ly, lz);
  };
  tile_pipe_init(pipe);
  warp_sweep_tiles(src, [ct](int64_t k) { return ct.first + k * ct.step; }, ct.count, pipe, g, a.status, a.wait,
                   static_cast<const Rec*>(nullptr), body);

#pragma unroll
  for (int p = 0; p < NP; ++p) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t il = first + bve_target<TPT>(2 * p + h);
      if (il < a.nt) {
        const float vx = h ? hx[p].y : hx[p].x, ex = h ? lx[p].y : lx[p].x;
        const float vy = h ? hy[p].y : hy[p].x, ey = h ? ly[p].y : ly[p].x;
        const float vz = h ? hz[p].y : hz[p].x, ez = h ? lz[p].y : lz[p].x;
        a.partial[(chunk * 3 + 0) * a.nt + il] = static_cast<double>(vx) + static_cast<double>(ex);
        a.partial[(chunk * 3 + 1) * a.nt + il] = static_cast<double>(vy) + static_cast<double>(ey);
        a.partial[(chunk * 3 + 2) * a.nt + il] = static_cast<double>(vz) + static_cast<double>(ez);
      }
    }
  }
}

// A unit-scaled position as hi/lo floats.
struct SplitPoint {
  float h[3], l[3];
};

__device__ __forceinline__ SplitPoint split_point(double px, double py, double pz) {
  SplitPoint s;
  split2(px, s.h[0], s.l[0]);
  split2(py, s.h[1], s.l[1]);
  split2(pz, s.h[2], s.l[2]);
  return s;
}

// The frame of the thread's group of G sources within a tile of TILE (one CTA of TILE
// threads, every thread one source): the origin o (the centroid in FP32: any point near it
// does, and one without a low part saves the targets' offsets an operation), the radius R about o,
// whether the group is compact (R <= a/2 and R <= 32 x the smallest distance h between
// consecutive sources) and whether every |c_j| <= 2^-30 h^2 (c_j negligible in q), c_j =
// |p|^2 - 1.  All of it in FP32 from the hi/lo positions (the offsets are exact to 2^-24): the FP64
// pipe would bound this kernel.  R is widened by its rounding.
struct GroupFrame {
  float o[3];
  float radius;
  bool compact, on_sphere;
};

template <int TILE, int G>
__device__ __forceinline__ GroupFrame sphere_group_frame(bool valid, const SplitPoint& sp, double cj,
                                                         float compact_radius = BveRel::kCompactRadius) {
  static_assert(G % 32 == 0 && TILE % G == 0, "whole warps per group");
  constexpr int NW = TILE / 32, WPG = G / 32;
  __shared__ float part[NW][4];
  __shared__ float last[NW][3];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w0 = wid / WPG * WPG;  // the group's first warp
  float v[4] = {valid ? sp.h[0] : 0.f, valid ? sp.h[1] : 0.f, valid ? sp.h[2] : 0.f, valid ? 1.f : 0.f};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
  if (WPG > 1) {
    if (lane == 0)
#pragma unroll
      for (int c = 0; c < 4; ++c) part[wid][c] = v[c];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      v[c] = 0.f;
#pragma unroll
      for (int w = 0; w < WPG; ++w) v[c] += part[w0 + w][c];
    }
    __syncthreads();
  }
  GroupFrame f;
  const float inv = v[3] > 0.f ? 1.f / v[3] : 0.f;
  f.o[0] = v[0] * inv;
  f.o[1] = v[1] * inv;
  f.o[2] = v[2] * inv;
  float d[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) d[c] = __fadd_rn(__fadd_rn(sp.h[c], -f.o[c]), sp.l[c]);
  float e[3];  // from the source before, in the group
#pragma unroll
  for (int c = 0; c < 3; ++c) e[c] = __shfl_up_sync(0xffffffffu, d[c], 1);
  if (WPG > 1) {
    if (lane == 31)
#pragma unroll
      for (int c = 0; c < 3; ++c) last[wid][c] = d[c];
    __syncthreads();
    if (lane == 0 && wid > w0)
#pragma unroll
      for (int c = 0; c < 3; ++c) e[c] = last[wid - 1][c];
  }
  const bool has_prev = valid && (lane > 0 || wid > w0);
  float rad = valid ? d[0] * d[0] + d[1] * d[1] + d[2] * d[2] : 0.f;
  if (!(rad == rad)) rad = __int_as_float(0x7f800000);  // a NaN source: an infinite radius
  const float ex = d[0] - e[0], ey = d[1] - e[1], ez = d[2] - e[2];
  float spc = has_prev ? ex * ex + ey * ey + ez * ez : 3.0e38f;
  float cm = valid ? fabsf(__double2float_rn(cj)) : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    rad = fmaxf(rad, __shfl_xor_sync(0xffffffffu, rad, o));
    spc = fminf(spc, __shfl_xor_sync(0xffffffffu, spc, o));
    cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
  }
  if (WPG > 1) {
    if (lane == 0) {
      part[wid][0] = rad;
      part[wid][1] = spc;
      part[wid][2] = cm;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < WPG; ++w) {
      rad = fmaxf(rad, part[w0 + w][0]);
      spc = fminf(spc, part[w0 + w][1]);
      cm = fmaxf(cm, part[w0 + w][2]);
    }
  }
  f.radius = sqrtf(rad) * 1.000001f;
  f.compact = f.radius <= compact_radius && f.radius <= BveRel::kCompactRatio * sqrtf(spc);
  // on the sphere: dropping every c_j moves q by <= 2^-30 h^2 relative to the smallest |d|^2
  // (a group of one source has no distance to compare with)
  f.on_sphere = spc < 3.0e38f && cm <= 9.313225746154785e-10f * spc;
  return f;
}

// Offsets of a unit-scaled position from its group's origin: rel2_fast for a compact
// group (the target's far-form operations), rel2 otherwise.
__device__ __forceinline__ void group_offsets(const GroupFrame& f, const SplitPoint& sp, float (&hi)[3],
                                              float (&lo)[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (f.compact) {
      rel2_fast(sp.h[c], sp.l[c], f.o[c], hi[c], lo[c]);
    } else {
      rel2(sp.h[c], sp.l[c], f.o[c], hi[c], lo[c]);
    }
  }
}

// The group record: origin, radius (0 for a compact group; the sweeps that have a near form for compact
// groups put its near radius there, negative), on-sphere flag.
__device__ __forceinline__ BveRel::Origin group_origin(const GroupFrame& f) {
  BveRel::Origin o;
  o.hi = make_float4(f.o[0], f.o[1], f.o[2], f.compact ? 0.f : f.radius);
  o.lo = make_float4(0.f, 0.f, 0.f, f.on_sphere ? 1.f : 0.f);
  return o;
}

// h . e + l . e + c as a pair hi + lo (about 2^-46 relative to the terms): products and sums with
// their FP32 errors carried (T. Ogita, S. M. Rump and S. Oishi, Accurate sum and dot product, SIAM J.
// Sci. Comput. 26, 2005).
__device__ __forceinline__ float2 dot_pair(const float (&h)[3], const float (&l)[3], const float (&e)[3], float c) {
  float s = c, err = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float p = __fmul_rn(h[k], e[k]);
    float t, q;
    two_sum(s, p, t, q);
    s = t;
    err += q + fmaf(h[k], e[k], -p) + l[k] * e[k];
  }
  return make_float2(s, err);
}

// The far form's basis of a group: e1 and e2 unit vectors about orthogonal to o and to each other
// (FP32), and what solving for a source's coefficients in it takes.  `singular`: o is too close to
// the centre of the sphere to be a basis vector (the group then never takes the far form).
struct GroupBasis {
  float e1[3], e2[3];
  float k1, k2;         // o.e1, o.e2
  float g11, g12, g22;  // e1.e1 - 1, e1.e2, e2.e2 - 1
  float inv_o2;         // 1 / |o|^2
  float k;              // (1 - |o|^2) / 2
  bool singular;
};

__device__ __forceinline__ GroupBasis group_basis(const GroupFrame& f) {
  GroupBasis b;
  const float zero[3] = {0.f, 0.f, 0.f};
  // e1 across o and the axis it is least along, e2 across both
  const float x = f.o[0], y = f.o[1], z = f.o[2];
  float ux, uy, uz;
  if (fabsf(x) <= fabsf(y) && fabsf(x) <= fabsf(z)) {
    ux = 0.f, uy = -z, uz = y;
  } else if (fabsf(y) <= fabsf(z)) {
    ux = z, uy = 0.f, uz = -x;
  } else {
    ux = -y, uy = x, uz = 0.f;
  }
  const float ru = rsqrtf(fmaxf(ux * ux + uy * uy + uz * uz, 1e-30f));
  ux *= ru, uy *= ru, uz *= ru;
  float vx = y * uz - z * uy, vy = z * ux - x * uz, vz = x * uy - y * ux;
  const float rv = rsqrtf(fmaxf(vx * vx + vy * vy + vz * vz, 1e-30f));
  vx *= rv, vy *= rv, vz *= rv;
  b.e1[0] = ux, b.e1[1] = uy, b.e1[2] = uz;
  b.e2[0] = vx, b.e2[1] = vy, b.e2[2] = vz;
  auto dot = [&](const float (&p)[3], const float (&q)[3], float c) {
    const float2 d = dot_pair(p, zero, q, c);
    return d.x + d.y;
  };
  b.k1 = dot(f.o, b.e1, 0.f);
  b.k2 = dot(f.o, b.e2, 0.f);
  b.g11 = dot(b.e1, b.e1, -1.f);
  b.g12 = dot(b.e1, b.e2, 0.f);
  b.g22 = dot(b.e2, b.e2, -1.f);
  b.k = -0.5f * dot(f.o, f.o, -1.f);
  const float o2 = x * x + y * y + z * z;
  b.singular = !(o2 >= 1e-3f);
  b.inv_o2 = b.singular ? 0.f : 1.f / o2;
  return b;
}

// The radius of the near test: the group's, and at least sqrt(|k|) / 2.  C = ct + k and the coordinates c (about
// 2k) are rounded at the size of k = (1 - |o|^2) / 2, which is R^2 / 4 for a patch of the sphere but up to 2^-24 for a
// tight cluster, whose origin is off the sphere by its own rounding (and more for points off the sphere); at
// |t| >= 1.5 sqrt(|k|) h is no smaller than |k|, so those roundings stay a few ulps of it.
__device__ __forceinline__ float near_radius(float r, const GroupBasis& b) { return fmaxf(r, 0.5f * sqrtf(fabsf(b.k))); }

// A source's coordinates in its group's basis, s_j = a e1 + b e2 + c o for its offset (hi, lo): the
// projections less their first-order coupling (2^-24 of them; the second order is 2^-48).
__device__ __forceinline__ void basis_coords(const GroupBasis& b, const GroupFrame& f, const float (&hi)[3],
                                             const float (&lo)[3], float& af, float& bf, float& cf) {
  const float2 a0 = dot_pair(hi, lo, b.e1, 0.f), b0 = dot_pair(hi, lo, b.e2, 0.f), so = dot_pair(hi, lo, f.o, 0.f);
  const float c0 = so.x * b.inv_o2;
  af = a0.x + (a0.y - (a0.x * b.g11 + b0.x * b.g12 + c0 * b.k1));
  bf = b0.x + (b0.y - (a0.x * b.g12 + b0.x * b.g22 + c0 * b.k2));
  cf = (so.x + (so.y - (af * b.k1 + bf * b.k2))) * b.inv_o2;
}

// Records and groups of one tile of TILE sources (one CTA of TILE threads; every thread
// one record).  `j` is the thread's particle (meaningful only if `valid`), `inv_a` and
// `s_scale` the tile's sphere scale.  Every record is written as the offset of p_j from its
// group's origin -- the operations the sweep uses for targets -- and in the group's basis.
template <int TILE>
__device__ __forceinline__ void bve_rel_prep_tile(const double* x, const double* y, const double* z,
                                                  const double* zeta, const double* area, bool valid, int32_t j,
                                                  double inv_a, double s_scale, BveRel::Rec* out,
                                                  BveRel::Group* og) {
  double px = 0.0, py = 0.0, pz = 0.0, cj = 0.0;
  if (valid) {
    px = x[j] * inv_a;
    py = y[j] * inv_a;
    pz = z[j] * inv_a;
    cj = fma(px, px, fma(py, py, fma(pz, pz, -1.0)));
  }
  const SplitPoint sp = split_point(px, py, pz);
  const GroupFrame f = sphere_group_frame<TILE, BveRel::kGroup>(valid, sp, cj);
  const GroupBasis b = group_basis(f);
  BveRel::Rec r;
  if (valid) {
    float hi[3], lo[3];
    group_offsets(f, sp, hi, lo);
    const float nc = __double2float_rn(-cj);
    float s, sl;
    split2(zeta[j] * area[j] * s_scale, s, sl);
    float af, bf, cf;
    basis_coords(b, f, hi, lo, af, bf, cf);
    // the strength times 1 + c, a and b, each rounded once
    auto times = [&](float v) {
      const float p = s * v;
      return p + fmaf(sl, v, fmaf(s, v, -p));
    };
    const float w = 0.5f * (s + fmaf(s, cf, sl)), aw = -0.5f * times(af), bw = -0.5f * times(bf);
    r.a = make_float4(-af, -af, -bf, -bf);
    r.b = make_float4(-cf, -cf, w, w);
    r.c = make_float4(aw, aw, bw, bw);
    r.d = make_float4(-hi[0], -hi[1], -hi[2], s);
    r.e = make_float4(-lo[0], -lo[1], -lo[2], nc);
  } else {
    // inert: at the origin with zero strength and zero -c (weight 0 times a finite value;
    // q > 0 through the target's 2^-100 offset when the target sits on o)
    r.a = r.b = r.c = r.d = r.e = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  *out = r;
  if (threadIdx.x % BveRel::kGroup == 0) {
    BveRel::Group g;
    g.o = group_origin(f);
    // The sign marks a compact group, whose far form starts at kCompactFar R, or kCompactFarSmall R if it is
    // small: there |h| >= R^2 / 8 (R^2 / 32), and the expanded form's roundings are at most about 20 (60) x 2^-24
    // of it, at the nearest of the group's sources alone, while the difference form near a compact group
    // carries an absolute 2^-24 R in d for all of them.  Relative L2 error of the velocity against FP64 over
    // all targets, two fields, with the far form from 3 R, 1.5 R and 1.25 R on: icosahedral nest 6 12.0e-8, 11.1e-8,
    // 10.9e-8; nest 7 6.26e-8, 5.86e-8, 5.77e-8; nest 8 3.69e-8, 3.51e-8, 3.46e-8; at nest 4, whose groups
    // are not small, 17.3e-8 and 17.5e-8.  1.5 R is 3 % faster than 3 R at nests 5 and 6, 1.25 R no faster.
    const float from = f.radius <= BveRel::kCompactSmall ? BveRel::kCompactFarSmall : BveRel::kCompactFar;
    g.o.hi.w = f.compact ? -near_radius(from / BveRel::kNearFactor * f.radius, b) : near_radius(f.radius, b);
    if (b.singular) g.o.hi.w = 1e15f;             // near every target
    g.o.lo.x = b.k;
    g.o.lo.y = 1.f - b.k;  // |o|^2 + k
    g.e1 = make_float4(b.e1[0], b.e1[1], b.e1[2], b.k1);
    g.e2 = make_float4(b.e2[0], b.e2[1], b.e2[2], b.k2);
    og[threadIdx.x / BveRel::kGroup] = g;
  }
}

// Tile-relative records of the Hilbert-sorted source list `sorted` (ns entries, records
// ns..npad-1 inert) and the groups (CTA t < n_tiles: tile t, TILE threads), then the nt targets from ib on.
template <int TILE>
__global__ void __launch_bounds__(TILE) bve_rel_prep_kernel(const double* x, const double* y, const double* z,
                                                            const double* zeta, const double* area,
                                                            const int32_t* sorted, int64_t ns, int64_t n_tiles,
                                                            double inv_a, double s_scale, int64_t ib, int64_t nt,
                                                            BveRel::Rec* out, BveRel::Group* org, BveRel::Tgt* tgt) {
  const int64_t t = blockIdx.x;
  if (t >= n_tiles) {
    const int64_t il = (t - n_tiles) * TILE + threadIdx.x;
    if (il < nt) tgt[il] = bve_split_target(BveF32::Params{x, y, z, inv_a}, ib + il);
    return;
  }
  const int64_t k = t * TILE + threadIdx.x;
  const bool valid = k < ns;
  const int32_t j = valid ? sorted[k] : 0;
  bve_rel_prep_tile<TILE>(x, y, z, zeta, area, valid, j, inv_a, s_scale, out + k,
                          org + t * (TILE / BveRel::kGroup));
}

}  // namespace lpm
