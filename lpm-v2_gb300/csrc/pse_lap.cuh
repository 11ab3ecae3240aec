// pse_lap.cuh -- the FP32C PSE Laplacians: K8 of the great-circle distance and the Gaussian of the
// chord on the sphere, K8 and the Gaussian of the distance in the plane.
//
// Reference, src/PSEDirectSum.f90 (kernels :611-640):
//   PSESphereLaplacianAtParticles (:502-535), PSEPlaneLaplacianAtParticles (:467-500)
//   L_i = eps^-4 sum_j (f_j - f_i) A_j K(r),  r = distance / eps
// Both kernels carry exp(-r^2); at r^2 >= 49 they are below 1e-17 of their peak, far below FP32 --
// and FP64 -- resolution of any sum they enter, so a warp skips a group of 32 sources that lies
// beyond that from its targets.  The result equals the all-pairs sum to FP32 rounding; the skipped
// pairs are counted as done.
//
// Layout: sources and targets in curve order.  A group of kGroup sources has an origin o near its
// centroid (in the plane with a low part: far from the coordinates' origin a float alone would make every
// group wide, and at a shift of 1e8 a sum at quad nest 7 took 3.9 ms instead of 0.5); positions (unit directions for
// the great circle, x / a for the chord, x in the plane) are held relative to it.  A pair needs only the exponent's base-2 argument y = -r^2 log2 e:
//   v = |t - s|^2 from the offsets (3 + 3 packed FP32x2 operations; 2 + 2 in the plane),
//   y = v (q0 + q1 v + ...)     for the great circle, theta^2 = 4 asin^2(sqrt(v) / 2) as a polynomial
//                               interpolated at Chebyshev nodes (within 5e-9; v <= 0.2 or 1.3),
//   y = q0 v                    for chords (the factor is in the target's and record's scale),
//   E = 2^y (2 MUFU, which run at twice the reciprocal's rate), K8 = E (p0 + p1 y + p2 y^2 + p3 y^3),
//   (f_j - f_i) A_j = A_j F_j - A_j F_i with F the field less a group constant: one FMA forms it from
//   floats, and one accumulates its product with K (near the group, where the difference is smaller than F:
//   F_j - F_i from float pairs in three operations, times A_j K).
// The kernel is smooth at r = 0, so that no pair needs more than the offsets' 2^-24: a group that is
// small against eps (R <= 2 eps) takes one form for every target, self pairs included (f_j - f_i =
// 0).  A wider group (particles far apart against eps, or a set far from its coordinates' origin)
// takes two-float offsets.
//
// Targets are split into floats once per call (PseLap::Tgt, by the prep kernel): a sweep has several
// CTAs per target block, and taking the FP64 positions apart in each of them (about 60 FP64
// instructions a target with the unit direction, at 2 lanes per clock and SM) cost a quarter of it.
#pragma once

#include "bve_rel.cuh"
#include "ops.cuh"
#include "plane_rel.cuh"
#include "pse_rel.cuh"

namespace lpm {

// How y comes from the squared offset distance: proportional, or by the angle's polynomial.
enum PseLapAngle { kLapChord = 0, kLapNear = 1, kLapFar = 2 };
constexpr double kLapNearMax = 0.43, kLapFarMax = 1.13;  // the largest cutoff chord of the polynomials

struct PseLap {
  struct __align__(16) Rec {
    float4 a;  // -sx, -sx, -sy, -sy
    float4 b;  // -sz, -sz, A, A
    float4 c;  // A F, A F, and F as a float pair
    float4 d;  // the offset's low parts -sx, -sy, -sz (wide groups), 0
  };
  struct __align__(16) Group {
    float4 o;  // origin, R
    float4 f;  // the field's group constant, 1 for a wide group, the origin's low part (plane)
  };
  struct __align__(16) Tgt {
    float4 h;  // position, field: high parts
    float4 l;  // low parts
  };
  static constexpr int kGroup = 32;  // the cutoff's granularity
  static constexpr float kWide = 2.0f / 7.0f;  // R beyond this share of the cutoff distance 7 eps
};

struct PseLapArgs {
  const PseLap::Rec* src;
  const PseLap::Group* grp;
  const PseLap::Tgt* tgt;
  const float4* tball;  // per source tile: centre (hi parts) and radius
  float c_cut;          // distance at which r^2 = 49
  float q[7];           // y's polynomial
  int64_t n_tiles, ib, nt;
  // targets in curve order: position k of the sweep is particle tperm[k] (nullptr: ib + k);
  // partial sums are stored at the particle's own place, (tperm[k] - ib)
  const int32_t* tperm;
  double* partial;  // [chunk][nt]
  int* status;
  WaitCfg wait;  // limits of the bounded waits (the test hook may shorten them and skip a tile)
};

template <int ANG>
__device__ __forceinline__ float2 lap_exponent(float2 v, const float (&q)[7]) {
  constexpr int D = ANG == kLapChord ? 0 : (ANG == kLapNear ? 3 : 6);
  float2 p = make_float2(q[D], q[D]);
#pragma unroll
  for (int k = D - 1; k >= 0; --k) p = __ffma2_rn(p, v, make_float2(q[k], q[k]));
  return __fmul2_rn(v, p);
}

// The kernel (times pi; the Gaussian without its 4) at y = -r^2 log2 e.
template <bool K8>
__device__ __forceinline__ float2 lap_kernel(float2 y) {
  const float2 e = make_float2(ex2_approx(y.x), ex2_approx(y.y));
  if (!K8) return e;
  // 40 - 40 r^2 + 10 r^4 - (2/3) r^6 with r^2 = -y ln 2
  float2 p = __ffma2_rn(make_float2(0.22201644f, 0.22201644f), y, make_float2(4.8045301f, 4.8045301f));
  p = __ffma2_rn(p, y, make_float2(27.725887f, 27.725887f));
  p = __ffma2_rn(p, y, make_float2(40.0f, 40.0f));
  return __fmul2_rn(e, p);
}

// Target pairs [P0, P1) of a warp against one group.  CLOSE: F_j - F_i from the float pairs, for targets
// so near the group that the difference is smaller than its terms; both pairs come from the same operations, so
// a particle's own pair is exactly zero (K is largest there, and a residue of 2^-48 f would be all that a set
// without neighbours in reach has).
template <bool SPHERE, bool K8, int ANG, bool CLOSE, int P0, int P1, int NP>
__device__ __forceinline__ void lap_group(const PseLap::Rec* __restrict__ gr, const float (&q)[7],
                                          const float2 (&tx)[NP], const float2 (&ty)[NP], const float2 (&tz)[NP],
                                          const float2 (&nf)[NP], const float2 (&nl)[NP], float2 (&acc)[NP]) {
#pragma unroll 4
  for (int j = 0; j < PseLap::kGroup; ++j) {
    const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c;
#pragma unroll
    for (int p = P0; p < P1; ++p) {
      const float2 dx = __fadd2_rn(tx[p], lo2(ra)), dy = __fadd2_rn(ty[p], hi2(ra));
      float2 v = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
      if (SPHERE) {
        const float2 dz = __fadd2_rn(tz[p], lo2(rb));
        v = __ffma2_rn(dz, dz, v);
      }
      const float2 k = lap_kernel<K8>(lap_exponent<ANG>(v, q));
      if (CLOSE) {
        const float2 m = __fadd2_rn(__fadd2_rn(make_float2(rc.z, rc.z), nf[p]), __fadd2_rn(make_float2(rc.w, rc.w), nl[p]));
        acc[p] = __ffma2_rn(m, __fmul2_rn(hi2(rb), k), acc[p]);
      } else {
        acc[p] = __ffma2_rn(__ffma2_rn(hi2(rb), nf[p], lo2(rc)), k, acc[p]);
      }
    }
  }
}

template <bool SPHERE, bool K8, int ANG, int THREADS, int TPT, int TILE, int MINB, int S>
__global__ void __launch_bounds__(THREADS, MINB) pse_lap_sweep_kernel(PseLapArgs a) {
  static_assert(TPT == 4, "two target pairs");
  constexpr int NP = TPT / 2;
  constexpr int G = PseLap::kGroup;
  constexpr int GPT = TILE / G;
  using Rec = PseLap::Rec;
  using Group = PseLap::Group;
  __shared__ TilePipe<Rec, TILE, S, Group, GPT> pipe;

  const int64_t chunk = blockIdx.y;  // this CTA's share of the target block's in-reach tiles
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (THREADS * TPT);
  const int64_t count = a.nt - first < THREADS * TPT ? a.nt - first : THREADS * TPT;
  float2 xh[NP], yh[NP], zh[NP], xl[NP], yl[NP], zl[NP], fh[NP], fl[NP], hs[NP], ls[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    PseLap::Tgt t[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int64_t il = bve_target<TPT>(2 * p + h);
      if (il >= count) il = count - 1;  // duplicates of a valid target; results not stored
      t[h] = a.tgt[first + il];
    }
    xh[p] = make_float2(t[0].h.x, t[1].h.x);
    yh[p] = make_float2(t[0].h.y, t[1].h.y);
    zh[p] = make_float2(t[0].h.z, t[1].h.z);
    fh[p] = make_float2(t[0].h.w, t[1].h.w);
    xl[p] = make_float2(t[0].l.x, t[1].l.x);
    yl[p] = make_float2(t[0].l.y, t[1].l.y);
    zl[p] = make_float2(t[0].l.z, t[1].l.z);
    fl[p] = make_float2(t[0].l.w, t[1].l.w);
    hs[p] = ls[p] = make_float2(0.f, 0.f);
  }
  // the ball around the CTA's targets (hi parts) for the tile culling
  __shared__ TargetBall ball;
  {
    float bx[2 * NP], by[2 * NP], bz[2 * NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      bx[2 * p] = xh[p].x;
      bx[2 * p + 1] = xh[p].y;
      by[2 * p] = yh[p].x;
      by[2 * p + 1] = yh[p].y;
      bz[2 * p] = zh[p].x;
      bz[2 * p + 1] = zh[p].y;
    }
    cta_target_ball<THREADS, 2 * NP>(bx, by, bz, ball);
  }

  tile_pipe_init(pipe);
  uint32_t g = 0;
  auto tile_body = [&](const Rec* tl, const Group* og) {
    // a group's terms are summed on their own: a running sum of the tile's four groups had 1.1 to
    // 1.3 times the error
    float2 acc[NP];
    auto flush = [&]() {
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        comp_add(hs[p].x, ls[p].x, acc[p].x);
        comp_add(hs[p].y, ls[p].y, acc[p].y);
      }
    };
#pragma unroll 1
    for (int g0 = 0; g0 < TILE; g0 += G) {
#pragma unroll
      for (int p = 0; p < NP; ++p) acc[p] = make_float2(0.f, 0.f);
      const Group o = og[g0 / G];
      const Rec* gr = tl + g0;
      float2 tx[NP], ty[NP], tz[NP], nf[NP], nl[NP];
      const float reach = o.o.w + a.c_cut, close = BveRel::kNearFactor * o.o.w;
      bool in[NP], near = false;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        tx[p] = SPHERE ? rel1x2(xh[p], xl[p], o.o.x) : rel1x2(xh[p], xl[p], o.o.x, o.f.z);
        ty[p] = SPHERE ? rel1x2(yh[p], yl[p], o.o.y) : rel1x2(yh[p], yl[p], o.o.y, o.f.w);
        tz[p] = SPHERE ? rel1x2(zh[p], zl[p], o.o.z) : make_float2(0.f, 0.f);
        float2 n2 = __ffma2_rn(ty[p], ty[p], __fmul2_rn(tx[p], tx[p]));
        if (SPHERE) n2 = __ffma2_rn(tz[p], tz[p], n2);
        // each target pair's 64 targets on their own: consecutive in curve order
        in[p] = __any_sync(0xffffffffu, !(n2.x >= reach * reach) | !(n2.y >= reach * reach));
        near |= !(n2.x > close * close) | !(n2.y > close * close);  // (a group of radius 0: its own particle)
        // -F_i = (f of the group) - f_i as a float pair, with the operations of the records
        const float2 fg = make_float2(o.f.x, o.f.x), mf = make_float2(-fh[p].x, -fh[p].y),
                     ml = make_float2(-fl[p].x, -fl[p].y);
        const float2 s = __fadd2_rn(fg, mf);
        const float2 b = __fadd2_rn(s, make_float2(-fg.x, -fg.y));  // TwoSum of fg and mf
        const float2 e = __fadd2_rn(__fadd2_rn(fg, __fadd2_rn(b, make_float2(-s.x, -s.y))),
                                    __fadd2_rn(mf, make_float2(-b.x, -b.y)));
        const float2 r = __fadd2_rn(e, ml);  // |r| <= |s| or s = 0
        nf[p] = __fadd2_rn(s, r);
        const float2 d = __fadd2_rn(nf[p], make_float2(-s.x, -s.y));
        nl[p] = __fadd2_rn(r, make_float2(-d.x, -d.y));
      }
      if (!in[0] && !in[1]) continue;  // every pair has r^2 > 49
      if (o.f.y == 0.f) {
        if (__any_sync(0xffffffffu, near)) {
          lap_group<SPHERE, K8, ANG, true, 0, 2>(gr, a.q, tx, ty, tz, nf, nl, acc);
        } else if (in[0] && in[1]) {
          lap_group<SPHERE, K8, ANG, false, 0, 2>(gr, a.q, tx, ty, tz, nf, nl, acc);
        } else if (in[0]) {
          lap_group<SPHERE, K8, ANG, false, 0, 1>(gr, a.q, tx, ty, tz, nf, nl, acc);
        } else {
          lap_group<SPHERE, K8, ANG, false, 1, 2>(gr, a.q, tx, ty, tz, nf, nl, acc);
        }
        flush();
        continue;
      }
      // wide group: d = (t_hi - s_hi) + (t_lo - s_lo)
      float2 ux[NP], uy[NP], uz[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        if (SPHERE) {
          rel2x2(xh[p], xl[p], o.o.x, tx[p], ux[p]);
          rel2x2(yh[p], yl[p], o.o.y, ty[p], uy[p]);
          rel2x2(zh[p], zl[p], o.o.z, tz[p], uz[p]);
        } else {
          rel2x2(xh[p], xl[p], o.o.x, o.f.z, tx[p], ux[p]);
          rel2x2(yh[p], yl[p], o.o.y, o.f.w, ty[p], uy[p]);
        }
      }
      for (int j = 0; j < G; ++j) {
        const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c, rd = gr[j].d;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const float2 dx = __fadd2_rn(__fadd2_rn(tx[p], lo2(ra)), __fadd2_rn(ux[p], make_float2(rd.x, rd.x)));
          const float2 dy = __fadd2_rn(__fadd2_rn(ty[p], hi2(ra)), __fadd2_rn(uy[p], make_float2(rd.y, rd.y)));
          float2 v = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
          if (SPHERE) {
            const float2 dz = __fadd2_rn(__fadd2_rn(tz[p], lo2(rb)), __fadd2_rn(uz[p], make_float2(rd.z, rd.z)));
            v = __ffma2_rn(dz, dz, v);
          }
          const float2 k = lap_kernel<K8>(lap_exponent<ANG>(v, a.q));
          const float2 m = __fadd2_rn(__fadd2_rn(make_float2(rc.z, rc.z), nf[p]), __fadd2_rn(make_float2(rc.w, rc.w), nl[p]));
          acc[p] = __ffma2_rn(m, __fmul2_rn(hi2(rb), k), acc[p]);
        }
      }
      flush();
    }
  };
  // this CTA's balanced share of the in-reach tiles of the whole source range (engine.cuh)
  sweep_culled_share<THREADS>(
      a.n_tiles, [&](int64_t t) { return tile_in_reach(a.tball[t], ball, a.c_cut); },
      [&](const int32_t* list, int cnt) {
        return warp_sweep_tiles(a.src, [list](int64_t k) { return static_cast<int64_t>(list[k]); }, cnt, pipe, g,
                                a.status, a.wait, a.grp, tile_body);
      });

#pragma unroll
  for (int p = 0; p < NP; ++p) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t il = bve_target<TPT>(2 * p + h);
      if (il >= count) continue;
      const int64_t at = a.tperm ? static_cast<int64_t>(a.tperm[first + il]) - a.ib : first + il;
      a.partial[chunk * a.nt + at] =
          static_cast<double>(h ? hs[p].y : hs[p].x) + static_cast<double>(h ? ls[p].y : ls[p].x);
    }
  }
}

// The frame of a warp's group of 32 planar sources: the centroid with its low part (planar sets lie
// anywhere, and a float origin is off by half the float spacing there), and the radius about it.  The mean
// is taken of the offsets from the first source.
struct PlaneFrame {
  float o[2], ol[2];
  float radius;
};

__device__ __forceinline__ PlaneFrame plane_group_frame(bool valid, const SplitPoint& sp) {
  PlaneFrame f;
  float d[2], n = valid ? 1.f : 0.f;
  double first[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const float h0 = __shfl_sync(0xffffffffu, sp.h[c], 0), l0 = __shfl_sync(0xffffffffu, sp.l[c], 0);
    first[c] = static_cast<double>(h0) + static_cast<double>(l0);
    d[c] = valid ? __fadd_rn(__fadd_rn(sp.h[c], -h0), __fadd_rn(sp.l[c], -l0)) : 0.f;
  }
  float m[2] = {d[0], d[1]};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m[0] += __shfl_xor_sync(0xffffffffu, m[0], o);
    m[1] += __shfl_xor_sync(0xffffffffu, m[1], o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  const float inv = n > 0.f ? 1.f / n : 0.f;
  float r = 0.f;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    split2(first[c] + static_cast<double>(m[c] * inv), f.o[c], f.ol[c]);
    const float e = valid ? __fadd_rn(__fadd_rn(sp.h[c], -f.o[c]), __fadd_rn(sp.l[c], -f.ol[c])) : 0.f;
    r += e * e;
  }
  if (!(r == r)) r = __int_as_float(0x7f800000);  // a NaN source: an infinite radius
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
  f.radius = sqrtf(r) * 1.000001f;
  return f;
}

// Records, groups and balls of the sorted sources (CTA t < n_tiles: tile t, TILE threads, every thread
// one source), then the targets in the order of the sweep.
template <bool SPHERE, int ANG, int TILE>
__global__ void __launch_bounds__(TILE) pse_lap_prep_kernel(const double* x, const double* y, const double* z,
                                                            const double* f, const double* area,
                                                            const int32_t* sorted, int64_t ns, int64_t n_tiles,
                                                            double inv_a, float c_cut, const int32_t* tperm,
                                                            int64_t ib, int64_t nt, PseLap::Rec* out,
                                                            PseLap::Group* grp, float4* tball, PseLap::Tgt* tgt) {
  constexpr int G = PseLap::kGroup, GPT = TILE / G;
  static_assert(G == 32, "a warp per group");
  auto position = [&](int64_t i) {
    double px, py, pz = 0.0;
    if constexpr (SPHERE) {
      pse_position<ANG == kLapChord ? kPseAngleChord : kPseAngleSeries>(x, y, z, i, inv_a, px, py, pz);
    } else {
      px = x[i];
      py = y[i];
    }
    return split_point(px, py, pz);
  };
  const int64_t t = blockIdx.x;
  if (t >= n_tiles) {
    const int64_t k = (t - n_tiles) * TILE + threadIdx.x;
    if (k >= nt) return;
    const int64_t i = tperm ? static_cast<int64_t>(tperm[k]) : ib + k;
    const SplitPoint sp = position(i);
    float fh, fl;
    split2(f[i], fh, fl);
    tgt[k] = PseLap::Tgt{make_float4(sp.h[0], sp.h[1], sp.h[2], fh), make_float4(sp.l[0], sp.l[1], sp.l[2], fl)};
    return;
  }
  const int64_t k = t * TILE + threadIdx.x;
  const bool valid = k < ns;
  const int32_t j = valid ? sorted[k] : 0;
  SplitPoint sp{};
  float fh = 0.f, fl = 0.f;
  if (valid) {
    sp = position(j);
    split2(f[j], fh, fl);
  }
  float og[3] = {0.f, 0.f, 0.f}, ogl[2] = {0.f, 0.f}, radius;  // the group's origin and radius
  if constexpr (SPHERE) {
    const GroupFrame fr = sphere_group_frame<TILE, G>(valid, sp, 0.0);
    for (int c = 0; c < 3; ++c) og[c] = fr.o[c];
    radius = fr.radius;
  } else {
    const PlaneFrame fr = plane_group_frame(valid, sp);
    for (int c = 0; c < 2; ++c) og[c] = fr.o[c], ogl[c] = fr.ol[c];
    radius = fr.radius;
  }
  const float fg = __shfl_sync(0xffffffffu, fh, 0);  // the first source's field
  PseLap::Rec r;
  if (valid) {
    float hi[3] = {0.f, 0.f, 0.f}, lo[3] = {0.f, 0.f, 0.f};
    if constexpr (SPHERE) {
#pragma unroll
      for (int c = 0; c < 3; ++c) rel2(sp.h[c], sp.l[c], og[c], hi[c], lo[c]);
    } else {
#pragma unroll
      for (int c = 0; c < 2; ++c) rel2(sp.h[c], sp.l[c], og[c], ogl[c], hi[c], lo[c]);
    }
    const float ar = __double2float_rn(area[j]);
    // f_j - f_g = fs + fe, fs rounded from all of it: the low part of f_j is the whole of F_j where f_j and f_g
    // round to the same float (every group of a field with a large mean, and a group's first source)
    float d, de, fs, fe;
    two_sum(fh, -fg, d, de);
    two_sum(d, de + fl, fs, fe);
    const float af = ar * fs;
    r.a = make_float4(-hi[0], -hi[0], -hi[1], -hi[1]);
    r.b = make_float4(-hi[2], -hi[2], ar, ar);
    r.c = make_float4(af, af, fs, fe);
    r.d = make_float4(-lo[0], -lo[1], -lo[2], 0.f);
  } else {
    r.a = r.b = r.c = r.d = make_float4(0.f, 0.f, 0.f, 0.f);  // zero area: no contribution
  }
  out[k] = r;
  __shared__ float4 ball[GPT];  // the groups' balls for the tile's ball (w < 0: empty group)
  if (threadIdx.x % G == 0) {
    PseLap::Group o;
    o.o = make_float4(og[0], og[1], og[2], radius);
    o.f = make_float4(fg, radius > PseLap::kWide * c_cut ? 1.f : 0.f, ogl[0], ogl[1]);
    grp[t * GPT + threadIdx.x / G] = o;
    ball[threadIdx.x / G] = valid ? o.o : make_float4(0.f, 0.f, 0.f, -1.f);
  }
  __syncthreads();
  if (threadIdx.x == 0) tball[t] = tile_ball_from_groups<GPT>(ball);
}

}  // namespace lpm
