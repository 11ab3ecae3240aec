// plane_rel.cuh -- the planar Biot-Savart FP32C sweep on spatially sorted sources in
// group-relative coordinates (7 packed FP32x2 operations per target pair and source).
//
// Reference: planarIncompressibleVelocity, src/PlaneIncompressibleSolver.f90:291-308:
//   u_i = -sum_j S_j (y_i - y_j) / (r^2 + delta^2),  v_i = sum_j S_j (x_i - x_j) / (r^2 + delta^2)
// with S_j = omega_j A_j / (2 pi) (delta = 0 in the reference, delta > 0 the regularised
// extension).  The structure is that of the sphere sweep (bve_rel.cuh): sources in 2-D
// Hilbert-curve order (sort.cu), each group of kGroup sources stored relative to its
// centroid o as rel2(p, o) with the group radius R, and per warp and group a far form
// d = t_hi - s_hi (every target at |t - o| >= 3R: relative error <= ~2^-23) or a near form
// in which each target forms (t_hi, t_lo) = rel2(t, o) with the sources' operations and
// keeps the lo parts (a self pair cancels bit for bit; delta^2 carries a 2^-100 offset so
// that the self weight is finite).  Per target pair and source, far:
//   d (2 FADD2), q = d.d + delta^2 (2 FFMA2), w = S rcp(q) (FMUL2 + 2 MUFU),
//   U += w dy, V += w dx (2 FFMA2);
// near: 4 more FADD2.  Each group's terms are summed in FP32 on their own and added to the
// tile's FP32 partial (2 FADD2 per group), which goes into compensated (hi, lo) pairs; the
// FP64 finish reduces the split-K chunks and sets u = -U, v = V.
#pragma once

#include "bve_x2.cuh"
#include "bve_rel.cuh"
#include "engine.cuh"
#include "ops.cuh"

namespace lpm {

// rel1 and rel2 (bve_rel.cuh) from an origin with a low part (planar sets lie anywhere).
__device__ __forceinline__ float2 rel1x2(float2 ph, float2 pl, float oh, float ol) {
  return __fadd2_rn(__fadd2_rn(ph, make_float2(-oh, -oh)), __fadd2_rn(pl, make_float2(-ol, -ol)));
}
__device__ __forceinline__ void rel2(float ph, float pl, float oh, float ol, float& rh, float& rl) {
  rel2(ph, __fadd_rn(pl, -ol), oh, rh, rl);
}
__device__ __forceinline__ void rel2x2(float2 ph, float2 pl, float oh, float ol, float2& rh, float2& rl) {
  rel2x2(ph, __fadd2_rn(pl, make_float2(-ol, -ol)), oh, rh, rl);
}

struct PlaneRel {
  struct __align__(16) Rec {
    float4 a;  // -sx_hi, -sx_hi, -sy_hi, -sy_hi
    float4 b;  // S_j, S_j, -sx_lo, -sx_lo
    float4 c;  // -sy_lo, -sy_lo, 0, 0
    __device__ static Rec make(float sxh, float sxl, float syh, float syl, float s, float) {
      return Rec{make_float4(-sxh, -sxh, -syh, -syh), make_float4(s, s, -sxl, -sxl), make_float4(-syl, -syl, 0.f, 0.f)};
    }
  };
  struct __align__(16) Origin {
    float4 o;  // o_hi.x, o_hi.y, o_lo.x, o_lo.y
    float4 f;  // R (the group radius about o), S_g hi, S_g lo (S_g = sum of the group's S_j), 0
  };
  struct Pair {
    float2 xh, yh, xl, yl;
  };
  // A target as floats, split once per sum by the prep kernel (every CTA of its block needs it): x_hi, y_hi,
  // x_lo, y_lo.
  using Tgt = float4;
  // sources per origin: 128 (the planar velocity, stream-function and SWE sweeps measured 0.2-2 %
  // faster than with 64)
  static constexpr int kGroup = 128;
  static constexpr float kNearFactor = 3.0f;  // near: |t - o| < kNearFactor R
};

template <class Rec>
struct PlaneRelArgs {
  float d2;  // delta^2 + 2^-100
  const Rec* src;
  const PlaneRel::Origin* org;
  const PlaneRel::Tgt* tgt;
  int64_t n_tiles, nt;
  double* partial;  // [chunk][components][nt]
  int* status;
};

// Target pairs of a sweep: targets first + bve_target(2p + h), clamped to the `count` valid ones
// (duplicates are computed but not stored).
template <int NP>
__device__ __forceinline__ void plane_load_pairs(const PlaneRel::Tgt* __restrict__ tgt, int64_t count,
                                                 PlaneRel::Pair (&pr)[NP]) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    int64_t i0 = bve_target<2 * NP>(2 * p), i1 = bve_target<2 * NP>(2 * p + 1);
    if (i0 >= count) i0 = count - 1;
    if (i1 >= count) i1 = count - 1;
    const float4 t0 = tgt[i0], t1 = tgt[i1];
    pr[p].xh = make_float2(t0.x, t1.x);
    pr[p].yh = make_float2(t0.y, t1.y);
    pr[p].xl = make_float2(t0.z, t1.z);
    pr[p].yl = make_float2(t0.w, t1.w);
  }
}

template <int THREADS, int TPT, int TILE, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) plane_rel_sweep_kernel(PlaneRelArgs<PlaneRel::Rec> a) {
  static_assert(TPT % 2 == 0, "targets come in pairs");
  static_assert(TILE % PlaneRel::kGroup == 0, "whole origin groups per tile");
  constexpr int NP = TPT / 2;
  constexpr int G = PlaneRel::kGroup;
  constexpr int GPT = TILE / G;
  using Rec = PlaneRel::Rec;
  __shared__ __align__(128) Rec stage[2][TILE];
  __shared__ __align__(8) uint64_t bars[2];

  const int64_t chunk = blockIdx.y;
  const ChunkTiles ct = chunk_tiles(a.n_tiles);

  PlaneRel::Pair pr[NP];
  float2 hu[NP], hv[NP], lu[NP], lv[NP];
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (THREADS * TPT);
  const int64_t count = a.nt - first < THREADS * TPT ? a.nt - first : THREADS * TPT;
  plane_load_pairs<NP>(a.tgt + first, count, pr);
#pragma unroll
  for (int p = 0; p < NP; ++p) hu[p] = hv[p] = lu[p] = lv[p] = make_float2(0.f, 0.f);
  const float2 d2 = make_float2(a.d2, a.d2);

  pipe_init(bars);
  uint32_t g = 0;
  auto body = [&](const Rec* tl, const PlaneRel::Origin* og) {
    float2 au[NP], av[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) au[p] = av[p] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int g0 = 0; g0 < TILE; g0 += G) {
      const PlaneRel::Origin o = og[g0 / G];
      const Rec* gr = tl + g0;
      float2 tx[NP], ty[NP];
      bool near = false;
      const float lim = (PlaneRel::kNearFactor * o.f.x) * (PlaneRel::kNearFactor * o.f.x);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        tx[p] = rel1x2(pr[p].xh, pr[p].xl, o.o.x, o.o.z);
        ty[p] = rel1x2(pr[p].yh, pr[p].yl, o.o.y, o.o.w);
        const float2 n2 = __ffma2_rn(ty[p], ty[p], __fmul2_rn(tx[p], tx[p]));
        near |= (n2.x < lim) | (n2.y < lim);
      }
      // the group's terms are summed on their own and then added to the tile's: a running
      // FP32 sum of a whole tile's terms (both signs, e.g. the two lobes of a dipole) rounds
      // at the size of the tile's partial sum 256 times, a group sum only 128 times
      float2 gu[NP], gv[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) gu[p] = gv[p] = make_float2(0.f, 0.f);
      if (!__any_sync(0xffffffffu, near)) {
        // far group: d = t_hi - s_hi
#pragma unroll 4
        for (int j = 0; j < G; ++j) {
          const float4 ra = gr[j].a, rb = gr[j].b;
          const float2 nsx = lo2(ra), nsy = hi2(ra), s2 = lo2(rb);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const float2 dx = __fadd2_rn(tx[p], nsx);
            const float2 dy = __fadd2_rn(ty[p], nsy);
            float2 q = __ffma2_rn(dx, dx, d2);
            q = __ffma2_rn(dy, dy, q);
            const float2 w = __fmul2_rn(s2, make_float2(rcp_approx(q.x), rcp_approx(q.y)));
            gu[p] = __ffma2_rn(w, dy, gu[p]);
            gv[p] = __ffma2_rn(w, dx, gv[p]);
          }
        }
      } else {
        // near group: d = (t_hi - s_hi) + (t_lo - s_lo)
        float2 txh[NP], tyh[NP], txl[NP], tyl[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          rel2x2(pr[p].xh, pr[p].xl, o.o.x, o.o.z, txh[p], txl[p]);
          rel2x2(pr[p].yh, pr[p].yl, o.o.y, o.o.w, tyh[p], tyl[p]);
        }
        for (int j = 0; j < G; ++j) {
          const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c;
          const float2 nsx = lo2(ra), nsy = hi2(ra), s2 = lo2(rb), nlx = hi2(rb), nly = lo2(rc);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const float2 dx = __fadd2_rn(__fadd2_rn(txh[p], nsx), __fadd2_rn(txl[p], nlx));
            const float2 dy = __fadd2_rn(__fadd2_rn(tyh[p], nsy), __fadd2_rn(tyl[p], nly));
            float2 q = __ffma2_rn(dx, dx, d2);
            q = __ffma2_rn(dy, dy, q);
            const float2 w = __fmul2_rn(s2, make_float2(rcp_approx(q.x), rcp_approx(q.y)));
            gu[p] = __ffma2_rn(w, dy, gu[p]);
            gv[p] = __ffma2_rn(w, dx, gv[p]);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        au[p] = __fadd2_rn(au[p], gu[p]);
        av[p] = __fadd2_rn(av[p], gv[p]);
      }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      comp_add(hu[p].x, lu[p].x, au[p].x);
      comp_add(hu[p].y, lu[p].y, au[p].y);
      comp_add(hv[p].x, lv[p].x, av[p].x);
      comp_add(hv[p].y, lv[p].y, av[p].y);
    }
  };
  int64_t tile = ct.first;
  staged_sweep<Rec, TILE>(a.src, ct.first, ct.count, stage[0], stage[1], bars, g, a.status, [&](const Rec* tl) {
    body(tl, a.org + tile * GPT);
    tile += ct.step;
  }, ct.step);

#pragma unroll
  for (int p = 0; p < NP; ++p) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t il = first + bve_target<TPT>(2 * p + h);
      if (il < a.nt) {
        a.partial[(chunk * 2 + 0) * a.nt + il] =
            static_cast<double>(h ? hu[p].y : hu[p].x) + static_cast<double>(h ? lu[p].y : lu[p].x);
        a.partial[(chunk * 2 + 1) * a.nt + il] =
            static_cast<double>(h ? hv[p].y : hv[p].x) + static_cast<double>(h ? lv[p].y : lv[p].x);
      }
    }
  }
}

// Records and origins of one tile of TILE sources (one CTA of TILE threads): each group of
// kGroup sources reduces its centroid o, its radius R about o and its total S_g (of the FP32
// strengths), and every record is written as rel2(p_j, o) -- the operations the sweep uses
// for targets.  s_scale = 1/(2 pi) for the velocity, 1/(4 pi) for the stream function.
// `second` (optional): a second strength second_j A_j s_scale (the SWE divergence).  CTA t < n_tiles writes
// tile t, the others split the nt targets from ib on.
template <int TILE, class Rec>
__global__ void __launch_bounds__(TILE) plane_rel_prep_kernel(const double* x, const double* y, const double* omega,
                                                              const double* area, const int32_t* sorted, int64_t ns,
                                                              int64_t n_tiles, double s_scale, int64_t ib, int64_t nt,
                                                              Rec* out, PlaneRel::Origin* org, PlaneRel::Tgt* tgt,
                                                              const double* second = nullptr) {
  constexpr int G = PlaneRel::kGroup;
  __shared__ double red[3][TILE];
  __shared__ float fmax_[TILE], cntf[TILE];
  const int64_t t = blockIdx.x;
  const int tid = threadIdx.x;
  if (t >= n_tiles) {
    const int64_t il = (t - n_tiles) * TILE + tid;
    if (il < nt) {
      float xh, xl, yh, yl;
      split2(x[ib + il], xh, xl);
      split2(y[ib + il], yh, yl);
      tgt[il] = make_float4(xh, yh, xl, yl);
    }
    return;
  }
  const int64_t k = t * TILE + tid;
  const bool valid = k < ns;
  const int32_t j = valid ? sorted[k] : 0;
  const int lane = tid % G;
  const double px = valid ? x[j] : 0.0, py = valid ? y[j] : 0.0;
  const float s = valid ? __double2float_rn(omega[j] * area[j] * s_scale) : 0.f;
  red[0][tid] = px;
  red[1][tid] = py;
  red[2][tid] = s;
  cntf[tid] = valid ? 1.f : 0.f;
  __syncthreads();
  for (int w = G / 2; w > 0; w >>= 1) {
    if (lane < w) {
      red[0][tid] += red[0][tid + w];
      red[1][tid] += red[1][tid + w];
      red[2][tid] += red[2][tid + w];
      cntf[tid] += cntf[tid + w];
    }
    __syncthreads();
  }
  const int g0 = tid - lane;
  const double cnt = cntf[g0] > 0.f ? static_cast<double>(cntf[g0]) : 1.0;
  const double cx = red[0][g0] / cnt, cy = red[1][g0] / cnt;
  fmax_[tid] = valid ? static_cast<float>(sqrt((px - cx) * (px - cx) + (py - cy) * (py - cy))) : 0.f;
  __syncthreads();
  for (int w = G / 2; w > 0; w >>= 1) {
    if (lane < w) fmax_[tid] = fmaxf(fmax_[tid], fmax_[tid + w]);
    __syncthreads();
  }
  float oxh, oxl, oyh, oyl;
  split2(cx, oxh, oxl);
  split2(cy, oyh, oyl);
  float sxh = 0.f, sxl = 0.f, syh = 0.f, syl = 0.f, s2 = 0.f;
  if (valid) {
    float h, l;
    split2(px, h, l);
    rel2(h, l, oxh, oxl, sxh, sxl);
    split2(py, h, l);
    rel2(h, l, oyh, oyl, syh, syl);
    if (second) s2 = __double2float_rn(second[j] * area[j] * s_scale);
  }
  // (past the sources: inert, at the origin with zero strength)
  out[k] = Rec::make(sxh, sxl, syh, syl, s, s2);
  if (lane == 0) {
    PlaneRel::Origin o;
    o.o = make_float4(oxh, oyh, oxl, oyl);
    float sgh, sgl;
    split2(red[2][g0], sgh, sgl);
    o.f = make_float4(fmax_[g0], sgh, sgl, 0.f);
    org[t * (TILE / G) + tid / G] = o;
  }
}

// ====================================================================== planar SWE integrals
// SWEPlaneRHSIntegrals, src/SWEPlaneSolver.f90:457-571, velocity and velocity-gradient part
// (the surface-height Laplacian is the planar PSE sweep, pse_lap.cuh).  With W = vort_j A_j / (2 pi),
// D = div_j A_j / (2 pi) and s = 1/r^2, the reference's terms are
//   u += s P, v += s Q,  P = D dx - W dy, Q = W dx + D dy,
//   ux += D s - 2 s dx (s P),  uy += -W s - 2 s dy (s P),
//   vx +=  W s - 2 s dx (s Q), vy += D s - 2 s dy (s Q)
// (1/(pi r^4) = 2 s^2 / (2 pi)).  In z = dx + i dy they are u - i v = (D - i W) / z and its
// derivative, so uy = vx and vy = -ux term by term, and with p = s dx, q = -s dy (1/z = p + i q),
//   u = D p + W q,  v = W p - D q,  -ux = D A - W T,  -vx = W A + D T,
//   A = p^2 - q^2 = s - 2 q^2,  T = -2 p q:
// 17 packed operations and 2 MUFU per target pair and source (far form), four sums instead of six (23
// operations).  Near groups add the lo parts and give the self pair s = 0.  Partials: [chunk][4][nt].
// Bound: the FP32 pipe.  The call took 7.69 ms at 131,585 points (1.00 at 33,025) with six sums of 23
// operations, 5.94 (0.82) with four of 17, and 6.33 (0.88) with running sums of 32 sources instead of a
// tile's 256, which brought the velocity's error from 1.5 times the former one to 0.3 times and the
// double dot product's to 0.7 times.  128 x 6 targets and 3 CTAs per SM: 6.56.
struct PlaneSwe {
  struct __align__(16) Rec {
    float4 a;  // -sx_hi, -sx_hi, sy_hi, sy_hi
    float4 b;  // W, W, D, D
    float4 c;  // -W, -W, -D, -D
    float4 d;  // -sx_lo, sy_lo, 0, 0   (near form)
    __device__ static Rec make(float sxh, float sxl, float syh, float syl, float w, float dv) {
      return Rec{make_float4(-sxh, -sxh, syh, syh), make_float4(w, w, dv, dv), make_float4(-w, -w, -dv, -dv),
                 make_float4(-sxl, syl, 0.f, 0.f)};
    }
  };
};

template <int THREADS, int TPT, int TILE, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) plane_swe_rel_sweep_kernel(PlaneRelArgs<PlaneSwe::Rec> a) {
  static_assert(TPT % 2 == 0, "targets come in pairs");
  static_assert(TILE % PlaneRel::kGroup == 0, "whole origin groups per tile");
  constexpr int NP = TPT / 2;
  constexpr int G = PlaneRel::kGroup;
  constexpr int GPT = TILE / G;
  constexpr int NC = 4;
  constexpr int FL = 32;  // sources to a running FP32 sum
  using Rec = PlaneSwe::Rec;
  __shared__ TilePipe<Rec, TILE, 2, PlaneRel::Origin, GPT> pipe;

  const int64_t chunk = blockIdx.y;
  const ChunkTiles ct = chunk_tiles(a.n_tiles);

  PlaneRel::Pair pr[NP];
  float2 hs[NP][NC], ls[NP][NC];
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (THREADS * TPT);
  const int64_t count = a.nt - first < THREADS * TPT ? a.nt - first : THREADS * TPT;
  plane_load_pairs<NP>(a.tgt + first, count, pr);
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int c = 0; c < NC; ++c) hs[p][c] = ls[p][c] = make_float2(0.f, 0.f);
  const float2 m2 = make_float2(-2.0f, -2.0f);

  tile_pipe_init(pipe);
  uint32_t g = 0;
  auto body = [&](const Rec* tl, const PlaneRel::Origin* og) {
    float2 acc[NP][NC];
    auto clear = [](float2 (&v)[NP][NC]) {
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int c = 0; c < NC; ++c) v[p][c] = make_float2(0.f, 0.f);
    };
    auto add = [&](const float2 (&v)[NP][NC]) {
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[p][c] = __fadd2_rn(acc[p][c], v[p][c]);
    };
    clear(acc);
    // one pair's terms from d = (dx, -dy) and s = 1/r^2 (0 for the self pair)
    auto terms = [&](float2 (&ac)[NC], float2 dx, float2 ndy, float2 sv, float4 rb, float4 rc) {
      const float2 pv = __fmul2_rn(sv, dx), qv = __fmul2_rn(sv, ndy);
      const float2 t = __fmul2_rn(qv, m2);
      const float2 av = __ffma2_rn(t, qv, sv), tv = __fmul2_rn(t, pv);
      ac[0] = __ffma2_rn(hi2(rb), pv, __ffma2_rn(lo2(rb), qv, ac[0]));
      ac[1] = __ffma2_rn(lo2(rb), pv, __ffma2_rn(hi2(rc), qv, ac[1]));
      ac[2] = __ffma2_rn(hi2(rb), av, __ffma2_rn(lo2(rc), tv, ac[2]));
      ac[3] = __ffma2_rn(lo2(rb), av, __ffma2_rn(hi2(rb), tv, ac[3]));
    };
#pragma unroll 1
    for (int g0 = 0; g0 < TILE; g0 += G) {
      const PlaneRel::Origin o = og[g0 / G];
      const Rec* gr = tl + g0;
      float2 tx[NP], ty[NP];  // x and -y of the offset
      bool near = false;
      const float lim = fmaxf((PlaneRel::kNearFactor * o.f.x) * (PlaneRel::kNearFactor * o.f.x),
                              7.888609052210118e-31f);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        tx[p] = rel1x2(pr[p].xh, pr[p].xl, o.o.x, o.o.z);
        const float2 y = rel1x2(pr[p].yh, pr[p].yl, o.o.y, o.o.w);
        ty[p] = make_float2(-y.x, -y.y);
        const float2 n2 = __ffma2_rn(ty[p], ty[p], __fmul2_rn(tx[p], tx[p]));
        near |= !(n2.x > lim) | !(n2.y > lim);
      }
      if (!__any_sync(0xffffffffu, near)) {
        // far group: d = t_hi - s_hi, r^2 > 0
#pragma unroll 1
        for (int j0 = 0; j0 < G; j0 += FL) {
          float2 sum[NP][NC];
          clear(sum);
#pragma unroll 2
          for (int j = j0; j < j0 + FL; ++j) {
            const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
              const float2 dx = __fadd2_rn(tx[p], lo2(ra));
              const float2 dy = __fadd2_rn(ty[p], hi2(ra));
              const float2 r2 = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
              terms(sum[p], dx, dy, make_float2(rcp_approx(r2.x), rcp_approx(r2.y)), rb, rc);
            }
          }
          add(sum);
        }
      } else {
        // near group: d = (t_hi - s_hi) + (t_lo - s_lo); the self pair has d = 0 exactly
        float2 txl[NP], tyl[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          rel2x2(pr[p].xh, pr[p].xl, o.o.x, o.o.z, tx[p], txl[p]);
          rel2x2(pr[p].yh, pr[p].yl, o.o.y, o.o.w, ty[p], tyl[p]);
          ty[p] = make_float2(-ty[p].x, -ty[p].y);
          tyl[p] = make_float2(-tyl[p].x, -tyl[p].y);
        }
#pragma unroll 1
        for (int j0 = 0; j0 < G; j0 += FL) {
          float2 sum[NP][NC];
          clear(sum);
          for (int j = j0; j < j0 + FL; ++j) {
            const float4 ra = gr[j].a, rb = gr[j].b, rc = gr[j].c, rd = gr[j].d;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
              const float2 dx =
                  __fadd2_rn(__fadd2_rn(tx[p], lo2(ra)), __fadd2_rn(txl[p], make_float2(rd.x, rd.x)));
              const float2 dy =
                  __fadd2_rn(__fadd2_rn(ty[p], hi2(ra)), __fadd2_rn(tyl[p], make_float2(rd.y, rd.y)));
              const float2 r2 = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
              const float2 sv = make_float2(r2.x > 0.f ? rcp_approx(r2.x) : 0.f, r2.y > 0.f ? rcp_approx(r2.y) : 0.f);
              terms(sum[p], dx, dy, sv, rb, rc);
            }
          }
          add(sum);
        }
      }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        comp_add(hs[p][c].x, ls[p][c].x, acc[p][c].x);
        comp_add(hs[p][c].y, ls[p][c].y, acc[p][c].y);
      }
  };
  warp_sweep_tiles(a.src, [ct](int64_t t) { return ct.first + t * ct.step; }, ct.count, pipe, g, a.status,
                   default_wait(), a.org, body);

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

}  // namespace lpm
