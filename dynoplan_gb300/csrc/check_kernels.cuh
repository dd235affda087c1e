// check_kernels.cuh -- exact checking of (primitive, node) pairs on sm_103a.
//
// Replaces LazyTraj::compute + check_lazy_trajectory
// (include/dynoplan/dbastar/dbastar.hpp:166-230, src/dbastar/dbastar.cpp:391-490)
// for every in-ball pair of a batch.
//
// Work decomposition: persistent warps take (primitive, 32 nodes) items from a
// device counter, longest primitives first.  check_pairs: the 32 lanes walk the
// same primitive in lockstep, so the per-state pose rows are warp-broadcast
// loads and the lanes differ only by their node offset.  check_pairs_slots
// (below, the default) gives every test of the item to a lane of its own.
//
// Transform: position_k = canonical_k + p0 (+ k*dt*v0), velocity_k =
// canonical_k + v0, other components canonical_k.  That is the translation of
// the stored states (unicycle1, car1) and, exactly, the re-rollout from the
// shifted start for quad2d / quadrotor (no dynamics term depends on position
// or velocity); the canonical rollout is FP64, once per upload.
//
// Obstacles (shared memory) are culled in the lockstep walk per lane in two levels, both with a
// margin of band + slack (+ kGapCap when min_gap is an output) so nothing that
// could touch the robot, fall in the FP64 band or set min_gap is dropped:
//   1. against the bounding box of the whole transformed primitive (once per
//      pair; bitmask over <= kMaxCullObs obstacles),
//   2. against the box of each chunk of R::CHUNK states (from the level-1 set),
// then every state tests its chunk's candidates (separating axes, AABB early
// reject).  Bounds tests run only in chunks whose box is not inside the
// bounds, and a chunk in which no lane has an obstacle or bounds test to make
// is stepped over as a whole.  A test whose FP32 gap lies within `band` of zero, and a bounds
// test within `band` of a bound, is recomputed in FP64 from the FP64 tables
// on the spot, so verdicts equal the FP64 oracle's.
#pragma once

#include <type_traits>

#include "expand_kernels.cuh"

namespace dpg {

struct CheckArgs {
  RobotParams rp;
  PrimView pv;
  NodeView nv;
  EnvView ev;
  PairView out;
  const unsigned long long *ord_pbase;
  const unsigned long long *ord_ibase;
  const uint32_t *item_pos;  // item -> order position (null: binary search over ord_ibase)
  DevCounters *ctr;
  const volatile int *abort_flag;
  double band;       // FP64 re-check band (0 on the FP64 path)
  float cull_margin; // obstacle culling margin
  // FP32 copies of the constants the state loop uses (GB300 runs FP64 and
  // double->float conversions at 1/64 of the FP32 rate)
  float dt32, half_len32, half_wid32, radius32, band32;
  float lo32[3], hi32[3];
  float lo_out[3], lo_in[3], hi_in[3], hi_out[3];  // the bounds less and plus the band
  float lo_box[3], hi_box[3];  // a box within these (band and slack inside) needs no bounds test
  // this launch takes work items [n_items cum[sub] / cum[nsub],
  // n_items cum[sub + 1] / cum[nsub]) (integer weights; nsub <= 1: all items)
  int sub, nsub;
  int sub_cum[kMaxSub + 1];
  // progress-driven copies (one launch, nsub = 1): the items fall into
  // n_ranges ranges by the same weights; a warp adds the items it finished
  // in a range to range_done when it moves to the next range or stops (after
  // a fence), and the add that completes a range sets range_flag[j] (mapped
  // host memory) after a system fence
  int n_ranges;
  int *range_flag;
  // when set, the pair's node id is written back through it (processing
  // order -> caller's numbering) once the pair is checked
  const uint32_t *perm;
  // slot variant: byte offset of the warps' scratch in dynamic shared memory,
  // and its bytes per warp
  int slot_offset, slot_stride;
};

// The FP32 bounds and the limits derived from them.
inline void set_bounds(CheckArgs &a, const double *lo, const double *hi) {
  for (int i = 0; i < 3; i++) {
    a.lo32[i] = (float)lo[i];
    a.hi32[i] = (float)hi[i];
    a.lo_out[i] = a.lo32[i] - a.band32;
    a.lo_in[i] = a.lo32[i] + a.band32;
    a.hi_in[i] = a.hi32[i] - a.band32;
    a.hi_out[i] = a.hi32[i] + a.band32;
    a.lo_box[i] = a.lo_in[i] + 1e-3f;
    a.hi_box[i] = a.hi_in[i] - 1e-3f;
  }
}

// Obstacle culling margin: every obstacle within the FP64 band, plus a slack
// for the FP32 box arithmetic, and within the min_gap cap when min_gap is an
// output (without it, obstacles farther than the band change no result).
inline float cull_margin(bool min_gap, double band) { return (min_gap ? kGapCap : 0.f) + (float)band + 1e-3f; }

template <class Real> __device__ __forceinline__ const Pose<Real> *pose_table(const PrimView &pv);
template <> __device__ __forceinline__ const Pose<float> *pose_table<float>(const PrimView &pv) { return pv.pose32; }
template <> __device__ __forceinline__ const Pose<double> *pose_table<double>(const PrimView &pv) { return pv.pose64; }

// node offset component i (position i < POSD, then velocity)
template <class Real> __device__ __forceinline__ Real node_off(const NodeView &nv, int64_t n, int i, int nx, int comp);
template <> __device__ __forceinline__ float node_off<float>(const NodeView &nv, int64_t n, int i, int nx, int comp) {
  return nv.off32[i * nv.N + n];
}
template <> __device__ __forceinline__ double node_off<double>(const NodeView &nv, int64_t n, int i, int nx, int comp) {
  return nv.x64[n * nx + comp];
}

// ------------------------------------------------------------ narrow phase --

// a b + c d with the rounding written out in FP32: every kernel that makes a
// test rounds it alike, so they send the same tests to FP64 (DPG_FLAG_CONTACT_RECHECK)
__device__ __forceinline__ float dot2(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ double dot2(double a, double b, double c, double d) { return a * b + c * d; }

// Oriented box (pose c,s; half extents a,b; axis-aligned half extents ex,ey)
// against an obstacle box.  Returns 0 clear, 1 contact, 2 ambiguous (|gap| <=
// band, FP32 path).  mg takes the axis-aligned clearance.
template <class Real, bool BAND>
__device__ __forceinline__ int planar_test(Real px, Real py, Real c, Real s, Real ex, Real ey,
                                           const Obs2<Real> &ob, Real a, Real b, Real band, Real &mg) {
  const Real dx = px - ob.cx, dy = py - ob.cy;
  const Real g = fmax(fabs(dx) - (ex + ob.hx), fabs(dy) - (ey + ob.hy));
  mg = fmin(mg, g);
  if (g > band) return 0;
  const Real ac = fabs(c), as = fabs(s);
  const Real du = dot2(dx, c, dy, s), dv = dot2(dy, c, -dx, s);
  const Real gu = fabs(du) - (a + ob.hx * ac + ob.hy * as);
  const Real gv = fabs(dv) - (b + ob.hx * as + ob.hy * ac);
  const Real gs = fmax(g, fmax(gu, gv));
  if (BAND) {
    if (gs > band) return 0;
    return gs < -band ? 1 : 2;
  }
  return gs <= Real(0) ? 1 : 0;
}

template <class Real, bool BAND>
__device__ __forceinline__ int sphere_test(Real px, Real py, Real pz, const Obs3<Real> &ob, Real rad,
                                           Real band, Real &mg) {
  const Real dx = fabs(px - ob.cx) - ob.hx, dy = fabs(py - ob.cy) - ob.hy, dz = fabs(pz - ob.cz) - ob.hz;
  const Real m = fmax(dx, fmax(dy, dz));
  const Real g = m - rad;
  mg = fmin(mg, g);
  if (g > band) return 0;
  const Real ux = fmax(dx, Real(0)), uy = fmax(dy, Real(0)), uz = fmax(dz, Real(0));
  const Real gs = (m <= Real(0) ? m : sqrt(ux * ux + uy * uy + uz * uz)) - rad;
  if (BAND) {
    if (gs > band) return 0;
    return gs < -band ? 1 : 2;
  }
  return gs <= Real(0) ? 1 : 0;
}

// FP64 position component i of state k (affine transform of the FP64 table)
template <int KIND>
__device__ __forceinline__ double pos64(const CheckArgs &A, int64_t row, int k, const double *x64, int i) {
  using R = Robot<KIND>;
  const Pose<double> ps = A.pv.pose64[row];  // part 0 = the state position
  double v = (i == 0 ? ps.cx : (i == 1 ? ps.cy : ps.c)) + x64[i];
  if (R::VELOFF) v += (double(k) * A.rp.dt) * x64[R::vel_comp(i)];
  return v;
}

// FP64 separating-axis gap of part q at state k against obstacle o (the
// oracle's formula, from the FP64 tables).
template <int KIND>
__device__ double gap64(const CheckArgs &A, int64_t s0, int k, int q, const double *x64, int o) {
  using R = Robot<KIND>;
  const RobotParams &rp = A.rp;
  double sx = x64[0], sy = x64[1], sz = R::POSD == 3 ? x64[2] : 0.0;
  if (R::VELOFF) {
    const double t = double(k) * rp.dt;
    sx += t * x64[R::vel_comp(0)];
    sy += t * x64[R::vel_comp(1)];
    if (R::POSD == 3) sz += t * x64[R::vel_comp(2)];
  }
  const Pose<double> ps = A.pv.pose64[q * A.pv.S + s0 + k];
  if constexpr (R::SPHERE) {
    const Obs3<double> ob = ((const Obs3<double> *)A.ev.obs64)[o];
    const double dx = fabs(ps.cx + sx - ob.cx) - ob.hx, dy = fabs(ps.cy + sy - ob.cy) - ob.hy,
                 dz = fabs(ps.c + sz - ob.cz) - ob.hz;
    const double m = fmax(dx, fmax(dy, dz));
    const double ux = fmax(dx, 0.0), uy = fmax(dy, 0.0), uz = fmax(dz, 0.0);
    return (m <= 0 ? m : sqrt(ux * ux + uy * uy + uz * uz)) - rp.radius;
  } else {
    const Obs2<double> ob = ((const Obs2<double> *)A.ev.obs64)[o];
    const double px = ps.cx + sx, py = ps.cy + sy;
    const double ac = fabs(ps.c), as = fabs(ps.s);
    const double a = rp.half_len, b = rp.half_wid;
    const double dx = px - ob.cx, dy = py - ob.cy;
    const double gx = fabs(dx) - (a * ac + b * as + ob.hx);
    const double gy = fabs(dy) - (a * as + b * ac + ob.hy);
    const double du = dx * ps.c + dy * ps.s, dv = -dx * ps.s + dy * ps.c;
    const double gu = fabs(du) - (a + ob.hx * ac + ob.hy * as);
    const double gv = fabs(dv) - (b + ob.hx * as + ob.hy * ac);
    return fmax(fmax(gx, gy), fmax(gu, gv));
  }
}

// box (centre cen, half hf) against obstacle box, with margin
template <int D, class Real>
__device__ __forceinline__ bool near_box(const float *cen, const float *hf, const void *obs_sm, int o, float M) {
  if constexpr (D == 2) {
    const Obs2<Real> ob = ((const Obs2<Real> *)obs_sm)[o];
    return fabsf(cen[0] - (float)ob.cx) <= hf[0] + (float)ob.hx + M &&
           fabsf(cen[1] - (float)ob.cy) <= hf[1] + (float)ob.hy + M;
  } else {
    const Obs3<Real> ob = ((const Obs3<Real> *)obs_sm)[o];
    return fabsf(cen[0] - (float)ob.cx) <= hf[0] + (float)ob.hx + M &&
           fabsf(cen[1] - (float)ob.cy) <= hf[1] + (float)ob.hy + M &&
           fabsf(cen[2] - (float)ob.cz) <= hf[2] + (float)ob.hz + M;
  }
}


// ------------------------------------------------------------- one pair ----

// NW: words of the per-lane obstacle bitmasks (obstacles <= 32 NW); 0 = no
// culling (more than kMaxCullObs obstacles), every state tests every obstacle.
// ES64: write the end state in FP64 (the FP64 canonical row plus the FP64
// node offset) while the tests run in Real.
template <int KIND, class Real, bool BAND, int NW, bool LOCKSTEP, bool ES64 = false>
__device__ void check_one(const CheckArgs &A, const void *obs_sm, int p, int64_t pair, uint32_t node,
                          bool active) {
  using R = Robot<KIND>;
  constexpr int D = R::POSD, V = R::VELOFF;
  const PrimView &pv = A.pv;
  const RobotParams &rp = A.rp;
  const int L = pv.len[p];
  const int64_t s0 = pv.soff[p];
  const Pose<Real> *pose = pose_table<Real>(pv);
  constexpr bool F32 = sizeof(Real) == 4;
  const Real band = BAND ? (F32 ? Real(A.band32) : Real(A.band)) : Real(0);
  const Real dtR = F32 ? Real(A.dt32) : Real(rp.dt);
  Real loR[3], hiR[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    loR[i] = F32 ? Real(A.lo32[i]) : Real(A.ev.lo[i]);
    hiR[i] = F32 ? Real(A.hi32[i]) : Real(A.ev.hi[i]);
  }
  const double *x64 = A.nv.x64 + (int64_t)(active ? node : 0) * R::NX;
  const int n_obs = A.ev.n_obs;

  Real off[D + V];
#pragma unroll
  for (int i = 0; i < D; i++) off[i] = active ? node_off<Real>(A.nv, node, i, R::NX, i) : Real(0);
#pragma unroll
  for (int i = 0; i < V; i++) off[D + i] = active ? node_off<Real>(A.nv, node, D + i, R::NX, R::vel_comp(i)) : Real(0);

  // bounds pre-check on the swept box of the positions: inside with a margin
  // (band + slack for the arithmetic) means no state needs a bounds test
  bool need_bounds = true;
  if (active) {
    const double *bx = pv.pbox + (int64_t)p * 2 * D;
    const float *bx32 = pv.pbox32 + (int64_t)p * 2 * D;
    const Real tmax = Real(L - 1) * dtR;
    const Real slack = F32 ? Real(1e-3f) : Real(0);
    bool inside = true;
#pragma unroll
    for (int i = 0; i < D; i++) {
      Real lo = (F32 ? Real(bx32[i]) : Real(bx[i])) + off[i];
      Real hi = (F32 ? Real(bx32[D + i]) : Real(bx[D + i])) + off[i];
      if (V) {
        const Real sv = tmax * off[D + i];
        lo += fmin(sv, Real(0));
        hi += fmax(sv, Real(0));
      }
      inside = inside && lo > loR[i] + band + slack && hi < hiR[i] - band - slack;
    }
    need_bounds = !inside;
  }

  // level-1 culling: obstacles near the whole transformed primitive
  constexpr bool CULL = NW > 0;
  constexpr int NWA = NW > 0 ? NW : 1;
  uint32_t l1[NWA] = {};
  const float M = A.cull_margin;
  if (CULL && active) {
    const float *tb = pv.tbox32 + (int64_t)p * 2 * D;
    const float tmax = float(L - 1) * A.dt32;
    float cen[D], hf[D];
#pragma unroll
    for (int i = 0; i < D; i++) {
      cen[i] = tb[i] + (float)off[i];
      hf[i] = tb[D + i];
      if (V) {
        const float sv = tmax * (float)off[D + i];
        cen[i] += 0.5f * sv;
        hf[i] += 0.5f * fabsf(sv);
      }
    }
#pragma unroll
    for (int w = 0; w < NWA; w++) {  // word by word: the masks stay in registers
      uint32_t bits = 0u;
      const int o0 = 32 * w, o1 = min(n_obs, o0 + 32);
      for (int o = o0; o < o1; o++)
        if (near_box<D, Real>(cen, hf, obs_sm, o, M)) bits |= 1u << (o - o0);
      l1[w] = bits;
    }
  }

  bool done = !active, collided = false, rechecked = false;
  int first_oob = L, first_col = L;
  Real mg = Real(INFINITY);
  const Real hl = F32 ? Real(A.half_len32) : Real(rp.half_len);
  const Real hw = F32 ? Real(A.half_wid32) : Real(rp.half_wid);
  const Real rad = F32 ? Real(A.radius32) : Real(rp.radius);
  uint32_t cm[NWA] = {};
  bool nb = need_bounds;  // bounds tests in the current chunk

  for (int k = 0; k < L; k++) {
    if (LOCKSTEP) {
      if (!__any_sync(kFull, !done)) break;
    } else if (done) {
      break;
    }
    const Real t = Real(k) * dtR;
    // at each chunk start: the chunk's box (the parts over its R::CHUNK states,
    // transformed), level-2 culling, and whether its states need bounds tests
    if (CULL && (k % R::CHUNK) == 0) {
      const float *cb = pv.cbox32 + (pv.coff[p] + k / R::CHUNK) * 2 * D;
      const float t0 = float(k) * A.dt32, t1 = float(min(L - 1, k + R::CHUNK - 1)) * A.dt32;
      float cen[D], hf[D];
#pragma unroll
      for (int i = 0; i < D; i++) {
        cen[i] = cb[i] + (float)off[i];
        hf[i] = cb[D + i];
        if (V) {
          const float v = (float)off[D + i];
          cen[i] += 0.5f * (t0 + t1) * v;
          hf[i] += 0.5f * (t1 - t0) * fabsf(v);
        }
      }
      if (!done && !collided) {
#pragma unroll
        for (int w = 0; w < NWA; w++) {
          uint32_t m = l1[w], c = 0;
          while (m) {
            const int b = __ffs(m) - 1;
            m &= m - 1;
            if (near_box<D, Real>(cen, hf, obs_sm, 32 * w + b, M)) c |= 1u << b;
          }
          cm[w] = c;
        }
      }
      // the box holds every state position of the chunk: inside the bounds
      // with the band and an arithmetic slack, no state of it is out
      if (need_bounds) {
        bool in = true;
#pragma unroll
        for (int i = 0; i < D; i++)
          in = in && cen[i] - hf[i] > A.lo32[i] + A.band32 + 1e-3f && cen[i] + hf[i] < A.hi32[i] - A.band32 - 1e-3f;
        nb = !in;
      }
      // no lane has an obstacle test or a bounds test to make in this chunk:
      // its states change nothing (no contact, no bound, no min_gap update)
      if (LOCKSTEP) {
        uint32_t any = 0u;
#pragma unroll
        for (int w = 0; w < NWA; w++) any |= cm[w];
        const bool idle = done || ((collided || any == 0u) && !nb);
        if (__all_sync(kFull, idle)) {
          k += R::CHUNK - 1;
          continue;
        }
      }
    }
    if (done) continue;
    // per-state geometry (identical for the 32 lanes)
    Pose<Real> ps[R::PARTS];
#pragma unroll
    for (int q = 0; q < R::PARTS; q++) ps[q] = pose[q * pv.S + s0 + k];
    Real sx = off[0], sy = off[1], sz = Real(0);
    if (V) { sx += t * off[D + 0]; sy += t * off[D + 1]; }
    if (D == 3) { sz = off[2]; if (V) sz += t * off[D + 2]; }
    if (nb) {
      const Real pv3[3] = {ps[0].cx + sx, ps[0].cy + sy, ps[0].c + sz};
      int bt = 0;
#pragma unroll
      for (int i = 0; i < D; i++) {
        int r;
        if (BAND) {
          const Real v = pv3[i];
          const Real lo = loR[i], hi = hiR[i];
          r = (v < lo - band || v > hi + band) ? 1 : ((v <= lo + band || v >= hi - band) ? 2 : 0);
          if (r == 2) {  // decide in FP64
            const double v64 = pos64<KIND>(A, s0 + k, k, x64, i);
            r = (v64 >= A.ev.lo[i] && v64 <= A.ev.hi[i]) ? 0 : 1;
            rechecked = true;
          }
        } else {
          r = (pv3[i] >= loR[i] && pv3[i] <= hiR[i]) ? 0 : 1;
        }
        bt |= r;
      }
      if (bt) { first_oob = k; done = true; continue; }
    }
    if (collided) continue;
    bool hit = false;
    auto test_obstacle = [&](int o) {
      if constexpr (R::SPHERE) {
        const Obs3<Real> ob = ((const Obs3<Real> *)obs_sm)[o];
        int r = sphere_test<Real, BAND>(ps[0].cx + sx, ps[0].cy + sy, ps[0].c + sz, ob, rad, band, mg);
        if (BAND && r == 2) { r = gap64<KIND>(A, s0, k, 0, x64, o) <= 0.0 ? 1 : 0; rechecked = true; }
        hit |= r == 1;
      } else {
        const Obs2<Real> ob = ((const Obs2<Real> *)obs_sm)[o];
#pragma unroll
        for (int q = 0; q < R::PARTS; q++) {
          const Real ac = fabs(ps[q].c), as = fabs(ps[q].s);
          const Real ex = dot2(hl, ac, hw, as), ey = dot2(hl, as, hw, ac);
          int r = planar_test<Real, BAND>(ps[q].cx + sx, ps[q].cy + sy, ps[q].c, ps[q].s, ex, ey, ob, hl, hw,
                                          band, mg);
          if (BAND && r == 2) { r = gap64<KIND>(A, s0, k, q, x64, o) <= 0.0 ? 1 : 0; rechecked = true; }
          hit |= r == 1;
        }
      }
    };
    if (CULL) {
#pragma unroll
      for (int w = 0; w < NWA; w++) {
        uint32_t m = cm[w];
        while (m) {
          const int b = __ffs(m) - 1;
          m &= m - 1;
          test_obstacle(32 * w + b);
        }
      }
    } else {
      for (int o = 0; o < n_obs; o++) test_obstacle(o);
    }
    if (hit) {
      collided = true;
      first_col = k;
      if (!need_bounds) done = true;
    }
  }

  const unsigned rmask = LOCKSTEP ? __ballot_sync(kFull, active && rechecked) : 0u;
  if (LOCKSTEP && (threadIdx.x & 31) == 0 && rmask) atomicAdd(&A.ctr->n_recheck, (unsigned long long)__popc(rmask));
  if (!active) return;
  const PairView &o = A.out;
  if (A.perm) o.node[pair] = A.perm[node];
  uint8_t verdict;
  int fi;
  if (first_oob < L) { verdict = DPG_OUT_OF_BOUNDS; fi = first_oob; }
  else if (collided) { verdict = DPG_COLLISION; fi = first_col; }
  else { verdict = DPG_VALID; fi = L; }
  const int er = first_oob < L ? first_oob : L - 1;  // end-state row
  const int64_t row_out = o.out_index ? (int64_t)o.out_index[pair] : pair;
  if (o.node_host) {
    o.node_host[row_out] = A.perm ? A.perm[node] : node;
    o.prim_host[row_out] = (uint32_t)p;
  }
  if (o.verdict) o.verdict[row_out] = verdict;
  if (o.first_invalid) o.first_invalid[row_out] = (int16_t)fi;
  if (o.min_gap)
    o.min_gap[row_out] = verdict == DPG_OUT_OF_BOUNDS ? __int_as_float(0x7fc00000)
                                                   : ((float)mg <= kGapCap ? (float)mg : __int_as_float(0x7f800000));
  if (o.flags) o.flags[row_out] = rechecked ? DPG_FLAG_CONTACT_RECHECK : 0;
  if (ES64 && o.end_state) {
    double *es = (double *)o.end_state + row_out * R::NX;
    const double t = double(er) * rp.dt;
    const double *xs = pv.st64 + (s0 + er) * R::NX;
#pragma unroll
    for (int c = 0; c < R::NX; c++) {
      double v = xs[c];
      if (c < D) {
        v += x64[c];
        if (V) v += t * x64[R::vel_comp(c)];
      }
#pragma unroll
      for (int i = 0; i < V; i++)
        if (c == R::vel_comp(i)) v += x64[R::vel_comp(i)];
      es[c] = v;
    }
  } else if (o.end_state) {
    Real *es = (Real *)o.end_state + row_out * R::NX;
    const Real t = Real(er) * dtR;
    const int64_t row = s0 + er;
#pragma unroll
    for (int c = 0; c < R::NX; c++) {
      Real v = sizeof(Real) == 4 ? Real(pv.st32[row * R::NXP + c]) : Real(pv.st64[row * R::NX + c]);
      if (c < D) {
        v += off[c];
        if (V) v += t * off[D + c];
      }
#pragma unroll
      for (int i = 0; i < V; i++)
        if (c == R::vel_comp(i)) v += off[D + i];
      es[c] = v;
    }
  }
}

// ------------------------------------------------- slot-parallel variant --
//
// The lockstep walk above makes every state cost the largest candidate count
// of any lane: lanes with fewer candidates (most have none) wait.  Here the
// warp goes through the primitive in windows of WIN chunks of R::CHUNK
// states and gives every test to a lane of its own:
//   - slots (lane, obstacle): the union of the lanes' window boxes selects the
//     obstacles near any lane (a lane per obstacle, one ballot per 32), each of
//     these is tested against the 32 lanes' boxes, and the lanes it is near to
//     append their slots;
//   - a lane per slot tests its obstacle against the boxes of each part over
//     the window's chunks at its owner's offset (a bit per chunk and part);
//   - the bounds are tested with a lane per (lane, state of a chunk);
//   - the near (slot, part, chunk) entries are listed in the chunks' order and
//     tested with a lane per (entry, state), 32 / CHUNK entries a step, up to
//     the owner's first state out of bounds.
// Per lane the first state out of bounds, the first contact and the first FP64
// decisions are kept in shared memory (one atomic per entry with a contact):
// decisions after the first contact do not count, which gives exactly the
// results of the sequential walk (every candidate is tested at every state up
// to the first contact).  FP32 tests with FP64 decisions in the band.
//
// Bound by instruction issue (77 % of the issue slots on car1, 27.1 active
// lanes an instruction, 82 % and 26.6 on the quadrotor; its table reads hit L1 / L2).  Check kernel, ms, against
// the form that dealt (lane, chunk, obstacle) slots out and walked a slot's
// states in one lane (17.7 active lanes), and against the first form of this
// one (a box for all parts of a chunk, bounds and tests chunk by chunk, every
// axis of an ambiguous test in FP64):
//   car1 100,000 x 5,000          1.91   1.34   1.03
//   quadrotor 50,000 x 5,000     10.6    6.6    5.2
//   unicycle1 FP64 10,000 x 1,000 0.127  0.106  0.098
//   quad2d 32 x 10,000            0.168  0.121  0.090
// Measured beside it: a lane walking its own states in the bounds tests when
// many lanes need them, quadrotor 6.6 -> 8.7; entries of several chunks listed
// before they are tested (fuller steps, but lanes past their contact), car1
// 1.06 at 4 entries, 1.08 at 12, 1.36 at 32; windows of 8 chunks instead of 4
// car1 1.06, of 4 instead of 2 the quadrotor 5.26; chunks of 8 or 32 states for
// the quadrotor 6.65 and 8.9 (first form); 3 blocks an SM car1 1.18, 5 (spills)
// 1.75.  End-state rows of 52 bytes written by a lane each cost the quadrotor
// 2.2 ms: they go out through shared memory.

constexpr int kSlotCap = 512;  // slots of a window held at a time; also the most obstacles of this variant
// Slots expected of a window from which it is WINDOW_MANY chunks: lanes meet an
// obstacle early there, and a long window's slots do not fit.  The line lies where
// both lengths take about the same time (quad2d, 8 and 3 chunks: random motions, 40
// obstacles of up to 1 m on 32 square metres, 355 slots expected: 145 and 131 us, 100
// smaller ones, 715: 289 and 197; hover motions, 65 obstacles, 63: 387 and 481, 128
// obstacles, 90: 571 and 721).
constexpr double kManySlots = 400;
constexpr int kListCap = 160;  // entries held at a time
constexpr int kListMin = 4;    // entries from which a listed chunk is tested at once
constexpr int kNever = 0x7fffffff;

template <int KIND, bool ES64> struct SlotScratch {
  static constexpr int C = Robot<KIND>::POSD + Robot<KIND>::VELOFF;
  using Es = std::conditional_t<ES64, double, float>;
  union {
    struct {
      // chunk of the window << 16 | part << 14 | obstacle << 5 | lane; bounds: lane
      uint32_t list[kListCap];
      uint16_t slot[kSlotCap];  // obstacle << 5 | lane
      std::conditional_t<Robot<KIND>::PARTS == 1, uint8_t, uint16_t>
          near_[kSlotCap];  // the window's chunks (8 bits a part) the slot's obstacle is near to
    };
    Es end[32 * Robot<KIND>::NX];  // the item's end states on their way out
  };
  float off[C][32];  // the lanes' node offsets
  uint32_t node[32];
  // per lane, the first state: out of bounds (L: none), with a contact, with a
  // bounds / an obstacle test decided in FP64 (kNever: none)
  int oob[32], contact[32], oob_amb[32], contact_amb[32];
};
// (with the min_gap output the warp's scratch is followed by (CHUNK + 1) x 32
// words: per state of the chunk and lane, the min axis-aligned gap as ordered
// bits, then each lane's minimum so far)

template <int KIND, bool ES64>
constexpr size_t slot_scratch_bytes(bool min_gap) {
  return (sizeof(SlotScratch<KIND, ES64>) + (min_gap ? sizeof(unsigned) * 32 * (Robot<KIND>::CHUNK + 1) : 0) + 15) / 16 * 16;
}

__device__ __forceinline__ unsigned ord_gap(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unord_gap(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// FP64 decision of an ambiguous obstacle test of part q at state k (rare: kept
// out of line).  Planar robots: an axis whose FP32 gap (px, py, c, s: the FP32
// pose) is below the band by more than the FP32 error is below zero in FP64
// too, so only the others, usually one, are evaluated (all four: 27 FP64
// instructions at 16 SM cycles each, an eighth of car1's check).
template <int KIND>
__device__ __noinline__ bool contact64(const CheckArgs &A, int p, int k, int q, uint32_t node, int o, float px,
                                       float py, float c, float s) {
  using R = Robot<KIND>;
  const double *x64 = A.nv.x64 + (int64_t)node * R::NX;
  const int64_t s0 = A.pv.soff[p];
  if constexpr (R::SPHERE) {
    return gap64<KIND>(A, s0, k, q, x64, o) <= 0.0;
  } else {
    const Obs2<float> of = ((const Obs2<float> *)A.ev.obs32)[o];
    const Obs2<double> ob = ((const Obs2<double> *)A.ev.obs64)[o];
    const Pose<double> ps = A.pv.pose64[q * A.pv.S + s0 + k];
    const float a32 = A.half_len32, b32 = A.half_wid32, fc = fabsf(c), fs = fabsf(s), dxf = px - of.cx, dyf = py - of.cy;
    const float cut = -(A.band32 + 1e-4f + 1e-6f * (fabsf(px) + fabsf(py)));
    double sx = x64[0], sy = x64[1];
    if (R::VELOFF) {
      const double t = double(k) * A.rp.dt;
      sx += t * x64[R::vel_comp(0)];
      sy += t * x64[R::vel_comp(1)];
    }
    const double a = A.rp.half_len, b = A.rp.half_wid, ac = fabs(ps.c), as = fabs(ps.s);
    const double dx = ps.cx + sx - ob.cx, dy = ps.cy + sy - ob.cy;
    bool in = true;
    if (fabsf(dxf) - (a32 * fc + b32 * fs + of.hx) > cut) in = fabs(dx) - (a * ac + b * as + ob.hx) <= 0.0;
    if (in && fabsf(dyf) - (a32 * fs + b32 * fc + of.hy) > cut) in = fabs(dy) - (a * as + b * ac + ob.hy) <= 0.0;
    if (in && fabsf(dxf * c + dyf * s) - (a32 + of.hx * fc + of.hy * fs) > cut)
      in = fabs(dx * ps.c + dy * ps.s) - (a + ob.hx * ac + ob.hy * as) <= 0.0;
    if (in && fabsf(dyf * c - dxf * s) - (b32 + of.hx * fs + of.hy * fc) > cut)
      in = fabs(-dx * ps.s + dy * ps.c) - (b + ob.hx * as + ob.hy * ac) <= 0.0;
    return in;
  }
}
// FP64 decision of an ambiguous bounds test of position component i
template <int KIND>
__device__ __noinline__ bool outside64(const CheckArgs &A, int p, int k, uint32_t node, int i) {
  const double v = pos64<KIND>(A, A.pv.soff[p] + k, k, A.nv.x64 + (int64_t)node * Robot<KIND>::NX, i);
  return !(v >= A.ev.lo[i] && v <= A.ev.hi[i]);
}

// Bounds test of state k (pose ps) for the lane whose offsets are in column
// `own` of S; `amb` set when a component was decided in FP64.
template <int KIND, class Scratch>
__device__ __forceinline__ bool out_of_bounds(const CheckArgs &A, const Scratch &S, const Pose<float> &ps, int p, int k,
                                              int own, bool &amb) {
  using R = Robot<KIND>;
  constexpr int D = R::POSD, V = R::VELOFF;
  const float tk = float(k) * A.dt32;
  float osh[D + V];
#pragma unroll
  for (int i = 0; i < D + V; i++) osh[i] = S.off[i][own];
  const float pv3[3] = {ps.cx + osh[0] + (V ? tk * osh[D] : 0.f), ps.cy + osh[1] + (V ? tk * osh[D + 1] : 0.f),
                        D == 3 ? ps.c + osh[2] + (V ? tk * osh[D + 2] : 0.f) : 0.f};
  int bt = 0;
#pragma unroll
  for (int i = 0; i < D; i++) {
    const float v = pv3[i];
    int r = (v < A.lo_out[i] || v > A.hi_out[i]) ? 1 : ((v <= A.lo_in[i] || v >= A.hi_in[i]) ? 2 : 0);
    if (r == 2) {  // decide in FP64
      r = outside64<KIND>(A, p, k, S.node[own], i) ? 1 : 0;
      amb = true;
    }
    bt |= r;
  }
  return bt != 0;
}

// centre and half extents of the culling box at `box` (D centres, D halves)
template <int D>
__device__ __forceinline__ void load_box(const float *box, float *c, float *h) {
  if constexpr (D == 2) {
    const float4 v = *reinterpret_cast<const float4 *>(box);
    c[0] = v.x; c[1] = v.y; h[0] = v.z; h[1] = v.w;
  } else {
    const float2 *v = reinterpret_cast<const float2 *>(box);
    const float2 v0 = v[0], v1 = v[1], v2 = v[2];
    c[0] = v0.x; c[1] = v0.y; c[2] = v1.x; h[0] = v1.y; h[1] = v2.x; h[2] = v2.y;
  }
}

// This lane is the first of its group of CH lanes in the ballot m (it is one of m).
template <int CH>
__device__ __forceinline__ bool first_of_group(unsigned m, int lane) {
  return ((m >> (lane & ~(CH - 1))) & ((1u << (lane & (CH - 1))) - 1u)) == 0u;
}

template <int KIND, bool ES64, int WIN>
__device__ __forceinline__ void check_item(const CheckArgs &A, const void *obs_sm, SlotScratch<KIND, ES64> &S, int p,
                                           uint32_t pair0, int count, uint32_t node) {
  using R = Robot<KIND>;
  using Ob = std::conditional_t<R::SPHERE, Obs3<float>, Obs2<float>>;
  constexpr int D = R::POSD, V = R::VELOFF, CH = R::CHUNK, PARTS = R::PARTS;
  constexpr int NE = 32 / CH;  // entries a step tests at once
  static_assert(32 % CH == 0 && WIN <= 8, "a lane per (entry, state); a byte of chunk bits");
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const bool active = lane < count;
  const PrimView &pv = A.pv;
  const int L = pv.len[p], n_chunks = (L + CH - 1) / CH;
  const float dt = A.dt32, M = A.cull_margin;
  const int n_obs = A.ev.n_obs;
  const PairView &o = A.out;
  const bool want_mg = o.min_gap != nullptr;
  unsigned *mgs = reinterpret_cast<unsigned *>(&S + 1);  // [CH + 1][32] with min_gap

#pragma unroll
  for (int i = 0; i < D; i++) S.off[i][lane] = active ? node_off<float>(A.nv, node, i, R::NX, i) : 0.f;
#pragma unroll
  for (int i = 0; i < V; i++)
    S.off[D + i][lane] = active ? node_off<float>(A.nv, node, D + i, R::NX, R::vel_comp(i)) : 0.f;
  S.node[lane] = node;
  S.oob[lane] = L;
  S.contact[lane] = S.oob_amb[lane] = S.contact_amb[lane] = kNever;
  if (want_mg)
    for (int i = 0; i <= CH; i++) mgs[32 * i + lane] = 0xffffffffu;
  if (active && (A.perm || o.node_host)) {  // the pair's node in the caller's numbering
    const uint32_t n = A.perm ? A.perm[node] : node;
    if (A.perm) o.node[pair0 + lane] = n;
    if (o.node_host) {
      o.node_host[pair0 + lane] = n;
      o.prim_host[pair0 + lane] = (uint32_t)p;
    }
  }

  // bounds pre-check on the swept box of the positions (as check_one)
  bool need_bounds;
  {
    const float *bx32 = pv.pbox32 + (int64_t)p * 2 * D;
    const float tmax = float(L - 1) * dt;
    bool inside = true;
#pragma unroll
    for (int i = 0; i < D; i++) {
      const float off = S.off[i][lane];
      float lo = bx32[i] + off, hi = bx32[D + i] + off;
      if constexpr (V > 0) {
        const float sv = tmax * S.off[D + i][lane];
        lo += fminf(sv, 0.f);
        hi += fmaxf(sv, 0.f);
      }
      inside = inside && lo > A.lo_box[i] && hi < A.hi_box[i];
    }
    need_bounds = active && !inside;
  }

  bool live = active, collided = false;
  const int j = lane % CH, sub = lane / CH;  // this lane's state of a chunk and its entry of a step
  const Pose<float> *pose = pv.pose32 + pv.soff[p];
  const float *cbox = pv.cbox32 + pv.coff[p] * 2 * D, *qbox = pv.qbox32 + pv.coff[p] * (PARTS * 2 * D);
  __syncwarp();

  for (int c0 = 0; c0 < n_chunks; c0 += WIN) {
    unsigned rest = __ballot_sync(kFull, live);  // lanes whose window is still to check
    if (!rest) break;
    const int nc = min(WIN, n_chunks - c0);
    // the lane's box over the window: the union of its chunks' boxes, moved by
    // the offset (and the velocity over the window's time); the chunks in
    // which the lane's box is not inside the bounds
    float cen[D], hf[D];
    unsigned nbw = 0u;
    const bool any_nb = __any_sync(kFull, live && need_bounds);
    {
      float lo[D], hi[D];
#pragma unroll
      for (int i = 0; i < D; i++) { lo[i] = INFINITY; hi[i] = -INFINITY; }
      for (int c = 0; c < nc; c++) {
        float cc[D], ch[D];
        load_box<D>(cbox + (c0 + c) * 2 * D, cc, ch);
#pragma unroll
        for (int i = 0; i < D; i++) {
          lo[i] = fminf(lo[i], cc[i] - ch[i]);
          hi[i] = fmaxf(hi[i], cc[i] + ch[i]);
        }
        if (any_nb) {
          const int k0 = (c0 + c) * CH;
          const float t0 = float(k0) * dt, t1 = float(min(L, k0 + CH) - 1) * dt;
          bool in = true;
#pragma unroll
          for (int i = 0; i < D; i++) {
            float x = cc[i] + S.off[i][lane], h = ch[i];
            if constexpr (V > 0) {
              const float v = S.off[D + i][lane];
              x += 0.5f * (t0 + t1) * v;
              h += 0.5f * (t1 - t0) * fabsf(v);
            }
            in = in && x - h > A.lo_box[i] && x + h < A.hi_box[i];
          }
          if (!in) nbw |= 1u << c;
        }
      }
      if (!(live && need_bounds)) nbw = 0u;
      const float tm0 = float(c0 * CH) * dt, tm1 = float(min(L, (c0 + nc) * CH) - 1) * dt;
#pragma unroll
      for (int i = 0; i < D; i++) {
        cen[i] = 0.5f * (lo[i] + hi[i]) + S.off[i][lane];
        hf[i] = 0.5f * (hi[i] - lo[i]);
        if constexpr (V > 0) {
          const float v = S.off[D + i][lane];
          cen[i] += 0.5f * (tm0 + tm1) * v;
          hf[i] += 0.5f * (tm1 - tm0) * fabsf(v);
        }
      }
    }

    // bounds: the (lane, chunk) entries of each chunk, tested with a lane per
    // (entry, state), so that a lane out of bounds has none in later chunks
    if (any_nb) {
      for (unsigned todo = __reduce_or_sync(kFull, nbw); todo; todo &= todo - 1) {
        const int c = __ffs(todo) - 1, k = (c0 + c) * CH + j;
        const bool nb = ((nbw >> c) & 1u) && S.oob[lane] == L;
        const unsigned nbm = __ballot_sync(kFull, nb);
        if (!nbm) continue;
        const Pose<float> ps = pose[min(k, L - 1)];
        const int n = __popc(nbm);
        if (nb) S.list[__popc(nbm & lt)] = (uint32_t)lane;
        __syncwarp();
        for (int i0 = 0; i0 < n; i0 += NE) {
          const int i = i0 + sub;
          bool out = false, amb = false;
          int own = 0;
          if (i < n && k < L) {
            own = (int)S.list[i];
            out = out_of_bounds<KIND>(A, S, ps, p, k, own, amb);
          }
          const unsigned ow = __ballot_sync(kFull, out), aw = __ballot_sync(kFull, amb);
          if (out && first_of_group<CH>(ow, lane)) S.oob[own] = k;
          if (aw && amb && first_of_group<CH>(aw, lane)) atomicMin(&S.oob_amb[own], k);
        }
        __syncwarp();
      }
    }

    // (usually one pass: all lanes; more slots than the list holds: as many
    // lanes as fit, then the others)
    rest = __ballot_sync(kFull, live && !collided);
    while (rest) {
      unsigned take = rest;
      int n_slot;
      while (true) {
        n_slot = 0;
        const bool inc = (take >> lane) & 1u;
        // union of the lanes' boxes, a little wider than their own tests (a
        // lane with a NaN offset is near no obstacle and stays out of it)
        float ulo[D], uhi[D];
#pragma unroll
        for (int i = 0; i < D; i++) {
          const float lo = cen[i] - hf[i], hi = cen[i] + hf[i];
          const bool ok = inc && lo <= hi;
          ulo[i] = unord_gap(__reduce_min_sync(kFull, ok ? ord_gap(lo) : ord_gap(INFINITY)));
          uhi[i] = unord_gap(__reduce_max_sync(kFull, ok ? ord_gap(hi) : ord_gap(-INFINITY)));
          const float m = M + 1e-3f + 1e-6f * (fabsf(ulo[i]) + fabsf(uhi[i]));
          ulo[i] -= m;
          uhi[i] += m;
        }
        for (int w0 = 0; w0 < n_obs; w0 += 32) {
          bool u = w0 + lane < n_obs;
          if (u) {
            const Ob ob = ((const Ob *)obs_sm)[w0 + lane];
            u = ob.cx + ob.hx >= ulo[0] && ob.cx - ob.hx <= uhi[0] && ob.cy + ob.hy >= ulo[1] && ob.cy - ob.hy <= uhi[1];
            if constexpr (D == 3) u = u && ob.cz + ob.hz >= ulo[2] && ob.cz - ob.hz <= uhi[2];
          }
          for (unsigned m = __ballot_sync(kFull, u); m; m &= m - 1) {
            const int ob = w0 + __ffs(m) - 1;
            const bool h = inc && near_box<D, float>(cen, hf, obs_sm, ob, M);
            const unsigned hm = __ballot_sync(kFull, h);
            const int pos = n_slot + __popc(hm & lt);
            if (h && pos < kSlotCap) S.slot[pos] = (uint16_t)(ob << 5 | lane);
            n_slot += __popc(hm);
          }
        }
        if (n_slot <= kSlotCap) break;
        // one lane always fits (at most kSlotCap obstacles): halve the set
        for (int k = __popc(take) / 2; k > 0; k--) take &= ~(0x80000000u >> __clz(take));
      }
      rest &= ~take;
      __syncwarp();
      // the window's chunks each slot is near to
      unsigned near_any = 0u;
      for (int b = lane; b < n_slot; b += 32) {
        const unsigned e = S.slot[b];
        const int own = (int)(e & 31u);
        const Ob ob = ((const Ob *)obs_sm)[e >> 5];
        float r[D], v[D], h[D];  // owner's offset from the obstacle's centre
        r[0] = S.off[0][own] - ob.cx;
        h[0] = ob.hx + M;
        r[1] = S.off[1][own] - ob.cy;
        h[1] = ob.hy + M;
        if constexpr (D == 3) {
          r[2] = S.off[2][own] - ob.cz;
          h[2] = ob.hz + M;
        }
#pragma unroll
        for (int i = 0; i < D; i++) v[i] = V > 0 ? S.off[(V > 0 ? D : 0) + i][own] : 0.f;
        unsigned near = 0u;
#pragma unroll 4
        for (int c = 0; c < nc; c++) {
#pragma unroll
          for (int q = 0; q < PARTS; q++) {
            float cc[D], ch[D];
            load_box<D>(qbox + ((c0 + c) * PARTS + q) * 2 * D, cc, ch);
            bool in = true;
            if constexpr (V > 0) {
              const int k0 = (c0 + c) * CH, k1 = min(L, k0 + CH) - 1;
              const float tm = 0.5f * dt * float(k0 + k1), th = 0.5f * dt * float(k1 - k0);
#pragma unroll
              for (int i = 0; i < D; i++) in = in && fabsf(cc[i] + tm * v[i] + r[i]) <= ch[i] + th * fabsf(v[i]) + h[i];
            } else {
#pragma unroll
              for (int i = 0; i < D; i++) in = in && fabsf(cc[i] + r[i]) <= ch[i] + h[i];
            }
            if (in) near |= 1u << (8 * q + c);
          }
        }
        S.near_[b] = near;
        near_any |= near;
      }
      near_any = __reduce_or_sync(kFull, near_any);
      if (PARTS > 1) near_any = (near_any | near_any >> 8) & 0xffu;
      __syncwarp();

      // obstacle tests: the near (slot, part) entries of the chunks in order,
      // listed until there are enough of them (a chunk at a time with min_gap,
      // whose gaps are kept per state of a chunk), then tested with a lane per
      // (entry, state)
      unsigned free_m = take;  // lanes of this pass without a contact yet
      int n_ent = 0, b = 0;
      while (near_any) {
        const int c = __ffs(near_any) - 1;
        for (; b < n_slot && n_ent <= kListCap - 32 * PARTS; b += 32) {
          unsigned near = b + lane < n_slot ? S.near_[b + lane] >> c : 0u;
          const unsigned e = near ? S.slot[b + lane] : 0u;
          if (!((free_m >> (e & 31u)) & 1u)) near = 0u;
#pragma unroll
          for (int q = 0; q < PARTS; q++) {
            const bool in = (near >> (8 * q)) & 1u;
            const unsigned m = __ballot_sync(kFull, in);
            if (in) S.list[n_ent + __popc(m & lt)] = (uint32_t)c << 16 | (uint32_t)q << 14 | e;
            n_ent += __popc(m);
          }
        }
        const bool whole = b >= n_slot;  // all of the chunk is listed
        if (whole) {
          b = 0;
          near_any &= near_any - 1;
          if (near_any && !want_mg && n_ent < kListMin) continue;
        }
        __syncwarp();
        for (int i0 = 0; i0 < n_ent; i0 += NE) {
          const bool in = i0 + sub < n_ent;
          const unsigned e = in ? S.list[i0 + sub] : 0u;
          const int own = (int)(e & 31u), ob_i = (int)(e >> 5 & (kSlotCap - 1u));
          const int k = (c0 + (int)(e >> 16)) * CH + j;
          bool hit = false, amb = false;
          if (in && k < S.oob[own] && k <= S.contact[own]) {
            const int q = PARTS > 1 ? (int)(e >> 14 & 1u) : 0;
            const Pose<float> ps = pose[(PARTS > 1 ? q * pv.S : 0) + k];
            const Ob ob = ((const Ob *)obs_sm)[ob_i];
            float sx = S.off[0][own], sy = S.off[1][own], sz = D == 3 ? S.off[D - 1][own] : 0.f;
            if constexpr (V > 0) {
              const float tk = float(k) * dt;
              sx += tk * S.off[D][own];
              sy += tk * S.off[D + 1][own];
              if constexpr (D == 3) sz += tk * S.off[D + 2][own];
            }
            float gmin = INFINITY;
            int r;
            if constexpr (R::SPHERE) {
              r = sphere_test<float, true>(ps.cx + sx, ps.cy + sy, ps.c + sz, ob, A.radius32, A.band32, gmin);
            } else {
              const float ac = fabsf(ps.c), as = fabsf(ps.s), hl = A.half_len32, hw = A.half_wid32;
              r = planar_test<float, true>(ps.cx + sx, ps.cy + sy, ps.c, ps.s, dot2(hl, ac, hw, as),
                                           dot2(hl, as, hw, ac), ob, hl, hw, A.band32, gmin);
            }
            if (r == 2) {  // decide in FP64
              r = contact64<KIND>(A, p, k, q, S.node[own], ob_i, ps.cx + sx, ps.cy + sy, ps.c, ps.s) ? 1 : 0;
              amb = true;
            }
            hit = r == 1;
            // gaps above the cap are reported as +inf: only smaller ones are merged
            if (want_mg && gmin <= kGapCap) atomicMin(&mgs[32 * j + own], ord_gap(gmin));
          }
          const unsigned hb = __ballot_sync(kFull, hit);
          if (hit && first_of_group<CH>(hb, lane)) atomicMin(&S.contact[own], k);
          if (amb) atomicMin(&S.contact_amb[own], k);
        }
        n_ent = 0;
        __syncwarp();
        // (a contact found amid a chunk may not be the chunk's first)
        if (!whole) continue;
        if (S.contact[lane] != kNever) collided = true;
        if (want_mg) {
          const int k0 = (c0 + c) * CH, last = S.contact[lane];
          unsigned mg = mgs[32 * CH + lane];
          for (int i = 0; i < CH; i++) {
            if (k0 + i <= last) mg = min(mg, mgs[32 * i + lane]);
            mgs[32 * i + lane] = 0xffffffffu;
          }
          mgs[32 * CH + lane] = mg;
          __syncwarp();
        }
        free_m &= __ballot_sync(kFull, !collided);
        if (!free_m) break;
      }
      __syncwarp();  // the next pass rewrites the slots
    }
    if ((collided && !need_bounds) || S.oob[lane] != L) live = false;
  }

  // what was tested after a lane's first contact or first state out of bounds does not count
  const int first_oob = S.oob[lane], first_contact = S.contact[lane];
  const bool oob = first_oob < L;
  const int fi = oob ? first_oob : (collided ? first_contact : L);
  const bool rechecked = (S.oob_amb[lane] != kNever && S.oob_amb[lane] <= first_oob) ||
                         (S.contact_amb[lane] != kNever && S.contact_amb[lane] <= first_contact);
  const unsigned rmask = __ballot_sync(kFull, active && rechecked);
  if (lane == 0 && rmask) atomicAdd(&A.ctr->n_recheck, (unsigned long long)__popc(rmask));
  const uint32_t row_out = active && o.out_index ? o.out_index[pair0 + lane] : pair0 + lane;
  if (active) {
    const uint8_t verdict = oob ? DPG_OUT_OF_BOUNDS : (collided ? DPG_COLLISION : DPG_VALID);
    if (o.verdict) o.verdict[row_out] = verdict;
    if (o.first_invalid) o.first_invalid[row_out] = (int16_t)fi;
    if (want_mg) {  // (no gap up to the cap: NaN bits, reported as +inf)
      const float mg = unord_gap(mgs[32 * CH + lane]);
      o.min_gap[row_out] = oob ? __int_as_float(0x7fc00000) : (mg <= kGapCap ? mg : __int_as_float(0x7f800000));
    }
    if (o.flags) o.flags[row_out] = rechecked ? DPG_FLAG_CONTACT_RECHECK : 0;
  }
  if (!o.end_state) return;
  // end states: each lane its row, then through shared memory so that the
  // stores of the item's rows are coalesced
  using Es = std::conditional_t<ES64, double, float>;
  Es *es = (Es *)o.end_state;
  Es v[R::NX];
  const int er = oob ? fi : L - 1;  // end-state row
  const int64_t s0 = pv.soff[p];
  if constexpr (ES64) {
    const double *st = pv.st64 + (s0 + er) * R::NX;
#pragma unroll
    for (int c = 0; c < R::NX; c++) v[c] = st[c];
    const double *x64 = A.nv.x64 + (int64_t)node * R::NX;
    const double t = double(er) * A.rp.dt;
#pragma unroll
    for (int i = 0; i < D; i++) {
      v[i] += x64[i];
      if (V) v[i] += t * x64[R::vel_comp(i)];
    }
#pragma unroll
    for (int i = 0; i < V; i++) v[R::vel_comp(i)] += x64[R::vel_comp(i)];
  } else {
    const float4 *st = reinterpret_cast<const float4 *>(pv.st32 + (s0 + er) * R::NXP);
#pragma unroll
    for (int c = 0; c < R::NXP / 4; c++) {
      const float4 x = st[c];
      const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (4 * c + i < R::NX) v[4 * c + i] = xs[i];
    }
    const float t = float(er) * dt;
#pragma unroll
    for (int i = 0; i < D; i++) {
      v[i] += S.off[i][lane];
      if constexpr (V > 0) v[i] += t * S.off[D + i][lane];
    }
    if constexpr (V > 0) {
#pragma unroll
      for (int i = 0; i < V; i++) v[R::vel_comp(i)] += S.off[D + i][lane];
    }
  }
  if (o.out_index) {  // rows of their own
    if (active)
#pragma unroll
      for (int c = 0; c < R::NX; c++) es[(int64_t)row_out * R::NX + c] = v[c];
    return;
  }
#pragma unroll
  for (int c = 0; c < R::NX; c++) S.end[lane * R::NX + c] = v[c];
  __syncwarp();
  Es *dst = es + (int64_t)pair0 * R::NX;
#pragma unroll
  for (int e = 0; e < 32 * R::NX; e += 32)
    if (e + lane < count * R::NX) dst[e + lane] = S.end[e + lane];
}

template <class Real, int KIND>
__device__ void load_obstacles(const EnvView &ev, void *sm) {
  using R = Robot<KIND>;
  if constexpr (R::SPHERE) {
    const Obs3<Real> *src = (const Obs3<Real> *)(sizeof(Real) == 4 ? ev.obs32 : ev.obs64);
    Obs3<Real> *dst = (Obs3<Real> *)sm;
    for (int i = threadIdx.x; i < ev.n_obs; i += blockDim.x) dst[i] = src[i];
  } else {
    const Obs2<Real> *src = (const Obs2<Real> *)(sizeof(Real) == 4 ? ev.obs32 : ev.obs64);
    Obs2<Real> *dst = (Obs2<Real> *)sm;
    for (int i = threadIdx.x; i < ev.n_obs; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
}

// The abort flag lies in host memory: a read of it crosses the host link, and
// the link serves about 150 M such reads a second whatever the SMs do, so a
// read per item bounded the whole check (car1, 100,000 nodes x 5,000 motions,
// 260,000 items: 1.73 ms for fetching the items alone, 0.18 ms without the
// reads).  So a warp reads it when it takes up every kAbortPoll-th item of the
// launch, the first included (one read in a few hundred nanoseconds of a full
// GPU); on an abort it moves the launch's item counter past its end.
constexpr uint32_t kAbortPoll = 64;
// Items a warp at the end of a launch that are drawn one by one.  Drawn ahead,
// each waited for its warp's current item: 3,000 unicycle nodes x 1,000 motions
// among 700 obstacles (walked lockstep) 3.6 ms, 2.8 with the last 2, 4 or 8 a
// warp drawn late (one by one throughout, with a host read each, 3.2); 1,500
// cars in FP64 3.05, 2.69; the quadrotor's slots, 33 items a warp, 0.897, 0.891.
constexpr uint32_t kTail = 8;
constexpr uint32_t kUndrawn = 0xffffffffu;
constexpr unsigned long long kNoMoreItems = 1ull << 62;

// Persistent warps over (primitive, 32 nodes) work items: item(p, pair, count,
// node) for each, `pair` its first pair, `count` (<= 32) its pairs, `node` the
// lane's node.
template <class Item>
__device__ __forceinline__ void for_items(const CheckArgs &A, Item item_fn) {
  const int lane = threadIdx.x & 31;
  // (items and pairs stay below 2^32: the capacity does)
  const unsigned long long n_all = A.ctr->n_items;
  const int nsub = A.nsub > 0 ? A.nsub : 1;
  const uint32_t i_lo = nsub > 1 ? (uint32_t)(n_all * A.sub_cum[A.sub] / A.sub_cum[nsub]) : 0u;
  const uint32_t n_items = (uint32_t)(nsub > 1 ? n_all * A.sub_cum[A.sub + 1] / A.sub_cum[nsub] : n_all);
  int cur_range = -1;    // progress-driven copies: the range of this warp's items,
  uint32_t cur_cnt = 0;  // and how many of them it finished
  auto range_end = [&](int j) {  // first item past range j
    return (uint32_t)(A.ctr->n_items * A.sub_cum[j + 1] / A.sub_cum[A.n_ranges]);
  };
  auto flush_range = [&]() {  // warp-uniform
    if (cur_cnt == 0) return;
    __threadfence();  // this lane's result writes, before the count
    __syncwarp();
    if (lane == 0) {
      const int j = cur_range;
      const uint32_t lo = j > 0 ? range_end(j - 1) : 0u, hi = range_end(j);
      if (atomicAdd(&A.ctr->range_done[j], (unsigned long long)cur_cnt) + cur_cnt == hi - lo) {
        __threadfence_system();
        reinterpret_cast<volatile int *>(A.range_flag)[j] = 1;
      }
    }
    cur_cnt = 0;
  };
  // A warp's first item is its number in the launch (consecutive items on
  // different blocks), the others are drawn from the counter: the next one
  // while the current one is checked, near the launch's end once it is done.
  const uint32_t warps = gridDim.x * (blockDim.x >> 5), w_id = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  uint32_t next = w_id < n_items - i_lo ? i_lo + w_id : n_items;
  auto draw = [&]() {
    if (lane == 0) {
      const unsigned long long drawn = atomicAdd(&A.ctr->next_sub[A.sub], 1ull);
      next = drawn + warps < n_items - i_lo ? i_lo + warps + (uint32_t)drawn : n_items;
    }
  };
  while (true) {
    const uint32_t item = __shfl_sync(kFull, next, 0);
    if (item >= n_items) break;
    if (lane == 0 && (item - i_lo) % kAbortPoll == 0 && *A.abort_flag) {
      A.ctr->status = DPG_ERR_ABORTED;  // every warp's next draw lies past the end
      atomicMax(&A.ctr->next_sub[A.sub], kNoMoreItems);
    }
    if (n_items - item > kTail * warps) draw();
    else next = kUndrawn;
    if (A.n_ranges > 1) {
      int j = 0;
      while (j + 1 < A.n_ranges && item >= range_end(j)) j++;
      if (j != cur_range) {
        flush_range();
        cur_range = j;
      }
      cur_cnt++;
    }
    // order position lo with ord_ibase[lo] <= item < ord_ibase[lo + 1]
    int lo = 0;
    if (A.item_pos) {
      lo = (int)A.item_pos[item];
    } else {
      int hi = A.pv.P;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (A.ord_ibase[mid] <= item) lo = mid; else hi = mid;
      }
    }
    const int p = A.pv.order[lo];
    const uint32_t first = (uint32_t)(A.ord_pbase[lo] + 32ull * (item - A.ord_ibase[lo]));
    const int count = (int)min(32u, (uint32_t)A.ord_pbase[lo + 1] - first);
    const uint32_t node = lane < count ? A.out.node[first + lane] : 0u;
    item_fn(p, first, count, node);
    if (next == kUndrawn) draw();
  }
  if (A.n_ranges > 1) flush_range();
}

// lockstep walk
template <int KIND, class Real, bool BAND, int NW, bool ES64 = false>
__global__ void __launch_bounds__(kCheckThreads, Robot<KIND>::CHECK_BLOCKS) check_pairs(CheckArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  load_obstacles<Real, KIND>(A.ev, smem);
  const int lane = threadIdx.x & 31;
  for_items(A, [&](int p, uint32_t pair, int count, uint32_t node) {
    check_one<KIND, Real, BAND, NW, true, ES64>(A, smem, p, (int64_t)pair + lane, node, lane < count);
  });
}

// slot-parallel tests (FP32 with the band), in windows of WIN chunks; the warps'
// scratch follows the obstacles at A.slot_offset, A.slot_stride bytes apart
template <int KIND, bool ES64, int WIN>
__global__ void __launch_bounds__(kCheckThreads, Robot<KIND>::SLOT_BLOCKS) check_pairs_slots(CheckArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  load_obstacles<float, KIND>(A.ev, smem);
  auto &scr = *reinterpret_cast<SlotScratch<KIND, ES64> *>(smem + A.slot_offset + (threadIdx.x >> 5) * A.slot_stride);
  for_items(A, [&](int p, uint32_t pair, int count, uint32_t node) {
    check_item<KIND, ES64, WIN>(A, smem, scr, p, pair, count, node);
    __syncwarp();  // the next item rewrites the scratch
  });
}

}  // namespace dpg
