// kt_group.cuh -- the exact KS kernel with 4 or 8 lanes per ray.
//
// One lane per ray (k_trace) needs a warp's 32 rays to fill its lanes and
// several warps per scheduler to hide the FP64 latency.  A frame with fewer
// rays is bound by the serial chain of its longest rays: ~150 attempts of 11
// right-hand sides of seven metric evaluations, 150 dependent and independent
// FP64 operations each.  Here the lanes of a group share one ray: every lane
// evaluates its own finite-difference points and carries its axis' components
// of the state, the stage sums and the stages, in registers (there is no
// record in shared memory).  A lane reads the other components with shuffles
// inside the group; step control and events are computed by all lanes of the
// group from the same values, so a group does not diverge in itself.  Every
// value comes from the expressions of the one-lane machine (KSRk4): the
// results are the same bit for bit.
//
// The rules are by rays per SM, 8 lanes up to 90 and 4 up to 540, one above:
// there the lanes are full anyway and the bookkeeping of a ray is paid by every
// lane of its group.  Measured on 148 SMs (ms; 8 lanes / 4 / one with 8 blocks
// per SM), the frames of three scenes:
//    4000 rays   2.2 / 2.3 / 5.5    1.9 / 2.1 / 5.6    3.1 / 3.3 / 7.7
//   12000        2.7 / 2.9 / 6.3    2.4 / 2.7 / 5.7    3.0 / 3.3 / 6.6
//   16000        3.4 / 3.1 / 6.9    2.9 / 2.9 / 6.0    3.1 / 3.4 / 6.9
//   24000        4.7 / 4.3 / 8.5    3.6 / 3.5 / 6.9    4.1 / 4.0 / 7.8
//   57600        7.5 / 7.0 / 9.1    7.8 / 6.8 / 7.3    7.2 / 6.3 / 9.1
//   72000        9.0 / 7.3 / 8.5    9.5 / 7.8 / 7.6    8.7 / 7.2 / 10.5
//   80000        9.8 / 8.1 / 8.9   10.5 / 8.6 / 7.8    9.5 / 7.9 / 9.3
//   90000       11.1 / 9.0 / 8.8   11.7 / 9.5 / 8.1   10.6 / 8.7 / 10.3
//  100000       12.2 / 9.9 / 10.1  12.9 / 10.5 / 8.9  11.6 / 9.5 / 10.4
// (A BL form, 4 lanes on the five points, measured no faster at any size: the
// one-lane right-hand side already has five independent metrics in flight.)
//
// The slot sequence and the queue are k_trace's.
#pragma once

#include "kt_trace_kernel.cuh"

namespace kt {

// Lanes of one ray's group: q within the group, mask of the group's lanes.
struct Lanes {
  unsigned base, mask;
  int q;
};
template <int G>
__device__ __forceinline__ Lanes group_lanes() {
  const unsigned lane = threadIdx.x & 31u;
  Lanes L;
  L.q = (int)(lane & (G - 1));
  L.base = lane & ~(unsigned)(G - 1);
  L.mask = ((G == 32) ? kFull : ((1u << G) - 1u)) << L.base;
  return L;
}
__device__ __forceinline__ double from_lane(const Lanes& L, double v, int q) {
  return __shfl_sync(L.mask, v, (int)L.base + q);
}

// ---- KS chart, G = 4 or 8 lanes ---------------------------------------------
// The lanes of axis a = 0, 1, 2 carry the coordinate and the momentum along it
// and evaluate the points +-eps on it (8 lanes: one point each); the lanes of
// axis 3 evaluate the centre, whose H and l^i every lane turns into its own
// dX^a/dlambda.
template <int G>
__device__ __forceinline__ void ks_rhs_group(const Lanes& L, const Metric& g, const double x[3],
                                             const double p[3], double pT, double k[2]) {
  constexpr int kPer = G / 4;  // lanes per axis
  const int a = L.q / kPer;
  uint32_t top = 0;
  bool ok = (g.tame != 0) & ks_coord_ok(x[0]) & ks_coord_ok(x[1]) & ks_coord_ok(x[2]);
  const double xa = (a == 0) ? x[0] : (a == 1) ? x[1] : x[2];
  const double e = 1e-5 * (fabs(xa) + 0.1);
  const double hi = xa + e, lo = xa - e;
  KSPoint P;
  double d;
  if (G == 8) {
    const double v = (L.q & 1) ? lo : hi;
    P = ks_point<true>(g, a == 0 ? v : x[0], a == 1 ? v : x[1], a == 2 ? v : x[2], &top, &ok);
    const double h = ks_ham2(P, pT, p[0], p[1], p[2]);
    const double other = __shfl_xor_sync(L.mask, h, 1);
    d = (L.q & 1) ? other - h : h - other;
  } else {
    P = ks_point<true>(g, a == 0 ? hi : x[0], a == 1 ? hi : x[1], a == 2 ? hi : x[2], &top, &ok);
    const KSPoint M = ks_point<false>(g, a == 0 ? lo : x[0], a == 1 ? lo : x[1], a == 2 ? lo : x[2],
                                      &top, &ok);
    d = ks_ham2(P, pT, p[0], p[1], p[2]) - ks_ham2(M, pT, p[0], p[1], p[2]);
  }
  if (a == 3) d = 0.0;  // the centre's two Hamiltonians are the same number
  k[1] = ks_slope(d, e, &top, &ok);
  // this axis' row of g^{ab} p_b at the centre (ks_rows)
  const double H = from_lane(L, P.H, 3 * kPer), l1 = from_lane(L, P.l1, 3 * kPer);
  const double l2 = from_lane(L, P.l2, 3 * kPer), l3 = from_lane(L, P.l3, 3 * kPer);
  const double ha = H * ((a == 0) ? l1 : (a == 1) ? l2 : l3);
  k[0] = (((0.0 + ha) * pT + ((a == 0 ? 1.0 : 0.0) - ha * l1) * p[0]) +
          ((a == 1 ? 1.0 : 0.0) - ha * l2) * p[1]) +
         ((a == 2 ? 1.0 : 0.0) - ha * l3) * p[2];
  ok = ok & ((top & kTopBit) == 0u);
  if (!__all_sync(L.mask, ok)) {
    double f[6];
    ks_rhs_rest(g, x[0], x[1], x[2], p[0], p[1], p[2], pT, f);
    k[0] = (a == 0) ? f[0] : (a == 1) ? f[1] : f[2];
    k[1] = (a == 0) ? f[3] : (a == 1) ? f[4] : f[5];
  }
}

template <int G>
struct GroupKSRk4 {
  static constexpr int kLanes = G, kSlots = KSRk4::kSlots, kPer = G / 4;
  double s[2], k1[2], sum[2], kp[2], A[2], B1[2];  // this axis: coordinate, momentum
  double pT, h, step_used, prev_r;
  int it, rejects;
  uint32_t attempts;
  bool need_k1, pending;

  __device__ __forceinline__ bool needs_k1() const { return need_k1; }
  __device__ __forceinline__ bool start(const Lanes& L, const Frame& f, uint32_t pix,
                                        uint32_t out_slot, uint32_t fb_key, const Fallback& fb) {
    KSState ks;
    if (!init_ks_state(f.g, camera_ray(f, pix), &ks)) {
      if (L.q == 0) {
        const uint32_t i = atomicAdd(fb.count, 1u);
        fb.pix[i] = fb_key;
        if (fb.slot) fb.slot[i] = out_slot;
      }
      return false;
    }
    const int a = L.q / kPer;
    s[0] = (a == 0) ? ks.X : (a == 1) ? ks.Y : ks.Z;
    s[1] = (a == 0) ? ks.pX : (a == 1) ? ks.pY : ks.pZ;
    pT = ks.pT;
    h = f.dlam0;
    step_used = h;
    prev_r = r_ks(f.g, ks.X, ks.Y, ks.Z);
    it = 0;
    rejects = 0;
    attempts = 0;
    need_k1 = true;
    pending = false;
    return true;
  }

  __device__ __forceinline__ void gather(const Lanes& L, const double v[2], double x[3],
                                         double p[3]) const {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      x[a] = from_lane(L, v[0], a * kPer);
      p[a] = from_lane(L, v[1], a * kPer);
    }
  }

  __device__ __forceinline__ void stop_at(const Frame& f, const double x[3], int status,
                                          uint32_t steps, RayResult* o) const {
    double rr, tt, pp;
    ks_to_bl(f.g, x[0], x[1], x[2], &rr, &tt, &pp);
    o->steps = steps;
    o->attempts = attempts;
    set_result(o, kOutEscaped, status, rr, 1.0, 1.0, tt, pp, 0.0);
  }

  // KSRk4::events; x is the current position, in every lane.
  __device__ __forceinline__ bool events(const Lanes& L, const Frame& f, const double x[3],
                                         RayResult* o) {
    const double r_now = r_ks(f.g, x[0], x[1], x[2]);
    double best_alpha = 2.0;
    int ev = kEvNone;
    double disk_r = 0.0, disk_red = 1.0, disk_phi = 0.0;
    const double sz = from_lane(L, A[0], 2 * kPer);
    if (sign_change(sz, x[2]) || (dmin(fabs(sz), fabs(x[2])) < 0.35)) {
      double alpha = 0.0;
      bool hit = first_event(sz, x[2], from_lane(L, kp[0], 2 * kPer), from_lane(L, k1[0], 2 * kPer),
                             step_used, 0.0, &alpha);
      if (!hit && sign_change(sz, x[2])) {
        const double denom = sz - x[2];
        alpha = (fabs(denom) > 1e-12) ? (sz / denom) : 0.5;
        alpha = dclamp(alpha, 0.0, 1.0);
        hit = true;
      }
      if (hit) {
        double v[2], xh[3], qh[3];
        for (int i = 0; i < 2; ++i) v[i] = hermite(A[i], s[i], kp[i], k1[i], step_used, alpha);
        gather(L, v, xh, qh);
        double r_hit, th_hit, ph_hit;
        ks_to_bl(f.g, xh[0], xh[1], xh[2], &r_hit, &th_hit, &ph_hit);
        if (r_hit >= f.r_in && r_hit <= f.r_out) {
          const double pphi_bl = ks_pphi_bl(r_hit, th_hit, ph_hit, f.g.a, qh[0], qh[1], qh[2]);
          disk_r = r_hit;
          disk_red = dclamp(disk_redshift(f.g, f.eq, r_hit, pT, pphi_bl), 0.0, 20.0);
          disk_phi = ph_hit;
          best_alpha = alpha;
          ev = kEvDisk;
        }
      }
    }
    horizon_escape(prev_r, r_now, f.rh_cut, f.r_esc, &best_alpha, &ev);
    if (ev != kEvNone) {
      o->steps = (uint32_t)it + 1;
      o->attempts = attempts;
      if (ev == kEvDisk) {
        set_result(o, kOutDisk, kStEvent, disk_r, disk_red, 1.0, disk_phi, 0.0, 0.0);
      } else if (ev == kEvHorizon) {
        set_result(o, kOutHorizon, kStEvent, prev_r + best_alpha * (r_now - prev_r), 0.0, 1.0, 0.0,
                   0.0, 0.0);
      } else {
        const double v = A[0] + best_alpha * (s[0] - A[0]);
        double re, te, pe;
        ks_to_bl(f.g, from_lane(L, v, 0), from_lane(L, v, kPer), from_lane(L, v, 2 * kPer), &re, &te,
                 &pe);
        set_result(o, kOutEscaped, kStEvent, re, 1.0, 1.0, te, pe, 0.0);
      }
      return true;
    }
    prev_r = r_now;
    ++it;
    rejects = 0;
    if (it >= f.max_steps) {
      stop_at(f, x, kStStepCap, (uint32_t)it, o);
      return true;
    }
    return false;
  }

  __device__ __forceinline__ bool slot(const Lanes& L, const Frame& f, int sl, RayResult* o) {
    double y[2], x[3], p[3], k[2];
    if (sl < 0) {
      y[0] = s[0];
      y[1] = s[1];
    } else if (sl == 6) {
      y[0] = B1[0];
      y[1] = B1[1];
    } else {
      const double c = doubling_coeff(sl, h);
      const bool on_s = sl < 6, use_k1 = (sl == 0 || sl == 3);
#pragma unroll
      for (int i = 0; i < 2; ++i) y[i] = (on_s ? s[i] : B1[i]) + c * (use_k1 ? k1[i] : kp[i]);
    }
    gather(L, y, x, p);
    ks_rhs_group<G>(L, f.g, x, p, pT, k);
    switch (sl) {
      case -1:
        for (int i = 0; i < 2; ++i) k1[i] = k[i];
        need_k1 = false;
        if (!pending) return false;
        pending = false;
        return events(L, f, x, o);
      case 0:
      case 3:
        for (int i = 0; i < 2; ++i) {
          sum[i] = k1[i] + 2.0 * k[i];
          kp[i] = k[i];
        }
        return false;
      case 1:
      case 4:
      case 7:
      case 8:
        for (int i = 0; i < 2; ++i) {
          sum[i] = sum[i] + 2.0 * k[i];
          kp[i] = k[i];
        }
        return false;
      case 6:
        for (int i = 0; i < 2; ++i) {
          sum[i] = k[i];
          kp[i] = k[i];
        }
        return false;
      case 2: {
        const double w = h / 6.0;
        for (int i = 0; i < 2; ++i) A[i] = s[i] + w * (sum[i] + k[i]);
        return false;
      }
      case 5: {
        const double w = (0.5 * h) / 6.0;
        for (int i = 0; i < 2; ++i) B1[i] = s[i] + w * (sum[i] + k[i]);
        return false;
      }
      default: {  // 9
        const double w = (0.5 * h) / 6.0;
        double B[2], ee[2], ex[3], ep[3];
        for (int i = 0; i < 2; ++i) {
          B[i] = B1[i] + w * (sum[i] + k[i]);
          const double e = A[i] - B[i];
          ee[i] = e * e;
        }
        gather(L, ee, ex, ep);
        const double err =
            sqrt(((((ex[0] + ex[1]) + ex[2]) + ep[0]) + ep[1]) + ep[2]) / 15.0;
        step_used = h;
        ++attempts;
        if (doubling_update(err, f.tol, &h) == 1) {
          for (int i = 0; i < 2; ++i) {
            A[i] = s[i];    // s_prev
            kp[i] = k1[i];  // f(s_prev)
            s[i] = B[i];
          }
          need_k1 = true;
          pending = true;
          return false;
        }
        int st;
        if (reject_cap(h, &rejects, &st)) {
          double xs[3], ps[3];
          gather(L, s, xs, ps);
          stop_at(f, xs, st, (uint32_t)it, o);
          return true;
        }
        return false;
      }
    }
  }
};

// ---- the persistent loop -----------------------------------------------------
constexpr int kGroupBlock = 64;
constexpr uint32_t kKs8RaysPerSm = 90, kKs4RaysPerSm = 540;

// Blocks per SM: 8 lanes at 128 registers; 4 lanes, which carry two points at a
// time, at 160 without a spill (320 x 180: 6.8 ms against 7.0 with 8 blocks).
template <class M> constexpr int kGroupMinBlocks = M::kLanes == 8 ? 8 : 6;

template <class M>
__global__ void __launch_bounds__(kGroupBlock, kGroupMinBlocks<M>)
    k_trace_group(const __grid_constant__ Frame f, const OutSoA out, const RayList rl,
                  uint32_t* __restrict__ queue, const Fallback fb) {
  constexpr int G = M::kLanes;
  M m;
  const Lanes L = group_lanes<G>();
  bool active = false;
  uint32_t out_slot = 0;
  const uint32_t n = rl.n_dev ? *rl.n_dev : rl.n;
  const unsigned lane = threadIdx.x & 31u;
  bool exhausted = false;
  for (;;) {
    // a warp takes its next 32 / G rays when all of them are done
    if (!exhausted && !__any_sync(kFull, active)) {
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(queue, 32u / G);
      base = __shfl_sync(kFull, base, 0);
      if (base + 32u / G >= n) exhausted = true;
      const unsigned idx = base + lane / G;
      if (idx < n) {
        const uint32_t pix = rl.pix ? rl.pix[idx] : idx;
        out_slot = rl.slot ? rl.slot[idx] : idx;
        active = m.start(L, f, pix, out_slot, pix, fb);
      }
    }
    if (!__any_sync(kFull, active)) {
      if (exhausted) break;
      continue;
    }
    KT_ROLLED
    for (int sl = -1; sl < M::kSlots; ++sl) {
      const bool part = active && (sl >= 0 || m.needs_k1());
      if (sl < 0 && !__any_sync(kFull, part)) continue;
      if (part) {
        RayResult res;
        if (m.slot(L, f, sl, &res)) {
          if (L.q == 0) write_result(out, out_slot, res);
          active = false;
        }
      }
    }
  }
}

// `sms` x resident blocks, or fewer where the rays need fewer.
template <class M>
static cudaError_t launch_group(const Frame& f, const OutSoA& out, const RayList& rl,
                                uint32_t* queue, const Fallback& fb, int sms, cudaStream_t stream) {
  const uint32_t per_block = kGroupBlock / M::kLanes;
  const uint32_t need = (rl.n + per_block - 1) / per_block;
  const uint32_t most = (uint32_t)(sms * kGroupMinBlocks<M>);
  k_trace_group<M><<<need < most ? need : most, kGroupBlock, 0, stream>>>(f, out, rl, queue, fb);
  return cudaGetLastError();
}

}  // namespace kt
