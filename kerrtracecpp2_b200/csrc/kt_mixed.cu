// kt_mixed.cu -- mixed-precision trace kernels (KT_PREC_MIXED); the bundle one is
// in kt_mixed_bundle.cu.
//
// Same persistent loop and the same FP64 integrators as the exact kernels
// (state, stage sums, embedded error estimate, step-size controller, event
// location and the disk-crossing root all stay FP64; in bundle mode the
// Jacobi map W and its determinant too), with a different right-hand side:
// the Hamiltonian gradient is evaluated analytically
// (bl_rhs_analytic / ks_rhs_analytic: one inverse metric with four
// reciprocals instead of five metrics with 26 correctly rounded divisions),
// in FP32 where the tolerance and the geometry allow it, else in FP64.
// FP32 is used for a warp's RHS only when every active lane of the warp is
// beyond r_fp32 and away from a radial or polar turning point, so lanes never
// diverge between the two paths.  This file is compiled with FMA
// contraction on; its results are not bit-identical to the reference and
// are compared with the FP64 oracle statistically.
#include <cmath>

#include "kt_trace_kernel.cuh"

namespace kt {

__device__ __forceinline__ bool warp_all(bool p) { return __all_sync(__activemask(), p); }

// BL: FP32 beyond r_fp32 unless p_r or p_theta/r is small against |p_t|.
__device__ __forceinline__ void bl_rhs_mixed(const Frame& f, const double y[4], double pt,
                                             double pphi, double k[5]) {
  const double lim = f.turn_frac * fabs(pt);
  const bool far = y[0] > f.r_fp32 && fabs(y[2]) > lim && fabs(y[3]) > lim * y[0];
  if (warp_all(far))
    bl_rhs_analytic<float>(f.g, y[0], y[1], y[2], y[3], pt, pphi, k);
  else
    bl_rhs_analytic<double>(f.g, y[0], y[1], y[2], y[3], pt, pphi, k);
}

// The single-ray mixed modes come in two instantiations: kFp32 (some frame
// of the launch has a finite r_fp32) carries the FP32 right-hand side and
// the constraint reprojection; the other, for tolerances below 1e-8, runs
// the FP64 analytic RHS alone, without that code in the kernel.
template <bool kFp32>
struct ModeBLRk4MixedT {
  using Machine = BLRk4;
  static constexpr int kSlots = BLRk4::kSlots;
  BLRk4* m;
  __device__ __forceinline__ bool needs_k1() const { return m->needs_k1(); }
  __device__ __forceinline__ bool start(const Frame& f, uint32_t pix, uint32_t, uint32_t, const Fallback&) {
    m->init(f, camera_ray(f, pix));
    return true;
  }
  __device__ __forceinline__ bool slot(const Frame& f, int s, RayResult* res) {
    double y[4], k[5];
    m->input(s, y);
    if constexpr (kFp32) {
      bl_rhs_mixed(f, y, m->pt, m->pphi, k);
      const int it0 = m->it;
      if (m->consume(f, s, k, res)) return true;
      mixed_after_slot(f, m, s, it0);
      return false;
    } else {
      bl_rhs_analytic<double>(f.g, y[0], y[1], y[2], y[3], m->pt, m->pphi, k);
      return m->consume(f, s, k, res);
    }
  }
};

template <bool kFp32>
struct ModeBLDopri5MixedT {
  using Machine = BLDopri5;
  static constexpr int kSlots = BLDopri5::kSlots;
  BLDopri5* m;
  __device__ __forceinline__ bool needs_k1() const { return m->needs_k1(); }
  __device__ __forceinline__ bool start(const Frame& f, uint32_t pix, uint32_t, uint32_t, const Fallback&) {
    m->init(f, camera_ray(f, pix));
    return true;
  }
  __device__ __forceinline__ bool slot(const Frame& f, int s, RayResult* res) {
    double y[4], k[5];
    m->input(s, y);
    if constexpr (kFp32) {
      bl_rhs_mixed(f, y, m->pt, m->pphi, k);
      const int it0 = m->it;
      if (m->consume(f, s, k, res)) return true;
      mixed_after_slot(f, m, s, it0);
      return false;
    } else {
      bl_rhs_analytic<double>(f.g, y[0], y[1], y[2], y[3], m->pt, m->pphi, k);
      return m->consume(f, s, k, res);
    }
  }
};

// KS: FP32 beyond r_fp32 unless the radial momentum x.p/|x| is small.
// kBlockwise (with kFp32): as blocks that go through the slots together.
template <bool kFp32, bool kBlockwise = false>
struct ModeKSRk4MixedT {
  using Machine = KSRk4;
  static constexpr int kSlots = KSRk4::kSlots;
  KSRk4* m;
  __device__ __forceinline__ bool needs_k1() const { return m->needs_k1(); }
  __device__ __forceinline__ bool start(const Frame& f, uint32_t pix, uint32_t out_slot,
                                        uint32_t fb_key, const Fallback& fb) {
    if (m->init(f, camera_ray(f, pix))) return true;
    const uint32_t i = atomicAdd(fb.count, 1u);
    fb.pix[i] = fb_key;
    if (fb.slot) fb.slot[i] = out_slot;
    return false;
  }
  __device__ __forceinline__ bool slot(const Frame& f, int s, RayResult* res) {
    double y[6], k[6];
    m->input(s, y);
    if constexpr (kFp32) {
      const double rr = sqrt(y[0] * y[0] + y[1] * y[1] + y[2] * y[2]);
      const double prad = (y[0] * y[3] + y[1] * y[4] + y[2] * y[5]) / rr;
      const bool far = rr > f.r_fp32 && fabs(prad) > f.turn_frac * fabs(m->pT);
      if (warp_all(far))
        ks_rhs_analytic<float>(f.g, y[0], y[1], y[2], y[3], y[4], y[5], m->pT, k);
      else
        ks_rhs_analytic<double>(f.g, y[0], y[1], y[2], y[3], y[4], y[5], m->pT, k);
      const int it0 = m->it;
      if (m->consume(f, s, k, res)) return true;
      mixed_after_slot(f, m, s, it0);
      return false;
    } else {
      ks_rhs_analytic<double>(f.g, y[0], y[1], y[2], y[3], y[4], y[5], m->pT, k);
      return m->consume(f, s, k, res);
    }
  }
};

// Launch shapes, measured on B200 as for the exact kernels: refilling a
// warp only when all 32 lanes are idle matters more here, since the FP32/FP64
// choice is made per warp and a warp of neighbouring rays that started
// together makes it alike (720p config 2 DOPRI5: 24.3 against 31.9 ms; BL
// RK4: 25.2 against 41.1; KS RK4: 22.3 against 52.1; 1080p bundles: 224
// against 243).
template <bool B> struct Shape<ModeBLRk4MixedT<B>> { static constexpr int kBlock = 64, kMinBlocks = 9, kRefill = 32; };
// A warp refills once all 32 lanes are idle, so its rays are always the same
// 32 consecutive rays of the queue and the per-warp FP32 choice does not
// depend on the schedule (refilling at 16 idle lanes measured 21.2 ms
// against 22.3 at 720p, tol 1e-8, but mixes the groups).  Block and minimum
// blocks are shared by both instantiations (see launch_shape_mixed).
#ifndef KT_MIXED32_DOPRI5_REFILL
#define KT_MIXED32_DOPRI5_REFILL 32
#endif
#ifndef KT_MIXED_DOPRI5_MINB
#define KT_MIXED_DOPRI5_MINB 9
#endif
template <bool B> struct Shape<ModeBLDopri5MixedT<B>> {
  static constexpr int kBlock = 64, kMinBlocks = KT_MIXED_DOPRI5_MINB,
                       kRefill = B ? KT_MIXED32_DOPRI5_REFILL : 32;
};
// KS with the FP32 branch, from 192 rays per SM on: 256-thread blocks whose
// warps go through the slots together (Lockstep; 512 x 512 6.8 ms, 6.9 as 320 x
// 2, 7.8 as 128 x 5, against 8.1 free-running as 64 x 9).  Fewer rays spread
// over the SMs as free-running blocks of 64.  Measured on 148 SMs (ms of the
// call, free-running / lockstep, three scenes):
//   12000 rays  3.1 / 3.1   2.3 / 2.7   3.4 / 3.5     37000  3.8 / 3.7   3.2 / 2.9   4.7 / 4.6
//   24000       4.2 / 4.2   2.8 / 2.8   4.1 / 4.1     57600  4.6 / 3.9   3.4 / 2.9   4.6 / 4.2
//   30000       4.1 / 3.8   3.1 / 2.9   3.7 / 3.5    130000  4.9 / 4.3   4.2 / 3.6   5.7 / 5.2
// Without the branch 8 blocks of 64 (512 x 512 at tol 1e-9: 3.9 ms against 4.0
// with 10).
constexpr int kKsLockstepRaysPerSm = 192;
template <> struct Shape<ModeKSRk4MixedT<true, true>> { static constexpr int kBlock = 256, kMinBlocks = 2, kRefill = 32; };
template <> struct Lockstep<ModeKSRk4MixedT<true, true>> { static constexpr bool value = true; };
template <> struct Shape<ModeKSRk4MixedT<true>> { static constexpr int kBlock = 64, kMinBlocks = 9, kRefill = 32; };
template <> struct Shape<ModeKSRk4MixedT<false>> { static constexpr int kBlock = 64, kMinBlocks = 8, kRefill = 32; };
template <class ModeT>
static cudaError_t launch_one(const Frame& f, const OutSoA& out, const RayList& rl,
                              uint32_t* queue, const Fallback& fb, const LaunchShape& s,
                              cudaStream_t stream) {
  k_trace<ModeT><<<s.grid, s.block, s.smem, stream>>>(f, out, rl, queue, fb);
  return cudaGetLastError();
}

// The three KS instantiations share their record and differ in block, blocks
// per SM and so in shared memory; s is the free-running FP64 one's shape.
template <class M>
static cudaError_t launch_ks(const Frame& f, const OutSoA& out, const RayList& rl,
                             uint32_t* queue, const Fallback& fb, const LaunchShape& s,
                             cudaStream_t stream) {
  LaunchShape t = s;
  t.block = Shape<M>::kBlock;
  t.grid = s.sms * Shape<M>::kMinBlocks;
  t.smem = smem_bytes<M>(t.block);
  return launch_one<M>(f, out, rl, queue, fb, t, stream);
}

// Both instantiations of a BL mode share its launch bounds, block and shared
// memory, so one shape (the kFp32 one's) serves either.
cudaError_t launch_shape_mixed(Mode mode, int device, LaunchShape* shape) {
  switch (mode) {
    case kModeBLRk4Mixed: return shape_for<ModeBLRk4MixedT<true>>(device, shape);
    case kModeBLDopri5Mixed: return shape_for<ModeBLDopri5MixedT<true>>(device, shape);
    case kModeKSRk4Mixed: {
      // the other instantiations' shared memory is set up here (launch_ks)
      cudaError_t e = shape_for<ModeKSRk4MixedT<true, true>>(device, shape);
      if (e == cudaSuccess) e = shape_for<ModeKSRk4MixedT<true>>(device, shape);
      return e != cudaSuccess ? e : shape_for<ModeKSRk4MixedT<false>>(device, shape);
    }
    case kModeBundleMixed: return launch_shape_mixed_bundle(device, shape);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_trace_mixed(Mode mode, const Frame& f, const OutSoA& out, const RayList& rl,
                               uint32_t* queue, const Fallback& fb, const LaunchShape& s,
                               cudaStream_t stream) {
  const bool fp32 = std::isfinite(f.r_fp32);
  switch (mode) {
    case kModeBLRk4Mixed:
      return fp32 ? launch_one<ModeBLRk4MixedT<true>>(f, out, rl, queue, fb, s, stream)
                  : launch_one<ModeBLRk4MixedT<false>>(f, out, rl, queue, fb, s, stream);
    case kModeBLDopri5Mixed:
      return fp32 ? launch_one<ModeBLDopri5MixedT<true>>(f, out, rl, queue, fb, s, stream)
                  : launch_one<ModeBLDopri5MixedT<false>>(f, out, rl, queue, fb, s, stream);
    case kModeKSRk4Mixed:
      if (!fp32) return launch_one<ModeKSRk4MixedT<false>>(f, out, rl, queue, fb, s, stream);
      return !rl.n_dev && rl.n < (uint32_t)(kKsLockstepRaysPerSm * s.sms)
                 ? launch_ks<ModeKSRk4MixedT<true>>(f, out, rl, queue, fb, s, stream)
                 : launch_ks<ModeKSRk4MixedT<true, true>>(f, out, rl, queue, fb, s, stream);
    case kModeBundleMixed: return launch_trace_mixed_bundle(f, out, rl, queue, fb, s, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t batch_shape_mixed(Mode mode, int variant, int device, LaunchShape* shape) {
  switch (mode) {
    case kModeBLRk4Mixed: return batch_shape<ModeBLRk4MixedT<true>>(variant, device, shape);
    case kModeBLDopri5Mixed: return batch_shape<ModeBLDopri5MixedT<true>>(variant, device, shape);
    case kModeKSRk4Mixed: return batch_shape<ModeKSRk4MixedT<true>>(variant, device, shape);
    case kModeBundleMixed: return batch_shape_mixed_bundle(variant, device, shape);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_batch_mixed(Mode mode, int variant, const BatchRays& br, uint32_t* queue,
                               const Fallback& fb, const LaunchShape& s, cudaStream_t st) {
  switch (mode) {
    case kModeBLRk4Mixed:
      return br.fp32 ? batch_launch<ModeBLRk4MixedT<true>>(variant, br, queue, fb, s, st)
                     : batch_launch<ModeBLRk4MixedT<false>>(variant, br, queue, fb, s, st);
    case kModeBLDopri5Mixed:
      return br.fp32 ? batch_launch<ModeBLDopri5MixedT<true>>(variant, br, queue, fb, s, st)
                     : batch_launch<ModeBLDopri5MixedT<false>>(variant, br, queue, fb, s, st);
    case kModeKSRk4Mixed:
      return br.fp32 ? batch_launch<ModeKSRk4MixedT<true>>(variant, br, queue, fb, s, st)
                     : batch_launch<ModeKSRk4MixedT<false>>(variant, br, queue, fb, s, st);
    case kModeBundleMixed: return launch_batch_mixed_bundle(variant, br, queue, fb, s, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kt
