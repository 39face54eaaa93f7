// kt_mixed_bundle.cu -- the mixed-precision bundle kernel (KT_PREC_MIXED with
// bundles), compiled with FMA contraction like kt_mixed.cu: the Hessian-vector
// products of the analytic gradient, W and its determinant, all in FP64.
//
// KTM_SINCOS_CASES: the camera's sincos with its separate path below pi/4.
// Without contraction the two forms agree bit for bit; with it they fuse other
// products, and the bundle's W, a difference of neighbouring camera rays,
// turns the last bit of a ray into 1e-11 of its record and another step count
// in 5 of 10,000 rays.
#define KTM_SINCOS_CASES 1
#include "kt_smooth.cuh"
#include "kt_trace_kernel.cuh"

namespace kt {

struct ModeBundleMixed {
  using Machine = Bundle;
  static constexpr int kSlots = Bundle::kSlots;
  Bundle* m;
  __device__ __forceinline__ bool needs_k1() const { return m->needs_k1(); }
  __device__ __forceinline__ bool start(const Frame& f, uint32_t pix, uint32_t, uint32_t, const Fallback&) {
    m->init(f, (int)(pix % (uint32_t)f.cam.W), (int)(pix / (uint32_t)f.cam.W));
    return true;
  }
  __device__ __forceinline__ bool slot(const Frame& f, int s, RayResult* res) {
    double y[4], yW[8], k[5], kW[8];
    m->input(s, y, yW);
    bundle_rhs_analytic(f.g, y, m->pt, m->pphi, yW, k, kW);
    return m->consume(f, s, k, kW, res);
  }
};

// Mixed bundles: 64-thread blocks, at least 6 per SM (168 registers, no
// spill), measured at 1080p: 90.8 ms against 97.2 for 128 x 1 (216
// registers), 98.3 for 128 x 3, 91.7 for 64 x 5; refilling at 16 or 8 idle
// lanes 101.0 / 101.6.
#ifndef KT_MIXED_BUNDLE_BLOCK
#define KT_MIXED_BUNDLE_BLOCK 64
#endif
#ifndef KT_MIXED_BUNDLE_MINB
#define KT_MIXED_BUNDLE_MINB 6
#endif
#ifndef KT_MIXED_BUNDLE_REFILL
#define KT_MIXED_BUNDLE_REFILL 32
#endif
template <> struct Shape<ModeBundleMixed> {
  static constexpr int kBlock = KT_MIXED_BUNDLE_BLOCK, kMinBlocks = KT_MIXED_BUNDLE_MINB,
                       kRefill = KT_MIXED_BUNDLE_REFILL;
};

cudaError_t launch_shape_mixed_bundle(int device, LaunchShape* shape) {
  return shape_for<ModeBundleMixed>(device, shape);
}

cudaError_t launch_trace_mixed_bundle(const Frame& f, const OutSoA& out, const RayList& rl,
                                      uint32_t* queue, const Fallback& fb, const LaunchShape& s,
                                      cudaStream_t stream) {
  k_trace<ModeBundleMixed><<<s.grid, s.block, s.smem, stream>>>(f, out, rl, queue, fb);
  return cudaGetLastError();
}

cudaError_t batch_shape_mixed_bundle(int variant, int device, LaunchShape* shape) {
  return batch_shape<ModeBundleMixed>(variant, device, shape);
}

cudaError_t launch_batch_mixed_bundle(int variant, const BatchRays& br, uint32_t* queue,
                                      const Fallback& fb, const LaunchShape& s, cudaStream_t st) {
  return batch_launch<ModeBundleMixed>(variant, br, queue, fb, s, st);
}

}  // namespace kt
