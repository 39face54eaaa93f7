// kt_kernels.cu -- the exact (bit-faithful FP64) trace kernels for sm_100a.
//
// Compiled with --fmad=false: every multiply and add of the reference's
// arithmetic is rounded separately, as in the reference's CPU build.
#include "kt_elliptic.cuh"
#include "kt_group.cuh"
#include "kt_trace_kernel.cuh"

namespace kt {

// Instantiations of the exact modes' right-hand sides.  kFlat: launches whose
// frames all have Lambda = 0 (bl_rhs_exact; 640 x 360 DOPRI5 without Lambda:
// 14.6 ms, and 14.7 to 15.9 with the Lambda kernel); kLambda: others.  kGeneral:
// a frame's parameters lie outside the quotients' range (Metric::tame: |Lambda|
// below 2^-90, as the observed one is in units of most black holes' masses, a
// or Q below 2^-40), so that every right-hand side would be evaluated in the
// exact form, refused and evaluated in the general one by a call (640 x 360
// DOPRI5 with Lambda = 4.5e-33 26.8 ms, 16.2 with kGeneral; KS with a = 1e-13 at
// 320 x 180 29.9 and 12.3; 200 x 120 bundles 74 and 45).
enum Form : int { kFlat = 0, kLambda = 1, kGeneral = 2 };
static Form form_of(bool lam, bool tame) { return !tame ? kGeneral : lam ? kLambda : kFlat; }

template <class M, Form kForm>
struct ModeBL {
  using Machine = M;
  static constexpr int kSlots = M::kSlots;
  M* m;
  __device__ __forceinline__ bool needs_k1() const { return m->needs_k1(); }
  __device__ __forceinline__ bool start(const Frame& f, uint32_t pix, uint32_t, uint32_t, const Fallback&) {
    m->init(f, camera_ray(f, pix));
    return true;
  }
  __device__ __forceinline__ bool slot(const Frame& f, int s, RayResult* res) {
    double y[4], k[5];
    m->input(s, y);
    if constexpr (kForm == kGeneral)
      bl_rhs(f.g, y[0], y[1], y[2], y[3], m->pt, m->pphi, k);
    else if (!bl_rhs_exact<kForm == kLambda>(f.g, y[0], y[1], y[2], y[3], m->pt, m->pphi, k))
      bl_rhs_rest(f.g, y[0], y[1], y[2], y[3], m->pt, m->pphi, k);
    return m->consume(f, s, k, res);
  }
};
template <Form kForm> using ModeBLRk4 = ModeBL<BLRk4, kForm>;
template <Form kForm> using ModeBLDopri5 = ModeBL<BLDopri5, kForm>;

// (The KS chart has no Lambda: kFlat or kGeneral.)
template <Form kForm>
struct ModeKSRk4 {
  using Machine = KSRk4;
  static constexpr int kSlots = KSRk4::kSlots;
  KSRk4* m;
  __device__ __forceinline__ bool needs_k1() const { return m->needs_k1(); }
  __device__ __forceinline__ bool start(const Frame& f, uint32_t pix, uint32_t out_slot,
                                        uint32_t fb_key, const Fallback& fb) {
    if (m->init(f, camera_ray(f, pix))) return true;
    // init_ks_state failed: the ray is traced in the BL chart by a second
    // launch over the fallback list.
    const uint32_t i = atomicAdd(fb.count, 1u);
    fb.pix[i] = fb_key;
    if (fb.slot) fb.slot[i] = out_slot;
    return false;
  }
  __device__ __forceinline__ bool slot(const Frame& f, int s, RayResult* res) {
    double y[6], k[6];
    m->input(s, y);
    if constexpr (kForm == kGeneral)
      ks_rhs(f.g, y[0], y[1], y[2], y[3], y[4], y[5], m->pT, k);
    else if (!ks_rhs_exact(f.g, y[0], y[1], y[2], y[3], y[4], y[5], m->pT, k))
      ks_rhs_rest(f.g, y[0], y[1], y[2], y[3], y[4], y[5], m->pT, k);
    return m->consume(f, s, k, res);
  }
};

struct ModeBundle {
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
    bundle_rhs(f.g, y[0], y[1], y[2], y[3], m->pt, m->pphi, yW, k, kW);
    return m->consume(f, s, k, kW, res);
  }
};

// Bundles with two lanes per ray (k_trace_pair): the right-hand side is
// split by bundle_half_exact, the halves swapped with one shuffle each, and
// bundle_combine_exact assembles it in bundle_rhs's order (bit-identical); the
// even lane runs the machine's bookkeeping.
__device__ __forceinline__ void swap_halves(unsigned mask, const BundleHalf& me, BundleHalf* other) {
#pragma unroll
  for (int t = 0; t < 3; ++t)
#pragma unroll
    for (int j = 0; j < 5; ++j) other->h5[t][j] = __shfl_xor_sync(mask, me.h5[t][j], 1);
#pragma unroll
  for (int i = 0; i < 4; ++i) other->h1[i] = __shfl_xor_sync(mask, me.h1[i], 1);
}

// The general form; both lanes of each pair (mask) call it together.
__device__ __forceinline__ void bundle_rhs_pair_general(const Metric& g, const double y[4], double pt,
                                                        double pphi, const double W[8], double k[5],
                                                        double kW[8], bool odd, unsigned mask) {
  BundleHalf me, other;
  bundle_rhs_half(g, y[0], y[1], y[2], y[3], pt, pphi, odd, &me);
  swap_halves(mask, me, &other);
  // the even lane's view (the odd lane's result is not used)
  bundle_rhs_combine(me, other, y[0], y[2], y[3], W, k, kW);
}

// ... out of line, for the states the exact quotients do not take.
__device__ __noinline__ void bundle_rhs_pair_rest(const Metric& g, const double y[4], double pt,
                                                  double pphi, const double W[8], double k[5],
                                                  double kW[8], bool odd, unsigned mask) {
  bundle_rhs_pair_general(g, y, pt, pphi, W, k, kW, odd, mask);
}

template <bool kLam>
__device__ __forceinline__ void bundle_rhs_paired(const Metric& g, const double y[4], double pt,
                                                  double pphi, const double W[8], double k[5],
                                                  double kW[8], bool odd, unsigned pmask) {
  BundleHalf me, other;
  bool ok = bundle_half_exact<kLam>(g, y[0], y[1], y[2], y[3], pt, pphi, odd, &me);
  swap_halves(pmask, me, &other);
  ok = bundle_combine_exact(me, other, y[0], y[2], y[3], W, k, kW) & ok;
  const unsigned pair = 3u << (threadIdx.x & 30u);
  if (!__all_sync(pair, ok)) bundle_rhs_pair_rest(g, y, pt, pphi, W, k, kW, odd, pair);
}

template <Form kForm>
struct ModeBundlePair {
  using Machine = Bundle;
  static constexpr int kSlots = Bundle::kSlots;
  Bundle* m;
  __device__ __forceinline__ bool needs_k1() const { return m->needs_k1(); }
  __device__ __forceinline__ bool start(const Frame& f, uint32_t pix, uint32_t, uint32_t, const Fallback&) {
    m->init(f, (int)(pix % (uint32_t)f.cam.W), (int)(pix / (uint32_t)f.cam.W));
    return true;
  }
  __device__ __forceinline__ bool slot(const Frame& f, int s, RayResult* res, bool odd,
                                       unsigned pmask) {
    double y[4], yW[8], k[5], kW[8];
    m->input(s, y, yW);
    if constexpr (kForm == kGeneral)
      bundle_rhs_pair_general(f.g, y, m->pt, m->pphi, yW, k, kW, odd, pmask);
    else
      bundle_rhs_paired<kForm == kLambda>(f.g, y, m->pt, m->pphi, yW, k, kW, odd, pmask);
    __syncwarp(pmask);  // both lanes have read the record
    int done = 0;
    if (!odd) done = m->consume(f, s, k, kW, res) ? 1 : 0;
    __syncwarp(pmask);  // the even lane's updates are visible to the odd lane
    return __shfl_sync(pmask, done, (int)((threadIdx.x & 31u) & ~1u)) != 0;
  }
};

// Separable Kerr (semi-analytic solver): rays that give up are appended to
// the fallback list for the BL RK4 launch and write no result here.
struct ModeSepRk4 {
  using Machine = SepRk4;
  static constexpr int kSlots = SepRk4::kSlots;
  SepRk4* m;
  Fallback fb;
  __device__ __forceinline__ bool needs_k1() const { return m->needs_k1(); }
  __device__ __forceinline__ void hand_back(uint32_t key, uint32_t out_slot) const {
    const uint32_t i = atomicAdd(fb.count, 1u);
    fb.pix[i] = key;
    if (fb.slot) fb.slot[i] = out_slot;
  }
  __device__ __forceinline__ bool start(const Frame& f, uint32_t pix, uint32_t out_slot,
                                        uint32_t fb_key, const Fallback& fbl) {
    fb = fbl;
    if (m->init(f, camera_ray(f, pix), fb_key, out_slot)) return true;
    hand_back(fb_key, out_slot);
    return false;
  }
  __device__ __forceinline__ bool slot(const Frame& f, int s, RayResult* res) {
    double y[2], k[3];
    m->input(s, y);
    const bool ok = m->rhs(s, y, k);
    if (!m->consume(f, s, k, ok, res)) return false;
    if (m->fallback) {
      hand_back(m->fb_key, m->out_slot);
      res->outcome = -1;
    }
    return true;
  }
};

template <Form kForm> struct Lockstep<ModeBundlePair<kForm>> { static constexpr bool value = true; };

template <> struct Defers<ModeSepRk4> { static constexpr bool value = true; };

// Launch shape per mode, measured on B200 (720p config-2 frame, BL chart
// DOPRI5 and RK4; 720p Kerr KS frame; 1080p config-3 bundles): the BL and KS
// single-ray kernels run best as 64-thread blocks, 8 per SM, the bundle
// kernel as 128-thread blocks.  Refilling a
// warp only once all its lanes are idle (kRefill 32) keeps the 32 rays of a
// warp neighbouring pixels that start together: the camera set-up and the
// first slots run converged and the rays' step sequences stay alike, which
// outweighs the lanes idling at the end of each group of 32 (with the
// division-based right-hand sides, KS: 62 against 73 ms, BL RK4: 66 against
// 68, DOPRI5: equal; bundles best at 16).
// The BL kernels with bl_rhs_exact: 8 blocks (16 warps) per SM at 128
// registers without a spill.  720p DOPRI5 41.1 ms against 43.0 with 10 blocks
// (96 registers, 22 B spilled) and 43.4 with 6; RK4 at 641 x 359 9.4 / 10.7 /
// 8.8 ms (that frame is short enough for its longest rays to show).
template <class M, Form kForm> struct Shape<ModeBL<M, kForm>> {
  static constexpr int kBlock = 64, kMinBlocks = 8, kRefill = 32;
};
template <class M, Form kForm> struct BatchMin0<ModeBL<M, kForm>> {
  static constexpr int value = batch_min_blocks(kModeBLRk4, 0);
};
template <Form kForm> struct BatchMin0<ModeKSRk4<kForm>> {
  static constexpr int value = batch_min_blocks(kModeKSRk4, 0);
};
// (720p KS frame 51.6 ms against 52.3 with 10 blocks of 96 registers.)
template <Form kForm> struct Shape<ModeKSRk4<kForm>> {
  static constexpr int kBlock = 64, kMinBlocks = 8, kRefill = 32;
};
template <> struct Shape<struct ModeBundle> { static constexpr int kBlock = 128, kMinBlocks = 1, kRefill = 16; };
// Paired bundles: 64 rays per 128-thread block; kRefill counts lanes.
#ifndef KT_BUNDLE_PAIR_BLOCK
#define KT_BUNDLE_PAIR_BLOCK 128
#endif
#ifndef KT_BUNDLE_PAIR_MINB
#define KT_BUNDLE_PAIR_MINB 3
#endif
#ifndef KT_BUNDLE_PAIR_REFILL
#define KT_BUNDLE_PAIR_REFILL 8
#endif
template <Form kForm> struct Shape<ModeBundlePair<kForm>> {
  static constexpr int kBlock = KT_BUNDLE_PAIR_BLOCK, kMinBlocks = KT_BUNDLE_PAIR_MINB,
                       kRefill = KT_BUNDLE_PAIR_REFILL;
};

template <class ModeT>
static cudaError_t launch_one(const Frame& f, const OutSoA& out, const RayList& rl,
                              uint32_t* queue, const Fallback& fb, const LaunchShape& s,
                              cudaStream_t stream) {
  k_trace<ModeT><<<s.grid, s.block, s.smem, stream>>>(f, out, rl, queue, fb);
  return cudaGetLastError();
}

template <class ModeT>
static cudaError_t launch_pair(const Frame& f, const OutSoA& out, const RayList& rl,
                               uint32_t* queue, const Fallback& fb, const LaunchShape& s,
                               cudaStream_t stream) {
  k_trace_pair<ModeT><<<s.grid, s.block, s.smem, stream>>>(f, out, rl, queue, fb);
  return cudaGetLastError();
}

// One launch of the mode's instantiation for a form.
template <template <Form> class ModeF>
static cudaError_t launch_form(Form form, const Frame& f, const OutSoA& out, const RayList& rl,
                               uint32_t* queue, const Fallback& fb, const LaunchShape& s,
                               cudaStream_t stream) {
  switch (form) {
    case kFlat: return launch_one<ModeF<kFlat>>(f, out, rl, queue, fb, s, stream);
    case kLambda: return launch_one<ModeF<kLambda>>(f, out, rl, queue, fb, s, stream);
    default: return launch_one<ModeF<kGeneral>>(f, out, rl, queue, fb, s, stream);
  }
}

template <template <Form> class ModeF>
static cudaError_t batch_launch_form(Form form, int variant, const BatchRays& br, uint32_t* queue,
                                     const Fallback& fb, const LaunchShape& s, cudaStream_t st) {
  switch (form) {
    case kFlat: return batch_launch<ModeF<kFlat>>(variant, br, queue, fb, s, st);
    case kLambda: return batch_launch<ModeF<kLambda>>(variant, br, queue, fb, s, st);
    default: return batch_launch<ModeF<kGeneral>>(variant, br, queue, fb, s, st);
  }
}

cudaError_t launch_shape(Mode mode, int device, LaunchShape* shape) {
  if (is_mixed_mode(mode)) return launch_shape_mixed(mode, device, shape);
  switch (mode) {
    case kModeBLRk4:
      return shape_for_all<ModeBLRk4<kLambda>, ModeBLRk4<kFlat>, ModeBLRk4<kGeneral>>(device, shape);
    case kModeBLDopri5:
      return shape_for_all<ModeBLDopri5<kLambda>, ModeBLDopri5<kFlat>, ModeBLDopri5<kGeneral>>(device, shape);
    case kModeKSRk4: return shape_for_all<ModeKSRk4<kFlat>, ModeKSRk4<kGeneral>>(device, shape);
    case kModeBundle:
      return shape_for_pair<ModeBundlePair<kLambda>, ModeBundlePair<kFlat>, ModeBundlePair<kGeneral>>(device,
                                                                                                     shape);
    case kModeSepRk4: return shape_for<ModeSepRk4>(device, shape);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_trace(Mode mode, const Frame& f, const OutSoA& out, const RayList& rl,
                         uint32_t* queue, const Fallback& fb, const LaunchShape& s,
                         cudaStream_t stream) {
  if (is_mixed_mode(mode)) return launch_trace_mixed(mode, f, out, rl, queue, fb, s, stream);
  const Form form = form_of(f.g.L != 0.0, f.g.tame != 0);
  switch (mode) {
    case kModeBLRk4: return launch_form<ModeBLRk4>(form, f, out, rl, queue, fb, s, stream);
    case kModeBLDopri5: return launch_form<ModeBLDopri5>(form, f, out, rl, queue, fb, s, stream);
    case kModeKSRk4:
      if (form == kGeneral) return launch_one<ModeKSRk4<kGeneral>>(f, out, rl, queue, fb, s, stream);
      // several lanes per ray where the rays do not fill the device
      // (kt_group.cuh); a count on the device is not known here
      if (!rl.n_dev && rl.n > 0 && rl.n <= kKs8RaysPerSm * (uint32_t)s.sms)
        return launch_group<GroupKSRk4<8>>(f, out, rl, queue, fb, s.sms, stream);
      if (!rl.n_dev && rl.n > 0 && rl.n <= kKs4RaysPerSm * (uint32_t)s.sms)
        return launch_group<GroupKSRk4<4>>(f, out, rl, queue, fb, s.sms, stream);
      return launch_one<ModeKSRk4<kFlat>>(f, out, rl, queue, fb, s, stream);
    case kModeBundle:
      switch (form) {
        case kFlat: return launch_pair<ModeBundlePair<kFlat>>(f, out, rl, queue, fb, s, stream);
        case kLambda: return launch_pair<ModeBundlePair<kLambda>>(f, out, rl, queue, fb, s, stream);
        default: return launch_pair<ModeBundlePair<kGeneral>>(f, out, rl, queue, fb, s, stream);
      }
    case kModeSepRk4: return launch_one<ModeSepRk4>(f, out, rl, queue, fb, s, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t batch_shape(Mode mode, int variant, int device, LaunchShape* shape) {
  switch (mode) {
    case kModeBLRk4:
      return batch_shape_all<ModeBLRk4<kLambda>, ModeBLRk4<kFlat>, ModeBLRk4<kGeneral>>(variant, device,
                                                                                        shape);
    case kModeBLDopri5:
      return batch_shape_all<ModeBLDopri5<kLambda>, ModeBLDopri5<kFlat>, ModeBLDopri5<kGeneral>>(
          variant, device, shape);
    case kModeKSRk4:
      return batch_shape_all<ModeKSRk4<kFlat>, ModeKSRk4<kGeneral>>(variant, device, shape);
    case kModeBundle:
      if (variant == kBatchPairVariant)
        return batch_shape_pair_for<kBatchBlock[kBatchPairVariant], kBatchMinBlocks[kBatchPairVariant],
                                    ModeBundlePair<kLambda>, ModeBundlePair<kFlat>,
                                    ModeBundlePair<kGeneral>>(device, shape);
      return batch_shape<ModeBundle>(variant, device, shape);
    case kModeSepRk4: return batch_shape<ModeSepRk4>(variant, device, shape);
    default: return batch_shape_mixed(mode, variant, device, shape);
  }
}

cudaError_t launch_batch(Mode mode, int variant, const BatchRays& br, uint32_t* queue,
                         const Fallback& fb, const LaunchShape& s, cudaStream_t st) {
  const Form form = form_of(br.lam, br.tame);
  switch (mode) {
    case kModeBLRk4: return batch_launch_form<ModeBLRk4>(form, variant, br, queue, fb, s, st);
    case kModeBLDopri5: return batch_launch_form<ModeBLDopri5>(form, variant, br, queue, fb, s, st);
    case kModeKSRk4:
      return form == kGeneral ? batch_launch<ModeKSRk4<kGeneral>>(variant, br, queue, fb, s, st)
                              : batch_launch<ModeKSRk4<kFlat>>(variant, br, queue, fb, s, st);
    case kModeBundle:
      if (variant == kBatchPairVariant) {
        constexpr int kB = kBatchBlock[kBatchPairVariant], kM = kBatchMinBlocks[kBatchPairVariant];
        if (form == kGeneral)
          k_trace_batch_pair<ModeBundlePair<kGeneral>, kB, kM><<<s.grid, s.block, s.smem, st>>>(br, queue, fb);
        else if (form == kLambda)
          k_trace_batch_pair<ModeBundlePair<kLambda>, kB, kM><<<s.grid, s.block, s.smem, st>>>(br, queue, fb);
        else
          k_trace_batch_pair<ModeBundlePair<kFlat>, kB, kM><<<s.grid, s.block, s.smem, st>>>(br, queue, fb);
        return cudaGetLastError();
      }
      return batch_launch<ModeBundle>(variant, br, queue, fb, s, st);
    case kModeSepRk4: return batch_launch<ModeSepRk4>(variant, br, queue, fb, s, st);
    default: return launch_batch_mixed(mode, variant, br, queue, fb, s, st);
  }
}

// ---- elliptic-closed solver -------------------------------------------------

// After the standard trace of the same rays (the reference's fallback and its
// horizon-precedence check, main.cpp:1227-1295): a ray whose closed-form
// equator crossing lies in the disk, and which the standard tracer did not
// end at the horizon, becomes that disk hit.  One thread per ray.
__global__ void __launch_bounds__(128) k_elliptic(const __grid_constant__ Frame f, const OutSoA out,
                                                  const RayList rl) {
  const uint32_t n = rl.n_dev ? *rl.n_dev : rl.n;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
    const uint32_t pix = rl.pix ? rl.pix[idx] : idx;
    const uint32_t slot = rl.slot ? rl.slot[idx] : idx;
    if (out.outcome[slot] == kOutHorizon) continue;
    double r, g;
    int why;
    if (!elliptic_closed_form(f, camera_ray(f, pix), &r, &g, &why)) continue;
    // TraceResult{DISK_HIT, r, g}: phi_disk and the escape angles stay 0
    out.outcome[slot] = (uint8_t)kOutDisk;
    out.r[slot] = r;
    out.red[slot] = g;
    out.magnif[slot] = 1.0;
    out.phi_disk[slot] = 0.0;
    out.th_esc[slot] = 0.0;
    out.ph_esc[slot] = 0.0;
  }
}

// The closed form's fallback reason per pixel (the reference's
// --debug-elliptic tag, main.cpp:2111-2121): 0 where it places the crossing
// in the disk, else the EllipticFallbackReason.
__global__ void __launch_bounds__(128) k_elliptic_reasons(const __grid_constant__ Frame f, uint32_t n,
                                                          uint8_t* __restrict__ reason) {
  for (uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x; pix < n; pix += gridDim.x * blockDim.x) {
    double r, g;
    int why = kEfNone;
    elliptic_closed_form(f, camera_ray(f, pix), &r, &g, &why);
    reason[pix] = (uint8_t)why;
  }
}

cudaError_t launch_elliptic_reasons(const Frame& f, uint32_t n, uint8_t* reason, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  uint64_t grid = ((uint64_t)n + 127) / 128;
  if (grid > 148 * 8) grid = 148 * 8;
  k_elliptic_reasons<<<(int)grid, 128, 0, stream>>>(f, n, reason);
  return cudaGetLastError();
}

cudaError_t launch_elliptic(const Frame& f, const OutSoA& out, const RayList& rl, cudaStream_t stream) {
  const uint64_t n = rl.n_dev ? (uint64_t)0xffffffffu : rl.n;
  if (n == 0) return cudaSuccess;
  uint64_t grid = (n + 127) / 128;
  if (grid > 148 * 8) grid = 148 * 8;
  k_elliptic<<<(int)grid, 128, 0, stream>>>(f, out, rl);
  return cudaGetLastError();
}

// ---- centre-out ray order ----------------------------------------------------
// The camera looks at the black hole, so the image centre holds the shadow
// and the critical curve, whose rays are the longest, and the edges hold
// short escaping rays.  A whole frame is traced in rings about the image
// centre, innermost first, in blocks of 8 x 4 pixels (ring_item): the long
// rays start early and the persistent kernel's tail is short, while a
// warp's 32 rays are one compact block of neighbours.  Each ray's
// arithmetic does not depend on when or beside which rays it runs, so the
// results are bit for bit those of the row-major trace.  Rings are 4
// pixels wide, wider where the frame needs more than kOrderClasses of them.
// The list is a stable counting sort of ring_item's order: per-tile ring
// counts, one exclusive scan in (ring, tile) order, then each tile scattered
// in item order (a "tile" here is the sort's chunk of items).

// counts[c * tiles + t]: pixels of ring c in tile t (tile = `tile` pixels)
__global__ void k_ring_count(int W, int H, uint32_t tile, uint32_t tiles, uint32_t* __restrict__ counts) {
  __shared__ uint32_t h[kOrderClasses];
  for (int i = threadIdx.x; i < kOrderClasses; i += blockDim.x) h[i] = 0;
  __syncthreads();
  const RingGeom g = ring_geom(W, H);
  const uint32_t n = (uint32_t)W * (uint32_t)H;
  const uint32_t t = blockIdx.x;
  const uint32_t end = min(n, (t + 1) * tile);
  for (uint32_t e = t * tile + threadIdx.x; e < end; e += blockDim.x) {
    uint32_t p;
    int c;
    ring_item(g, e, &p, &c);
    atomicAdd(&h[c], 1u);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < kOrderClasses; c += blockDim.x) counts[(uint32_t)c * tiles + t] = h[c];
}

// Exclusive scan of counts[0..m) in place, one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_ring_scan(uint32_t* __restrict__ a, uint32_t m) {
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t base = 0; base < m; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = (i < m) ? a[i] : 0u;
    uint32_t x = v;  // inclusive warp scan
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, x, d);
      if ((int)lane >= d) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t s = warp_sum[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, s, d);
        if ((int)lane >= d) s += y;
      }
      warp_sum[lane] = s;  // inclusive over warps
    }
    __syncthreads();
    const uint32_t before = carry + (warp ? warp_sum[warp - 1] : 0u) + (x - v);
    if (i < m) a[i] = before;
    __syncthreads();
    if (threadIdx.x == 0) carry += warp_sum[31];
    __syncthreads();
  }
}

// One warp per tile: the tile's pixels in order, each ring's in consecutive
// places from that ring's offset for the tile.
__global__ void k_ring_place(int W, int H, uint32_t tile, uint32_t tiles,
                             const uint32_t* __restrict__ offsets, uint32_t base,
                             uint32_t* __restrict__ list) {
  __shared__ uint32_t next[kOrderClasses];
  const uint32_t t = blockIdx.x;
  for (int c = threadIdx.x; c < kOrderClasses; c += 32) next[c] = offsets[(uint32_t)c * tiles + t];
  __syncwarp();
  const RingGeom g = ring_geom(W, H);
  const uint32_t n = (uint32_t)W * (uint32_t)H;
  const uint32_t end = min(n, (t + 1) * tile);
  const unsigned lane = threadIdx.x;
  for (uint32_t e0 = t * tile; e0 < end; e0 += 32) {
    const uint32_t e = e0 + lane;
    uint32_t p = 0;
    int c = -1;
    if (e < end) ring_item(g, e, &p, &c);
    const unsigned same = __match_any_sync(kFull, c);
    uint32_t at = 0;
    if (c >= 0) at = next[c] + (uint32_t)__popc(same & ((1u << lane) - 1u));
    __syncwarp();
    if (c >= 0) {
      list[at] = base + p;
      if ((int)lane == __ffs(same) - 1) next[c] += (uint32_t)__popc(same);
    }
    __syncwarp();
  }
}

cudaError_t launch_ring_order(int W, int H, uint32_t base, uint32_t* scratch, uint32_t* list,
                              cudaStream_t stream) {
  const uint64_t n = (uint64_t)W * (uint64_t)H;
  const uint32_t tile = ring_tile(n), tiles = (uint32_t)((n + tile - 1) / tile);
  k_ring_count<<<tiles, 256, 0, stream>>>(W, H, tile, tiles, scratch);
  k_ring_scan<<<1, 1024, 0, stream>>>(scratch, (uint32_t)kOrderClasses * tiles);
  k_ring_place<<<tiles, 32, 0, stream>>>(W, H, tile, tiles, scratch, base, list);
  return cudaGetLastError();
}

// ---- the order of a batch ----------------------------------------------------

// One warp per chunk of 32 rays, its lanes dealing the classes of frames among
// them (kt_batch_order.h); the warps past the last chunk copy the rays beyond
// each frame's whole chunks.  A rank over all frames instead of their classes
// made this kernel's time quadratic in the number of frames (creating a batch
// of 40,000 frames of 16 x 16: 2170 ms, 690 this way and without the order).
__global__ void k_batch_order(const BatchOrder o, const uint64_t* __restrict__ offsets,
                              const uint32_t* __restrict__ in, uint32_t* __restrict__ out) {
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t nf = o.n_frames, whole = o.first_chunk()[nf];
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < whole + nf; w += warps) {
    if (w < whole) {  // chunk j of frame k
      const uint32_t k = count_at_most(o.first_chunk(), nf + 1, w) - 1;
      const uint32_t j = w - o.first_chunk()[k];
      const uint32_t rank = __reduce_add_sync(kFull, chunk_rank(o, k, j, lane, 32));
      out[(uint64_t)rank * 32 + lane] = in[offsets[k] + (uint64_t)j * 32 + lane];
    } else {  // frame k's remainder
      const uint32_t k = w - whole, n = o.rest()[k + 1] - o.rest()[k];
      if (lane < n) out[(uint64_t)whole * 32 + o.rest()[k] + lane] = in[offsets[k + 1] - n + lane];
    }
  }
}

cudaError_t launch_batch_order(const BatchOrder& order, uint64_t n_rays, const uint64_t* offsets,
                               const uint32_t* in, uint32_t* out, cudaStream_t stream) {
  const uint64_t warps = n_rays / 32 + order.n_frames;
  uint64_t grid = (warps + 7) / 8;
  if (grid > 148 * 8) grid = 148 * 8;
  k_batch_order<<<(int)grid, 256, 0, stream>>>(order, offsets, in, out);
  return cudaGetLastError();
}

// Chunks of 32 spread over an order list, one warp each: chunk i of m lies at
// (i + f) whole / m, f the fractional part of i times the golden ratio (a fixed
// stride would meet the same frame of an interleaved list every time).
__global__ void k_sample_order(const uint32_t* __restrict__ order, uint64_t whole, uint64_t m,
                               uint32_t* __restrict__ sample) {
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= m) return;
  uint64_t at = i;
  if (m < whole) {
    const double f = (double)i * 0.6180339887498949;
    at = min(whole - 1, (uint64_t)(((double)i + (f - floor(f))) * ((double)whole / (double)m)));
  }
  sample[i * 32 + lane] = order[at * 32 + lane];
}

cudaError_t launch_sample_order(const uint32_t* order, uint64_t whole, uint64_t m, uint32_t* sample,
                                cudaStream_t stream) {
  k_sample_order<<<(unsigned)((m + 7) / 8), 256, 0, stream>>>(order, whole, m, sample);
  return cudaGetLastError();
}

// ---- colour ------------------------------------------------------------------

// One pixel of colorize_buffer (main.cpp:1817-1866), both palettes.  The
// reference colours from float32 GeoPixel fields; the same rounding is
// applied here.
__device__ __forceinline__ void pixel_colour(const ColourConst& cc, int oc, double r, double red,
                                             double magnif, double phi_disk, double th_esc,
                                             double ph_esc, const uint8_t* __restrict__ bg, int bg_w,
                                             int bg_h, uint8_t c[3]) {
  c[0] = c[1] = c[2] = 0;
  if (oc == kOutDisk && cc.palette == 1) {
    disk_colour_interstellar(cc, (double)(float)r, (double)(float)phi_disk, (double)(float)red,
                             (double)(float)magnif, c);
  } else if (oc == kOutDisk) {
    disk_colour(cc, (double)(float)r, (double)(float)red, (double)(float)magnif, c);
  } else if (oc == kOutEscaped && bg != nullptr) {
    bg_sample(bg, bg_w, bg_h, (double)(float)th_esc, (double)(float)ph_esc, c);
  }
}

__global__ void k_colorize(const ColourConst cc, int64_t n, const uint8_t* __restrict__ outcome,
                           const double* __restrict__ r, const double* __restrict__ red,
                           const double* __restrict__ magnif, const double* __restrict__ phi_disk,
                           const double* __restrict__ th_esc,
                           const double* __restrict__ ph_esc, const uint8_t* __restrict__ bg,
                           int bg_w, int bg_h, uint8_t* __restrict__ rgb) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint8_t c[3];
    pixel_colour(cc, outcome[i], r[i], red[i], magnif[i], phi_disk[i], th_esc[i], ph_esc[i], bg,
                 bg_w, bg_h, c);
    rgb[3 * i + 0] = c[0];
    rgb[3 * i + 1] = c[1];
    rgb[3 * i + 2] = c[2];
  }
}

cudaError_t launch_colorize(const ColourConst& cc, int64_t n, const uint8_t* outcome,
                            const double* r, const double* red, const double* magnif,
                            const double* phi_disk, const double* th_esc, const double* ph_esc,
                            const uint8_t* bg,
                            int bg_w, int bg_h, uint8_t* rgb, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const int block = 256;
  int64_t grid = (n + block - 1) / block;
  if (grid > 148 * 32) grid = 148 * 32;
  k_colorize<<<(int)grid, block, 0, stream>>>(cc, n, outcome, r, red, magnif, phi_disk, th_esc,
                                              ph_esc, bg, bg_w, bg_h, rgb);
  return cudaGetLastError();
}

// ---- camera supersampling ------------------------------------------------------

// render_image's camera_spp > 1 branch (main.cpp:2280-2321) after all passes
// are traced: per pixel, the colour of every pass, taken to linear light
// pow(clamp(c/255, 0, 1), gamma) and summed in pass order (the sum of the
// first pass is the value itself), then lround(255 pow(clamp(sum/n, 0, 1),
// 1/gamma)), lround's half-away-from-zero rounding written out for a
// non-negative value.  The 256 linear values of the 8-bit levels are
// computed once per block.
__global__ void k_spp_colorize(const ColourConst cc, int64_t n, int spp, const SppPasses P,
                               const uint8_t* __restrict__ bg, int bg_w, int bg_h, double gamma,
                               uint8_t* __restrict__ rgb) {
  __shared__ double lin[256];
  for (int c = threadIdx.x; c < 256; c += blockDim.x)
    lin[c] = ktm_pow(dclamp((double)c / 255.0, 0.0, 1.0), gamma);
  __syncthreads();
  const double inv_n = 1.0 / (double)spp;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double acc[3] = {0.0, 0.0, 0.0};
    for (int s = 0; s < spp; ++s) {
      const int64_t j = (int64_t)s * n + i;
      uint8_t c[3];
      pixel_colour(cc, P.outcome[j], P.r[j], P.red[j], P.magnif[j], P.phi_disk[j], P.th_esc[j],
                   P.ph_esc[j], bg, bg_w, bg_h, c);
#pragma unroll
      for (int ch = 0; ch < 3; ++ch) acc[ch] = (s == 0) ? lin[c[ch]] : acc[ch] + lin[c[ch]];
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      const double x = 255.0 * ktm_pow(dclamp(acc[ch] * inv_n, 0.0, 1.0), 1.0 / gamma);
      const double t = trunc(x);
      rgb[3 * i + ch] = (uint8_t)(int)((x - t >= 0.5) ? t + 1.0 : t);
    }
  }
}

cudaError_t launch_spp_colorize(const ColourConst& cc, int64_t n, int spp, const SppPasses& P,
                                const uint8_t* bg, int bg_w, int bg_h, double gamma, uint8_t* rgb,
                                cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  int64_t grid = (n + 255) / 256;
  if (grid > 148 * 16) grid = 148 * 16;
  k_spp_colorize<<<(int)grid, 256, 0, stream>>>(cc, n, spp, P, bg, bg_w, bg_h, gamma, rgb);
  return cudaGetLastError();
}

// ---- FP64 pipe probe -----------------------------------------------------------

// Eight independent dependent-FMA chains per thread: measures the FP64 FMA
// issue rate the trace kernels are bounded by (2 flops per FMA).
__global__ void k_fp64_probe(double* out, int n_iter) {
  double a0 = threadIdx.x * 1e-9, a1 = a0 + 1e-9, a2 = a0 + 2e-9, a3 = a0 + 3e-9;
  double a4 = a0 + 4e-9, a5 = a0 + 5e-9, a6 = a0 + 6e-9, a7 = a0 + 7e-9;
  const double m = 0.999999999, c = 1e-12;
  for (int i = 0; i < n_iter; ++i) {
    a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
    a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
  }
  const double s = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
  if (s == 12345.678) out[blockIdx.x] = s;  // keeps the chains alive
}

cudaError_t launch_fp64_probe(double* out, int n_iter, int grid, int block, cudaStream_t stream) {
  k_fp64_probe<<<grid, block, 0, stream>>>(out, n_iter);
  return cudaGetLastError();
}

// Throughput of the operations the algorithmic flop count weights (division,
// x/3, square root, sincos, pow): eight independent recurrences per thread,
// each step one operation plus `kOpProbeExtra[op]` FMA-pipe operations that
// keep its argument in range (2.5/x; sqrt(3x); x/3 + 1; 1.2 + 0.3 sin x +
// 0.001 cos x; 0.3 + 0.5 x^-0.2).  Op 0 is the FMA chain of k_fp64_probe.
template <int OP>
__global__ void k_op_probe(double* out, int n_iter) {
  double v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 1.0 + (threadIdx.x * 8 + j) * 1e-7;
  for (int i = 0; i < n_iter; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      double x = v[j];
      if (OP == 0) x = fma(x, 0.999999999, 1e-12);
      if (OP == 1) x = 2.5 / x;
      if (OP == 2) x = ktm_div3(x) + 1.0;
      if (OP == 3) x = sqrt(x * 3.0);
      if (OP == 4) {
        double sn, cs;
        ktm_sincos(x, &sn, &cs);
        x = fma(0.3, sn, fma(1e-3, cs, 1.2));
      }
      if (OP == 5) x = fma(0.5, ktm_pow(x, -0.2), 0.3);
      v[j] = x;
    }
  }
  const double s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  if (s == 12345.678) out[blockIdx.x] = s;  // keeps the recurrences alive
}

cudaError_t launch_op_probe(int op, double* out, int n_iter, int grid, int block, cudaStream_t stream) {
  switch (op) {
    case 0: k_op_probe<0><<<grid, block, 0, stream>>>(out, n_iter); break;
    case 1: k_op_probe<1><<<grid, block, 0, stream>>>(out, n_iter); break;
    case 2: k_op_probe<2><<<grid, block, 0, stream>>>(out, n_iter); break;
    case 3: k_op_probe<3><<<grid, block, 0, stream>>>(out, n_iter); break;
    case 4: k_op_probe<4><<<grid, block, 0, stream>>>(out, n_iter); break;
    case 5: k_op_probe<5><<<grid, block, 0, stream>>>(out, n_iter); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace kt
