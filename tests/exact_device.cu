// exact_device.cu -- TEST-ONLY: kt_exact.cuh and the exact right-hand sides on
// the device, against the device's IEEE division and square root and the
// general forms, bit for bit.  Built (--fmad=false, as the exact kernels) and
// called by test_gpu_exact_device.py; every call returns a CUDA error code.
#include <cuda_runtime.h>
#include <string.h>

#include "kt_machines.cuh"

using namespace kt;

static __device__ bool differ(double a, double b) {
  return __double_as_longlong(a) != __double_as_longlong(b);
}
template <int N>
static __device__ bool differ(const double* a, const double* b) {
  bool d = false;
  for (int i = 0; i < N; ++i) d = d || differ(a[i], b[i]);
  return d;
}

// Largest |1 - b y0| (root: |1 - x y0^2| / 2) over every top 20 significand
// bits, both ends of the range of the low word and every exponent in
// [-350, 300): for one seed the error is monotone in b, so the ends bound all
// of it, given that the seed depends on the high word alone (*other: low words
// with another seed).
__global__ void k_seeds(bool root, unsigned long long* worst, unsigned long long* other) {
  const uint32_t top = blockIdx.x * blockDim.x + threadIdx.x;
  if (top >= (1u << 20)) return;
  double w = 0.0;
  unsigned long long diff = 0;
  for (int e = -350; e < 300; ++e) {
    const uint64_t hi = ((uint64_t)(1023 + e) << 52) | ((uint64_t)top << 32);
    const double b0 = ktm_from_bits(hi), b1 = ktm_from_bits(hi | 0xffffffffu);
    const double bm = ktm_from_bits(hi | ((top * 2654435761u) ^ (uint32_t)(e * 40503)));
    const double y0 = root ? rsqrt_seed(b0) : rcp_seed(b0);
    diff += differ(y0, root ? rsqrt_seed(b1) : rcp_seed(b1));
    diff += differ(y0, root ? rsqrt_seed(bm) : rcp_seed(bm));
    for (int j = 0; j < 2; ++j) {
      const double b = j ? b1 : b0;
      double err;
      if (root) {
        const double p = b * y0, pl = fma(b, y0, -p);
        err = 0.5 * fabs(fma(-p, y0, 1.0) - pl * y0);
      } else {
        err = fabs(fma(-b, y0, 1.0));
      }
      w = fmax(w, err);
    }
  }
  atomicMax(worst, (unsigned long long)__double_as_longlong(w));
  if (diff) atomicAdd(other, diff);
}

__global__ void k_quot(long n, const double* a, const double* b, unsigned long long* bad) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    if (top_ones(b[i]) & kTopBit) continue;
    const Rcp R = make_rcp(b[i]);
    if (differ(quot_signed(a[i], R), a[i] / b[i]) || differ(quot_one(R), 1.0 / b[i])) atomicAdd(bad, 1ull);
  }
}

__global__ void k_root(long n, const double* x, unsigned long long* bad) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    if (top_edge(x[i]) & kTopBit) continue;
    const Root r = make_root(x[i]);
    const double s = sqrt(x[i]), q = s * s, a = x[i] + 1.0;
    bool d = differ(r.g, s);
    if (!((top_ones(s) | top_ones(q)) & kTopBit))
      d = d || differ(quot(a, make_rcp_from(s, r.y)), a / s) ||
          differ(quot(a, make_rcp_from(q, r.y * r.y)), a / q);
    if (d) atomicAdd(bad, 1ull);
  }
}

__global__ void k_libm(long n, const double* x, unsigned long long* bad) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double s, c, s2, c2;
    ktm_sincos(x[i], &s, &c);
    ktm_sincos_any(x[i], &s2, &c2);
    if (differ(s, s2) || differ(c, c2) || differ(pow_ctl(x[i], 0.2), ktm_pow(x[i], 0.2)) ||
        differ(pow_ctl(x[i], 0.25), ktm_pow(x[i], 0.25)))
      atomicAdd(bad, 1ull);
  }
}

// kind 0 BL (6 numbers a state), 1 KS (7), 2 the two-lane bundles (14).
template <int kKind, bool kLam>
__global__ void k_rhs(const Metric g, long n, const double* y, unsigned long long* bad,
                      unsigned long long* refused) {
  constexpr int kN = kKind == 0 ? 6 : kKind == 1 ? 7 : 14;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double* s = y + kN * i;
    double k[13], e[13];
    for (int j = 0; j < 13; ++j) k[j] = e[j] = 0.0;
    bool ok;
    if constexpr (kKind == 0) {
      ok = bl_rhs_exact<kLam>(g, s[0], s[1], s[2], s[3], s[4], s[5], k);
      bl_rhs(g, s[0], s[1], s[2], s[3], s[4], s[5], e);
    } else if constexpr (kKind == 1) {
      ok = ks_rhs_exact(g, s[0], s[1], s[2], s[3], s[4], s[5], s[6], k);
      ks_rhs(g, s[0], s[1], s[2], s[3], s[4], s[5], s[6], e);
    } else {
      BundleHalf H[2];
      ok = bundle_half_exact<kLam>(g, s[0], s[1], s[2], s[3], s[4], s[5], false, &H[0]);
      ok = bundle_half_exact<kLam>(g, s[0], s[1], s[2], s[3], s[4], s[5], true, &H[1]) && ok;
      ok = bundle_combine_exact(H[0], H[1], s[0], s[2], s[3], s + 6, k, k + 5) && ok;
      bundle_rhs(g, s[0], s[1], s[2], s[3], s[4], s[5], s + 6, e, e + 5);
    }
    if (!ok) atomicAdd(refused, 1ull);
    else if (differ<13>(k, e)) atomicAdd(bad, 1ull);
  }
}

namespace {
struct Dev {  // device copies, freed on return
  void* p[4] = {nullptr, nullptr, nullptr, nullptr};
  int n = 0;
  cudaError_t e = cudaSuccess;
  template <class T>
  T* get(size_t count, const T* host) {
    void* q = nullptr;
    if (e == cudaSuccess) e = cudaMalloc(&q, count * sizeof(T));
    if (q) p[n++] = q;
    if (e == cudaSuccess)
      e = host ? cudaMemcpy(q, host, count * sizeof(T), cudaMemcpyHostToDevice)
               : cudaMemset(q, 0, count * sizeof(T));
    return (T*)q;
  }
  int take(unsigned long long* host, const unsigned long long* dev, size_t count) {
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(host, dev, count * 8, cudaMemcpyDeviceToHost);
    return (int)e;
  }
  ~Dev() {
    while (n) cudaFree(p[--n]);
  }
};
constexpr int kGrid = 592, kBlock = 128;
constexpr unsigned long long* kZeros = nullptr;
}  // namespace

extern "C" {

int ed_seeds(int root, double* worst, unsigned long long* other) {
  Dev d;
  unsigned long long h[2], *o = d.get(2, kZeros);
  if (d.e == cudaSuccess) k_seeds<<<8192, kBlock>>>(root != 0, o, o + 1);
  const int r = d.take(h, o, 2);
  memcpy(worst, h, 8);
  *other = h[1];
  return r;
}

int ed_quot(long n, const double* a, const double* b, unsigned long long* bad) {
  Dev d;
  const double *da = d.get(n, a), *db = d.get(n, b);
  unsigned long long* o = d.get(1, kZeros);
  if (d.e == cudaSuccess) k_quot<<<kGrid, kBlock>>>(n, da, db, o);
  return d.take(bad, o, 1);
}

// what: 0 square roots and quotients by them, 1 sincos and the controllers' pow
int ed_values(int what, long n, const double* x, unsigned long long* bad) {
  Dev d;
  const double* dx = d.get(n, x);
  unsigned long long* o = d.get(1, kZeros);
  if (d.e == cudaSuccess) {
    if (what == 0) k_root<<<kGrid, kBlock>>>(n, dx, o);
    else k_libm<<<kGrid, kBlock>>>(n, dx, o);
  }
  return d.take(bad, o, 1);
}

int ed_rhs(int kind, int lam, double M, double a, double Q, double L, long n, const double* y,
           unsigned long long* bad_refused) {
  const Metric g = make_metric(M, a, Q, L);
  Dev d;
  const double* dy = d.get((size_t)n * (kind == 0 ? 6 : kind == 1 ? 7 : 14), y);
  unsigned long long* o = d.get(2, kZeros);
  if (d.e == cudaSuccess) {
    if (kind == 1) k_rhs<1, false><<<kGrid, kBlock>>>(g, n, dy, o, o + 1);
    else if (kind == 0 && lam) k_rhs<0, true><<<kGrid, kBlock>>>(g, n, dy, o, o + 1);
    else if (kind == 0) k_rhs<0, false><<<kGrid, kBlock>>>(g, n, dy, o, o + 1);
    else if (lam) k_rhs<2, true><<<kGrid, kBlock>>>(g, n, dy, o, o + 1);
    else k_rhs<2, false><<<kGrid, kBlock>>>(g, n, dy, o, o + 1);
  }
  return d.take(bad_refused, o, 2);
}
}
