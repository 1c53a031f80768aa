// acg_cdist_fx.cu -- the FP64 cost matrices on the integer pipes.
//
// ||x - y|| over K features takes 2 K FP64 instructions and a root (about 44 at
// K = 17), each 16 SM cycles per warp: the FP64 edge matrix ran at 0.2 TB/s.
// Here a feature is fixed point of W = 57 to 61 bits (the fewer features, the more:
// FxWindow) in two parts, a difference two 32-bit subtractions, and the sum of
// squares three 64-bit accumulators fed by one wide multiply-add each, so five
// integer instructions per feature and pair; the sum of the rounded features'
// squares is exact, and fx_root forms its root.
// The unit is 2^(a - W) with 2^a twice to four times the largest feature of the
// pattern and of a sample of the rows.  The sample is the same in every block: a
// row's costs depend on its values, not on its place, and equal rows have equal
// costs.  Pairs so close that the unit would show beside FP64's own roundings, and
// rows or patterns with values outside the range (or not finite) are formed in
// FP64.
//
// One thread per row: its features in registers, the pattern's parts in shared
// memory (broadcast 16-byte loads of two features), two columns at a time.
// R-MAT 20, 17 features x 64 columns: 90.7 -> 12.7 ms (8.6 GB written, 2.8 GB
// of rows gathered: 1.7 ms at the copy bandwidth); the multiply-adds bound it.
// Where many pairs are left to FP64, the call for them is still no slower than forming
// the whole matrix in FP64 with the row in registers, as the FP64 pipe charges the
// lanes that are active: 131,072 vertices, 16 edges each, 13 and 17 features, a 32/64
// pattern, one iteration: N(0, 1) 4.2 / 13.1 ms; lognormal, sigma 1 and 2, 4.4 / 13.1
// and 11.2 / 13.8; one feature 100 or 10,000 times the others 11.9 / 13.2 and 17.9 / 18.8.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "acg_cdist.cuh"
#include "acg_device.cuh"

namespace acg {

namespace {

constexpr int kXT = 256;
constexpr int kSample = 64;  // rows that the scale is formed from, spread over all

// FP64 form of one pair, for what fixed point does not cover.
__device__ __noinline__ double pair_fp64(const double* __restrict__ x, const double* __restrict__ y,
                                         int K) {
  double s = 0.0;
  for (int k = 0; k < K; ++k) {
    const double t = __ldg(x + k) - __ldg(y + k);
    s = fma(t, t, s);
  }
  return sqrt(s);
}

// One feature: |x - y|, where squaring it neither overflows nor underflows the root
// of its square.
__device__ __forceinline__ double pair_one(double x, double y) {
  const double t = x - y, u = fabs(t);
  const uint32_t e = (uint32_t)__double2hiint(u) >> 20;
  return e > 1023 - 500 && e < 1023 + 500 ? u : sqrt(t * t);
}
__device__ void rows_one(const CdistRbArgs<double, double>& a) {
  const double* y = a.y;
  for (long long r = (long long)blockIdx.x * kXT + threadIdx.x; r < a.nrows;
       r += (long long)gridDim.x * kXT) {
    const double* xr = a.x + (size_t)(a.row ? (long long)__ldg(a.row + r) : r) * a.kstride;
    const double x = __ldg(xr);
    double* orow = a.out + (size_t)r * a.ostride;
    for (int q0 = 0; q0 < a.Pp; q0 += 2) {
      double d[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        d[j] = q0 + j < a.P ? pair_one(x, __ldg(y + q0 + j)) : 0.0;
        if (a.wide && q0 + j < a.P) d[j] = edge_word(d[j], a.wide);
      }
      *reinterpret_cast<double2*>(orow + q0) = make_double2(d[0], d[1]);
    }
  }
}

template <int KM>
__global__ void __launch_bounds__(kXT) cdist_fx_kernel(const CdistRbArgs<double, double> a) {
  dep_launch();
  dep_wait();
  if constexpr (KM == 2)
    if (a.K == 1) {
      rows_one(a);
      return;
    }
  extern __shared__ __align__(16) unsigned char smem[];
  FxPart* s_y = reinterpret_cast<FxPart*>(smem);  // [Pp][KM], zero past P and K
  __shared__ int s_exp, s_bad;
  const int K = a.K, P = a.P, Pp = a.Pp;
  if (threadIdx.x == 0) {
    s_exp = 0;
    s_bad = 0;
  }
  __syncthreads();
  {
    int e = 0;
    auto see = [&](double v) {
      const int x = (__double2hiint(v) >> 20) & 0x7ff;
      if (x != 0x7ff) e = max(e, x);
    };
    // (kLanes threads to a sampled row, their loads in flight together)
    constexpr int kLanes = kXT / kSample;
    const int k0 = threadIdx.x % kLanes;
    const long long r = threadIdx.x / kLanes * a.nrows / kSample;
    const double* xr = a.x + (size_t)(a.row ? (long long)__ldg(a.row + r) : r) * a.kstride;
    double v[(KM + kLanes - 1) / kLanes];
#pragma unroll
    for (int k = 0; k < KM; k += kLanes) v[k / kLanes] = k0 + k < K ? __ldg(xr + k0 + k) : 0.0;
    // (and the thread's own first row on its way)
    const long long r0 = (long long)blockIdx.x * kXT + threadIdx.x;
    if (r0 < a.nrows) {
      const double* x0 = a.x + (size_t)(a.row ? (long long)__ldg(a.row + r0) : r0) * a.kstride;
#pragma unroll
      for (int k = 0; k < KM; k += 16)
        if (k < K) asm volatile("prefetch.global.L1 [%0];" ::"l"(x0 + k));
      asm volatile("prefetch.global.L1 [%0];" ::"l"(x0 + K - 1));
    }
    for (int t = threadIdx.x; t < P * K; t += kXT) see(a.y[t]);
#pragma unroll
    for (int k = 0; k < KM; k += kLanes) see(v[k / kLanes]);
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_exp, e);
  }
  __syncthreads();
  // the largest is below 2^(e - 1022); beyond +-2^480 squares leave FP64's range
  const int ax = min(480, max(-480, s_exp - 1021));
  {
    bool bad = false;
    for (int t = threadIdx.x; t < Pp * KM; t += kXT) {
      const int q = t / KM, k = t % KM;
      s_y[t] = (q < P && k < K) ? fx_part<KM>(a.y[(size_t)q * K + k], ax, &bad) : FxPart{0, 0};
    }
    if (bad) s_bad = 1;
  }
  __syncthreads();
  const bool ybad = s_bad != 0;
  for (long long r = (long long)blockIdx.x * kXT + threadIdx.x; r < a.nrows;
       r += (long long)gridDim.x * kXT) {
    const double* xr = a.x + (size_t)(a.row ? (long long)__ldg(a.row + r) : r) * a.kstride;
    FxPart x[KM];
    bool big = ybad;
#pragma unroll
    for (int k = 0; k < KM; ++k) {
      x[k] = FxPart{0, 0};
      if (k < K) x[k] = fx_part<KM>(__ldg(xr + k), ax, &big);
    }
    double* orow = a.out + (size_t)r * a.ostride;
    for (int q0 = 0; q0 < Pp; q0 += 2) {
      double d[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int4* yq = reinterpret_cast<const int4*>(s_y + (size_t)(q0 + j) * KM);
        uint64_t sh = 0, sl = 0;
        int64_t sc = 0;
#pragma unroll
        for (int k = 0; k < KM; k += 2) {
          const int4 y = yq[k / 2];
          const int h0 = x[k].h - y.x, l0 = x[k].l - y.y, h1 = x[k + 1].h - y.z, l1 = x[k + 1].l - y.w;
          sh += (uint64_t)((int64_t)h0 * h0);
          sc += (int64_t)h0 * l0;
          sl += (uint64_t)((int64_t)l0 * l0);
          sh += (uint64_t)((int64_t)h1 * h1);
          sc += (int64_t)h1 * l1;
          sl += (uint64_t)((int64_t)l1 * l1);
        }
        if (q0 + j >= P) d[j] = 0.0;
        else if (big || fx_small<KM>(sh)) d[j] = pair_fp64(xr, a.y + (size_t)(q0 + j) * K, K);
        else d[j] = fx_root<KM>(sh, sc, sl, ax);
        if (a.wide && q0 + j < P) d[j] = edge_word(d[j], a.wide);
      }
      *reinterpret_cast<double2*>(orow + q0) = make_double2(d[0], d[1]);
    }
  }
}

// Column statistics of the vertex costs d (StatSpec{P, 2P}): max(-d), LSE(d),
// LSE(-d) as block partials.  Thread t takes column t % P of rows t / P,
// t / P + 256 / P, ... of the block's contiguous rows.
__global__ void __launch_bounds__(kXT)
cdist_stats_kernel(const double* d, long long nrows, int P, int stride, double* part) {
  dep_launch();
  dep_wait();
  __shared__ FxLse s_p[kXT], s_n[kXT];
  __shared__ double s_m[kXT];
  const int nb = gridDim.x, rs = kXT / P;
  const int c = threadIdx.x % P, rl = threadIdx.x / P;
  const long long r0 = nrows * blockIdx.x / nb, r1 = nrows * (blockIdx.x + 1) / nb;
  FxLse lp, ln;
  fx_init(lp);
  fx_init(ln);
  double mn = CUDART_INF;
  if (rl < rs) {
    for (long long r = r0 + rl; r < r1; r += rs) {
      const double x = d[(size_t)r * stride + c];
      mn = fmin(mn, x);
      fx_add(lp, x);
      fx_add(ln, -x);
    }
  }
  s_p[threadIdx.x] = lp;
  s_n[threadIdx.x] = ln;
  s_m[threadIdx.x] = -mn;
  __syncthreads();
  if (threadIdx.x < P) {
    double mx = -mn;
    for (int k = 1; k < rs; ++k) {
      fx_merge(lp, s_p[k * P + c]);
      fx_merge(ln, s_n[k * P + c]);
      mx = fmax(mx, s_m[k * P + c]);
    }
    double m, s;
    part[(size_t)c * nb + blockIdx.x] = mx;
    fx_pair(lp, m, s);
    part[(size_t)(P + 2 * c) * nb + blockIdx.x] = m;
    part[(size_t)(P + 2 * c + 1) * nb + blockIdx.x] = s;
    fx_pair(ln, m, s);
    part[(size_t)(P + 2 * (P + c)) * nb + blockIdx.x] = m;
    part[(size_t)(P + 2 * (P + c) + 1) * nb + blockIdx.x] = s;
  }
}

}  // namespace

#define ACG_FX_CASE(KM_)                                                                         \
  if (km == KM_) {                                                                               \
    const size_t sm = sizeof(FxPart) * (size_t)a.Pp * KM_; /* at most 64 KB */                   \
    if (sm > 48 * 1024)                                                                          \
      ACG_CUDA_TRY(cudaFuncSetAttribute(cdist_fx_kernel<KM_>,                                    \
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));  \
    ACG_CUDA_TRY(launch_kernel(a.early, cdist_fx_kernel<KM_>, blocks, kXT, sm, s, a));                 \
    return ACG_OK;                                                                               \
  }

bool cdist_fx_eligible(int K) { return K >= 1 && K <= 32; }

acg_status launch_cdist_fx(const CdistRbArgs<double, double>& a, int blocks, cudaStream_t s) {
  if (a.P == 0 || a.nrows == 0) return ACG_OK;
  const int km = (a.K + 1) / 2 * 2;
  ACG_FX_CASE(2) ACG_FX_CASE(4) ACG_FX_CASE(6) ACG_FX_CASE(8)
  ACG_FX_CASE(10) ACG_FX_CASE(12) ACG_FX_CASE(14) ACG_FX_CASE(16)
  ACG_FX_CASE(18) ACG_FX_CASE(20) ACG_FX_CASE(22) ACG_FX_CASE(24)
  ACG_FX_CASE(26) ACG_FX_CASE(28) ACG_FX_CASE(30) ACG_FX_CASE(32)
  return set_error(ACG_ERR_UNSUPPORTED, "fixed-point cdist: feature dim %d", a.K);
}

acg_status launch_cdist_vertex_fx(const CdistRbArgs<double, double>& a, int blocks, cudaStream_t s) {
  if (a.P == 0) return ACG_OK;
  if (a.P > kXT) return set_error(ACG_ERR_UNSUPPORTED, "cdist: %d columns", a.P);
  ACG_TRY(launch_cdist_fx(a, std::max(1, std::min(ceil_div(a.nrows, kXT), blocks * 4)), s));
  ACG_CUDA_TRY(launch_kernel(a.early, cdist_stats_kernel, blocks, kXT, 0, s, a.out, a.nrows, a.P, a.ostride, a.bpart));
  return ACG_OK;
}

}  // namespace acg
