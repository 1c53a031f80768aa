// acg_device.cuh -- device helpers shared by the matcher's kernels.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>

#include <cstdint>

#include "acg_common.h"
#include "acg_fx.cuh"

#define ACG_CUDA_TRY(expr)                                                    \
  do {                                                                        \
    cudaError_t acg_e_ = (expr);                                              \
    if (acg_e_ != cudaSuccess)                                                \
      return acg::set_error(acg_e_ == cudaErrorMemoryAllocation               \
                                ? ACG_ERR_OUT_OF_MEMORY : ACG_ERR_CUDA,       \
                            "%s:%d: %s: %s", __FILE__, __LINE__, #expr,       \
                            cudaGetErrorString(acg_e_));                      \
  } while (0)

#define ACG_LAUNCH_CHECK()                                                    \
  do {                                                                        \
    cudaError_t acg_e_ = cudaGetLastError();                                  \
    if (acg_e_ != cudaSuccess)                                                \
      return acg::set_error(ACG_ERR_CUDA, "%s:%d: launch: %s", __FILE__,      \
                            __LINE__, cudaGetErrorString(acg_e_));            \
  } while (0)

namespace acg {

// Programmatic dependent launch: a kernel launched early may start while the one
// before it in the stream still runs; until dep_wait() returns (the
// one before has completed and its writes are visible) it touches only what no
// kernel of a match writes.  dep_launch() lets the next such kernel start early.
// An iteration of a small graph is four to five kernels of about 8 us, so the
// gaps between them and their prologues count (1,000 vertices: FP64 571 -> 457 us a
// match, mixed 480 -> 413).
// Such a kernel lives while its predecessors still write, so it reads what they
// write by ordinary loads (or ld_cs, or cp.async), which stay behind dep_wait():
// __ldg and const __restrict__ parameters are for memory that nobody writes in the
// kernel's life, and the compiler may move those loads ahead of the wait.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... KA, typename... A>
cudaError_t launch_kernel(bool early, void (*kernel)(KA...), int blocks, int threads, size_t smem,
                                cudaStream_t s, const A&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)blocks);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, KA(args)...);
}

// Streaming loads (evicted first), not moved across dep_wait().
__device__ __forceinline__ float ld_cs(const float* p) {
  float x;
  asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(x) : "l"(p));
  return x;
}
__device__ __forceinline__ double ld_cs(const double* p) {
  double x;
  asm volatile("ld.global.cs.f64 %0, [%1];" : "=d"(x) : "l"(p));
  return x;
}
__device__ __forceinline__ float4 ld_cs(const float4* p) {
  float4 x;
  asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "l"(p));
  return x;
}
__device__ __forceinline__ double2 ld_cs(const double2* p) {
  double2 x;
  asm volatile("ld.global.cs.v2.f64 {%0, %1}, [%2];" : "=d"(x.x), "=d"(x.y) : "l"(p));
  return x;
}

constexpr int kNumSMs = 152;  // GB300: 2 dies x 76 SMs

template <typename T>
__device__ __forceinline__ T neg_inf();
template <>
__device__ __forceinline__ double neg_inf<double>() { return -CUDART_INF; }
template <>
__device__ __forceinline__ float neg_inf<float>() { return -CUDART_INF_F; }

template <typename T>
__device__ __forceinline__ T pos_inf() { return -neg_inf<T>(); }

__device__ __forceinline__ double dev_exp(double x) { return exp(x); }
__device__ __forceinline__ float dev_exp(float x) { return expf(x); }
__device__ __forceinline__ double dev_log(double x) { return log(x); }
__device__ __forceinline__ float dev_log(float x) { return logf(x); }

// Running log-sum-exp over a stream of values: the sum of exp(x - m) for the
// largest value m seen so far.  The FP32 form keeps a Kahan compensation term
// so that a thread's partial sum carries only O(eps) relative error however
// many terms it adds; partials are combined in FP64 (LseD below).
template <typename T>
struct OnlineLse;

template <>
struct OnlineLse<double> {
  FxLse a;  // integer arithmetic (acg_fx.cuh)
  __device__ __forceinline__ void init() { fx_init(a); }
  __device__ __forceinline__ void add(double x) { fx_add(a, x); }
  // add x = hi + lo (lo tiny next to hi)
  __device__ __forceinline__ void add2(double hi, double lo) { add(hi + lo); }
  __device__ __forceinline__ void add2_fast(double hi, double lo) { add(hi + lo); }
  __device__ __forceinline__ void add_fast(double x) { add(x); }
  __device__ __forceinline__ double mval() const {
    double m, s;
    fx_pair(a, m, s);
    return m;
  }
  __device__ __forceinline__ double sval() const {
    double m, s;
    fx_pair(a, m, s);
    return s;
  }
};

template <>
struct OnlineLse<float> {
  float m, s, c;
  __device__ __forceinline__ void init() {
    m = -CUDART_INF_F;
    s = 0.f;
    c = 0.f;
  }
  __device__ __forceinline__ void kahan(float e) {
    float y = e - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ void add(float x) {
    if (!(x > -CUDART_INF_F)) return;
    if (x > m) {
      float sc = expf(m - x);
      s *= sc;
      c *= sc;
      m = x;
      kahan(1.f);
    } else {
      kahan(expf(x - m));
    }
  }
  // add x = hi + lo (lo tiny next to hi): exp(hi + lo - m) = exp(hi - m)(1 + lo)
  // to first order, so the low part of a compensated value is not lost
  __device__ __forceinline__ void add2(float hi, float lo) {
    if (!(hi > -CUDART_INF_F)) return;
    if (hi > m) {
      float sc = expf(m - hi);
      s *= sc;
      c *= sc;
      m = hi;
      kahan(1.f + lo);
    } else {
      kahan(expf(hi - m) * (1.f + lo));
    }
  }
  // add2 for finite hi, branch-free with the fast exponential (hot path)
  __device__ __forceinline__ void add2_fast(float hi, float lo) {
    const float mn = fmaxf(m, hi);
    const float sc = __expf(m - mn);  // m = -inf -> 0
    s *= sc;
    c *= sc;
    kahan(__expf(hi - mn) * (1.f + lo));
    m = mn;
  }
  // Branch-free variant with the fast exponential, for the hot per-vertex
  // statistics: m' = max(m, x); s = s e^(m - m') + e^(x - m').  Terms near the
  // running maximum dominate the sum and carry ~1e-7 relative error.
  __device__ __forceinline__ void add_fast(float x) {
    if (x > -CUDART_INF_F) add_fast_some(x);
  }
  // the same for x known to be above -inf
  __device__ __forceinline__ void add_fast_some(float x) {
    const float mn = fmaxf(m, x);
    const float sc = __expf(m - mn);  // m = -inf -> 0
    s *= sc;
    c *= sc;
    kahan(__expf(x - mn));
    m = mn;
  }
  // Four values at once (-inf entries add nothing): one rescale of the running
  // sum for the block's maximum, the four terms summed in FP32 first.
  __device__ __forceinline__ void add4_fast(float x0, float x1, float x2, float x3) {
    const float m4 = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3));
    if (!(m4 > -CUDART_INF_F)) return;
    const float mn = fmaxf(m, m4);
    const float sc = __expf(m - mn);  // m = -inf -> 0
    s *= sc;
    c *= sc;
    kahan((__expf(x0 - mn) + __expf(x1 - mn)) + (__expf(x2 - mn) + __expf(x3 - mn)));
    m = mn;
  }
  // add2_fast of four compensated values hi + lo (hi = -inf: nothing)
  __device__ __forceinline__ void add2x4_fast(const float (&hi)[4], const float (&lo)[4]) {
    const float m4 = fmaxf(fmaxf(hi[0], hi[1]), fmaxf(hi[2], hi[3]));
    if (!(m4 > -CUDART_INF_F)) return;
    const float mn = fmaxf(m, m4);
    const float sc = __expf(m - mn);
    s *= sc;
    c *= sc;
    float e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = __expf(hi[i] - mn) * (1.f + lo[i]);
    kahan((e[0] + e[1]) + (e[2] + e[3]));
    m = mn;
  }
  __device__ __forceinline__ double mval() const { return (double)m; }
  __device__ __forceinline__ double sval() const { return (double)s - (double)c; }
};

// FP64 edge costs dE and messages Z are kept where the FP64 edge phase can read
// their high words as floats (acg_iter.cu): magnitudes from 2^-100 (smaller
// ones, and zeros, take 2^-100: 2^48 times below the last place of anything
// they are added to) to 2^126; *wide is set where one is larger or a NaN, and
// the edge phase then compares in FP64.
__device__ __forceinline__ double edge_word(double x, int* wide) {
  const uint32_t t = (uint32_t)__double2hiint(x) & 0x7fffffffu;
  if (t >= 0x47d00000u) *wide = 1;
  return t < 0x39b00000u ? 0x1p-100 : x;
}

// (max, scaled sum) pair in FP64 for combining partial log-sum-exps.
struct LseD {
  double m, s;
  __device__ __forceinline__ void init() {
    m = -CUDART_INF;
    s = 0.0;
  }
  __device__ __forceinline__ void merge(double m2, double s2) {
    if (!(m2 > -CUDART_INF) || s2 == 0.0) return;
    if (!(m > -CUDART_INF)) {
      m = m2;
      s = s2;
      return;
    }
    if (m2 > m) {
      s = s * exp(m - m2) + s2;
      m = m2;
    } else {
      s += s2 * exp(m2 - m);
    }
  }
  __device__ __forceinline__ double value() const {
    return (m > -CUDART_INF && s > 0.0) ? m + log(s) : -CUDART_INF;
  }
};

__device__ __forceinline__ void lse_merge(double& m, double& s, double m2, double s2) {
  LseD a{m, s};
  a.merge(m2, s2);
  m = a.m;
  s = a.s;
}

// exp(d) for d <= 0, the factor that rescales a partial sum when partial
// log-sum-exps are merged: kMergeF32, the FP32 exponential (relative error ~1e-7,
// that of the FP32 partial sums it scales) for the iterations' statistics of FP32
// kernels; kMergeF64, CUDA's FP64 exponential, for what FP32 plans form once per
// match; kMergeFx, the integer pipes', for FP64 plans (FP64 transcendentals are
// slow on this GPU).
enum MergeExp { kMergeF64 = 0, kMergeF32 = 1, kMergeFx = 2 };
__device__ __forceinline__ double merge_exp(double d, int mode) {
  return mode == kMergeF32 ? (double)expf((float)d) : mode == kMergeFx ? fx_expd(d) : exp(d);
}
// A partial (m, s) that holds no term: m = -inf or s = 0.
__device__ __forceinline__ bool lse_nonempty(double m, double s) {
  return m > -CUDART_INF && s != 0.0;
}

// Per-block statistics written as partials [slot][column]: `nmax` maxima, then
// `nlse` log-sum-exps as (m, s) pairs.  red[w * slots + slot] holds warp w's
// value; warps are combined in order, so the result does not depend on timing.
// Each log-sum-exp is merged in two passes (the largest m, then the sum of
// s_w exp(m_w - m)): one independent exponential per partial, no chain.
__device__ __forceinline__ void write_block_partials(const double* red, int nwarps, int nmax,
                                                     int nlse, double* bpart, int ncols,
                                                     int col, int mode = kMergeF64) {
  const int slots = nmax + 2 * nlse;
  for (int j = threadIdx.x; j < nmax + nlse; j += blockDim.x) {
    if (j < nmax) {
      double m = -CUDART_INF;
      for (int w = 0; w < nwarps; ++w) m = fmax(m, red[w * slots + j]);
      bpart[(size_t)j * ncols + col] = m;
    } else {
      const int sm = nmax + 2 * (j - nmax);
      double m = -CUDART_INF, s = 0.0;
      for (int w = 0; w < nwarps; ++w) {
        const double m2 = red[w * slots + sm], s2 = red[w * slots + sm + 1];
        if (lse_nonempty(m2, s2)) m = fmax(m, m2);
      }
      if (m > -CUDART_INF) {
        for (int w = 0; w < nwarps; ++w) {
          const double m2 = red[w * slots + sm], s2 = red[w * slots + sm + 1];
          if (lse_nonempty(m2, s2)) s += s2 * merge_exp(m2 - m, mode);
        }
      }
      bpart[(size_t)sm * ncols + col] = m;
      bpart[(size_t)(sm + 1) * ncols + col] = s;
    }
  }
}

// The same for FP32 statistics, maxima kept as floats: warp w's are red_m[w * (nmax +
// nlse) ...], its sums red_s[w * nlse ...].  The results are write_block_partials'
// with kMergeF32, bit for bit: a difference of two floats rounds to FP32 alike from
// FP64 and from the exact value.
__device__ __forceinline__ void write_block_partials_f32(const float* red_m, const double* red_s,
                                                         int nwarps, int nmax, int nlse,
                                                         double* bpart, int ncols, int col) {
  const int nm = nmax + nlse;
  for (int j = threadIdx.x; j < nm; j += blockDim.x) {
    float m = -CUDART_INF_F;
    if (j < nmax) {
      for (int w = 0; w < nwarps; ++w) m = fmaxf(m, red_m[w * nm + j]);
      bpart[(size_t)j * ncols + col] = (double)m;
    } else {
      const int i = j - nmax;
      double s = 0.0;
      auto nonempty = [&](int w) {
        return red_m[w * nm + j] > -CUDART_INF_F && (__double_as_longlong(red_s[w * nlse + i]) << 1) != 0;
      };
      for (int w = 0; w < nwarps; ++w)
        if (nonempty(w)) m = fmaxf(m, red_m[w * nm + j]);
      if (m > -CUDART_INF_F)
        for (int w = 0; w < nwarps; ++w)
          if (nonempty(w)) s += red_s[w * nlse + i] * (double)expf(red_m[w * nm + j] - m);
      bpart[(size_t)(nmax + 2 * i) * ncols + col] = (double)m;
      bpart[(size_t)(nmax + 2 * i + 1) * ncols + col] = s;
    }
  }
}

// Compensated running sum for FP32 (TwoSum: hi + lo carries the exact sum of
// the added terms to within one rounding); plain sum for FP64.
template <typename T>
struct CSum;
template <>
struct CSum<float> {
  float hi, lo;
  __device__ __forceinline__ void init(float x) {
    hi = x;
    lo = 0.f;
  }
  __device__ __forceinline__ void add(float x) {
    const float s = hi + x;
    const float bp = s - hi;
    lo += (hi - (s - bp)) + (x - bp);
    hi = s;
  }
  __device__ __forceinline__ float value() const { return hi + lo; }
  // (hi + lo) - y with a single final rounding of the small part
  __device__ __forceinline__ float minus(float y) const { return (hi - y) + lo; }
  __device__ __forceinline__ double dvalue() const { return (double)hi + (double)lo; }
};
template <>
struct CSum<double> {
  double hi;
  double lo = 0.0;  // always zero: FP64 needs no compensation here
  __device__ __forceinline__ void init(double x) { hi = x; }
  __device__ __forceinline__ void add(double x) { hi += x; }
  __device__ __forceinline__ double value() const { return hi; }
  __device__ __forceinline__ double minus(double y) const { return hi - y; }
  __device__ __forceinline__ double dvalue() const { return hi; }
};

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned r;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
  return r;
}

}  // namespace acg
