// acg_iter.cu -- one BP iteration as two kernels (see acg_bp.cu's header for
// the algebra).
//
// Phase A, edge_max_kernel -- the segmented (max, -) reduction over the
// destination-sorted CSR:  M'[v][q] = max_{e in in(v)} VR'[s_e][q] - dE[e][q].
//   One warp per work item (a light vertex's in-edges, or one chunk of a heavy
//   vertex's).  The 32 lanes are (edge slot, 16-byte column) pairs: NPOW lanes
//   cover one [Pp] row, S = 32 / NPOW in-edges are loaded per instruction and
//   kU instructions are issued back to back, so each warp keeps S * kU pairs of
//   (streamed dE row, gathered VR' row) in flight.  The items are cut into
//   contiguous ranges of near-equal cost (load steps plus a per-item
//   overhead; built on the device once per data graph), up to 32 per launched
//   warp: a warp walks its own range, then claims further ranges from a
//   counter as it finishes, so the SMs stay full until the last ranges.  Every
//   item is written by exactly one warp, whichever it is, so the result does
//   not depend on the order of the claims.  A chunk writes a partial row; the max
//   of a heavy vertex's partial rows is taken by the warp that finishes the last
//   one (FP32 without argmax) or by heavy_combine_kernel.
//
// Phase B, vertex_warp_kernel (FP32, patterns up to 64 x 64) -- one warp per
//   contiguous vertex range, rows staged per warp with cp.async; see its own
//   comment.  FP32 patterns of more than 64 edge columns take acg_vertex_wide.cu's
//   kernel, FP64 ones acg_vertex_fx.cu's; the block-tile form below is left with
//   FP32 patterns of up to 64 edge columns and more than 64 vertices, and with wide
//   ones around a hub or of few vertices (vertex_wide_schedule).
//
// Phase B, vertex_update_kernel -- everything per vertex, streamed with
//   coalesced 16-byte accesses: FMax, RMax, MU_raw (compensated sum), the next
//   VF', VR', and per-column statistics.  One thread per (vertex, 16-byte
//   column) for the q-side and per (vertex, pattern vertex) for MU; a block
//   walks fixed tiles of consecutive vertices and every thread owns fixed
//   columns, so statistics are accumulated in registers in a fixed order and
//   results are bit-reproducible.  No kernel waits on another block.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <limits>
#include <vector>

#include "acg_device.cuh"
#include "acg_iter.cuh"
#include "acg_vschedule.h"

namespace acg {

namespace {

constexpr int kAT = 256;       // threads per block, phase A
// 3 steps in flight measured fastest at RMAT-22 (4.07 ms per edge phase; 2: 4.44,
// 4: 4.47, 5: 4.36, 6: 5.37, 8: 5.21 ms)
#ifndef ACG_EDGE_KU
#define ACG_EDGE_KU 3
#endif
constexpr int kU = ACG_EDGE_KU;  // edge steps issued back to back
constexpr int kBT = 256;       // threads per block, phase B

template <typename T>
struct VecT;
template <>
struct VecT<double> {
  using type = double2;
  static constexpr int W = 2;
};
template <>
struct VecT<float> {
  using type = float4;
  static constexpr int W = 4;
};
template <typename T>
__device__ __forceinline__ T vg(const typename VecT<T>::type& v, int w) {
  return reinterpret_cast<const T*>(&v)[w];
}
template <typename T>
__device__ __forceinline__ void vs(typename VecT<T>::type& v, int w, T x) {
  reinterpret_cast<T*>(&v)[w] = x;
}
template <typename T>
__device__ __forceinline__ typename VecT<T>::type vfill(T x) {
  typename VecT<T>::type r;
#pragma unroll
  for (int w = 0; w < VecT<T>::W; ++w) vs<T>(r, w, x);
  return r;
}

__host__ __device__ inline size_t a16(size_t b) { return (b + 15) & ~size_t(15); }

// ------------------------------------------------------------------ phase A
// (An explicit minimum of one block per SM lets the compiler keep more of the
// pipelined loads in registers: 72 registers and 3 blocks/SM measured faster
// than 56 registers and 4 blocks/SM at RMAT-22, 4.47 ms against 5.30 ms.)
#ifndef ACG_EDGE_MINB
#define ACG_EDGE_MINB 1
#endif
// ARG: also the first maximal dst-CSR position of each maximum (adjoint
// recording): ties go to the smaller position.
// The max of heavy vertex h's cnt partial rows into its M row; one warp, lanes
// over columns.  The rows were written by other warps of this launch: read
// through L2.
template <typename T>
__device__ __forceinline__ void heavy_finish(const T* partial, T* M, size_t b0, size_t out, int cnt,
                                             int Pp) {
  const int lane = threadIdx.x & 31;
  for (int q = lane; q < Pp; q += 32) {
    T m = neg_inf<T>();
    for (int r = 0; r < cnt; ++r) m = fmax(m, __ldcg(partial + b0 + (size_t)r * Pp + q));
    M[out + q] = m;
  }
}

// FP64 maxima without FP64 arithmetic per element.  A difference and a maximum
// in FP64 occupy an SM for 32 cycles per warp (2 lanes per clock), which bounds
// the FP64 edge phase at twice the time of its bytes.  Instead each element
// x - y gets an interval [l, u] from the high words of x and y read as floats,
// and a column keeps the pair (x, y) of its largest element so far.  Per step,
// the elements (and the pair kept) whose interval reaches the largest lower
// bound are candidates; a single one is the new pair, and only where there are
// more (two elements within 2^-18 of the operands) are the differences formed
// in FP64 and compared.  The difference of the pair that remains is formed once
// per item.  FP64 rounding is monotone, so the result has the bits of the
// element-wise FP64 maximum.
// The integer pipe (shifts, logic, selects: 16 lanes a clock per scheduler) is
// the next bound, so the values are stored within a float's range (edge_word)
// and a high word becomes a float by one multiply-add.
// R-MAT 20, pattern 32/64 (9.1 GB, 1.4 ms at the copy bandwidth): 4.31 ms an
// iteration in FP64, 1.99 with intervals from clamped words, 1.78
// so.
struct LazyMax {
  double x, y;  // the largest element so far is x - y (none yet: about -2^127)
  __device__ __forceinline__ void init() {
    x = -0x1p127;
    y = 1.0;
  }
  __device__ __forceinline__ double value() const { return x - y; }
  __device__ __forceinline__ void set(bool r, double nx, double ny) {
    x = r ? nx : x;
    y = r ? ny : y;
  }
};
// The float of a double's high word, truncated toward zero to 20 mantissa bits
// (magnitudes of edge_word): the exponent rebased from 1023 to 127.  rebase is
// 8; as a multiplier it keeps the shift off the integer pipe.
__device__ __forceinline__ float high_float(double x, uint32_t rebase) {
  const uint32_t h = (uint32_t)__double2hiint(x);
  return __uint_as_float((h * rebase + 0x40000000u) | (h & 0x80000000u));
}
__device__ __forceinline__ float high_float_pos(double x, uint32_t rebase) {
  return __uint_as_float((uint32_t)__double2hiint(x) * rebase + 0x40000000u);
}
// [l, u] of x - y, y > 0: truncation is below 2^-20 of each operand, the
// roundings here below 2^-22.
__device__ __forceinline__ void diff_bounds(double x, double y, uint32_t rebase, float& l, float& u) {
  const float fx = high_float(x, rebase), fy = high_float_pos(y, rebase);
  const float d = fx - fy, w = fabsf(fx) + fy;
  l = fmaf(w, -0x1p-19f, d);
  u = fmaf(w, 0x1p-19f, d);
}
// One step of a column: N elements x - y, ok where there is one (below the
// others' range where not), at positions e, e + stride, ...; the whole warp
// calls it.  col: a pattern edge's column, not one of the row's padding, whose
// zeros would tie with each other.  ARG: pos, the first maximal position.
template <int N, bool ARG>
__device__ __forceinline__ void lazy_step(LazyMax& b, int& pos, const double (&x)[N],
                                          const double (&y)[N], const bool (&ok)[N], bool col, int e,
                                          int stride, uint32_t rebase) {
  float l[N], u[N], top, bu;
  diff_bounds(b.x, b.y, rebase, top, bu);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    diff_bounds(x[i], y[i], rebase, l[i], u[i]);
    top = fmaxf(top, l[i]);
  }
  bool c[N], any = bu >= top, two = false;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    c[i] = ok[i] && u[i] >= top;
    two = two || (any && c[i]);
    any = any || c[i];
  }
  if (__any_sync(0xffffffffu, two && col)) {
    // in FP64, in order (volatile: not computed ahead of the vote)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      double v, m;
      asm volatile("sub.f64 %0, %1, %2;" : "=d"(v) : "d"(x[i]), "d"(y[i]));
      asm volatile("sub.f64 %0, %1, %2;" : "=d"(m) : "d"(b.x), "d"(b.y));
      const bool r = ok[i] && v > m;
      b.set(r, x[i], y[i]);
      if constexpr (ARG) pos = r ? e + i * stride : pos;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      b.set(c[i], x[i], y[i]);
      if constexpr (ARG) pos = c[i] ? e + i * stride : pos;
    }
  }
}
// max of two doubles that are not NaN, as integers
__device__ __forceinline__ double max_bits(double a, double b) {
  const long long ia = __double_as_longlong(a), ib = __double_as_longlong(b);
  const long long ka = ia ^ ((ia >> 63) & 0x7fffffffffffffffll);
  const long long kb = ib ^ ((ib >> 63) & 0x7fffffffffffffffll);
  return ka >= kb ? a : b;
}

// One range of a warp's items, [it, it_end).
template <typename T, int NPOW, int NQV, bool ARG, bool LAZY>
__device__ __forceinline__ void edge_max_range(const EdgeMaxArgs<T>& a, int it, const int it_end,
                                               const int slot, const int qc) {
  using VT = typename VecT<T>::type;
  constexpr int W = VecT<T>::W;
  constexpr int S = 32 / NPOW;
  constexpr int NQ = NQV * W;
  constexpr int STEP = S * kU;
  const int Pp = a.Pp;
  if (it >= it_end) return;

  // Software pipeline over the warp's steps (kU in-edges per slot per step,
  // crossing item boundaries): the source indices of step k+1 are loaded while
  // the gathered rows of step k are in flight.
  int4 item = __ldg(a.items + it);
  int4 item_next = it + 1 < it_end ? __ldg(a.items + it + 1) : make_int4(0, 0, 0, -1);
  int base = item.y;
  int sidx[kU];
#pragma unroll
  for (int u = 0; u < kU; ++u) {
    const int e = base + slot + S * u;
    sidx[u] = e < item.z ? __ldg(a.src_of + e) : 0;
  }
  constexpr bool kLazy = LAZY;
  T acc[NQ];
  LazyMax best[kLazy ? NQ : 1];
  int pos[ARG ? NQ : 1];
  bool col[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    acc[k] = neg_inf<T>();
    col[k] = (qc + NPOW * (k / W)) * W + k % W < a.Pe;
    if constexpr (kLazy) best[k].init();
    if constexpr (ARG) pos[k] = -1;
  }
  for (;;) {
    // rows of this step
    VT x[kU][NQV], y[kU][NQV];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int e = base + slot + S * u;
      const bool ok = e < item.z;
#pragma unroll
      for (int k = 0; k < NQV; ++k) {
        const int qv = qc + NPOW * k;
        if (ok && qv * W < Pp) {
          x[u][k] = reinterpret_cast<const VT*>(a.vr_in + (size_t)sidx[u] * Pp)[qv];
          y[u][k] = ld_cs(reinterpret_cast<const VT*>(a.dE + (size_t)e * Pp) + qv);
        } else {
          x[u][k] = vfill<T>(kLazy ? T(-0x1p127) : neg_inf<T>());
          y[u][k] = vfill<T>(T(kLazy ? 1 : 0));
        }
      }
    }
    // next step's position, and its source indices (in flight with the rows)
    const bool item_done = base + STEP >= item.z;
    int nbase = base + STEP, nend = item.z;
    bool more = true;
    if (item_done) {
      more = it + 1 < it_end;
      nbase = item_next.y;
      nend = item_next.z;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int e = nbase + slot + S * u;
      sidx[u] = (more && e < nend) ? __ldg(a.src_of + e) : 0;
    }
    if constexpr (kLazy) {
      bool ok[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) ok[u] = base + slot + S * u < item.z;
#pragma unroll
      for (int k = 0; k < NQV; ++k)
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const int j = k * W + w;
          double xs[kU], ys[kU];
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            xs[u] = vg<T>(x[u][k], w);
            ys[u] = vg<T>(y[u][k], w);
          }
          lazy_step<kU, ARG>(best[j], pos[ARG ? j : 0], xs, ys, ok, col[j], base + slot, S, a.rebase);
        }
    } else {
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if constexpr (ARG) {
        const int e = base + slot + S * u;
        if (e < item.z) {
#pragma unroll
          for (int k = 0; k < NQV; ++k)
#pragma unroll
            for (int w = 0; w < W; ++w) {
              const T v = vg<T>(x[u][k], w) - vg<T>(y[u][k], w);
              if (pos[k * W + w] < 0 || v > acc[k * W + w]) {
                acc[k * W + w] = v;
                pos[k * W + w] = e;
              }
            }
        }
      } else {
#pragma unroll
        for (int k = 0; k < NQV; ++k)
#pragma unroll
          for (int w = 0; w < W; ++w)
            acc[k * W + w] = fmax(acc[k * W + w], vg<T>(x[u][k], w) - vg<T>(y[u][k], w));
      }
    }
    }
    if (item_done) {
      if constexpr (kLazy) {
#pragma unroll
        for (int k = 0; k < NQ; ++k) acc[k] = best[k].value();
      }
      if constexpr (ARG) {
#pragma unroll
        for (int o = NPOW; o < 32; o <<= 1)
#pragma unroll
          for (int k = 0; k < NQ; ++k) {
            const T ob = __shfl_xor_sync(0xffffffffu, acc[k], o);
            const int op = __shfl_xor_sync(0xffffffffu, pos[k], o);
            if (op >= 0 && (pos[k] < 0 || ob > acc[k] || (ob == acc[k] && op < pos[k]))) {
              acc[k] = ob;
              pos[k] = op;
            }
          }
      } else {
#pragma unroll
        for (int o = NPOW; o < 32; o <<= 1)
#pragma unroll
          for (int k = 0; k < NQ; ++k) {
            const T ob = __shfl_xor_sync(0xffffffffu, acc[k], o);
            if constexpr (sizeof(T) == 8) acc[k] = max_bits(acc[k], ob);
            else acc[k] = fmax(acc[k], ob);
          }
      }
      if (slot == 0) {
        T* row = item.w >= 0 ? a.partial + (size_t)item.w * Pp : a.M + (size_t)item.x * Pp;
#pragma unroll
        for (int k = 0; k < NQV; ++k) {
          const int qv = qc + NPOW * k;
          if (qv * W < Pp) {
            VT o;
#pragma unroll
            for (int w = 0; w < W; ++w) vs<T>(o, w, acc[k * W + w]);
            reinterpret_cast<VT*>(row)[qv] = o;
            if constexpr (ARG) {
              int* prow = item.w >= 0 ? a.ppos + (size_t)item.w * Pp : a.argpos + (size_t)item.x * Pp;
#pragma unroll
              for (int w = 0; w < W; ++w) prow[qv * W + w] = pos[k * W + w];
            }
          }
        }
      }
      // (FP32 without argmax only: in the other forms the finisher would cost
      // the edge loop registers, 64 -> 72..94; they keep heavy_combine)
      if (sizeof(T) == 4 && !ARG && item.w >= 0 && a.hcnt) {
        // a chunk: its rows are fenced before the count; the warp that
        // completes the heavy vertex's last chunk fences again and combines
        __threadfence();
        __syncwarp();
        const int h = __ldg(a.pheavy + item.w);
        const int cnt = __ldg(a.hcount + h);
        int last = 0;
        if ((threadIdx.x & 31) == 0) last = atomicAdd(a.hcnt + h, 1) == cnt - 1;
        if (__shfl_sync(0xffffffffu, last, 0)) {
          __threadfence();
          heavy_finish<T>(a.partial, a.M, (size_t)__ldg(a.hbase + h) * Pp,
                          (size_t)__ldg(a.hvert + h) * Pp, cnt, Pp);
          if ((threadIdx.x & 31) == 0) a.hcnt[h] = 0;  // ready for the next launch
        }
      }
#pragma unroll
      for (int k = 0; k < NQ; ++k) {
        acc[k] = neg_inf<T>();
        if constexpr (kLazy) best[k].init();
        if constexpr (ARG) pos[k] = -1;
      }
      if (!more) break;
      ++it;
      item = item_next;
      item_next = it + 1 < it_end ? __ldg(a.items + it + 1) : make_int4(0, 0, 0, -1);
    }
    base = nbase;
  }
}

// (FP64: four blocks per SM hide the longer chains; RMAT-20 edge phases 57.1 ms,
// three blocks 60.3, two 67; the wide shapes keep what their registers allow.)
template <typename T, int NQV>
constexpr int edge_min_blocks() {
  return sizeof(T) == 4 ? ACG_EDGE_MINB : NQV == 1 ? 4 : NQV == 2 ? 2 : 1;
}
template <typename T, int NPOW, int NQV, bool ARG>
__global__ void __launch_bounds__(kAT, (edge_min_blocks<T, NQV>()))
edge_max_kernel(const EdgeMaxArgs<T> a) {
  const int lane = threadIdx.x & 31;
  const int slot = lane / NPOW, qc = lane % NPOW;
  const int nw = (int)gridDim.x * (kAT / 32);
  const int gw = (blockIdx.x * kAT + threadIdx.x) >> 5;
  dep_launch();
  dep_wait();
  const bool wide = sizeof(T) == 8 && *a.wide != 0;
  // The warp's own range first, then claimed ones (the claim of the next is in
  // flight while this one runs): warps that finish early keep taking work, so
  // the SMs stay full until the last ranges instead of waiting on the slowest
  // warp of a static split.
  for (int r = gw; r < a.nranges;) {
    int rn = a.nranges;
    if (a.ctr && lane == 0) rn = nw + atomicAdd(a.ctr, 1);
    const int it = __ldg(a.wsplit + r), it_end = __ldg(a.wsplit + r + 1);
    if constexpr (sizeof(T) == 8) {
      if (wide) edge_max_range<T, NPOW, NQV, ARG, false>(a, it, it_end, slot, qc);
      else edge_max_range<T, NPOW, NQV, ARG, true>(a, it, it_end, slot, qc);
    } else {
      edge_max_range<T, NPOW, NQV, ARG, false>(a, it, it_end, slot, qc);
    }
    r = __shfl_sync(0xffffffffu, rn, 0);
  }
  if (a.ctr && lane == 0) {
    __threadfence();  // this warp's claims come before its finish count
    if (atomicAdd(a.ctr + 1, 1) == nw - 1) {  // every warp has made its last claim
      a.ctr[0] = 0;
      a.ctr[1] = 0;
    }
  }
}

template <typename T>
__device__ __forceinline__ T max_of(T a, T b) {
  if constexpr (sizeof(T) == 8) return max_bits(a, b);
  else return fmaxf(a, b);
}

// Max over each heavy vertex's partial rows: one block per heavy vertex, its
// warps over the rows (a hub has hundreds; one warp over all of them took 64 us
// at R-MAT 20), lanes over the columns.
constexpr int kHeavyCols = 256;  // columns of a row at most
template <typename T>
__global__ void __launch_bounds__(256)
heavy_combine_kernel(const T* partial, const int* __restrict__ hbase,
                     const int* __restrict__ hcount, const int* __restrict__ hvert, int Pp, T* M) {
  __shared__ T part[8][kHeavyCols];
  dep_launch();
  dep_wait();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const T* p0 = partial + (size_t)hbase[blockIdx.x] * Pp;
  const int cnt = hcount[blockIdx.x];
  for (int q = lane; q < Pp; q += 32) {
    T m = neg_inf<T>();
    int r = w;
    for (; r + 24 < cnt; r += 32) {
      const T a0 = p0[(size_t)r * Pp + q], a1 = p0[(size_t)(r + 8) * Pp + q];
      const T a2 = p0[(size_t)(r + 16) * Pp + q], a3 = p0[(size_t)(r + 24) * Pp + q];
      m = max_of(m, max_of(max_of(a0, a1), max_of(a2, a3)));
    }
    for (; r < cnt; r += 8) m = max_of(m, p0[(size_t)r * Pp + q]);
    part[w][q] = m;
  }
  __syncthreads();
  T* row = M + (size_t)hvert[blockIdx.x] * Pp;
  for (int q = threadIdx.x; q < Pp; q += 256) {
    T m = part[0][q];
#pragma unroll
    for (int k = 1; k < 8; ++k) m = max_of(m, part[k][q]);
    row[q] = m;
  }
}

// The same with the chunks' argmax positions (chunks in order: an earlier
// chunk keeps a tie).
template <typename T>
__global__ void __launch_bounds__(256)
heavy_combine_arg_kernel(const T* __restrict__ partial, const int* __restrict__ ppos,
                         const int* __restrict__ hbase, const int* __restrict__ hcount,
                         const int* __restrict__ hvert, int nheavy, int Pp, T* __restrict__ M,
                         int* __restrict__ A) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= nheavy) return;
  const size_t b0 = (size_t)hbase[warp] * Pp, out = (size_t)hvert[warp] * Pp;
  const int cnt = hcount[warp];
  for (int q = lane; q < Pp; q += 32) {
    T m = neg_inf<T>();
    int bi = -1;
    auto take = [&](T x, int px) {
      if (px >= 0 && (bi < 0 || x > m)) {
        m = x;
        bi = px;
      }
    };
    int c = 0;
    for (; c + 4 <= cnt; c += 4) {  // four rows in flight, applied in order
      const size_t r = b0 + (size_t)c * Pp + q;
      const T x0 = partial[r], x1 = partial[r + Pp], x2 = partial[r + 2 * (size_t)Pp],
              x3 = partial[r + 3 * (size_t)Pp];
      const int p0 = ppos[r], p1 = ppos[r + Pp], p2 = ppos[r + 2 * (size_t)Pp],
                p3 = ppos[r + 3 * (size_t)Pp];
      take(x0, p0);
      take(x1, p1);
      take(x2, p2);
      take(x3, p3);
    }
    for (; c < cnt; ++c) {
      const size_t r = b0 + (size_t)c * Pp + q;
      take(partial[r], ppos[r]);
    }
    M[out + q] = m;
    A[out + q] = bi;
  }
}

// ------------------------------------------------------------------ phase B
struct UpdSmem {
  size_t pat, fill, lq, F, R, MU, red, stage, sM, sVF, sEM, sB, sCV, sCVl, sOff, stage_bytes, total;
  __host__ __device__ UpdSmem(int V, int Pn, int Pe, int Pp, int Pnp, int sz) {
    size_t o = 0;
    pat = o; o += a16(sizeof(int) * (size_t)(4 * Pe + 2 * (Pn + 1)));
    fill = o; o += a16((size_t)2 * Pp * sz);  // fillF, fillR (padded to Pp)
    lq = o; o += a16((size_t)8 * Pp * sz);    // dF, dR, cR', cF' as hi/lo pairs (padded to Pp)
    F = o; o += a16((size_t)V * Pp * sz);
    R = o; o += a16((size_t)V * Pp * sz);
    MU = o; o += a16((size_t)V * 2 * Pn * sz);  // hi, lo
    red = o; o += a16(sizeof(double) * (size_t)kBT * 6);
    // one stage: the tile's M, Y, dEmin, B rows, CV (hi, lo) rows, in-degree offsets
    size_t so = 0;
    sM = so; so += a16((size_t)V * Pp * sz);
    sVF = so; so += a16((size_t)V * Pp * sz);
    sEM = so; so += a16((size_t)V * Pp * sz);
    sB = so; so += a16((size_t)V * Pp * sz);
    sCV = so; so += a16((size_t)V * Pnp * sz);
    sCVl = so; so += sz == 4 ? a16((size_t)V * Pnp * sz) : 0;
    sOff = so; so += a16(sizeof(int) * (size_t)(V + 1));
    stage_bytes = so;
    stage = o; o += 2 * so;
    total = o;
  }
};

__device__ __forceinline__ unsigned sm_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp16(void* sdst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sm_u32(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp4(void* sdst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sm_u32(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

template <typename T>
__global__ void __launch_bounds__(kBT, 2)
vertex_update_kernel(const VertexUpdArgs<T> a) {
  using VT = typename VecT<T>::type;
  constexpr int W = VecT<T>::W;
  extern __shared__ __align__(16) unsigned char smem[];
  const int Pe = a.Pe, Pn = a.Pn, Pp = a.Pp, Pnp = a.Pnp, Dn = a.Dn;
  const int nvec = Pp / W;
  const int V = kBT / nvec;  // vertices per tile
  const UpdSmem L(V, Pn, Pe, Pp, Pnp, sizeof(T));
  int* s_pat = reinterpret_cast<int*>(smem + L.pat);
  T* s_fillF = reinterpret_cast<T*>(smem + L.fill);
  T* s_fillR = s_fillF + Pp;
  T* s_dF = reinterpret_cast<T*>(smem + L.lq);  // hi, lo of each constant
  T* s_dFlo = s_dF + Pp;
  T* s_dR = s_dFlo + Pp;
  T* s_dRlo = s_dR + Pp;
  T* s_cR = s_dRlo + Pp;
  T* s_cRlo = s_cR + Pp;
  T* s_cF = s_cRlo + Pp;
  T* s_cFlo = s_cF + Pp;
  T* s_F = reinterpret_cast<T*>(smem + L.F);
  T* s_R = reinterpret_cast<T*>(smem + L.R);
  T* s_MU = reinterpret_cast<T*>(smem + L.MU);  // [V][Pn] hi then [V][Pn] lo
  T* s_MUlo = s_MU + (size_t)V * Pn;
  double* s_red = reinterpret_cast<double*>(smem + L.red);
  const int* s_psrc = s_pat;
  const int* s_pdst = s_pat + Pe;
  const int* s_inoff = s_pat + 2 * Pe;
  const int* s_inq = s_inoff + Pn + 1;
  const int* s_outoff = s_inq + Pe;
  const int* s_outq = s_outoff + Pn + 1;
  const int tid = threadIdx.x;

  for (int t = tid; t < 4 * Pe + 2 * (Pn + 1); t += kBT) s_pat[t] = a.pat[t];
  __syncthreads();
  {
    // Shifted storage: Y = VF' - dEmin - cR and Z = VR' - cF with per-q FP64
    // shifts, so that the entries that can win a max are small numbers and an
    // FP32 store keeps their low bits.  With dR = lR - cR, dF = lF - cF
    // (statistics of the previous pass, in that pass's shifts):
    //   RMax = max(fillR, Y - dR)       FMax = max(fillF, max_e(Z[s_e] - dE) - dF)
    // New shifts for this pass's stores: lR, lF of the pass before the previous
    // one (the iteration has period two, so that value tracks lR, lF closely);
    // the first pass uses the previous pass's own.  Any finite shift is exact.
    const double* g = a.glob_in;
    const int x0 = 4 * Pe + Pn;
    auto split = [](double x, T* hi, T* lo, int q) {
      const T h = (T)x;
      hi[q] = h;
      lo[q] = (T)(x - (double)h);
    };
    for (int q = tid; q < Pp; q += kBT) {
      if (q >= Pe) {
        s_fillF[q] = s_fillR[q] = T(0);
        s_dF[q] = s_dFlo[q] = s_dR[q] = s_dRlo[q] = T(0);
        s_cR[q] = s_cRlo[q] = s_cF[q] = s_cFlo[q] = T(0);
        continue;
      }
      const double cRu = g[x0 + q], cFu = g[x0 + Pe + q];
      const double dR = g[2 * Pe + q], dF = g[3 * Pe + q];
      double fr = g[q] + cRu - g[4 * Pe + s_pdst[q]];
      double ff = g[Pe + q] + cFu - g[4 * Pe + s_psrc[q]];
      if (a.cnull) {
        fr -= a.cnull[q];
        ff -= a.cnull[q];
      }
      s_fillR[q] = (T)fr;
      s_fillF[q] = (T)ff;
      split(dR, s_dR, s_dRlo, q);
      split(dF, s_dF, s_dFlo, q);
      const double lRp = cRu + dR, lFp = cFu + dF;
      double cRn = a.first ? lRp : g[x0 + 2 * Pe + q];
      double cFn = a.first ? lFp : g[x0 + 3 * Pe + q];
      if (!isfinite(cRn)) cRn = 0.0;
      if (!isfinite(cFn)) cFn = 0.0;
      split(cRn, s_cR, s_cRlo, q);
      split(cFn, s_cF, s_cFlo, q);
      if (blockIdx.x == 0) {
        double* o = a.glob_out;
        o[x0 + q] = (double)s_cR[q] + (double)s_cRlo[q];
        o[x0 + Pe + q] = (double)s_cF[q] + (double)s_cFlo[q];
        o[x0 + 2 * Pe + q] = lRp;
        o[x0 + 3 * Pe + q] = lFp;
      }
    }
  }
  __syncthreads();

  // fixed columns: q-vector qv (vertex j0 of the tile), pattern vertex pc.
  // Everything a thread indexes in shared memory is fixed across tiles, so the
  // pointers and the pattern endpoints of its columns are set up once.
  const int qv = tid % nvec, j0 = tid / nvec;
  const bool qact = j0 < V;
  const int pc = tid % Pn, jp0 = tid / Pn, prows = kBT / Pn;
  T* const myF = s_F + j0 * Pp + qv * W;
  T* const myR = s_R + j0 * Pp + qv * W;
  const T* const myMU = s_MU + j0 * Pn;
  const T* const myMUlo = s_MUlo + j0 * Pn;
  const int qoff = j0 * Pp + qv * W;  // offset in a [V][Pp] stage block
  int pdst[W], psrc[W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const int q = qv * W + w;
    pdst[w] = q < Pe ? s_pdst[q] : 0;
    psrc[w] = q < Pe ? s_psrc[q] : 0;
  }
  const int in0 = s_inoff[pc], in1 = s_inoff[pc + 1];
  const int out0 = s_outoff[pc], out1 = s_outoff[pc + 1];
  const bool my_last = __ldg(a.iters_p + pc) == a.t;
  T mxF[W], mxR[W];
  OnlineLse<T> lr[W], lf[W], lmu;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    mxF[w] = neg_inf<T>();
    mxR[w] = neg_inf<T>();
    lr[w].init();
    lf[w].init();
  }
  lmu.init();

  const int ntiles = (Dn + V - 1) / V;
  const int cvec = Pnp / W;
  // Stage a tile's rows into shared memory with asynchronous 16-byte copies
  // (its vertices are consecutive, so every row block is contiguous).
  auto issue = [&](int tile, int k) {
    if (tile >= ntiles) return;
    unsigned char* st = smem + L.stage + (size_t)(k & 1) * L.stage_bytes;
    const int v0 = tile * V;
    const int nv = min(V, Dn - v0);
    const T* gM = a.M + (size_t)v0 * Pp;
    const T* gVF = a.vf + (size_t)v0 * Pp;
    const T* gEM = a.dEmin + (size_t)v0 * Pp;
    const T* gB = a.B + (size_t)v0 * Pp;
    T* sM = reinterpret_cast<T*>(st + L.sM);
    T* sVF = reinterpret_cast<T*>(st + L.sVF);
    T* sEM = reinterpret_cast<T*>(st + L.sEM);
    T* sB = reinterpret_cast<T*>(st + L.sB);
    for (int c = tid * W; c < nv * Pp; c += kBT * W) {
      cp16(sM + c, gM + c);
      cp16(sVF + c, gVF + c);
      cp16(sEM + c, gEM + c);
      cp16(sB + c, gB + c);
    }
    const T* gCV = a.CV + (size_t)v0 * Pnp;
    T* sCV = reinterpret_cast<T*>(st + L.sCV);
    for (int c = tid * W; c < nv * Pnp; c += kBT * W) cp16(sCV + c, gCV + c);
    const T* gCVl = a.CVlo + (size_t)v0 * Pnp;
    T* sCVl = reinterpret_cast<T*>(st + L.sCVl);
    for (int c = tid * W; c < nv * Pnp; c += kBT * W) cp16(sCVl + c, gCVl + c);
    int* sOff = reinterpret_cast<int*>(st + L.sOff);
    for (int j = tid; j <= nv; j += kBT) cp4(sOff + j, a.d_off + v0 + j);
  };
  (void)cvec;
  issue(blockIdx.x, 0);
  cp_commit();
  int k = 0;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++k) {
    issue(tile + gridDim.x, k + 1);  // next tile's copies fly while this one computes
    cp_commit();
    cp_wait1();
    __syncthreads();
    const unsigned char* st = smem + L.stage + (size_t)(k & 1) * L.stage_bytes;
    const T* sCV = reinterpret_cast<const T*>(st + L.sCV);
    const int* sOff = reinterpret_cast<const int*>(st + L.sOff);
    const int v0 = tile * V;
    const int v = v0 + j0;
    const bool vok = qact && v < Dn;
    VT bv = vfill<T>(T(0)), emv = vfill<T>(T(0));
    if (vok) {
      const bool has_in = sOff[j0 + 1] > sOff[j0];
      const VT mv = has_in ? *reinterpret_cast<const VT*>(reinterpret_cast<const T*>(st + L.sM) + qoff)
                           : vfill<T>(neg_inf<T>());
      const VT yv = *reinterpret_cast<const VT*>(reinterpret_cast<const T*>(st + L.sVF) + qoff);
      emv = *reinterpret_cast<const VT*>(reinterpret_cast<const T*>(st + L.sEM) + qoff);
      bv = *reinterpret_cast<const VT*>(reinterpret_cast<const T*>(st + L.sB) + qoff);
      // per-q constants of the thread's columns (16-byte shared loads)
      const VT fF = *reinterpret_cast<const VT*>(s_fillF + qv * W);
      const VT fR = *reinterpret_cast<const VT*>(s_fillR + qv * W);
      const VT dF = *reinterpret_cast<const VT*>(s_dF + qv * W);
      const VT dFl = *reinterpret_cast<const VT*>(s_dFlo + qv * W);
      const VT dR = *reinterpret_cast<const VT*>(s_dR + qv * W);
      const VT dRl = *reinterpret_cast<const VT*>(s_dRlo + qv * W);
      VT fo, ro;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        // no in-edges: M = -inf; no out-edges: Y = -inf; the fill wins
        vs<T>(fo, w, fmax(vg<T>(fF, w), (vg<T>(mv, w) - vg<T>(dF, w)) - vg<T>(dFl, w)));
        vs<T>(ro, w, fmax(vg<T>(fR, w), (vg<T>(yv, w) - vg<T>(dR, w)) - vg<T>(dRl, w)));
      }
      *reinterpret_cast<VT*>(myF) = fo;
      *reinterpret_cast<VT*>(myR) = ro;
    }
    __syncthreads();
    // MU_raw = -CV + sum F + sum R, compensated (CV carries a low part)
    for (int j = jp0; j < V && jp0 < prows; j += prows) {
      const int vv = v0 + j;
      if (vv >= Dn) break;
      const T* rowF = s_F + j * Pp;
      const T* rowR = s_R + j * Pp;
      CSum<T> mu;
      mu.init(-sCV[j * Pnp + pc]);
      mu.lo = -reinterpret_cast<const T*>(st + L.sCVl)[j * Pnp + pc];
      for (int t = in0; t < in1; ++t) mu.add(rowF[s_inq[t]]);
      for (int t = out0; t < out1; ++t) mu.add(rowR[s_outq[t]]);
      s_MU[j * Pn + pc] = mu.hi;
      s_MUlo[j * Pn + pc] = mu.lo;
      lmu.add2(mu.hi, mu.lo);
      if (my_last) a.mu_raw[(size_t)vv * Pn + pc] = mu.dvalue();
    }
    __syncthreads();
    if (!a.last && vok) {
      const VT fo = *reinterpret_cast<const VT*>(myF);
      const VT ro = *reinterpret_cast<const VT*>(myR);
      const VT cR = *reinterpret_cast<const VT*>(s_cR + qv * W);
      const VT cF = *reinterpret_cast<const VT*>(s_cF + qv * W);
      VT nf, nr;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        // f = VF' - cR, r = VR' - cF; the shift is taken off the compensated
        // MU_raw first (for the entries that matter the two are close, so the
        // difference is exact) and the small message after
        const VT cRl = *reinterpret_cast<const VT*>(s_cRlo + qv * W);
        const VT cFl = *reinterpret_cast<const VT*>(s_cFlo + qv * W);
        const T f = ((myMU[pdst[w]] - vg<T>(cR, w)) - vg<T>(fo, w)) + (myMUlo[pdst[w]] - vg<T>(cRl, w));
        T r = ((myMU[psrc[w]] - vg<T>(cF, w)) - vg<T>(ro, w)) + (myMUlo[psrc[w]] - vg<T>(cFl, w));
        T y;
        if (qv * W + w < Pe) {
          mxF[w] = fmax(mxF[w], f);
          mxR[w] = fmax(mxR[w], r);
          const T b = vg<T>(bv, w);
          lr[w].add_fast(f + b);
          lf[w].add_fast(r + b);
          y = f - vg<T>(emv, w);  // no out-edges: dEmin = +inf, Y = -inf
        } else {
          y = T(0);
          r = T(0);
        }
        vs<T>(nf, w, y);
        vs<T>(nr, w, r);
      }
      const size_t go = (size_t)v * Pp + (size_t)qv * W;
      *reinterpret_cast<VT*>(a.vf + go) = nf;
      *reinterpret_cast<VT*>(a.vr_out + go) = nr;
    }
    __syncthreads();  // the tile's smem rows and this stage are free
  }
  cp_wait0();

  // ---- block partials: mVF, mVR (max), lR, lF, S (lse); rows combined in order
  const int nmax = 2 * Pe;
  const int ncols = gridDim.x, col = blockIdx.x;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    __syncthreads();
    double* e = s_red + (size_t)tid * 6;
    e[0] = (double)mxF[w];
    e[1] = (double)mxR[w];
    e[2] = lr[w].mval();
    e[3] = lr[w].sval();
    e[4] = lf[w].mval();
    e[5] = lf[w].sval();
    __syncthreads();
    for (int c = tid; c < nvec; c += kBT) {
      const int q = c * W + w;
      if (q >= Pe) continue;
      double f = -CUDART_INF, r = -CUDART_INF, m1 = -CUDART_INF, s1 = 0, m2 = -CUDART_INF, s2 = 0;
      for (int row = 0; row < V; ++row) {
        const double* x = s_red + (size_t)(row * nvec + c) * 6;
        f = fmax(f, x[0]);
        r = fmax(r, x[1]);
        lse_merge(m1, s1, x[2], x[3]);
        lse_merge(m2, s2, x[4], x[5]);
      }
      a.bpart[(size_t)q * ncols + col] = f;
      a.bpart[(size_t)(Pe + q) * ncols + col] = r;
      a.bpart[(size_t)(nmax + 2 * q) * ncols + col] = m1;
      a.bpart[(size_t)(nmax + 2 * q + 1) * ncols + col] = s1;
      a.bpart[(size_t)(nmax + 2 * (Pe + q)) * ncols + col] = m2;
      a.bpart[(size_t)(nmax + 2 * (Pe + q) + 1) * ncols + col] = s2;
    }
  }
  __syncthreads();
  s_red[tid * 2] = lmu.mval();
  s_red[tid * 2 + 1] = lmu.sval();
  __syncthreads();
  for (int p = tid; p < Pn; p += kBT) {
    double m = -CUDART_INF, s = 0;
    for (int row = 0; row < prows; ++row)
      lse_merge(m, s, s_red[(row * Pn + p) * 2], s_red[(row * Pn + p) * 2 + 1]);
    a.bpart[(size_t)(nmax + 2 * (2 * Pe + p)) * ncols + col] = m;
    a.bpart[(size_t)(nmax + 2 * (2 * Pe + p) + 1) * ncols + col] = s;
  }
}


// ------------------------------------------------------ phase B, warp form
// Patterns with Pp <= 64 and Pn <= 64.  Lane l owns the QPL contiguous edge
// columns q = l * QPL + k and the pattern vertices p = l + 32 j (j < PPL); the
// per-q constants and statistics of its columns live in registers.  Each warp
// walks a contiguous range of vertices; their rows are staged into a per-warp
// double-buffered ring (kVps vertices per stage) with cp.async, so a warp never
// waits on another.  Per stage:
//   1. F, R of each staged vertex from its M, Y rows, written over them in the
//      stage;
//   2. the compensated sums MU_raw[v][p] = -CV[v][p] + sum F + sum R of all
//      staged vertices through a per-lane schedule built on the host
//      (vertex_warp_schedule): each (vertex, p) sum is one job whose terms are
//      -CV, then F[q] of the in-edges q of p ascending, then R[q] of its
//      out-edges ascending -- the order of the tile form -- and the jobs are
//      spread over the lanes longest first, so a lane runs ~1/32 of the
//      stage's terms instead of the largest pattern degree for every vertex;
//   3. per staged vertex: the MU_raw statistics and outputs of the lane's p,
//      and the new Y, Z of its columns from MU_raw[dst_q], MU_raw[src_q].
// Every sum keeps its terms and their order, so the results do not depend on
// how the jobs are spread.  Vertices without in-edges have M rows of -inf (set
// once, never written by phase A).
// Bound by instruction issue (2.7 of 4 a cycle from 16 warps an SM) and the shared
// memory pipe: one more load a term cost 5%.  R-MAT 22, pattern 32/64 (7.5 GB,
// 1.11 ms at the copy bandwidth): 1.74 ms an iteration with 102.9 M instructions
// and 10.1 M conflict cycles at R-MAT 18, 1.59 ms with 88.7 M and 5.3 M so.  The
// tail of a stage by a branch (predicated: 1% slower).  On a small graph a launch
// is its constants and its block partials.
constexpr int kVps = 4;  // vertices per stage (one add4_fast per column)
constexpr int kVw = kBT / 32;
template <int PPL>
struct VwSmem {
  size_t pat, sched, ring, mu, total, stage, warp_ring, mu_n;
  __host__ __device__ VwSmem(int Pn, int Pe, int Pp, int Pnp, int nterms) {
    const size_t sz = sizeof(float);
    size_t o = 0;
    pat = o; o += a16(sizeof(int) * (size_t)(4 * Pe + 2 * (Pn + 1)));
    sched = o; o += a16(sizeof(uint32_t) * (size_t)nterms * 32);
    stage = (size_t)VwStage(Pp, Pnp, true, kVps).n * sz;  // row sizes are 16-byte multiples
    warp_ring = 2 * stage;
    const size_t red = sizeof(double) * (size_t)kVw * (6 * Pe + 2 * Pn);  // aliases the rings
    ring = o; o += a16(red > kVw * warp_ring ? red : kVw * warp_ring);
    mu_n = 2 * kVps * (32 * PPL + 1);  // MU_raw hi | lo rows of the staged vertices
    mu = o; o += a16((size_t)kVw * mu_n * sz);
    total = o;
  }
};

// Two FP32 additions or subtractions in one instruction, each rounded to nearest
// as by itself; the last step of a message, ((u - c) - m) + (l - cl), on pairs.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
      " add.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
      " sub.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 message2(float2 u, float2 c, float2 m, float2 l, float2 cl) {
  return add2(sub2(sub2(u, c), m), sub2(l, cl));
}

template <int N>
__device__ __forceinline__ void lds_n(const float* p, float (&x)[N]) {
  if constexpr (N == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    x[0] = v.x;
    x[1] = v.y;
  } else {
    x[0] = *p;
  }
}
template <int N>
__device__ __forceinline__ void st_n(float* p, const float (&x)[N]) {
  if constexpr (N == 2) *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  else *p = x[0];
}

// Two blocks per SM bounds the registers at 128
template <int QPL, int PPL, bool REC>
__global__ void __launch_bounds__(kBT, 2)
vertex_warp_kernel(const VertexUpdArgs<float> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int Pe = a.Pe, Pn = a.Pn, Pp = a.Pp, Pnp = a.Pnp, Dn = a.Dn, nterms = a.vterms;
  const VwSmem<PPL> L(Pn, Pe, Pp, Pnp, nterms);
  const VwStage G(Pp, Pnp, true, kVps);
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  int* s_pat = reinterpret_cast<int*>(smem + L.pat);
  uint32_t* s_sched = reinterpret_cast<uint32_t*>(smem + L.sched);
  for (int t = tid; t < 4 * Pe + 2 * (Pn + 1); t += kBT) s_pat[t] = a.pat[t];
  for (int t = tid; t < nterms * 32; t += kBT) s_sched[t] = a.vsched[t];
  __syncthreads();
  dep_launch();
  dep_wait();
  const int* s_psrc = s_pat;
  const int* s_pdst = s_pat + Pe;

  // per-q constants (see the tile form for the algebra), formed once per block: FP64
  // arithmetic, 16 cycles an instruction and SM.  By every warp for its lanes they
  // were 8 us of a launch at 64 columns, whatever the graph's size.
  const double* g = a.glob_in;
  const int x0 = 4 * Pe + Pn;
  const int qo = lane * QPL;
  const bool qon = qo < Pp;
  float* s_cst = reinterpret_cast<float*>(smem + L.mu);  // [10][Pp], before the first sums
  for (int q = tid; q < Pp; q += kBT) {
    float c[10] = {};
    if (q < Pe) {
      const double cRu = g[x0 + q], cFu = g[x0 + Pe + q];
      const double dR = g[2 * Pe + q], dF = g[3 * Pe + q];
      double fr = g[q] + cRu - g[4 * Pe + s_pdst[q]];
      double ff = g[Pe + q] + cFu - g[4 * Pe + s_psrc[q]];
      if (a.cnull) {
        fr -= a.cnull[q];
        ff -= a.cnull[q];
      }
      const double lRp = cRu + dR, lFp = cFu + dF;
      double cRn = a.first ? lRp : g[x0 + 2 * Pe + q];
      double cFn = a.first ? lFp : g[x0 + 3 * Pe + q];
      if (!isfinite(cRn)) cRn = 0.0;
      if (!isfinite(cFn)) cFn = 0.0;
      c[0] = (float)ff;
      c[1] = (float)fr;
      c[2] = (float)dF;
      c[3] = (float)(dF - (double)c[2]);
      c[4] = (float)dR;
      c[5] = (float)(dR - (double)c[4]);
      c[6] = (float)cRn;
      c[7] = (float)(cRn - (double)c[6]);
      c[8] = (float)cFn;
      c[9] = (float)(cFn - (double)c[8]);
      if (blockIdx.x == 0) {
        double* o = a.glob_out;
        o[x0 + q] = (double)c[6] + (double)c[7];
        o[x0 + Pe + q] = (double)c[8] + (double)c[9];
        o[x0 + 2 * Pe + q] = lRp;
        o[x0 + 3 * Pe + q] = lFp;
      }
    }
#pragma unroll
    for (int x = 0; x < 10; ++x) s_cst[x * Pp + q] = c[x];
  }
  __syncthreads();
  float fF[QPL], fR[QPL], dFh[QPL], dFl[QPL], dRh[QPL], dRl[QPL], cRh[QPL], cRl[QPL], cFh[QPL], cFl[QPL];
  int qd[QPL], qs[QPL];
#pragma unroll
  for (int k = 0; k < QPL; ++k) {
    const int q = min(qo + k, Pp - 1);
    fF[k] = s_cst[q];
    fR[k] = s_cst[Pp + q];
    dFh[k] = s_cst[2 * Pp + q];
    dFl[k] = s_cst[3 * Pp + q];
    dRh[k] = s_cst[4 * Pp + q];
    dRl[k] = s_cst[5 * Pp + q];
    cRh[k] = s_cst[6 * Pp + q];
    cRl[k] = s_cst[7 * Pp + q];
    cFh[k] = s_cst[8 * Pp + q];
    cFl[k] = s_cst[9 * Pp + q];
    qd[k] = q < Pe ? s_pdst[q] : 0;
    qs[k] = q < Pe ? s_psrc[q] : 0;
  }
  __syncthreads();  // the MU_raw rows take the constants' place
  float mxF[QPL], mxR[QPL];
  OnlineLse<float> lr[QPL], lf[QPL], lmu[PPL];
  bool any_last = false;
  bool plast[PPL];  // this iteration is the last of pattern vertex p's pattern
#pragma unroll
  for (int k = 0; k < QPL; ++k) {
    mxF[k] = mxR[k] = neg_inf<float>();
    lr[k].init();
    lf[k].init();
  }
#pragma unroll
  for (int j = 0; j < PPL; ++j) {
    lmu[j].init();
    const int p = lane + 32 * j;
    plast[j] = p < Pn && __ldg(a.iters_p + p) == a.t;
    any_last = any_last || plast[j];
  }
  any_last = __any_sync(0xffffffffu, any_last);  // (one branch a vertex, none of the FP64 sums)

  const long long nw = (long long)gridDim.x * kVw;
  const long long gw = (long long)blockIdx.x * kVw + wib;
  const int vb = (int)(gw * Dn / nw), ve = (int)((gw + 1) * Dn / nw);
  unsigned char* ring = smem + L.ring + (size_t)wib * L.warp_ring;
  float* smu = reinterpret_cast<float*>(smem + L.mu) + (size_t)wib * L.mu_n;
  // MU_raw rows of the staged vertices, one word apart in bank order so that
  // the lanes ending jobs of one p for different vertices do not collide
  constexpr int kMuRow = 32 * PPL + 1;
  constexpr int kMuLo = kVps * kMuRow;  // the low parts after the high parts
  const size_t rowb = (size_t)Pp * sizeof(float), crow = (size_t)Pnp * sizeof(float);
  auto issue = [&](int v0, int buf) {
    const int nv = min(kVps, ve - v0);
    if (nv <= 0) return;
    unsigned char* st = ring + (size_t)buf * L.stage;
    const int n16 = (int)((size_t)nv * rowb / 16);
    const size_t go = (size_t)v0 * rowb;
    for (int c = lane; c < n16; c += 32) {
      cp16(st + G.oM * sizeof(float) + c * 16, reinterpret_cast<const unsigned char*>(a.M) + go + c * 16);
      cp16(st + G.oY * sizeof(float) + c * 16, reinterpret_cast<const unsigned char*>(a.vf) + go + c * 16);
      cp16(st + G.oE * sizeof(float) + c * 16, reinterpret_cast<const unsigned char*>(a.dEmin) + go + c * 16);
      cp16(st + G.oB * sizeof(float) + c * 16, reinterpret_cast<const unsigned char*>(a.B) + go + c * 16);
    }
    const int c16 = (int)((size_t)nv * crow / 16);
    const size_t co = (size_t)v0 * crow;
    for (int c = lane; c < c16; c += 32) {
      cp16(st + G.oC * sizeof(float) + c * 16, reinterpret_cast<const unsigned char*>(a.CV) + co + c * 16);
      cp16(st + G.oCl * sizeof(float) + c * 16, reinterpret_cast<const unsigned char*>(a.CVlo) + co + c * 16);
    }
  };
  issue(vb, 0);
  cp_commit();
  int buf = 0;
  for (int v0 = vb; v0 < ve; v0 += kVps, buf ^= 1) {
    issue(v0 + kVps, buf ^ 1);  // the next stage flies while this one computes
    cp_commit();
    cp_wait1();
    __syncwarp();
    float* st = reinterpret_cast<float*>(ring + (size_t)buf * L.stage);
    const int nv = min(kVps, ve - v0);
    // ---- 1. F over M, R over Y (a vertex past the stage's: unused)
    if (qon) {
#pragma unroll
      for (int jv = 0; jv < kVps; ++jv) {
        float m[QPL], y[QPL];
        float* sm_ = st + G.oM + jv * Pp + qo;
        float* sy_ = st + G.oY + jv * Pp + qo;
        lds_n<QPL>(sm_, m);
        lds_n<QPL>(sy_, y);
        // no in-edges: M = -inf; no out-edges: Y = -inf; the fill wins
        if constexpr (QPL == 2) {
          const float2 f2 = sub2(sub2({m[0], m[1]}, {dFh[0], dFh[1]}), {dFl[0], dFl[1]});
          const float2 r2 = sub2(sub2({y[0], y[1]}, {dRh[0], dRh[1]}), {dRl[0], dRl[1]});
          m[0] = fmaxf(fF[0], f2.x);
          m[1] = fmaxf(fF[1], f2.y);
          y[0] = fmaxf(fR[0], r2.x);
          y[1] = fmaxf(fR[1], r2.y);
        } else {
          const float2 v = sub2(sub2({m[0], y[0]}, {dFh[0], dRh[0]}), {dFl[0], dRl[0]});
          m[0] = fmaxf(fF[0], v.x);
          y[0] = fmaxf(fR[0], v.y);
        }
        st_n<QPL>(sm_, m);
        st_n<QPL>(sy_, y);
      }
    }
    __syncwarp();
    // ---- 2. the compensated sums of the stage's (vertex, p) jobs, four terms
    // per step: their schedule words in one 16-byte load, their values loaded
    // before the dependent additions
    {
      float hi = 0.f, lo = 0.f;
      const uint4* sch = reinterpret_cast<const uint4*>(s_sched) + lane;
      for (int t4 = 0; t4 < nterms / 4; ++t4) {
        const uint4 w4 = sch[t4 * 32];
        const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
        float x[4], xl[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float* xp = st + (w[u] & 0xfffu);
          x[u] = *xp;
          xl[u] = 0.f;
          if (w[u] & kSchedStart) xl[u] = xp[G.oCl - G.oC];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          // a job starts from (-CV_hi, -CV_lo)
          const bool first = (w[u] & kSchedStart) != 0;
          const float sm = hi + x[u];
          const float bp = sm - hi;
          const float l = lo + ((hi - (sm - bp)) + (x[u] - bp));
          hi = first ? -x[u] : sm;
          lo = first ? -xl[u] : l;
          if (w[u] & kSchedEnd) {
            const int slot = (int)((w[u] >> 16) & 0x1ffu);
            smu[slot] = hi;
            smu[kMuLo + slot] = lo;
          }
        }
      }
    }
    __syncwarp();
    // ---- 3. per staged vertex: MU_raw outputs, new Y and Z; the column
    // log-sum-exps take the stage's values four at a time (-inf: nothing)
    float lrv[QPL][kVps], lfv[QPL][kVps], muh[PPL][kVps], mul[PPL][kVps];
#pragma unroll
    for (int jv = 0; jv < kVps; ++jv) {
#pragma unroll
      for (int k = 0; k < QPL; ++k) lrv[k][jv] = lfv[k][jv] = neg_inf<float>();
#pragma unroll
      for (int j = 0; j < PPL; ++j) {
        muh[j][jv] = neg_inf<float>();
        mul[j][jv] = 0.f;
      }
    }
#pragma unroll
    for (int jv = 0; jv < kVps; ++jv) {
      if (jv >= nv) break;
      const size_t v = v0 + jv;
      const float* mu_hi = smu + jv * kMuRow;
#pragma unroll
      for (int j = 0; j < PPL; ++j) {
        const int p = lane + 32 * j;
        const bool pon = p < Pn;
        const float h = mu_hi[p], l = mu_hi[kMuLo + p];
        muh[j][jv] = pon ? h : neg_inf<float>();
        mul[j][jv] = pon ? l : 0.f;
        if (any_last && pon && plast[j]) a.mu_raw[v * Pn + p] = (double)h + (double)l;
        if constexpr (REC) {
          if (pon && a.rec_mh) {
            a.rec_mh[v * Pn + p] = h;
            a.rec_ml[v * Pn + p] = l;
          }
        }
      }
      if (!a.last && qon) {
        float F[QPL], R[QPL], em[QPL], b[QPL], f[QPL], r[QPL], yo[QPL];
        lds_n<QPL>(st + G.oM + jv * Pp + qo, F);
        lds_n<QPL>(st + G.oY + jv * Pp + qo, R);
        lds_n<QPL>(st + G.oE + jv * Pp + qo, em);
        lds_n<QPL>(st + G.oB + jv * Pp + qo, b);
        // f = VF' - cR, r = VR' - cF: the shift comes off the compensated
        // MU_raw first, the small message after
        if constexpr (QPL == 2) {
          const float2 f2 = message2({mu_hi[qd[0]], mu_hi[qd[1]]}, {cRh[0], cRh[1]}, {F[0], F[1]},
                                     {mu_hi[kMuLo + qd[0]], mu_hi[kMuLo + qd[1]]}, {cRl[0], cRl[1]});
          const float2 r2 = message2({mu_hi[qs[0]], mu_hi[qs[1]]}, {cFh[0], cFh[1]}, {R[0], R[1]},
                                     {mu_hi[kMuLo + qs[0]], mu_hi[kMuLo + qs[1]]}, {cFl[0], cFl[1]});
          f[0] = f2.x;
          f[1] = f2.y;
          r[0] = r2.x;
          r[1] = r2.y;
        } else {
          const float2 v2 = message2({mu_hi[qd[0]], mu_hi[qs[0]]}, {cRh[0], cFh[0]}, {F[0], R[0]},
                                     {mu_hi[kMuLo + qd[0]], mu_hi[kMuLo + qs[0]]}, {cRl[0], cFl[0]});
          f[0] = v2.x;
          r[0] = v2.y;
        }
#pragma unroll
        for (int k = 0; k < QPL; ++k) {
          if (qo + k < Pe) {
            mxF[k] = fmaxf(mxF[k], f[k]);
            mxR[k] = fmaxf(mxR[k], r[k]);
            lrv[k][jv] = f[k] + b[k];
            lfv[k][jv] = r[k] + b[k];
          }
          yo[k] = qo + k < Pe ? f[k] - em[k] : 0.f;  // no out-edges: dEmin = +inf, Y = -inf
          if (qo + k >= Pe) f[k] = r[k] = 0.f;
        }
        st_n<QPL>(a.vf + v * Pp + qo, yo);
        st_n<QPL>(a.vr_out + v * Pp + qo, r);
        if constexpr (REC) {
          if (a.rec_f) {
            st_n<QPL>(a.rec_f + v * Pp + qo, f);
            st_n<QPL>(a.rec_r + v * Pp + qo, r);
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < QPL; ++k) {
      lr[k].add4_fast(lrv[k][0], lrv[k][1], lrv[k][2], lrv[k][3]);
      lf[k].add4_fast(lfv[k][0], lfv[k][1], lfv[k][2], lfv[k][3]);
    }
#pragma unroll
    for (int j = 0; j < PPL; ++j) lmu[j].add2x4_fast(muh[j], mul[j]);
    __syncwarp();  // this stage's buffer is free for the stage after next
  }
  cp_wait0();
  __syncthreads();  // the rings become the reduction area

  const int nmax = 2 * Pe, nlse = 2 * Pe + Pn;
  double* red_s = reinterpret_cast<double*>(smem + L.ring);
  float* red_m = reinterpret_cast<float*>(red_s + (size_t)kVw * nlse);
  double* rs = red_s + (size_t)wib * nlse;
  float* rm = red_m + (size_t)wib * (nmax + nlse);
#pragma unroll
  for (int k = 0; k < QPL; ++k) {
    const int q = qo + k;
    if (q < Pe) {
      rm[q] = mxF[k];
      rm[Pe + q] = mxR[k];
      rm[nmax + q] = lr[k].m;
      rs[q] = lr[k].sval();
      rm[nmax + Pe + q] = lf[k].m;
      rs[Pe + q] = lf[k].sval();
    }
  }
#pragma unroll
  for (int j = 0; j < PPL; ++j) {
    const int p = lane + 32 * j;
    if (p < Pn) {
      rm[nmax + 2 * Pe + p] = lmu[j].m;
      rs[2 * Pe + p] = lmu[j].sval();
    }
  }
  __syncthreads();
  write_block_partials_f32(red_m, red_s, kVw, nmax, nlse, a.bpart, gridDim.x, blockIdx.x);
}

template <typename T>
__global__ void fill_kernel(T* __restrict__ p, size_t n, T v) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    p[i] = v;
}

#define ACG_EDGE_SHAPES(X) \
  X(1, 1) X(2, 1) X(4, 1) X(8, 1) X(16, 1) X(32, 1) X(32, 2) X(32, 4)

}  // namespace

int edge_step(WarpShape ws) { return (32 / ws.npow) * kU; }

WarpShape choose_warp_shape(int elem_bytes, int pp) {
  const int W = 16 / elem_bytes;
  const int nvec = (pp + W - 1) / W;
  WarpShape ws{32, 1};
  if (nvec <= 32) {
    int np = 1;
    while (np < nvec) np <<= 1;
    ws.npow = np;
    ws.nqv = 1;
  } else {
    ws.npow = 32;
    ws.nqv = nvec <= 64 ? 2 : 4;
  }
  return ws;
}

#define ACG_EDGE_LAUNCH(NP_, NQ_)                                           \
  if (ws.npow == NP_ && ws.nqv == NQ_) {                                    \
    if (a.argpos)                                                           \
      ACG_CUDA_TRY(launch_kernel(a.early, edge_max_kernel<T, NP_, NQ_, true>, blocks, kAT, 0, s, a));  \
    else                                                                    \
      ACG_CUDA_TRY(launch_kernel(a.early, edge_max_kernel<T, NP_, NQ_, false>, blocks, kAT, 0, s, a)); \
    return ACG_OK;                                                          \
  }

template <typename T>
acg_status launch_edge_max(const EdgeMaxArgs<T>& a, WarpShape ws, int blocks, cudaStream_t s) {
  if (a.nitems == 0) return ACG_OK;
  ACG_EDGE_SHAPES(ACG_EDGE_LAUNCH)
  return set_error(ACG_ERR_UNSUPPORTED, "no edge kernel for npow=%d nqv=%d", ws.npow, ws.nqv);
}

#define ACG_EDGE_OCC(NP_, NQ_)                                                        \
  if (ws.npow == NP_ && ws.nqv == NQ_) {                                             \
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, edge_max_kernel<T, NP_, NQ_, false>, \
                                                      kAT, 0) != cudaSuccess)        \
      nb = 1;                                                                        \
  }

template <typename T>
int edge_max_blocks_per_sm(WarpShape ws) {
  int nb = 1;
  ACG_EDGE_SHAPES(ACG_EDGE_OCC)
  return nb < 1 ? 1 : nb;
}


template <typename T>
acg_status launch_heavy_combine_arg(const T* partial, const int* ppos, const int* hbase,
                                    const int* hcount, const int* hvert, int nheavy, int Pp, T* M,
                                    int* A, cudaStream_t s) {
  if (nheavy == 0) return ACG_OK;
  heavy_combine_arg_kernel<T><<<ceil_div(nheavy, 8), 256, 0, s>>>(partial, ppos, hbase, hcount, hvert,
                                                                   nheavy, Pp, M, A);
  ACG_LAUNCH_CHECK();
  return ACG_OK;
}
template <typename T>
acg_status launch_heavy_combine(const T* partial, const int* hbase, const int* hcount,
                                const int* hvert, int nheavy, int Pp, T* M, bool early, cudaStream_t s) {
  if (nheavy == 0) return ACG_OK;
  if (Pp > kHeavyCols) return set_error(ACG_ERR_UNSUPPORTED, "heavy vertices: %d columns", Pp);
  ACG_CUDA_TRY(launch_kernel(early, heavy_combine_kernel<T>, nheavy, 256, 0, s, partial, hbase, hcount, hvert, Pp, M));
  return ACG_OK;
}

template <typename T>
size_t vertex_update_smem(int pn, int pe, int pp) {
  const int nvec = pp / VecT<T>::W;
  const int pnp = (pn + VecT<T>::W - 1) / VecT<T>::W * VecT<T>::W;
  return UpdSmem(kBT / nvec, pn, pe, pp, pnp, sizeof(T)).total;
}

template <int QPL, int PPL, bool REC>
size_t vertex_warp_setup(int pn, int pe, int pp, int pnp, int nterms) {
  const size_t sm = VwSmem<PPL>(pn, pe, pp, pnp, nterms).total;
  if (sm > 48 * 1024)
    cudaFuncSetAttribute(vertex_warp_kernel<QPL, PPL, REC>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  return sm;
}

// Calls f.template operator()<QPL, PPL>() for the warp form's shape; false if
// the pattern is too large for it.
template <typename F>
bool warp_form(int pn, int pp, F&& f) {
  if (pp > 64 || pn > 64) return false;
  if (pp <= 32 && pn <= 32) f.template operator()<1, 1>();
  else if (pp <= 32) f.template operator()<1, 2>();
  else if (pn <= 32) f.template operator()<2, 1>();
  else f.template operator()<2, 2>();
  return true;
}

template <typename T>
acg_status launch_vertex_update(const VertexUpdArgs<T>& a, int blocks, cudaStream_t s) {
  if (a.Pp > 64 && a.vsched) return launch_vertex_wide(a, blocks, s);
  cudaError_t le = cudaSuccess;
  if (a.vsched == nullptr && a.Pn > 0 && a.Pn <= 64 && a.Pp <= 64)
    return set_error(ACG_ERR_INVALID_ARGUMENT, "vertex phase: no schedule for the warp form");
  const bool warp = warp_form(a.Pn, a.Pp, [&]<int QPL, int PPL>() {
    auto go = [&]<bool REC>() {
      const size_t sm = vertex_warp_setup<QPL, PPL, REC>(a.Pn, a.Pe, a.Pp, a.Pnp, a.vterms);
      le = launch_kernel(a.early, vertex_warp_kernel<QPL, PPL, REC>, blocks, kBT, sm, s, a);
    };
    if (a.rec_f || a.rec_mh) go.template operator()<true>();
    else go.template operator()<false>();
  });
  if (warp) {
    if (le != cudaSuccess)
      return set_error(ACG_ERR_CUDA, "vertex_warp_kernel launch: %s", cudaGetErrorString(le));
    return ACG_OK;
  }
  const size_t sm = vertex_update_smem<T>(a.Pn, a.Pe, a.Pp);
  if (sm > 48 * 1024)
    ACG_CUDA_TRY(cudaFuncSetAttribute(vertex_update_kernel<T>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  vertex_update_kernel<T><<<blocks, kBT, sm, s>>>(a);
  ACG_LAUNCH_CHECK();
  return ACG_OK;
}

template <typename T>
int vertex_update_blocks(int pn, int pe, int pp, int pnp, int nterms, int num_sms, int dn) {
  int nb = 0;
  const bool warp = warp_form(pn, pp, [&]<int QPL, int PPL>() {
    const size_t sm = vertex_warp_setup<QPL, PPL, false>(pn, pe, pp, pnp, nterms);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, vertex_warp_kernel<QPL, PPL, false>, kBT,
                                                      sm) != cudaSuccess)
      nb = 1;
  });
  // (two per SM at most, whatever registers the compiler takes: the grid fixes the
  // warps' ranges of vertices, and with them the statistics' order of summation)
  if (warp) return num_sms * std::min(std::max(nb, 1), 2);
  const int V = kBT / (pp / VecT<T>::W);
  const long long tiles = (dn + V - 1) / V;
  const long long b = (long long)num_sms * vertex_update_blocks_per_sm<T>(pn, pe, pp);
  return (int)(tiles < 1 ? 1 : (tiles < b ? tiles : b));
}

int vertex_warp_schedule(const int* pat, int pn, int pe, int pp, int pnp, std::vector<uint32_t>* out) {
  return vertex_warp_schedule(pat, pn, pe, pp, pnp, kVps, out);
}

template <typename T>
acg_status launch_fill(T* p, size_t n, T v, cudaStream_t s) {
  if (n == 0) return ACG_OK;
  fill_kernel<T><<<(unsigned)std::min<size_t>((n + 255) / 256, 4096), 256, 0, s>>>(p, n, v);
  ACG_LAUNCH_CHECK();
  return ACG_OK;
}

template <typename T>
int vertex_update_blocks_per_sm(int pn, int pe, int pp) {
  const size_t sm = vertex_update_smem<T>(pn, pe, pp);
  if (sm > 48 * 1024)
    cudaFuncSetAttribute(vertex_update_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  int nb = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, vertex_update_kernel<T>, kBT, sm) !=
      cudaSuccess)
    nb = 1;
  return nb < 1 ? 1 : nb;
}

template acg_status launch_edge_max<double>(const EdgeMaxArgs<double>&, WarpShape, int, cudaStream_t);
template acg_status launch_edge_max<float>(const EdgeMaxArgs<float>&, WarpShape, int, cudaStream_t);
template acg_status launch_heavy_combine_arg<double>(const double*, const int*, const int*, const int*, const int*, int, int, double*, int*, cudaStream_t);
template acg_status launch_heavy_combine_arg<float>(const float*, const int*, const int*, const int*, const int*, int, int, float*, int*, cudaStream_t);
template acg_status launch_heavy_combine<double>(const double*, const int*, const int*, const int*, int, int, double*, bool, cudaStream_t);
template acg_status launch_heavy_combine<float>(const float*, const int*, const int*, const int*, int, int, float*, bool, cudaStream_t);
template acg_status launch_vertex_update<float>(const VertexUpdArgs<float>&, int, cudaStream_t);
template int edge_max_blocks_per_sm<double>(WarpShape);
template int edge_max_blocks_per_sm<float>(WarpShape);
template int vertex_update_blocks<float>(int, int, int, int, int, int, int);
template acg_status launch_fill<double>(double*, size_t, double, cudaStream_t);
template acg_status launch_fill<float>(float*, size_t, float, cudaStream_t);
template int vertex_update_blocks_per_sm<float>(int, int, int);

}  // namespace acg
