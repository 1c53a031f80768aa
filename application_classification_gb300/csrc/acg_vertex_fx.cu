// acg_vertex_fx.cu -- the vertex phase of FP64 plans (see acg_iter.cu for the
// algebra) in fixed-point arithmetic on the integer pipes.
//
// What bounds it: an FP64 instruction occupies an SM for 16 cycles (2 lanes per
// clock), and the phase needs 11 FP64 additions per (vertex, pattern edge)
// besides its log-sum-exps, 2.9 times the time its bytes take.  As 64-bit
// integers the same additions cost two integer instructions each and are exact.
// So a warp converts the rows it has staged to fixed point with Q fraction
// bits, forms F, R, MU_raw and the next f, r as integers, feeds their
// log-sum-exps without a conversion (fx_exp_scaled), and converts back only
// what it stores.  The arrays in memory stay FP64.
//
// Q is chosen per launch from the iteration's own constants, so that every
// quantity fits 60 bits: |F| <= |fill| + 1 (the edge term never exceeds 0, since
// M <= LSE(Z + B)), |CV| <= LSE(dV), hence |MU_raw| <= LSE(dV) + the fills of
// its edges, and f, r by the shifts on top.  With patterns of up to 48 vertices
// and unit features Q is 48 to 50, finer than a double's last place above 8.
// A stage that holds any other value, and a launch whose constants exceed 2^13
// or are not finite, run the same steps in FP64 (Fp64Ar); so every input the
// FP64 form took is handled as it was.
//
// A group of NW warps shares a stage of kFxVps vertices; the lanes of the group
// own QPL columns each (QPL = 2 and NW up to 4 cover 256 pattern edges) and
// PPL pattern vertices.  Two vertices per stage keep two blocks (16 warps) on
// an SM; the stage of four of the FP32 kernel would leave one.
// R-MAT 20, pattern 32/64 (1.05 M vertices, 3.5 GB, 0.52 ms at the copy
// bandwidth): FP64 8.77 ms an iteration, with integer exponentials 5.9, in fixed
// point 1.71, with the range checked on the words already in registers and the
// larger exponential table 1.42.  ncu: 900 warp instructions per vertex, the
// integer (ALU) pipe 59% busy, FP64 pipe 9%, DRAM 25%.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "acg_device.cuh"
#include "acg_iter.cuh"
#include "acg_vschedule.h"

namespace acg {

namespace {

constexpr int kFT = 256;     // threads per block
constexpr int kFW = kFxWarps;
static_assert(kFT == 32 * kFxWarps && kFxTableBytes == (int)sizeof(uint64_t) * kFxTable);

__device__ __forceinline__ void fcp16(void* sdst, const void* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc) : "memory");
}

// The group's barrier (a warp, or NW warps on named barrier 1 + group).
template <int NW>
__device__ __forceinline__ void group_sync(int group) {
  if constexpr (NW == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;\n" ::"r"(1 + group), "n"(32 * NW) : "memory");
}
// The same, returning whether any thread of the group passed true.
template <int NW>
__device__ __forceinline__ bool group_or(int group, bool x) {
  if constexpr (NW == 1) {
    const bool r = __any_sync(0xffffffffu, x);
    __syncwarp();
    return r;
  } else {
    int r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.s32 p, %3, 0;\n"
        " barrier.red.or.pred q, %1, %2, p;\n selp.s32 %0, 1, 0, q;\n}\n"
        : "=r"(r) : "r"(1 + group), "n"(32 * NW), "r"((int)x) : "memory");
    return r != 0;
  }
}

// Fixed point, and FP64 for the stages fixed point does not cover: the same
// operations on values of type V, kept in the stage in place of the doubles.
struct FxAr {
  using V = long long;
  int Q;
  int32_t c;            // fx_scaled_factor(Q)
  uint32_t lim;         // the high word of 2^(60 - Q)
  const uint64_t* tab;
  __device__ __forceinline__ V in(double x) const { return fx_from_double(x, Q); }
  __device__ __forceinline__ double out(V v) const { return fx_to_double(v, Q); }
  __device__ __forceinline__ V max2(V a, V b) const { return a > b ? a : b; }
  __device__ __forceinline__ void add(FxLse& l, V x) const {
    int k;
    const uint64_t f = fx_exp_scaled(x, Q, c, tab, k);
    fx_add_term(l, k, f);  // (no sum is wide here: see run_stage)
  }
};
struct Fp64Ar {
  using V = double;
  __device__ __forceinline__ V in(double x) const { return x; }
  __device__ __forceinline__ double out(V v) const { return v; }
  __device__ __forceinline__ V max2(V a, V b) const { return fmax(a, b); }
  __device__ __forceinline__ void add(FxLse& l, V x) const { fx_add(l, x); }
};

// What a lane carries across its vertices.
template <int QPL, int PPL>
struct LaneStats {
  FxLse lr[QPL], lf[QPL], lmu[PPL];
  long long mxF[QPL], mxR[QPL];  // maxima of the fixed-point stages
};

struct StageCtx {
  const VertexUpdArgs<double>* a;
  double* st;            // the stage
  double* smu;           // MU_raw rows of the staged vertices
  const uint32_t* sched;
  double* mxd;           // [2 Pp] maxima of the group's FP64 stages
  int gl, group, v0, nv, mu_row;
};

// One stage in arithmetic A; the column constants are the lane's.  In fixed
// point it returns true, before anything but the stage's M, Y and CV rows is
// changed, when the stage holds a value that fixed point does not cover: M or Y
// at 2^(60 - Q) or beyond (low ones only lose to the fill, as -inf does), CV
// outside +-2^(60 - Q), a NaN with a clear sign (fmax drops a NaN; a set sign
// reads as a low value), or a sum that is in the wide form.  B may lie anywhere:
// the terms of a vertex with a finite B outside +-2^(60 - Q) are added by
// fx_add_far once the stage's others are, so that fx_add_term never meets the wide
// form such a term may leave behind (beyond 2^24; the next stage then runs in FP64,
// whose ordinary terms bring the sum back).
template <typename A, int QPL, int PPL, int NW>
__device__ __forceinline__ bool run_stage(const A ar, const StageCtx& x, const typename A::V (&fF)[QPL],
                                          const typename A::V (&fR)[QPL], const typename A::V (&dF)[QPL],
                                          const typename A::V (&dR)[QPL], const typename A::V (&cF)[QPL],
                                          const typename A::V (&cR)[QPL], const int (&qd)[QPL],
                                          const int (&qs)[QPL], unsigned plast, LaneStats<QPL, PPL>& S) {
  using V = typename A::V;
  constexpr bool kFx = !std::is_same<V, double>::value;
  const VertexUpdArgs<double>& a = *x.a;
  const int Pe = a.Pe, Pn = a.Pn, Pp = a.Pp, Pnp = a.Pnp;
  const VwStage G(Pp, Pnp, false, kFxVps);
  V* const sv = reinterpret_cast<V*>(x.st);
  V* const smu = reinterpret_cast<V*>(x.smu);
  const int qo = x.gl * QPL;
  const bool qon = qo < Pp;
  bool bad = false;
  if constexpr (kFx) {
    uint32_t wide = 0;
#pragma unroll
    for (int k = 0; k < QPL; ++k) wide |= S.lr[k].w[3] | S.lf[k].w[3];
#pragma unroll
    for (int j = 0; j < PPL; ++j) wide |= S.lmu[j].w[3];
    bad = (int32_t)wide < 0;
  }
  // ---- 1. F over M, R over Y; -CV in place
#pragma unroll
  for (int jv = 0; jv < kFxVps; ++jv) {
    if (jv >= x.nv) break;
    if (qon) {
      const int im = G.oM + jv * Pp + qo, iy = G.oY + jv * Pp + qo;
      double m[QPL], y[QPL];
#pragma unroll
      for (int k = 0; k < QPL; ++k) {
        m[k] = x.st[im + k];
        y[k] = x.st[iy + k];
      }
#pragma unroll
      for (int k = 0; k < QPL; ++k) {
        if constexpr (kFx)
          bad |= __double2hiint(m[k]) >= (int)ar.lim || __double2hiint(y[k]) >= (int)ar.lim;
        // no in-edges: M = -inf; no out-edges: Y = -inf; the fill wins
        sv[im + k] = ar.max2(fF[k], ar.in(m[k]) - dF[k]);
        sv[iy + k] = ar.max2(fR[k], ar.in(y[k]) - dR[k]);
      }
    }
#pragma unroll
    for (int j = 0; j < PPL; ++j) {
      const int p = x.gl + 32 * NW * j;
      if (p < Pn) {
        const int ic = G.oC + jv * Pnp + p;
        const double cv = x.st[ic];
        if constexpr (kFx) bad |= ((uint32_t)__double2hiint(cv) & 0x7fffffffu) >= ar.lim;
        sv[ic] = -ar.in(cv);
      }
    }
  }
  if constexpr (kFx) {
    if (group_or<NW>(x.group, bad)) return true;
  } else {
    group_sync<NW>(x.group);
  }
  // ---- 2. the sums MU_raw of the stage's (vertex, p) jobs
  {
    V s = V(0);
    const uint4* sch = reinterpret_cast<const uint4*>(x.sched) + x.gl;
    for (int t4 = 0; t4 < a.vterms / 4; ++t4) {
      const uint4 w4 = sch[t4 * 32 * NW];
      const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
      V t[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) t[u] = sv[w[u] & 0xfffu];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s = ((w[u] & kSchedStart) ? V(0) : s) + t[u];
        if (w[u] & kSchedEnd) smu[(w[u] >> 16) & 0x1ffu] = s;
      }
    }
  }
  group_sync<NW>(x.group);
  // ---- 3. MU_raw outputs and statistics, the new Y and Z
  bool far = false;
#pragma unroll
  for (int jv = 0; jv < kFxVps; ++jv) {
    if (jv >= x.nv) break;
    const size_t v = (size_t)(x.v0 + jv);
    const V* mu = smu + jv * x.mu_row;
#pragma unroll
    for (int j = 0; j < PPL; ++j) {
      const int p = x.gl + 32 * NW * j;
      if (p < Pn) {
        const V h = mu[p];
        ar.add(S.lmu[j], h);
        if (((plast >> j) & 1u) || a.rec_mh) {
          const double d = ar.out(h);
          if ((plast >> j) & 1u) a.mu_raw[v * Pn + p] = d;
          if (a.rec_mh) {
            a.rec_mh[v * Pn + p] = d;
            a.rec_ml[v * Pn + p] = 0.0;
          }
        }
      }
    }
    if (!a.last && qon) {
      double yo[QPL], zo[QPL], fo[QPL];
#pragma unroll
      for (int k = 0; k < QPL; ++k) {
        yo[k] = zo[k] = fo[k] = 0.0;
        const int i = jv * Pp + qo + k;
        const V f = (mu[qd[k]] - cR[k]) - sv[G.oM + i];
        const V r = (mu[qs[k]] - cF[k]) - sv[G.oY + i];
        const double em = x.st[G.oE + i], b = x.st[G.oB + i];
        if (qo + k < Pe) {
          if constexpr (kFx) {
            S.mxF[k] = ar.max2(S.mxF[k], f);
            S.mxR[k] = ar.max2(S.mxR[k], r);
            const uint32_t hb = (uint32_t)__double2hiint(b);
            if ((hb & 0x7fffffffu) < ar.lim) {
              const V bx = ar.in(b);
              ar.add(S.lr[k], f + bx);
              ar.add(S.lf[k], r + bx);
            } else {
              far |= hb != 0xfff00000u;  // (no out-edges, B = -inf: adds nothing)
            }
          } else {
            x.mxd[qo + k] = fmax(x.mxd[qo + k], f);
            x.mxd[Pp + qo + k] = fmax(x.mxd[Pp + qo + k], r);
            ar.add(S.lr[k], f + b);
            ar.add(S.lf[k], r + b);
          }
          // Y from the rounded f: the adjoint restores it from a checkpoint of
          // f as this same difference (no out-edges: dEmin = +inf, Y = -inf)
          fo[k] = ar.out(f);
          yo[k] = fo[k] - em;
          zo[k] = ar.out(r);
          if constexpr (kFx) zo[k] = r == 0 ? 0x1p-100 : zo[k];  // (edge_word)
          else zo[k] = edge_word(zo[k], a.wide);
        }
      }
      double* gy = a.vf + v * Pp + qo;
      double* gz = a.vr_out + v * Pp + qo;
      if constexpr (QPL == 2) {
        *reinterpret_cast<double2*>(gy) = make_double2(yo[0], yo[1]);
        *reinterpret_cast<double2*>(gz) = make_double2(zo[0], zo[1]);
      } else {
        gy[0] = yo[0];
        gz[0] = zo[0];
      }
      if (a.rec_f) {
#pragma unroll
        for (int k = 0; k < QPL; ++k) {
          a.rec_f[v * Pp + qo + k] = fo[k];
          a.rec_r[v * Pp + qo + k] = zo[k];
        }
      }
    }
  }
  if constexpr (kFx) {
    if (far) {  // (a.last leaves it clear; the stage's rows are as above)
#pragma unroll 1
      for (int jv = 0; jv < x.nv; ++jv) {
        const V* mu = smu + jv * x.mu_row;
#pragma unroll
        for (int k = 0; k < QPL; ++k) {
          const int i = jv * Pp + qo + k;
          const double b = x.st[G.oB + i];
          if (qo + k >= Pe || ((uint32_t)__double2hiint(b) & 0x7fffffffu) < ar.lim) continue;
          S.lr[k] = fx_add_far(S.lr[k], ar.out((mu[qd[k]] - cR[k]) - sv[G.oM + i]) + b);
          S.lf[k] = fx_add_far(S.lf[k], ar.out((mu[qs[k]] - cF[k]) - sv[G.oY + i]) + b);
        }
      }
    }
  }
  return false;
}

// GS: the schedule stays in global memory (acg_vschedule.h).
template <int QPL, int PPL, int NW, bool GS>
__global__ void __launch_bounds__(kFT, 2) vertex_fx_kernel(const VertexUpdArgs<double> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int Pe = a.Pe, Pn = a.Pn, Pp = a.Pp, Pnp = a.Pnp, Dn = a.Dn, nterms = a.vterms;
  constexpr int kNG = kFW / NW;
  const FxSmem L(Pn, Pe, Pp, Pnp, nterms, NW, GS);
  const VwStage G(Pp, Pnp, false, kFxVps);
  const int tid = threadIdx.x;
  int* s_pat = reinterpret_cast<int*>(smem + L.pat);
  uint32_t* s_sched = reinterpret_cast<uint32_t*>(smem + L.sched);
  double* s_cst = reinterpret_cast<double*>(smem + L.cst);
  double* s_mxd = reinterpret_cast<double*>(smem + L.mxd);
  float* s_amp = reinterpret_cast<float*>(smem + L.amp);
  int* s_bound = reinterpret_cast<int*>(smem + L.flags);  // float bits: [0] columns, [1] MU_raw
  for (int t = tid; t < 4 * Pe + 2 * (Pn + 1); t += kFT) s_pat[t] = a.pat[t];
  if constexpr (!GS)
    for (int t = tid; t < nterms * 32 * NW; t += kFT) s_sched[t] = a.vsched[t];
  for (int t = tid; t < 2 * Pp * kNG; t += kFT) s_mxd[t] = -CUDART_INF;
  for (int t = tid; t < kFxTable; t += kFT) reinterpret_cast<uint64_t*>(smem + L.tab)[t] = fx_table_entry(t);
  if (tid < 2) s_bound[tid] = 0;
  __syncthreads();
  dep_launch();
  dep_wait();
  const int* s_psrc = s_pat;
  const int* s_pdst = s_pat + Pe;

  const int gl = tid % (32 * NW), group = tid / (32 * NW);
  const long long ng = (long long)gridDim.x * kNG;
  const long long gg = (long long)blockIdx.x * kNG + group;
  const int vb = (int)(gg * Dn / ng), ve = (int)((gg + 1) * Dn / ng);
  unsigned char* ring = smem + L.ring + (size_t)group * L.group_ring;
  const size_t rowb = (size_t)Pp * 8, crow = (size_t)Pnp * 8;
  auto issue = [&](int v0, int buf) {
    const int nv = min(kFxVps, ve - v0);
    if (nv <= 0) return;
    unsigned char* st = ring + (size_t)buf * L.stage;
    const int n16 = (int)((size_t)nv * rowb / 16);
    const size_t go = (size_t)v0 * rowb;
    for (int c = gl; c < n16; c += 32 * NW) {
      fcp16(st + G.oM * 8 + c * 16, reinterpret_cast<const unsigned char*>(a.M) + go + c * 16);
      fcp16(st + G.oY * 8 + c * 16, reinterpret_cast<const unsigned char*>(a.vf) + go + c * 16);
      fcp16(st + G.oE * 8 + c * 16, reinterpret_cast<const unsigned char*>(a.dEmin) + go + c * 16);
      fcp16(st + G.oB * 8 + c * 16, reinterpret_cast<const unsigned char*>(a.B) + go + c * 16);
    }
    const int c16 = (int)((size_t)nv * crow / 16);
    const size_t co = (size_t)v0 * crow;
    for (int c = gl; c < c16; c += 32 * NW)
      fcp16(st + G.oC * 8 + c * 16, reinterpret_cast<const unsigned char*>(a.CV) + co + c * 16);
  };
  issue(vb, 0);  // (flies while the constants are formed)
  asm volatile("cp.async.commit_group;\n" ::: "memory");

  // ---- the columns' constants (acg_iter.cu has the algebra), their bounds
  const double* g = a.glob_in;
  const int x0 = 4 * Pe + Pn;
  for (int q = tid; q < Pp; q += kFT) {
    double fF = 0, fR = 0, dF = 0, dR = 0, cF = 0, cR = 0;
    if (q < Pe) {
      const double cRu = g[x0 + q], cFu = g[x0 + Pe + q];
      dR = g[2 * Pe + q];
      dF = g[3 * Pe + q];
      fR = g[q] + cRu - g[4 * Pe + s_pdst[q]];
      fF = g[Pe + q] + cFu - g[4 * Pe + s_psrc[q]];
      if (a.cnull) {
        fR -= a.cnull[q];
        fF -= a.cnull[q];
      }
      const double lRp = cRu + dR, lFp = cFu + dF;
      cR = a.first ? lRp : g[x0 + 2 * Pe + q];
      cF = a.first ? lFp : g[x0 + 3 * Pe + q];
      if (!isfinite(cR)) cR = 0.0;
      if (!isfinite(cF)) cF = 0.0;
      // (rounded up; NaN and infinities come out above every limit)
      const float aF = __double2float_ru(fabs(fF) + 1.0), aR = __double2float_ru(fabs(fR) + 1.0);
      s_amp[q] = aF;
      s_amp[Pp + q] = aR;
      const double m = fabs(dF) + fabs(dR) + fabs(cF) + fabs(cR) + fabs(fF) + fabs(fR);
      const float mf = m < 1e9 ? __double2float_ru(m) + 2.f : 1e9f;
      atomicMax(s_bound, __float_as_int(mf));
      if (blockIdx.x == 0) {
        double* o = a.glob_out;
        o[x0 + 2 * Pe + q] = lRp;
        o[x0 + 3 * Pe + q] = lFp;
      }
    }
    s_cst[q] = fF;
    s_cst[Pp + q] = fR;
    s_cst[2 * Pp + q] = dF;
    s_cst[3 * Pp + q] = dR;
    s_cst[4 * Pp + q] = cF;
    s_cst[5 * Pp + q] = cR;
  }
  __syncthreads();
  {
    const int* inoff = s_pat + 2 * Pe;
    const int* inq = inoff + Pn + 1;
    const int* outoff = inq + Pe;
    const int* outq = outoff + Pn + 1;
    for (int p = tid; p < Pn; p += kFT) {
      const double l = fabs(a.lse_pos[p]);
      float m = l < 1e9 ? __double2float_ru(l) + 1.f : 1e9f;
      for (int t = inoff[p]; t < inoff[p + 1]; ++t) m += s_amp[inq[t]];
      for (int t = outoff[p]; t < outoff[p + 1]; ++t) m += s_amp[Pp + outq[t]];
      atomicMax(s_bound + 1, __float_as_int(m < 1e9f ? m : 1e9f));  // NaN, inf: 1e9
    }
  }
  __syncthreads();
  // every |MU_raw|, |f|, |r| is below the bound, so below 2^60 with Q fraction bits
  const float bound = (__int_as_float(s_bound[0]) + __int_as_float(s_bound[1])) * 1.001f + 64.f;
  const bool fixed = bound < 8192.f;
  // (at most 50: finer than a double from 4 on, and B, dEmin may reach 2^10)
  const int Q = fixed ? min(50, 60 - ((__float_as_int(bound) >> 23) - 126)) : 47;

  // in fixed point, once per block (the second stage of the first group's ring: not
  // yet in use; 48 Pp bytes of at least 64 Pp); the shifts also as they are
  // subtracted: multiples of 2^-Q, exact as doubles
  static_assert(kFxVps >= 2, "room for the columns' constants");
  long long* s_fix = reinterpret_cast<long long*>(smem + L.ring + L.stage);
  for (int t = tid; t < 6 * Pp; t += kFT) {
    const long long k = fixed ? __double2ll_rn(s_cst[t] * (double)(1ull << Q)) : 0ll;
    s_fix[t] = k;
    if (fixed && t >= 4 * Pp) s_cst[t] = (double)k * (1.0 / (double)(1ull << Q));
  }
  __syncthreads();

  const int qo = gl * QPL;
  uint64_t* s_tab = reinterpret_cast<uint64_t*>(smem + L.tab);
  const FxAr fx{Q, fx_scaled_factor(Q), (uint32_t)(1083 - Q) << 20, s_tab};
  long long fFx[QPL], fRx[QPL], dFx[QPL], dRx[QPL], cFx[QPL], cRx[QPL];
  int qd[QPL], qs[QPL];
  LaneStats<QPL, PPL> S;
#pragma unroll
  for (int k = 0; k < QPL; ++k) {
    const int q = qo + k;
    const bool on = q < Pp;
    auto cst = [&](int i) { return on ? s_fix[i * Pp + q] : 0ll; };  // rounded to Q fraction bits
    fFx[k] = cst(0);
    fRx[k] = cst(1);
    dFx[k] = cst(2);
    dRx[k] = cst(3);
    cFx[k] = cst(4);
    cRx[k] = cst(5);
    qd[k] = q < Pe ? s_pdst[q] : 0;
    qs[k] = q < Pe ? s_psrc[q] : 0;
    fx_init(S.lr[k]);
    fx_init(S.lf[k]);
    S.mxF[k] = S.mxR[k] = (long long)0x8000000000000000ull;
  }
  __syncthreads();  // s_fix is read: the ring may fill
  if (blockIdx.x == 0)
    for (int q = tid; q < Pe; q += kFT) {
      a.glob_out[x0 + q] = s_cst[5 * Pp + q];
      a.glob_out[x0 + Pe + q] = s_cst[4 * Pp + q];
    }
  unsigned plast = 0;  // bit j: this iteration is the last of the lane's j-th pattern vertex
#pragma unroll
  for (int j = 0; j < PPL; ++j) {
    fx_init(S.lmu[j]);
    const int p = gl + 32 * NW * j;
    if (p < Pn && __ldg(a.iters_p + p) == a.t) plast |= 1u << j;
  }

  // The stage's M, Y and CV rows again, where fixed point had begun on them (Y's
  // row in memory is rewritten at the end of its stage only).
  auto restage = [&](int v0, int nv, unsigned char* st) {
    const int n16 = (int)((size_t)nv * rowb / 16), c16 = (int)((size_t)nv * crow / 16);
    for (int c = gl; c < n16; c += 32 * NW) {
      *reinterpret_cast<uint4*>(st + G.oM * 8 + c * 16) =
          *reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(a.M) + (size_t)v0 * rowb + c * 16);
      *reinterpret_cast<uint4*>(st + G.oY * 8 + c * 16) =
          *reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(a.vf) + (size_t)v0 * rowb + c * 16);
    }
    for (int c = gl; c < c16; c += 32 * NW)
      *reinterpret_cast<uint4*>(st + G.oC * 8 + c * 16) =
          *reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(a.CV) + (size_t)v0 * crow + c * 16);
  };
  StageCtx x{&a, nullptr, reinterpret_cast<double*>(smem + L.mu) + (size_t)group * L.mu_n, GS ? a.vsched : s_sched,
             s_mxd + (size_t)group * 2 * Pp, gl, group, 0, 0, L.mu_row};
  int buf = 0;
  for (int v0 = vb; v0 < ve; v0 += kFxVps, buf ^= 1) {
    issue(v0 + kFxVps, buf ^ 1);  // the next stage flies while this one computes
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    unsigned char* st = ring + (size_t)buf * L.stage;
    x.st = reinterpret_cast<double*>(st);
    x.v0 = v0;
    x.nv = min(kFxVps, ve - v0);
    group_sync<NW>(group);
    if (!fixed || run_stage<FxAr, QPL, PPL, NW>(fx, x, fFx, fRx, dFx, dRx, cFx, cRx, qd, qs, plast, S)) {
      if (fixed) {
        restage(v0, x.nv, st);
        group_sync<NW>(group);
      }
      double fF[QPL], fR[QPL], dF[QPL], dR[QPL], cF[QPL], cR[QPL];
#pragma unroll
      for (int k = 0; k < QPL; ++k) {
        const int q = qo + k;
        auto cst = [&](int i) { return q < Pp ? s_cst[i * Pp + q] : 0.0; };
        fF[k] = cst(0);
        fR[k] = cst(1);
        dF[k] = cst(2);
        dR[k] = cst(3);
        cF[k] = cst(4);
        cR[k] = cst(5);
      }
      run_stage<Fp64Ar, QPL, PPL, NW>(Fp64Ar{}, x, fF, fR, dF, dR, cF, cR, qd, qs, plast, S);
    }
    group_sync<NW>(group);  // this stage's buffer is free for the stage after next
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();  // the rings become the reduction area

  // ---- block partials: 2 Pe maxima (doubles), then the 2 Pe + Pn sums (four words each)
  const int nmax = 2 * Pe, nlse = 2 * Pe + Pn;
  double* rmx = reinterpret_cast<double*>(smem + L.ring);                // [kNG][nmax]
  FxLse* rls = reinterpret_cast<FxLse*>(rmx + (size_t)kNG * nmax);       // [kNG][nlse]
#pragma unroll
  for (int k = 0; k < QPL; ++k) {
    const int q = qo + k;
    if (q < Pe) {
      const long long none = (long long)0x8000000000000000ull;
      double f = x.mxd[q], r = x.mxd[Pp + q];
      if (S.mxF[k] != none) f = fmax(f, fx.out(S.mxF[k]));
      if (S.mxR[k] != none) r = fmax(r, fx.out(S.mxR[k]));
      rmx[(size_t)group * nmax + q] = f;
      rmx[(size_t)group * nmax + Pe + q] = r;
      rls[(size_t)group * nlse + q] = S.lr[k];
      rls[(size_t)group * nlse + Pe + q] = S.lf[k];
    }
  }
#pragma unroll
  for (int j = 0; j < PPL; ++j) {
    const int p = gl + 32 * NW * j;
    if (p < Pn) rls[(size_t)group * nlse + 2 * Pe + p] = S.lmu[j];
  }
  __syncthreads();
  const int ncols = gridDim.x, col = blockIdx.x;
  for (int j = tid; j < nmax + nlse; j += kFT) {
    if (j < nmax) {
      double m = rmx[j];
      for (int w = 1; w < kNG; ++w) m = fmax(m, rmx[(size_t)w * nmax + j]);
      a.bpart[(size_t)j * ncols + col] = m;
    } else {
      const int i = j - nmax;
      FxLse l = rls[i];
      for (int w = 1; w < kNG; ++w) fx_merge(l, rls[(size_t)w * nlse + i]);
      double m, s;
      fx_pair(l, m, s);
      a.bpart[(size_t)(nmax + 2 * i) * ncols + col] = m;
      a.bpart[(size_t)(nmax + 2 * i + 1) * ncols + col] = s;
    }
  }
}

// The shape for a pattern: NW warps a group (64 columns and 64 pattern vertices
// each), QPL columns and PPL pattern vertices a lane.
template <typename F>
void fx_form(int pn, int pp, F&& f) {
  if (pp <= 64 && pn <= 64) {
    if (pp <= 32 && pn <= 32) f.template operator()<1, 1, 1>();
    else if (pp <= 32) f.template operator()<1, 2, 1>();
    else if (pn <= 32) f.template operator()<2, 1, 1>();
    else f.template operator()<2, 2, 1>();
  } else if (pp <= 128) {
    if (pn <= 64) f.template operator()<2, 1, 2>();
    else f.template operator()<2, 2, 2>();
  } else {
    f.template operator()<2, 1, 4>();
  }
}

}  // namespace

int vertex_fx_warps(int pn, int pp) { return pp <= 64 && pn <= 64 ? 1 : pp <= 128 ? 2 : 4; }

int vertex_fx_schedule(const int* pat, int pn, int pe, int pp, int pnp, std::vector<uint32_t>* out) {
  return vertex_warp_schedule(pat, pn, pe, pp, pnp, kFxVps, out, 32 * vertex_fx_warps(pn, pp), 2, 8);
}

// f(kernel, shared memory) of the kernel for a pattern.
template <typename F>
static void fx_kernel(int pn, int pe, int pp, int pnp, int nterms, F&& f) {
  fx_form(pn, pp, [&]<int QPL, int PPL, int NW>() {
    const size_t sm = FxSmem(pn, pe, pp, pnp, nterms, NW, false).total;
    if constexpr (NW == 4)  // (fewer warps' schedules fit, of every pattern)
      if (sm > kBlockSmem) {
        f(vertex_fx_kernel<QPL, PPL, NW, true>, FxSmem(pn, pe, pp, pnp, nterms, NW, true).total);
        return;
      }
    f(vertex_fx_kernel<QPL, PPL, NW, false>, sm);
  });
}

acg_status launch_vertex_fx(const VertexUpdArgs<double>& a, int blocks, cudaStream_t s) {
  if (a.vsched == nullptr)
    return set_error(ACG_ERR_INVALID_ARGUMENT, "vertex phase: no schedule of the sums");
  cudaError_t le = cudaSuccess;
  fx_kernel(a.Pn, a.Pe, a.Pp, a.Pnp, a.vterms, [&](auto kernel, size_t sm) {
    if (sm > 48 * 1024)
      le = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (le != cudaSuccess) return;
    le = launch_kernel(a.early, kernel, blocks, kFT, sm, s, a);
  });
  if (le != cudaSuccess)
    return set_error(ACG_ERR_CUDA, "vertex_fx_kernel launch: %s", cudaGetErrorString(le));
  return ACG_OK;
}

int vertex_fx_blocks(int pn, int pe, int pp, int pnp, int nterms, int num_sms, int dn) {
  int nb = 0;
  fx_kernel(pn, pe, pp, pnp, nterms, [&](auto kernel, size_t sm) {
    if (sm > 48 * 1024)
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, kFT, sm) != cudaSuccess) nb = 1;
  });
  // (a stage per group at least: fewer partials to finalise on small graphs)
  const int per = kFxVps * kFW / vertex_fx_warps(pn, pp);
  return std::min(num_sms * (nb < 1 ? 1 : nb), std::max(1, ceil_div(dn, per)));
}

}  // namespace acg
