// acg_vertex_wide.cu -- the vertex phase of FP32 plans with more than 64 padded
// edge columns (see acg_iter.cu for the algebra and vertex_update_kernel, whose
// results these are, bit for bit).
//
// The block-tile form spent its time at its four block barriers per tile of 4 to
// 15 vertices and in the sums MU_raw, where a thread walked one pattern
// vertex's edges for two or three rows while the others of its warp waited (500
// cycles a vertex and SM at 120 columns, against 150 for its bytes).  Here a
// row of the tile belongs to one warp (two above 128 columns) for the whole
// launch: its lanes own four columns each, statistics in registers, its vertices (one per tile) are staged two at a time with cp.async,
// and the sums run through the balanced per-lane schedule of the warp form.
// What ties the rows of a block together, the statistics of MU_raw, whose order
// runs over the rows of each tile, is added from a shared copy of MU_raw after
// one block barrier per two tiles.
// A thread's columns, rows and pattern vertices, and the order of every sum, are
// those of the tile form: a block of V = 256 / (Pp / 4) rows walks the tiles
// blockIdx.x, blockIdx.x + gridDim.x, ...
// R-MAT 18, pattern 40/120 (0.84 GB, 124 us at the copy bandwidth): 458 us an
// iteration as block tiles, 233 so (and 48 of merges, in a batch beside the edge phase);
// 131,072 vertices, patterns of 132 to 192 columns: 284 -> 190 us.  Two columns a
// lane with twice the warps was slower (435 us: the copies, the schedule and the
// barriers are per warp), and so were constants held in registers (326).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "acg_device.cuh"
#include "acg_iter.cuh"
#include "acg_vschedule.h"

namespace acg {

namespace {

constexpr int kTileThreads = 256;  // the tile form's block, which fixes V
// Terms a lane above which a pattern whose rows take two warps is left to the
// block-tile form: a hub's sum is one lane's, in each row, while the tile form's
// threads share out the rows.  100,000 vertices, ten iterations, tile form / this one:
// 136 edges, longest sum 86 and 110 terms 7.13 / 7.00 and 7.42 / 7.66 ms; 170, 105 and
// 138: 8.46 / 8.43 and 9.07 / 9.35; 254, 79 and 155: 9.07 / 8.70 and 10.91 / 11.03; a
// star of 254: 12.95 / 14.03.  Rows of one warp gain for every hub (a star of 128
// edges 6.40 / 5.45).
constexpr int kWideTerms = 104;

__device__ __forceinline__ void wcp16(void* sdst, const void* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc) : "memory");
}
// The warps of one row: a warp, or two on named barrier 1 + row (at most 7 rows).
template <int NW>
__device__ __forceinline__ void row_sync(int row) {
  if constexpr (NW == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;\n" ::"r"(1 + row), "n"(32 * NW) : "memory");
}
__device__ __forceinline__ void ld4(const float* p, float (&x)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  x[0] = v.x;
  x[1] = v.y;
  x[2] = v.z;
  x[3] = v.w;
}
__device__ __forceinline__ void st4(float* p, const float (&x)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}

// The block has 32 NW V threads; kThreads bounds them, kBlocks of such blocks fit
// an SM's registers.
template <int NW, int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks) vertex_wide_kernel(const VertexUpdArgs<float> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int Pe = a.Pe, Pn = a.Pn, Pp = a.Pp, Pnp = a.Pnp, Dn = a.Dn, nterms = a.vterms;
  const int nvec = Pp / 4, V = kTileThreads / nvec;
  const WideSmem L(V, Pn, Pe, Pp, Pnp, nterms, NW);
  const VwStage G(Pp, Pnp, true, kWv);
  const int tid = threadIdx.x, nt = blockDim.x;
  int* s_pat = reinterpret_cast<int*>(smem + L.pat);
  uint32_t* s_sched = reinterpret_cast<uint32_t*>(smem + L.sched);
  float* s_cst = reinterpret_cast<float*>(smem + L.cst);  // [10][Pp]
  for (int t = tid; t < 2 * Pe; t += nt) s_pat[t] = a.pat[t];
  for (int t = tid; t < nterms * 32 * NW; t += nt) s_sched[t] = a.vsched[t];
  __syncthreads();
  const int* s_psrc = s_pat;
  const int* s_pdst = s_pat + Pe;
  {
    const double* g = a.glob_in;
    const int x0 = 4 * Pe + Pn;
    for (int q = tid; q < Pp; q += nt) {
      float c[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};  // fF fR dF dFlo dR dRlo cR cRlo cF cFlo
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
        auto split = [](double x, float& hi, float& lo) {
          hi = (float)x;
          lo = (float)(x - (double)hi);
        };
        c[0] = (float)ff;
        c[1] = (float)fr;
        split(dF, c[2], c[3]);
        split(dR, c[4], c[5]);
        split(cRn, c[6], c[7]);
        split(cFn, c[8], c[9]);
        if (blockIdx.x == 0) {
          double* o = a.glob_out;
          o[x0 + q] = (double)c[6] + (double)c[7];
          o[x0 + Pe + q] = (double)c[8] + (double)c[9];
          o[x0 + 2 * Pe + q] = lRp;
          o[x0 + 3 * Pe + q] = lFp;
        }
      }
#pragma unroll
      for (int i = 0; i < 10; ++i) s_cst[i * Pp + q] = c[i];
    }
  }
  __syncthreads();

  // ---- the lane's columns (four) and its row; the columns' constants stay in
  // shared memory and are read once per stage
  const int gl = tid % (32 * NW), row = tid / (32 * NW);
  const bool qon = gl < nvec;
  const int qo = gl * 4;
  const unsigned act = __ballot_sync(0xffffffffu, qon);
  int qd[4], qs[4];
  float mxF[4], mxR[4];
  OnlineLse<float> lr[4], lf[4], lmu;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    qd[w] = qon && qo + w < Pe ? s_pdst[qo + w] : 0;
    qs[w] = qon && qo + w < Pe ? s_psrc[qo + w] : 0;
    mxF[w] = mxR[w] = neg_inf<float>();
    lr[w].init();
    lf[w].init();
  }
  lmu.init();
  // the pattern vertex and rows of this thread in the statistics of MU_raw
  const int pc = tid % Pn, jp0 = tid / Pn, prows = kTileThreads / Pn;
  const bool pon = tid < kTileThreads && jp0 < prows;
  const bool my_last = pon && __ldg(a.iters_p + pc) == a.t;

  const int ntiles = (Dn + V - 1) / V;
  const int bx = blockIdx.x, gx = gridDim.x;
  const int mine = bx < ntiles ? (ntiles - bx + gx - 1) / gx : 0;  // tiles of this block
  unsigned char* ring = smem + L.ring + (size_t)row * L.row_ring;
  float* s_mu = reinterpret_cast<float*>(smem + L.mu);
  auto vertex_of = [&](int k) {  // of the block's k-th tile in this row; -1: none
    if (k >= mine) return -1;
    const int v = (bx + k * gx) * V + row;
    return v < Dn ? v : -1;
  };
  auto issue = [&](int k0, int buf) {
    float* st = reinterpret_cast<float*>(ring + (size_t)buf * L.stage);
#pragma unroll
    for (int jv = 0; jv < kWv; ++jv) {
      const int v = vertex_of(k0 + jv);
      if (v < 0) continue;
      if (qon) {
        const size_t go = (size_t)v * Pp + qo;
        const int so = jv * Pp + qo;
        wcp16(st + G.oM + so, a.M + go);
        wcp16(st + G.oY + so, a.vf + go);
        wcp16(st + G.oE + so, a.dEmin + go);
        wcp16(st + G.oB + so, a.B + go);
      }
      for (int c = gl * 4; c < Pnp; c += 32 * NW * 4) {
        wcp16(st + G.oC + jv * Pnp + c, a.CV + (size_t)v * Pnp + c);
        wcp16(st + G.oCl + jv * Pnp + c, a.CVlo + (size_t)v * Pnp + c);
      }
    }
  };
  issue(0, 0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  int buf = 0;
  for (int k0 = 0; k0 < mine; k0 += kWv, buf ^= 1) {
    issue(k0 + kWv, buf ^ 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    row_sync<NW>(row);
    float* st = reinterpret_cast<float*>(ring + (size_t)buf * L.stage);
    float* mu = s_mu + (size_t)(buf * V + row) * 2 * L.mu_n;  // hi rows, then lo rows
    // ---- F over M, R over Y; -CV (and its low part) in place
    if (qon) {
      float f[4], c[4], cl[4];
      ld4(s_cst + qo, f);
      ld4(s_cst + 2 * Pp + qo, c);
      ld4(s_cst + 3 * Pp + qo, cl);
#pragma unroll
      for (int jv = 0; jv < kWv; ++jv) {
        float m[4];
        ld4(st + G.oM + jv * Pp + qo, m);
#pragma unroll
        for (int w = 0; w < 4; ++w) m[w] = fmaxf(f[w], (m[w] - c[w]) - cl[w]);  // no in-edges: M = -inf
        st4(st + G.oM + jv * Pp + qo, m);
      }
      ld4(s_cst + Pp + qo, f);
      ld4(s_cst + 4 * Pp + qo, c);
      ld4(s_cst + 5 * Pp + qo, cl);
#pragma unroll
      for (int jv = 0; jv < kWv; ++jv) {
        float y[4];
        ld4(st + G.oY + jv * Pp + qo, y);
#pragma unroll
        for (int w = 0; w < 4; ++w) y[w] = fmaxf(f[w], (y[w] - c[w]) - cl[w]);  // no out-edges: Y = -inf
        st4(st + G.oY + jv * Pp + qo, y);
      }
    }
    for (int c = gl * 4; c < kWv * Pnp; c += 32 * NW * 4) {  // (a stage without a second vertex: unused)
      float x[4];
      ld4(st + G.oC + c, x);
      st4(st + G.oC + c, {-x[0], -x[1], -x[2], -x[3]});
      ld4(st + G.oCl + c, x);
      st4(st + G.oCl + c, {-x[0], -x[1], -x[2], -x[3]});
    }
    row_sync<NW>(row);
    // ---- the compensated sums MU_raw through the lanes' schedule (acg_iter.cu)
    {
      float hi = 0.f, lo = 0.f;
      const uint4* sch = reinterpret_cast<const uint4*>(s_sched) + gl;
      for (int t4 = 0; t4 < nterms / 4; ++t4) {
        const uint4 w4 = sch[t4 * 32 * NW];
        const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
        float x[4], xl[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float* xp = st + (w[u] & 0xfffu);
          x[u] = *xp;
          xl[u] = (w[u] & kSchedStart) ? xp[G.oCl - G.oC] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool first = (w[u] & kSchedStart) != 0;
          const float h0 = first ? 0.f : hi, l0 = first ? xl[u] : lo;
          const float sm = h0 + x[u];
          const float bp = sm - h0;
          lo = l0 + ((h0 - (sm - bp)) + (x[u] - bp));
          hi = sm;
          if (w[u] & kSchedEnd) {
            const int slot = (int)((w[u] >> 16) & 0x1ffu);
            mu[slot] = hi;
            mu[L.mu_n + slot] = lo;
          }
        }
      }
    }
    row_sync<NW>(row);
    // ---- the new Y, Z and their statistics
    if (!a.last && qon) {
      float cR[4], cRl[4], cF[4], cFl[4];
      ld4(s_cst + 6 * Pp + qo, cR);
      ld4(s_cst + 7 * Pp + qo, cRl);
      ld4(s_cst + 8 * Pp + qo, cF);
      ld4(s_cst + 9 * Pp + qo, cFl);
#pragma unroll
      for (int jv = 0; jv < kWv; ++jv) {
        const int v = vertex_of(k0 + jv);
        if (v < 0) continue;
        const float* mh = mu + jv * L.mu_row;
        const float* ml = mh + L.mu_n;
        float F[4], R[4], em[4], b[4], y[4], z[4], xr[4], xf[4];
        bool some = true;
        ld4(st + G.oM + jv * Pp + qo, F);
        ld4(st + G.oY + jv * Pp + qo, R);
        ld4(st + G.oE + jv * Pp + qo, em);
        ld4(st + G.oB + jv * Pp + qo, b);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          // f = VF' - cR, r = VR' - cF: the shift comes off the compensated
          // MU_raw first, the small message after
          const float f = ((mh[qd[w]] - cR[w]) - F[w]) + (ml[qd[w]] - cRl[w]);
          const float r = ((mh[qs[w]] - cF[w]) - R[w]) + (ml[qs[w]] - cFl[w]);
          // (the padding's statistics are never written)
          mxF[w] = fmaxf(mxF[w], f);
          mxR[w] = fmaxf(mxR[w], r);
          xr[w] = f + b[w];
          xf[w] = r + b[w];
          some = some && (xr[w] > neg_inf<float>() && xf[w] > neg_inf<float>() || qo + w >= Pe);
          const bool in = qo + w < Pe;
          y[w] = in ? f - em[w] : 0.f;  // no out-edges: dEmin = +inf, Y = -inf
          z[w] = in ? r : 0.f;
        }
        // a vertex has out-edges (B above -inf) in all its columns or in none
        if (__all_sync(act, some)) {
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            lr[w].add_fast_some(xr[w]);
            lf[w].add_fast_some(xf[w]);
          }
        } else {
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            lr[w].add_fast(xr[w]);
            lf[w].add_fast(xf[w]);
          }
        }
        st4(a.vf + (size_t)v * Pp + qo, y);
        st4(a.vr_out + (size_t)v * Pp + qo, z);
      }
    }
    // ---- the statistics of MU_raw: rows of a tile in the tile form's order.
    // (The other stage's copy is rewritten only after the next barrier.)
    __syncthreads();
    if (pon) {
#pragma unroll
      for (int jv = 0; jv < kWv; ++jv) {
        if (k0 + jv >= mine) break;
        const int v0 = (bx + (k0 + jv) * gx) * V;
        for (int j = jp0; j < V && v0 + j < Dn; j += prows) {
          const float* m = s_mu + (size_t)(buf * V + j) * 2 * L.mu_n + jv * L.mu_row + pc;
          const float h = m[0], l = m[L.mu_n];
          lmu.add2(h, l);
          if (my_last) a.mu_raw[(size_t)(v0 + j) * Pn + pc] = (double)h + (double)l;
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");

  // ---- the rows' statistics, merged by wide_partials_kernel
  if (qon) {
    float* rp = a.rowpart + (size_t)(bx * V + row) * 8 * Pp + qo;
    auto put = [&](int i, float x0, float x1, float x2, float x3) { st4(rp + (size_t)i * Pp, {x0, x1, x2, x3}); };
    put(0, mxF[0], mxF[1], mxF[2], mxF[3]);
    put(1, lr[0].m, lr[1].m, lr[2].m, lr[3].m);
    put(2, lr[0].s, lr[1].s, lr[2].s, lr[3].s);
    put(3, lr[0].c, lr[1].c, lr[2].c, lr[3].c);
    put(4, mxR[0], mxR[1], mxR[2], mxR[3]);
    put(5, lf[0].m, lf[1].m, lf[2].m, lf[3].m);
    put(6, lf[0].s, lf[1].s, lf[2].s, lf[3].s);
    put(7, lf[0].c, lf[1].c, lf[2].c, lf[3].c);
  }
  if (tid < kTileThreads) {
    float* rm = a.rowpart + (size_t)gx * V * 8 * Pp + (size_t)bx * 3 * kTileThreads + tid;
    rm[0] = lmu.m;
    rm[kTileThreads] = lmu.s;
    rm[2 * kTileThreads] = lmu.c;
  }
}

// Block b's partials from its rows' statistics: mVF, mVR (max), lR, lF, S (lse),
// rows combined in order.  The merges are FP64 exponentials, 37 us of the FP64
// pipe at 120 columns; as a launch of their own they spread over all threads of a
// block, and in a batch run beside the next edge phase, which does not read them.
__global__ void __launch_bounds__(256)
wide_partials_kernel(const float* __restrict__ rowpart, int V, int Pe, int Pn, int Pp,
                     double* __restrict__ bpart) {
  const int bx = blockIdx.x, gx = gridDim.x, nmax = 2 * Pe;
  const int rows = min(kTileThreads / Pn, V);  // (threads beyond the tile's rows added nothing)
  for (int j = threadIdx.x; j < 2 * Pe + Pn; j += 256) {
    double m = -CUDART_INF, s = 0;
    if (j < 2 * Pe) {
      const int k = j >= Pe, q = j - k * Pe;
      double f = -CUDART_INF;
      const float* rp = rowpart + (size_t)bx * V * 8 * Pp + (size_t)4 * k * Pp + q;
      for (int r = 0; r < V; ++r, rp += 8 * Pp) {
        f = fmax(f, (double)rp[0]);
        lse_merge(m, s, (double)rp[Pp], (double)rp[2 * Pp] - (double)rp[3 * Pp]);
      }
      bpart[(size_t)j * gx + bx] = f;
    } else {
      const float* rm = rowpart + (size_t)gx * V * 8 * Pp + (size_t)bx * 3 * kTileThreads + (j - 2 * Pe);
      for (int r = 0; r < rows; ++r, rm += Pn)
        lse_merge(m, s, (double)rm[0], (double)rm[kTileThreads] - (double)rm[2 * kTileThreads]);
    }
    bpart[(size_t)(nmax + 2 * j) * gx + bx] = m;
    bpart[(size_t)(nmax + 2 * j + 1) * gx + bx] = s;
  }
}

int wide_warps(int pp) { return pp <= 128 ? 1 : 2; }  // of a row

template <int NW, int kThreads, int kBlocks>
acg_status launch_wide(const VertexUpdArgs<float>& a, int V, int blocks, cudaStream_t s) {
  const size_t sm = WideSmem(V, a.Pn, a.Pe, a.Pp, a.Pnp, a.vterms, NW).total;
  if (sm > 48 * 1024)
    ACG_CUDA_TRY(cudaFuncSetAttribute(vertex_wide_kernel<NW, kThreads, kBlocks>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  vertex_wide_kernel<NW, kThreads, kBlocks><<<blocks, 32 * NW * V, sm, s>>>(a);
  ACG_LAUNCH_CHECK();
  return ACG_OK;
}

}  // namespace

// Few pattern vertices share many edges: their long sums are a few lanes' of each
// row, and a large graph has the tiles over which the tile form spreads them.  Ten
// iterations, tile form / this one: 33,000 vertices, 8 and 132, 8 and 256: 2.40 / 2.55,
// 2.79 / 2.90 ms (20,000: 1.94 / 1.94, 2.06 / 2.20); 200,000, 16 and 132, 20 and 144:
// 7.98 / 8.98, 8.24 / 8.53 (33,000: 2.45 / 2.45, 2.47 / 2.36); rows of one warp, 2 and
// 100, 4 and 100: 200,000 6.08 / 7.80, 5.97 / 6.60, 33,000 2.22 / 2.13, 2.18 / 1.96.
static bool few_vertices(int pn, int pp, int dn) {
  if (wide_warps(pp) == 1) return pn <= 2 && dn >= 1 << 16;
  return (pn <= 8 && dn >= 1 << 15) || (pn <= 16 && kTileThreads / (pp / 4) >= 6 && dn >= 1 << 16);
}

int vertex_wide_schedule(const int* pat, int pn, int pe, int pp, int pnp, int dn, std::vector<uint32_t>* out) {
  out->clear();
  if (few_vertices(pn, pp, dn)) return 0;
  const int nt = vertex_warp_schedule(pat, pn, pe, pp, pnp, kWv, out, 32 * wide_warps(pp), 4);
  if (wide_warps(pp) == 1 || nt <= kWideTerms) return nt;
  out->clear();
  return 0;
}

size_t wide_rowpart_floats(int pp, int blocks) {
  return pp <= 64 ? 0 : (size_t)blocks * ((size_t)kTileThreads / (pp / 4) * 8 * pp + 3 * kTileThreads);
}

acg_status launch_wide_partials(const VertexUpdArgs<float>& a, int blocks, cudaStream_t s) {
  wide_partials_kernel<<<blocks, 256, 0, s>>>(a.rowpart, kTileThreads / (a.Pp / 4), a.Pe, a.Pn, a.Pp, a.bpart);
  ACG_LAUNCH_CHECK();
  return ACG_OK;
}

acg_status launch_vertex_wide(const VertexUpdArgs<float>& a, int blocks, cudaStream_t s) {
  if (a.vsched == nullptr || a.Pp <= 64 || a.Pp > 256)
    return set_error(ACG_ERR_INVALID_ARGUMENT, "vertex phase: %d columns, %d schedule terms", a.Pp, a.vterms);
  const int V = kTileThreads / (a.Pp / 4);  // 8 to 15 rows of one warp, 4 to 7 of two
  if (wide_warps(a.Pp) == 1)
    return V <= 8 ? launch_wide<1, 256, 2>(a, V, blocks, s) : launch_wide<1, 480, 1>(a, V, blocks, s);
  return V <= 4   ? launch_wide<2, 256, 2>(a, V, blocks, s)
         : V <= 5 ? launch_wide<2, 320, 2>(a, V, blocks, s)
         : V <= 6 ? launch_wide<2, 384, 2>(a, V, blocks, s)
                  : launch_wide<2, 448, 1>(a, V, blocks, s);
}

}  // namespace acg
