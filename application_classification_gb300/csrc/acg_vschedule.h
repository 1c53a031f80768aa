// acg_vschedule.h -- the vertex phase's per-lane schedule of its compensated
// MU_raw sums (warp form of vertex_warp_kernel, acg_iter.cu), host code that
// nvcc and the host compiler both build (the CPU tests compile it directly).
//
// A warp stages kVps data vertices at a time.  Each (staged vertex jv, pattern
// vertex p) sum is one job: the terms -CV[jv][p], then F[jv][q] for the in-edges
// q of p (dst_q = p) ascending, then R[jv][q] for its out-edges (src_q = p)
// ascending -- the order of the tile form.  The jobs go to the 32 lanes longest
// first, each to the least loaded lane, so a lane runs ~1/32 of the stage's terms
// instead of the largest pattern degree for every vertex.  Every sum keeps its
// terms and their order, so the result does not depend on the spread.  Within a
// lane the jobs' order is free, and chosen for the shared memory's banks.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define ACG_VS_HD __host__ __device__
#else
#define ACG_VS_HD
#endif

namespace acg {

// schedule word: element offset of the term in the stage (bits 0-11), first
// term of its job (bit 12), last term (bit 13), the job's slot
// jv * row + p (row: Pn rounded up to 32, plus 1) in the per-warp MU_raw rows (bits 16-24); stored
// [t / 4][lane][t % 4] so that a lane's four next words are one 16-byte load
constexpr uint32_t kSchedStart = 1u << 12, kSchedEnd = 1u << 13;

// Element offsets of one stage of vps vertices: M, Y, dEmin, B rows [vps][Pp],
// then the CV rows [vps][Pnp] and (FP32) their low parts.
struct VwStage {
  int oM, oY, oE, oB, oC, oCl, n;
  ACG_VS_HD VwStage(int Pp, int Pnp, bool lo, int vps) {
    oM = 0;
    oY = vps * Pp;
    oE = 2 * vps * Pp;
    oB = 3 * vps * Pp;
    oC = 4 * vps * Pp;
    oCl = oC + vps * Pnp;
    n = oCl + (lo ? vps * Pnp : 0);
  }
};

// The schedule for a pattern whose incidence arrays (build_incidence's layout:
// psrc[pe], pdst[pe], in_off[pn + 1], in_q[pe], out_off[pn + 1], out_q[pe])
// are at pat, for stages of vps vertices.  Returns the terms per lane (a
// multiple of 4) and fills out[terms * nlanes] for nlanes lanes (32, or the
// lanes of a group of warps) and stage elements of elem bytes; 0 when the pattern has more than per_lane
// vertices or padded edge columns per lane, or the stage is too large for the word's
// fields.
inline int vertex_warp_schedule(const int* pat, int pn, int pe, int pp, int pnp, int vps,
                                std::vector<uint32_t>* out, int nlanes = 32, int per_lane = 2,
                                int elem = 4) {
  out->clear();
  if (pn <= 0 || pn > per_lane * nlanes || pp > per_lane * nlanes || vps <= 0) return 0;
  const int row = (pn + 31) / 32 * 32 + 1;  // a vertex's MU_raw row
  const VwStage G(pp, pnp, false, vps);  // offsets of M, Y, CV (the same for FP32 and FP64)
  // every offset and slot must fit its field of the word
  if (G.oC + vps * pnp > 0x1000 || vps * row > 0x200) return 0;
  const int* inoff = pat + 2 * pe;
  const int* inq = inoff + pn + 1;
  const int* outoff = inq + pe;
  const int* outq = outoff + pn + 1;
  // jobs (jv, p), longest first (ties: jv, then p), each to the least loaded
  // lane (ties: the lowest)
  struct Job {
    int jv, p, len;
  };
  std::vector<Job> jobs;
  for (int jv = 0; jv < vps; ++jv)
    for (int p = 0; p < pn; ++p)
      jobs.push_back({jv, p, 1 + inoff[p + 1] - inoff[p] + outoff[p + 1] - outoff[p]});
  std::stable_sort(jobs.begin(), jobs.end(), [](const Job& x, const Job& y) { return x.len > y.len; });
  std::vector<std::vector<Job>> lanes(nlanes);
  std::vector<int> load(nlanes, 0);
  for (const Job& j : jobs) {
    const int best = (int)(std::min_element(load.begin(), load.end()) - load.begin());
    lanes[best].push_back(j);
    load[best] += j.len;
  }
  const int nt = (*std::max_element(load.begin(), load.end()) + 3) / 4 * 4;
  auto term = [&](const Job& j, int i) {
    const int ni = inoff[j.p + 1] - inoff[j.p];
    if (i == 0) return (uint32_t)(G.oC + j.jv * pnp + j.p);                         // -CV
    if (i <= ni) return (uint32_t)(G.oM + j.jv * pp + inq[inoff[j.p] + i - 1]);     // F[q], dst_q = p
    return (uint32_t)(G.oY + j.jv * pp + outq[outoff[j.p] + i - 1 - ni]);           // R[q], src_q = p
  };
  // A lane's jobs in the order that meets the fewest bank conflicts with the lanes
  // before it, jobs of the next lane of the same length taken in exchange: a load
  // of 32 lanes (of 8-byte elements 16, on 16 banks of two words) takes as many
  // passes as its busiest bank has words, hits[t][group][bank] so far.  Passes per
  // load of random patterns of 16/32, 32/64 and 40/120: 4.2, 4.5 and 2.9 in the
  // order of assignment (a pattern vertex's jobs for the staged vertices side by
  // side, on the same banks), 3.2, 2.5 and 2.5 so.
  const int gl = 128 / elem, groups = (nlanes + gl - 1) / gl;
  std::vector<uint8_t> hits((size_t)nt * groups * gl, 0), most((size_t)nt * groups, 0);
  // padding terms (word 0) come after a lane's last job and change nothing it stores
  out->assign((size_t)nt * nlanes, 0u);
  for (int l = 0; l < nlanes; ++l) {
    std::vector<Job>& L = lanes[l];
    int t0 = 0;
    for (size_t k = 0; k < L.size(); ++k) {
      size_t best = k;
      Job* other = nullptr;
      int cost = -1;
      auto price = [&](const Job& j) {
        int x = 0;
        for (int i = 0; i < j.len; ++i) {
          const size_t tg = (size_t)(t0 + i) * groups + l / gl;
          const int h = hits[tg * gl + term(j, i) % gl];
          x += h == most[tg] ? 16 + h : h;
        }
        return x * 64 / j.len;
      };
      for (size_t c = k; c < L.size(); ++c) {
        const int x = price(L[c]);
        if (cost < 0 || x < cost) {
          best = c;
          cost = x;
          other = nullptr;
        }
        if (l + 1 == nlanes) continue;
        for (Job& j : lanes[l + 1]) {
          if (j.len != L[c].len) continue;
          const int y = price(j);
          if (y < cost) {
            best = c;
            cost = y;
            other = &j;
          }
        }
      }
      if (other) std::swap(L[best], *other);
      std::swap(L[k], L[best]);
      const Job& j = L[k];
      const uint32_t slot = (uint32_t)(j.jv * row + j.p) << 16;
      for (int i = 0; i < j.len; ++i) {
        const int t = t0 + i;
        const uint32_t w = term(j, i);
        const size_t tg = (size_t)t * groups + l / gl;
        const uint8_t h = ++hits[tg * gl + w % gl];
        most[tg] = std::max(most[tg], h);
        (*out)[(size_t)(t / 4) * 4 * nlanes + l * 4 + t % 4] =
            w | slot | (i == 0 ? kSchedStart : 0u) | (i == j.len - 1 ? kSchedEnd : 0u);
      }
      t0 += j.len;
    }
  }
  return nt;
}

// ---- shared memory of the kernels that share a stage between warps
constexpr size_t kBlockSmem = 227 * 1024;  // sm_103a, dynamic
ACG_VS_HD inline size_t vs16(size_t b) { return (b + 15) & ~size_t(15); }

// vertex_fx_kernel (acg_vertex_fx.cu): groups of nw warps share a stage.
constexpr int kFxVps = 2;           // vertices per stage
constexpr int kFxWarps = 8;         // of a block
constexpr int kFxTableBytes = 8192; // 2^(j / 1024)
// A lane's terms are as many as its longest job's, 1 + twice the pattern's edges for
// a vertex that all of them leave and enter: of such hubs the schedule of a group of
// four warps is up to 264 KB.  Where it does not fit a block's memory beside the rest
// it stays in global memory (in_global).
struct FxSmem {
  size_t pat, sched, tab, cst, mxd, amp, flags, ring, mu, total, stage, group_ring, mu_n;
  int mu_row;
  ACG_VS_HD FxSmem(int Pn, int Pe, int Pp, int Pnp, int nterms, int nw, bool in_global) {
    const int ng = kFxWarps / nw;  // groups
    size_t o = 0;
    pat = o; o += vs16(sizeof(int) * (size_t)(4 * Pe + 2 * (Pn + 1)));
    sched = o; o += in_global ? 0 : vs16(sizeof(uint32_t) * (size_t)nterms * 32 * nw);
    tab = o; o += kFxTableBytes;
    cst = o; o += vs16(sizeof(double) * (size_t)6 * Pp);   // fF fR dF dR cF cR
    mxd = o; o += vs16(sizeof(double) * (size_t)2 * Pp * ng);  // maxima of FP64 stages
    amp = o; o += vs16(sizeof(float) * (size_t)2 * Pp);    // |F|, |R| bounds
    flags = o; o += 16;
    stage = sizeof(double) * (size_t)VwStage(Pp, Pnp, false, kFxVps).n;
    group_ring = 2 * stage;
    const size_t red = sizeof(uint32_t) * (size_t)ng * (4 * Pe + 4 * (2 * Pe + Pn));  // aliases the rings
    ring = o; o += vs16(red > ng * group_ring ? red : ng * group_ring);
    mu_row = (Pn + 31) / 32 * 32 + 1;
    mu_n = (size_t)kFxVps * mu_row;
    mu = o; o += vs16(sizeof(double) * ng * mu_n);
    total = o;
  }
};

// vertex_wide_kernel (acg_vertex_wide.cu): V rows of nw warps; schedules of more
// than kWideTerms terms a lane are not made.
constexpr int kWv = 2;  // vertices (tiles) per stage
struct WideSmem {
  size_t pat, sched, cst, ring, mu, total, stage, row_ring, mu_n;
  int mu_row;
  ACG_VS_HD WideSmem(int V, int Pn, int Pe, int Pp, int Pnp, int nterms, int nw) {
    size_t o = 0;
    pat = o; o += vs16(sizeof(int) * (size_t)(2 * Pe));
    sched = o; o += vs16(sizeof(uint32_t) * (size_t)nterms * 32 * nw);
    cst = o; o += vs16(sizeof(float) * (size_t)10 * Pp);
    stage = sizeof(float) * (size_t)VwStage(Pp, Pnp, true, kWv).n;
    row_ring = 2 * stage;
    ring = o; o += vs16(V * row_ring);
    mu_row = (Pn + 31) / 32 * 32 + 1;  // (the schedule's slots)
    mu_n = (size_t)kWv * mu_row;
    mu = o; o += vs16(sizeof(float) * 2 * 2 * V * mu_n);  // two stages: hi, lo of each row
    total = o;
  }
};

}  // namespace acg
