// Host-side work plans of the persistent time-loop sweeps (persist.cuh): which CTA
// takes which (row group, j range) segments, and for the cluster form which CTA
// finalises each row group shared by several CTAs of a cluster.  Plain C++ (no device
// code), built once per context.
#pragma once

#include <algorithm>
#include <vector>

#include "layout.h"

namespace lddmm {

constexpr int kPlanSub = 32;          // j entries per staged sub-tile (kSub)
constexpr int kPlanMaxJobParts = 8;   // parts of a row group in the cluster form (kMaxJobParts)

// Work plan of the persistent sweeps: the units' (64-row tiles') j ranges laid end to end
// and dealt to at most G CTAs, each up to the same cost, a segment costing its entries plus
// kSegCost (a CTA's combine and finalise, in entries of pair time: with 64 instead of 256 a
// step of 4000 points took 15.2 / 23.0 us shooting / adjoint instead of 14.6 / 22.2); the
// smallest such cost is found by bisection.  Cuts fall on multiples of 16 entries and leave
// at least kMinSeg.  A CTA takes no less than a tenth of the longest range: a tile's parts are
// read ten at a time.  With sms given, G being twice that, one CTA per SM is preferred where
// its shares are under 0.8 of what two CTAs of an SM take together: two hide each other's
// latency, but a few SMs with two would be waited for (1200 points: 152 CTAs took 5.5 / 7.4 us
// per step, 133 take 5.1 / 6.5).
struct HostPlan {
  std::vector<int4> segs;       // (unit, j begin, j end, part) in CTA order
  std::vector<int> cta_seg;     // G + 1 offsets into segs
  std::vector<int2> unit_parts; // (parts, first partial slot)
  int slots = 0;
};

constexpr int kSegCost = 256;
constexpr int kMinSeg = 32;

inline HostPlan plan_sweeps(const std::vector<int2> &units, const std::vector<PairDesc> &hpd,
                            int G, int sms = 0) {
  const int nu = (int)units.size();
  HostPlan h;
  auto deal = [&](long long cap, bool emit) {
    int ctas = 1;
    long long left = cap;
    for (int u = 0; u < nu; ++u) {
      const int J = hpd[units[u].x].Npad;
      int part = 0;
      for (int x = 0; x < J;) {
        int n = (int)std::min<long long>(J - x, std::max(left - kSegCost, 0LL) / 16 * 16);
        if (n < J - x && J - x - n < kMinSeg) n = J - x - kMinSeg;
        if (n < std::min(kMinSeg, J - x)) {  // no room here: the next CTA
          ++ctas;
          left = cap;
          if (emit) h.cta_seg.push_back((int)h.segs.size());
          continue;
        }
        if (emit) h.segs.push_back(make_int4(u, x, x + n, part));
        ++part;
        left -= n + kSegCost;
        x += n;
      }
      if (emit) {
        h.unit_parts.push_back(make_int2(part, h.slots));
        if (part > 1) h.slots += part;
      }
    }
    return ctas;
  };
  long long lo = 2 * kMinSeg, hi = kSegCost;
  for (int u = 0; u < nu; ++u) {
    const int J = hpd[units[u].x].Npad;
    lo = std::max(lo, (J + 159LL) / 160 * 16);
    hi += J + kSegCost;
  }
  lo += kSegCost;
  auto smallest = [&](int ctas) {
    long long l = lo, r = std::max(hi, lo);
    while (l < r) {
      const long long mid = (l + r) / 2;
      if (deal(mid, false) <= ctas) r = mid;
      else l = mid + 1;
    }
    return l;
  };
  long long cap = smallest(std::max(G, 1));
  if (sms > 0 && deal(cap, false) > sms) {
    const long long one = smallest(sms);
    if (one - kSegCost < 0.8 * 2 * (cap - kSegCost)) cap = one;
  }
  h.cta_seg.push_back(0);
  deal(cap, true);
  h.cta_seg.push_back((int)h.segs.size());
  return h;
}

constexpr long long kMinPart = 32;  // shortest part of a cut row group (cluster form)

// Work plan of the cluster-form persistent sweeps: the row groups split into ncl
// contiguous ranges of whole row groups, one per cluster, minimising the largest
// range's work (binary search on the bound, greedy fill); each cluster's entries cut
// into C equal CTA shares.  Only a CTA's first and last segment can be part
// of a row group shared with other CTAs (slots 0 and 1); the CTA holding a shared row
// group's first part finalises it (at most one per CTA: only a CTA's last segment can
// be a first part).  CTA k * C + r is rank r of cluster k.  max_share: the largest CTA
// share in entries.
struct ClusterHostPlan {
  std::vector<int4> segs;       // (unit, j begin, j end, kind: 0 whole, 1 / 2 slot 0 / 1)
  std::vector<int> cta_seg;     // ncl * C + 1 offsets into segs
  std::vector<int2> job;        // per CTA: (unit, parts) or (-1, 0)
  std::vector<int> job_src;     // per CTA x kPlanMaxJobParts: rank << 1 | slot
  long long max_share = 0;
  bool ok = false;
};

inline ClusterHostPlan plan_cluster_sweeps(const std::vector<int2> &units,
                                           const std::vector<PairDesc> &hpd, int C, int ncl) {
  ClusterHostPlan h;
  const int nu = (int)units.size();
  if (nu == 0 || C < 1 || C > kPlanMaxJobParts || ncl < 1) return h;
  std::vector<long long> w(nu);
  long long tot = 0, wmax = 0;
  for (int u = 0; u < nu; ++u) {
    w[u] = hpd[units[u].x].Npad;
    tot += w[u];
    wmax = std::max(wmax, w[u]);
  }
  auto ranges = [&](long long cap) {
    int g = 1;
    long long acc = 0;
    for (int u = 0; u < nu; ++u) {
      if (acc + w[u] > cap) {
        ++g;
        acc = 0;
      }
      acc += w[u];
    }
    return g;
  };
  long long lo = wmax, hi = tot;
  while (lo < hi) {
    const long long mid = (lo + hi) / 2;
    if (ranges(mid) <= ncl) hi = mid;
    else lo = mid + 1;
  }
  std::vector<int> ub(1, 0);  // unit range of each cluster
  {
    long long acc = 0;
    for (int u = 0; u < nu; ++u) {
      if (acc + w[u] > lo) {
        ub.push_back(u);
        acc = 0;
      }
      acc += w[u];
    }
    while ((int)ub.size() < ncl + 1) ub.push_back(nu);
  }
  const int G = ncl * C;
  h.cta_seg.assign(G + 1, 0);
  h.job.assign(G, make_int2(-1, 0));
  h.job_src.assign((size_t)G * kPlanMaxJobParts, 0);
  for (int k = 0; k < ncl; ++k) {
    const int u0 = ub[k], u1 = ub[k + 1];
    std::vector<long long> us(1, 0);
    for (int u = u0; u < u1; ++u) us.push_back(us.back() + w[u]);
    const long long L = us.back();
    std::vector<long long> b(C + 1, 0);
    b[C] = L;
    for (int r = 1; r < C; ++r) {
      const long long x = L * r / C;
      int v = (int)(std::upper_bound(us.begin(), us.end(), x) - us.begin()) - 1;
      v = std::min(std::max(v, 0), std::max(u1 - u0 - 1, 0));
      long long off = 0;
      if (u1 > u0) {
        const long long J = us[v + 1] - us[v];
        off = (x - us[v] + kPlanSub / 2) / kPlanSub * kPlanSub;
        if (off < kMinPart) off = 0;
        else if (J - off < kMinPart) off = J;
      }
      b[r] = std::max(b[r - 1], std::min(us[v] + off, L));
    }
    std::vector<std::vector<int2>> parts(u1 - u0);  // (rank, slot) per shared row group
    for (int r = 0; r < C; ++r) {
      const int cta = k * C + r;
      h.cta_seg[cta] = (int)h.segs.size();
      h.max_share = std::max(h.max_share, b[r + 1] - b[r]);
      const int first = (int)h.segs.size();
      for (int v = 0; v < u1 - u0; ++v) {
        const long long lo2 = std::max(b[r], us[v]) - us[v];
        const long long hi2 = std::min(b[r + 1], us[v + 1]) - us[v];
        if (hi2 > lo2) h.segs.push_back(make_int4(u0 + v, (int)lo2, (int)hi2, 0));
      }
      const int last = (int)h.segs.size() - 1;
      for (int q = first; q <= last; ++q) {
        int4 &sg = h.segs[q];
        if (sg.y == 0 && sg.z == (int)w[sg.x]) continue;  // a whole row group
        if (q != first && q != last) return h;  // cannot happen: middle segments are whole
        const int slot = (q == first) ? 0 : 1;
        sg.w = 1 + slot;
        parts[sg.x - u0].push_back(make_int2(r, slot));
      }
    }
    for (int v = 0; v < u1 - u0; ++v) {
      const std::vector<int2> &pv = parts[v];
      if (pv.empty()) continue;
      if ((int)pv.size() > kPlanMaxJobParts) return h;
      const int cta = k * C + pv[0].x;
      if (h.job[cta].x >= 0) return h;  // one job per CTA
      h.job[cta] = make_int2(u0 + v, (int)pv.size());
      for (size_t q = 0; q < pv.size(); ++q)
        h.job_src[(size_t)cta * kPlanMaxJobParts + q] = (pv[q].x << 1) | pv[q].y;
    }
  }
  h.cta_seg[G] = (int)h.segs.size();
  h.ok = true;
  return h;
}

}  // namespace lddmm
