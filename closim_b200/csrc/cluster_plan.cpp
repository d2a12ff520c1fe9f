// Builds the per-CTA element lists of the one-cluster PCG (cluster_plan.hpp)
// from the membrane and hinge incidence CSRs.
#include "cluster_plan.hpp"

#include <algorithm>

#include "setup.hpp"

namespace cs {

namespace {

// A set of ids below `n` that empties itself in ascending order: marking is one
// bit, and a CTA's ids lie close together, so the scan is short.
struct IdSet {
  std::vector<uint64_t> words;
  size_t lo, hi;
  explicit IdSet(int n) : words((size_t)n / 64 + 1, 0), lo(words.size()), hi(0) {}
  void add(int id) {
    const size_t w = (size_t)id >> 6;
    words[w] |= 1ull << (id & 63);
    lo = std::min(lo, w);
    hi = std::max(hi, w + 1);
  }
  void drain(std::vector<int>& out) {
    out.clear();
    for (size_t w = lo; w < hi; w++) {
      for (uint64_t b = words[w]; b; b &= b - 1) out.push_back((int)(w * 64 + (size_t)__builtin_ctzll(b)));
      words[w] = 0;
    }
    lo = words.size();
    hi = 0;
  }
};

int range_begin(int n, int nrank, int r) { return (int)((int64_t)r * n / nrank); }

}  // namespace

size_t cluster_plan_least_smem(const HostMesh& me, int nrank, bool hinges) {
  size_t least = 0;
  for (int r = 0; r < nrank; r++) {
    const int v0 = range_begin(me.n, nrank, r), v1 = range_begin(me.n, nrank, r + 1);
    const int ti = (int)(me.memOff[v1] - me.memOff[v0]), hi = hinges ? (int)(me.hinOff[v1] - me.hinOff[v0]) : 0;
    least = std::max(least, (size_t)cl_smem_layout(v1 - v0, ti / 3, hi / 4, ti + hi, v1 - v0, 0, hinges).total);
  }
  return least;
}

void build_cluster_plan(const HostMesh& me, int nrank, int warpsPerCta, ClusterPlanHost& p, bool domains,
                        bool hinges) {
  p = ClusterPlanHost{};
  p.nrank = nrank;
  p.warpsPerCta = warpsPerCta;
  p.nwarps = nrank * warpsPerCta;
  p.ok = nrank > 0 && warpsPerCta > 0 && (!domains || me.D <= 3 * p.nwarps);
  if (!p.ok) return;
  const int n = me.n;
  // phase B: domain slots per CTA and where each vertex's dofs live
  p.vDst.assign(n, -1);
  p.nSlots.assign(nrank, 0);
  for (int dom = 0; domains && dom < me.D; dom++) {
    const int gw = dom % p.nwarps, u = dom / p.nwarps, r = gw / warpsPerCta, slot = u * warpsPerCta + gw % warpsPerCta;
    p.nSlots[r] = std::max(p.nSlots[r], slot + 1);
    for (int l = 0; l < me.domStart[dom + 1] - me.domStart[dom]; l++) {
      const int v = me.domVerts[me.domStart[dom] + l];
      if (l >= 8 || v < 0 || v >= n || p.vDst[v] != -1) { p.ok = false; return; }
      p.vDst[v] = (r << 24) | (slot * 24 + l * 3);
    }
  }
  for (int v = 0; domains && v < n; v++)
    if (p.vDst[v] < 0) { p.ok = false; return; }
  p.vb.resize(nrank + 1);
  for (int r = 0; r <= nrank; r++) p.vb[r] = range_begin(n, nrank, r);
  p.haloOff.assign(1, 0);
  p.triOff.assign(1, 0);
  p.hinOff.assign(1, 0);
  p.incOff.assign(n + 1, 0);
  p.incHin.assign(n, 0);
  p.ownHalo.assign(n, 0);
  p.inc.resize(me.memRec.size() + (hinges ? me.hinRec.size() : 0));
  int nextInc = 0;
  std::vector<int> loc(n, -1), tslot(me.m, -1), hslot(me.hg, -1);
  std::vector<int> tris, hins, halo;
  IdSet triSet(me.m), hinSet(me.hg), haloSet(n);
  for (int r = 0; r < nrank; r++) {
    const int v0 = p.vb[r], v1 = p.vb[r + 1];
    for (int v = v0; v < v1; v++) haloSet.add(v);
    for (uint32_t q = me.memOff[v0]; q < me.memOff[v1]; q++) triSet.add((int)(me.memRec[q] >> 2));
    if (hinges)
      for (uint32_t q = me.hinOff[v0]; q < me.hinOff[v1]; q++) hinSet.add((int)(me.hinRec[q] >> 2));
    triSet.drain(tris);
    hinSet.drain(hins);
    for (int t : tris)
      for (int c = 0; c < 3; c++) haloSet.add((int)me.idx[3 * (size_t)t + c]);
    for (int h : hins)
      for (int c = 0; c < 4; c++) haloSet.add(me.hinge[4 * (size_t)h + c]);
    haloSet.drain(halo);
    if (halo.size() > 65535) p.ok = false;
    for (size_t i = 0; i < halo.size(); i++) loc[halo[i]] = (int)i;
    p.triLoc.resize(p.triLoc.size() + 4 * tris.size(), 0);
    uint16_t* tl = p.triLoc.data() + p.triLoc.size() - 4 * tris.size();
    for (size_t s = 0; s < tris.size(); s++, tl += 4) {
      const int t = tris[s];
      tslot[t] = (int)s;
      for (int c = 0; c < 3; c++) tl[c] = (uint16_t)loc[me.idx[3 * (size_t)t + c]];
    }
    p.hinLoc.resize(p.hinLoc.size() + 4 * hins.size());
    uint16_t* hl = p.hinLoc.data() + p.hinLoc.size() - 4 * hins.size();
    for (size_t s = 0; s < hins.size(); s++, hl += 4) {
      const int h = hins[s];
      hslot[h] = (int)s;
      for (int c = 0; c < 4; c++) hl[c] = (uint16_t)loc[me.hinge[4 * (size_t)h + c]];
    }
    const int inc0 = nextInc;
    for (int v = v0; v < v1; v++) {
      p.incOff[v] = nextInc;
      for (uint32_t q = me.memOff[v]; q < me.memOff[v + 1]; q++) {
        const uint32_t rec = me.memRec[q];
        p.inc[nextInc++] = ((uint32_t)tslot[rec >> 2] << 2) | (rec & 3);
      }
      p.incHin[v] = nextInc;
      for (uint32_t q = me.hinOff[v]; hinges && q < me.hinOff[v + 1]; q++) {
        const uint32_t rec = me.hinRec[q];
        p.inc[nextInc++] = ((uint32_t)hslot[rec >> 2] << 2) | (rec & 3);
      }
      p.ownHalo[v] = loc[v];
    }
    const int nInc = nextInc - inc0, nOwn = v1 - v0;
    p.triId.insert(p.triId.end(), tris.begin(), tris.end());
    p.hinId.insert(p.hinId.end(), hins.begin(), hins.end());
    p.halo.insert(p.halo.end(), halo.begin(), halo.end());
    p.triOff.push_back((int)p.triId.size());
    p.hinOff.push_back((int)p.hinId.size());
    p.haloOff.push_back((int)p.halo.size());
    const int nh = (int)halo.size(), nt = (int)tris.size(), ng = (int)hins.size();
    const int ns = p.nSlots[r];
    p.smemNoHinge = std::max(p.smemNoHinge, (size_t)cl_smem_layout(nh, nt, ng, nInc, nOwn, ns, false).total);
    p.smemHinge = std::max(p.smemHinge, (size_t)cl_smem_layout(nh, nt, ng, nInc, nOwn, ns, true).total);
  }
  p.incOff[n] = nextInc;
}

}  // namespace cs
