// Per-candidate and per-seed steps of one clone-engine layer iteration.
// Each function restates the cited reference routine for one candidate
// (one CUDA thread) or one seed (8 lanes); the plain form calls them from
// separate kernels, the batched persistent form from one kernel.
#pragma once

#include "find_dev.cuh"

namespace mkfg {

// Layer of region `reg` at layer-plan step `step` (>= 1), or -1.
__device__ __forceinline__ int plan_layer(const FindConfigDev& C, int reg, int step) {
  const int idx = C.pickup[reg] + step;
  return idx < C.plan_len[reg] ? C.plan[reg][idx] : -1;
}

__device__ __forceinline__ void load_state(const CandSoA& B, int slot, float (&par)[6],
                                           float (&err)[21]) {
#pragma unroll
  for (int e = 0; e < 6; ++e) par[e] = B.par[e * B.cap + slot];
#pragma unroll
  for (int e = 0; e < 21; ++e) err[e] = B.err[e * B.cap + slot];
}

__device__ __forceinline__ void store_state(const CandSoA& B, int slot, const float (&par)[6],
                                            const float (&err)[21]) {
#pragma unroll
  for (int e = 0; e < 6; ++e) B.par[e * B.cap + slot] = par[e];
#pragma unroll
  for (int e = 0; e < 21; ++e) B.err[e * B.cap + slot] = err[e];
}

// Appends a hit-on-track node to seed s's arena (CombCandidate::AddHit).
__device__ __forceinline__ int arena_append(const EventDev& E, int s, int index, int layer,
                                            float chi2, int prev) {
  const int pos = atomicAdd(&E.hot_size[s], 1);
  if (pos >= E.hot_cap) {
    atomicOr(E.err_flags, kErrArena);
    return prev;
  }
  const size_t k = (size_t)s * E.hot_cap + pos;
  E.node_hot[k] = hot_pack(index, layer);
  E.node_chi2[k] = chi2;
  E.node_prev[k] = prev;
  return pos;
}

__device__ __forceinline__ int node_hot_of(const EventDev& E, int s, int node) {
  return E.node_hot[(size_t)s * E.hot_cap + node];
}

// Dynamic hit-selection windows (MkFinder::getHitSelDynamicWindows,
// mkFit/MkFinder.cc:166-195).
__device__ __forceinline__ void dynamic_windows(const LayerDev& L, float invpt, float theta,
                                                float& min_dq, float& max_dq, float& min_dphi,
                                                float& max_dphi) {
  float max_invpt = invpt;
  if (invpt > 10.0) max_invpt = 10.0f;
  const float this_dq = fmaf(L.c_dq_1, theta, L.c_dq_0 * max_invpt) + L.c_dq_2;
  if (L.c_dq_sf * this_dq > 0.f) {
    min_dq = L.c_dq_sf * this_dq;
    max_dq = 2.0f * min_dq;
  }
  const float this_dphi = fmaf(L.c_dp_1, theta, L.c_dp_0 * max_invpt) + L.c_dp_2;
  if (L.c_dp_sf * this_dphi > min_dphi) {
    min_dphi = L.c_dp_sf * this_dphi;
    max_dphi = 2.0f * min_dphi;
  }
}

// Dynamic chi2 cut (MkFinder::getHitSelDynamicChi2Cut, :203-220).
__device__ __forceinline__ float dynamic_chi2_cut(const LayerDev& L, float chi2_min,
                                                  const float (&par)[6]) {
  const float invpt = par[3];
  const float theta = fabsf(par[5] - kPIOver2);
  float max_invpt = invpt;
  if (invpt > 10.0) max_invpt = 10.0f;
  const float this_c2 = fmaf(L.c_c2_1, theta, L.c_c2_0 * max_invpt) + L.c_c2_2;
  if (L.c_c2_sf * this_c2 > chi2_min) return L.c_c2_sf * this_c2;
  return chi2_min;
}

__device__ __forceinline__ int q_bin_checked(const LayerDev& L, float q) {
  const int b = (int)((q - L.qmin) * L.fq);
  return min(max(b, 0), L.nq - 1);
}

__device__ __forceinline__ int phi_bin(float phi) {
  constexpr float fphi_fine = 1024 / kTwoPI;
  return ((int)floorf(fphi_fine * (phi + kPI))) >> 2;
}

__device__ __forceinline__ float cdist(float a) { return a > kPI ? kTwoPI - a : a; }

// SelectHitIndices for one candidate (mkFit/MkFinder.cc:227-684) including
// the sensitive-region test (TrackerInfo.h:118-138). `bins` is the layer's
// (q bin, phi bin) table of the candidate's event. Writes up to 16 hit
// indices (index within layer) in bin-scan order; returns XHitSize (-1 when
// outside the layer) and the WSR code. kGenericBins: `bins` may point to
// shared memory (a staged copy of the table), so it is read with generic
// loads rather than through the read-only data path.
template <bool kGenericBins = false>
__device__ __forceinline__ int select_hits(const EventDev& E, const LayerDev& L,
                                           const uint32_t* __restrict__ bins, int hit_base,
                                           const float (&par)[6],
                                           const float (&err)[21], int* xhit, int xstride,
                                           int& wsr) {
  float min_dq = L.min_dq, max_dq = L.max_dq, min_dphi = L.min_dphi, max_dphi = L.max_dphi;
  const float invpt = par[3];
  const float theta = fabsf(par[5] - kPIOver2);
  dynamic_windows(L, invpt, theta, min_dq, max_dq, min_dphi, max_dphi);

  const float x = par[0], y = par[1];
  const float r2 = x * x + y * y;
  const float dphidx = -y / r2, dphidy = x / r2;
  const float dphi2 = fmaf(2 * dphidx * dphidy, err[1],
                           fmaf(dphidx * dphidx, err[0], dphidy * dphidy * err[2]));
  const float phi = f_atan2(y, x);
  float dphi = fmaxf(3.f * sqrtf(fabsf(dphi2)), min_dphi);
  float q, dq;
  if (L.is_barrel) {
    const float z = par[2];
    dq = fabsf(3.f * sqrtf(err[5]));
    const float edgeCorr = fabsf(0.5f * (L.rout - L.rin) / f_tan(par[5]));
    const float d = sqrtf(fmaf(dq, dq, edgeCorr * edgeCorr));
    if (z > L.zmax + d || z < L.zmin - d)
      wsr = kWsrOutside;
    else if (z < L.zmax - d && z > L.zmin + d)
      wsr = kWsrInside;
    else
      wsr = kWsrEdge;
    q = z;
  } else {
    const float r = sqrtf(r2);
    dq = 3.f * sqrtf(fabsf(fmaf(2 * x * y, err[1], fmaf(x * x, err[0], y * y * err[2]))) / r2);
    const float edgeCorr = fabsf(0.5f * (L.zmax - L.zmin) * f_tan(par[5]));
    const float d = sqrtf(fmaf(dq, dq, edgeCorr * edgeCorr));
    if (r > L.rout + d || r < L.rin - d) {
      wsr = kWsrOutside;
    } else if (r < L.rout - d && r > L.rin + d) {
      wsr = kWsrInside;
      if (L.has_hole) {
        if (r < L.hole_max - d && r > L.hole_min + d)
          wsr = kWsrOutside;
        else if (r < L.hole_max + d && r > L.hole_min - d)
          wsr = kWsrEdge;
      }
    } else {
      wsr = kWsrEdge;
    }
    q = r;
  }
  if (wsr == kWsrOutside) return -1;

  dphi = fminf(fmaxf(fabsf(dphi), min_dphi), max_dphi);
  dq = fminf(fmaxf(dq, min_dq), max_dq);
  const int qb1 = q_bin_checked(L, q - dq);
  const int qb2 = q_bin_checked(L, q + dq) + 1;
  const int pb1 = phi_bin(phi - dphi);
  const int pb2 = phi_bin(phi + dphi) + 1;

  // Bins in scan order (q row, then phi bin mod 256), read eight at a time
  // so the loads of a row are in flight together.
  constexpr int kBinChunk = 8;
  int n = 0;
  for (int qi = qb1; qi < qb2; ++qi) {
    const uint32_t* row = bins + qi * 256;
    for (int p0 = pb1; p0 < pb2; p0 += kBinChunk) {
      uint32_t bv[kBinChunk];
#pragma unroll
      for (int k = 0; k < kBinChunk; ++k)
        bv[k] = p0 + k < pb2 ? (kGenericBins ? row[(p0 + k) & 0xff] : __ldg(row + ((p0 + k) & 0xff)))
                             : 0u;
#pragma unroll
      for (int k = 0; k < kBinChunk; ++k) {
        const int first = bv[k] & 0xffff, last = bv[k] >> 16;
        for (int hi = first; hi < last; ++hi) {
          if (n >= kMaxXHits) break;
          const float4 hs = __ldg(reinterpret_cast<const float4*>(E.sorted_hits + hit_base + hi));
          const float ddq = fabsf(q - hs.x);
          const float ddphi = cdist(fabsf(phi - hs.y));
          if (ddq >= dq) continue;
          if (ddphi >= dphi) continue;
          xhit[n * xstride] = __float_as_int(hs.z);
          ++n;
        }
      }
    }
  }
  return n;
}

// isStripQCompatible (mkFit/MkFinder.cc:837-860).
__device__ __forceinline__ bool strip_q_compatible(bool barrel, const float (&perr)[21],
                                                   const float (&ppar)[6], const float (&mpos)[3],
                                                   const float (&merr)[6]) {
  if (barrel) {
    const float res = fabsf(mpos[2] - ppar[2]);
    const float hitHL = sqrtf(merr[5] * 3.f);
    const float qErr = sqrtf(perr[5]);
    return hitHL + fmaxf(3.f * qErr, 0.5f) > res;
  }
  const float res0 = mpos[0] - ppar[0], res1 = mpos[1] - ppar[1];
  const float hitT2 = merr[0] + merr[2];
  const float hitT2inv = 1.f / hitT2;
  const float proj0 = merr[0] * hitT2inv, proj1 = merr[1] * hitT2inv, proj2 = merr[2] * hitT2inv;
  const float qErr = sqrtf(fabsf(fmaf(perr[2], proj2, fmaf(perr[0], proj0, 2.f * perr[1] * proj1))));
  const float resProj =
      sqrtf(fmaf(res1 * proj2, res1, fmaf(res0 * proj0, res0, 2.f * res1 * proj1 * res0)));
  return sqrtf(hitT2 * 3.f) + fmaxf(3.f * qErr, 0.5f) > resProj;
}

// passStripChargePCMfromTrack (mkFit/MkFinder.cc:867-896).
__device__ __forceinline__ bool strip_charge_ok(bool barrel, unsigned pcm, const float (&ppar)[6],
                                                const float (&merr)[6]) {
  constexpr unsigned kMaxPcm = 1620 + (0xfe << 3);
  if (pcm >= kMaxPcm) return true;
  float qSF;
  if (barrel) {
    const float hitT2 = merr[0] + merr[2];
    const float hitT2inv = 1.f / hitT2;
    const float proj0 = merr[0] * hitT2inv, proj1 = merr[1] * hitT2inv, proj2 = merr[2] * hitT2inv;
    const bool detXY_OK = fabsf(fmaf(proj0, proj2, -(proj1 * proj1))) < 0.1f;
    const float cosP = f_cos(ppar[4]);
    const float sinP = f_sin(ppar[4]);
    const float sinT = fabsf(f_sin(ppar[5]));
    qSF = detXY_OK ? sinT * sqrtf(fabsf(fmaf(-2.f * cosP * sinP, proj1,
                                             fmaf(sinP * sinP, proj2, fmaf(cosP * cosP, proj0, 1.f)))))
                   : 1.f;
  } else {
    qSF = fabsf(f_cos(ppar[5]));
  }
  const float qCorr = pcm * qSF;
  return qCorr > 1620u;
}

// HitMatchPair (mkFit/HitStructures.h:343-393).
struct HitMatchPair {
  int hit[2];
  int module[2];
  float chi2[2];
  __device__ void reset() {
    hit[0] = hit[1] = -1;
    module[0] = module[1] = -1;
    chi2[0] = chi2[1] = 1e9f;
  }
  __device__ void consider(int h, int m, float c2) {
    if (m == module[0]) {
      if (c2 < chi2[0]) { chi2[0] = c2; hit[0] = h; }
    } else if (m == module[1]) {
      if (c2 < chi2[1]) { chi2[1] = c2; hit[1] = h; }
    } else {
      if (chi2[0] > chi2[1]) {
        if (c2 < chi2[0]) { hit[0] = h; module[0] = m; chi2[0] = c2; }
      } else {
        if (c2 < chi2[1]) { hit[1] = h; module[1] = m; chi2[1] = c2; }
      }
    }
  }
  // Returns 0/1 for the chosen match, or -1.
  __device__ int find(int h, int m) const {
    (void)h;
    if (m == module[0]) return hit[1] >= 0 ? 1 : -1;
    if (m == module[1]) return hit[0] >= 0 ? 0 : -1;
    if (chi2[0] <= chi2[1]) return hit[0] >= 0 ? 0 : -1;
    return hit[1] >= 0 ? 1 : -1;
  }
};

}  // namespace mkfg

namespace mkfg {

//------------------------------------------------------------------------------
// Shared step implementations (plain kernels and the fused persistent kernel)
//------------------------------------------------------------------------------

// Every value is loaded before the first store: the compiler cannot tell
// the two buffers apart, and interleaved loads and stores would wait for
// one another (37 memory round trips instead of one).
__device__ __forceinline__ void copy_slot(const CandSoA& from, int fs, const CandSoA& to, int ts) {
  float par[6], err[21];
#pragma unroll
  for (int e = 0; e < 6; ++e) par[e] = from.par[e * from.cap + fs];
#pragma unroll
  for (int e = 0; e < 21; ++e) err[e] = from.err[e * from.cap + fs];
  const int chg = from.chg[fs], last = from.last[fs], nfound = from.nfound[fs];
  const int nmiss = from.nmiss[fs], nover = from.nover[fs], ninside = from.ninside[fs];
  const int ntail = from.ntail[fs];
  const float chi2 = from.chi2[fs], score = from.score[fs];
#pragma unroll
  for (int e = 0; e < 6; ++e) to.par[e * to.cap + ts] = par[e];
#pragma unroll
  for (int e = 0; e < 21; ++e) to.err[e * to.cap + ts] = err[e];
  to.chg[ts] = chg;
  to.chi2[ts] = chi2;
  to.score[ts] = score;
  to.last[ts] = last;
  to.nfound[ts] = nfound;
  to.nmiss[ts] = nmiss;
  to.nover[ts] = nover;
  to.ninside[ts] = ninside;
  to.ntail[ts] = ntail;
}

// TrackCand::addHitIdx counters (mkFit/HitStructures.h:714-735).
__device__ __forceinline__ void add_hit_counts(int hit, float chi2, int& nfound, int& nmiss,
                                               int& ninside, int& ntail, float& tchi2) {
  if (hit >= 0 || hit == -9) {
    ++nfound;
    tchi2 += chi2;
    ninside += ntail;
    ntail = 0;
  } else {
    ++nmiss;
    if (hit == -1) ++ntail;
  }
}

// Seed state at the start of layer-plan step `step`: a dormant seed starts
// finding at the step after its pickup layer (find_tracks_unroll_candidates,
// mkFit/MkBuilder.cc:1503-1566).
__device__ __forceinline__ int wake_seed(const FindConfigDev& C, int reg, int layer, int step,
                                         int state, int pickup_layer) {
  if (layer >= 0 && state == kDormant && pickup_layer == C.plan[reg][C.pickup[reg] + step - 1])
    return kFinding;
  return state;
}

// Output of the candidate preparation of one layer step.
struct PrepOut {
  bool active = false;  // candidate takes part in this layer
  int xs = 0;           // XHitSize
  int wsr = kWsrOutside;
  int extra = 0;        // held back: 1 plain copy, 2 copy with a stop node
  int extra_last = -1;  // arena node of the stop node (extra == 2)
  bool hole = false;    // a hole record was produced
  int hole_hit = 0;
  float hole_score = 0.f;
  float ppar[6];
  float perr[21];
};

// Unroll + looper stop (mkFit/MkBuilder.cc:1503-1566) for a candidate of a
// seed already in Finding state: a candidate whose last node is a stop (-2)
// is inactive; a low-pT looper outside r = 25 cm turning back gets a stop
// node and is inactive. Returns whether the candidate is active.
__device__ __forceinline__ bool cand_is_active(const EventDev& E, const CandSoA& B, int s, int slot,
                                               int layer, bool looper_stop) {
  // Parameters first: their loads overlap the stop-node lookup.
  const float x = B.par[0 * B.cap + slot], y = B.par[1 * B.cap + slot];
  const float ipt = B.par[3 * B.cap + slot], phi = B.par[4 * B.cap + slot];
  const int last = B.last[slot];
  if (hot_index(node_hot_of(E, s, last)) == -2) return false;
  const float pt = fabsf(1.f / ipt);
  if (looper_stop && pt < 1.2f) {  // IT_FwdSearch only
    const float dphi = fabsf(f_atan2(y, x) - phi);
    if (fmaf(x, x, y * y) > 625.f && dphi > 1.371f && dphi < 4.512f) {
      B.last[slot] = arena_append(E, s, -2, layer, 0.f, last);
      B.nmiss[slot] += 1;
      return false;
    }
  }
  return true;
}

// cand_is_active, loading the state of an active candidate.
__device__ __forceinline__ bool activate_cand(const EventDev& E, const CandSoA& B, int s, int slot,
                                              int layer, bool looper_stop, float (&par)[6],
                                              float (&err)[21], int& chg) {
  if (!cand_is_active(E, B, s, slot, layer, looper_stop)) return false;
  load_state(B, slot, par, err);
  chg = B.chg[slot];
  return true;
}

// Propagation to the layer, SelectHitIndices, missed-layer handling
// (mkFit/MkBuilder.cc:1568-1637) and the hole record (MkFinder.cc:1245-1283)
// for an active candidate. xhit receives up to 16 indices with stride xstride.
template <bool kGenericBins = false>
__device__ __forceinline__ void select_cand(const EventDev& E, const FindConfigDev& C,
                                            const LayerDev& L, const uint32_t* layer_bins,
                                            int hit_base, int reg, int layer, int s,
                                            const CandSoA& B, int slot, const float (&ppar)[6],
                                            const float (&perr)[21], int* xhit, int xstride,
                                            PrepOut& o);

template <bool kGenericBins = false>
__device__ __forceinline__ void prep_cand(const EventDev& E, const FindConfigDev& C,
                                          const LayerDev& L, const uint32_t* layer_bins,
                                          int hit_base, int reg, int layer, int s, const CandSoA& B,
                                          int slot, const float (&par)[6], const float (&err)[21],
                                          int chg, int* xhit, int xstride, PrepOut& o) {
  if (L.is_barrel)
    propagate_to_r<false>(par, err, chg, L.propagate_to, C.inter_pflags, C.mat, false, o.ppar, o.perr);
  else
    propagate_to_z(par, err, chg, L.propagate_to, C.inter_pflags, C.mat, false, o.ppar, o.perr);
  select_cand<kGenericBins>(E, C, L, layer_bins, hit_base, reg, layer, s, B, slot, o.ppar, o.perr,
                            xhit, xstride, o);
}

// The part of prep_cand after the propagation: SelectHitIndices on the
// propagated state, missed-layer handling and the hole record.
template <bool kGenericBins>
__device__ __forceinline__ void select_cand(const EventDev& E, const FindConfigDev& C,
                                            const LayerDev& L, const uint32_t* layer_bins,
                                            int hit_base, int reg, int layer, int s,
                                            const CandSoA& B, int slot, const float (&ppar)[6],
                                            const float (&perr)[21], int* xhit, int xstride,
                                            PrepOut& o) {
  o.active = true;
  o.xs = select_hits<kGenericBins>(E, L, layer_bins, hit_base, ppar, perr, xhit, xstride, o.wsr);
  const float cand_r = hypot_f(ppar[0], ppar[1]);
  if (L.is_barrel && cand_r < L.rin) {
    o.xs = 0;
    o.wsr = kWsrOutside;
    o.extra = (reg == 2) ? 2 : 1;
    if (o.extra == 2) o.extra_last = arena_append(E, s, -2, layer, 0.f, B.last[slot]);
  } else if (o.wsr == kWsrOutside) {
    o.extra = 1;
  }
  if (o.xs < 0) o.xs = 0;
  if (o.wsr != kWsrOutside) {
    const int nin = B.ninside[slot], ntl = B.ntail[slot];
    int fake = ((nin + ntl) < C.max_holes && ntl < C.max_consec_holes) ? -1 : -2;
    if (o.wsr == kWsrEdge) fake = -3;
    const int ntail_rec = fake == -1 ? ntl + 1 : ntl;
    const float pt = fabsf(1.0f / ppar[3]);
    o.hole = true;
    o.hole_hit = fake;
    o.hole_score = score_struct(B.nfound[slot], ntail_rec, B.nover[slot], nin, B.chi2[slot], pt);
  }
}

// The chi2 and the cuts of one (candidate, hit) evaluation
// (MkFinder::FindCandidatesCloneEngine, mkFit/MkFinder.cc:1142-1193, with
// kalmanPropagateAndComputeChi2[Endcap]): dynamic chi2 cut, strip
// compatibility and strip charge. The pixel same-layer check is the
// caller's. Returns whether the hit passes; fills chi2 and module.
__device__ __forceinline__ bool pair_accept(const EventDev& E, const FindConfigDev& C,
                                            const LayerDev& L, int g, const float (&ppar)[6],
                                            const float (&perr)[21], int chg, float& chi2_out,
                                            int& module_out) {
  float mpos[3], merr[6];
  load_hit(E, g, mpos, merr);
  const uint32_t info = __ldg(E.hinfo + g);
  float hpar[6], herr_[21];
  float chi2;
  if (L.is_barrel) {
    propagate_to_r<false>(ppar, perr, chg, hypot_f(mpos[0], mpos[1]), C.intra_pflags, C.mat, false,
                         hpar, herr_);
    chi2 = kalman_barrel<true, false>(hpar, herr_, mpos, merr, hpar, herr_);
  } else {
    propagate_to_z(ppar, perr, chg, mpos[2], C.intra_pflags, C.mat, false, hpar, herr_);
    chi2 = kalman_endcap<true, false>(hpar, herr_, mpos, merr, hpar, herr_);
  }
  chi2 = fabsf(chi2);
  bool ok = chi2 < dynamic_chi2_cut(L, C.chi2_cut_min, ppar);
  if (ok && !L.is_pix) {
    ok = strip_q_compatible(L.is_barrel, perr, hpar, mpos, merr);
    ok &= strip_charge_ok(L.is_barrel, info >> 12, hpar, merr);
  }
  chi2_out = chi2;
  module_out = info & 0xfff;
  return ok;
}

// Score of an accepted hit record (IdxChi2List with nhits + 1, no tail
// holes, MkFinder.cc:1222-1233).
__device__ __forceinline__ float hit_record_score(const float (&ppar)[6], int nfound, int nover,
                                                  int nholes, float cand_chi2, float chi2) {
  const float pt = fabsf(1.0f / ppar[3]);
  return score_struct(nfound + 1, 0, nover, nholes, cand_chi2 + chi2, pt);
}

// One (candidate, hit) evaluation (MkFinder::FindCandidatesCloneEngine,
// mkFit/MkFinder.cc:1142-1240). Returns whether the hit is accepted; fills
// chi2, score, module.
__device__ __forceinline__ bool eval_pair(const EventDev& E, const FindConfigDev& C,
                                          const LayerDev& L, int layer, int s, int g,
                                          const float (&ppar)[6], const float (&perr)[21], int chg,
                                          int nfound, int nover, int nholes, float cand_chi2,
                                          float& chi2_out, float& score_out, int& module_out) {
  float chi2;
  bool ok = pair_accept(E, C, L, g, ppar, perr, chg, chi2, module_out);
  if (ok && L.is_pix) {
    // No second hit on a pixel layer of the first three hit-on-track nodes
    // (MkFinder.cc:1195-1210: ccand.m_hots[0 .. min(nFound, 2)]). Those are
    // the seed's own nodes, the first ones of its arena; for a seed with
    // fewer than three hits the reference reads past the nodes it holds, so
    // only the seed's nodes are checked here.
    const int n_seed = E.init_hot[s];
    for (int i = 0; i <= nfound && i <= 2 && i < n_seed; ++i)
      if (hot_layer(node_hot_of(E, s, i)) == layer) ok = false;
  }
  if (!ok) return false;
  chi2_out = chi2;
  score_out = hit_record_score(ppar, nfound, nover, nholes, cand_chi2, chi2);
  return true;
}

// UpdateWithLastHit on a state in registers (mkFit/MkFinder.cc:1291-1308;
// kalmanPropagateAndUpdate[Endcap], KalmanUtilsMPlex.cc:471-505, 697-731):
// propagation to the hit with the inter-layer flags, the update, and the
// charge flip of a negative 1/pT; g is the hit's global index.
__device__ __forceinline__ void update_state(const EventDev& E, const FindConfigDev& C,
                                             const LayerDev& L, int g, float (&par)[6],
                                             float (&err)[21], int& chg) {
  float mpos[3], merr[6];
  load_hit(E, g, mpos, merr);
  float ppar[6], perr[21];
  if (L.is_barrel) {
    propagate_to_r<false>(par, err, chg, hypot_f(mpos[0], mpos[1]), C.inter_pflags, C.mat, false, ppar,
                         perr);
    kalman_barrel<false, true>(ppar, perr, mpos, merr, par, err);
  } else {
    propagate_to_z(par, err, chg, mpos[2], C.inter_pflags, C.mat, false, ppar, perr);
    kalman_endcap<false, true>(ppar, perr, mpos, merr, par, err);
  }
  if (par[3] < 0) {
    chg = -chg;
    par[3] = -par[3];
  }
}

// UpdateWithLastHit + CopyOutParErr for the new candidate in slot `slot` of
// buffer N (MkFinder.cc:1291-1335): the state of its parent (slot `src` of
// buffer B, which the clone step leaves where it is) updated with the hit
// of global index g on layer L.
__device__ __forceinline__ void update_cand_at(const EventDev& E, const FindConfigDev& C,
                                               const LayerDev& L, int g, const CandSoA& B, int src,
                                               const CandSoA& N, int slot) {
  float par[6], err[21];
  load_state(B, src, par, err);
  int chg = B.chg[src];
  update_state(E, C, L, g, par, err, chg);
  store_state(N, slot, par, err);
  N.chg[slot] = chg;
}

// Records and per-candidate step results of one seed, wherever they live
// (global memory in the plain form, shared memory in the fused form).
struct SeedRecords {
  const Record* rec_;      // kRecPerSeed records
  const uint32_t* mask_;   // per candidate: bit h set = record h present
  const int* wsr_;         // WSR code | extra kind << 8, per candidate
  const int* extra_last_;  // stop node of a kind-2 extra, per candidate
  __device__ Record rec(int idx) const { return rec_[idx]; }
  __device__ uint32_t mask(int c) const { return mask_[c]; }
  __device__ int extra_kind(int c) const { return wsr_[c] >> 8; }
  __device__ int extra_last(int c) const { return extra_last_[c]; }
};

// Total order of record scores as integers: the float order, with -0 taken
// as +0 and NaN below every number (NaN records go last, in record order)
// but above kNoKey, the key of an empty place.
constexpr int kNoKey = INT_MIN;
__device__ __forceinline__ int score_key(float score) {
  const float z = __fadd_rn(score, 0.f);
  const int k = __float_as_int(z);
  return z != z ? kNoKey + 1 : (k >= 0 ? k : k ^ 0x7fffffff);
}
// The score a key stands for (+0 for -0, a NaN for any NaN).
__device__ __forceinline__ float key_score(int key) {
  return __int_as_float(key >= 0 ? key : key ^ 0x7fffffff);
}

// Writes a hit-on-track node at arena position pos of seed s (allocated by
// the caller); returns pos, or prev after an overflow (flagged).
__device__ __forceinline__ int arena_put(const EventDev& E, int s, int pos, int index, int layer,
                                         float chi2, int prev) {
  if (pos >= E.hot_cap) {
    atomicOr(E.err_flags, kErrArena);
    return prev;
  }
  const size_t k = (size_t)s * E.hot_cap + pos;
  E.node_hot[k] = hot_pack(index, layer);
  E.node_chi2[k] = chi2;
  E.node_prev[k] = prev;
  return pos;
}

// A seed's new candidates as the ranking leaves them, in the registers of
// the 8 lanes that work on the seed: lane i holds new candidate i < n.
struct CloneList {
  int n;          // new candidates
  int n_records;  // records present
  int rec;        // record taken (index in the seed's records)
  int parent;     // parent's slot
  int kind;       // held-back copy: 1 plain, 2 with a stop node; 0 a record's candidate
  int ov;         // parent's record of the overlap hit, or -1
  int node;       // arena position of the candidate's first node
  bool upd;       // takes an update
};

// Shared-memory scratch of a seed's clone step: the records present (or,
// then, the best of them in order).
constexpr int kCloneList = 32;
struct CloneScratch {
  int key[kCloneList];  // score_key
  int id[kCloneList];   // record index, bit 8: a stop (-2), bit 9: a hit
};
__device__ __forceinline__ int clone_id(int idx, int hit) {
  return idx | (hit == -2 ? 256 : 0) | (hit >= 0 ? 512 : 0);
}

// First half of CandCloner::ProcessSeedRange (mkFit/CandCloner.cc:36-189)
// for the seeds of a warp, 8 lanes per seed (lane c of them works on
// candidate c, then on new candidate c): the top records by (score desc,
// record order), merged with the held-back candidates into the list of new
// candidates, the best short candidate, and the arena space of the step.
// All lanes of the warp call it; `on` is false for the lanes of a seed that
// takes no part. The lanes own the seed.
__device__ __forceinline__ CloneList clone_rank(const EventDev& E, const FindConfigDev& C, bool on,
                                                int s, int layer, int ncand, int cur,
                                                const SeedRecords& R, CloneScratch& X, int lane) {
  constexpr unsigned kFull = 0xffffffffu;
  const CandSoA& B = E.cand[cur];
  const int M = C.max_cands;
  const int c = lane & 7, g0 = lane & 24, s0 = s * kSlots;
  const unsigned gmask = 0xffu << g0;
  const bool is_cand = on && c < ncand;
  const int hot0 = on ? E.hot_size[s] : 0;
  const bool bs_valid = on && E.bshort_valid[s];
  const float bs_in = on ? E.bshort.score[s] : 0.f;

  // Records present in record order: candidate c's start at place `at`.
  const uint32_t cm = is_cand ? R.mask(c) : 0u;
  const int kind = is_cand ? R.extra_kind(c) : 0;
  int at = __popc(cm);
#pragma unroll
  for (int off = 1; off < kSlots; off <<= 1) {
    const int v = __shfl_up_sync(kFull, at, off, kSlots);
    if (c >= off) at += v;
  }
  const int n_valid = __shfl_sync(kFull, at, kSlots - 1, kSlots);
  at -= __popc(cm);
  const unsigned em0 = (__ballot_sync(kFull, kind != 0) >> g0) & 0xffu;

  // Top-num_hits records in (score desc, record index asc) order: the
  // reference's std::sort by score; on exact score ties this order is the
  // stable one. Record p goes to the place given by the count of those
  // before it. More records than places are taken in rounds, the best so far
  // first. The 8 lanes take the records in turn, whosever they are: a seed
  // in dense noise has one candidate's dozen hits, and one lane would wait
  // for them one after the other.
  const int num_hits = min(n_valid, M);
  constexpr int kPer = kCloneList / kSlots;
  int base = 0, kept = 0;
  do {
    const bool more = base < n_valid;
    const int n = more ? min(kept + n_valid - base, kCloneList) : 0;
    if (more) {
      int p = kept + at - base;
      for (uint32_t m = cm; m; m &= m - 1, ++p)
        if (p >= kept && p < n) X.id[p] = c * kRecPerCand + __ffs(m) - 1;
    }
    __syncwarp();
    int key[kPer], id[kPer], rank[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int p = c + kSlots * k;
      rank[k] = p < n ? 0 : kCloneList;
      key[k] = kNoKey;
      id[k] = 0;
      if (p < n) {
        id[k] = X.id[p];
        if (p >= kept) {
          const Record r = R.rec(id[k]);
          key[k] = score_key(r.score);
          id[k] = clone_id(id[k], r.hit);
        } else {
          key[k] = X.key[p];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (c + kSlots * k < n) X.key[c + kSlots * k] = key[k];
    __syncwarp();
    if (n <= kSlots) {
      for (int j = 0; j < n; ++j) {
        const int kj = X.key[j];
        rank[0] += (kj > key[0]) || (kj == key[0] && j < c);
      }
    } else {
      for (int j = 0; j < n; ++j) {
        const int kj = X.key[j];
#pragma unroll
        for (int k = 0; k < kPer; ++k)
          rank[k] += (kj > key[k]) || (kj == key[k] && j < c + kSlots * k);
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (rank[k] < num_hits) {
        X.key[rank[k]] = key[k];
        X.id[rank[k]] = id[k];
      }
    if (more) {
      base += n - kept;
      kept = min(n, num_hits);
    }
  } while (__any_sync(kFull, base < n_valid));
  __syncwarp();

  // The new candidate list. The best short candidate's score decides
  // whether a stop (-2) record replaces it.
  CloneList out{0, n_valid, 0, 0, 0, -1, 0, false};
  int bs_from = -1;
  float bs_score = bs_valid ? bs_in : -1e16f;  // getScoreWorstPossible
  const bool has = c < num_hits;
  const int my_id = has ? X.id[c] : 0;
  const unsigned stop_m = (__ballot_sync(kFull, has && (my_id & 256)) >> g0) & 0xffu;
  const unsigned push_m = (__ballot_sync(kFull, has && !(my_id & 256)) >> g0) & 0xffu;
  if (n_valid == 0) {
    // hitsForSeed empty (CandCloner.cc:163-172): the extras survive.
    out.n = __popc(em0);
    out.parent = c < out.n ? (int)__fns(em0, 0, c + 1) : 0;
  } else if (em0 == 0) {
    // No extras: the records in order, less the stops, of which the first
    // (best) may replace the best short candidate. All lanes at once.
    out.n = __popc(push_m);
    if (stop_m) {
      const int f = __ffs(stop_m) - 1;
      if (key_score(X.key[f]) > bs_score) bs_from = X.id[f] & 255;
    }
    out.rec = X.id[c < out.n ? (stop_m ? (int)__fns(push_m, 0, c + 1) : c) : 0];
    out.parent = (out.rec & 255) / kRecPerCand;
  } else {
    // Extras and records in turn, the same in every lane of the seed.
    const float my_score = is_cand ? B.score[s0 + c] : 0.f;
    unsigned em = em0;
    auto push = [&](int rec, int parent) {
      if (c == out.n) {
        out.rec = rec;
        out.parent = parent;
      }
      ++out.n;
    };
    for (int ih = 0; ih < num_hits; ++ih) {
      const int rid = X.id[ih];
      const float score = key_score(X.key[ih]);
      if (rid & 256) {
        if (score > bs_score) {
          bs_score = score;
          bs_from = rid & 255;
        }
        continue;
      }
      while (em && out.n < M) {
        const int e = __ffs(em) - 1;
        if (!(__shfl_sync(gmask, my_score, e, kSlots) > score)) break;
        push(-1, e);
        em &= em - 1;
      }
      if (out.n >= M) break;
      push(rid, (rid & 255) / kRecPerCand);
    }
    for (; em && out.n < M; em &= em - 1) push(-1, __ffs(em) - 1);
  }
  // Lane i < n: candidate i's record (held-back copies have none).
  const bool mine = c < out.n;
  const bool from_rec = mine && n_valid > 0 && out.rec >= 0;
  const bool hit = from_rec && (out.rec & 512);
  out.rec = from_rec ? out.rec & 255 : 0;
  out.kind = __shfl_sync(kFull, kind, out.parent, kSlots);
  if (from_rec || !mine) out.kind = 0;

  // The overlap hit (CandCloner.cc:120-124): the parent's hit records under
  // the overlap chi2 cut, considered in hit order as MkFinder does
  // (:1212-1216). A record's own hit never pairs with itself, so a parent
  // without another one needs no look.
  const uint32_t pm = __shfl_sync(kFull, cm, out.parent, kSlots) & ((1u << kMaxXHits) - 1u);
  if (hit) {
    const int h = out.rec - out.parent * kRecPerCand;
    if ((pm & ~(1u << h)) && fabsf(1.f / B.par[3 * B.cap + s0 + out.parent]) > C.pt_cut_overlap) {
      HitMatchPair p;
      p.reset();
      int module = 0;
      for (uint32_t m = pm; m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        const Record q = R.rec(out.parent * kRecPerCand + k);
        if (k == h) module = q.module;
        if (q.chi2 < C.chi2_cut_overlap) p.consider(k, q.module, q.chi2);
      }
      const int f = p.find(h, module);
      if (f >= 0) out.ov = out.parent * kRecPerCand + (f ? p.hit[1] : p.hit[0]);
    }
  }
  out.upd = hit;

  // Arena nodes of this step, one allocation for the seed: the best short
  // candidate's hole node first, then one or two nodes per new candidate
  // with a record, in candidate order.
  const int own = from_rec ? 1 + (out.ov >= 0) : 0;
  int nodes = own;
#pragma unroll
  for (int off = 1; off < kSlots; off <<= 1) {
    const int v = __shfl_up_sync(kFull, nodes, off, kSlots);
    if (c >= off) nodes += v;
  }
  const int total = __shfl_sync(kFull, nodes, kSlots - 1, kSlots) + (bs_from >= 0);
  if (on && c == 0 && total) E.hot_size[s] = hot0 + total;
  out.node = hot0 + (bs_from >= 0) + nodes - own;

  // Best short candidate (a -2 record scoring above the current best): the
  // parent with the stop as its last node; its state by all 8 lanes. Loads
  // first (see copy_slot).
  if (bs_from >= 0) {
    const int src = s0 + bs_from / kRecPerCand;
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int e = c + kSlots * k;
      if (e < 27) v[k] = (e < 6 ? B.par + e * B.cap : B.err + (e - 6) * B.cap)[src];
    }
    if (c == 0) {
      int nfound = B.nfound[src], nmiss = B.nmiss[src], nin = B.ninside[src], ntl = B.ntail[src];
      float chi2 = B.chi2[src];
      const int chg = B.chg[src], nover = B.nover[src], last = B.last[src];
      const float score = R.rec(bs_from).score;
      add_hit_counts(-2, 0.f, nfound, nmiss, nin, ntl, chi2);
      E.bshort.last[s] = arena_put(E, s, hot0, -2, layer, 0.f, last);
      E.bshort.chg[s] = chg;
      E.bshort.chi2[s] = chi2;
      E.bshort.score[s] = score;
      E.bshort.nfound[s] = nfound;
      E.bshort.nmiss[s] = nmiss;
      E.bshort.nover[s] = nover;
      E.bshort.ninside[s] = nin;
      E.bshort.ntail[s] = ntl;
      E.bshort_valid[s] = 1;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int e = c + kSlots * k;
      if (e < 27)
        (e < 6 ? E.bshort.par + e * E.bshort.cap : E.bshort.err + (e - 6) * E.bshort.cap)[s] = v[k];
    }
  }
  return out;
}

// Second half, by lane i < l.n of the seed's 8: new candidate i written
// into the other buffer -- counters and hit-on-track nodes, and the
// parent's parameters and covariance unless an update follows, which reads
// them from the parent and writes the updated ones (copy_all: always).
// Returns its update code: 1 + the index in the layer of the last hit added
// (the overlap hit if any), 0 for none.
__device__ __forceinline__ int clone_write(const EventDev& E, int s, int layer, int cur,
                                           const SeedRecords& R, const CloneList& l, int i,
                                           bool copy_all) {
  const CandSoA& B = E.cand[cur];
  const CandSoA& N = E.cand[cur ^ 1];
  const int src = s * kSlots + l.parent, dst = s * kSlots + i;
  Record r{0, 0, 0.f, 0.f}, q{0, 0, 0.f, 0.f};
  if (!l.kind) r = R.rec(l.rec);
  if (l.ov >= 0) q = R.rec(l.ov);
  // Loads first (see copy_slot).
  const int chg = B.chg[src];
  int nfound = B.nfound[src], nmiss = B.nmiss[src], nover = B.nover[src];
  int nin = B.ninside[src], ntl = B.ntail[src], last = B.last[src];
  float chi2 = B.chi2[src], score = B.score[src];
  if (copy_all || !l.upd) {
    float par[6], err[21];
    load_state(B, src, par, err);
    store_state(N, dst, par, err);
  }
  int upd = 0;
  if (l.kind) {
    if (l.kind == 2) {
      last = R.extra_last(l.parent);
      ++nmiss;
    }
  } else {
    add_hit_counts(r.hit, r.chi2, nfound, nmiss, nin, ntl, chi2);
    last = arena_put(E, s, l.node, r.hit, layer, r.chi2, last);
    score = r.score;
    int hit = r.hit;
    if (l.ov >= 0) {
      add_hit_counts(q.hit, q.chi2, nfound, nmiss, nin, ntl, chi2);
      last = arena_put(E, s, l.node + 1, q.hit, layer, q.chi2, last);
      ++nover;
      hit = q.hit;
    }
    if (l.upd) upd = 1 + hit;
  }
  N.chg[dst] = chg;
  N.chi2[dst] = chi2;
  N.score[dst] = score;
  N.last[dst] = last;
  N.nfound[dst] = nfound;
  N.nmiss[dst] = nmiss;
  N.nover[dst] = nover;
  N.ninside[dst] = nin;
  N.ntail[dst] = ntl;
  return upd;
}

// Candidate score for the final merge: getScoreCand with default arguments
// (mkFit/HitStructures.h:519-531).
__device__ __forceinline__ float cand_score(const CandSoA& B, int slot) {
  const float pt = fabsf(1.f / B.par[3 * B.cap + slot]);
  float chi2 = B.chi2[slot];
  if (chi2 < 0) chi2 = 0.f;
  return score_calc(B.nfound[slot], 0, B.nover[slot], B.ninside[slot], chi2, pt, false);
}

// CombCandidate::MergeCandsAndBestShortOne(update_score, sort_cands)
// (mkFit/HitStructures.cc:511-552) for one seed; writes the final list into
// buffer cur ^ 1 and returns the final candidate count. When the list
// stays as it is (already in score order, no best short candidate to
// insert) only the scores are written, in place, and `moved` is false.
__device__ __forceinline__ int merge_seed(const EventDev& E, const FindConfigDev& C, int s,
                                          int n, int cur, bool& moved) {
  const CandSoA& B = E.cand[cur];
  const CandSoA& N = E.cand[cur ^ 1];
  float score[kSlots + 1];
  int order[kSlots + 1];
  for (int c = 0; c < n; ++c) {
    score[c] = cand_score(B, s * kSlots + c);
    order[c] = c;
  }
  // Insertion sort by score, descending (std::sort on <= 16 elements).
  for (int i = 1; i < n; ++i) {
    const int o = order[i];
    const float v = score[o];
    int j = i;
    while (j > 0 && score[order[j - 1]] < v) {
      order[j] = order[j - 1];
      --j;
    }
    order[j] = o;
  }
  const bool has_bs = E.bshort_valid[s];
  // With candidates left the best short candidate's score is recomputed
  // with theirs; with none it is appended as it is, keeping the score of
  // the record that made it (getScoreStruct, in-finding weights, tail holes
  // counted) -- HitStructures.cc:515-548.
  const float bs = has_bs ? (n > 0 ? cand_score(E.bshort, s) : E.bshort.score[s]) : 0.f;
  int ins = -1;
  if (n > 0) {
    if (has_bs && bs > score[order[n - 1]]) {
      int ci = 0;
      while (score[order[ci]] > bs) ++ci;
      if (n >= C.max_cands) --n;
      ins = ci;
    }
  } else if (has_bs) {
    ins = 0;
  }
  bool identity = ins < 0;
  for (int i = 0; i < n && identity; ++i) identity = order[i] == i;
  moved = !identity;
  if (identity) {
    for (int c = 0; c < n; ++c) B.score[s * kSlots + c] = score[c];
    E.bshort_valid[s] = 0;
    return n;
  }
  int w = 0;
  for (int i = 0; i <= n; ++i) {
    if (i == ins) {
      const int dst = s * kSlots + w;
      copy_slot(E.bshort, s, N, dst);
      N.score[dst] = bs;
      ++w;
    }
    if (i == n) break;
    const int src = s * kSlots + order[i];
    const int dst = s * kSlots + w;
    copy_slot(B, src, N, dst);
    N.score[dst] = score[order[i]];
    ++w;
  }
  E.bshort_valid[s] = 0;
  return w;
}

}  // namespace mkfg
