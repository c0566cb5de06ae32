// Fused clone-engine finding: one thread block carries a chunk of W
// consecutive seeds through every layer-plan step and the final merge in a
// single launch. Per step the block runs the same phases as the plain
// form's kernels (prep, chi2, clone, update), separated by block
// barriers, but the step scratch -- states propagated to the layer, selected
// hit lists, the (candidate, hit) pair list, and the IdxChi2List records
// -- lives in shared memory and never
// goes to DRAM. Candidate buffers, seed scalars and the hit-on-track arena
// stay in global memory (each seed's data is touched by one block only, so
// they stay in L1/L2 between phases).
//
// The per-candidate and per-seed work is the code the plain kernels call
// (find_steps.cuh), with every rounding written out, so results are the plain
// form's bit for bit; a chunk stops stepping once none of its seeds can change
// any more.
//
// Bound by latency: a step is the chain of its four phases in one block
// (18.5 us per step for 120 seeds, 8 per block: 0.78 ms per run). With a
// warp per seed in the clone phase 1.18 ms; with the branch-free arithmetic
// (flat_math.cuh) 0.58, measured when the compiler chose the FMAs and other
// ones turned near-ties of the ranking in one small event out of ten.
#pragma once

#include "find_steps.cuh"

namespace mkfg {

template <int W>
struct FusedShared {
  static constexpr int T = W * kSlots;  // threads: one per candidate slot
  float ppar[6 * T];
  float perr[21 * T];
  int xhit[kMaxXHits * T];
  int wsr[T];
  int extra_last[T];
  Record rec[W * kRecPerSeed];
  uint32_t rmask[T];
  unsigned short pairs[T * kMaxXHits];
  CloneScratch scratch[W];
  int n_pairs;
  int pairs_end[2];   // of them in barrel and endcap layers
};

template <int W>
__global__ void __launch_bounds__(W * kSlots) k_find_fused(EventDev E,
                                                           const FindConfigDev* __restrict__ Cp) {
  constexpr int T = W * kSlots;
  static_assert(T % 32 == 0, "chunk must fill whole warps");
  extern __shared__ __align__(16) unsigned char fused_smem[];
  FusedShared<W>& S = *reinterpret_cast<FusedShared<W>*>(fused_smem);
  const FindConfigDev& C = *Cp;
  const int tid = threadIdx.x, lane = tid & 31;
  const int s0 = blockIdx.x * W;
  const int ls = tid / kSlots, c = tid % kSlots;  // local seed, candidate slot
  const int s = s0 + ls;
  const bool in_range = s < E.n_seeds;
  const int slot = s * kSlots + c;
  const unsigned grp = 0xffu << (lane & ~7);
  const int reg = in_range ? E.region[s] : 0;
  const int ev = in_range ? E.seed_event[s] : 0;
  const int pickup_layer = in_range ? E.pickup_layer[s] : -1;
  const int* lb = E.layer_begin + ev * E.lb_stride;
  const int n_local = min(W, E.n_seeds - s0);

  if (tid == 0) S.n_pairs = S.pairs_end[0] = S.pairs_end[1] = 0;
  __syncthreads();

  for (int step = 1; step <= C.max_steps; ++step) {
    //-------------------------------------------------------------- prep
    int layer = -1, state = kFinished, ncand = 0, buf = 0;
    if (in_range) {
      layer = plan_layer(C, reg, step);
      state = wake_seed(C, reg, layer, step, E.state[s], pickup_layer);
      ncand = E.n_cands[s];
      buf = E.cur[s];
    }
    const CandSoA& B = E.cand[buf];
    float par[6], err[21];
    int chg = 0;
    const bool active = in_range && layer >= 0 && state == kFinding && c < ncand &&
                        activate_cand(E, B, s, slot, layer, C.looper_stop != 0, par, err, chg);
    const unsigned act = __ballot_sync(0xffffffffu, active) & grp;
    int* cnt = E.step_count + step * kCntN;
    const bool barrel = layer >= 0 && C.layer[layer].is_barrel;
    {
      const unsigned all = __ballot_sync(0xffffffffu, active);
      const unsigned nb = __popc(__ballot_sync(0xffffffffu, active && barrel));
      const unsigned nf = __popc(__ballot_sync(0xffffffffu, c == 0 && act != 0));
      if (lane == 0 && all) {
        atomicAdd(&E.work[step * kWorkN + 0], __popc(all));
        if (nb) atomicAdd(cnt + kCntActBarrel, nb);
        if (nb < __popc(all)) atomicAdd(cnt + kCntActEndcap, __popc(all) - nb);
        atomicAdd(cnt + kCntFind, nf);
      }
    }
    if (in_range && c == 0) {
      if (layer >= 0 && state == kFinding && act == 0) state = kFinished;
      E.state[s] = state;
    }
    const int rbase = ls * kRecPerSeed + c * kRecPerCand;
    PrepOut o;
    if (active) {
      const LayerDev& L = C.layer[layer];
      prep_cand(E, C, L, E.bins + (size_t)ev * E.n_bins + L.bin_offset, lb[layer], reg, layer, s,
                B, slot, par, err, chg, S.xhit + tid, T, o);
      if (o.extra == 2) S.extra_last[tid] = o.extra_last;
#pragma unroll
      for (int e = 0; e < 6; ++e) S.ppar[e * T + tid] = o.ppar[e];
#pragma unroll
      for (int e = 0; e < 21; ++e) S.perr[e * T + tid] = o.perr[e];
      if (o.xs > 0) {
        atomicAdd(S.pairs_end + !barrel, o.xs);
        const int base = atomicAdd(&S.n_pairs, o.xs);
        for (int h = 0; h < o.xs; ++h) S.pairs[base + h] = (unsigned short)(tid * kMaxXHits + h);
      }
    }
    if (o.hole) S.rec[rbase + kMaxXHits] = Record{o.hole_hit, -1, 0.f, o.hole_score};
    S.rmask[tid] = o.hole ? 1u << kMaxXHits : 0u;
    S.wsr[tid] = o.wsr | (o.extra << 8);
    __syncthreads();

    //-------------------------------------------------------------- chi2
    const int np = S.n_pairs;
    if (tid == 0 && np) {
      atomicAdd(&E.pair_count[step], np);
      atomicAdd(&E.work[step * kWorkN + 2], np);
      if (S.pairs_end[0]) atomicAdd(cnt + kCntPairBarrel, S.pairs_end[0]);
      if (S.pairs_end[1]) atomicAdd(cnt + kCntPairEndcap, S.pairs_end[1]);
    }
    for (int p = tid; p < np; p += T) {
      const int code = S.pairs[p];
      const int lt = code / kMaxXHits, h = code % kMaxXHits;
      const int pls = lt / kSlots, pc = lt % kSlots;
      const int ps = s0 + pls, pslot = ps * kSlots + pc;
      const int player = plan_layer(C, E.region[ps], step);
      const LayerDev& L = C.layer[player];
      float ppar[6], perr[21];
#pragma unroll
      for (int e = 0; e < 6; ++e) ppar[e] = S.ppar[e * T + lt];
#pragma unroll
      for (int e = 0; e < 21; ++e) perr[e] = S.perr[e * T + lt];
      const CandSoA& PB = E.cand[E.cur[ps]];
      const int hidx = S.xhit[h * T + lt];
      const int g = E.layer_begin[E.seed_event[ps] * E.lb_stride + player] + hidx;
      float chi2, score;
      int module;
      const int r = pls * kRecPerSeed + pc * kRecPerCand + h;
      if (eval_pair(E, C, L, player, ps, g, ppar, perr, PB.chg[pslot], PB.nfound[pslot],
                    PB.nover[pslot], PB.ninside[pslot] + PB.ntail[pslot], PB.chi2[pslot], chi2,
                    score, module)) {
        S.rec[r] = Record{hidx, module, chi2, score};
        atomicOr(S.rmask + lt, 1u << h);
      }
    }
    __syncthreads();

    //-------------------------------------------------------------- clone
    if (tid == 0) S.n_pairs = S.pairs_end[0] = S.pairs_end[1] = 0;
    // The 8 threads of a seed rank its records, then each writes a new
    // candidate and updates it with the hit it took.
    {
      const bool on = in_range && layer >= 0 && state == kFinding && act != 0;
      const SeedRecords R{S.rec + ls * kRecPerSeed, S.rmask + ls * kSlots, S.wsr + ls * kSlots,
                          S.extra_last + ls * kSlots};
      const CloneList l = clone_rank(E, C, on, on ? s : 0, layer, ncand, buf, R, S.scratch[ls], lane);
      if (on && c == 0) {
        atomicAdd(&E.work[step * kWorkN + 3], 1);
        atomicAdd(&E.work[step * kWorkN + 4], l.n_records);
        atomicAdd(&E.work[step * kWorkN + 5], l.n);
        E.n_cands[s] = l.n;
        E.cur[s] = buf ^ 1;
      }
      if (on && c < l.n) {
        const int upd = clone_write(E, s, layer, buf, R, l, c, false);
        //-------------------------------------------------------------- update
        if (upd) {
          atomicAdd(&E.work[step * kWorkN + 1], 1);
          atomicAdd(cnt + (barrel ? kCntUpdBarrel : kCntUpdEndcap), 1);
          update_cand_at(E, C, C.layer[layer], lb[layer] + upd - 1, E.cand[buf],
                         s * kSlots + l.parent, E.cand[buf ^ 1], slot);
        }
      }
    }
    // A seed can still change if it is dormant (it may wake up) or finding
    // with layers left in its plan.
    bool live = false;
    if (in_range && c == 0)
      live = state == kDormant || (state == kFinding && plan_layer(C, reg, step + 1) >= 0);
    if (!__syncthreads_or(live)) break;
  }

  //---------------------------------------------------------------- merge
  if (tid < n_local) {
    const int ms = s0 + tid;
    const int cur = E.cur[ms];
    bool moved = true;
    E.n_cands[ms] = merge_seed(E, C, ms, E.n_cands[ms], cur, moved);
    if (moved) E.cur[ms] = cur ^ 1;
  }
}

}  // namespace mkfg
