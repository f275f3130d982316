// bbs_kernels.cuh -- kernel templates of the GB300 path.
//
//   mcmc_kernel   persistent chain runner, src/Application.hpp:398-496.
//                 A chain is one warp, or `wpc` warps that split its cells
//                 (the block is then that one chain).  The chain's current
//                 and proposed ancestor rows are double-buffered in shared
//                 memory.  Proposals are read off a table of every node of the
//                 current tree (bbs_incr.cuh), or every node is evaluated, the
//                 cell rows loaded for each evaluation.
//   batch_kernel  the same over many datasets, from a work list.
//   init_kernel   the chains' initial states.
//   score_*       TreeScorer::logscore_tree over a batch: score_few_kernel a
//                 block per tree; score_walk_kernel and score_tree_kernel, a
//                 block or a warp per tree, codes inherited along the tree;
//                 score_kernel, a warp per tree, masked popcounts.
//   apply_kernel  realize_raw_move_sample + update ctor over a batch.
//   grad_kernel   sum-over-attachments score with its fused adjoint.
#pragma once
#include <cuda_runtime.h>

#include <cmath>

#include "bbs_device.cuh"
#include "bbs_incr.cuh"

namespace bbs {

// Rows x = 32 r + lane for the node groups r owned by warp `wic` of `wpc`.
template <int W32>
__device__ __forceinline__ void copy_rows_part(const uint32_t *src,
                                               uint32_t *dst, int n, int wpc,
                                               int wic, int lane) {
  constexpr int RS = rs_of_w32(W32);
  for (int r = wic; r < W32; r += wpc) {
    const int x = 32 * r + lane;
    if (x < n) {
      uint32_t v[W32];
      ld_row<W32>(src + x * RS, v);
      st_row<W32>(dst + x * RS, v);
    }
  }
}

template <int W32>
__device__ __forceinline__ void copy_rows(const uint32_t *src, uint32_t *dst,
                                          int n, int lane) {
  copy_rows_part<W32>(src, dst, n, 1, 0, lane);
}

// The scratch pieces of a slot: parent vectors and warp wic's scratch.
// (Host-callable too: the layout test walks it over every shape.)
struct SlotSum {
  uint8_t *par0, *par1;
  SumCtx sx;
};

__host__ __device__ __forceinline__ SlotSum slot_sum(uint8_t *slot, int n,
                                                     int rs, int wpc, int wic,
                                                     int w32, int q,
                                                     bool counts) {
  SlotSum o{};
  uint8_t *p = slot + slot_head_bytes(n, rs, wpc);
  o.par0 = p;
  o.par1 = p + n;
  p += align16(2 * n) + wic * sum_warp_bytes(n, w32, q, counts);
  // (rows of up to four words: position 1 on 8 bytes, as sum_cells_table reads
  // it, and three zeros past the end)
  o.sx.ord = reinterpret_cast<uint16_t *>(p) + (w32 <= 4 ? 3 : 0);
  p += order_bytes(n, w32);
  o.sx.hist = reinterpret_cast<int *>(p);
  p += align16(4 * 32 * ((n + 31) / 32));
  if (counts && w32 <= 4) o.sx.cnt = reinterpret_cast<uint32_t *>(p);
  if (counts && w32 > 4) {
    o.sx.ring = reinterpret_cast<uint32_t *>(p);
    o.sx.gt = reinterpret_cast<uint32_t *>(p + align16(ring_bytes(q)));
  }
  return o;
}

// Warp wic's part of the table of a slot without increments
// (table_slot_bytes).
__host__ __device__ __forceinline__ uint32_t *table_part(uint8_t *slot, int n,
                                                         int rs, int wpc,
                                                         int wic, int w32,
                                                         int q, int chunks) {
  return reinterpret_cast<uint32_t *>(
      slot + slot_bytes(n, rs, wpc, true, w32, q, false) +
      wic * table_part_bytes(n, q, chunks));
}

// The block's increment tables: for warp part wic of wpc and lane l, the
// cells c = 32 wic + 32 wpc q + l (q < Q; zero past the dataset's cells),
// as load_cells takes them; gene j's entry packs D bit | M bit << 8 of each
// such cell as the count table packs counts.  Cell rows are read with the
// stride rs that load_cells uses.
template <int Q>
__device__ __forceinline__ void build_increments(uint8_t *table, int wpc,
                                                 const DatasetDev &ds, int rs) {
  constexpr int NW = kPackWords<Q>;
  const int n = ds.n_nodes;
  for (int idx = threadIdx.x; idx < wpc * n * 32; idx += blockDim.x) {
    const int wic = idx / (n * 32);
    const int rem = idx - wic * n * 32;
    const int j = rem >> 5, l = rem & 31;
    uint32_t k[NW];
#pragma unroll
    for (int w = 0; w < NW; w++) k[w] = 0u;
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int c = 32 * wic + 32 * wpc * q + l;
      uint32_t v = 0;
      if (c < ds.n_cells) {
        const uint32_t kw = __ldg(ds.K + (size_t)c * rs + (j >> 5));
        const uint32_t mw = __ldg(ds.M + (size_t)c * rs + (j >> 5));
        const uint32_t bit = 1u << (j & 31);
        v = ((kw & ~mw & bit) ? 1u : 0u) | ((mw & bit) ? 256u : 0u);
      }
      k[q >> 1] |= v << (16 * (q & 1));
    }
    st_pack<Q>(reinterpret_cast<uint32_t *>(table + (size_t)wic * inc_table_bytes(n, Q)),
               j * 32 + l, k);
  }
}

// An evaluated tree: the score S = data term + prior, the (exact or
// expected) class counts e[4], the class sums sk and sm of the max score and
// the max score itself (S for the max score; for the sum score, sum_c max_j
// s_cj + prior).
struct Evaluated {
  float score, smax;
  float e[4];
  int sk, sm;
};

// The chain's class sums from its warps' (one block barrier when wpc > 1).
__device__ __forceinline__ Evaluated finish_max(const DatasetDev &ds,
                                                const LogTable &L, float prior,
                                                int a, int b, int wpc, int wic,
                                                int lane, int *part,
                                                int parity) {
  if (wpc > 1) {
    int *pp = part + parity * 12 * wpc;
    if (lane == 0) {
      pp[12 * wic] = a;
      pp[12 * wic + 1] = b;
    }
    __syncthreads();
    a = b = 0;
    for (int w = 0; w < wpc; w++) {
      a += pp[12 * w];
      b += pp[12 * w + 1];
    }
  }
  Evaluated o;
  o.sk = a;
  o.sm = b;
  int N[4];
  class_totals(ds, a, b, N);
#pragma unroll
  for (int i = 0; i < 4; i++) o.e[i] = (float)N[i];
  o.score = o.smax = tree_score(ds, a, b, L, prior);
  return o;
}

// The same for the sum score's fixed-point sums.
__device__ __forceinline__ Evaluated finish_sum(const DatasetDev &ds,
                                                float prior,
                                                long long (&acc)[6], int wpc,
                                                int wic, int lane, int *part,
                                                int parity) {
  if (wpc > 1) {
    long long *pp = reinterpret_cast<long long *>(part) + parity * 6 * wpc;
    if (lane == 0)
      for (int i = 0; i < 6; i++) pp[6 * wic + i] = acc[i];
    __syncthreads();
    for (int i = 0; i < 6; i++) acc[i] = 0;
    for (int w = 0; w < wpc; w++)
      for (int i = 0; i < 6; i++) acc[i] += pp[6 * w + i];
  }
  complete_expected_counts(ds, acc);
  Evaluated o;
  o.sk = o.sm = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) o.e[i] = ll_to_float(acc[i + 1]) * (1.0f / kFixScale);
  o.smax = __fadd_rn(ll_to_float(acc[5]) * (1.0f / kScoreScale), prior);
  o.score = __fadd_rn(ll_to_float(acc[0]) * (1.0f / kScoreScale), prior);
  return o;
}

// Evaluates a tree for the whole chain (all wpc warps) from its rows.
template <int W32, int Q, bool SUM>
__device__ __forceinline__ Evaluated evaluate(const uint32_t *rows, int n,
                                              const DatasetDev &ds,
                                              const LogTable &L, float prior,
                                              int wpc, int wic, int lane,
                                              int *part, int parity,
                                              const SumCtx &sx) {
  if constexpr (!SUM) {
    int a, b;
    score_part<W32, Q>(rows, n, ds, L, wpc, wic, lane, a, b, sx);
    return finish_max(ds, L, prior, a, b, wpc, wic, lane, part, parity);
  } else {
    long long acc[6];
    sum_part<W32, Q>(rows, n, ds, L, wpc, wic, lane, acc, sx);
    return finish_sum(ds, prior, acc, wpc, wic, lane, part, parity);
  }
}

// One chain for n_steps steps: src/Application.hpp:408-487 with the
// error-rate move chosen by md.error_move.  `chain_id` keys the Philox
// stream.  All wpc warps of the chain run this with the same arguments.
template <int W32, int Q, bool SUM>
__device__ __forceinline__ void run_chain(
    const DatasetDev &ds, const ModelDev &md, uint32_t chain_id,
    uint32_t *g, uint32_t *gbest, uint64_t *lhash, float *lbeta, int K,
    ChainState *gstate,
    const bbs_raw_move *moves, bbs_step_trace *trace, int n_steps,
    const volatile int *cancel, int *status, uint32_t *buf0, uint32_t *buf1,
    int *part, volatile int *sflag, uint4 *pbuf, const SlotSum &ss,
    int wpc, int wic, int lane) {
  const int n = ds.n_nodes;
  const bool multi = wpc > 1;
  const ChainState st = *gstate;
  copy_rows_part<W32>(g, buf0, n, wpc, wic, lane);
  if (multi) __syncthreads(); else __syncwarp();
  uint32_t *cur = buf0, *prop = buf1;
  // Rows of five to eight words inherit their counts through the ring, which
  // needs the parent vectors of the current tree and of the proposal.  A
  // parent vector is used only after it has been checked against its rows: a
  // realised move whose k-th (non)descendant fell back to node 0 (the
  // reference's rule when floor(u * count) reaches the count) changes the
  // rows in a way the parent-vector form does not follow, and may leave rows
  // that are no tree.  Such trees, and streamed cells of narrower rows, are
  // scored with masked popcounts, which take any rows.
  uint8_t *cpar = nullptr, *ppar = nullptr;
  bool cur_par_ok = false;  // cpar describes cur
  const bool track = W32 > 4 && ss.sx.ring != nullptr;
  if (track) {
    cpar = ss.par0;
    ppar = ss.par1;
    if (wic == 0) derive_parents<W32>(cur, n, cpar, ss.sx.hist, lane);
    if (multi) __syncthreads(); else __syncwarp();
    cur_par_ok = parents_match_rows<W32>(cur, n, cpar, lane);
  }
  SumCtx sx = ss.sx;
  float alpha = st.alpha, beta = st.beta, score = st.score, prior = st.prior;
  LogTable L{st.l00, st.l10, st.l01, st.l11};
  float ec[4] = {st.ec[0], st.ec[1], st.ec[2], st.ec[3]};
  int csk = st.sk, csm = st.sm;
  bool has_best = st.has_best != 0;
  float best_score = st.best_score, best_alpha = st.best_alpha,
        best_beta = st.best_beta;
  int bsk = st.best_sk, bsm = st.best_sm;
  uint32_t err_prop = st.err_proposed, err_acc = st.err_accepted;
  uint32_t lcount = st.list_count;  // co-optimal trees listed (K > 1)
  const bool learn = md.error_move != 0;
  int i = 0;
  bool cancelled = false;
  for (; i < n_steps; i++) {
    if (cancel != nullptr && (i & 255) == 0) {
      // one reader, then a chain-uniform decision
      if (wic == 0 && lane == 0) *sflag = *cancel;
      if (multi) __syncthreads(); else __syncwarp();
      const int c = *sflag;
      if (multi) __syncthreads(); else __syncwarp();
      if (c) {
        cancelled = true;
        break;
      }
    }
    // Philox blocks of the next 16 steps (a warp-uniform condition; the
    // previous step's reads ended at its closing __syncwarp)
    if (moves == nullptr && (i & 15) == 0) {
      philox_fill(pbuf, md.seed, chain_id, st.steps_done + (uint64_t)i, lane);
      __syncwarp();
    }
    const bbs_raw_move raw =
        moves != nullptr
            ? moves[i]
            : move_from_words(md.mp, (uint32_t)n, pbuf[2 * (i & 15)],
                              pbuf[2 * (i & 15) + 1], trace != nullptr);
    const bool err_move = raw.move_type == BBS_MOVE_CHANGE_BETA;
    float palpha = alpha, pbeta = beta, pprior = prior;
    LogTable PL = L;
    const uint32_t *scored = cur;
    float corr = 1.0f;
    RateProposal rates{};  // learned error moves
    bool fallback_move = false;  // the realised move took node 0 by fallback
    uint32_t Dv[W32], Dw[W32];
    if (!err_move) {
      const Realized R = realize_move<W32>(cur, n, beta, raw, lane, Dv, Dw);
      const uint32_t top = max(max(max(R.p.v, R.p.w), max(R.p.parent_of_v, R.p.parent_of_w)),
                               max(R.p.descendant_of_v, R.p.nondescendant_of_v));
      if (!device_check(top < (uint32_t)n, status, kCheckMoveNode, top, (uint32_t)n)) {
        cancelled = true;  // the chain stops where it is
        break;
      }
      build_proposal<W32>(cur, prop, n, R.p, Dv, Dw, R.related, wpc, wic,
                          lane);
      fallback_move = R.fallback;
      if (cur_par_ok && wic == 0)
        propose_parents(cpar, ppar, n, R.p, R.related, lane);
      scored = prop;
      // src/Application.hpp:443-450
      if (raw.move_type == BBS_MOVE_SWAP_SUBTREES && R.related)
        corr = __fdiv_rn((float)R.ndv, (float)R.ndw);
    } else if (!learn) {
      // reference ChangeBeta: beta + jump reflected into [0, 1]
      // (src/MutationTree.hpp:345-351)
      float nb = __fadd_rn(beta, raw.beta_jump);
      if (nb < 0.0f) nb = fabsf(nb);
      if (nb > 1.0f) nb = __fsub_rn(nb, __fmul_rn(2.0f, __fsub_rn(nb, 1.0f)));
      pbeta = nb;
      beta_terms(ds, pbeta, PL.l01, PL.l11, pprior);
    } else {
      // (preconditioned) random walk or Langevin step in logit space, with
      // the geometry of the current state from its class counts
      rates = propose_rates(ds, md, alpha, beta, ec, raw, lane);
      palpha = rates.palpha;
      pbeta = rates.pbeta;
      pprior = rates.pprior;
      PL = rates.PL;
    }
    if (multi) __syncthreads(); else __syncwarp();
    // The evaluated tree's parent vector.  It is checked against the rows
    // where it can be wrong -- a proposal whose move took node 0 by
    // fallback -- and used only where it checks out; checked builds check
    // every one and record a mismatch outside that case as a failed device
    // check.
    bool par_ok = false;
    if (cpar != nullptr && cur_par_ok) {
      const bool suspect = scored != cur && fallback_move;
      bool check = suspect;
#ifdef BBS_CHECKED
      check = true;
#endif
      par_ok = true;
      if (check) {
        par_ok = parents_match_rows<W32>(scored, n,
                                         scored == cur ? cpar : ppar, lane);
#ifdef BBS_CHECKED
        if (!suspect)
          device_check(par_ok, status, kCheckParent,
                       (uint32_t)raw.move_type, 4u);
#endif
      }
    }
    sx.par = par_ok ? (scored == cur ? cpar : ppar) : nullptr;
    const bool prop_par_ok = par_ok && scored != cur;
    const Evaluated ev = evaluate<W32, Q, SUM>(scored, n, ds, PL, pprior, wpc,
                                               wic, lane, part, i & 1, sx);
    const float pscore = ev.score, psmax = ev.smax;
    const float (&e)[4] = ev.e;
    const int sk = ev.sk, sm = ev.sm;
    bool accept;
    if (err_move && learn) {
      accept = accept_rates(ds, md, rates, alpha, beta, score, pscore, e,
                            raw.acceptance_level, lane);
      err_prop++;
      if (accept) err_acc++;
    } else {
      // src/Application.hpp:452-455
      const float ratio = __fmul_rn(
          corr, expf(__fmul_rn(__fsub_rn(pscore, score), md.gamma)));
      accept = ratio > raw.acceptance_level;
      if (err_move) {
        err_prop++;
        if (accept) err_acc++;
      }
    }
    // src/Application.hpp:456, best over proposals by the reference's max
    // score (the chain's own score unless it samples the sum score)
    if (!has_best || psmax > best_score) {
      has_best = true;
      best_score = psmax;
      best_alpha = palpha;
      best_beta = pbeta;
      bsk = sk;
      bsm = sm;
      copy_rows_part<W32>(scored, gbest, n, wpc, wic, lane);
      if (K > 1) {
        // a new best: the co-optimal list restarts with it
        const uint64_t h = tree_hash<W32>(scored, n, lane);
        if (wic == 0 && lane == 0) {
          lhash[0] = h;
          lbeta[0] = pbeta;
        }
        lcount = 1;
      }
    } else if (K > 1 && psmax == best_score && lcount < (uint32_t)K) {
      // a tie with the best: listed when it is a tree not listed yet
      const uint64_t h = tree_hash<W32>(scored, n, lane);
      const bool seen =
          __any_sync(BBS_FULL_MASK, lane < (int)lcount && lhash[lane] == h);
      if (!seen) {
        copy_rows_part<W32>(scored, gbest + (size_t)lcount * n * rs_of_w32(W32),
                            n, wpc, wic, lane);
        if (wic == 0 && lane == 0) {
          lhash[lcount] = h;
          lbeta[lcount] = pbeta;
        }
        lcount++;
      }
    }
    if (trace != nullptr && wic == 0 && lane == 0) {
      bbs_step_trace *t = trace + i;
      t->move = raw;
      t->proposed_score = pscore;
      t->current_score = accept ? pscore : score;
      t->proposed_beta = pbeta;
      t->accepted = accept ? 1u : 0u;
      t->proposed_alpha = palpha;
      t->proposed_max_score = psmax;
#pragma unroll
      for (int k = 0; k < 2; k++) t->reserved[k] = 0;
#pragma unroll
      for (int k = 0; k < 4; k++)
        t->proposed_counts[k] = SUM ? 0ull : (uint64_t)e[k];
    }
    if (accept) {
      if (!err_move) {
        uint32_t *t = cur;
        cur = prop;
        prop = t;
        uint8_t *tp = cpar;
        cpar = ppar;
        ppar = tp;
        cur_par_ok = prop_par_ok;
        if (cpar != nullptr && !cur_par_ok) {
          // the new tree's own parent vector, where its rows are a tree
          if (multi) __syncthreads(); else __syncwarp();
          if (wic == 0) derive_parents<W32>(cur, n, cpar, ss.sx.hist, lane);
          if (multi) __syncthreads(); else __syncwarp();
          cur_par_ok = parents_match_rows<W32>(cur, n, cpar, lane);
        }
      }
      alpha = palpha;
      beta = pbeta;
      score = pscore;
      prior = pprior;
      L = PL;
#pragma unroll
      for (int k = 0; k < 4; k++) ec[k] = e[k];
      csk = sk;
      csm = sm;
    }
    __syncwarp();
  }
  copy_rows_part<W32>(cur, g, n, wpc, wic, lane);
  if (wic == 0 && lane == 0) {
    ChainState o = st;
    o.alpha = alpha;
    o.beta = beta;
    o.score = score;
    o.prior = prior;
    o.l00 = L.l00;
    o.l10 = L.l10;
    o.l01 = L.l01;
    o.l11 = L.l11;
#pragma unroll
    for (int k = 0; k < 4; k++) o.ec[k] = ec[k];
    o.sk = csk;
    o.sm = csm;
    o.has_best = has_best ? 1u : 0u;
    o.best_alpha = best_alpha;
    o.best_beta = best_beta;
    o.best_score = best_score;
    o.best_sk = bsk;
    o.best_sm = bsm;
    o.steps_done = st.steps_done + (uint64_t)i;
    o.err_proposed = err_prop;
    o.err_accepted = err_acc;
    o.list_count = lcount;
    *gstate = o;
    if (cancelled && status != nullptr) atomicOr(status, 1);
  }
  if (multi) __syncthreads(); else __syncwarp();
}

template <int N>
struct IntConst {
  static constexpr int value = N;
};

// A tree scored from its rows, off the hot path: proposals that are not
// followed node by node, and error moves of the max score.
template <int W32, int Q, bool SUM>
__device__ __noinline__ Evaluated evaluate_rows(const uint32_t *rows,
                                                const DatasetDev *ds,
                                                const LogTable L, float prior,
                                                int wpc, int wic, int lane,
                                                int *part, int parity,
                                                SumCtx sx) {
  sx.par = nullptr;
  return evaluate<W32, Q, SUM>(rows, ds->n_nodes, *ds, L, prior, wpc, wic,
                               lane, part, parity, sx);
}

// A proposal's rows and, for a tree whose parent vector is known, its parent
// vector.
template <int W32>
__device__ __forceinline__ void propose_tree(
    const uint32_t *cur, uint32_t *prop, const uint8_t *cpar, uint8_t *ppar,
    int n, const bbs_move_params &p, const NodeSets<W32> &D, bool related,
    bool tree_ok, int wpc, int wic, int lane) {
  build_proposal<W32>(cur, prop, n, p, D.v, D.w, related, wpc, wic, lane);
  if (tree_ok && wic == 0) propose_parents(cpar, ppar, n, p, related, lane);
  if (wpc > 1) __syncthreads(); else __syncwarp();
}

// The same out of line, for proposals that are not described by classes.
// (Structures passed by value to functions that are not inlined go through
// local memory: with this and the table's update called that way on every
// proposal summed, 95 x 96 took 12.2 us a step, inlined 10.9.)
template <int W32>
__device__ __noinline__ void propose_tree_call(
    const uint32_t *cur, uint32_t *prop, const uint8_t *cpar, uint8_t *ppar,
    int n, const bbs_move_params p, const NodeSets<W32> D, bool related,
    bool tree_ok, int wpc, int wic, int lane) {
  propose_tree<W32>(cur, prop, cpar, ppar, n, p, D, related, tree_ok, wpc, wic,
                    lane);
}

// run_chain with a table of bbs_incr.cuh: `chunks` chunks of the warp's cells
// in tab, one for the sum score, which holds counts (rows of up to four words).
// Max score chains hold codes or, with COUNTS, counts (up to four words). Bound
// at 95 x 96 (1024 one-warp chains, 1.8 warps per scheduler) by the latency of
// one step's serial chain -- draw, descendant sets, table loads, reductions --
// no longer by the node loop's instructions.
template <int W32, int Q, bool SUM, bool COUNTS>
__device__ __forceinline__ void run_chain_table(
    const DatasetDev &ds, const ModelDev &md, uint32_t chain_id,
    uint32_t *g, uint32_t *gbest, uint64_t *lhash, float *lbeta, int K,
    ChainState *gstate, const bbs_raw_move *moves, bbs_step_trace *trace,
    int n_steps, const volatile int *cancel, int *status, uint32_t *buf0,
    uint32_t *buf1, int *part, volatile int *sflag, uint4 *pbuf,
    const SlotSum &ss, const Table<W32, Q> tab, int chunks, int wpc, int wic,
    int lane) {
  constexpr int NW = kPackWords<Q>;
  constexpr bool CODES = !SUM && !COUNTS;
  const int n = ds.n_nodes;
  const bool multi = wpc > 1;
  const int stride = 32 * wpc, c0 = 32 * wic;
  const ChainState st = *gstate;
  copy_rows_part<W32>(g, buf0, n, wpc, wic, lane);
  if (multi) __syncthreads(); else __syncwarp();
  uint32_t *cur = buf0, *prop = buf1;
  uint8_t *cpar = ss.par0, *ppar = ss.par1;
  float alpha = st.alpha, beta = st.beta, score = st.score, prior = st.prior;
  LogTable L{st.l00, st.l10, st.l01, st.l11};
  float ec[4] = {st.ec[0], st.ec[1], st.ec[2], st.ec[3]};
  int csk = st.sk, csm = st.sm;
  bool has_best = st.has_best != 0;
  float best_score = st.best_score, best_alpha = st.best_alpha,
        best_beta = st.best_beta;
  int bsk = st.best_sk, bsm = st.best_sm;
  uint32_t err_prop = st.err_proposed, err_acc = st.err_accepted;
  uint32_t lcount = st.list_count;
  const bool learn = md.error_move != 0;
  // the current tree's parent vector holds (its rows are a tree, and the
  // table and, for the sum score, the order and cell sums follow it)
  bool tree_ok = false;
  bool ord_ok = false;  // ss.sx.ord is the current tree's order
  if constexpr (SUM)
    if (lane < 3) ss.sx.ord[n + lane] = 0;  // (read in groups of four)
  MaxCode code{};
  CellSums<Q> cs;
  float pd[Q], pm[Q];
  float smax = 0.0f, eps = 0.0f, slack = 0.0f;  // of the sum score's bound
  int bounded = 0, rejected = 0, skip = 0;      // proposals bounded, rejected
  if constexpr (SUM) {
    Cells<W32, Q> cb;
    load_cells<W32, Q>(cb, ds, c0, stride, lane);
#pragma unroll
    for (int q = 0; q < Q; q++) {
      pd[q] = cb.pdb[q] - 8388608.0f;
      pm[q] = cb.pmb[q] - 8388608.0f;
    }
  }
  // The bound's tolerances for the current rates.  Exponents lie within
  // 1.45 n_genes max|l| + 105 in size and carry a few roundings each; a
  // cell's stored terms are rounded to 2^-16 and at their own size.
  auto tolerances = [&]() {
    const float big =
        (float)n * fmaxf(fmaxf(fabsf(L.l00), fabsf(L.l01)),
                         fmaxf(fabsf(L.l10), fabsf(L.l11))) + 73.0f;
    eps = big * 2.3841858e-06f;  // 10 roundings of twice 2^-24 big / ln 2
    slack = (float)ds.n_cells * fmaf(big, 4.7683716e-07f, 3.0517578e-05f);
  };
  // Set at the start and after an accepted tree that was not followed node
  // by node: the parent vector (where the rows are a tree), the codes and the
  // table anew from the rows; and, for the max score, after accepted rates
  // (the codes and the table).
  bool fresh_rows = true, fresh_table = true;
  uint8_t *const list = reinterpret_cast<uint8_t *>(ss.sx.hist);
  int i = 0;
  bool cancelled = false;
  while (i < n_steps) {
    const bool fresh = fresh_table;
    bool err_move = false;
    bbs_raw_move raw{};
    if (!fresh) {
      if (cancel != nullptr && (i & 255) == 0) {
        if (wic == 0 && lane == 0) *sflag = *cancel;
        if (multi) __syncthreads(); else __syncwarp();
        const int c = *sflag;
        if (multi) __syncthreads(); else __syncwarp();
        if (c) {
          cancelled = true;
          break;
        }
      }
      if (moves == nullptr && (i & 15) == 0) {
        moves_fill(pbuf, md, (uint32_t)n, chain_id, st.steps_done + (uint64_t)i,
                   trace != nullptr, lane);
        __syncwarp();
      }
      raw = moves != nullptr
                ? moves[i]
                : reinterpret_cast<const bbs_raw_move *>(pbuf)[i & 15];
      err_move = raw.move_type == BBS_MOVE_CHANGE_BETA;
    }
    float palpha = alpha, pbeta = beta, pprior = prior;
    LogTable PL = L;
    float corr = 1.0f;
    RateProposal rates{};  // learned error moves
    Evaluated ev;
    CellSums<Q> pcs;
    NodeSets<W32> D, C;
    Packed<NW> dv{}, dw{};
    Delta delta{};
    bbs_move_params mp{};
    bool related = false;
    bool classes = false;    // the proposal is described by classes
    int nc = 0, nv = 0;      // their nodes (list), those of the first class
    bool built = false;      // prop holds the proposal's rows
    bool applied = false;    // the table holds the proposal's counts
    bool from_rows = false;  // scored from its rows
    bool from_table = false; // summed over the table in the order of
    const uint32_t *order = nullptr;  // these rows (null: sx.ord holds it)
    if (fresh) {
      if (fresh_rows) {
        if (multi) __syncthreads(); else __syncwarp();
        if (wic == 0) derive_parents<W32>(cur, n, cpar, ss.sx.hist, lane);
        if (multi) __syncthreads(); else __syncwarp();
        tree_ok = parents_match_rows<W32>(cur, n, cpar, lane);
      }
      fresh_rows = fresh_table = false;
      if constexpr (CODES)
        code = make_code(L.l00, L.l01, L.l10, L.l11, ds.max_d, ds.max_m, lane);
      else if constexpr (SUM)
        tolerances();
      if (!tree_ok || (CODES && !code.usable)) continue;
      from_table = SUM;
      order = cur;
    } else if (!err_move) {
      bool general = true;
      if (tree_ok) {
        mp = realize_classes<W32>(cur, cpar, n, raw, lane, D.v, D.w, related,
                                  general, corr);
      }
      if constexpr (CODES) general = general || !code.usable;
      if (general) {
        corr = 1.0f;
        const Realized R = realize_move<W32>(cur, n, beta, raw, lane, D.v, D.w);
        mp = R.p;
        related = R.related;
        if (raw.move_type == BBS_MOVE_SWAP_SUBTREES && R.related)
          corr = __fdiv_rn((float)R.ndv, (float)R.ndw);
      }
      const uint32_t top = max(max(max(mp.v, mp.w), max(mp.parent_of_v, mp.parent_of_w)),
                               max(mp.descendant_of_v, mp.nondescendant_of_v));
      if (!device_check(top < (uint32_t)n, status, kCheckMoveNode, top, (uint32_t)n)) {
        cancelled = true;  // the chain stops where it is
        break;
      }
      classes = !general;
      from_rows = general;
    } else if (!learn) {
      // reference ChangeBeta (src/MutationTree.hpp:345-351)
      float nb = __fadd_rn(beta, raw.beta_jump);
      if (nb < 0.0f) nb = fabsf(nb);
      if (nb > 1.0f) nb = __fsub_rn(nb, __fmul_rn(2.0f, __fsub_rn(nb, 1.0f)));
      pbeta = nb;
      beta_terms(ds, pbeta, PL.l01, PL.l11, pprior);
    } else {
      rates = propose_rates(ds, md, alpha, beta, ec, raw, lane);
      palpha = rates.palpha;
      pbeta = rates.pbeta;
      pprior = rates.pprior;
      PL = rates.PL;
    }
    if (classes) {
      delta = move_classes<W32>(mp, related, D, C);
      nc = list_nodes<W32>(C, list, lane, nv);
      if constexpr (COUNTS) {
        const int2 km = scan_counts<W32, Q>(tab, &ds, L, chunks, wpc, wic, lane,
                                            list, nc, nv, delta);
        ev = finish_max(ds, L, prior, km.x, km.y, wpc, wic, lane, part, i & 1);
      } else if constexpr (CODES) {
        int sk = 0, sm = 0;
        // CH chunks of cells from chunk c on
        auto read_off = [&](auto CHT, int c) {
          constexpr int CH = decltype(CHT)::value;
          Packed<NW> pv[CH], pw[CH];
          uint32_t best[CH * NW];
#pragma unroll
          for (int k = 0; k < CH; k++)
            class_deltas<W32, Q>(tab.chunk(c + k, n), delta, lane, pv[k], pw[k]);
          scan_codes<W32, Q, CH>(tab.chunk(c, n), n, C, list, nv, nc, pv, pw,
                                 lane, best);
#pragma unroll
          for (int k = 0; k < CH; k++)
#pragma unroll
            for (int q = 0; q < Q; q++) {
              const uint32_t T = (best[k * NW + (q >> 1)] >> (16 * (q & 1))) & 0xFFFFu;
              int d, m;
              decode<(W32 > 4)>(code, T, d, m);
              sk += d + m;
              sm += m;
            }
          dv = pv[0];  // (kept for accepted proposals of one chunk)
          dw = pw[0];
        };
        int c = 0;
        for (; c + 2 <= chunks; c += 2) read_off(IntConst<2>{}, c);
        if (c < chunks) read_off(IntConst<1>{}, c);
        sk = __reduce_add_sync(BBS_FULL_MASK, sk);
        sm = __reduce_add_sync(BBS_FULL_MASK, sm);
        ev = finish_max(ds, L, prior, sk, sm, wpc, wic, lane, part, i & 1);
        if (!code.exact) {
          // the codes' choice is within the margin per cell of the
          // reference's: enough to reject, otherwise score the rows
          const float tol = fmaf((float)ds.n_cells, code.margin,
                                 fabsf(ev.score) * 1.0e-6f + 1.0e-3f);
          const float up = ev.score + tol;
          from_rows = !(trace == nullptr && md.gamma > 0.0f && has_best &&
                        up < best_score &&
                        corr * expf((up - score) * md.gamma) * 1.001f <
                            raw.acceptance_level);
        }
      } else {
        // Where the bound rejects less than a sixth of the proposals it is left
        // out for a while: it costs about a tenth of the exact sum (few cells,
        // flat likelihoods.  1000 steps of 750 Langevin chains, left out below
        // a third and below a sixth: 67 x 9 6.78, 6.38 ms; 100 x 16 8.39, 7.41;
        // 127 x 32 9.13, 8.15).
        const bool bound = trace == nullptr && md.gamma > 0.0f && has_best &&
                           skip == 0;
        if (skip > 0) skip--;
        float up[2] = {0.0f, 0.0f};
        class_deltas<W32, Q>(tab, delta, lane, dv, dw);
        if (bound)
          bound_proposal<W32, Q>(tab, delta, list, nv, nc, cs, L, eps, c0,
                                 stride, ds.n_cells, lane, up);
        if (bound) {
          if ((++bounded & 31) == 0) {
            if (rejected < 5) skip = 96;
            rejected = 0;
          }
          if (multi) {
            float *pp = reinterpret_cast<float *>(part + (i & 1) * 12 * wpc);
            if (lane == 0) {
              pp[12 * wic] = up[0];
              pp[12 * wic + 1] = up[1];
            }
            __syncthreads();
            up[0] = up[1] = 0.0f;
            for (int w = 0; w < wpc; w++) {
              up[0] += pp[12 * w];
              up[1] += pp[12 * w + 1];
            }
          }
          const float tol = slack + fabsf(score) * 4.8e-07f +
                            fabsf(smax) * 4.8e-07f + 1.0e-3f;
          const float ds_up = fmaf(up[0], kLn2 / kBoundUnit, tol);
          const float dm_up = fmaf(up[1], kLn2 / kBoundUnit, tol);
          if (smax + dm_up < best_score &&
              corr * expf(ds_up * md.gamma) * 1.001f < raw.acceptance_level) {
            __syncwarp();
            rejected++;
            i++;
            continue;  // rejected: the chain's state stays as it is
          }
        }
        from_table = true;
        order = prop;
      }
    } else if (SUM && err_move && tree_ok) {
      from_table = true;
      if (!ord_ok) order = cur;
    } else if (COUNTS && err_move && tree_ok) {
      if constexpr (COUNTS) {
        const int2 km = scan_counts<W32, Q>(tab, &ds, PL, chunks, wpc, wic,
                                            lane, list, 0, 0, delta);
        ev = finish_max(ds, PL, pprior, km.x, km.y, wpc, wic, lane, part, i & 1);
      }
    } else if (!fresh) {
      from_rows = true;
    }
    if (classes ? (SUM || from_rows) : (from_rows && !err_move)) {
      if constexpr (SUM)
        propose_tree<W32>(cur, prop, cpar, ppar, n, mp, D, related, tree_ok,
                          wpc, wic, lane);
      else  // (rarely: out of line)
        propose_tree_call<W32>(cur, prop, cpar, ppar, n, mp, D, related,
                               tree_ok, wpc, wic, lane);
      built = true;
    }
    if constexpr (SUM) {
      if (classes) {
        apply_classes<W32, Q>(tab, list, nc, nv, delta, dv, dw, false, lane);
        applied = true;
      }
    }
    if (order != nullptr && (SUM || ss.sx.inc != nullptr))
      canonical_order<W32>(order, n, fresh ? cpar : nullptr, ss.sx.ord,
                           ss.sx.hist, lane);
    if (fresh) {
      const int off = CODES ? code.off : 0, wd = CODES ? -code.s * code.P : 1,
                wm = CODES ? code.s * code.Q : 256;
      if (ss.sx.inc != nullptr)
        fill_table_inherit<Q>(ss.sx, n, lane, off, wd, wm);
      else
        fill_table<W32, Q>(cur, &ds, tab, chunks, wpc, wic, lane, off, wd, wm);
    }
    if constexpr (SUM) {
      if (from_table) {
        long long acc[6] = {0, 0, 0, 0, 0, 0};
        sum_cells_table<W32, Q>(tab, ss.sx.ord, n, pd, pm, PL, c0, stride, lane,
                                ds.n_cells, acc, pcs);
        acc[0] = warp_sum_ll(acc[0]);
        acc[2] = warp_sum_ll(acc[2]);
        acc[4] = warp_sum_ll(acc[4]);
        acc[5] = warp_sum_ll(acc[5]);
        ev = finish_sum(ds, pprior, acc, wpc, wic, lane, part, i & 1);
      }
    }
    if (fresh) {
      ord_ok = true;
      if constexpr (SUM) {
        cs = pcs;
        smax = ev.smax;
        if (multi) __syncthreads();  // step i writes the same partial sums
      }
      continue;
    }
    if (from_rows)
      ev = evaluate_rows<W32, Q, SUM>(err_move ? cur : prop, &ds, PL, pprior,
                                      wpc, wic, lane, part, i & 1, ss.sx);
    if (order != nullptr || from_rows) ord_ok = order == cur && !from_rows;
    const float pscore = ev.score, psmax = ev.smax;
    bool accept;
    if (err_move && learn) {
      accept = accept_rates(ds, md, rates, alpha, beta, score, pscore, ev.e,
                            raw.acceptance_level, lane);
      err_prop++;
      if (accept) err_acc++;
    } else {
      // src/Application.hpp:452-455
      const float ratio = __fmul_rn(
          corr, expf(__fmul_rn(__fsub_rn(pscore, score), md.gamma)));
      accept = ratio > raw.acceptance_level;
      if (err_move) {
        err_prop++;
        if (accept) err_acc++;
      }
    }
    // src/Application.hpp:456 and the co-optimal list, as in run_chain
    const bool better = !has_best || psmax > best_score;
    const bool tie = !better && K > 1 && psmax == best_score &&
                     lcount < (uint32_t)K;
    if constexpr (!SUM)
      if (!err_move && !built && (accept || better || tie))
        propose_tree<W32>(cur, prop, cpar, ppar, n, mp, D, related, tree_ok,
                          wpc, wic, lane);
    const uint32_t *scored_rows = err_move ? cur : prop;
    if (better) {
      has_best = true;
      best_score = psmax;
      best_alpha = palpha;
      best_beta = pbeta;
      bsk = ev.sk;
      bsm = ev.sm;
      copy_rows_part<W32>(scored_rows, gbest, n, wpc, wic, lane);
      if (K > 1) {
        const uint64_t h = tree_hash<W32>(scored_rows, n, lane);
        if (multi) __syncthreads();  // before the rows are written again
        if (wic == 0 && lane == 0) {
          lhash[0] = h;
          lbeta[0] = pbeta;
        }
        lcount = 1;
      }
    } else if (tie) {
      const uint64_t h = tree_hash<W32>(scored_rows, n, lane);
      const bool seen =
          __any_sync(BBS_FULL_MASK, lane < (int)lcount && lhash[lane] == h);
      if (multi) __syncthreads();  // before rows or list are written again
      if (!seen) {
        copy_rows_part<W32>(scored_rows,
                            gbest + (size_t)lcount * n * rs_of_w32(W32), n, wpc,
                            wic, lane);
        if (wic == 0 && lane == 0) {
          lhash[lcount] = h;
          lbeta[lcount] = pbeta;
        }
        lcount++;
      }
    }
    if (trace != nullptr && wic == 0 && lane == 0) {
      bbs_step_trace *t = trace + i;
      t->move = raw;
      t->proposed_score = pscore;
      t->current_score = accept ? pscore : score;
      t->proposed_beta = pbeta;
      t->accepted = accept ? 1u : 0u;
      t->proposed_alpha = palpha;
      t->proposed_max_score = psmax;
#pragma unroll
      for (int k = 0; k < 2; k++) t->reserved[k] = 0;
#pragma unroll
      for (int k = 0; k < 4; k++)
        t->proposed_counts[k] = SUM ? 0ull : (uint64_t)ev.e[k];
    }
    if (accept) {
      alpha = palpha;
      beta = pbeta;
      score = pscore;
      prior = pprior;
      L = PL;
#pragma unroll
      for (int k = 0; k < 4; k++) ec[k] = ev.e[k];
      csk = ev.sk;
      csm = ev.sm;
      smax = psmax;
      if (!err_move) {
        uint32_t *t = cur;
        cur = prop;
        prop = t;
        uint8_t *tp = cpar;
        cpar = ppar;
        ppar = tp;
        if (classes) {
          if constexpr (!SUM) {
            for (int c = 0; c < chunks; c++) {
              const Table<W32, Q> tc = tab.chunk(c, n);
              if (COUNTS || chunks > 1)
                class_deltas<W32, Q>(tc, delta, lane, dv, dw);
              apply_classes<W32, Q>(tc, list, nc, nv, delta, dv, dw, false,
                                    lane);
            }
          } else {
            cs = pcs;
            ord_ok = true;
          }
#ifdef BBS_CHECKED
          device_check(parents_match_rows<W32>(cur, n, cpar, lane), status,
                       kCheckParent, (uint32_t)raw.move_type, 4u);
#endif
        } else {
          fresh_rows = fresh_table = true;
        }
      } else if (tree_ok) {
        if constexpr (SUM) {
          cs = pcs;
          tolerances();
        } else {
          fresh_table = CODES;
        }
      }
    } else if (applied) {
      take_back<W32, Q>(tab, list, delta, C, dv, dw, lane);
    }
    __syncwarp();
    i++;
  }
  copy_rows_part<W32>(cur, g, n, wpc, wic, lane);
  if (wic == 0 && lane == 0) {
    ChainState o = st;
    o.alpha = alpha;
    o.beta = beta;
    o.score = score;
    o.prior = prior;
    o.l00 = L.l00;
    o.l10 = L.l10;
    o.l01 = L.l01;
    o.l11 = L.l11;
#pragma unroll
    for (int k = 0; k < 4; k++) o.ec[k] = ec[k];
    o.sk = csk;
    o.sm = csm;
    o.has_best = has_best ? 1u : 0u;
    o.best_alpha = best_alpha;
    o.best_beta = best_beta;
    o.best_score = best_score;
    o.best_sk = bsk;
    o.best_sm = bsm;
    o.steps_done = st.steps_done + (uint64_t)i;
    o.err_proposed = err_prop;
    o.err_accepted = err_acc;
    o.list_count = lcount;
    *gstate = o;
    if (cancelled && status != nullptr) atomicOr(status, 1);
  }
  if (multi) __syncthreads(); else __syncwarp();
}

// A warp's table in a slot of rows of five to eight words, its nodes from ns
// on in global memory (`table`, a part per slot of the launch and warp).
template <int W32, int Q>
__device__ __forceinline__ Table<W32, Q> wide_table(uint8_t *slot_base, int n,
                                                    int rs, int wpc, int wic,
                                                    int chunks, int ns,
                                                    uint32_t *table,
                                                    int slot) {
  uint8_t *p = slot_base + slot_bytes(n, rs, wpc, true, W32, Q, false) +
               wic * wide_part_bytes(Q, chunks, ns);
  return Table<W32, Q>{reinterpret_cast<uint32_t *>(p),
                       table + (size_t)(slot * wpc + wic) * chunks *
                                   (pack_table_bytes(n - ns, Q) / 4),
                       ns};
}

// Launch bounds of each variant (bbs_layout.h).
template <int W32, int Q, int TAB>
struct ChainBounds {
  static constexpr int threads = chain_max_threads(Q);
  static constexpr int min_blocks = chain_blocks(W32, Q, TAB != 0);
};

// One dataset: chains 0..n_chains-1, one warp per chain (blocks of `cpb`
// chains) or wpc warps per chain (the block is one chain).  REC: recorded
// moves and/or a step trace (replays and tests); without them the move and
// trace paths compile away.
// TAB: 1 or 2, proposals are read off a table (a.chunks > 0), of counts for 2;
// 0, every node is evaluated.  Kernels of their own, so that none carries
// another's code and registers (with codes and counts in one, 20 x 24 took 11 %
// longer and 63 x 64 4 %).
template <int W32, int Q, bool SUM, bool REC, int TAB>
__global__ void __launch_bounds__((ChainBounds<W32, Q, TAB>::threads),
                                  (ChainBounds<W32, Q, TAB>::min_blocks))
    mcmc_kernel(const RunArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  const int wpc = a.wpc;
  const int cpb = wpb / wpc;
  const int slot = wib / wpc, wic = wib - slot * wpc;
  const int n = a.ds.n_nodes;
  // the launcher's plan, for the whole block
  const bool inc = a.with_inc != 0, ring = W32 > 4 && TAB == 0;
  constexpr bool wide = W32 > 4 && TAB != 0;
  constexpr bool scratch = SUM || W32 > 4 || TAB != 0;
  const int sb =
      wide ? wide_slot_bytes(n, RS, wpc, W32, Q, a.chunks, a.ns)
      : TAB != 0 && !inc ? table_slot_bytes(n, RS, wpc, W32, Q, a.chunks)
                    : slot_bytes(n, RS, wpc, scratch, W32, Q, inc || ring);
  uint8_t *slot_base = reinterpret_cast<uint8_t *>(smem) + (size_t)slot * sb;
  uint32_t *buf0 = reinterpret_cast<uint32_t *>(slot_base);
  uint32_t *buf1 = buf0 + n * RS;
  int *part = reinterpret_cast<int *>(buf0 + 2 * n * RS);
  volatile int *sflag = part + 24 * wpc;
  uint4 *pbuf = reinterpret_cast<uint4 *>(
      slot_base + 4 * (2 * n * RS + 24 * wpc + 4) + kPhiloxBytes * wic);
  SlotSum ss{};
  if (scratch) ss = slot_sum(slot_base, n, RS, wpc, wic, W32, Q, inc || ring);
  Table<W32, Q> tab{};
  if constexpr (TAB != 0) {
    if constexpr (wide) {
      tab = wide_table<W32, Q>(slot_base, n, RS, wpc, wic, a.chunks, a.ns,
                               a.table, blockIdx.x * cpb + slot);
    } else {
      if (inc) {
        uint8_t *table = reinterpret_cast<uint8_t *>(smem) + (size_t)cpb * sb;
        build_increments<Q>(table, wpc, a.ds, RS);
        __syncthreads();
        ss.sx.inc = reinterpret_cast<const uint32_t *>(
            table + (size_t)wic * inc_table_bytes(n, Q));
      } else {
        ss.sx.cnt = table_part(slot_base, n, RS, wpc, wic, W32, Q, a.chunks);
      }
      tab = Table<W32, Q>{ss.sx.cnt, nullptr, n};
    }
  }
  for (int chain = blockIdx.x * cpb + slot; chain < a.n_chains;
       chain += gridDim.x * cpb) {
    const bbs_raw_move *moves = nullptr;
    bbs_step_trace *trace = nullptr;
    if constexpr (REC) {
      if (a.moves != nullptr) moves = a.moves + (size_t)chain * a.n_steps;
      if (a.trace != nullptr) trace = a.trace + (size_t)chain * a.n_steps;
    }
    const int K = a.list_hash != nullptr ? a.md.treelist : 1;
    uint32_t *rows = a.rows + (size_t)chain * n * RS;
    uint32_t *best = a.best_rows + (size_t)chain * K * n * RS;
    uint64_t *lhash = K > 1 ? a.list_hash + (size_t)chain * K : nullptr;
    float *lbeta = K > 1 ? a.list_beta + (size_t)chain * K : nullptr;
    if constexpr (TAB != 0)
      run_chain_table<W32, Q, SUM, TAB == 2>(
          a.ds, a.md, (uint32_t)chain, rows, best, lhash, lbeta, K,
          a.states + chain, moves, trace, a.n_steps, a.cancel, a.status, buf0,
          buf1, part, sflag, pbuf, ss, tab, a.chunks, wpc, wic, lane);
    else
      run_chain<W32, Q, SUM>(a.ds, a.md, (uint32_t)chain, rows, best, lhash,
                             lbeta, K, a.states + chain, moves, trace,
                             a.n_steps, a.cancel, a.status, buf0, buf1, part,
                             sflag, pbuf, ss, wpc, wic, lane);
  }
}

// One work unit of the batched launch: chain `chain` of dataset `d`, run
// by the wpc warps of its slot (warp wic of them).
template <int W32, int Q, bool SUM, int TAB>
__device__ __forceinline__ void batch_unit(const BatchArgs &b,
                                           const DatasetDev &ds,
                                           const ModelDev &md, uint32_t chain,
                                           uint32_t d, uint32_t *buf0,
                                           int *part, volatile int *sflag,
                                           uint4 *pbuf, const SlotSum &ss,
                                           const Table<W32, Q> &slot_tab,
                                           int wpc, int wic, int lane) {
  constexpr int RS = rs_of_w32(W32);
  // the dataset's node count is within this launch's row width
  uint32_t *buf1 = buf0 + ds.n_nodes * RS;
  const uint64_t off = b.chain_off[chain];
  // Philox key: the chain's number within its dataset, so a dataset's
  // chains draw the same moves here as in a one-dataset run.
  const uint32_t local = chain - d * (uint32_t)b.chains_per_dataset;
  if constexpr (TAB != 0) {
    // (this dataset's chunks and nodes: a launch's largest dataset sizes the
    // slots)
    const int span = 32 * wpc * Q;
    Table<W32, Q> tab = slot_tab;
    tab.ns = min(tab.ns, ds.n_nodes);
    run_chain_table<W32, Q, SUM, TAB == 2>(
        ds, md, local, b.rows + off, b.best_rows + off, nullptr, nullptr, 1,
        b.states + chain, nullptr, nullptr, b.n_steps, b.cancel, b.status, buf0,
        buf1, part, sflag, pbuf, ss, tab, (ds.n_cells + span - 1) / span, wpc,
        wic, lane);
  } else {
    run_chain<W32, Q, SUM>(ds, md, local, b.rows + off, b.best_rows + off,
                           nullptr, nullptr, 1, b.states + chain, nullptr,
                           nullptr, b.n_steps, b.cancel, b.status, buf0, buf1,
                           part, sflag, pbuf, ss, wpc, wic, lane);
  }
}

// Many datasets: warps take chains from a shared work list (costliest
// first); each chain brings its own dataset and rules.  One warp per chain
// (blocks of one-warp slots), or wpc warps per chain (the block is one
// slot and takes its chains together).
// MULTI: chains of b.wpc > 1 warps; without it every chain is one warp,
// known at compile time.
template <int W32, int Q, bool SUM, bool MULTI, int TAB>
__global__ void __launch_bounds__((ChainBounds<W32, Q, TAB>::threads),
                                  (W32 > 4 ? 1
                                           : ChainBounds<W32, Q, TAB>::min_blocks))
    batch_kernel(const BatchArgs b) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int wpc = MULTI ? b.wpc : 1;
  const int slot = wib / wpc, wic = wib - slot * wpc;
  // the host's plan, the same in every thread
  const bool inc = b.with_inc != 0, ring = W32 > 4 && TAB == 0;
  constexpr bool wide = W32 > 4 && TAB != 0;
  constexpr bool scratch = SUM || W32 > 4 || TAB != 0;
  const int sb =
      wide ? wide_slot_bytes(b.max_nodes, RS, wpc, W32, Q, b.chunks, b.ns)
      : TAB != 0 && !inc
          ? table_slot_bytes(b.max_nodes, RS, wpc, W32, Q, b.chunks)
          : slot_bytes(b.max_nodes, RS, wpc, scratch, W32, Q, inc || ring);
  uint8_t *slot_base = reinterpret_cast<uint8_t *>(smem) + (size_t)slot * sb;
  uint32_t *buf0 = reinterpret_cast<uint32_t *>(slot_base);
  int *part = reinterpret_cast<int *>(buf0 + 2 * b.max_nodes * RS);
  volatile int *sflag = part + 24 * wpc;
  // the slot's next unit, shared by its warps (the flag words' second)
  volatile unsigned int *sunit =
      reinterpret_cast<volatile unsigned int *>(sflag + 1);
  uint4 *pbuf = reinterpret_cast<uint4 *>(
      slot_base + 4 * (2 * b.max_nodes * RS + 24 * wpc + 4) +
      kPhiloxBytes * wic);
  SlotSum ss{};
  if (scratch)
    ss = slot_sum(slot_base, b.max_nodes, RS, wpc, wic, W32, Q, inc || ring);
  Table<W32, Q> tab{};
  if constexpr (TAB != 0) {
    if constexpr (wide) {
      tab = wide_table<W32, Q>(
          slot_base, b.max_nodes, RS, wpc, wic, b.chunks, b.ns, b.table,
          blockIdx.x * ((blockDim.x >> 5) / wpc) + slot);
    } else {
      if (inc) {
        // the increment table of the launch's one dataset
        uint8_t *table = reinterpret_cast<uint8_t *>(smem) +
                         (size_t)((blockDim.x >> 5) / wpc) * sb;
        const DatasetDev &tds = b.ds[b.table_ds];
        build_increments<Q>(table, wpc, tds, RS);
        __syncthreads();
        ss.sx.inc = reinterpret_cast<const uint32_t *>(
            table + (size_t)wic * inc_table_bytes(tds.n_nodes, Q));
      } else {
        ss.sx.cnt = table_part(slot_base, b.max_nodes, RS, wpc, wic, W32, Q,
                               b.chunks);
      }
      tab = Table<W32, Q>{ss.sx.cnt, nullptr, b.max_nodes};
    }
  }
  for (;;) {
    unsigned int unit = 0;
    if constexpr (!MULTI) {
      if (lane == 0) unit = atomicAdd(b.next_unit, 1u);
      unit = __shfl_sync(BBS_FULL_MASK, unit, 0);
    } else {
      // the block's warps take each unit together (the previous unit's
      // reads of *sunit ended before the first barrier)
      __syncthreads();
      if (threadIdx.x == 0) *sunit = atomicAdd(b.next_unit, 1u);
      __syncthreads();
      unit = *sunit;
    }
    if (unit >= (unsigned int)b.n_units) break;
    const uint32_t chain = b.units[unit];
    if (!device_check(chain < (uint32_t)b.n_chains, b.status, kCheckUnit, chain,
                      (uint32_t)b.n_chains))
      continue;
    const uint32_t d = b.chain_ds[chain];
    if (!device_check(d < (uint32_t)b.n_datasets, b.status, kCheckDataset, d,
                      (uint32_t)b.n_datasets))
      continue;
    // The sum score reads the dataset and model tables in place (fewer
    // registers, measured faster); the max score keeps register copies
    // (measured faster there).
    if constexpr (SUM) {
      batch_unit<W32, Q, SUM, TAB>(b, b.ds[d], b.md[d], chain, d, buf0, part,
                              sflag, pbuf, ss, tab, wpc, wic, lane);
    } else {
      const DatasetDev ds = b.ds[d];
      const ModelDev md = b.md[d];
      batch_unit<W32, Q, SUM, TAB>(b, ds, md, chain, d, buf0, part, sflag, pbuf,
                              ss, tab, wpc, wic, lane);
    }
  }
}

// Initial chain states: each chain's tree evaluated at (alpha_mean,
// beta_mean); one warp per chain.
template <int W32, int Q, bool SUM>
__global__ void __launch_bounds__(128) init_kernel(const InitArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  const int idx = blockIdx.x * wpb + wib;
  if (idx >= a.n_chains) return;  // whole warp
  const int chain = a.chain_list != nullptr ? (int)a.chain_list[idx] : idx;
  const uint32_t d = a.chain_ds != nullptr ? a.chain_ds[chain] : 0u;
  const DatasetDev ds = a.ds[d];
  const ModelDev md = a.md[d];
  const int n = ds.n_nodes;
  const uint64_t off = a.chain_off != nullptr ? a.chain_off[chain]
                                              : (uint64_t)chain * n * RS;
  // per warp: the tree's rows, then (sum score) the canonical order and
  // its histogram
  const int wb = 4 * a.max_nodes * RS +
                 (SUM ? align16(2 * a.max_nodes) + align16(4 * 32 * ((a.max_nodes + 31) / 32)) : 0);
  uint8_t *mine = reinterpret_cast<uint8_t *>(smem) + (size_t)wib * wb;
  uint32_t *rows = reinterpret_cast<uint32_t *>(mine);
  SumCtx sx{};
  if constexpr (SUM) {
    sx.ord = reinterpret_cast<uint16_t *>(mine + 4 * a.max_nodes * RS);
    sx.hist = reinterpret_cast<int *>(mine + 4 * a.max_nodes * RS + align16(2 * a.max_nodes));
  }
  copy_rows<W32>(a.rows + off, rows, n, lane);
  __syncwarp();
  const float *tm = a.terms + 8 * (size_t)d;
  const LogTable L{tm[2], tm[3], tm[4], tm[5]};
  const float alpha = tm[0], beta = tm[1], prior = tm[6];
  const Evaluated ev = evaluate<W32, Q, SUM>(rows, n, ds, L, prior, 1, 0, lane,
                                             nullptr, 0, sx);
  if (lane == 0) {
    ChainState o;
    o.alpha = alpha;
    o.beta = beta;
    o.score = ev.score;
    o.prior = prior;
    o.l00 = L.l00;
    o.l10 = L.l10;
    o.l01 = L.l01;
    o.l11 = L.l11;
#pragma unroll
    for (int k = 0; k < 4; k++) o.ec[k] = ev.e[k];
    o.sk = ev.sk;
    o.sm = ev.sm;
    o.has_best = 0;
    o.best_alpha = alpha;
    o.best_beta = beta;
    o.best_score = -INFINITY;
    o.best_sk = 0;
    o.best_sm = 0;
    o.steps_done = 0;
    o.err_proposed = 0;
    o.err_accepted = 0;
    o.list_count = 0;
    for (int k = 0; k < 7; k++) o.pad[k] = 0;
    a.states[chain] = o;
  }
}

__device__ __forceinline__ void write_score(const ScoreArgs &a, int tree,
                                            int sk, int sm, const LogTable &L,
                                            float prior) {
  const float s = tree_score(a.ds, sk, sm, L, prior);
  if (a.scores) a.scores[tree] = s;
  if (a.counts) {
    int N[4];
    class_totals(a.ds, sk, sm, N);
    for (int q = 0; q < 4; q++) a.counts[4 * (size_t)tree + q] = (uint64_t)N[q];
  }
}

// Shared memory of score_walk_kernel: the rows, parents, order and depth
// histogram (n ints and the node -> position map fit it), then each warp's
// ring and gene table.
struct WalkLayout {
  int par, ord, hist, warps, per_warp;
  __host__ __device__ WalkLayout(int n, int rs) {
    par = 4 * n * rs;
    ord = par + align16(n);
    hist = ord + align16(2 * n);
    warps = hist + align16(4 * 32 * ((n + 31) / 32));
    per_warp = align16(ring_bytes(2)) + align16(gene_table_bytes(n, 2));
  }
  __host__ __device__ int bytes(int n_warps) const {
    return warps + n_warps * per_warp;
  }
};

// Scores of many trees by masked popcounts, one warp per tree: rows of up to
// four words with few nodes or cells, where finding the parents and the order
// of a walk would cost as much as it saves.
template <int W32, int Q, bool ATTACH>
__global__ void __launch_bounds__(128) score_kernel(const ScoreArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  const int tree = blockIdx.x * wpb + wib;
  if (tree >= a.n_trees) return;  // whole warp
  const int n = a.ds.n_nodes;
  uint32_t *rows = smem + (size_t)wib * n * RS;
  copy_rows<W32>(a.rows + (size_t)tree * n * RS, rows, n, lane);
  __syncwarp();
  const float *bt = a.beta_terms + 4 * (size_t)tree;
  const LogTable L{a.ds.l00, a.ds.l10, bt[1], bt[2]};
  const float prior = bt[3];
  Cells<W32, Q> cb;
  int k = 0, m = 0;
  for (int c0 = 0; c0 < a.ds.n_cells; c0 += 32 * Q) {
    load_cells<W32, Q>(cb, a.ds, c0, 32, lane);
    int bj[Q];
    best_nodes<W32, Q>(rows, n, cb, L.l00, L.l01, L.l10, L.l11, a.ds.neg_zero,
                          bj);
    counts_at<W32, Q>(rows, cb, bj, k, m);
    if constexpr (ATTACH) {
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int c = c0 + 32 * q + lane;
        if (c < a.ds.n_cells)
          a.attach[(size_t)tree * a.ds.n_cells + c] = (uint32_t)bj[q];
      }
    }
  }
  const int sk = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)k);
  const int sm = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)m);
  if (lane == 0) {
    write_score(a, tree, sk, sm, L, prior);
  }
}

// Scores of few trees: one block per tree, its warps split the chunks of 32
// cells and, four ways, the nodes, so that a call for one tree waits for some
// 25 nodes' latency instead of all nodes of two chunks (kernel time of one tree
// at 95 x 96: 20.5 -> 5.6 us; at 255 x 512 the call went from 434 to 98 us).
inline constexpr int kFewRanges = 4, kFewGroups = 4;

template <int W32, bool ATTACH>
__global__ void __launch_bounds__(32 * kFewRanges * kFewGroups)
    score_few_kernel(const ScoreArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32);
  __shared__ float part_s[kFewGroups][kFewRanges][32];
  __shared__ int part_j[kFewGroups][kFewRanges][32];
  __shared__ int sums[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = warp / kFewRanges, range = warp % kFewRanges;
  const int n = a.ds.n_nodes, tree = blockIdx.x;
  const uint32_t *src = a.rows + (size_t)tree * n * RS;
  for (int i = threadIdx.x; i < n * RS; i += blockDim.x) smem[i] = src[i];
  if (threadIdx.x < 2) sums[threadIdx.x] = 0;
  __syncthreads();
  const float *bt = a.beta_terms + 4 * (size_t)tree;
  const LogTable L{a.ds.l00, a.ds.l10, bt[1], bt[2]};
  const int j0 = n * range / kFewRanges, j1 = n * (range + 1) / kFewRanges;
  int k = 0, m = 0;
  for (int base = 0; base < a.ds.n_cells; base += 32 * kFewGroups) {
    const int c0 = base + 32 * group;
    Cells<W32, 1> cb;
    load_cells<W32, 1>(cb, a.ds, c0, 32, lane);
    if (j0 < j1) {
      float best[1];
      int bj[1];
      best_nodes_of<W32, 1>(smem, j0, j1, cb, L.l00, L.l01, L.l10, L.l11,
                            a.ds.neg_zero, best, bj);
      part_s[group][range][lane] = best[0];
      part_j[group][range][lane] = bj[0];
    } else {
      part_j[group][range][lane] = -1;  // fewer nodes than ranges
    }
    __syncthreads();
    if (range == 0) {
      // the first maximum: ranges are in node order, an equal score later on
      // does not win
      float best = 0.0f;
      int bj[1] = {-1};
#pragma unroll
      for (int r = 0; r < kFewRanges; r++) {
        const int j = part_j[group][r][lane];
        const float s = part_s[group][r][lane];
        if (j >= 0 && (bj[0] < 0 || s > best)) {
          best = s;
          bj[0] = j;
        }
      }
      counts_at<W32, 1>(smem, cb, bj, k, m);
      if constexpr (ATTACH) {
        const int c = c0 + lane;
        if (c < a.ds.n_cells)
          a.attach[(size_t)tree * a.ds.n_cells + c] = (uint32_t)bj[0];
      }
    }
    __syncthreads();  // the partial results are written again
  }
  k = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)k);
  m = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)m);
  if (range == 0 && lane == 0) {
    atomicAdd(&sums[0], k);
    atomicAdd(&sums[1], m);
  }
  __syncthreads();
  if (threadIdx.x == 0) write_score(a, tree, sums[0], sums[1], L, bt[3]);
}

// The parents of the tree with ancestor rows `rows` -- the deepest proper
// ancestors -- by `threads` threads, a warp's or a block's: whether this
// thread's nodes agree with them (rows that are not a tree's do not).
template <int W32>
__device__ __forceinline__ bool walk_parents(const uint32_t *rows, int n,
                                             uint8_t *par, int *hist, int id,
                                             int threads) {
  constexpr int RS = rs_of_w32(W32);
  for (int x = id; x < n; x += threads) {
    uint32_t r[W32];
    ld_row<W32>(rows + x * RS, r);
    int pc = 0;
#pragma unroll
    for (int k = 0; k < W32; k++) pc += __popc(r[k]);
    hist[x] = pc;
  }
  if (threads > 32) __syncthreads(); else __syncwarp();
  bool ok = true;
  for (int x = id; x < n; x += threads) {
    uint32_t r[W32], q[W32];
    ld_row<W32>(rows + x * RS, r);
    // a tree's parent has one ancestor less
    int p = x == n - 1 ? x : -1;
#pragma unroll
    for (int k = 0; k < W32; k++) {
      uint32_t v = k == (x >> 5) ? r[k] & ~(1u << (x & 31)) : r[k];
      while (v != 0u && p < 0) {
        const int y = 32 * k + __ffs(v) - 1;
        v &= v - 1u;
        if (y < n && hist[y] == hist[x] - 1) p = y;
      }
    }
    if (p < 0) {
      ok = false;
      p = n - 1;
    }
    par[x] = (uint8_t)p;
    ld_row<W32>(rows + p * RS, q);
#pragma unroll
    for (int k = 0; k < W32; k++) {
      const uint32_t own = k == (x >> 5) ? 1u << (x & 31) : 0u;
      ok = ok && (x == n - 1 ? r[k] == own
                             : r[k] == (q[k] | own) && (q[k] & own) == 0u);
    }
  }
  return ok;
}

// The nodes with the highest codes of the lane's two cells, each node's codes
// its parent's from the ring plus its gene's (sx: the order's entries in hist,
// ring and gene table): the class sums and, with attachments, the nodes.
template <bool ATTACH>
__device__ __forceinline__ void walk_codes(const SumCtx &sx,
                                           const MaxCode &code, int n,
                                           int lane, int (&bj)[2], int &k,
                                           int &m) {
  const uint32_t wd = (uint32_t)(-code.s * code.P), wm = (uint32_t)(code.s * code.Q);
  // T of both cells in one word; with attachments, keys T << 8 | 255 - j
  uint32_t best = (uint32_t)code.off * 0x10001u;
  uint32_t key0 = 0u, key1 = 0u;
  auto see = [&](uint32_t t, uint32_t o) {
    if constexpr (ATTACH) {
      const uint32_t jj = 255u - (uint32_t)ring_node(o);
      key0 = max(key0, __byte_perm(t, jj, 0x5104u));
      key1 = max(key1, __byte_perm(t, jj, 0x5324u));
    } else {
      best = __vmaxu2(best, t);
    }
  };
  auto gene = [&](uint32_t g, uint32_t o) {
    const uint32_t b = ring_gene(g, o);
    return (b & 0x00010001u) * wd + ((b >> 8) & 0x00010001u) * wm;
  };
  sx.ring[32 + lane] = best;
  see(best, (uint32_t)(n - 1) >> 3 << 23 | ((uint32_t)(n - 1) & 7u));
  int i = 1;
#pragma unroll 2
  for (; i + 1 < n; i += 2) {
    const uint2 o = ring_pair(sx, i);
    uint32_t g0, g1;
    const uint32_t a0 = ring_counts(sx, o.x, lane, g0);
    const uint32_t a1 = ring_counts(sx, o.y, lane, g1);
    const uint32_t t0 = a0 + gene(g0, o.x);
    const uint32_t t1 = ((o.y & 32u) ? t0 : a1) + gene(g1, o.y);
    const uint32_t at = (uint32_t)(i + 1) * 32u & (kRingBytes / 4 - 32u);
    sx.ring[at + lane] = t0;
    sx.ring[at + 32 + lane] = t1;
    see(t0, o.x);
    see(t1, o.y);
  }
  if (i < n) {
    const uint32_t o = (uint32_t)sx.hist[i - 1];
    uint32_t g;
    const uint32_t t = ring_counts(sx, o, lane, g);
    see(t + gene(g, o), o);
  }
#pragma unroll
  for (int q = 0; q < 2; q++) {
    int d, mm;
    if constexpr (ATTACH) {
      const uint32_t key = q ? key1 : key0;
      bj[q] = 255 - (int)(key & 0xFFu);
      decode<true>(code, key >> 8, d, mm);
    } else {
      decode<true>(code, (best >> (16 * q)) & 0xFFFFu, d, mm);
    }
    k += d + mm;
    m += mm;
  }
}

// Scores of many trees with rows of five to eight words: one block per tree,
// four warps over its chunks of 64 cells.  Where the rows are a tree whose
// order fits the ring and its rates have exact codes (bbs_incr.cuh), each node
// takes its parent's codes from the ring plus its gene's, some 20 instructions
// a node for 64 cells; otherwise masked popcounts, which run the
// population-count pipe at its peak (255 x 512, 1500 trees: 735 us, walked 230
// us, and another 9 us less a call with offsets in the order's entries; bound
// by the latency of the walk at three blocks per SM).
template <int W32, bool ATTACH>
__global__ void __launch_bounds__(128) score_walk_kernel(const ScoreArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32), Q = 2, WARPS = 4;
  __shared__ int sums[2], fits;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = a.ds.n_nodes, tree = blockIdx.x;
  const WalkLayout w(n, RS);
  uint8_t *base = reinterpret_cast<uint8_t *>(smem);
  uint32_t *rows = smem;
  uint8_t *par = base + w.par;
  uint16_t *ord = reinterpret_cast<uint16_t *>(base + w.ord);
  int *hist = reinterpret_cast<int *>(base + w.hist);
  uint32_t *ring = reinterpret_cast<uint32_t *>(base + w.warps + warp * w.per_warp);
  uint32_t *gt = ring + ring_bytes(Q) / 4;
  SumCtx sx{};
  sx.hist = hist;
  sx.ring = ring;
  sx.gt = gt;
  copy_rows_part<W32>(a.rows + (size_t)tree * n * RS, rows, n, WARPS, warp, lane);
  if (threadIdx.x < 2) sums[threadIdx.x] = 0;
  __syncthreads();
  const float *bt = a.beta_terms + 4 * (size_t)tree;
  const LogTable L{a.ds.l00, a.ds.l10, bt[1], bt[2]};
  bool ok = walk_parents<W32>(rows, n, par, hist, threadIdx.x, blockDim.x);
  ok = __syncthreads_and(ok);
  const MaxCode code =
      make_code(L.l00, L.l01, L.l10, L.l11, a.ds.max_d, a.ds.max_m, lane);
  ok = ok && code.usable && code.exact;
  if (ok && warp == 0) {
    const bool f = ring_order<W32>(rows, n, par, ord, hist, lane);
    if (lane == 0) fits = f ? 1 : 0;
  }
  __syncthreads();
  ok = ok && fits != 0;
  int k = 0, m = 0;
  for (int c0 = 64 * warp; c0 < a.ds.n_cells; c0 += 64 * WARPS) {
    Cells<W32, Q> cb;
    load_cells<W32, Q>(cb, a.ds, c0, 32, lane);
    int bj[Q];
    if (ok) {
      build_gene_table<W32, Q>(cb, gt, n, lane);
      walk_codes<ATTACH>(sx, code, n, lane, bj, k, m);
      __syncwarp();
    } else {
      best_nodes<W32, Q>(rows, n, cb, L.l00, L.l01, L.l10, L.l11,
                         a.ds.neg_zero, bj);
      counts_at<W32, Q>(rows, cb, bj, k, m);
    }
    if constexpr (ATTACH) {
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int c = c0 + 32 * q + lane;
        if (c < a.ds.n_cells)
          a.attach[(size_t)tree * a.ds.n_cells + c] = (uint32_t)bj[q];
      }
    }
  }
  k = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)k);
  m = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)m);
  if (lane == 0) {
    atomicAdd(&sums[0], k);
    atomicAdd(&sums[1], m);
  }
  __syncthreads();
  if (threadIdx.x == 0) write_score(a, tree, sums[0], sums[1], L, bt[3]);
}

// The same for rows of up to four words, one warp per tree (4096 trees at 95 x
// 96: the call went from 255 to 240 us, at 95 x 500 from 390 to 268 us; the
// rest is the copy of the trees).
template <int W32, bool ATTACH>
__global__ void __launch_bounds__(128) score_tree_kernel(const ScoreArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32), Q = 2;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int tree = blockIdx.x * (blockDim.x >> 5) + wib;
  if (tree >= a.n_trees) return;  // whole warp
  const int n = a.ds.n_nodes;
  const WalkLayout w(n, RS);
  uint8_t *base = reinterpret_cast<uint8_t *>(smem) + wib * w.bytes(1);
  uint32_t *rows = reinterpret_cast<uint32_t *>(base);
  uint8_t *par = base + w.par;
  uint16_t *ord = reinterpret_cast<uint16_t *>(base + w.ord);
  SumCtx sx{};
  sx.hist = reinterpret_cast<int *>(base + w.hist);
  sx.ring = reinterpret_cast<uint32_t *>(base + w.warps);
  sx.gt = sx.ring + ring_bytes(Q) / 4;
  copy_rows<W32>(a.rows + (size_t)tree * n * RS, rows, n, lane);
  __syncwarp();
  const float *bt = a.beta_terms + 4 * (size_t)tree;
  const LogTable L{a.ds.l00, a.ds.l10, bt[1], bt[2]};
  const MaxCode code =
      make_code(L.l00, L.l01, L.l10, L.l11, a.ds.max_d, a.ds.max_m, lane);
  bool ok = code.usable && code.exact;
  if (ok)
    ok = __all_sync(BBS_FULL_MASK,
                    walk_parents<W32>(rows, n, par, sx.hist, lane, 32)) &&
         ring_order<W32>(rows, n, par, ord, sx.hist, lane);
  int k = 0, m = 0;
  for (int c0 = 0; c0 < a.ds.n_cells; c0 += 32 * Q) {
    Cells<W32, Q> cb;
    load_cells<W32, Q>(cb, a.ds, c0, 32, lane);
    int bj[Q];
    if (ok) {
      build_gene_table<W32, Q>(cb, sx.gt, n, lane);
      walk_codes<ATTACH>(sx, code, n, lane, bj, k, m);
    } else {
      best_nodes<W32, Q>(rows, n, cb, L.l00, L.l01, L.l10, L.l11,
                         a.ds.neg_zero, bj);
      counts_at<W32, Q>(rows, cb, bj, k, m);
    }
    if constexpr (ATTACH) {
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int c = c0 + 32 * q + lane;
        if (c < a.ds.n_cells)
          a.attach[(size_t)tree * a.ds.n_cells + c] = (uint32_t)bj[q];
      }
    }
  }
  k = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)k);
  m = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)m);
  if (lane == 0) write_score(a, tree, k, m, L, bt[3]);
}

template <int W32>
__global__ void __launch_bounds__(128) apply_kernel(const ApplyArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  const int tree = blockIdx.x * wpb + wib;
  if (tree >= a.n_trees) return;
  const int n = a.n_nodes;
  uint32_t *rows = smem + (size_t)wib * n * RS;
  copy_rows<W32>(a.rows + (size_t)tree * n * RS, rows, n, lane);
  __syncwarp();
  const float beta = a.betas[tree];
  uint32_t Dv[W32], Dw[W32];
  bbs_move_params p;
  bool related;
  if (a.raw != nullptr) {
    const Realized R = realize_move<W32>(rows, n, beta, a.raw[tree], lane, Dv, Dw);
    p = R.p;
    related = R.related;
  } else {
    p = a.params[tree];
    p.v = min(p.v, (uint32_t)(n - 1));
    p.w = min(p.w, (uint32_t)(n - 1));
    descendant_sets<W32>(rows, n, p.v, p.w, lane, Dv, Dw);
    related = has_bit<W32>(Dw, p.v);
  }
  uint32_t *out = a.rows_out + (size_t)tree * n * RS;
  build_proposal<W32>(rows, out, n, p, Dv, Dw, related, 1, 0, lane);
  if (lane == 0) {
    if (a.params_out) a.params_out[tree] = p;
    if (a.beta_out)
      a.beta_out[tree] = p.move_type == BBS_MOVE_CHANGE_BETA ? p.new_beta : beta;
  }
}

// Sum-over-attachments score and adjoint: one block per tree, its warps over
// the chunks of 32 cells.  Per cell exp(s_j - r) is summed against r = ub -
// 72, ub >= every s_j (as in sum_cells: no term overflows), with the
// softmax-weighted sums of d and m; a cell whose maximum lies more than 80
// below r is summed again against its maximum.  An online maximum per term,
// as before, took both sides of a branch and two exponentials for most nodes
// (4096 trees at 95 x 96: 110 us, now 85 us, bound by instruction issue).  The
// expected class counts give dlogL / dtheta = sum_c sum_k E_pi[n_k] dl_k /
// dtheta.
// With posteriors a warp keeps its cells' scores in shared memory (`tile`
// floats per cell) and writes the 32 cells' rows as one contiguous piece; a
// store per lane and node went to 32 lines each (50 trees at 61 x 201: 83 ->
// 15 us).
template <int W32, bool POST>
__global__ void __launch_bounds__(256) grad_kernel(const GradArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int RS = rs_of_w32(W32);
  __shared__ float sums[8][5];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  const int n = a.ds.n_nodes, tree = blockIdx.x;
  const int tile = n | 1;  // odd: a node's 32 scores lie in 32 banks
  float *mine = reinterpret_cast<float *>(smem + n * RS) + warp * 32 * tile;
  const uint32_t *src = a.rows + (size_t)tree * n * RS;
  for (int i = threadIdx.x; i < n * RS; i += blockDim.x) smem[i] = src[i];
  __syncthreads();
  const float *tb = a.tables + 6 * (size_t)tree;
  const float l00 = tb[2], l01 = tb[3], l10 = tb[4], l11 = tb[5];
  const LogTable2 L2{dup2(l00), dup2(l01), dup2(l10), dup2(l11),
                     dup2(a.ds.neg_zero)};
  // Chunk c adds to sum c % 8, whichever warp takes it: the totals are the
  // same with any number of warps (posteriors leave room for fewer).
  for (int slot = warp; slot < 8; slot += warps) {
    float acc[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};  // lse, n00, n01, n10, n11
    for (int c0 = 32 * slot; c0 < a.ds.n_cells; c0 += 32 * 8) {
      Cells<W32, 1> cb;
      load_cells<W32, 1>(cb, a.ds, c0, 32, lane);
      const float pd = cb.pdb[0] - 8388608.0f, pm = cb.pmb[0] - 8388608.0f;
      float r = fmaf(pd, fmaxf(l00, l01), pm * fmaxf(l10, l11)) - 72.0f;
      float mx, z, ed, em;
      auto sum = [&](bool first) {
        mx = -INFINITY;
        float2 z2 = dup2(0.0f), d2 = z2, m2 = z2;
        int j = 0;
#pragma unroll 2
        for (; j + 1 < n; j += 2) {
          uint32_t ra[W32], rb[W32];
          ld_row<W32>(smem + j * RS, ra);
          ld_row<W32>(smem + (j + 1) * RS, rb);
          const float2 db = make_float2(
              __int_as_float(0x4B000000 + masked_popc<W32>(cb.D[0], ra)),
              __int_as_float(0x4B000000 + masked_popc<W32>(cb.D[0], rb)));
          const float2 mb = make_float2(
              __int_as_float(0x4B000000 + masked_popc<W32>(cb.M[0], ra)),
              __int_as_float(0x4B000000 + masked_popc<W32>(cb.M[0], rb)));
          const float2 s =
              pair_score_b2(db, mb, dup2(cb.pdb[0]), dup2(cb.pmb[0]), L2);
          mx = fmax3(mx, s.x, s.y);
          if (POST && first) {
            mine[lane * tile + j] = s.x;
            mine[lane * tile + j + 1] = s.y;
          }
          const float2 e = make_float2(expf(s.x - r), expf(s.y - r));
          const float2 bias = dup2(8388608.0f);
          z2 = fadd2(z2, e);
          d2 = ffma2(e, fsub2(db, bias), d2);
          m2 = ffma2(e, fsub2(mb, bias), m2);
        }
        z = z2.x + z2.y;
        ed = d2.x + d2.y;
        em = m2.x + m2.y;
        if (j < n) {
          uint32_t ra[W32];
          ld_row<W32>(smem + j * RS, ra);
          const int d = masked_popc<W32>(cb.D[0], ra);
          const int m = masked_popc<W32>(cb.M[0], ra);
          const float s =
              pair_score(d, m, cb.pdb[0], cb.pmb[0], l00, l01, l10, l11);
          mx = fmaxf(mx, s);
          if (POST && first) mine[lane * tile + j] = s;
          const float e = expf(s - r);
          z += e;
          ed = fmaf(e, (float)d, ed);
          em = fmaf(e, (float)m, em);
        }
      };
      sum(true);
      const bool bad = !(mx - r >= -80.0f);
      if (__any_sync(BBS_FULL_MASK, bad)) {
        if (bad) r = mx;
        sum(false);
      }
      // (against the maximum: r + log z would round a log of up to 72)
      const float lse = mx + logf(z * expf(r - mx));
      if (c0 + lane < a.ds.n_cells) {
        const float Ed = ed / z, Em = em / z;
        acc[0] += lse;
        acc[1] += pd - Ed;
        acc[2] += Ed;
        acc[3] += pm - Em;
        acc[4] += Em;
      }
      if constexpr (POST) {
        // against the maximum, where the differences of the scores are exact
        float zm = 0.0f;
        for (int j = 0; j < n; j++) {
          const float e = expf(mine[lane * tile + j] - mx);
          zm += e;
          mine[lane * tile + j] = e;
        }
        const float inv = 1.0f / zm;
        for (int j = 0; j < n; j++) mine[lane * tile + j] *= inv;
        __syncwarp();
        const int cells = min(32, a.ds.n_cells - c0);
        float *post = a.posterior + ((size_t)tree * a.ds.n_cells + c0) * n;
        // lane l starts at element l; 32 elements further is (n + l) / n cells
        int cell = 0, j = lane;
        while (j >= n) {
          j -= n;
          cell++;
        }
        for (int i = lane; i < cells * n; i += 32) {
          post[i] = mine[cell * tile + j];
          j += 32;
          while (j >= n) {
            j -= n;
            cell++;
          }
        }
        __syncwarp();
      }
    }
#pragma unroll
    for (int k = 0; k < 5; k++) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        acc[k] += __shfl_xor_sync(BBS_FULL_MASK, acc[k], off);
      if (lane == 0) sums[slot][k] = acc[k];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float t[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int w = 0; w < 8; w++)
      for (int k = 0; k < 5; k++) t[k] += sums[w][k];
    const double al = tb[0], be = tb[1];
    a.logl[tree] = t[0];
    if (a.dalpha)
      a.dalpha[tree] = (float)(-(double)t[1] / (1.0 - al) + (double)t[3] / al);
    if (a.dbeta)
      a.dbeta[tree] = (float)((double)t[2] / be - (double)t[4] / (1.0 - be));
  }
}

}  // namespace bbs
