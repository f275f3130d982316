// bbs_incr.cuh -- proposals evaluated from what they change.
//
// A tree move leaves most nodes' ancestor sets as they are; the others, two
// disjoint classes of nodes, all change by the same genes, so every cell's
// counts (d, m) change there by one constant per class and cell.  A chain
// therefore keeps a table of every node and cell of its current tree and
// reads a proposal off it:
//   - max score: the table holds integer codes that order a cell's nodes as
//     their scores do (MaxCode), 16 bits per cell; a proposal's best nodes
//     are the maxima over the unchanged nodes and the two shifted classes.
//     Where rates change often, or have no codes, it holds the counts, and a
//     proposal scores every node from them (scan_counts);
//   - sum score (rows of up to four words): the table holds the counts.  A
//     proposal is first bounded from above by the terms that move (two
//     exponentials per class and cell); only one that the bound does not
//     reject is summed, over the proposal's canonical order, term by term as
//     everywhere else.
// The rows, the parent vector and the table follow accepted moves only.
// Decisions, scores and trees are those of an evaluation of every node.
//
// Measured against evaluating every node of every proposal (GB300, 10-30 % of
// the proposals accepted): 1024 chains at 95 x 96 max score 98 -> 380 M
// chain-steps/s, sum score with Langevin error moves 121 -> 188 M; at 255 x
// 512 max score 8.0 -> 18.7 M; 128 uneven datasets of 32 chains 4.4 times as
// fast; 8 chains at 63 x 64 6.3 -> 2.0 us a step.
// What bounds it now is a step's serial chain of short dependent pieces (draw,
// descendant sets, table loads, maxima, reductions: some 4 clocks for each of
// 1,300 instructions at 1.8 warps per scheduler), and for the sum score the
// special-function unit where a proposal is summed (six exponentials for two
// nodes and three cells, 8 clocks each).
#pragma once
#include "bbs_device.cuh"

namespace bbs {

// ------------------------------------------------------------------------
// Integer codes of the max score
// ------------------------------------------------------------------------
// With fixed rates a cell's score at a node is, but for rounding, affine in
// its counts: const + c1 d + c2 m with c1 = l01 - l00 and c2 = l11 - l10 of
// opposite signs.  Two nodes compare as the ratio |c1| / |c2| compares with
// a fraction (difference of m) / (difference of d), of which only finitely
// many can occur.  Any weights with a ratio between the same two
// neighbouring fractions al/bl < |c1|/|c2| < au/bu order all nodes alike;
// their mediant P/Q is the smallest: T = s (Q m - P d) + off fits 16 bits
// (P <= 2 mmax, Q <= 2 dmax, dmax and mmax the largest counts of a cell; at
// most 4 x 127 x 127).  Different (d, m) give different T, and au Q - bu P =
// 1 turns T back into (d, m).
//   exact: no two counts of a cell lie so close that the rounding of the
//          reference-order float score could tie or swap them, so the
//          largest T is the reference's choice.  Otherwise its score is
//          within `margin` of it, and only decides what `margin` leaves no
//          doubt about.
//   usable: the codes exist at all (rates with alpha + beta = 1 or
//          non-finite logs have none).
struct MaxCode {
  int P, Q, s, au, bu, off;
  uint32_t invP, invQ;  // floor(2^32 / P) + 1: quotients of x < 2^24
  float margin;
  int ties;  // denominators up to dmax that come that close
  bool usable, exact;
};

// Neighbouring fractions al / bl < |c1| / |c2| < au / bu, found so far.
struct Neighbours {
  int al = 0, bl = 1, au = 1, bu = 0;
  int ties = 0;
  __host__ __device__ void below(int a, int b) {
    if (a * bl > al * b || (a * bl == al * b && b < bl)) {
      al = a;
      bl = b;
    }
  }
  __host__ __device__ void above(int a, int b) {
    if (a * bu < au * b || (a * bu == au * b && b < bu)) {
      au = a;
      bu = b;
    }
  }
  // the fractions with denominator b; near-ties count as below
  __host__ __device__ void denominator(int b, float a1, float a2,
                                       float margin, int mmax) {
    int a = (int)fminf(floorf((float)b * (a1 / a2)), (float)mmax);
    const float x = (float)b * a1;
    if (a < mmax && (float)(a + 1) * a2 - x <= margin) a++;
    ties += fabsf(x - (float)a * a2) > margin ? 0 : 1;
    below(a, b);
    if (a < mmax) above(a + 1, b);
  }
};

// What the log table alone says: sign, margin, whether codes can exist.
__host__ __device__ inline MaxCode code_begin(float l00, float l01, float l10,
                                              float l11, int dmax, int mmax,
                                              float &a1, float &a2) {
  MaxCode k;
  const float c1 = l01 - l00, c2 = l11 - l10;
  a1 = fabsf(c1);
  a2 = fabsf(c2);
  k.s = c1 < 0.0f && c2 > 0.0f ? 1 : -1;
  // rounding of two scores (four products and three sums each, all within
  // `big`), of c1 and c2 and of the gaps: 16 units of 2^-24 big
  const float big = dmax * fmaxf(fabsf(l00), fabsf(l01)) +
                    mmax * fmaxf(fabsf(l10), fabsf(l11));
  k.margin = big * 1.9073486e-06f;  // 2^-19: twice that
  k.usable = c1 * c2 < 0.0f && a1 > 1.0e-6f && a2 > 1.0e-6f && big < 1.0e6f;
  k.exact = a1 > k.margin && a2 > k.margin;
  return k;
}

__host__ __device__ inline void code_end(MaxCode &k, const Neighbours &f,
                                         int dmax, int mmax) {
  k.P = f.al + f.au;
  k.Q = f.bl + f.bu;
  if (k.P == 1) {  // decode divides by P > 1: the next weights in between
    k.P += f.au;
    k.Q += f.bu;
  }
  k.au = f.au;
  k.bu = f.bu;
  k.off = k.s > 0 ? k.P * dmax : k.Q * mmax;
  // neighbours in lowest terms; near-ties sorted inconsistently are not
  k.usable = k.usable && f.au * f.bl - f.al * f.bu == 1 &&
             k.P * dmax + k.Q * mmax <= 65535;
  k.ties = f.ties;
  k.exact = k.exact && f.ties == 0;
  k.invP = 0xFFFFFFFFu / (uint32_t)k.P + 1u;
  k.invQ = 0xFFFFFFFFu / (uint32_t)k.Q + 1u;
}

// The codes of a log table, the denominators spread over the lanes.
inline __device__ __noinline__ MaxCode make_code(float l00, float l01,
                                                 float l10, float l11,
                                                 int dmax, int mmax,
                                                 int lane) {
  float a1, a2;
  MaxCode k = code_begin(l00, l01, l10, l11, dmax, mmax, a1, a2);
  Neighbours f;
  if (k.usable)
    for (int b = lane + 1; b <= dmax; b += 32)
      f.denominator(b, a1, a2, k.margin, mmax);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int xa = __shfl_xor_sync(BBS_FULL_MASK, f.al, o),
              xb = __shfl_xor_sync(BBS_FULL_MASK, f.bl, o),
              ya = __shfl_xor_sync(BBS_FULL_MASK, f.au, o),
              yb = __shfl_xor_sync(BBS_FULL_MASK, f.bu, o);
    f.below(xa, xb);
    f.above(ya, yb);
  }
  f.ties = (int)__reduce_add_sync(BBS_FULL_MASK, (unsigned)f.ties);
  code_end(k, f, dmax, mmax);
  return k;
}

// The same on the host: whether a launch plans for them.
inline MaxCode make_code_host(float l00, float l01, float l10, float l11,
                              int dmax, int mmax) {
  float a1, a2;
  MaxCode k = code_begin(l00, l01, l10, l11, dmax, mmax, a1, a2);
  Neighbours f;
  if (k.usable)
    for (int b = 1; b <= dmax; b++) f.denominator(b, a1, a2, k.margin, mmax);
  code_end(k, f, dmax, mmax);
  return k;
}

// (d, m) of a code: T0 = Q m - P d.  The solutions are (bu T0 - Q t,
// au T0 - P t); with T0 >= 0 the smallest d >= 0 gives m >= 0, with T0 < 0
// the smallest m >= 0 gives d > 0, and the next ones exceed the cell's bits.
// The quotient t comes from a reciprocal, exact for dividends below 2^23 (at
// most 128 nodes); WIDE dividends reach 2^24 and may give one too many.
template <bool WIDE>
__device__ __forceinline__ void decode(const MaxCode &k, uint32_t T, int &d,
                                       int &m) {
  const int T0 = k.s * ((int)T - k.off);
  const uint32_t a = (uint32_t)abs(T0);
  const bool up = T0 >= 0;
  const uint32_t x = up ? (uint32_t)k.bu * a
                        : (uint32_t)(k.au * (int)a + k.P - 1);
  uint32_t q = __umulhi(x, up ? k.invQ : k.invP);
  if constexpr (WIDE) {
    const uint32_t den = (uint32_t)(up ? k.Q : k.P);
    if (q * den > x) q--;
  }
  const int t = up ? (int)q : -(int)q;
  d = k.bu * T0 - k.Q * t;
  m = k.au * T0 - k.P * t;
}

// ------------------------------------------------------------------------
// The table: entry [chunk][node][lane] of (Q + 1) / 2 words, 16 bits per
// cell: off + wd d + wm m of the cell at the node.  Counts are off = 0, wd
// = 1, wm = 256.  Chunk c holds the warp's cells from 32 wpc Q c on, as
// load_cells takes them.
// ------------------------------------------------------------------------
// One chunk's part of it: nodes below ns in shared memory, the others (rows
// of five to eight words only, where 256 nodes x 512 cells take 256 KB) in
// global memory, which stays in L2 for the chains at work.
template <int W32, int Q>
struct Table {
  static constexpr int NW = kPackWords<Q>;
  uint32_t *s, *g;
  int ns;
  __device__ __forceinline__ uint32_t *at(int j) const {
    if constexpr (W32 <= 4) return s + j * 32 * NW;
    return j < ns ? s + j * 32 * NW : g + (j - ns) * 32 * NW;
  }
  __device__ __forceinline__ void ld(int j, int lane,
                                     uint32_t (&k)[NW]) const {
    ld_pack<Q>(at(j), lane, k);
  }
  __device__ __forceinline__ void st(int j, int lane,
                                     const uint32_t (&k)[NW]) const {
    st_pack<Q>(at(j), lane, k);
  }
  __device__ __forceinline__ Table chunk(int c, int n) const {
    return Table{s + c * ns * 32 * NW, g + c * (n - ns) * 32 * NW, ns};
  }
};

// From the ancestor rows by masked popcounts (any rows): at the start of a
// launch and after the rare moves that are not followed node by node.
template <int W32, int Q>
__device__ __noinline__ void fill_table(const uint32_t *rows,
                                        const DatasetDev *ds,
                                        const Table<W32, Q> tab,
                                        int chunks, int wpc, int wic,
                                        int lane, int off, int wd, int wm) {
  constexpr int RS = rs_of_w32(W32);
  constexpr int NW = kPackWords<Q>;
  const int n = ds->n_nodes;
  for (int c = 0; c < chunks; c++) {
    Cells<W32, Q> cb;
    load_cells<W32, Q>(cb, *ds, 32 * (wpc * Q * c + wic), 32 * wpc, lane);
#pragma unroll 1
    for (int j = 0; j < n; j++) {
      uint32_t a[W32], k[NW];
      ld_row<W32>(rows + j * RS, a);
#pragma unroll
      for (int w = 0; w < NW; w++) k[w] = 0u;
#pragma unroll
      for (int q = 0; q < Q; q++)
        k[q >> 1] += (uint32_t)(off + wd * masked_popc<W32>(cb.D[q], a) +
                                wm * masked_popc<W32>(cb.M[q], a))
                     << (16 * (q & 1));
      tab.chunk(c, n).st(j, lane, k);
    }
  }
  __syncwarp();
}

// The same from the block's increment table, along a parents-first order
// (canonical_order with the tree's parent vector): one chunk, each lane its
// own column.
template <int Q>
__device__ __noinline__ void fill_table_inherit(const SumCtx sx, int n,
                                                int lane, int off, int wd,
                                                int wm) {
  constexpr int NW = kPackWords<Q>;
  {
    uint32_t k[NW];
#pragma unroll
    for (int w = 0; w < NW; w++) k[w] = (uint32_t)off * 0x10001u;
    st_pack<Q>(sx.cnt, (int)(sx.ord[0] & 0xFF) * 32 + lane, k);
  }
#pragma unroll 2
  for (int i = 1; i < n; i++) {
    const uint32_t o = sx.ord[i];
    const int j = (int)(o & 0xFF), p = (int)(o >> 8);
    uint32_t a[NW], g[NW];
    ld_pack<Q>(sx.cnt, p * 32 + lane, a);
    ld_pack<Q>(sx.inc, j * 32 + lane, g);
#pragma unroll
    for (int w = 0; w < NW; w++)
      a[w] += (g[w] & 0x00010001u) * (uint32_t)wd +
              ((g[w] >> 8) & 0x00010001u) * (uint32_t)wm;
    st_pack<Q>(sx.cnt, j * 32 + lane, a);
  }
}

// ------------------------------------------------------------------------
// A realised tree move as two classes of changed nodes
// ------------------------------------------------------------------------
// Entries of class v change by T[a0] - T[b0], those of class w by T[a1] -
// T[b1].  SwapNodes(v, w) changes the two classes by opposite amounts, +-
// (T[a0] - T[b0] - T[a1] + T[b1]) with a1, b1 = v and its parent, a0, b0 = w
// and its parent, and then exchanges the entries of v and w.
struct Delta {
  uint32_t v, w, a0, b0, a1, b1;
  bool swap;
};

// select_bit without its branches: each lane ranks its own nodes.
template <int W32>
__device__ __forceinline__ uint32_t kth_bit(const uint32_t (&S)[W32],
                                            uint32_t k, int lane) {
  const uint32_t below = (1u << lane) - 1u;
  uint32_t before = 0, result = 0;
#pragma unroll
  for (int r = 0; r < W32; r++) {
    const bool hit = ((S[r] >> lane) & 1u) &&
                     before + (uint32_t)__popc(S[r] & below) == k;
    const uint32_t b = __ballot_sync(BBS_FULL_MASK, hit);
    if (b) result = 32u * r + (uint32_t)(__ffs(b) - 1);
    before += (uint32_t)__popc(S[r]);
  }
  return result;
}

// realize_move for a tree whose parent vector is known; what the move does
// not use is not drawn.  `general`: a k-th (non)descendant beyond the count
// (the reference's node-0 rule), a move of the root or of one node onto
// itself: not expressed as classes.
template <int W32>
__device__ __forceinline__ bbs_move_params realize_classes(
    const uint32_t *rows, const uint8_t *par, int n, const bbs_raw_move &raw,
    int lane, uint32_t (&Dv)[W32], uint32_t (&Dw)[W32], bool &related,
    bool &general, float &corr) {
  constexpr int RS = rs_of_w32(W32);
  bbs_move_params p;
  uint32_t v = min(raw.raw_v, (uint32_t)(n - 1));
  uint32_t w = min(raw.raw_w, (uint32_t)(n - 1));
  // every load before the first use: is_ancestor(v, w), both parents and
  // both descendant sets, exchanged afterwards where v is above w
  const bool above = (rows[w * RS + (v >> 5)] >> (v & 31u)) & 1u;
  const uint32_t pv = par[v], pw = par[w];
  descendant_sets<W32>(rows, n, v, w, lane, Dv, Dw);
  if (above) {
    const uint32_t t = v;
    v = w;
    w = t;
#pragma unroll
    for (int r = 0; r < W32; r++) {
      const uint32_t d = Dv[r];
      Dv[r] = Dw[r];
      Dw[r] = d;
    }
  }
  p.parent_of_v = above ? pw : pv;
  p.parent_of_w = above ? pv : pw;
  p.move_type = raw.move_type;
  p.v = v;
  p.w = w;
  p.descendant_of_v = p.nondescendant_of_v = 0;
  p.new_beta = 0.0f;
  related = has_bit<W32>(Dw, v);
  general = v == w || w == (uint32_t)(n - 1) || v == (uint32_t)(n - 1);
  int ndv = 0;
#pragma unroll
  for (int r = 0; r < W32; r++) ndv += __popc(Dv[r]);
  if (raw.move_type == BBS_MOVE_PRUNE_REATTACH) {
    const int nnd = n - ndv;
    const uint32_t k = __float2uint_rz(
        floorf(__fmul_rn(raw.raw_nondescendant_of_v, (float)nnd)));
    uint32_t ND[W32];
#pragma unroll
    for (int r = 0; r < W32; r++) ND[r] = ~Dv[r] & group_mask(r, n);
    p.nondescendant_of_v = kth_bit<W32>(ND, k, lane);
    general = general || k >= (uint32_t)nnd;
  } else if (raw.move_type == BBS_MOVE_SWAP_SUBTREES && related) {
    int ndw = 0;
#pragma unroll
    for (int r = 0; r < W32; r++) ndw += __popc(Dw[r]);
    const uint32_t k = __float2uint_rz(
        floorf(__fmul_rn(raw.raw_descendant_of_v, (float)ndv)));
    p.descendant_of_v = kth_bit<W32>(Dv, k, lane);
    general = general || k >= (uint32_t)ndv;
    corr = __fdiv_rn((float)ndv, (float)ndw);  // src/Application.hpp:443-450
  }
  return p;
}

// Two sets of nodes: the descendants of v and of w, or the two classes.
template <int W32>
struct NodeSets {
  uint32_t v[W32], w[W32];
};

// The classes of a realised move (not a general one).
template <int W32>
__device__ __forceinline__ Delta move_classes(const bbs_move_params &p,
                                              bool related,
                                              const NodeSets<W32> &D,
                                              NodeSets<W32> &C) {
  Delta x;
  const bool prune = p.move_type == BBS_MOVE_PRUNE_REATTACH;
  x.swap = p.move_type == BBS_MOVE_SWAP_NODES;
  x.v = p.v;
  x.w = p.w;
  x.b0 = x.b1 = p.parent_of_v;
  x.a0 = prune ? p.nondescendant_of_v : p.parent_of_w;
  x.a1 = p.descendant_of_v;
  if (x.swap) {
    x.a0 = p.w;
    x.b0 = p.parent_of_w;
    x.a1 = p.v;
  } else if (!related) {
    x.a1 = p.parent_of_v;
    x.b1 = p.parent_of_w;
  }
#pragma unroll
  for (int r = 0; r < W32; r++) {
    C.v[r] = x.swap ? D.v[r] & ~D.w[r] : D.v[r];
    C.w[r] = prune ? 0u : D.w[r] & ~D.v[r];
  }
  return x;
}

// The changed nodes as a list in shared memory, class v first: a loop over
// it is one copy of its body, whatever the row width (the chain kernels are
// bound by instruction fetch before anything else when their step code is
// unrolled per row word).  nv: nodes of class v; returns the total.
template <int W32>
__device__ __forceinline__ int list_nodes(const NodeSets<W32> &C,
                                          uint8_t *list, int lane, int &nv) {
  const uint32_t below = (1u << lane) - 1u;
  int at = 0;
#pragma unroll
  for (int r = 0; r < W32; r++) {
    if ((C.v[r] >> lane) & 1u)
      list[at + __popc(C.v[r] & below)] = (uint8_t)(32 * r + lane);
    at += __popc(C.v[r]);
  }
  nv = at;
#pragma unroll
  for (int r = 0; r < W32; r++) {
    if ((C.w[r] >> lane) & 1u)
      list[at + __popc(C.w[r] & below)] = (uint8_t)(32 * r + lane);
    at += __popc(C.w[r]);
  }
  __syncwarp();
  return at;
}

// Packed differences by value.
template <int NW>
struct Packed {
  uint32_t k[NW];
};

// The classes' changes as packed differences (their sum with an entry is the
// new entry, field borrows included).
template <int W32, int Q, int NW = kPackWords<Q>>
__device__ __forceinline__ void class_deltas(const Table<W32, Q> &tab,
                                             const Delta &x, int lane,
                                             Packed<NW> &dv, Packed<NW> &dw) {
  uint32_t a[NW], b[NW], c[NW], e[NW];
  tab.ld((int)x.a0, lane, a);
  tab.ld((int)x.b0, lane, b);
  tab.ld((int)x.a1, lane, c);
  tab.ld((int)x.b1, lane, e);
#pragma unroll
  for (int i = 0; i < NW; i++) {
    dv.k[i] = a[i] - b[i];
    dw.k[i] = c[i] - e[i];
    if (x.swap) {
      dv.k[i] -= dw.k[i];
      dw.k[i] = 0u - dv.k[i];
    }
  }
}

// Adds the classes' changes to the table, or takes them back: the nodes of
// list_nodes (nc of them, nv of the first class).
template <int W32, int Q, int NW = kPackWords<Q>>
__device__ __forceinline__ void apply_classes(const Table<W32, Q> &tab,
                                              const uint8_t *list, int nc,
                                              int nv, const Delta &x,
                                              Packed<NW> dv, Packed<NW> dw,
                                              bool back, int lane) {
  auto swap_entries = [&]() {
    uint32_t a[NW], b[NW];
    tab.ld((int)x.v, lane, a);
    tab.ld((int)x.w, lane, b);
    tab.st((int)x.v, lane, b);
    tab.st((int)x.w, lane, a);
  };
  if (back && x.swap) swap_entries();
  if (back) {
#pragma unroll
    for (int i = 0; i < NW; i++) {
      dv.k[i] = 0u - dv.k[i];
      dw.k[i] = 0u - dw.k[i];
    }
  }
  // (every load of a batch before its stores: one node at a time waited some
  // 100 clocks for each)
  constexpr int B = W32 > 4 ? 8 : 4;
#pragma unroll 1
  for (int c0 = 0; c0 < nc; c0 += B) {
    uint32_t k[B][NW];
    int j[B];
#pragma unroll
    for (int b = 0; b < B; b++) j[b] = (int)list[min(c0 + b, nc - 1)];
#pragma unroll
    for (int b = 0; b < B; b++) tab.ld(j[b], lane, k[b]);
#pragma unroll
    for (int b = 0; b < B; b++) {
#pragma unroll
      for (int i = 0; i < NW; i++) k[b][i] += c0 + b < nv ? dv.k[i] : dw.k[i];
      if (c0 + b < nc) tab.st(j[b], lane, k[b]);
    }
  }
  if (!back && x.swap) swap_entries();
  __syncwarp();  // the list has been read
}

// Taking a rejected proposal back, out of line: the bound leaves few of them.
template <int W32, int Q, int NW = kPackWords<Q>>
__device__ __noinline__ void take_back(const Table<W32, Q> tab, uint8_t *list,
                                       const Delta x, const NodeSets<W32> C,
                                       const Packed<NW> dv,
                                       const Packed<NW> dw, int lane) {
  int nv;
  const int nc = list_nodes<W32>(C, list, lane, nv);
  apply_classes<W32, Q>(tab, list, nc, nv, x, dv, dw, true, lane);
}

// ------------------------------------------------------------------------
// Max score: a proposal's largest codes
// ------------------------------------------------------------------------
// best = max(best, k) field by field over the nodes b < 8 whose bit of u is
// set.  Codes are at least 0 and the root always counts, so the others are
// masked to 0; as branches or predicated maxima a group of eight took 216 and
// 144 clocks, masked 100 (one warp, two words an entry).
template <int NW>
__device__ __forceinline__ void max8(uint32_t (&best)[NW],
                                     const uint32_t (&k)[8][NW], uint32_t u) {
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const uint32_t m = (uint32_t)((int)(u << (31 - b)) >> 31);
#pragma unroll
    for (int i = 0; i < NW; i++) best[i] = __vmaxu2(best[i], k[b][i] & m);
  }
}

// A node's entries in CH chunks of a table, side by side.
template <int Q, int CH, int NW = kPackWords<Q>>
__device__ __forceinline__ void ld_chunks(const uint32_t *t, int chunk_words,
                                          int idx, uint32_t (&k)[CH * NW]) {
#pragma unroll
  for (int c = 0; c < CH; c++) {
    uint32_t e[NW];
    ld_pack<Q>(t + c * chunk_words, idx, e);
#pragma unroll
    for (int i = 0; i < NW; i++) k[c * NW + i] = e[i];
  }
}

// max8 over nodes first .. first + count - 1 (first a multiple of 8) at t:
// whole groups, the next one's loads under the current one, then what is
// left.
template <int W32, int Q, int CH, int NW = kPackWords<Q>>
__device__ __forceinline__ void max_nodes(uint32_t (&best)[CH * NW],
                                          const uint32_t *t, int chunk_words,
                                          const uint32_t (&un)[W32], int first,
                                          int count, int lane) {
  auto bits = [&](int j) {
    return pick<W32>(un, (uint32_t)j >> 5) >> (j & 31);
  };
  int j = 0;
#pragma unroll 2
  for (; j + 8 <= count; j += 8) {
    uint32_t k[8][CH * NW];
#pragma unroll
    for (int b = 0; b < 8; b++)
      ld_chunks<Q, CH>(t, chunk_words, (j + b) * 32 + lane, k[b]);
    max8<CH * NW>(best, k, bits(first + j));
  }
  if (j < count) {
    uint32_t k[8][CH * NW];
#pragma unroll
    for (int b = 0; b < 8; b++)
      ld_chunks<Q, CH>(t, chunk_words, min(j + b, count - 1) * 32 + lane, k[b]);
    max8<CH * NW>(best, k, bits(first + j) & ((1u << (count - j)) - 1u));
  }
}

// The largest code of each cell of CH chunks over the proposal's nodes: the
// unchanged ones (the root is always one) and each class's largest, shifted.
// list holds the nc changed nodes, the first nv of class v.  Two chunks at a
// time share the masks and the list and have twice the loads in flight.
template <int W32, int Q, int CH, int NW = kPackWords<Q>>
__device__ __forceinline__ void scan_codes(const Table<W32, Q> &tab, int n,
                                           const NodeSets<W32> &C,
                                           const uint8_t *list, int nv, int nc,
                                           const Packed<NW> (&dv)[CH],
                                           const Packed<NW> (&dw)[CH],
                                           int lane,
                                           uint32_t (&best)[CH * NW]) {
  uint32_t un[W32], tv[CH * NW], tw[CH * NW];
#pragma unroll
  for (int r = 0; r < W32; r++) un[r] = ~(C.v[r] | C.w[r]) & group_mask(r, n);
#pragma unroll
  for (int i = 0; i < CH * NW; i++) best[i] = tv[i] = tw[i] = 0u;
  const int sw = tab.ns * 32 * NW;
  if constexpr (W32 <= 4) {
    max_nodes<W32, Q, CH>(best, tab.s, sw, un, 0, n, lane);
  } else {
    // the global part's loads, eight nodes at a time, each under its share of
    // the nodes in shared memory (ns is a multiple of 8, or n)
    const int ne = n - tab.ns, groups = (ne + 7) >> 3, gw = ne * 32 * NW;
    const int share =
        groups > 0 ? ((tab.ns + 8 * groups - 1) / (8 * groups)) * 8 : tab.ns;
    int j = 0;
#pragma unroll 1
    for (int e = 0; j < tab.ns || e < ne; e += 8) {
      uint32_t x[8][CH * NW];
      if (e < ne) {
#pragma unroll
        for (int b = 0; b < 8; b++)
          ld_chunks<Q, CH>(tab.g, gw, min(e + b, ne - 1) * 32 + lane, x[b]);
      }
      const int count = min(share, tab.ns - j);
      max_nodes<W32, Q, CH>(best, tab.s + j * 32 * NW, sw, un, j, count, lane);
      j += count;
      if (e < ne) {
        uint32_t u = pick<W32>(un, (uint32_t)(tab.ns + e) >> 5) >> ((tab.ns + e) & 31);
        if (ne - e < 8) u &= (1u << (ne - e)) - 1u;
        max8<CH * NW>(best, x, u);
      }
    }
  }
  constexpr int B = W32 > 4 ? 8 : 4;
#pragma unroll 1
  for (int c0 = 0; c0 < nc; c0 += B) {
    uint32_t k[B][CH * NW];
#pragma unroll
    for (int b = 0; b < B; b++) {
      const int j = (int)list[min(c0 + b, nc - 1)];
      if (W32 <= 4 || j < tab.ns)
        ld_chunks<Q, CH>(tab.s, sw, j * 32 + lane, k[b]);
      else
        ld_chunks<Q, CH>(tab.g, (n - tab.ns) * 32 * NW,
                         (j - tab.ns) * 32 + lane, k[b]);
    }
#pragma unroll
    for (int b = 0; b < B; b++) {
      const bool in_v = min(c0 + b, nc - 1) < nv;
#pragma unroll
      for (int i = 0; i < CH * NW; i++) {
        tv[i] = __vmaxu2(tv[i], in_v ? k[b][i] : 0u);
        tw[i] = __vmaxu2(tw[i], in_v ? 0u : k[b][i]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < CH; c++)
#pragma unroll
    for (int i = 0; i < NW; i++) {
      uint32_t &o = best[c * NW + i];
      if (nv > 0) o = __vmaxu2(o, tv[c * NW + i] + dv[c].k[i]);
      if (nc > nv) o = __vmaxu2(o, tw[c * NW + i] + dw[c].k[i]);
    }
}

// The max score over a table of counts: lane sums of k and m at each cell's
// best node by its reference-order score at the rates of L, the first in node
// order (best_nodes); of the current tree or, with nc > 0 nodes in list, of the
// proposal x, to whose counts the table goes and back.  For chains whose codes
// do not exist, tie at many nodes or would be made anew too often; out of line,
// as the others' steps need the room.
template <int W32, int Q, int NW = kPackWords<Q>>
__device__ __noinline__ int2 scan_counts(const Table<W32, Q> tab,
                                         const DatasetDev *ds,
                                         const LogTable L, int chunks, int wpc,
                                         int wic, int lane,
                                         const uint8_t *list, int nc, int nv,
                                         const Delta x) {
  const int n = ds->n_nodes;
  const LogTable2 L2 = log_table2(L, ds->neg_zero);
  int sk = 0, sm = 0;
#pragma unroll 1
  for (int c = 0; c < chunks; c++) {
    const Table<W32, Q> tc = tab.chunk(c, n);
    Packed<NW> dv, dw;
    if (nc > 0) {
      class_deltas<W32, Q>(tc, x, lane, dv, dw);
      apply_classes<W32, Q>(tc, list, nc, nv, x, dv, dw, false, lane);
    }
    float best[Q];
    uint32_t at[Q];  // the best node's entry
    float2 pdb[Q], pmb[Q];
    {
      Cells<W32, Q> cb;
      load_cells<W32, Q>(cb, *ds, 32 * (wpc * Q * c + wic), 32 * wpc, lane);
      uint32_t k[NW];
      tc.ld(0, lane, k);
#pragma unroll
      for (int q = 0; q < Q; q++) {
        pdb[q] = dup2(cb.pdb[q]);
        pmb[q] = dup2(cb.pmb[q]);
        at[q] = k[q >> 1];
        best[q] = pair_score_b(pack_d_biased(at[q], q), pack_m_biased(at[q], q),
                               cb.pdb[q], cb.pmb[q], L.l00, L.l01, L.l10,
                               L.l11);
      }
    }
    // (past the end the last node again, whose score is not above itself)
#pragma unroll 1
    for (int j = 1; j < n; j += 2) {
      uint32_t a[NW], b[NW];
      tc.ld(j, lane, a);
      tc.ld(min(j + 1, n - 1), lane, b);
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const uint32_t u = a[q >> 1], v = b[q >> 1];
        const float2 s = pair_score_b2(
            make_float2(pack_d_biased(u, q), pack_d_biased(v, q)),
            make_float2(pack_m_biased(u, q), pack_m_biased(v, q)), pdb[q],
            pmb[q], L2);
        at[q] = s.x > best[q] ? u : at[q];
        best[q] = s.x > best[q] ? s.x : best[q];
        at[q] = s.y > best[q] ? v : at[q];
        best[q] = s.y > best[q] ? s.y : best[q];
      }
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int d = (int)((at[q] >> (16 * (q & 1))) & 0xFFu),
                m = (int)((at[q] >> (16 * (q & 1) + 8)) & 0xFFu);
      sk += d + m;
      sm += m;
    }
    if (nc > 0)
      apply_classes<W32, Q>(tc, list, nc, nv, x, dv, dw, true, lane);
  }
  sk = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)sk);
  sm = (int)__reduce_add_sync(BBS_FULL_MASK, (uint32_t)sm);
  return make_int2(sk, sm);
}

// ------------------------------------------------------------------------
// Sum score
// ------------------------------------------------------------------------
// Terms below 2^-126 are flushed to zero: 2^-118 is above 128 of them and as
// much again.
inline constexpr float kFlushed = 3.0092655e-36f;

// What the bound keeps of the current tree, for the lane's Q cells: the
// exponents' offset, the sum of the terms and its reciprocal, and the
// largest exponent (all against the reference the sum was taken against).
template <int Q>
struct CellSums {
  float base[Q], z[Q], rz[Q], mx[Q];
};

// The second pass over the far-off cells of one cell slot (resum_cells'
// terms in the same order), counts from the table.  One slot at a time, eight
// nodes' loads and exponentials in flight: what is left is the chain of
// additions (a dataset whose rates leave one cell far below its bound takes
// this pass in every evaluation).
struct Resum1 {
  float z, ed, em;
};

template <int W32, int Q>
__device__ __noinline__ Resum1 resum_slot_table(const Table<W32, Q> tab,
                                                const uint16_t *ord, int n,
                                                int lane, float c1, float c2,
                                                float base, int q) {
  constexpr int NW = kPackWords<Q>;
  const int word = lane * NW + (q >> 1);
  const uint32_t sd = (q & 1) ? 0x7542u : 0x7540u;
  Resum1 o{0.0f, 0.0f, 0.0f};
  auto term = [&](uint32_t k) {
    const float fd =
        __int_as_float((int)__byte_perm(k, 0x4B000000u, sd)) - 8388608.0f;
    const float fm =
        __int_as_float((int)__byte_perm(k, 0x4B000000u, sd + 1u)) - 8388608.0f;
    const float e = ex2_approx(fmaf(fd, c1, fmaf(fm, c2, base)));
    o.z += e;
    o.ed = fmaf(e, fd, o.ed);
    o.em = fmaf(e, fm, o.em);
  };
#pragma unroll 8
  for (int i = 0; i < n; i++) term(tab.at((int)(ord[i] & 0xFF))[word]);
  return o;
}

// sum_cells with the counts of every node in the table and the tree's
// canonical order (ord): the same terms in the same pairs and
// order, so the same sums.  The table's entries are all in place before the
// loop, so its loads wait for nothing but the order.  ord + 1 is 8-byte
// aligned and followed by three zeros (slot_sum).
template <int W32, int Q>
__device__ __forceinline__ void sum_cells_table(
    const Table<W32, Q> &tab, const uint16_t *ord, int n, const float (&pd)[Q],
    const float (&pm)[Q], const LogTable &L, int c0, int stride, int lane,
    int n_cells, long long (&acc)[6], CellSums<Q> &cs) {
  constexpr int NW = kPackWords<Q>;
  const float c1 = (L.l01 - L.l00) * kLog2E;
  const float c2 = (L.l11 - L.l10) * kLog2E;
  const float2 c1p = dup2(c1), c2p = dup2(c2);
  const float u0 = fmaxf(L.l00, L.l01), u1 = fmaxf(L.l10, L.l11);
  float r[Q], base[Q], mx[Q];
  float2 base2[Q], z2[Q], ed2[Q], em2[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) {
    r[q] = fmaf(pd[q], u0, pm[q] * u1) - 72.0f;
    base[q] = (fmaf(pd[q], L.l00, pm[q] * L.l10) - r[q]) * kLog2E;
    base2[q] = dup2(base[q]);
    mx[q] = base[q];  // the root has no counted bits
    z2[q] = make_float2(ex2_approx(base[q]), 0.0f);
    ed2[q] = em2[q] = make_float2(0.0f, 0.0f);
  }
  // Four nodes an iteration, in the pairs (1, 2), (3, 4), ... of the other
  // count sources: their entries are loaded an iteration ahead of the float
  // work and the order, four nodes a load, two ahead.  (96 nodes, one warp
  // per scheduler, one and three cells per lane: 46 and 85 clocks a pair; one
  // node a load and one pair ahead 58 and 95.)  Past the order's end stand
  // zeros, past its last group that group again: loaded, not summed.
  if (n > 1) {
    const int last = (n - 2) >> 2;
    auto order4 = [&](int g) {
      return *reinterpret_cast<const uint2 *>(ord + 1 + 4 * min(g, last));
    };
    auto entries = [&](uint2 o, uint32_t (&k)[4][NW]) {
      tab.ld((int)__byte_perm(o.x, 0u, 0x4440u), lane, k[0]);
      tab.ld((int)__byte_perm(o.x, 0u, 0x4442u), lane, k[1]);
      tab.ld((int)__byte_perm(o.y, 0u, 0x4440u), lane, k[2]);
      tab.ld((int)__byte_perm(o.y, 0u, 0x4442u), lane, k[3]);
    };
    uint32_t k[4][NW];
    entries(order4(0), k);
    uint2 o = order4(1);
    int left = n - 1;  // positions not summed yet
#pragma unroll 1
    for (int g = 2; left >= 4; left -= 4, g++) {
      uint32_t next[4][NW];
      entries(o, next);
      o = order4(g);
      sum_counts2<Q, NW>(k[0], k[1], c1p, c2p, base2, mx, z2, ed2, em2);
      sum_counts2<Q, NW>(k[2], k[3], c1p, c2p, base2, mx, z2, ed2, em2);
#pragma unroll
      for (int b = 0; b < 4; b++)
#pragma unroll
        for (int w = 0; w < NW; w++) k[b][w] = next[b][w];
    }
    if (left >= 2) {
      sum_counts2<Q, NW>(k[0], k[1], c1p, c2p, base2, mx, z2, ed2, em2);
#pragma unroll
      for (int w = 0; w < NW; w++) k[0][w] = k[2][w];
    }
    if (left & 1) {
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const float fd = pack_d_biased(k[0][q >> 1], q) - 8388608.0f;
        const float fm = pack_m_biased(k[0][q >> 1], q) - 8388608.0f;
        const float t = fmaf(fd, c1, fmaf(fm, c2, base[q]));
        const float e = ex2_approx(t);
        mx[q] = fmaxf(mx[q], t);
        z2[q].x += e;
        ed2[q].x = fmaf(e, fd, ed2[q].x);
        em2[q].x = fmaf(e, fm, em2[q].x);
      }
    }
  }
  float z[Q], ed[Q], em[Q];
  bool bad[Q], any = false;
#pragma unroll
  for (int q = 0; q < Q; q++) {
    z[q] = z2[q].x + z2[q].y;
    ed[q] = ed2[q].x + ed2[q].y;
    em[q] = em2[q].x + em2[q].y;
    bad[q] = !(mx[q] >= -80.0f * kLog2E);
    any |= bad[q];
  }
  if (__any_sync(BBS_FULL_MASK, any)) {
#pragma unroll
    for (int q = 0; q < Q; q++) {
      if (!__any_sync(BBS_FULL_MASK, bad[q])) continue;
      const Resum1 o = resum_slot_table<W32, Q>(
          tab, ord, n, lane, c1, c2, bad[q] ? base[q] - mx[q] : base[q], q);
      if (bad[q]) {
        r[q] = fmaf(mx[q], kLn2, r[q]);
        base[q] -= mx[q];
        mx[q] = 0.0f;
        z[q] = o.z;
        ed[q] = o.ed;
        em[q] = o.em;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const float inv = __frcp_rn(z[q]);
    cs.base[q] = base[q];
    cs.z[q] = z[q];
    cs.rz[q] = inv;
    cs.mx[q] = mx[q];
    const int c = c0 + stride * q + lane;
    if (c >= n_cells) continue;
    const float Ed = ed[q] * inv, Em = em[q] * inv;
    acc[0] += (long long)__float2int_rn((r[q] + logf(z[q])) * kScoreScale);
    acc[2] += (long long)__float2int_rn(Ed * kFixScale);
    acc[4] += (long long)__float2int_rn(Em * kFixScale);
    acc[5] += (long long)__float2int_rn(fmaf(mx[q], kLn2, r[q]) * kScoreScale);
  }
}

// The current tree's terms at the listed nodes: their sum and largest
// exponent per cell.
template <int W32, int Q, int NW = kPackWords<Q>>
__device__ __forceinline__ void class_terms(const Table<W32, Q> &tab,
                                            const uint8_t *list, int n_list,
                                            float c1, float c2,
                                            const float (&base)[Q], int lane,
                                            float (&zo)[Q], float (&mo)[Q]) {
  const float2 c1p = dup2(c1), c2p = dup2(c2);
  float2 z2[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) {
    z2[q] = make_float2(0.0f, 0.0f);
    mo[q] = -INFINITY;
  }
  uint32_t a0[NW], a1[NW];
  tab.ld((int)list[0], lane, a0);
  tab.ld((int)list[n_list > 1 ? 1 : 0], lane, a1);
#pragma unroll 1
  for (int c = 0; c < n_list; c += 2) {
    // an odd last node is paired with itself; its copy's term is dropped
    const bool two = c + 1 < n_list;
    float2 fd[Q], fm[Q];
    pack_to_float2<Q, NW>(a0, a1, fd, fm);
    // the next pair's entries (the last loads again past the end)
    tab.ld((int)list[min(c + 2, n_list - 1)], lane, a0);
    tab.ld((int)list[min(c + 3, n_list - 1)], lane, a1);
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const float2 t = ffma2(fd[q], c1p, ffma2(fm[q], c2p, dup2(base[q])));
      const float e1 = ex2_approx(t.y);
      z2[q] = fadd2(z2[q], make_float2(ex2_approx(t.x), two ? e1 : 0.0f));
      mo[q] = fmax3(mo[q], t.x, t.y);
    }
  }
#pragma unroll
  for (int q = 0; q < Q; q++) zo[q] = z2[q].x + z2[q].y;
}

// Exponent shift of cell slot q between two table entries a and b (their
// signed count differences times c1 and c2).
template <int NW>
__device__ __forceinline__ float entry_shift(const uint32_t (&a)[NW],
                                             const uint32_t (&b)[NW], int q,
                                             float c1, float c2) {
  const float dd = pack_d_biased(a[q >> 1], q) - pack_d_biased(b[q >> 1], q);
  const float dm = pack_m_biased(a[q >> 1], q) - pack_m_biased(b[q >> 1], q);
  return fmaf(dd, c1, dm * c2);
}

inline constexpr float kBoundUnit = 4096.0f;  // 2^-12 of a base-2 log

// A lane's sum as an integer not below it, in units of 1 / kBoundUnit; 8192,
// where inf and NaN end too, for a larger one.
__device__ __forceinline__ int lane_bound(float s) {
  s = s < 8192.0f ? fmaxf(s, -64.0f) : 8192.0f;
  return __float2int_ru(s * kBoundUnit) + 1;
}

// Adds upper bounds of a proposal's sum score and max score over one chunk of
// this warp's cells, relative to the current tree, to up: up[0] bounds sum_c
// log2(z'_c / z_c), up[1] bounds sum_c (largest exponent' - largest exponent),
// in units of 1 / kBoundUnit.  eps bounds the relative rounding of a term
// against its shifted form.  Sums of up to 128 terms are good to 2^-17 of the
// largest partial sum, so a cell's remainder z - zo is taken with 2^-15 z on
// top.  kFlushed, on zo and on z, covers the flushed terms of the nodes that
// move and of those that stay: where a cell's best node moves far away, the
// exact sum takes the others against their own maximum and counts them again.
template <int W32, int Q, int NW = kPackWords<Q>>
__device__ __forceinline__ void bound_proposal(
    const Table<W32, Q> &tab, const Delta &x, const uint8_t *list, int nv, int nc,
    const CellSums<Q> &cs, const LogTable &L, float eps, int c0, int stride,
    int n_cells, int lane, float (&up)[2]) {
  const float c1 = (L.l01 - L.l00) * kLog2E;
  const float c2 = (L.l11 - L.l10) * kLog2E;
  float hv[Q], hw[Q], z1[Q], gain[Q], rest[Q];
  {
    uint32_t a[NW], b[NW], c[NW], e[NW];
    tab.ld((int)x.a0, lane, a);
    tab.ld((int)x.b0, lane, b);
    tab.ld((int)x.a1, lane, c);
    tab.ld((int)x.b1, lane, e);
#pragma unroll
    for (int q = 0; q < Q; q++) {
      hv[q] = entry_shift<NW>(a, b, q, c1, c2);
      hw[q] = entry_shift<NW>(c, e, q, c1, c2);
      if (x.swap) {
        hv[q] -= hw[q];
        hw[q] = -hv[q];
      }
      z1[q] = 0.0f;
      gain[q] = -INFINITY;
      rest[q] = cs.z[q] + kFlushed;
    }
  }
#pragma unroll 1
  for (int cls = 0; cls < 2; cls++) {
    const int at = cls ? nv : 0, count = cls ? nc - nv : nv;
    if (count > 0) {
      float zo[Q], mo[Q];
      class_terms<W32, Q>(tab, list + at, count, c1, c2, cs.base, lane, zo, mo);
#pragma unroll
      for (int q = 0; q < Q; q++) {
        rest[q] -= zo[q];
        z1[q] = fmaf(zo[q] + kFlushed, ex2_approx(hv[q]), z1[q]);
        gain[q] = fmaxf(gain[q], mo[q] + hv[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < Q; q++) hv[q] = hw[q];
  }
  float s = 0.0f, g = 0.0f;
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const float left = fmaxf(rest[q], 0.0f) + 3.0517578e-05f * cs.z[q];
    const float zu = fmaf(z1[q], 1.0f + eps, left);
    // the largest exponent left is at most the current one and at most the
    // logarithm of what is left of the sum
    const float top = fmaxf(fminf(cs.mx[q], __log2f(left) + eps), gain[q] + eps);
    if (c0 + stride * q + lane < n_cells) {
      s += __log2f(zu * cs.rz[q]);
      g += top - cs.mx[q];
    }
  }
  // A lane loses 15 a cell at most (what is left is at least 2^-15 z), so that
  // lane_bound's -64 is not below it.  Its 8192 is no bound; but no other lanes
  // bring that sum back below 4096, and a warp above 4096 has no bound (the
  // rates are far below those of real data), nor has the proposal then.
  const int si = __reduce_add_sync(BBS_FULL_MASK, lane_bound(s));
  const int gi = __reduce_add_sync(BBS_FULL_MASK, lane_bound(g));
  constexpr int most = 4096 * (int)kBoundUnit;
  up[0] += si < most ? (float)si : INFINITY;
  up[1] += gi < most ? (float)gi : INFINITY;
}

}  // namespace bbs
