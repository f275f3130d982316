// bbs_layout.h -- shared-memory layout of the chain kernels: the sizes the
// kernels carve their dynamic shared memory by and the host launchers
// request (host and device code).
#pragma once
#include <algorithm>

#include "bbs_internal.h"

namespace bbs {

// Bytes of a packed count table of n nodes x 32 lanes for q cells per
// lane: (q + 1) / 2 32-bit words per entry.
__host__ __device__ inline int pack_table_bytes(int n, int q) {
  return 4 * ((q + 1) / 2) * n * 32;
}

// Shared memory of the chain kernels, in bytes (16-byte aligned pieces).
__host__ __device__ inline int align16(int b) { return (b + 15) & ~15; }

// Rows of five to eight words: a warp's ring of the packed counts of the
// last kRing nodes in the canonical order, and its gene table, one entry
// of NW words per 8 genes and lane laid out as the counts are packed (word
// h: byte 0 the D bits of the 8 genes for cell slot 2h, byte 1 their M
// bits, bytes 2 and 3 the same for cell slot 2h + 1).
__host__ __device__ inline int ring_bytes(int q) {
  return 4 * ((q + 1) / 2) * kRing * 32;
}
__host__ __device__ inline int gene_table_bytes(int n, int q) {
  return 4 * ((q + 1) / 2) * ((n + 7) / 8) * 32;
}

// The canonical node order; rows of up to four words with three entries
// before and three after it (slot_sum).
__host__ __device__ inline int order_bytes(int n, int w32) {
  return align16(w32 <= 4 ? 2 * n + 12 : 2 * n);
}

// Per warp of a chain with the node-order scratch (every sum-score chain:
// its order is canonical; every chain that inherits counts): the canonical
// node order, its depth histogram and, with `counts`, the packed counts of
// every node for the lane's cells (rows of up to four words) or the ring
// and gene table (wider rows).
__host__ __device__ inline int sum_warp_bytes(int n, int w32, int q,
                                              bool counts) {
  int b = order_bytes(n, w32) + align16(4 * 32 * ((n + 31) / 32));
  if (counts)
    b += w32 <= 4 ? align16(pack_table_bytes(n, q))
                  : align16(ring_bytes(q)) + align16(gene_table_bytes(n, q));
  return b;
}

// Each warp's Philox blocks of 16 steps: 32 x 16 bytes.
inline constexpr int kPhiloxBytes = 512;

// The head of a chain slot: two row buffers, the partial sums of both step
// parities (2 x wpc x 12 words), a flag word (16 bytes) and each warp's
// Philox blocks.
__host__ __device__ inline int slot_head_bytes(int n, int rs, int wpc) {
  return 4 * (2 * n * rs + 24 * wpc + 4) + kPhiloxBytes * wpc;
}

// One chain slot: its head and, with the scratch, the current and proposed
// parent vectors and each warp's scratch.
__host__ __device__ inline int slot_bytes(int n, int rs, int wpc, bool scratch,
                                          int w32, int q, bool counts) {
  int b = slot_head_bytes(n, rs, wpc);
  if (scratch) b += align16(2 * n) + wpc * sum_warp_bytes(n, w32, q, counts);
  return b;
}

// After the slots, with `counts`: the block's tables of per-gene
// increments, one per warp part of a chain (wpc), each for that warp's
// 32 q cell slots.
__host__ __device__ inline int inc_table_bytes(int n, int q) {
  return align16(pack_table_bytes(n, q));
}
__host__ __device__ inline int table_bytes(int n, int w32, int q, int wpc,
                                           bool counts) {
  return counts && w32 <= 4 ? wpc * inc_table_bytes(n, q) : 0;
}

// Chain-kernel blocks: one-warp chains of one dataset share the block's
// increment table.  The launch bounds of each cells-per-lane variant aim
// at 16, 12 and 8 resident warps per SM for 1, 2 and 3-4 cells per lane
// (registers per thread 128, 168, 255), in blocks of up to 4, 4 and 8
// warps: eight warps of three or four cells per lane fill an SM alone.
// (The batched kernel for rows of five to eight words takes up to 255
// registers: shared memory limits those launches first.)
inline constexpr int kMaxBlockThreads = 256;
__host__ __device__ constexpr int chain_max_threads(int q) {
  return q >= 3 ? 256 : 128;
}
// Kernels that read proposals off a table (tab) get more registers: at 128 and
// 168 for one and two cells per lane they spilled (20 x 12, sum score: 5.8 ms
// against 4.6 ms per 1346 steps; 63 x 64, 8 chains: 3.4 against 2.1 us a step).
// So do the batched kernels of wide rows, whose blocks shared memory limits
// first.
__host__ __device__ constexpr int chain_blocks(int w32, int q, bool tab) {
  if (tab) return w32 > 4 ? 1 : (q == 1 ? 3 : (q == 2 ? 2 : 1));
  return q == 1 ? 4 : (q == 2 ? 3 : 1);
}
__host__ __device__ constexpr int chain_regs(int q, bool tab) {
  if (tab) return q == 1 ? 168 : 255;
  return q == 1 ? 128 : (q == 2 ? 168 : 255);
}

// Dynamic shared memory of a chain-kernel launch: `slots` chain slots of
// `wpc` warps and, with inherited counts, the increment tables.
__host__ __device__ inline int chain_launch_smem(int n, int n_cells, int q,
                                                 int wpc, int slots,
                                                 bool sum) {
  const int w32 = w32_of_nodes(n);
  const bool counts = inherits_counts(w32, n_cells, 32 * wpc * q);
  return slots * slot_bytes(n, rs_of_w32(w32), wpc, sum || counts, w32, q,
                            counts) +
         table_bytes(n, w32, q, wpc, counts);
}

// The table of every node that proposals are read off (bbs_incr.cuh).
//   chunks  chunks of 32 wpc q cells the table holds (0: no table, the cells
//           are streamed); the sum score takes one.
//   inc     rows of up to four words: the block's increment tables come with
//           it, which fill it, and again after a chain's rates change its codes:
//           one-warp chains of one dataset in one chunk share one (the layout
//           with `counts` above).  Other launches fill their tables from the
//           rows and keep the room.
//   ns, global  rows of five to eight words: what of it is in shared memory and
//           what in global memory.
struct TablePlan {
  int chunks;
  bool inc;
  int smem;         // dynamic shared memory of the launch
  int ns;           // nodes whose entries are in shared memory
  size_t global;    // bytes of table per slot in global memory (the others')
};

__host__ __device__ inline int table_part_bytes(int n, int q, int chunks) {
  return chunks * align16(pack_table_bytes(n, q));
}
// A slot with its table but without increments: the slot with the scratch,
// then each warp's part of the table.
__host__ __device__ inline int table_slot_bytes(int n, int rs, int wpc,
                                                int w32, int q, int chunks) {
  return slot_bytes(n, rs, wpc, true, w32, q, false) +
         wpc * table_part_bytes(n, q, chunks);
}

// Rows of five to eight words: a warp's part of a slot holds the table's
// first ns nodes.
__host__ __device__ inline int wide_part_bytes(int q, int chunks, int ns) {
  return chunks * align16(pack_table_bytes(ns, q));
}
__host__ __device__ inline int wide_slot_bytes(int n, int rs, int wpc, int w32,
                                               int q, int chunks, int ns) {
  return slot_bytes(n, rs, wpc, true, w32, q, false) +
         wpc * wide_part_bytes(q, chunks, ns);
}

inline constexpr int kFewCells = 12;

// What the chains of a launch read proposals off.
enum class Tables { none, codes, counts };

// The choice for max-score chains of up to 128 nodes: `load` chains per SM,
// error moves a share pb of all, the rates' codes (where pb is 0).
//   none    Few nodes and cells: an evaluation from the rows costs less than
//           following the table does, the more so the more often rates change,
//           which makes codes and table anew, and the more chains share an SM.
//   counts  Otherwise, where rates change so often that codes do not pay, and at
//           fixed rates without codes or with codes that tie at most counts (a
//           ratio of the log differences like 1 or 1/2) and so leave many
//           proposals to an evaluation from the rows: the table holds counts,
//           and a proposal scores every node from them.
//   codes   The rest.
// A step, us, by rows / codes / counts, one move in eleven an error move
// (Langevin): 2432 chains of 8 x 24 2.0 / 5.8 / 4.8, 608 of 32 x 64 3.5 / 2.8 /
// 3.3, 608 of 95 x 96 10.4 / 5.7 / 7.8; one in two: 608 of 95 x 96 10.8 / 14.7
// / 8.1.  Fitted to chains past their first thousands of steps, 4 to 127 genes,
// 8 to 256 cells, 8 to 2432 chains, none to half of the moves: the choice takes
// 1 % longer than the best of the three on average, codes alone 28 %.
struct CodeQuality {
  bool usable;
  int ties, most;  // of the denominators that tie, and how many could
};
inline Tables max_score_tables(int n, int n_cells, double load, float pb,
                               const CodeQuality &codes) {
  const int work = n * ((n_cells + 31) / 32);
  const bool poor = pb == 0.0f && (!codes.usable || 5 * codes.ties >= 2 * codes.most);
  const double crowd = 1.0 + 0.35 * std::max(0.0, std::min(load, 8.0) - 1.0);
  const double base = pb == 0.0f && load > 12.0 ? 17.0 : 5.0;
  if (work <= (poor ? 100.0 : std::min(100.0, base + 190.0 * pb * crowd)))
    return Tables::none;
  if (poor) return Tables::counts;
  const float often = load < 1.0 || (n_cells > 128 && n >= 64) ? 0.25f
                      : load >= 4.0 && n <= 64 && n_cells <= 128 ? 0.12f
                                                                 : 0.2f;
  return pb > often ? Tables::counts : Tables::codes;
}

// The plan of a launch of `slots` chain slots per block, its largest dataset of
// n nodes and n_cells cells.  Where the tables do not fit a block, or a
// sum-score chain's cells of rows of up to four words do not fit one chunk, the
// cells are streamed as before (such launches are bound by their masked
// popcounts). Nor does the sum score of at most 32 nodes and kFewCells cells
// take one: nearly every proposal is accepted, so the bound rejects little, and
// the sum over so few nodes costs less than following the table (1000 steps of
// 750 Langevin chains, every node and table: 8 x 4 2.28, 3.54 ms; 8 x 9 2.27,
// 3.07; 20 x 9 2.83, 3.48; 8 x 16 2.28, 2.57; at fixed rates 8 x 9 2.12, 1.80;
// 20 x 9 2.70, 2.28; 8 x 16 2.12, 1.54.  From 33 nodes on the table is no
// slower). Max-score chains take one where `max_table` says so.  With rows of
// five to eight words it is in shared memory where that leaves an SM four
// warps; else one chain per SM keeps as many nodes there as fit (255 x 512: 216
// of 256), the others in global memory.  The sum score keeps the ring at that
// width: half of its proposals are accepted in the runs measured (255 x 512)
// and then summed over every node, which with a table was slower (200 x 150: 17
// M against 22 M chain-steps/s).
inline TablePlan plan_tables(int n, int w32, int n_cells, int q, int wpc,
                             int slots, bool sum, bool one_dataset,
                             bool max_table, int smem_block, int smem_sm,
                             bool any_table = true) {
  const int rs = rs_of_w32(w32), span = 32 * wpc * q;
  const int chunks = (n_cells + span - 1) / span;
  if (w32 > 4) {
    const TablePlan ring{0, false,
                         chain_launch_smem(n, n_cells, q, wpc, slots, sum), 0, 0};
    if (!max_table || sum || !any_table) return ring;
    auto smem_of = [&](int ns) {
      return slots * wide_slot_bytes(n, rs, wpc, w32, q, chunks, ns);
    };
    const int full = smem_of(n);
    if (full <= smem_block &&
        smem_sm / (full + 1024) * slots * wpc >= 4)
      return TablePlan{chunks, false, full, n, 0};
    if (slots > 1) return ring;
    int ns = n & ~7;
    while (ns > 0 && smem_of(ns) > smem_block) ns -= 8;
    if (ns < n / 2) return ring;
    return TablePlan{chunks, false, smem_of(ns), ns,
                     (size_t)wpc * chunks * pack_table_bytes(n - ns, q)};
  }
  const TablePlan p{0, false, slots * slot_bytes(n, rs, wpc, sum, w32, q, false),
                    n, 0};
  if (!any_table ||
      (sum ? chunks > 1 || (w32 == 1 && n_cells <= kFewCells) : !max_table))
    return p;
  const bool inc = wpc == 1 && one_dataset && chunks == 1;
  const int smem =
      inc ? chain_launch_smem(n, n_cells, q, wpc, slots, sum)
          : slots * table_slot_bytes(n, rs, wpc, w32, q, chunks);
  if (smem > smem_block) return p;
  return TablePlan{chunks, inc, smem, n, 0};
}

// Resident warps per SM of such a launch (blocks of warps_per_block
// warps), from the SM's shared memory (smem_sm bytes, reserved_per_block
// of them taken by each block, at most smem_block per block) and registers.
inline int chain_resident_warps(int smem, int warps_per_block,
                                int regs_per_thread, int smem_sm,
                                int smem_block, int reserved_per_block) {
  if (smem > smem_block) return 0;
  const int by_smem = smem_sm / (smem + reserved_per_block);
  const int regs = (regs_per_thread + 7) & ~7;
  const int by_regs = 65536 / (regs * 32 * warps_per_block);
  const int blocks = by_smem < by_regs ? by_smem : by_regs;
  return blocks * warps_per_block;
}

}  // namespace bbs
