// Slots with a table of every node but no increment tables, walked on the
// host over node counts 2..128, 1..4 cells per lane, 1..4 warps per chain and
// 1..4 chunks: the table parts follow the slot's other pieces, inside the
// slot, disjoint and aligned; and plan_tables asks for that many bytes, or
// for the streamed layout where they do not fit a block.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "bbs_kernels.cuh"

int main() {
  constexpr int kBlock = 232448;
  long cases = 0;
  std::vector<uint8_t> mem(1 << 22);
  uint8_t *base = mem.data();
  for (int n = 2; n <= 128; n++)
    for (int q = 1; q <= 4; q++)
      for (int wpc = 1; wpc <= 4; wpc++)
        for (int chunks = 1; chunks <= 4; chunks++) {
          const int w32 = bbs::w32_of_nodes(n), rs = bbs::rs_of_w32(w32);
          const int sb = bbs::table_slot_bytes(n, rs, wpc, w32, q, chunks);
          size_t end = 0;
          for (int wic = 0; wic < wpc; wic++) {
            const bbs::SlotSum ss =
                bbs::slot_sum(base, n, rs, wpc, wic, w32, q, false);
            const size_t hist =
                (size_t)(reinterpret_cast<uint8_t *>(ss.sx.hist) - base) +
                4 * 32 * ((n + 31) / 32);
            if (hist > end) end = hist;
          }
          for (int wic = 0; wic < wpc; wic++) {
            const size_t lo =
                (size_t)(reinterpret_cast<uint8_t *>(bbs::table_part(
                             base, n, rs, wpc, wic, w32, q, chunks)) -
                         base);
            const size_t bytes = (size_t)chunks * bbs::pack_table_bytes(n, q);
            if (lo < end || lo % (4 * ((q + 1) / 2)) != 0 ||
                lo + bytes > (size_t)sb || sb % 16 != 0) {
              std::printf("FAIL n=%d q=%d wpc=%d chunks=%d wic=%d\n", n, q,
                          wpc, chunks, wic);
              return 1;
            }
            end = lo + bytes;
          }
          // cells that need just that many chunks, two datasets in the launch
          const int span = 32 * wpc * q, cells = span * (chunks - 1) + 1;
          for (int slots = 1; slots <= (wpc > 1 ? 1 : 4); slots++)
            for (int sum = 0; sum < 2; sum++) {
              const bbs::TablePlan p = bbs::plan_tables(
                  n, w32, cells, q, wpc, slots, sum != 0, false, true, kBlock,
                  kBlock + 1024);
              const bool few = w32 == 1 && cells <= bbs::kFewCells;
              const bool fits =
                  slots * sb <= kBlock && !(sum && (chunks > 1 || few));
              if (p.inc || p.chunks != (fits ? chunks : 0) ||
                  p.smem != slots * (fits ? sb
                                          : bbs::slot_bytes(n, rs, wpc,
                                                            sum != 0, w32, q,
                                                            false))) {
                std::printf("FAIL plan n=%d q=%d wpc=%d chunks=%d slots=%d\n",
                            n, q, wpc, chunks, slots);
                return 1;
              }
              cases++;
            }
        }
  // rows of five to eight words: plans that fit a block, the nodes that do not
  // in global memory; the sum score takes none
  for (int n = 129; n <= 256; n++)
    for (int q = 1; q <= 2; q++)
      for (int wpc = 1; wpc <= 4; wpc++)
        for (int sum = 0; sum < 2; sum++)
          for (int cells : {1, 33, 150, 512, 2049}) {
            const int w32 = bbs::w32_of_nodes(n), rs = bbs::rs_of_w32(w32);
            const int chunks = (cells + 32 * wpc * q - 1) / (32 * wpc * q);
            const bbs::TablePlan p =
                bbs::plan_tables(n, w32, cells, q, wpc, 1, sum != 0, true, true,
                                 kBlock, kBlock + 1024);
            bool ok = p.smem <= kBlock && !(sum && p.chunks > 0);
            if (p.chunks > 0)
              ok = ok && p.chunks == chunks && p.ns >= n / 2 && p.ns <= n &&
                   (p.ns == n || p.ns % 8 == 0) &&
                   p.smem == bbs::wide_slot_bytes(n, rs, wpc, w32, q, chunks,
                                                  p.ns) &&
                   p.global == (size_t)wpc * chunks *
                                   bbs::pack_table_bytes(n - p.ns, q);
            if (!ok) {
              std::printf("FAIL wide n=%d q=%d wpc=%d sum=%d cells=%d\n", n, q,
                          wpc, sum, cells);
              return 1;
            }
            cases++;
          }
  std::printf("tables ok %ld\n", cases);
  return 0;
}
