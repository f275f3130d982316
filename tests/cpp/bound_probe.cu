// The sum score's bound against exact sums: tables of every node are made on
// the host, one warp per case sums the current tree, bounds a proposal, brings
// the table to it and sums it, as a chain does.  The bound plus a chain's
// tolerance has to be at least the change of the score and of the max score.
//   far   one cell whose best node, 100 to 116 powers of two below the cell's
//         reference, moves away, while the other nodes lie about where a term
//         leaves the range of normal floats (2^-126)
//   high  one lane whose cells gain more than the bound counts, beside lanes
//         that lose less than that
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "bbs_kernels.cuh"

namespace {

struct Case {
  int q, n, n_cells, nv, nc;
  bbs::LogTable L;
  bbs::Delta x;
  std::vector<uint8_t> list;
  std::vector<uint16_t> entry;  // [node][slot][lane]: d | m << 8
  std::vector<float> pd, pm;    // [slot][lane]
};

struct Result {
  float up[2];
  double before[2], after[2];  // score and max score, data terms
};

__device__ float bound_eps(const bbs::LogTable &L, int n) {
  const float big =
      (float)n * fmaxf(fmaxf(fabsf(L.l00), fabsf(L.l01)),
                       fmaxf(fabsf(L.l10), fabsf(L.l11))) + 73.0f;
  return big * 2.3841858e-06f;
}

template <int Q>
__global__ void run_case(const uint32_t *table, const uint8_t *list_in,
                         const float *cells, bbs::LogTable L, bbs::Delta x,
                         int n, int n_cells, int nv, int nc, Result *out) {
  constexpr int NW = bbs::kPackWords<Q>;
  __shared__ __align__(8) uint16_t order[136];
  __shared__ __align__(8) uint32_t mem[128 * 32 * NW];
  __shared__ uint8_t list[128];
  const int lane = threadIdx.x;
  for (int i = lane; i < n * 32 * NW; i += 32) mem[i] = table[i];
  for (int i = lane; i < nc; i += 32) list[i] = list_in[i];
  uint16_t *ord = order + 3;
  // the root, which is the last node, first
  for (int i = lane; i < n + 3; i += 32)
    ord[i] = (uint16_t)(i == 0 ? n - 1 : i < n ? i - 1 : 0);
  __syncwarp();
  const bbs::Table<4, Q> tab{mem, nullptr, n};
  float pd[Q], pm[Q];
  for (int q = 0; q < Q; q++) {
    pd[q] = cells[(2 * q) * 32 + lane];
    pm[q] = cells[(2 * q + 1) * 32 + lane];
  }
  auto sum = [&](bbs::CellSums<Q> &cs, double (&o)[2]) {
    long long acc[6] = {0, 0, 0, 0, 0, 0};
    bbs::sum_cells_table<4, Q>(tab, ord, n, pd, pm, L, 0, 32, lane, n_cells,
                               acc, cs);
    o[0] = (double)bbs::warp_sum_ll(acc[0]) / (double)bbs::kScoreScale;
    o[1] = (double)bbs::warp_sum_ll(acc[5]) / (double)bbs::kScoreScale;
  };
  bbs::CellSums<Q> cs, pcs;
  double before[2], after[2];
  sum(cs, before);
  float up[2] = {0.0f, 0.0f};
  bbs::Packed<NW> dv, dw;
  bbs::class_deltas<4, Q>(tab, x, lane, dv, dw);
  bbs::bound_proposal<4, Q>(tab, x, list, nv, nc, cs, L, bound_eps(L, n), 0, 32,
                            n_cells, lane, up);
  bbs::apply_classes<4, Q>(tab, list, nc, nv, x, dv, dw, false, lane);
  sum(pcs, after);
  if (lane == 0)
    for (int k = 0; k < 2; k++) {
      out->up[k] = up[k];
      out->before[k] = before[k];
      out->after[k] = after[k];
    }
}

bbs::LogTable logs(double alpha, double beta) {
  bbs::LogTable L;
  L.l00 = (float)std::log1p(-alpha);
  L.l10 = (float)std::log(alpha);
  L.l01 = (float)std::log(beta);
  L.l11 = (float)std::log1p(-beta);
  return L;
}

Case empty_case(int q, int n, int n_cells, const bbs::LogTable &L) {
  Case c;
  c.q = q;
  c.n = n;
  c.n_cells = n_cells;
  c.L = L;
  c.x = bbs::Delta{};
  c.entry.assign((size_t)n * q * 32, 0);
  c.pd.assign((size_t)q * 32, 0.0f);
  c.pm.assign((size_t)q * 32, 0.0f);
  return c;
}

uint16_t field(int d, int m) { return (uint16_t)(d | m << 8); }

template <int Q>
void launch(const Case &c, const uint32_t *t, const uint8_t *l, const float *f,
            Result *r) {
  run_case<Q><<<1, 32>>>(t, l, f, c.L, c.x, c.n, c.n_cells, c.nv, c.nc, r);
}

// What a chain adds to the bound (run_chain_table).
double tolerance(const Case &c, const Result &r) {
  const double big =
      c.n * std::fmax(std::fmax(std::fabs(c.L.l00), std::fabs(c.L.l01)),
                      std::fmax(std::fabs(c.L.l10), std::fabs(c.L.l11))) + 73.0;
  return c.n_cells * (big * 4.7683716e-07 + 3.0517578e-05) +
         (std::fabs(r.before[0]) + std::fabs(r.before[1])) * 4.8e-07 + 1.0e-3;
}

// One cell: node 0 the best, `others` nodes at (d2, m2), a node far below that
// the best one is moved by, and the root.  lift: half of the others move too,
// one step up.
Case far_case(const bbs::LogTable &L, int pd, int pm, int d, int m, int d2,
              int m2, int others, bool lift) {
  Case c = empty_case(1, others + 4, 1, L);
  const int far = others + 1, step = others + 2, root = others + 3;
  auto set = [&](int node, int dd, int mm) {
    c.entry[(size_t)node * 32] = field(dd, mm);
  };
  set(0, d, m);
  for (int k = 1; k <= others; k++) set(k, d2, m2);
  set(far, 60, 0);
  set(step, 0, 1);
  set(root, 0, 0);
  c.pd[0] = (float)pd;
  c.pm[0] = (float)pm;
  c.x.a0 = (uint32_t)far;
  c.x.a1 = (uint32_t)step;
  c.x.b0 = c.x.b1 = (uint32_t)root;
  c.list.push_back(0);
  c.nv = 1;
  if (lift)
    for (int k = 1; k <= others / 2; k++) c.list.push_back((uint8_t)k);
  c.nc = (int)c.list.size();
  return c;
}

void far_cases(std::vector<Case> &cases) {
  for (double alpha : {1.0e-2, 1.0e-3, 1.0e-4, 1.0e-5, 1.0e-6})
    for (double beta : {0.1, 0.3, 0.45})
      for (int pm : {25, 58, 100}) {
        const bbs::LogTable L = logs(alpha, beta);
        const double c1 = (L.l01 - L.l00) * 1.4426950408889634,
                     c2 = (L.l11 - L.l10) * 1.4426950408889634;
        auto t = [&](int d, int m) {
          return 72.0 * 1.4426950408889634 + (m - pm) * c2 + d * c1;
        };
        for (int target = 100; target <= 116; target++) {
          // the node nearest to the target, and one either side of -126
          int bd = -1, bm = 0, nd[2] = {-1, -1}, nm[2] = {0, 0};
          for (int m = 0; m <= pm; m++)
            for (int d = 0; d <= 40; d++) {
              const double v = t(d, m);
              if (std::fabs(v + target) < 0.5 &&
                  (bd < 0 || std::fabs(v + target) < std::fabs(t(bd, bm) + target))) {
                bd = d;
                bm = m;
              }
              for (int s = 0; s < 2; s++) {
                const double off = s ? v + 126.0 : -126.0 - v;
                const double old =
                    nd[s] < 0 ? 1e9 : std::fabs(t(nd[s], nm[s]) + 126.0);
                if (off > 0.0 && off < old) {
                  nd[s] = d;
                  nm[s] = m;
                }
              }
            }
          if (bd < 0) continue;
          for (int s = 0; s < 2; s++)
            for (int others : {1, 6, 31, 123})
              for (int lift = 0; lift < 2; lift++)
                if (nd[s] >= 0)
                  cases.push_back(far_case(L, 100, pm, bd, bm, nd[s], nm[s],
                                           others, lift != 0));
        }
      }
  // a cell of 32 zeros and 58 ones at alpha 1e-4, beta 0.3
  for (int others : {1, 6})
    cases.push_back(far_case(logs(1.0e-4, 0.3), 32, 58, 1, 41, 0, 40, others, false));
}

// Four cells per lane, a node moved from one branch to another: lane 0's cells
// have 60 of their 120 mutations in either, `lose` other lanes' lose `down`.
Case high_case(int lose, int down) {
  const bbs::LogTable L = logs(1.0e-20, 0.2);
  Case c = empty_case(4, 8, 128, L);
  for (int q = 0; q < 4; q++)
    for (int lane = 0; lane < 32; lane++) {
      const size_t at = (size_t)q * 32 + lane;
      const bool gains = lane == 0, loses = lane > 0 && lane <= lose;
      c.pm[at] = gains || loses ? 120.0f : 0.0f;
      c.entry[(size_t)0 * 128 + at] = field(0, gains ? 60 : loses ? 120 : 0);
      c.entry[(size_t)1 * 128 + at] = field(0, gains ? 60 : 0);
      c.entry[(size_t)2 * 128 + at] = field(0, loses ? down : 0);
    }
  c.x.a0 = 1;
  c.x.b0 = 2;
  c.x.a1 = c.x.b1 = 7;
  c.list = {0};
  c.nv = c.nc = 1;
  return c;
}

void high_cases(std::vector<Case> &cases) {
  for (int lose : {0, 1, 31})
    for (int down : {1, 60}) cases.push_back(high_case(lose, down));
}

}  // namespace

int main(int argc, char **argv) {
  const std::string kind = argc > 1 ? argv[1] : "";
  std::vector<Case> cases;
  if (kind == "far") far_cases(cases);
  if (kind == "high") high_cases(cases);
  if (cases.empty()) return 2;

  // everything in one allocation each
  std::vector<uint32_t> tables;
  std::vector<uint8_t> lists;
  std::vector<float> cells;
  std::vector<size_t> at_t, at_l, at_f;
  for (const Case &c : cases) {
    const int nw = (c.q + 1) / 2;
    at_t.push_back(tables.size());
    for (int j = 0; j < c.n; j++)
      for (int lane = 0; lane < 32; lane++)
        for (int w = 0; w < nw; w++) {
          uint32_t v = 0;
          for (int h = 0; h < 2 && 2 * w + h < c.q; h++)
            v |= (uint32_t)c.entry[((size_t)j * c.q + 2 * w + h) * 32 + lane]
                 << (16 * h);
          tables.push_back(v);
        }
    at_l.push_back(lists.size());
    lists.insert(lists.end(), c.list.begin(), c.list.end());
    at_f.push_back(cells.size());
    for (int q = 0; q < c.q; q++)
      for (int k = 0; k < 2; k++)
        for (int lane = 0; lane < 32; lane++)
          cells.push_back((k ? c.pm : c.pd)[(size_t)q * 32 + lane]);
  }
  uint32_t *d_t;
  uint8_t *d_l;
  float *d_f;
  Result *d_r;
  if (cudaMalloc(&d_t, 4 * tables.size()) != cudaSuccess ||
      cudaMalloc(&d_l, lists.size()) != cudaSuccess ||
      cudaMalloc(&d_f, 4 * cells.size()) != cudaSuccess ||
      cudaMalloc(&d_r, sizeof(Result) * cases.size()) != cudaSuccess)
    return 2;
  cudaMemcpy(d_t, tables.data(), 4 * tables.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(d_l, lists.data(), lists.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(d_f, cells.data(), 4 * cells.size(), cudaMemcpyHostToDevice);
  for (size_t i = 0; i < cases.size(); i++) {
    const Case &c = cases[i];
    (c.q == 1 ? launch<1> : launch<4>)(c, d_t + at_t[i], d_l + at_l[i],
                                       d_f + at_f[i], d_r + i);
  }
  std::vector<Result> res(cases.size());
  if (cudaMemcpy(res.data(), d_r, sizeof(Result) * cases.size(),
                 cudaMemcpyDeviceToHost) != cudaSuccess) {
    std::printf("FAIL %s\n", cudaGetErrorString(cudaGetLastError()));
    return 2;
  }
  int bad = 0;
  for (size_t i = 0; i < cases.size(); i++) {
    const Case &c = cases[i];
    const Result &r = res[i];
    const double tol = tolerance(c, r);
    for (int k = 0; k < 2; k++) {
      const double bound = r.up[k] * 0.6931471805599453 / bbs::kBoundUnit + tol;
      const double change = r.after[k] - r.before[k];
      // (written so that a bound that is no number fails)
      if (!(bound >= change) && bad++ < 20)
        std::printf("FAIL %s case %zu: %s changes by %.4f, bound %.4f\n",
                    kind.c_str(), i, k ? "max score" : "score",
                    change, bound);
      // a bound that bounds something: near the change where nothing saturates
      if (kind == "far" && !(bound <= change + 40.0) && bad++ < 20)
        std::printf("FAIL case %zu: a loose bound, %.4f for %.4f\n", i, bound,
                    change);
    }
  }
  if (bad) {
    std::printf("%d of %zu cases\n", bad, cases.size());
    return 1;
  }
  std::printf("bound ok %zu\n", cases.size());
  return 0;
}
