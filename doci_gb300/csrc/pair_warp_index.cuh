// pair_warp_index.cuh -- tiling and tables of the warp-per-unit pair form
// (sigma_pair_warp.cu), shared with its host-side index check.
//
// Mirrored orbitals [0, P) are the column part, [P, L) the row part.  A unit
// is the row part R' (a mask over the na = L - P row orbitals, kp elements) of
// the (N-1)-pair sets; its sets run over the jp = N - 1 - kp subsets of the
// column orbitals (column c = C(P, jp) - 1 - colex).  Its own row R' (jp + 1
// column elements) holds S u a for a in the column part, the rows R' u b (jp
// column elements, the set's own column c) those with a row-part hole b.
#pragma once

#include <cstdint>
#include <vector>

#include "addressing.cuh"

namespace doci {
namespace pw {

constexpr uint32_t kNone = 0xffffffffu;

// Row buffers of a warp in shared memory: C(P, P/2) elements and one cell past
// them (the last) that stands for an orbital already in the set.
__host__ __device__ constexpr int cells(int P) { return P >= 12 ? 1024 : P >= 10 ? 256 : 128; }
__host__ __device__ constexpr uint32_t sentinel(int P) { return (static_cast<uint32_t>(cells(P)) - 1u) * 4u; }

// Insertion table by set and orbital: the byte offset (element x 4) of S u o in
// the own row, sentinel(P) when o is in S or no column orbital.  Eight u16 of
// orbitals 0..7 per set in `a` and, for P > 8, four of orbitals 8..11 in `b`;
// the sets of jp elements start at off[jp] (off has P + 2 entries), padded to
// whole warps with sets whose every entry is the sentinel.
__host__ __device__ constexpr uint32_t padded(uint32_t n) { return (n + 31u) & ~31u; }
inline void build_tables(int P, const uint32_t *B, int stride, std::vector<uint16_t> &a, std::vector<uint16_t> &b,
                         std::vector<uint32_t> &off) {
  off.assign(P + 2, 0);
  for (int j = 0; j <= P; ++j) off[j + 1] = off[j] + padded(B[P * stride + j]);
  a.assign(8 * static_cast<size_t>(off[P + 1]), static_cast<uint16_t>(sentinel(P)));
  b.assign(4 * static_cast<size_t>(off[P + 1]), static_cast<uint16_t>(sentinel(P)));
  for (uint32_t M = 0; M < (1u << P); ++M) {
    uint32_t s = 0;
    int j = 0;
    for (int d = 0; d < P; ++d)
      if (M >> d & 1u) s += B[d * stride + (++j)];
    const size_t at = off[j] + (B[P * stride + j] - 1 - s);
    for (int o = 0; o < P; ++o) {
      if (M >> o & 1u) continue;
      uint32_t t = 0;
      int k = 0;
      for (int d = 0; d < P; ++d)
        if ((M | (1u << o)) >> d & 1u) t += B[d * stride + (++k)];
      const uint32_t pos = 4u * (B[P * stride + k] - 1 - t);
      if (o < 8) a[8 * at + o] = static_cast<uint16_t>(pos);
      else b[4 * at + o - 8] = static_cast<uint16_t>(pos);
    }
  }
}

// start of the row with row part `mask` (kNone when it has no column sets)
DOCI_HD uint32_t row_start(uint32_t mask, int P, int na, int N, uint32_t D, const uint32_t *B, int stride) {
  uint32_t base = 0;
  int k = 0;
  for (int a = 0; a < na; ++a) k += static_cast<int>(mask >> a & 1u);
  const int j = N - k;
  if (j < 0 || j > P) return kNone;
  int t = 0;
  for (int a = 0; a < na; ++a)
    if (mask >> a & 1u) {
      base += B[(P + a) * stride + j + t + 1];
      ++t;
    }
  return D - base - B[P * stride + j];
}

// The unit list: the row-part sizes kp by decreasing number of sets (equal
// ones by increasing kp), last the rows without a column element (kp = N: no
// sets, only their diagonal), each size's masks in colex order, padded to a
// multiple of four (four units of one size share the tiles).
struct Groups {
  int n = 0;
  int kp[34];
  uint32_t first[35];  // first entry of the group in the list
  uint32_t count[34];  // masks of the group
};
inline Groups groups(int P, int na, int N, const uint32_t *B, int stride) {
  Groups g;
  for (int kp = 0; kp <= na && kp <= N; ++kp)
    if (N - 1 - kp <= P) g.kp[g.n++] = kp;
  auto sets = [&](int kp) { return N - 1 - kp < 0 ? 0u : B[P * stride + N - 1 - kp]; };
  for (int i = 1; i < g.n; ++i)
    for (int j = i; j > 0 && sets(g.kp[j]) > sets(g.kp[j - 1]); --j) {
      const int t = g.kp[j];
      g.kp[j] = g.kp[j - 1];
      g.kp[j - 1] = t;
    }
  uint32_t at = 0;
  for (int i = 0; i < g.n; ++i) {
    g.first[i] = at;
    g.count[i] = B[na * stride + g.kp[i]];
    at += (g.count[i] + 3u) & ~3u;
  }
  g.first[g.n] = at;
  return g;
}

// Column orbitals of an (L, N) space for `slots` tile rows in flight, and the unit
// list (0: fewer than 10 orbitals).  The more the fewer units: 12 as long as that
// leaves four units per tile row, else 10 as long as it leaves one and a half (with
// 1.36 the second round keeps a third of the rows busy: FP32 L=22 N=7 30.0 us, with
// 8 24.6; with 1.56 both take 30.8 at L=22 N=8, with 2.1 10 is the faster, 37.0
// against 43.0 at L=22 N=11), else 8; but no
// more than 20 row orbitals, whose row starts take 4 MiB.  (That bounds only
// spaces of few pairs or holes, up to 35,960 determinants, which run from their
// neighbour table unless asked: L=32, N=2 would have 2^24 row starts for its 496
// determinants.)
constexpr int kMaxRowOrbitals = 20;
inline int column_orbitals(int L, int N, uint32_t slots, const uint32_t *B, int stride, Groups *g) {
  int P = 0;
  for (int p : {12, 10, 8}) {
    if (L - p < 2 || L - p > kMaxRowOrbitals) continue;
    P = p;
    *g = groups(P, L - P, N, B, stride);
    if (g->first[g->n] / 2 >= (p == 12 ? 8 : 3) * slots) break;
  }
  return P;
}

}  // namespace pw
}  // namespace doci
