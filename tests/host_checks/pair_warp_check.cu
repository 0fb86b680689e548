// Host-side check of the warp-per-unit pair form's index arithmetic
// (doci_gb300/csrc/pair_warp_index.cuh), compiled by nvcc and run on the CPU:
// the unit list, row starts and insertion tables the library builds, the
// kernel's formulas applied to them (own row start + table offset / 4, row
// start of R' u b + c), every neighbour rank recomputed from first principles.
// Every set visits each orbital outside it exactly once at the right rank;
// over a whole space every determinant is reached N times and lies in exactly
// one unit's own row.
//   usage: pair_warp_check L N P [unit_stride] [set_stride]
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../doci_gb300/csrc/pair_warp_index.cuh"

constexpr int BC = 35;
static uint64_t binom(unsigned n, unsigned k) {
  if (k > n) return 0;
  uint64_t r = 1;
  for (unsigned d = 1; d <= k; ++d) r = r * (n - k + d) / d;
  return r;
}
static uint64_t direct_rank_mirrored(uint32_t M, int L, int N) {
  uint64_t s = 0;
  int e = 0;
  for (int o = 0; o < L; ++o)
    if (M >> (L - 1 - o) & 1u) {
      s += binom(L - 1 - o, N - e);
      ++e;
    }
  return binom(L, N) - 1 - s;
}

int main(int argc, char **argv) {
  if (argc < 4) return 2;
  const int L = std::atoi(argv[1]), N = std::atoi(argv[2]), P = std::atoi(argv[3]);
  const int us = argc > 4 ? std::atoi(argv[4]) : 1, ss = argc > 5 ? std::atoi(argv[5]) : 1;
  const int na = L - P;
  std::vector<uint32_t> B(33 * BC, 0);
  for (int n = 0; n <= 32; ++n)
    for (int k = 0; k < BC; ++k) B[n * BC + k] = static_cast<uint32_t>(binom(n, k));
  const uint64_t D = binom(L, N);
  std::vector<uint16_t> a, b;
  std::vector<uint32_t> off;
  doci::pw::build_tables(P, B.data(), BC, a, b, off);
  const doci::pw::Groups g = doci::pw::groups(P, na, N, B.data(), BC);
  const bool full = us == 1 && ss == 1;
  std::vector<uint8_t> hits(full ? D : 0, 0), owned(full ? D : 0, 0);
  uint64_t bad = 0, sets = 0, entries = 0;
  uint32_t prev_n = ~0u;
  for (int k = 0; k < g.n; ++k) {
    const int jp = N - 1 - g.kp[k];
    const uint32_t n_s = jp >= 0 ? B[P * BC + jp] : 0;
    const uint32_t n_own = jp + 1 <= P ? B[P * BC + jp + 1] : 0;
    if (n_s > prev_n || (g.first[k] & 3u)) ++bad;
    prev_n = n_s;
    for (uint32_t i = 0; i < g.count[k]; i += us) {
      const uint32_t mask = doci::dev::colex_unrank<BC>(i, na, g.kp[k], B.data());
      ++entries;
      if (__builtin_popcount(mask) != g.kp[k] || mask >> na) ++bad;
      const uint32_t own = n_own ? doci::pw::row_start(mask, P, na, N, static_cast<uint32_t>(D), B.data(), BC) : 0;
      if (n_own && (own == doci::pw::kNone || own + static_cast<uint64_t>(n_own) > D)) ++bad;
      if (full)
        for (uint32_t c = 0; c < n_own; ++c) ++owned[own + c];
      for (uint32_t c = 0; c < n_s; c += ss) {
        const uint32_t S = doci::dev::colex_unrank<BC>(n_s - 1 - c, P, jp, B.data()) | (mask << P);
        ++sets;
        for (int o = 0; o < 12; ++o) {
          const uint32_t e = o < 8 ? a[8 * (off[jp] + c) + o] : b[4 * (off[jp] + c) + o - 8];
          const bool hole = o < P && !(S >> o & 1u);
          if (!hole) {
            if (e != doci::pw::sentinel(P)) ++bad;
            continue;
          }
          if (e / 4 >= n_own || e % 4) { ++bad; continue; }
          if (own + e / 4 != direct_rank_mirrored(S | (1u << o), L, N)) ++bad;
          else if (full) ++hits[own + e / 4];
        }
        for (int r = 0; r < na; ++r) {
          if (mask >> r & 1u) continue;
          const uint64_t at = static_cast<uint64_t>(
              doci::pw::row_start(mask | (1u << r), P, na, N, static_cast<uint32_t>(D), B.data(), BC)) + c;
          if (at >= D || at != direct_rank_mirrored(S | (1u << (P + r)), L, N)) ++bad;
          else if (full) ++hits[at];
        }
      }
    }
  }
  if (full)
    for (uint64_t t = 0; t < D; ++t) bad += (hits[t] != N) + (owned[t] != 1);
  std::printf("L=%d N=%d P=%d units=%llu sets=%llu bad=%llu\n", L, N, P, static_cast<unsigned long long>(entries),
              static_cast<unsigned long long>(sets), static_cast<unsigned long long>(bad));
  return bad ? 1 : 0;
}
