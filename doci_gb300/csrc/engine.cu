// engine.cu -- block Davidson for many Hamiltonians at once, device-resident.
//
// The batch engine behind doci_batch_solve, doci_solve_roots and the request
// server's solves (no counterpart in the reference, whose Davidson is
// single-root and single-problem: davidson.c:33-128).  Every problem of a
// batch advances in lockstep: one iteration is a fixed sequence of batched
// launches, each covering all problems at once through a shared work space
// of determinant tiles (sigma) and vector chunks (the vector passes):
//
//   subspace eigenproblem (one block per problem, Jacobi in FP64)
//   -> thick restart where the basis is full (deflation pass)
//   -> residuals and diagonal-preconditioned corrections of every root
//   -> convergence / stall decisions (one thread per problem)
//   -> classical Gram-Schmidt of each correction of an unconverged root
//      against the basis, a second pass when the first leaves less than half
//      of its norm (projection passes with FP64 sums)
//   -> sigma of the new basis vectors (one multi-problem, multi-vector pass)
//   -> the new columns of the subspace matrices.
//
// All control lives on the device (basis sizes, active roots, flags), so the
// host only replays the iteration -- captured once as a CUDA graph -- and
// reads one flag per problem after it.  Per-problem arithmetic never depends
// on the other problems of the batch: a problem's determinants and vector
// chunks are the same whatever else runs, every reduction finishes in a fixed
// order (per-chunk partial rows summed by the problem's last chunk to
// finish), and the batched sigma has no atomics -- so a result is
// bit-identical alone and in any batch.  Large problems (from 2^22
// determinants, or as the shape's autotuning decides) take their sigmas from
// the single-problem kernels (launch_sigma: the pair form for FP32) on
// staging buffers instead (each on one of up to eight streams forked from
// and joined back into the engine's stream, so that several problems'
// kernels overlap); their results still do not depend on the batch,
// but the FP32 pair form's atomic adds make their last bits vary from run to
// run.  Mixed mode: an FP32 phase on H - s (s = the lowest diagonal
// element; FP32 basis, sigma and vector arithmetic with FP64 sums), ending at
// mixed_tol or when the largest residual has not reached a new minimum for
// 15 iterations, then the FP64 phase from its Ritz vectors.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "addressing.cuh"
#include "engine.h"
#include "internal.h"
#include "warp_sums.cuh"

namespace doci {
namespace {

constexpr int kET = 256;                // threads per block of the batched passes
// vector-pass elements per thread of a problem of D determinants (FP32 partial
// sums over them): a chunk is kET times that.  Small problems take short
// chunks, for blocks on more SMs (12 problems of L=12..18 are 15 chunks of 32
// per thread); large ones long ones, whose block sums (2 us of FP64 adds) are
// then small against their reads.
__host__ __device__ constexpr int elems_per_thread(uint32_t D) { return D < (1u << 19) ? 4 : 32; }
constexpr int kMaxR = 8;                // roots
constexpr int kMaxV = 32;               // basis vectors

struct EProb {
  uint32_t D;
  int L, N, nh;
  const uint32_t *nbr;  // neighbour table (small spaces; sigma.cu), or null
  const void *K;        // mirrored K (32 x 32) in the phase's type
  const void *diag_s;   // the sigma's diagonal in the phase's type (FP32 phase: diag - shift)
  const double *diag;   // FP64 diagonal (preconditioner)
  double shift;         // the operator is H - shift
  void *V, *VA, *T;     // basis and its sigmas (D x maxv), corrections (D x R), phase's type
  double *X;            // Ritz vectors (D x R, FP64)
  uint32_t tile0, chunk0, nchunks;
  int max_its;          // this problem's iteration limit in the phase
  int eper;             // vector-pass elements per thread (elems_per_thread)
  int dpt;              // sigma tile: kET * dpt determinants, dpt per thread (autotuned per shape)
};

struct EState {
  int m, m0, its, done, converged, stall, restart, kk, nact, pend, sigmas, idx0, need2;
  int act[kMaxR];
  double best, n0, scale;
  double res[kMaxR];
  double w[kMaxV];
  double c[kMaxV];
  double S[kMaxV * kMaxV];  // subspace matrix, column-major, leading dimension kMaxV
  double Y[kMaxV * kMaxV];  // its eigenvectors (columns), ascending eigenvalues w
};

struct EArgs {
  int n, R, maxv, keep, max_its, stall_window;
  double tol;
  EProb *P;
  EState *St;
  const uint32_t *tile0;   // n + 1 prefix offsets (sigma tiles)
  const uint32_t *chunk0;  // n + 1 prefix offsets (vector chunks)
  int ldp;                 // partial-row length: kMaxV + 2 or R kMaxV
  double *part;            // chunk x ldp partial rows
  unsigned *cnt;           // per-problem arrival counters (zero between passes)
  const uint32_t *binom;
  int *flags;              // per problem: 1 while running (host reads it)
};

// the problem that owns global index b of a prefix table (n + 1 entries)
__device__ __forceinline__ int owner(const uint32_t *pre, int n, uint32_t b) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(pre + mid) <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

template <typename S>
__device__ __forceinline__ S *colp(void *base, uint32_t D, int c) {
  return static_cast<S *>(base) + static_cast<size_t>(c) * D;
}

// Per-chunk sums of NK values (the block's threads each hold acc[k]) into the
// chunk's partial row from column `first` on, NK of `width` values by this
// block and the others by `groups` - 1 other blocks of the chunk; the
// problem's last block to arrive sums the rows in chunk order into
// out[0..width) and returns true (in every thread of that block).  Results do
// not depend on timing or on the other problems.
template <int NK, typename S>
__device__ bool chunk_reduce(S (&acc)[NK], int width, const EArgs &a, const EProb &pb, int p, uint32_t chunk,
                             double *out, int first = 0, int groups = 1) {
  __shared__ double red[kET / 32][NK];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  warp_sums<NK>(acc, red[warp]);
  __syncthreads();
  double *row = a.part + static_cast<size_t>(pb.chunk0 + chunk) * a.ldp + first;
  if (threadIdx.x < NK && first + static_cast<int>(threadIdx.x) < width) {
    double s = 0;
    for (int w = 0; w < kET / 32; ++w) s += red[w][threadIdx.x];
    row[threadIdx.x] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(a.cnt + p, 1u) == pb.nchunks * groups - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  // up to 16 threads per output, each over every such row, then over the
  // threads in order: the order depends only on the problem's chunk count and
  // the width.  (One warp per output and a shuffle tree took seven of the
  // Gram-Schmidt step's 25 us: nine outputs per warp, one after the other.)
  __shared__ double part[kET];
  const double *r0 = a.part + static_cast<size_t>(pb.chunk0) * a.ldp;
  const int fit = width < kET ? kET / width : 1, per = fit < 16 ? fit : 16;
  for (int k0 = 0; k0 < width; k0 += kET) {
    const int w = width - k0 < kET ? width - k0 : kET, k = threadIdx.x % w, g = threadIdx.x / w;
    double s = 0;
    if (g < per) {
#pragma unroll 8
      for (uint32_t c = g; c < pb.nchunks; c += per) s += __ldcg(r0 + static_cast<size_t>(c) * a.ldp + k0 + k);
    }
    part[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x < w) {
      for (int i = 1; i < per; ++i) s += part[i * w + threadIdx.x];
      out[k0 + threadIdx.x] = s;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) a.cnt[p] = 0;
  __syncthreads();
  return true;
}

// ---------------------------------------------------------------- sigma
// VA[:, m0 + v] = (H - shift) V[:, m0 + v] for the v < m - m0 new basis
// vectors of every running problem: a tile of kET * dpt determinants per
// block (dpt per thread, a per-shape choice of the tile autotuner), the
// neighbours by the prefix-sum ranks of addressing.cuh, every vector at once.
// The tile shape changes no arithmetic: each determinant's sum is the same.
template <typename S, int NH>
__global__ void __launch_bounds__(kET) eng_sigma(EArgs a) {
  __shared__ uint32_t B[kBinomRows * kBinomCols];
  for (int t = threadIdx.x; t < kBinomRows * kBinomCols; t += kET) B[t] = a.binom[t];
  __syncthreads();
  if (blockIdx.x >= __ldg(a.tile0 + a.n)) return;
  const int p = owner(a.tile0, a.n, blockIdx.x);
  const EProb &pb = a.P[p];
  const EState &st = a.St[p];
  if (st.done) return;
  const int m0 = st.m0, nv = st.m - st.m0;
  if (nv <= 0) return;
  const S *K = static_cast<const S *>(pb.K);
  const S *x = colp<S>(pb.V, pb.D, m0);
  S *y = colp<S>(pb.VA, pb.D, m0);
  const uint32_t tile_first = (blockIdx.x - pb.tile0) * kET * pb.dpt + threadIdx.x;
  for (int e = 0; e < pb.dpt; ++e) {
  const uint32_t r = tile_first + e * kET;
  if (r >= pb.D) return;
  struct Acc {
    const S *K, *x;
    uint32_t D;
    int nv;
    const S *Krow;
    S acc[kMaxR];
    __device__ __forceinline__ void begin(int m) { Krow = K + m * 32; }
    __device__ __forceinline__ void hop(int, int q, uint32_t idx) {
      const S kv = __ldg(Krow + q);
#pragma unroll
      for (int v = 0; v < kMaxR; ++v)
        if (v < nv) acc[v] += kv * __ldg(x + static_cast<size_t>(v) * D + idx);
    }
  } f{K, x, pb.D, nv, K, {}};
  const S d = static_cast<const S *>(pb.diag_s)[r];
#pragma unroll
  for (int v = 0; v < kMaxR; ++v)
    if (v < nv) f.acc[v] = d * x[static_cast<size_t>(v) * pb.D + r];
  if (pb.nbr) {  // the same hops in the same order, from the table
    const int hops = pb.N * pb.nh;
    const uint32_t *t = pb.nbr + r;
    constexpr int kB = 4;
    for (int h = 0; h < hops; h += kB, t += static_cast<size_t>(kB) * pb.D) {
      uint32_t en[kB];
#pragma unroll
      for (int i = 0; i < kB; ++i) en[i] = h + i < hops ? __ldg(t + static_cast<size_t>(i) * pb.D) : 0u;
#pragma unroll
      for (int i = 0; i < kB; ++i)
        if (h + i < hops) {
          const uint32_t at = en[i] >> 21, m = (at * 1986u) >> 16;  // 33 m + q
          f.Krow = K + 32 * m;
          f.hop(0, static_cast<int>(at - 33 * m), en[i] & 0x1fffffu);
        }
    }
  } else {
    const uint32_t Dm1 = pb.D - 1, R = Dm1 - r;
    const uint32_t M = dev::colex_unrank<kBinomCols>(R, pb.L, pb.N, B);
    dev::Neighbours<NH, kBinomCols> nb;
    nb.precompute(M, R, pb.L, pb.nh, B);
    nb.visit(M, R, Dm1, pb.N, pb.nh, B, f);
  }
#pragma unroll
  for (int v = 0; v < kMaxR; ++v)
    if (v < nv) y[static_cast<size_t>(v) * pb.D + r] = f.acc[v];
  }
}

// ---------------------------------------------------------------- vector passes
// three resident blocks per SM for the FP32 phase's passes (register
// budget 85; at two per SM the projection passes ran at ~2.4 TB/s); the
// FP64 phase's few iterations keep the registers their arrays need
template <typename S>
constexpr int eng_minb() { return sizeof(S) == 4 ? 3 : 1; }

// chunk-local element range of this thread: j = base + e * kET, e < eper
#define ENG_CHUNK_PROLOGUE                                      \
  const int p = owner(a.chunk0, a.n, blockIdx.x);               \
  const EProb &pb = a.P[p];                                     \
  EState &st = a.St[p];                                         \
  const uint32_t chunk = blockIdx.x - pb.chunk0;                \
  const int eper = pb.eper;                                     \
  const uint32_t jbase = chunk * (kET * eper) + threadIdx.x;

// The new columns of the subspace matrix, V_k . VA_i for the i = m0 + j new
// vectors (j < R) and all k <= i: a block takes eight k (blockIdx.y) and four
// j (blockIdx.z), so that a basis vector is read once for four columns;
// products summed over the thread's elements in S, then in FP64 (FP32 ones over
// the warp as pairs of floats: 17 us against 37 with FP64 adds)
constexpr int kCk = 8, kCj = 4;
template <typename S>
__global__ void __launch_bounds__(kET) eng_subcol(EArgs a) {
  ENG_CHUNK_PROLOGUE
  if (st.done) return;
  const int m = st.m, m0 = st.m0, k0 = blockIdx.y * kCk, j0 = blockIdx.z * kCj;
  const S *V = static_cast<const S *>(pb.V) + static_cast<size_t>(k0) * pb.D;
  const S *W = static_cast<const S *>(pb.VA) + static_cast<size_t>(m0 + j0) * pb.D;
  const int nk = m - k0 < kCk ? m - k0 : kCk, nj = m - m0 - j0 < kCj ? m - m0 - j0 : kCj;
  S f[kCj][kCk];
#pragma unroll
  for (int j = 0; j < kCj; ++j)
#pragma unroll
    for (int k = 0; k < kCk; ++k) f[j][k] = S(0);
  if (nk > 0 && nj > 0) {
    for (int e = 0; e < eper; ++e) {
      const uint32_t jj = jbase + e * kET;
      if (jj >= pb.D) break;
      S v[kCk], w[kCj];
#pragma unroll
      for (int k = 0; k < kCk; ++k) v[k] = k < nk ? V[static_cast<size_t>(k) * pb.D + jj] : S(0);
#pragma unroll
      for (int j = 0; j < kCj; ++j) w[j] = j < nj ? W[static_cast<size_t>(j) * pb.D + jj] : S(0);
#pragma unroll
      for (int j = 0; j < kCj; ++j)
        if (j < nj) {
#pragma unroll
          for (int k = 0; k < kCk; ++k) f[j][k] += v[k] * w[j];
        }
    }
  }
  S acc[kCj * kCk];
#pragma unroll
  for (int j = 0; j < kCj; ++j)
#pragma unroll
    for (int k = 0; k < kCk; ++k) acc[j * kCk + k] = f[j][k];
  const int kg = gridDim.y, first = (blockIdx.z * kg + blockIdx.y) * kCj * kCk;
  __shared__ double out[kMaxR * kMaxV];
  if (chunk_reduce<kCj * kCk>(acc, gridDim.z * kg * kCj * kCk, a, pb, p, chunk, out, first, kg * gridDim.z)) {
    for (int t = threadIdx.x; t < (m - m0) * m; t += kET) {
      const int j = t / m, k = t % m, i = m0 + j;
      if (k > i) continue;
      const double v = out[((j / kCj) * kg + k / kCk) * kCj * kCk + (j % kCj) * kCk + k % kCk];
      st.S[i * kMaxV + k] = v;
      st.S[k * kMaxV + i] = v;
    }
  }
}

// residuals of up to four roots q0.. (blockIdx.y) in one read of V and VA:
// x = V y, r = VA y - theta x, t = r / |diag - shift - theta| (cutoff 1e-12,
// davidson.c:214-227); sums |r|^2
constexpr int kRq = 4;
template <typename S>
__global__ void __launch_bounds__(kET) eng_residual(EArgs a) {
  ENG_CHUNK_PROLOGUE
  if (st.done) return;
  const int m = st.m, q0 = blockIdx.y * kRq, nr = a.R < m ? a.R : m;
  const int nq = nr - q0 < kRq ? nr - q0 : kRq;
  __shared__ S ys[kMaxV][kRq];
  for (int t = threadIdx.x; t < kMaxV * kRq; t += kET) {
    const int k = t / kRq, q = t % kRq;
    ys[k][q] = (k < m && q < nq) ? static_cast<S>(st.Y[(q0 + q) * kMaxV + k]) : S(0);
  }
  __syncthreads();
  const S *V = static_cast<const S *>(pb.V), *VA = static_cast<const S *>(pb.VA);
  S f[kRq];
#pragma unroll
  for (int q = 0; q < kRq; ++q) f[q] = S(0);
  for (int e = 0; e < eper && nq > 0; ++e) {
    const uint32_t jj = jbase + e * kET;
    if (jj >= pb.D) break;
    S xv[kRq], av[kRq];
#pragma unroll
    for (int q = 0; q < kRq; ++q) xv[q] = av[q] = S(0);
    const S *vp = V + jj, *ap = VA + jj;
#pragma unroll 8
    for (int k = 0; k < m; ++k) {
      const S v = vp[static_cast<size_t>(k) * pb.D], w = ap[static_cast<size_t>(k) * pb.D];
#pragma unroll
      for (int q = 0; q < kRq; ++q) {
        xv[q] += v * ys[k][q];
        av[q] += w * ys[k][q];
      }
    }
    const double d = pb.diag[jj];
#pragma unroll
    for (int q = 0; q < kRq; ++q)
      if (q < nq) {
        const double th = st.w[q0 + q];
        const S r = av[q] - static_cast<S>(th) * xv[q];
        f[q] += r * r;
        const S dd = static_cast<S>(fabs(d - (th + pb.shift)));
        colp<S>(pb.T, pb.D, q0 + q)[jj] = dd > S(1e-12) ? r / dd : r / S(1e-12);
      }
  }
  __shared__ double out[kMaxR];
  if (chunk_reduce<kRq>(f, gridDim.y * kRq, a, pb, p, chunk, out, q0, gridDim.y))
    if (static_cast<int>(threadIdx.x) < nr) st.res[threadIdx.x] = sqrt(out[threadIdx.x]);
}

// One step of the Gram-Schmidt orthogonalisation of the corrections t_q =
// T[:, act[q]], in one read of the basis: t_q -= sum_k c_k V_k with the
// projections c of the step before, then the sums t_q.t_q and V_k.t_q, and for
// the next correction t_{q+1}.t_{q+1}, V_k.t_{q+1} and t_q.t_{q+1} (q = -1: only
// those of t_0).  When t_q keeps more than half of its norm (the Daniel-Gragg-
// Kaufman-Stewart test) it becomes the basis vector V_m = t_q / |t_q|, whose
// projection on t_{q+1} is t_q.t_{q+1} / |t_q|: the next step starts from these
// and writes V_m on its way.  Otherwise the step runs a second time (`pass` 2)
// with the new projections.
// A step is bound by its latency (launch, one round of loads, the block's sums,
// the last block's), so it does all that the data in its registers allow: a
// projection and an update pass per correction, a pass writing the vector and
// one counting it took 12 problems of up to 32 vectors 52 us per correction, 32
// so (FP32 phase).
template <typename S, int KM>
__global__ void __launch_bounds__(kET, sizeof(S) == 4 ? 2 : 1) eng_gs(EArgs a, int q, int pass) {
  ENG_CHUNK_PROLOGUE
  if (st.done || q >= st.nact) return;
  if (pass == 2 && !st.need2) return;
  const int m = st.m, pend = pass == 1 ? st.pend : -1;
  const bool own = q >= 0, next = q + 1 < st.nact;
  __shared__ S cs[KM];
  if (threadIdx.x < KM) cs[threadIdx.x] = (own && threadIdx.x < m) ? static_cast<S>(st.c[threadIdx.x]) : S(0);
  __syncthreads();
  S *V = static_cast<S *>(pb.V);
  S *t = colp<S>(pb.T, pb.D, own ? st.act[q] : 0);
  const S *tn = colp<S>(pb.T, pb.D, next ? st.act[q + 1] : 0), *tp = colp<S>(pb.T, pb.D, pend >= 0 ? st.act[pend] : 0);
  const S psc = pend >= 0 ? static_cast<S>(st.scale) : S(0);
  constexpr int NK = 3 + 2 * KM;  // t.t, tn.tn, t.tn, then per column V.t, V.tn
  S f[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) f[k] = S(0);
  for (int e = 0; e < eper; ++e) {
    const uint32_t jj = jbase + e * kET;
    if (jj >= pb.D) break;
    S tv = own ? t[jj] : S(0);
    const S nv = next ? tn[jj] : S(0);
    const S pv = pend >= 0 ? tp[jj] * psc : S(0);
    S v[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k)
      if (k < m) v[k] = (pend >= 0 && k == m - 1) ? pv : V[static_cast<size_t>(k) * pb.D + jj];
    if (pend >= 0) V[static_cast<size_t>(m - 1) * pb.D + jj] = pv;
    if (own) {
#pragma unroll
      for (int k = 0; k < KM; ++k)
        if (k < m) tv -= cs[k] * v[k];
      t[jj] = tv;
    }
    f[0] += tv * tv;
    f[1] += nv * nv;
    f[2] += tv * nv;
#pragma unroll
    for (int k = 0; k < KM; ++k)
      if (k < m) {
        f[3 + 2 * k] += v[k] * tv;
        f[4 + 2 * k] += v[k] * nv;
      }
  }
  __shared__ double out[NK], scale;
  __shared__ bool settled;
  if (!chunk_reduce<NK>(f, 3 + 2 * m, a, pb, p, chunk, out)) return;
  if (threadIdx.x == 0) {
    settled = true;  // no second pass for t_q
    bool add = false;
    if (own) {
      const double n0 = st.n0, n1 = out[0];
      if (pass == 1) st.need2 = !(n1 > 0.25 * n0);
      settled = pass == 2 || !st.need2;
      // keep the correction if an independent direction is left
      add = settled && n0 > 0 && n1 > 0 && n1 > 1e-20 * n0 && m < a.maxv;
    }
    scale = add ? 1.0 / sqrt(out[0]) : 0.0;
    st.pend = add ? q : -1;
    if (add) {
      st.scale = scale;
      st.m = m + 1;
    }
    if (settled && next) st.n0 = out[1];
  }
  __syncthreads();
  const int k = threadIdx.x;
  if (!settled) {
    if (k < m) st.c[k] = out[3 + 2 * k];
  } else if (next) {
    if (k < m) st.c[k] = out[4 + 2 * k];
    else if (k == m && m < kMaxV) st.c[k] = scale * out[2];
  }
}

// The last step's vector, if it became one; then a basis that did not grow
// ends the solve, else the new vectors get their sigmas.  (A problem whose
// basis did not grow has no vector to write, so its blocks need not agree on
// `done`.)
template <typename S>
__global__ void __launch_bounds__(kET) eng_gs_finish(EArgs a) {
  ENG_CHUNK_PROLOGUE
  if (st.done) return;
  const int m = st.m;
  if (st.pend >= 0) {
    const S *t = colp<S>(pb.T, pb.D, st.act[st.pend]);
    S *out = colp<S>(pb.V, pb.D, m - 1);
    const S sc = static_cast<S>(st.scale);
    for (int e = 0; e < eper; ++e) {
      const uint32_t jj = jbase + e * kET;
      if (jj >= pb.D) break;
      out[jj] = t[jj] * sc;
    }
  }
  if (chunk == 0 && threadIdx.x == 0) {
    if (m == st.m0) {
      st.done = 1;
      a.flags[p] = 0;
    } else {
      st.sigmas += m - st.m0;
    }
  }
}

// thick restart: V[:, c] = sum_k V[:, k] Y[k, c], c < kk, in place (each
// element's row is read before it is written), the same for VA
template <typename S, int KM>
__global__ void __launch_bounds__(kET) eng_deflate(EArgs a) {
  ENG_CHUNK_PROLOGUE
  if (st.done || !st.restart) return;
  const int m = st.m, kk = st.kk;
  __shared__ S Ys[KM * KM];
  for (int i = threadIdx.x; i < KM * KM; i += kET) {
    const int k = i % KM, c = i / KM;
    Ys[i] = (k < m && c < kk) ? static_cast<S>(st.Y[c * kMaxV + k]) : S(0);
  }
  __syncthreads();
  for (int which = 0; which < 2; ++which) {
    S *V = static_cast<S *>(which ? pb.VA : pb.V);
    for (int e = 0; e < eper; ++e) {
      const uint32_t jj = jbase + e * kET;
      if (jj >= pb.D) break;
      S v[KM];
#pragma unroll
      for (int k = 0; k < KM; ++k)
        if (k < m) v[k] = V[static_cast<size_t>(k) * pb.D + jj];
      for (int c = 0; c < kk; ++c) {
        S s = S(0);
#pragma unroll
        for (int k = 0; k < KM; ++k)
          if (k < m) s += v[k] * Ys[c * KM + k];
        V[static_cast<size_t>(c) * pb.D + jj] = s;
      }
    }
  }
}

// X[:, r] = V Y[:, r] (FP64) for r < min(R, m)
template <typename S, int KM>
__global__ void __launch_bounds__(kET) eng_combine(EArgs a) {
  ENG_CHUNK_PROLOGUE
  const int m = st.m, nr = a.R < m ? a.R : m;
  const S *V = static_cast<const S *>(pb.V);
  for (int e = 0; e < eper; ++e) {
    const uint32_t jj = jbase + e * kET;
    if (jj >= pb.D) break;
    for (int r = 0; r < nr; ++r) {
      double s = 0;
#pragma unroll
      for (int k = 0; k < KM; ++k)
        if (k < m) s += static_cast<double>(V[static_cast<size_t>(k) * pb.D + jj]) * st.Y[r * kMaxV + k];
      pb.X[static_cast<size_t>(r) * pb.D + jj] = s;
    }
  }
}

// large problems take their sigmas from the single-problem kernels
// (launch_sigma) on fixed staging buffers: the new basis vectors are copied in
// (xs[v] = V[:, m0 + v], v < m - m0) and the sigmas out (VA[:, m0 + v] = ys[v])
template <typename S>
__global__ void eng_stage(EArgs a, int p, S *xs, const S *ys, int out) {
  const EProb &pb = a.P[p];
  const EState &st = a.St[p];
  if (st.done) return;
  const int m0 = st.m0, nv = st.m - st.m0;
  const size_t n = static_cast<size_t>(nv > 0 ? nv : 0) * pb.D;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    if (out) static_cast<S *>(pb.VA)[static_cast<size_t>(m0) * pb.D + i] = ys[i];
    else xs[i] = static_cast<const S *>(pb.V)[static_cast<size_t>(m0) * pb.D + i];
  }
}

// start vectors: T[:, r] = unit vector on the r-th smallest diagonal element
// (the first on ties; davidson's HF start, executable.c:276-288, extended)
template <typename S>
__global__ void __launch_bounds__(kET) eng_unit(EArgs a) {
  ENG_CHUNK_PROLOGUE
  for (int r = 0; r < a.R; ++r) {
    S *t = colp<S>(pb.T, pb.D, r);
    const int idx = reinterpret_cast<const int *>(st.act)[r];
    for (int e = 0; e < eper; ++e) {
      const uint32_t jj = jbase + e * kET;
      if (jj >= pb.D) break;
      t[jj] = static_cast<int>(jj) == idx ? S(1) : S(0);
    }
  }
}

// ---------------------------------------------------------------- per-problem control
// round r of the start-vector choice: the r-th smallest diagonal element
// (the first index on ties, excluding the r already chosen), stored in
// act[r]; every chunk finds its minimum, the problem's last chunk to arrive
// takes the minimum over the chunks in chunk order
__global__ void __launch_bounds__(kET) eng_lowest(EArgs a, int r) {
  ENG_CHUNK_PROLOGUE
  const int R = a.R < static_cast<int>(pb.D) ? a.R : static_cast<int>(pb.D);
  if (r >= R) return;
  __shared__ double wv[kET / 32];
  __shared__ uint32_t wi[kET / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v = 1e308;
  uint32_t id = 0xffffffffu;
  for (int e = 0; e < eper; ++e) {
    const uint32_t jj = jbase + e * kET;
    if (jj >= pb.D) break;
    bool taken = false;
    for (int q = 0; q < r; ++q) taken |= static_cast<uint32_t>(st.act[q]) == jj;
    const double d = pb.diag[jj];
    if (!taken && (d < v || (d == v && jj < id))) {
      v = d;
      id = jj;
    }
  }
  auto better = [](double v2, uint32_t i2, double v1, uint32_t i1) { return v2 < v1 || (v2 == v1 && i2 < i1); };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double v2 = __shfl_down_sync(0xffffffffu, v, o);
    const uint32_t i2 = __shfl_down_sync(0xffffffffu, id, o);
    if (better(v2, i2, v, id)) {
      v = v2;
      id = i2;
    }
  }
  if (lane == 0) {
    wv[warp] = v;
    wi[warp] = id;
  }
  __syncthreads();
  double *row = a.part + static_cast<size_t>(pb.chunk0 + chunk) * a.ldp;
  if (threadIdx.x == 0) {
    double bv = wv[0];
    uint32_t bi = wi[0];
    for (int w = 1; w < kET / 32; ++w)
      if (better(wv[w], wi[w], bv, bi)) {
        bv = wv[w];
        bi = wi[w];
      }
    row[0] = bv;
    row[1] = static_cast<double>(bi);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(a.cnt + p, 1u) == pb.nchunks - 1;
  __syncthreads();
  if (!last || warp != 0) return;
  __threadfence();
  const double *r0 = a.part + static_cast<size_t>(pb.chunk0) * a.ldp;
  v = 1e308;
  id = 0xffffffffu;
  for (uint32_t c = lane; c < pb.nchunks; c += 32) {
    const double v2 = __ldcg(r0 + static_cast<size_t>(c) * a.ldp);
    const uint32_t i2 = static_cast<uint32_t>(__ldcg(r0 + static_cast<size_t>(c) * a.ldp + 1));
    if (better(v2, i2, v, id)) {
      v = v2;
      id = i2;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double v2 = __shfl_down_sync(0xffffffffu, v, o);
    const uint32_t i2 = __shfl_down_sync(0xffffffffu, id, o);
    if (better(v2, i2, v, id)) {
      v = v2;
      id = i2;
    }
  }
  if (lane == 0) {
    st.act[r] = static_cast<int>(id);
    if (r == 0) st.idx0 = static_cast<int>(id);
    a.cnt[p] = 0;
  }
}

// fresh state of a phase: empty basis, every start vector to be added
__global__ void eng_init_state(EArgs a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.n) return;
  EState &st = a.St[p];
  st.m = st.m0 = st.its = st.done = st.converged = st.stall = st.restart = st.kk = st.sigmas = 0;
  st.pend = -1;
  st.best = 1e300;
  const int R = a.R < static_cast<int>(a.P[p].D) ? a.R : static_cast<int>(a.P[p].D);
  st.nact = R;
  for (int r = 0; r < kMaxR; ++r) {
    st.act[r] = r;
    st.res[r] = 1e300;
  }
  for (int i = 0; i < kMaxV * kMaxV; ++i) st.S[i] = st.Y[i] = 0.0;
  for (int i = 0; i < kMaxV; ++i) st.w[i] = st.c[i] = 0.0;
  a.flags[p] = 1;
}

// The subspace eigenproblem of every running problem: one block, Jacobi in
// FP64 with the round-robin (tournament) ordering: each round rotates n/2
// disjoint index pairs at once, n-1 rounds a sweep, until the off-diagonal
// part is below 1e-30 of the whole; ascending eigenvalues; then the restart
// decision.
//
// The FP64 units (two lanes per clock and SM) bound it, so most of the way is
// gone in FP32: Jacobi on the matrix rounded to FP32, its vectors V made
// orthogonal to FP64 accuracy (with V^T V = 1 + E, E about 1e-6, V (1 - E/2 +
// 3 E^2 / 8) is orthogonal to E^3), and the FP64 Jacobi then starts from V^T A V,
// whose off-diagonal part is about 1e-6 of the whole: two sweeps instead of six
// or seven, with fewer FP64 roundings than those (vectors orthogonal to 5e-15
// instead of 1e-14 at n = 32).
//
// A rotation's tangent, which only steers the convergence, is computed in FP32
// from differences in the matrix's type, the cosine in that type (an FP32
// reciprocal square root and one third-order step for FP64), so that the
// rotations stay orthogonal to its accuracy; and a pair whose square is below
// `skip`, which cannot keep the off-diagonal part above its limit, is left alone.
// Measured on 12 problems of up to 32 vectors (average over a solve): 1,609 us
// with one warp and FP64 tangents, 468 us with 256 threads in FP64 alone, 197 us
// with FP32 sweeps of the FP64 sweeps' form and FP64 sums for the stopping test,
// 163 us so.  At 24 vectors 150 us of FP32 and FP64 sweeps are latency (900
// clocks a round) and FP64 work in about equal parts, 40 us the products.
constexpr int kEigT = 256;
constexpr int kLdA = kMaxV + 1;
constexpr int kHalfV = kMaxV / 2;
constexpr int kPreMinN = 8;  // below, six FP64 sweeps cost less than the way through FP32

template <typename Real>
struct Rotations {  // one round's pairs (twice: this round's and the next one's)
  Real c[2][kHalfV], s[2][kHalfV];
  int p[2][kHalfV], q[2][kHalfV];
};

// pair `k` of a round (n2 = n rounded up to even; with n odd one pair a round
// holds n and is idle)
__device__ __forceinline__ void eig_pair(int n2, int round, int k, int &pp, int &qq) {
  auto player = [&](int i) {  // i - 1 + round modulo n2 - 1, plus one
    const int j = i + round;
    return i == 0 ? 0 : j > n2 - 1 ? j - (n2 - 1) : j;
  };
  const int pl = player(k), ql = player(n2 - 1 - k);
  pp = min(pl, ql);
  qq = max(pl, ql);
}

// the rotation of a pair, without branches (the idle pair's entries are zero)
template <typename Real>
__device__ __forceinline__ void eig_rotation(const Real *A, int pp, int qq, Real skip, Real &cs, Real &sn) {
  const Real apq = A[qq * kLdA + pp];
  // t = sign(d) b / (|d| + sqrt(d^2 + b^2)), d = aqq - app, b = 2 apq (A is
  // scaled to about 1 and apq not below `skip`: no under- or overflow)
  const float d = static_cast<float>(A[qq * kLdA + qq] - A[pp * kLdA + pp]), b = 2 * static_cast<float>(apq);
  const float h = d * d + b * b, tf = __fdividef(d >= 0 ? b : -b, fabsf(d) + h * rsqrtf(h));
  const Real t = tf, u = 1 + t * t;
  Real y = rsqrtf(static_cast<float>(u));
  if constexpr (sizeof(Real) == 8) {  // y has 22 bits; 1/sqrt(u) = y / sqrt(1 - e), e = 1 - u y^2, to e^3
    const Real e = 1 - u * (y * y);
    y += y * (e * (0.5 + 0.375 * e));
  }
  const bool turned = apq * apq > skip;
  cs = turned ? y : Real(1);
  sn = turned ? t * y : Real(0);
}

// off <= stop * tot for the squares of A's off-diagonal part and of all of it
// (A is scaled to about 1: FP32 holds squares of 1e-30 of it); tot is returned
template <typename Real>
__device__ __forceinline__ bool eig_settled(const Real *A, int n, float stop, float (*part)[kEigT / 32], float &tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float off = 0;
  tot = 0;
  for (int c = warp; c < n; c += kEigT / 32) {
    const float v = lane < n ? static_cast<float>(A[c * kLdA + lane]) : 0.f;
    tot += v * v;
    off += lane == c ? 0.f : v * v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    off += __shfl_xor_sync(0xffffffffu, off, o);
    tot += __shfl_xor_sync(0xffffffffu, tot, o);
  }
  if (lane == 0) {
    part[0][warp] = off;
    part[1][warp] = tot;
  }
  __syncthreads();
  off = tot = 0;
#pragma unroll
  for (int w = 0; w < kEigT / 32; ++w) {
    off += part[0][w];
    tot += part[1][w];
  }
  return off == 0 || off <= stop * tot;
}

// The FP32 sweeps: a round is bound by its latency, so it has one barrier.
// Every thread computes the two rotations of its 2 x 2 block (all blocks of a
// pair get the same bits), reads the block from A and writes it to B, which
// change places; the vectors are turned one round behind.
__device__ void eig_jacobi32(float *A, float *B, float *V, int n, float stop, float skip_rel, int sweeps,
                             Rotations<float> &rot, float (*part)[kEigT / 32]) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n2 = n + (n & 1), half = n2 / 2, bi = tid % kHalfV, bj = tid / kHalfV;
  auto turn = [&](int b) {
#pragma unroll
    for (int i = 0; i < kHalfV * 32 / kEigT; ++i) {
      const int k = warp + i * (kEigT / 32);
      if (k >= half || lane >= n) continue;
      const int pp = rot.p[b][k], qq = rot.q[b][k];
      const float c = rot.c[b][k], s = rot.s[b][k];
      const float vp = V[pp * kLdA + lane], vq = V[qq * kLdA + lane];
      V[pp * kLdA + lane] = c * vp - s * vq;
      V[qq * kLdA + lane] = s * vp + c * vq;
    }
  };
  int done = 0;  // rounds so far
  for (int sweep = 0; sweep < sweeps; ++sweep) {
    float tot;
    if (eig_settled<float>(A, n, stop, part, tot)) break;
    const float skip = skip_rel * tot;
    for (int round = 0; round < n2 - 1; ++round, ++done) {
      if (bi < half && bj < half) {  // rows (p, q) of pair i, columns (p, q) of pair j
        int pi, qi, pj, qj;
        float ci, si, cj, sj;
        eig_pair(n2, round, bi, pi, qi);
        eig_pair(n2, round, bj, pj, qj);
        const float a00 = A[pj * kLdA + pi], a01 = A[qj * kLdA + pi], a10 = A[pj * kLdA + qi], a11 = A[qj * kLdA + qi];
        eig_rotation<float>(A, pi, qi, skip, ci, si);
        eig_rotation<float>(A, pj, qj, skip, cj, sj);
        const float x0 = cj * a00 - sj * a01, x1 = sj * a00 + cj * a01;
        const float y0 = cj * a10 - sj * a11, y1 = sj * a10 + cj * a11;
        B[pj * kLdA + pi] = ci * x0 - si * y0;
        B[pj * kLdA + qi] = si * x0 + ci * y0;
        B[qj * kLdA + pi] = ci * x1 - si * y1;
        B[qj * kLdA + qi] = si * x1 + ci * y1;
        if (bi == bj) {
          rot.p[done & 1][bi] = pi;
          rot.q[done & 1][bi] = qi;
          rot.c[done & 1][bi] = ci;
          rot.s[done & 1][bi] = si;
        }
      }
      if (done > 0) turn((done - 1) & 1);
      __syncthreads();
      float *t = A;
      A = B;
      B = t;
    }
  }
  if (done > 0) turn((done - 1) & 1);
  __syncthreads();
}

// The FP64 sweeps on A (symmetric, full) with the vectors V until the
// off-diagonal squares are below `stop` of the whole (at most `sweeps`).
// A round rotates the 2 x 2 blocks of A, one thread per block of the upper
// triangle (its columns and rows at once, the mirror written along) while the
// free warps turn 7/16 of the vectors; then warp 0 computes the next round's
// rotations while the others turn the rest, so that the SM's four quarters have
// about the same FP64 work in both steps.
__device__ void eig_jacobi64(double *A, double *V, int n, float stop, double skip_rel, int sweeps,
                             Rotations<double> &rot, float (*part)[kEigT / 32]) {
  using Real = double;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n2 = n + (n & 1), half = n2 / 2;
  int bi = tid, bj = 1;  // this thread's block of the upper triangle (threads 0 to 127)
  while (bi >= bj && bj < half) bi -= bj++;
  const bool off_block = tid < half * (half - 1) / 2;
  auto turn = [&](int b, int first, int step, int end) {  // the vectors by the pairs first, first + step, ...
    if (lane >= n) return;
#pragma unroll 3
    for (int k = first; k < end; k += step) {
      const int pp = rot.p[b][k], qq = rot.q[b][k];
      const Real c = rot.c[b][k], s = rot.s[b][k];
      const Real vp = V[pp * kLdA + lane], vq = V[qq * kLdA + lane];
      V[pp * kLdA + lane] = c * vp - s * vq;
      V[qq * kLdA + lane] = s * vp + c * vq;
    }
  };
  for (int sweep = 0; sweep < sweeps && n > 1; ++sweep) {
    float tot;
    if (eig_settled<double>(A, n, stop, part, tot)) break;
    const double skip = skip_rel * static_cast<double>(tot);
    auto rotation = [&](int round, int k, int buf) {
      int pp, qq;
      double cs, sn;
      eig_pair(n2, round, k, pp, qq);
      eig_rotation<double>(A, pp, qq, skip, cs, sn);
      rot.p[buf][k] = pp;
      rot.q[buf][k] = qq;
      rot.c[buf][k] = cs;
      rot.s[buf][k] = sn;
    };
    if (tid < half) rotation(0, tid, 0);
    __syncthreads();
    for (int round = 0; round < n2 - 1; ++round) {
      const int b = round & 1;
      if (off_block) {  // rows (p, q) of pair i, columns (p, q) of pair j
        const int pi = rot.p[b][bi], qi = rot.q[b][bi], pj = rot.p[b][bj], qj = rot.q[b][bj];
        const Real ci = rot.c[b][bi], si = rot.s[b][bi], cj = rot.c[b][bj], sj = rot.s[b][bj];
        if (si != 0 || sj != 0) {
          const Real a00 = A[pj * kLdA + pi], a01 = A[qj * kLdA + pi], a10 = A[pj * kLdA + qi], a11 = A[qj * kLdA + qi];
          const Real x0 = cj * a00 - sj * a01, x1 = sj * a00 + cj * a01;
          const Real y0 = cj * a10 - sj * a11, y1 = sj * a10 + cj * a11;
          const Real r00 = ci * x0 - si * y0, r10 = si * x0 + ci * y0;
          const Real r01 = ci * x1 - si * y1, r11 = si * x1 + ci * y1;
          A[pj * kLdA + pi] = A[pi * kLdA + pj] = r00;
          A[pj * kLdA + qi] = A[qi * kLdA + pj] = r10;
          A[qj * kLdA + pi] = A[pi * kLdA + qj] = r01;
          A[qj * kLdA + qi] = A[qi * kLdA + qj] = r11;
        }
      } else if (tid >= 128 && tid < 128 + half) {  // a pair's own block: app + e, aqq - e
        const int k = tid - 128, pp = rot.p[b][k], qq = rot.q[b][k];
        const Real c = rot.c[b][k], s = rot.s[b][k];
        if (s != 0) {
          const Real app = A[pp * kLdA + pp], apq = A[qq * kLdA + pp], aqq = A[qq * kLdA + qq];
          const Real d = aqq - app, g = c * apq, f = g - s * d, e = -s * (f + g);
          A[pp * kLdA + pp] = app + e;
          A[qq * kLdA + pp] = A[pp * kLdA + qq] = c * f - s * (s * apq);
          A[qq * kLdA + qq] = aqq - e;
        }
      }
      const int early = half * 7 / 16;
      if (warp > 4) turn(b, warp - 5, 3, early);
      __syncthreads();
      if (warp == 0) {
        if (lane < half && round + 1 < n2 - 1) rotation(round + 1, lane, 1 - b);
      } else if (warp != 4) {
        turn(b, early + (warp < 4 ? warp - 1 : warp - 2), 6, half);
      }
      __syncthreads();
    }
  }
  __syncthreads();
}

// C = op(A) B for n x n matrices, columns of length kLdA (op: transpose)
template <bool TRANS, typename TA, typename TB, typename Out>
__device__ __forceinline__ void eig_matmul(const TA *A, const TB *B, int n, Out out) {
  const int r0 = threadIdx.x % kHalfV, c0 = threadIdx.x / kHalfV;  // elements (r0 + 0/16, c0 + 0/16)
  double s[2][2] = {{0, 0}, {0, 0}};
  for (int k = 0; k < n; ++k) {
    double a[2], b[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = r0 + i * kHalfV, c = c0 + i * kHalfV;
      a[i] = static_cast<double>(TRANS ? A[r * kLdA + k] : A[k * kLdA + r]);
      b[i] = static_cast<double>(B[c * kLdA + k]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (r0 + i * kHalfV < n && c0 + j * kHalfV < n) s[i][j] += a[i] * b[j];
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (r0 + i * kHalfV < n && c0 + j * kHalfV < n) out(r0 + i * kHalfV, c0 + j * kHalfV, s[i][j]);
}

__global__ void __launch_bounds__(kEigT) eng_eig(EArgs a) {
  const int p = blockIdx.x;
  EState &st = a.St[p];
  if (st.done) return;
  __shared__ double A[kMaxV * kLdA], Vv[kMaxV * kLdA], T[kMaxV * kLdA];
  __shared__ float A32[kMaxV * kLdA], B32[kMaxV * kLdA], V32[kMaxV * kLdA];
  __shared__ Rotations<double> rot;
  __shared__ Rotations<float> rot32;
  __shared__ double sum[kEigT / 32];
  __shared__ float part[2][kEigT / 32];
  __shared__ double wv[kMaxV];
  __shared__ int idx[kMaxV];
  const int n = st.m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double big = 0;
  for (int i = tid; i < kMaxV * kMaxV; i += kEigT) {
    const int r = i % kMaxV, c = i / kMaxV;
    const double v = (r < n && c < n) ? st.S[i] : 0.0;
    A[c * kLdA + r] = v;
    Vv[c * kLdA + r] = (r == c) ? 1.0 : 0.0;
    V32[c * kLdA + r] = (r == c) ? 1.f : 0.f;
    big += fabs(v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) big += __shfl_xor_sync(0xffffffffu, big, o);
  if (lane == 0) sum[warp] = big;
  __syncthreads();
  big = 0;
  for (int w = 0; w < kEigT / 32; ++w) big += sum[w];
  __syncthreads();
  const int ex = big > 0 && big < 1e300 ? ilogb(big) : 0;  // A is scaled to about 1
  for (int i = tid; i < kMaxV * kMaxV; i += kEigT) {
    const int at = i / kMaxV * kLdA + i % kMaxV;
    const double v = scalbn(A[at], -ex);
    A[at] = v;
    A32[at] = static_cast<float>(v);
  }
  __syncthreads();
  if (n >= kPreMinN && big > 0 && big < 1e300) {
    eig_jacobi32(A32, B32, V32, n, 1e-10f, 1e-18f, 12, rot32, part);
    float *E = A32;
    eig_matmul<true>(V32, V32, n, [&](int r, int c, double v) {
      const double e = r == c ? v - 1.0 : v;
      T[c * kLdA + r] = e;
      E[c * kLdA + r] = static_cast<float>(e);
    });
    __syncthreads();
    for (int i = tid; i < n * n; i += kEigT) {  // (E^2 is 1e-12: FP32 does for it)
      const int r = i % n, c = i / n;
      float e2 = 0;
      for (int k = 0; k < n; ++k) e2 += E[k * kLdA + r] * E[c * kLdA + k];
      T[c * kLdA + r] = 0.5 * T[c * kLdA + r] - 0.375 * static_cast<double>(e2);
    }
    __syncthreads();
    eig_matmul<false>(V32, T, n, [&](int r, int c, double v) {
      Vv[c * kLdA + r] = static_cast<double>(V32[c * kLdA + r]) - v;
    });
    __syncthreads();
    eig_matmul<false>(A, Vv, n, [&](int r, int c, double v) { T[c * kLdA + r] = v; });
    __syncthreads();
    eig_matmul<true>(Vv, T, n, [&](int r, int c, double v) {
      if (r <= c) A[c * kLdA + r] = A[r * kLdA + c] = v;
    });
    __syncthreads();
  }
  eig_jacobi64(A, Vv, n, 1e-30f, 1e-34, 100, rot, part);
  if (tid < n) {  // rank of each eigenvalue (ties by index; NaNs, from integrals that are not finite, last)
    auto before = [&](int i, int j) {
      const double wi = A[i * (kLdA + 1)], wj = A[j * (kLdA + 1)];
      const bool ni = isnan(wi), nj = isnan(wj);
      return wi < wj || (!ni && nj) || ((wi == wj || (ni && nj)) && i < j);
    };
    int rank = 0;
    for (int j = 0; j < n; ++j) rank += before(j, tid) ? 1 : 0;
    idx[rank] = tid;
    wv[rank] = scalbn(A[tid * (kLdA + 1)], ex);
  }
  __syncthreads();
  for (int i = warp; i < n; i += kEigT / 32) {
    if (lane < n) st.Y[i * kMaxV + lane] = Vv[idx[i] * kLdA + lane];
  }
  if (tid < n) st.w[tid] = wv[tid];
  if (tid == 0) {
    ++st.its;
    st.restart = n + a.R > a.maxv;
    st.kk = a.keep < n ? a.keep : n;
  }
}

// after a deflation: the basis holds the kk lowest Ritz vectors, so the
// subspace matrix is diag(w) and its eigenvectors the unit vectors
__global__ void eng_after_restart(EArgs a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.n) return;
  EState &st = a.St[p];
  if (st.done || !st.restart) return;
  const int kk = st.kk;
  for (int c = 0; c < kMaxV; ++c)
    for (int r = 0; r < kMaxV; ++r) {
      st.S[c * kMaxV + r] = (r == c && c < kk) ? st.w[c] : 0.0;
      st.Y[c * kMaxV + r] = (r == c && c < kk) ? 1.0 : 0.0;
    }
  st.m = kk;
  st.restart = 0;
}

// convergence (every root's residual <= tol), iteration limit, stall window;
// the unconverged roots become the corrections to add
__global__ void eng_control(EArgs a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.n) return;
  EState &st = a.St[p];
  if (st.done) return;
  const int nr = a.R < st.m ? a.R : st.m;
  double worst = 0;
  int nact = 0;
  for (int r = 0; r < nr; ++r) {
    worst = st.res[r] > worst ? st.res[r] : worst;
    if (st.res[r] > a.tol) st.act[nact++] = r;
  }
  st.nact = nact;
  st.pend = -1;
  st.m0 = st.m;
  if (worst <= a.tol) {
    st.done = 1;
    st.converged = 1;
  } else if (st.its >= a.P[p].max_its) {
    st.done = 1;
  } else if (a.stall_window > 0) {
    if (worst < st.best) {
      st.best = worst;
      st.stall = 0;
    } else if (++st.stall >= a.stall_window) {
      st.done = 1;
    }
  }
  if (st.done) a.flags[p] = 0;
}

// ---------------------------------------------------------------- host side
template <typename T>
struct DBuf {
  T *p = nullptr;
  cudaStream_t st = nullptr;
  int alloc(size_t n, cudaStream_t s) {
    st = s;
    DOCI_CUDA(cudaMallocAsync(&p, sizeof(T) * (n ? n : 1), s));
    return DOCI_OK;
  }
  ~DBuf() {
    if (p) cudaFreeAsync(p, st);
  }
};

inline unsigned nblk(uint64_t n) { return static_cast<unsigned>(n < 1 ? 1 : n); }

constexpr size_t kSideStreams = 8;

// streams forked from the engine's stream and joined back into it
struct SideStreams {
  int n = 0;
  cudaStream_t s[kSideStreams] = {};
  cudaEvent_t fork_ev = nullptr, join_ev[kSideStreams] = {};
  int make(int count) {
    DOCI_CUDA(cudaEventCreateWithFlags(&fork_ev, cudaEventDisableTiming));
    for (int i = 0; i < count; ++i) {
      DOCI_CUDA(cudaStreamCreateWithFlags(&s[i], cudaStreamNonBlocking));
      DOCI_CUDA(cudaEventCreateWithFlags(&join_ev[i], cudaEventDisableTiming));
      n = i + 1;
    }
    return DOCI_OK;
  }
  cudaError_t fork(cudaStream_t st) {
    cudaError_t e = cudaEventRecord(fork_ev, st);
    for (int i = 0; i < n && e == cudaSuccess; ++i) e = cudaStreamWaitEvent(s[i], fork_ev, 0);
    return e;
  }
  cudaError_t join(cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < n && e == cudaSuccess; ++i) {
      e = cudaEventRecord(join_ev[i], s[i]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(st, join_ev[i], 0);
    }
    return e;
  }
  ~SideStreams() {
    for (int i = 0; i < n; ++i) {
      cudaStreamDestroy(s[i]);
      cudaEventDestroy(join_ev[i]);
    }
    if (fork_ev) cudaEventDestroy(fork_ev);
  }
};

// a problem whose sigmas come from launch_sigma (its handle, or the FP32
// phase's shifted view of it) through staging buffers of R vectors
struct BigProb {
  int p;
  const doci_ham *h;
  void *xs, *ys;
  size_t D;
};

template <typename S, int KM, int NH>
int run_phase(EArgs &a, uint32_t ntiles, uint32_t nchunks, cudaStream_t st, bool unit_start,
              const std::vector<BigProb> &big) {
  const int n = a.n, R = a.R;
  const int prec = sizeof(S) == 8 ? DOCI_FP64 : DOCI_FP32;
  std::vector<char> big_running(big.size(), 1);
  const unsigned small = (n + 127) / 128;
  // side streams for the large problems' sigmas: each problem's copies and
  // kernels run on one of them, so that several problems' kernels overlap
  // (forked from and joined back into st with events, also inside the graph)
  SideStreams side;
  if (big.size() > 1) {
    const int ns = static_cast<int>(std::min<size_t>(big.size(), kSideStreams));
    if (const int se = side.make(ns)) return se;
  }
  eng_init_state<<<small, 128, 0, st>>>(a);
  if (unit_start) {
    for (int r = 0; r < R; ++r) eng_lowest<<<nblk(nchunks), kET, 0, st>>>(a, r);
    eng_unit<S><<<nblk(nchunks), kET, 0, st>>>(a);
    eng_init_state<<<small, 128, 0, st>>>(a);
  }
  DOCI_CUDA(cudaGetLastError());
  // the orthonormalisation of the corrections and the sigmas and subspace
  // columns of the vectors added (the start block is the first "corrections")
  auto extend = [&]() -> int {
    eng_gs<S, KM><<<nblk(nchunks), kET, 0, st>>>(a, -1, 0);
    for (int q = 0; q < R; ++q) {
      eng_gs<S, KM><<<nblk(nchunks), kET, 0, st>>>(a, q, 1);
      eng_gs<S, KM><<<nblk(nchunks), kET, 0, st>>>(a, q, 2);
    }
    eng_gs_finish<S><<<nblk(nchunks), kET, 0, st>>>(a);
    if (ntiles > 0) eng_sigma<S, NH><<<nblk(ntiles), kET, 0, st>>>(a);
    if (side.n > 0) DOCI_CUDA(side.fork(st));
    for (size_t b = 0, k = 0; b < big.size(); ++b) {
      if (!big_running[b]) continue;
      const BigProb &bp = big[b];
      cudaStream_t sb = side.n > 0 ? side.s[k++ % side.n] : st;
      eng_stage<S><<<nblk(std::min<uint64_t>((bp.D * R + 255) / 256, 4096)), 256, 0, sb>>>(
          a, bp.p, static_cast<S *>(bp.xs), nullptr, 0);
      for (int v = 0; v < R; ++v) {
        const int sv = launch_sigma(bp.h, static_cast<S *>(bp.xs) + v * bp.D, static_cast<S *>(bp.ys) + v * bp.D,
                                    prec, sb);
        if (sv) return sv;
      }
      eng_stage<S><<<nblk(std::min<uint64_t>((bp.D * R + 255) / 256, 4096)), 256, 0, sb>>>(
          a, bp.p, nullptr, static_cast<const S *>(bp.ys), 1);
    }
    if (side.n > 0) DOCI_CUDA(side.join(st));
    eng_subcol<S><<<dim3(nblk(nchunks), (KM + kCk - 1) / kCk, (R + kCj - 1) / kCj), kET, 0, st>>>(a);
    DOCI_CUDA(cudaGetLastError());
    return DOCI_OK;
  };
  int s = extend();
  if (s) return s;
  // one iteration, captured and replayed (captured again when a large
  // problem finishes, so that its sigmas are no longer launched)
  cudaGraphExec_t exec = nullptr;
  auto capture = [&]() -> int {
    if (exec) {
      cudaGraphExecDestroy(exec);
      exec = nullptr;
    }
    cudaGraph_t graph = nullptr;
    DOCI_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeRelaxed));
    eng_eig<<<n, kEigT, 0, st>>>(a);
    eng_deflate<S, KM><<<nblk(nchunks), kET, 0, st>>>(a);
    eng_after_restart<<<small, 128, 0, st>>>(a);
    eng_residual<S><<<dim3(nblk(nchunks), (R + kRq - 1) / kRq), kET, 0, st>>>(a);
    eng_control<<<small, 128, 0, st>>>(a);
    const int se = extend();
    cudaError_t ce = cudaStreamEndCapture(st, &graph);
    if (se) {
      if (graph) cudaGraphDestroy(graph);
      return se;
    }
    DOCI_CUDA(ce);
    ce = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    DOCI_CUDA(ce);
    return DOCI_OK;
  };
  s = capture();
  if (s) return s;
  std::vector<int> flags(n);
  int status = DOCI_OK;
  for (int it = 0; it <= a.max_its + 1; ++it) {
    cudaError_t e = cudaGraphLaunch(exec, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(flags.data(), a.flags, sizeof(int) * n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
      status = cuda_status(e, "batch engine iteration");
      break;
    }
    if (std::none_of(flags.begin(), flags.end(), [](int f) { return f != 0; })) break;
    bool changed = false;
    for (size_t b = 0; b < big.size(); ++b)
      if (big_running[b] && !flags[big[b].p]) {
        big_running[b] = 0;
        changed = true;
      }
    if (changed && (status = capture())) break;
  }
  if (exec) cudaGraphExecDestroy(exec);
  if (status) return status;
  eng_combine<S, KM><<<nblk(nchunks), kET, 0, st>>>(a);
  DOCI_CUDA(cudaGetLastError());
  return DOCI_OK;
}

template <typename S, int KM>
int run_phase_nh(EArgs &a, int nh_max, uint32_t ntiles, uint32_t nchunks, cudaStream_t st, bool unit_start,
                 const std::vector<BigProb> &big) {
  if (nh_max <= 8) return run_phase<S, KM, 8>(a, ntiles, nchunks, st, unit_start, big);
  if (nh_max <= 16) return run_phase<S, KM, 16>(a, ntiles, nchunks, st, unit_start, big);
  if (nh_max <= 24) return run_phase<S, KM, 24>(a, ntiles, nchunks, st, unit_start, big);
  return run_phase<S, KM, 32>(a, ntiles, nchunks, st, unit_start, big);
}

template <typename S>
int run_phase_km(EArgs &a, int nh_max, uint32_t ntiles, uint32_t nchunks, cudaStream_t st, bool unit_start,
                 const std::vector<BigProb> &big) {
  if (a.maxv <= 8) return run_phase_nh<S, 8>(a, nh_max, ntiles, nchunks, st, unit_start, big);
  if (a.maxv <= 16) return run_phase_nh<S, 16>(a, nh_max, ntiles, nchunks, st, unit_start, big);
  return run_phase_nh<S, 32>(a, nh_max, ntiles, nchunks, st, unit_start, big);
}

__global__ void shifted_diag32_kernel(const double *d, double shift, float *out, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = static_cast<float>(d[i] - shift);
}

// sigma choice per (device, L, N): the tile shape of the batched pass
// (determinants per thread: 1, 2 or 4) and whether the problem's sigmas come
// from the single-problem kernels instead (untuned: from 2^22 determinants,
// where those kernels' row tilings beat the per-determinant gather)
struct TileChoice {
  int dpt = 1;
  int kernels = -1;  // -1 untuned
};
std::mutex g_tile_mu;
std::map<std::tuple<int, int, int>, TileChoice> g_tile;
constexpr uint32_t kBigD = 1u << 22;

TileChoice tile_choice(const doci_ham *h) {
  std::lock_guard<std::mutex> lk(g_tile_mu);
  auto it = g_tile.find(std::make_tuple(h->device, h->L, h->N));
  TileChoice c = it == g_tile.end() ? TileChoice{} : it->second;
  if (c.kernels < 0) c.kernels = h->D >= kBigD ? 1 : 0;
  return c;
}

__global__ void eng_tune_state(EState *st, int nv) {
  st->m0 = 0;
  st->m = nv;
  st->done = 0;
}

template <int NH>
void launch_tune_sigma(const EArgs &a, unsigned ntiles, cudaStream_t st) {
  eng_sigma<float, NH><<<ntiles, kET, 0, st>>>(a);
}

}  // namespace

int engine_tune(doci_ham *h, int nv, int *dpt_out) {
  if (!h || nv < 1 || nv > kMaxR) return DOCI_ERR_INVALID;
  cudaStream_t st = h->stream;
  const size_t D = h->D;
  DBuf<float> V, VA;
  DBuf<EProb> dP;
  DBuf<EState> dS;
  DBuf<uint32_t> dT0;
  int s;
  if ((s = V.alloc(D * nv, st)) || (s = VA.alloc(D * nv, st)) || (s = dP.alloc(1, st)) || (s = dS.alloc(1, st)) ||
      (s = dT0.alloc(2, st)))
    return s;
  DOCI_CUDA(cudaMemsetAsync(V.p, 0, sizeof(float) * D * nv, st));
  eng_tune_state<<<1, 1, 0, st>>>(dS.p, nv);
  EProb pb{};
  pb.D = h->D;
  pb.L = h->L;
  pb.N = h->N;
  pb.nh = h->nh;
  pb.nbr = h->d_nbr;
  pb.K = h->d_Kmir32;
  pb.diag_s = h->d_diag32;
  pb.diag = h->d_diag;
  pb.V = V.p;
  pb.VA = VA.p;
  pb.tile0 = 0;
  EArgs a{};
  a.n = 1;
  a.R = nv;
  a.P = dP.p;
  a.St = dS.p;
  a.tile0 = dT0.p;
  a.binom = h->d_binom;
  cudaEvent_t e0, e1;
  DOCI_CUDA(cudaEventCreate(&e0));
  DOCI_CUDA(cudaEventCreate(&e1));
  int best = 1;
  float best_ms = 1e30f;
  for (int dpt : {1, 2, 4}) {
    pb.dpt = dpt;
    const uint32_t nt = static_cast<uint32_t>((D + static_cast<size_t>(kET) * dpt - 1) / (static_cast<size_t>(kET) * dpt));
    const uint32_t t0[2] = {0, nt};
    if (cudaMemcpyAsync(dP.p, &pb, sizeof pb, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(dT0.p, t0, sizeof t0, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      break;
    auto run = [&] {
      if (h->nh <= 8) launch_tune_sigma<8>(a, nt, st);
      else if (h->nh <= 16) launch_tune_sigma<16>(a, nt, st);
      else if (h->nh <= 24) launch_tune_sigma<24>(a, nt, st);
      else launch_tune_sigma<32>(a, nt, st);
    };
    run();  // warm-up
    cudaEventRecord(e0, st);
    for (int k = 0; k < 3; ++k) run();
    cudaEventRecord(e1, st);
    if (cudaEventSynchronize(e1) != cudaSuccess) break;
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best_ms) {
      best_ms = ms;
      best = dpt;
    }
  }
  // the single-problem kernels on the same vectors, one sigma per vector
  int kernels = 0;
  {
    bool ok = true;
    for (int k = 0; k < 4 && ok; ++k) {  // warm-up, then three timed rounds
      if (k == 1) cudaEventRecord(e0, st);
      for (int v = 0; v < nv && ok; ++v)
        ok = launch_sigma(h, V.p + static_cast<size_t>(v) * D, VA.p + static_cast<size_t>(v) * D, DOCI_FP32, st) ==
             DOCI_OK;
    }
    cudaEventRecord(e1, st);
    float ms = 1e30f;
    if (ok && cudaEventSynchronize(e1) == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    kernels = ms < best_ms ? 1 : 0;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  DOCI_CUDA(cudaGetLastError());
  if ((s = ham_device_error(h, st))) return s;
  {
    std::lock_guard<std::mutex> lk(g_tile_mu);
    TileChoice c;
    c.dpt = best;
    c.kernels = kernels;
    g_tile[std::make_tuple(h->device, h->L, h->N)] = c;
  }
  if (dpt_out) *dpt_out = kernels ? 0 : best;
  return DOCI_OK;
}

int64_t engine_footprint(int L, int N, const doci_batch_opts &o) {
  if (L < 1 || L > 32 || N < 0 || N > L) return -1;
  const int64_t D = static_cast<int64_t>(binom64(L, N));
  const int64_t R = std::max(1, std::min(o.nroots, kMaxR));
  const int64_t mv = std::min(kMaxV, std::max(o.max_vec, 2 * o.nroots));
  // the handle's diagonals and tables
  const int64_t ham = D * 12 + (16ll << 20) + static_cast<int64_t>(nbr_table_bytes(L, N, D));
  const int64_t x = D * R * 8;                 // Ritz vectors
  const int64_t p64 = 2 * mv * D * 8 + R * D * 8 + 2 * R * D * 8;  // + staging of a large problem
  const int64_t p32 = o.mode == DOCI_MODE_MIXED ? 2 * mv * D * 4 + R * D * 4 + D * 4 + 2 * R * D * 4 : 0;
  return ham + x + p64 + p32 + (1ll << 20);
}

int engine_solve(int n, doci_ham *const *hams, const doci_batch_opts &o, cudaStream_t st, doci_root_result *res,
                 double *const *vecs) {
  if (n < 1) return DOCI_OK;
  const int R = o.nroots;
  if (R < 1 || R > kMaxR) return DOCI_ERR_INVALID;
  EArgs a{};
  a.n = n;
  a.R = R;
  a.maxv = std::min(kMaxV, std::max(o.max_vec, 2 * R));
  // thick restart: by default keep 2 nroots Ritz vectors, at least a quarter
  // of the basis (keeping only the nroots wanted ones restarts every few
  // blocks and stalls the higher roots)
  a.keep = o.keep > 0 ? o.keep : std::max(2 * R, a.maxv / 4);
  if (a.keep < R) a.keep = R;
  if (a.keep > a.maxv - R) a.keep = a.maxv - R;
  a.tol = o.tol;
  a.ldp = std::max(kMaxV + 2, ((R + kCj - 1) / kCj) * kCj * kMaxV);
  std::vector<uint32_t> tile0(n + 1, 0), chunk0(n + 1, 0);
  std::vector<int> dpt(n, 1), big_idx;
  size_t total = 0;
  int nh_max = 1;
  for (int i = 0; i < n; ++i) {
    const doci_ham *h = hams[i];
    if (!h || static_cast<int64_t>(h->D) < 1) return DOCI_ERR_INVALID;
    const TileChoice tc = tile_choice(h);
    dpt[i] = tc.dpt;
    if (tc.kernels) big_idx.push_back(i);
    tile0[i + 1] = tile0[i] + (tc.kernels ? 0u : static_cast<uint32_t>((h->D + kET * dpt[i] - 1) / (kET * dpt[i])));
    const uint32_t chunk = static_cast<uint32_t>(kET * elems_per_thread(h->D));
    chunk0[i + 1] = chunk0[i] + (h->D + chunk - 1) / chunk;
    total += h->D;
    nh_max = std::max(nh_max, h->nh);
  }
  const uint32_t ntiles = tile0[n], nchunks = chunk0[n];
  DBuf<EProb> dP;
  DBuf<EState> dS;
  DBuf<uint32_t> dT0, dC0;
  DBuf<double> dpart, dX;
  DBuf<unsigned> dcnt;
  DBuf<int> dflags;
  int s;
  if ((s = dP.alloc(n, st)) || (s = dS.alloc(n, st)) || (s = dT0.alloc(n + 1, st)) || (s = dC0.alloc(n + 1, st)) ||
      (s = dpart.alloc(static_cast<size_t>(nchunks) * a.ldp, st)) || (s = dcnt.alloc(n, st)) ||
      (s = dflags.alloc(n, st)) || (s = dX.alloc(total * R, st)))
    return s;
  DOCI_CUDA(cudaMemcpyAsync(dT0.p, tile0.data(), sizeof(uint32_t) * (n + 1), cudaMemcpyHostToDevice, st));
  DOCI_CUDA(cudaMemcpyAsync(dC0.p, chunk0.data(), sizeof(uint32_t) * (n + 1), cudaMemcpyHostToDevice, st));
  DOCI_CUDA(cudaMemsetAsync(dcnt.p, 0, sizeof(unsigned) * n, st));
  a.St = dS.p;
  a.tile0 = dT0.p;
  a.chunk0 = dC0.p;
  a.part = dpart.p;
  a.cnt = dcnt.p;
  a.flags = dflags.p;
  a.binom = hams[0]->d_binom;
  a.P = dP.p;
  std::vector<EProb> P(n);
  std::vector<EState> host_st(n);
  auto upload = [&]() -> int {
    DOCI_CUDA(cudaMemcpyAsync(dP.p, P.data(), sizeof(EProb) * n, cudaMemcpyHostToDevice, st));
    return DOCI_OK;
  };
  auto fill_common = [&](size_t elem, void *V, void *VA, void *T) {
    size_t off = 0;
    for (int i = 0; i < n; ++i) {
      const doci_ham *h = hams[i];
      EProb &pb = P[i];
      pb.D = h->D;
      pb.L = h->L;
      pb.N = h->N;
      pb.nh = h->nh;
      pb.nbr = h->d_nbr;
      pb.diag = h->d_diag;
      pb.V = static_cast<char *>(V) + off * a.maxv * elem;
      pb.VA = static_cast<char *>(VA) + off * a.maxv * elem;
      pb.T = static_cast<char *>(T) + off * R * elem;
      pb.X = dX.p + off * R;
      pb.tile0 = tile0[i];
      pb.eper = elems_per_thread(h->D);
      pb.dpt = dpt[i];
      pb.chunk0 = chunk0[i];
      pb.nchunks = chunk0[i + 1] - chunk0[i];
      off += h->D;
    }
  };
  // a device wait that ran out in a large problem's sigmas (its FP32 view shares
  // the handle's error word)
  std::vector<int> status(n, DOCI_OK);
  auto check_waits = [&]() -> int {
    for (int i : big_idx) {
      const int e = ham_device_error(hams[i], st);
      if (e == DOCI_ERR_DEVICE_TIMEOUT) status[i] = e;
      else if (e) return e;
    }
    return DOCI_OK;
  };
  std::vector<double> e32(static_cast<size_t>(n) * R, 0.0);
  std::vector<int> its32v(n, 0), sig32(n, 0);
  bool have_start = false;  // the FP64 phase starts from the FP32 phase's Ritz vectors
  if (o.mode == DOCI_MODE_MIXED) {
    DBuf<float> V, VA, T, d32;
    if ((s = V.alloc(total * a.maxv, st)) || (s = VA.alloc(total * a.maxv, st)) || (s = T.alloc(total * R, st)) ||
        (s = d32.alloc(total, st)))
      return s;
    fill_common(sizeof(float), V.p, VA.p, T.p);
    // shift = the lowest diagonal element of each problem
    {
      for (int i = 0; i < n; ++i) {
        P[i].K = hams[i]->d_Kmir32;
        P[i].shift = 0;
        P[i].diag_s = nullptr;
      }
      if ((s = upload())) return s;
      eng_init_state<<<(n + 127) / 128, 128, 0, st>>>(a);
      eng_lowest<<<nblk(nchunks), kET, 0, st>>>(a, 0);
      DOCI_CUDA(cudaGetLastError());
      DOCI_CUDA(cudaMemcpyAsync(host_st.data(), dS.p, sizeof(EState) * n, cudaMemcpyDeviceToHost, st));
      DOCI_CUDA(cudaStreamSynchronize(st));
      size_t off = 0;
      for (int i = 0; i < n; ++i) {
        double sh = 0;
        DOCI_CUDA(cudaMemcpyAsync(&sh, hams[i]->d_diag + host_st[i].idx0, sizeof(double), cudaMemcpyDeviceToHost,
                                  st));
        DOCI_CUDA(cudaStreamSynchronize(st));
        P[i].shift = sh;
        P[i].diag_s = d32.p + off;
        shifted_diag32_kernel<<<nblk(std::min<uint64_t>((hams[i]->D + 255) / 256, 4096)), 256, 0, st>>>(
            hams[i]->d_diag, sh, d32.p + off, hams[i]->D);
        off += hams[i]->D;
      }
      DOCI_CUDA(cudaGetLastError());
      if ((s = upload())) return s;
    }
    // large problems: shifted views (FP32 diagonal - shift) and staging
    std::vector<std::unique_ptr<doci_ham>> views;
    std::vector<std::unique_ptr<DBuf<float>>> stg;
    std::vector<BigProb> big;
    for (int i : big_idx) {
      views.emplace_back(new doci_ham(*hams[i]));
      views.back()->d_diag32 = static_cast<float *>(const_cast<void *>(P[i].diag_s));
      views.back()->sigma_kernel = hams[i]->sigma_kernel;
      stg.emplace_back(new DBuf<float>());
      if ((s = stg.back()->alloc(2 * static_cast<size_t>(hams[i]->D) * R, st))) return s;
      big.push_back(BigProb{i, views.back().get(), stg.back()->p, stg.back()->p + static_cast<size_t>(hams[i]->D) * R,
                            hams[i]->D});
    }
    EArgs a32 = a;
    a32.tol = o.mixed_tol > o.tol ? o.mixed_tol : o.tol;
    a32.stall_window = 15;
    a32.max_its = o.max_its;
    for (int i = 0; i < n; ++i) P[i].max_its = o.max_its;
    if ((s = upload())) return s;
    s = run_phase_km<float>(a32, nh_max, ntiles, nchunks, st, true, big);
    if (s || (s = check_waits())) return s;
    DOCI_CUDA(cudaMemcpyAsync(host_st.data(), dS.p, sizeof(EState) * n, cudaMemcpyDeviceToHost, st));
    DOCI_CUDA(cudaStreamSynchronize(st));
    for (int i = 0; i < n; ++i) {
      its32v[i] = host_st[i].its;
      sig32[i] = host_st[i].sigmas;
      for (int r = 0; r < R; ++r) e32[static_cast<size_t>(i) * R + r] = host_st[i].w[r] + P[i].shift;
    }
    have_start = true;
  }
  // FP64 phase
  {
    DBuf<double> V, VA, T;
    if ((s = V.alloc(total * a.maxv, st)) || (s = VA.alloc(total * a.maxv, st)) || (s = T.alloc(total * R, st)))
      return s;
    fill_common(sizeof(double), V.p, VA.p, T.p);
    for (int i = 0; i < n; ++i) {
      P[i].K = hams[i]->d_Kmir64;
      P[i].diag_s = hams[i]->d_diag;
      P[i].shift = 0;
    }
    if ((s = upload())) return s;
    if (have_start) DOCI_CUDA(cudaMemcpyAsync(T.p, dX.p, sizeof(double) * total * R, cudaMemcpyDeviceToDevice, st));
    EArgs a64 = a;
    a64.stall_window = 0;
    // the FP64 phase may run max_its less the problem's FP32 iterations
    int max64 = 1;
    for (int i = 0; i < n; ++i) {
      P[i].max_its = have_start ? std::max(1, o.max_its - its32v[i]) : o.max_its;
      max64 = std::max(max64, P[i].max_its);
    }
    if ((s = upload())) return s;
    a64.max_its = max64;
    std::vector<std::unique_ptr<DBuf<double>>> stg;
    std::vector<BigProb> big;
    for (int i : big_idx) {
      stg.emplace_back(new DBuf<double>());
      if ((s = stg.back()->alloc(2 * static_cast<size_t>(hams[i]->D) * R, st))) return s;
      big.push_back(BigProb{i, hams[i], stg.back()->p, stg.back()->p + static_cast<size_t>(hams[i]->D) * R,
                            hams[i]->D});
    }
    s = run_phase_km<double>(a64, nh_max, ntiles, nchunks, st, !have_start, big);
    if (s || (s = check_waits())) return s;
    DOCI_CUDA(cudaMemcpyAsync(host_st.data(), dS.p, sizeof(EState) * n, cudaMemcpyDeviceToHost, st));
    DOCI_CUDA(cudaStreamSynchronize(st));
  }
  size_t off = 0;
  for (int i = 0; i < n; ++i) {
    doci_root_result &r = res[i];
    const EState &es = host_st[i];
    const int nr = std::min(R, es.m);
    r.nroots = R;
    for (int k = 0; k < nr; ++k) {
      r.energy[k] = es.w[k];
      r.residual[k] = es.res[k];
      r.energy_fp32[k] = e32[static_cast<size_t>(i) * R + k];
    }
    r.iterations = es.its + its32v[i];
    r.iterations_fp32 = its32v[i];
    r.sigmas = es.sigmas + sig32[i];
    r.converged = es.converged;
    r.status = status[i];
    if (vecs && vecs[i]) {
      DOCI_CUDA(cudaMemcpyAsync(vecs[i], dX.p + off * R, sizeof(double) * hams[i]->D * R, cudaMemcpyDeviceToHost,
                                st));
    }
    off += hams[i]->D;
  }
  DOCI_CUDA(cudaStreamSynchronize(st));
  return DOCI_OK;
}

}  // namespace doci
