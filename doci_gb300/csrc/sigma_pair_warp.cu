// sigma_pair_warp.cu -- FP32 sigma in the (N-1)-pair form (sigma_pair.cu has
// the regrouping: sigma[T] = diag[T] x[T] + sum_{i in T} Y_{T\i}[i],
// Y_S = X_S K), one warp per unit, the product with K on the 5th-generation
// tensor cores.  This is what kind 6 runs from 10 orbitals on.
//
// A unit (pair_warp_index.cuh) belongs to two warps, which walk its sets 32 at
// a time, one set per lane, which is also the set's lane in tensor memory: one
// gathers a set's values and splits them into the A operand, the other reads
// the product back and scatters it, while the first is at the next 32 sets.
// The unit's own row, at most C(12,6) = 924 elements, is private to them in
// shared memory, its x with the one and its sums with the other: the random
// accesses of the column orbitals stay on chip, and since S -> S u o is one to
// one the sums are plain read-modify-writes, one orbital after the other, with
// no atomics.  The rows of the row-part holes are read and added to at the
// set's own column, 32 consecutive elements at a time.  The orbital axis is
// not compacted, so K (high and low TF32 parts, 64 x 32, the B operand) is the
// same for every unit and four warps with units of their own share one
// 128-row MMA tile; tensor memory holds four tiles.
//
// TF32 three ways (x high x K high, x high x K low, x low x K high): the first
// two as one MMA of 64 columns, since an MMA of 128 rows takes the same 51
// cycles for 32 and for 64 columns on GB300 (24.6 ns in a run of 96; 72 cycles
// at 128 columns).  The two halves are added when they are read back.
//
// Column orbitals: 12, 10 or 8 (pw::column_orbitals).  Larger rows mean fewer
// set-ups and fewer row-part orbitals to look at, smaller ones more units to
// spread.  Measured with one warp doing both jobs (us, 12 / 10 / 8): L=32 N=16
// 19,120 / 22,940 / 38,470; L=26 N=13 347 / 362 / 562; L=24 N=12
// 107 / 103 / 138; L=22 N=11 70 / 38 / 46; L=21 N=9 70 / 27.6 / 25.1;
// L=18 N=9 69 / 27 / 16.8.
//
// Measured against the one-block-per-unit mma.sync kernel of sigma_pair.cu:
// L=32 N=16 33.9 -> 17.1 ms (one warp for both jobs 19.1), L=28 N=14 1.82 ->
// 1.11 ms (1.23), L=27 N=11 524 -> 305 us (331), L=20 N=10 28.0 -> 20.4 us
// (20.9).  Bound by instruction issue (65 % of the slots, 690 warp instructions
// per 32 sets), the shared-memory pipe (60 %) and the latency of the hole rows.
// Two sets per lane, two tiles per warp pair: fewer instructions (628), but
// half the warps, 1.33 ms at L=28; only the live row-part orbitals, at
// tensor-memory columns known at run time: 1.77 ms (their addresses go
// through uniform registers one by one).
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "addressing.cuh"
#include "internal.h"
#include "pair_warp.h"
#include "pair_warp_index.cuh"
#include "tcgen.cuh"

namespace doci {
namespace {

constexpr int kSlots = 4;                   // tiles in flight
constexpr int kThreads = 2 * 128 * kSlots;  // a gathering and a scattering warpgroup per tile
constexpr uint32_t kTmemCols = 512;         // per tile: A high 32 | A low 32 | D 64
// tcgen05 instruction descriptor: D FP32, A and B TF32, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc(uint32_t n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
constexpr int kOffBar = 64 * 128;           // after K: 64 rows (high, low) x 32 columns, swizzled
constexpr int kOffStart = kOffBar + 128;    // row starts of a warp's hole rows, 24 per warp
constexpr int kOffRows = kOffStart + 4 * 24 * (kThreads / 32);
constexpr size_t kMinSmem = 120 * 1024;     // one block per SM: it allocates all of the tensor memory

__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(id), "r"(acc));
}
// nearest TF32 (10-bit mantissa), ties away from zero: half a TF32 ulp added to
// the magnitude, the low 13 bits cut (two integer instructions; cvt.rna.tf32
// measured about five)
__device__ __forceinline__ uint32_t tf32_rna(float f) { return (__float_as_uint(f) + 0x1000u) & 0xffffe000u; }

// DET: what is added to hole rows is stored instead, each contribution in a
// place of its own (`slab`: the sum that element e of the target's row part
// contributes to determinant T at e D + T), and the own row is stored; the
// sums then have a fixed order (sum_slabs_kernel).
template <int P, bool DET>
__global__ void __launch_bounds__(kThreads, 1)
sigma_pair_warp_kernel(const __grid_constant__ PwShape s, const uint32_t *__restrict__ units,
                       const uint32_t *__restrict__ rowstart, const uint4 *__restrict__ tab_a,
                       const uint2 *__restrict__ tab_b, const float *__restrict__ g_ksplit,
                       const float *__restrict__ diag, const float *__restrict__ x, float *__restrict__ y,
                       float *__restrict__ slab, int *__restrict__ err) {
  constexpr int NR = 32 - P;
  constexpr int XC = pw::cells(P);
  extern __shared__ __align__(1024) uint8_t sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, slot = (warp >> 2) & (kSlots - 1), w4 = warp & 3;
  const bool gatherer = warp < 4 * kSlots;
  const uint32_t base = su32(sm);
  if (base & 1023u) {  // the swizzled K tile needs a 1024-byte aligned base
    if (tid == 0) atomicCAS(err, 0, 3);
    return;
  }
  const uint32_t bar_done = base + kOffBar + 8 * slot, bar_free = bar_done + 8 * kSlots;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + kOffBar + 16 * kSlots) + slot;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + kOffBar + 20 * kSlots);
  // the own row's x (gathering warps) or sums (scattering warps)
  float *cells = reinterpret_cast<float *>(sm + kOffRows) + warp * XC;
  const uint32_t ca = su32(cells), ra = base + kOffStart + warp * 96;

  for (int e = tid; e < 64 * 32; e += kThreads) {
    const int r = e >> 5, k = e & 31;
    *reinterpret_cast<float *>(sm + sw128(r, k)) = g_ksplit[(r >> 5) * 1024 + (r & 31) * 32 + k];
  }
  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(base + kOffBar + 8 * i));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(base + kOffBar + 8 * (kSlots + i)));
      reinterpret_cast<volatile int *>(sm + kOffBar + 16 * kSlots)[i] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (lane == 0) cells[XC - 1] = 0.f;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tslot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t tg = tmem + 128u * slot, tw = tg + (static_cast<uint32_t>(32 * w4) << 16);
  const int nks = (s.L + 7) >> 3;  // >= 2 (L >= 10)

  uint32_t n = 0;  // tiles of this slot so far
  bool ok = true, fail = false;
  for (int q = blockIdx.x * kSlots + slot; q < s.nquads && ok; q += gridDim.x * kSlots) {
    const uint32_t mask = units[4 * q + w4];
    const int jp = s.N - 1 - __popc(units[4 * q]);
    const uint32_t n_s = jp >= 0 ? s.n[jp] : 0u;
    const bool real = mask != pw::kNone;
    const uint32_t n_own = real ? s.n[jp + 1] : 0u;
    const uint32_t holes = real ? ~mask & ((1u << s.na) - 1u) : 0u;
    const uint32_t own = n_own ? rowstart[mask] : 0u;
    for (uint32_t c = lane; c < n_own; c += 32) cells[c] = gatherer ? __ldg(x + own + c) : 0.f;
    // (a unit without sets has no hole rows either)
    if (lane < 24) {
      const bool hole = n_s && ((holes >> lane) & 1u);
      uint32_t r = hole ? rowstart[mask | (1u << lane)] : 0u;
      if (DET && hole && !gatherer) r += s.D * static_cast<uint32_t>(__popc(mask & ((1u << lane) - 1u)));
      reinterpret_cast<uint32_t *>(sm + kOffStart)[warp * 24 + lane] = r;
    }
    __syncwarp();
    const uint4 *ta = tab_a + (n_s ? s.off[jp] : 0u) + lane;
    const uint2 *tb = tab_b + (n_s ? s.off[jp] : 0u) + lane;
    const uint32_t last = n_s - 1;

    if (gatherer) {
      for (uint32_t c0 = 0; c0 < n_s; c0 += 32, ++n) {
        // the set's 32 values by orbital: row-part holes from their rows, column
        // orbitals from the own row (the zero cell where the orbital is in the
        // set; the table ends each set size with a full warp of zero cells)
        float v[32];
        const float *xl = x + min(c0 + lane, last);
#pragma unroll
        for (int b = 0; b < NR; b += 4) {
          const uint4 r = lds128(ra + 4 * b);
          v[P + b] = ldg_if(xl + r.x, holes & (1u << b));
          v[P + b + 1] = ldg_if(xl + r.y, holes & (1u << (b + 1)));
          if (b + 2 < NR) v[P + b + 2] = ldg_if(xl + r.z, holes & (1u << (b + 2)));
          if (b + 3 < NR) v[P + b + 3] = ldg_if(xl + r.w, holes & (1u << (b + 3)));
        }
        uint32_t w[6];
        const uint4 ea = __ldg(ta + c0);
        w[0] = ea.x, w[1] = ea.y, w[2] = ea.z, w[3] = ea.w;
        if (P > 8) {
          const uint2 eb = __ldg(tb + c0);
          w[4] = eb.x, w[5] = eb.y;
        }
#pragma unroll
        for (int o = 0; o < P; ++o) v[o] = lds(ca + (o & 1 ? w[o >> 1] >> 16 : w[o >> 1] & 0xffffu));
        if (n > 0 && !warp_wait(bar_done, (n - 1) & 1u, s.spin_limit, abort_flag, err, 21)) fail = true;
        if (!fail) {  // (else an MMA may still read the tile)
          fence_after();
          // split into TF32 high and low parts in this lane's row of the tile
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            uint32_t r[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = tf32_rna(v[8 * h + i]);
            tst8(tw + 8 * h, r);
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(v[8 * h + i] - __uint_as_float(r[i]));
            tst8(tw + 32 + 8 * h, r);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          fence_before();
        }
        if (group_meet(slot, fail)) {
          ok = false;
          break;
        }
        if (w4 == 0) {
          // the sums of the tile before have to be read
          if (n > 0 && !warp_wait(bar_free, (n - 1) & 1u, s.spin_limit, abort_flag, err, 22)) fail = true;
          if (!fail && lane == 0) {
            fence_after();
            const uint64_t desc = smem_desc(base);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              if (ks < 2 || ks < nks) mma_ts(tg + 64, tg + 8 * ks, desc + 2 * ks, idesc(64), ks > 0);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              if (ks < 2 || ks < nks) mma_ts(tg + 64, tg + 32 + 8 * ks, desc + 2 * ks, idesc(32), 1);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_done)
                         : "memory");
          }
          __syncwarp();
        }
      }
    } else {
      for (uint32_t c0 = 0; c0 < n_s; c0 += 32, ++n) {
        uint32_t w[6];
        const uint4 ea = __ldg(ta + c0);
        w[0] = ea.x, w[1] = ea.y, w[2] = ea.z, w[3] = ea.w;
        if (P > 8) {
          const uint2 eb = __ldg(tb + c0);
          w[4] = eb.x, w[5] = eb.y;
        }
        if (!warp_wait(bar_done, n & 1u, s.spin_limit, abort_flag, err, 23)) {
          ok = false;
          break;
        }
        fence_after();
        float yv[32];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          float r[8], l[8];
          tld8(tw + 64 + 8 * h, r);
          tld8(tw + 96 + 8 * h, l);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 8; ++i) yv[8 * h + i] = r[i] + l[i];
        }
        fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_free) : "memory");
        float *yl = (DET ? slab : y) + c0 + lane;
        const uint32_t add = c0 + lane <= last ? holes : 0u;
        auto put = [](float *p, float v, uint32_t on) {
          if (DET) st_if(p, v, on);
          else red_if(p, v, on);
        };
#pragma unroll
        for (int b = 0; b < NR; b += 4) {
          const uint4 r = lds128(ra + 4 * b);
          put(yl + r.x, yv[P + b], add & (1u << b));
          put(yl + r.y, yv[P + b + 1], add & (1u << (b + 1)));
          if (b + 2 < NR) put(yl + r.z, yv[P + b + 2], add & (1u << (b + 2)));
          if (b + 3 < NR) put(yl + r.w, yv[P + b + 3], add & (1u << (b + 3)));
        }
        // own row: one orbital at a time no two sets meet (S -> S u o is one to
        // one), and the warp alone adds to it
#pragma unroll
        for (int o = 0; o < P; ++o) {
          const uint32_t a = ca + (o & 1 ? w[o >> 1] >> 16 : w[o >> 1] & 0xffffu);
          sts(a, lds(a) + yv[o]);
          __syncwarp();
        }
      }
      __syncwarp();
      if (ok)
        for (uint32_t c = lane; c < n_own; c += 32) {
          const float v = fmaf(diag[own + c], __ldg(x + own + c), cells[c]);
          if (DET) y[own + c] = v;
          else atomicAdd(y + own + c, v);
        }
      __syncwarp();
    }
  }
  // the last tile's MMAs complete by themselves; whatever side gave up, wait
  // for them (bounded) before the tensor memory is freed
  if (gatherer && w4 == 0 && n > 0)
    for (long i = 0; i < kTcSpinLimit && !mbar_try(bar_done, (n - 1) & 1u); ++i) {
    }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

__global__ void zero_kernel(float *__restrict__ y, uint32_t n) {
  const uint32_t head = min(n, static_cast<uint32_t>((16 - (reinterpret_cast<uintptr_t>(y) & 15)) & 15) / 4);
  const uint32_t n4 = (n - head) / 4, i0 = blockIdx.x * blockDim.x + threadIdx.x;
  float4 *y4 = reinterpret_cast<float4 *>(y + head);
  for (uint32_t i = i0; i < n4; i += gridDim.x * blockDim.x) y4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i0 < head) y[i0] = 0.f;
  if (i0 < n - head - 4 * n4) y[head + 4 * n4 + i0] = 0.f;
}

// sigma[T] += the slabs of the elements of T's row part, in ascending order; a
// warp per row
template <typename T>
__global__ void __launch_bounds__(256)
sum_slabs_kernel(const __grid_constant__ PwShape s, const uint32_t *__restrict__ units,
                 const uint32_t *__restrict__ rowstart, const T *__restrict__ slab, T *__restrict__ y) {
  const int lane = threadIdx.x & 31;
  for (int u = (blockIdx.x * 256 + threadIdx.x) >> 5; u < 4 * s.nquads; u += gridDim.x * 8) {
    const uint32_t mask = units[u];
    if (mask == pw::kNone) continue;
    const int k = __popc(mask);
    const uint32_t n = s.n[s.N - k], r = n ? rowstart[mask] : 0u;
    for (uint32_t c = lane; c < n; c += 32) {
      T v = y[r + c];
      const T *p = slab + r + c;
#pragma unroll 4
      for (int e = 0; e < k; ++e) v += p[static_cast<size_t>(e) * s.D];
      y[r + c] = v;
    }
  }
}

__global__ void build_starts_kernel(uint32_t *out, int P, int na, int N, uint32_t D, const uint32_t *binom) {
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << na); m += gridDim.x * blockDim.x)
    out[m] = pw::row_start(m, P, na, N, D, binom, kBinomCols);
}
__global__ void build_units_kernel(uint32_t *out, pw::Groups g, int na, const uint32_t *binom) {
  const uint32_t total = g.first[g.n];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    int k = 0;
    while (k + 1 < g.n && g.first[k + 1] <= i) ++k;
    const uint32_t j = i - g.first[k];
    out[i] = j < g.count[k] ? dev::colex_unrank<kBinomCols>(j, na, g.kp[k], binom) : pw::kNone;
  }
}

// the insertion tables, once per device and column-orbital count
struct PwTables {
  uint4 *a = nullptr;
  uint2 *b = nullptr;
};
int pw_tables(int device, int P, PwTables *out) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, PwTables> cache;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(device, P);
  auto it = cache.find(key);
  if (it == cache.end()) {
    std::vector<uint32_t> B(kBinomRows * kBinomCols), off;
    std::vector<uint16_t> a, b;
    fill_binom_table(B.data());
    pw::build_tables(P, B.data(), kBinomCols, a, b, off);
    PwTables t;
    DOCI_CUDA(cudaMalloc(&t.a, a.size() * sizeof(uint16_t)));
    DOCI_CUDA(cudaMalloc(&t.b, b.size() * sizeof(uint16_t)));
    DOCI_CUDA(cudaMemcpy(t.a, a.data(), a.size() * sizeof(uint16_t), cudaMemcpyHostToDevice));
    DOCI_CUDA(cudaMemcpy(t.b, b.data(), b.size() * sizeof(uint16_t), cudaMemcpyHostToDevice));
    it = cache.emplace(key, t).first;
  }
  *out = it->second;
  return DOCI_OK;
}

template <int P, bool DET>
int launch_p(const doci_ham *h, const PwShape &s, const float *x, float *y, float *slab, cudaStream_t st) {
  const size_t smem = std::max(kMinSmem, static_cast<size_t>(kOffRows) + 4 * pw::cells(P) * (kThreads / 32));
  int per_sm = 1;
  const int r = kernel_blocks(reinterpret_cast<const void *>(sigma_pair_warp_kernel<P, DET>), kThreads, smem, &per_sm);
  if (r != DOCI_OK) return r;
  const int grid = std::min(device_sm_count(), (s.nquads + kSlots - 1) / kSlots);
  sigma_pair_warp_kernel<P, DET><<<grid, kThreads, smem, st>>>(s, h->d_wunits, h->d_wstart,
                                                          static_cast<const uint4 *>(h->d_wtab_a),
                                                          static_cast<const uint2 *>(h->d_wtab_b),
                                                          reinterpret_cast<const float *>(h->d_kfrag), h->d_diag32, x,
                                                          y, slab, h->d_tc_err);
  DOCI_CUDA(cudaGetLastError());
  return DOCI_OK;
}

}  // namespace

bool pair_warp_fits(const doci_ham *h) { return h->wsplit > 0; }

int ham_build_pair_warp(doci_ham *h) {
  h->wsplit = 0;
  const int L = h->L, N = h->N;
  if (L < 10 || N < 1) return DOCI_OK;
  int major = 0, minor = 0;
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, h->device);
  cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, h->device);
  if (major != 10 || minor != 3) return DOCI_OK;
  std::vector<uint32_t> B(kBinomRows * kBinomCols);
  fill_binom_table(B.data());
  pw::Groups g;
  const int P = pw::column_orbitals(L, N, static_cast<uint32_t>(kSlots * device_sm_count()), B.data(), kBinomCols, &g);
  const int na = L - P;
  const uint32_t total = g.first[g.n];
  DOCI_CUDA(cudaMallocAsync(&h->d_wstart, sizeof(uint32_t) << na, h->stream));
  DOCI_CUDA(cudaMallocAsync(&h->d_wunits, sizeof(uint32_t) * total, h->stream));
  const int blocks = 4 * device_sm_count();
  build_starts_kernel<<<std::min(blocks, ((1 << na) + 255) / 256), 256, 0, h->stream>>>(h->d_wstart, P, na, N, h->D,
                                                                                       h->d_binom);
  build_units_kernel<<<std::min<int>(blocks, (total + 255) / 256), 256, 0, h->stream>>>(h->d_wunits, g, na,
                                                                                       h->d_binom);
  DOCI_CUDA(cudaGetLastError());
  h->nwquads = static_cast<int>(total / 4);
  PwTables t;
  const int r = pw_tables(h->device, P, &t);
  if (r != DOCI_OK) return r;
  if (const int k = ham_build_kdigits(h)) return k;
  h->d_wtab_a = t.a;
  h->d_wtab_b = t.b;
  h->wsplit = P;
  return DOCI_OK;
}

PwShape pair_warp_shape(const doci_ham *h) {
  const int P = h->wsplit;
  PwShape s{};
  s.D = h->D;
  s.L = h->L;
  s.N = h->N;
  s.na = h->L - P;
  s.nquads = h->nwquads;
  s.spin_limit = tc_spin_limit();
  uint32_t at = 0;
  for (int j = 0; j <= P; ++j) {
    s.n[j] = static_cast<uint32_t>(binom64(P, j));
    s.off[j] = at;
    at += pw::padded(s.n[j]);
  }
  return s;
}

int launch_pair_warp(const doci_ham *h, const float *x, float *y, cudaStream_t st) {
  if (!pair_warp_fits(h)) return DOCI_ERR_INVALID;
  const PwShape s = pair_warp_shape(h);
  zero_kernel<<<static_cast<unsigned>(std::min<uint64_t>((h->D / 4 + 256) / 256, 8ull * device_sm_count())), 256, 0,
                st>>>(y, h->D);
  DOCI_CUDA(cudaGetLastError());
  if (h->wsplit == 12) return launch_p<12, false>(h, s, x, y, nullptr, st);
  if (h->wsplit == 10) return launch_p<10, false>(h, s, x, y, nullptr, st);
  return launch_p<8, false>(h, s, x, y, nullptr, st);
}

// slabs of the reproducible form: the largest row part
int pair_warp_slabs(const doci_ham *h) { return std::min(h->L - h->wsplit, h->N); }

int launch_pair_warp_det(const doci_ham *h, const float *x, float *y, float *slab, cudaStream_t st) {
  if (!pair_warp_fits(h)) return DOCI_ERR_INVALID;
  const PwShape s = pair_warp_shape(h);
  const int r = h->wsplit == 12   ? launch_p<12, true>(h, s, x, y, slab, st)
                : h->wsplit == 10 ? launch_p<10, true>(h, s, x, y, slab, st)
                                  : launch_p<8, true>(h, s, x, y, slab, st);
  return r == DOCI_OK ? launch_sum_slabs(h, slab, y, st) : r;
}

template <typename T>
int launch_sum_slabs(const doci_ham *h, const T *slab, T *y, cudaStream_t st) {
  const PwShape s = pair_warp_shape(h);
  sum_slabs_kernel<T><<<std::min(16 * device_sm_count(), (4 * s.nquads + 7) / 8), 256, 0, st>>>(s, h->d_wunits,
                                                                                              h->d_wstart, slab, y);
  return cuda_ok("sum_slabs_kernel");
}
template int launch_sum_slabs<float>(const doci_ham *, const float *, float *, cudaStream_t);
template int launch_sum_slabs<double>(const doci_ham *, const double *, double *, cudaStream_t);

}  // namespace doci
