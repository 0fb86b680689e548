// sigma_pair_warp64.cu -- FP64-accurate sigma in the (N-1)-pair form, one warp
// per unit, the product with K in exact integer arithmetic on the
// 5th-generation tensor cores.  This is what kind 9 runs from 10 orbitals on,
// where K allows it (ham_build_kdigits) and sets have more than eight open slots.
//
// The tiling, unit lists and tables are those of the FP32 form
// (sigma_pair_warp.cu).  The product Y_S = X_S K of a set needs about 50 bits.
// On the FP32 units a product and its sum in float pairs take 12 operations,
// and GB300's FP64 units do 1/64 of the FP32 rate.  Here a set's values
// are brought to a common exponent (the largest value's) and cut into five
// signed digits of eleven bits, K likewise once per handle; both are integers of
// magnitude at most 1,088 and exact in FP16, and a digit of X times a digit of K over
// the set's open slots is an integer that FP32 accumulates exactly (Ozaki, Ogita, Oishi
// and Rump, "Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication and its applications", 2012).  Digits i of
// X and j of K go into the accumulator of i + j = 2..6, digit 2 times digit 2 into
// one of its own.  |x_1| <= 512 and the host's check of K's digits keep the
// accumulators of i + j = 2, 3 and 4 below 2^24 for any X (with 2 x 2 in the
// accumulator of 4 a constant K of 24 open slots passed 2^24, at 1.5e-13); those of
// the smaller sums round only if the digits' signs conspire, by a few units of 2^-55
// where the largest |x| |K| is 2^-6 to 2^-4 (constant vectors and K, emulated: 2.6e-15
// of the sum of the terms).  What is cut is below 2^-51 of the largest |x| |K|.  The
// six sums are put together as a float
// pair with exact rounding errors.  The own row's sums stay float pairs in
// shared memory; what leaves the SM is widened to double by integer
// operations and added with FP64 atomics to sigma = diag x.
//
// Tensor memory holds two tiles (four digits of X: 64 columns, six
// accumulators: 192; the fifth digits lie in shared memory), so that warps 0-7
// gather, cut and hand over the next tile of a slot while warps 8-15 read and
// scatter the one before.
//
// Measured against one unit per block with float pairs on the FP32 units: L=32 N=16
// 134.6 -> 59.4 ms, L=28 N=14 7.33 -> 3.84 ms, L=23 N=9 159 -> 84 us (3.58 ms and
// 80 us with 2 x 2 in the accumulator of 4); the hop sums' error against FP64 sums 2.0e-15 to
// 3.3e-15 of their norm, from 3.5e-15 to 5.4e-15.  Bound by instruction issue
// (1,980 warp instructions per 32 sets, 58 % of the issue slots).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <numeric>
#include <vector>

#include "addressing.cuh"
#include "f32x2.cuh"
#include "ff.cuh"
#include "internal.h"
#include "pair_warp.h"
#include "pair_warp_index.cuh"
#include "tcgen.cuh"

namespace doci {
namespace {

constexpr int kSlots = 2;                   // tiles in flight
constexpr int kThreads64 = 2 * 128 * kSlots;
constexpr uint32_t kTmemCols = 512;         // per slot: A digits 1-4, 16 each (0..63) | D 6 x 32 (64..255)
// the accumulators of i + j = 2, 3, 4 (without 2 + 2), 5, 6 and of digits 2 and 2
constexpr int kColD = 64, kCol22 = kColD + 5 * 32;
// tcgen05 instruction descriptor: D FP32, A and B FP16, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc16(uint32_t n) {
  return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
// after K (5 digits x 32 rows of 32 FP16, 64 of 128 bytes, swizzled): a slot's
// fifth digits of X, 128 rows of the same form
constexpr int kOffX5 = 160 * 128, kX5Bytes = 128 * 128;
constexpr int kOffBar = kOffX5 + kSlots * kX5Bytes;
constexpr int kOffExp = kOffBar + 128;      // the sets' exponents: two tiles of 128 per slot
constexpr int kOffStart = kOffExp + kSlots * 2 * 128 * 4;
constexpr int kOffCells = kOffStart + 4 * 24 * (kThreads64 / 32);
constexpr size_t kMinSmem = 120 * 1024;     // one block per SM: it allocates all of the tensor memory

__device__ __forceinline__ uint32_t half2_bits(f2 v) {  // (FP16 of the first) | (FP16 of the second) << 16
  float a, b;
  up(v, a, b);
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ float2 lds64(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts64(uint32_t a, float x, float y) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ float2 ldg64_if(const ff *p, uint32_t on) {
  float2 v;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t@q "
      "ld.global.nc.v2.f32 {%0, %1}, [%2];\n\t}\n"
      : "=&f"(v.x), "=&f"(v.y)
      : "l"(p), "r"(on));
  return v;
}
__device__ __forceinline__ void red64_if(double *p, double v, uint32_t on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q red.global.add.f64 [%0], %1;\n\t}\n" ::"l"(p), "d"(v),
               "r"(on)
               : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// D = A B (+ D), A in tensor memory or, by its descriptor, in shared memory
__device__ __forceinline__ void mma_f16_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(id), "r"(acc));
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(id), "r"(acc));
}
// (h + l) 2^e as a double by integer operations, |l| at most an ulp of h, h 0
// or of magnitude 2^-74 .. 2^120 (the FP64 units convert one lane in 64
// cycles per quarter SM); nan: or-ed into the high word
__device__ __forceinline__ double widen(float h, float l, int e, uint32_t nan) {
  const uint32_t u = __float_as_uint(h), mag = u & 0x7fffffffu;
  const float unit = __uint_as_float((306u - (mag >> 23)) << 23);  // 2^52 / 2^exponent of h
  const int s = static_cast<int>(u) >> 31;
  int low = (__float2int_rn(l * unit) ^ s) - s;  // l in units of the double's last place, along h's sign
  if ((mag & 0x7fffffu) == 0 && low < 0) low += low;  // below a power of two the last place is half as much
  const unsigned long long m = (static_cast<unsigned long long>(mag) << 29) + static_cast<long long>(low);
  uint32_t hi = static_cast<uint32_t>(m >> 32) + 0x38000000u + (static_cast<uint32_t>(e) << 20);
  uint32_t lo = static_cast<uint32_t>(m);
  if (mag == 0) hi = lo = 0;
  return __hiloint2double(static_cast<int>(hi | (u & 0x80000000u) | nan), static_cast<int>(lo));
}

// DET: as in sigma_pair_warp.cu, contributions stored in slabs instead of added
template <int P, bool DET>
__global__ void __launch_bounds__(kThreads64, 1)
sigma_pair_warp64_kernel(const __grid_constant__ PwShape s, const uint32_t *__restrict__ units,
                         const uint32_t *__restrict__ rowstart, const uint4 *__restrict__ tab_a,
                         const uint2 *__restrict__ tab_b, const uint16_t *__restrict__ g_kdig, int kexp,
                         const ff *__restrict__ x, double *__restrict__ y, double *__restrict__ slab,
                         int *__restrict__ err) {
  constexpr int NR = 32 - P;
  constexpr int XC = pw::cells(P);
  extern __shared__ __align__(1024) uint8_t sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, slot = (warp >> 2) & 1, w4 = warp & 3;
  const bool gatherer = warp < 4 * kSlots;
  const uint32_t base = su32(sm);
  if (base & 1023u) {  // the swizzled K tile needs a 1024-byte aligned base
    if (tid == 0) atomicCAS(err, 0, 3);
    return;
  }
  const uint32_t bar_done = base + kOffBar + 8 * slot, bar_free = base + kOffBar + 16 + 8 * slot;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + kOffBar + 64) + slot;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + kOffBar + 96);
  float2 *cells = reinterpret_cast<float2 *>(sm + kOffCells) + warp * XC;
  const uint32_t ca = su32(cells), ra = base + kOffStart + warp * 96;

  for (int e = tid; e < 160 * 32; e += kThreads64) {
    const uint32_t r = e >> 5, k = e & 31;  // row (digit, orbital), orbital
    const uint32_t at = (r >> 3) * 1024u + (r & 7u) * 128u + ((((k >> 3) ^ r) & 7u) << 4) + (k & 7u) * 2u;
    *reinterpret_cast<uint16_t *>(sm + at) = g_kdig[e];
  }
  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) {
      // a tile's MMAs and the issuing thread (which makes the exponents visible)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(base + kOffBar + 8 * i));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(base + kOffBar + 16 + 8 * i));
      reinterpret_cast<volatile int *>(sm + kOffBar + 64)[i] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (lane == 0) cells[XC - 1] = make_float2(0.f, 0.f);
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
  const uint32_t tg = tmem + 256u * slot, tw = tg + (static_cast<uint32_t>(32 * w4) << 16);
  const int nks = (s.L + 15) >> 4;
  const uint64_t desc = smem_desc(base), desc5 = smem_desc(base + kOffX5 + slot * kX5Bytes);
  const uint32_t row5 = base + kOffX5 + slot * kX5Bytes + (4 * w4 + (lane >> 3)) * 1024 + (lane & 7) * 128;
  volatile uint32_t *exps = reinterpret_cast<volatile uint32_t *>(sm + kOffExp) + slot * 256 + 32 * w4 + lane;

  uint32_t n = 0;  // tiles of this slot so far
  bool ok = true, fail = false;
  for (int q = blockIdx.x * kSlots + slot; q < s.nquads && ok; q += gridDim.x * kSlots) {
    const uint32_t mask = units[4 * q + w4];
    const int jp = s.N - 1 - __popc(units[4 * q]);
    const uint32_t n_s = jp >= 0 ? s.n[jp] : 0u;
    const bool real = mask != pw::kNone;
    const uint32_t n_own = real && n_s ? s.n[jp + 1] : 0u;  // (without sets sigma is diag x, set before)
    const uint32_t holes = real ? ~mask & ((1u << s.na) - 1u) : 0u;
    const uint32_t own = n_own ? rowstart[mask] : 0u;
    for (uint32_t c = lane; c < n_own; c += 32) {
      float2 v = make_float2(0.f, 0.f);
      if (gatherer) v = __ldg(reinterpret_cast<const float2 *>(x) + own + c);
      cells[c] = v;
    }
    if (lane < 24) {
      const bool hole = n_s && ((holes >> lane) & 1u);
      uint32_t r = hole ? rowstart[mask | (1u << lane)] : 0u;
      if (DET && hole && !gatherer) r += s.D * static_cast<uint32_t>(__popc(mask & ((1u << lane) - 1u)));
      reinterpret_cast<uint32_t *>(sm + kOffStart)[warp * 24 + lane] = r;
    }
    __syncwarp();
    if (n_s == 0) continue;
    const uint4 *ta = tab_a + s.off[jp];
    const uint2 *tb = tab_b + s.off[jp];
    const uint32_t last = n_s - 1;

    if (gatherer) {
      for (uint32_t c0 = 0; c0 < n_s; c0 += 32, ++n) {
        float xh[32], xl[32];
        const ff *xr = x + min(c0 + lane, last);
#pragma unroll
        for (int b = 0; b < NR; b += 4) {
          const uint4 r = lds128(ra + 4 * b);
          const uint32_t st[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (b + i < NR) {
              const float2 v = ldg64_if(xr + st[i], holes & (1u << (b + i)));
              xh[P + b + i] = v.x;
              xl[P + b + i] = v.y;
            }
        }
        {
          uint32_t w[6];
          const uint4 ea = __ldg(ta + c0 + lane);
          w[0] = ea.x, w[1] = ea.y, w[2] = ea.z, w[3] = ea.w;
          if (P > 8) {
            const uint2 eb = __ldg(tb + c0 + lane);
            w[4] = eb.x, w[5] = eb.y;
          }
#pragma unroll
          for (int o = 0; o < P; ++o) {
            const float2 v = lds64(ca + 2 * (o & 1 ? w[o >> 1] >> 16 : w[o >> 1] & 0xffffu));
            xh[o] = v.x;
            xl[o] = v.y;
          }
        }
        // the set's exponent: the largest magnitude just below 2^(eb - 126)
        float big = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) big = fmaxf(big, fabsf(xh[i]));
        uint32_t eb = __float_as_uint(big) >> 23;
        eb = eb < 30u ? 30u : eb;
        const bool inf = eb == 255u;
        const float f1 = inf ? __uint_as_float(0x7fc00000u) : __uint_as_float((262u - eb) << 23);  // 2^(135 - eb)
        const float f3 = __uint_as_float((284u - (inf ? 30u : eb)) << 23);                         // 2^(157 - eb)
        if (n > 0 && !warp_wait(bar_done, (n - 1) & 1u, s.spin_limit, abort_flag, err, 31)) fail = true;
        if (!fail) {  // (else an MMA may still read the tile)
          fence_after();
          // five signed digits of eleven bits, most significant first:
          // X 2^(124 - eb) = sum_i d_i 2^(-11 i), below 1/4, d_i the nearest
          // integer each time, every remainder exact but the last bits of h + l
          // past 2^-57
          const f2 c2048 = pk(2048.f, 2048.f);
          const f2 magic = pk(12582912.f, 12582912.f), nmagic = pk(-12582912.f, -12582912.f);
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t d1[8], d2[8], d3[8], d4[8], d5[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int a = 16 * hf + 2 * i;
              const f2 r1 = pk(xh[a] * f1, xh[a + 1] * f1), lo = pk(xl[a] * f3, xl[a + 1] * f3);
              const f2 s1 = addp(addp(r1, magic), nmagic);
              const f2 r2 = mulp(subp(r1, s1), c2048);
              const f2 s2 = addp(addp(r2, magic), nmagic);
              const f2 u = subp(r2, s2);
              const f2 s3 = addp(addp(fma2(u, c2048, lo), magic), nmagic);
              const f2 r4 = mulp(addp(fma2(u, c2048, mulp(s3, pk(-1.f, -1.f))), lo), c2048);
              const f2 s4 = addp(addp(r4, magic), nmagic);
              const f2 r5 = mulp(subp(r4, s4), c2048);
              const f2 s5 = addp(addp(r5, magic), nmagic);
              d1[i] = half2_bits(s1);
              d2[i] = half2_bits(s2);
              d3[i] = half2_bits(s3);
              d4[i] = half2_bits(s4);
              d5[i] = half2_bits(s5);
            }
            tst8(tw + 8 * hf, d1);
            tst8(tw + 16 + 8 * hf, d2);
            tst8(tw + 32 + 8 * hf, d3);
            tst8(tw + 48 + 8 * hf, d4);
            sts128(row5 + (((2 * hf) ^ (lane & 7)) << 4), d5[0], d5[1], d5[2], d5[3]);
            sts128(row5 + (((2 * hf + 1) ^ (lane & 7)) << 4), d5[4], d5[5], d5[6], d5[7]);
          }
          exps[128 * (n & 1u)] = eb;
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          fence_before();
        }
        if (group_meet(slot, fail)) {
          ok = false;
          break;
        }
        if (w4 == 0) {
          // D of the tile before has to be read
          if (n > 0 && !warp_wait(bar_free, (n - 1) & 1u, s.spin_limit, abort_flag, err, 32)) fail = true;
          if (!fail && lane == 0) {
            fence_after();
            // digit i of X times digits 1..6-i of K (32 rows of 128 bytes per
            // digit) into the accumulators of i + j; 2 x 2 apart
            auto kd = [&](int j, int ks) { return desc + 256 * (j - 1) + 2 * ks; };
            auto col = [&](int g) { return tg + kColD + 32 * (g - 2); };
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
              if (ks < nks) mma_f16(col(2), tg + 8 * ks, kd(1, ks), idesc16(160), ks);
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
              if (ks < nks) {
                const uint32_t x2 = tg + 16 + 8 * ks;
                mma_f16(col(3), x2, kd(1, ks), idesc16(32), 1);
                mma_f16(tg + kCol22, x2, kd(2, ks), idesc16(32), ks);
                mma_f16(col(5), x2, kd(3, ks), idesc16(64), 1);
                mma_f16(col(4), tg + 32 + 8 * ks, kd(1, ks), idesc16(96), 1);
                mma_f16(col(5), tg + 48 + 8 * ks, kd(1, ks), idesc16(64), 1);
                mma_f16_ss(col(6), desc5 + 2 * ks, kd(1, ks), idesc16(32), 1);
              }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_done)
                         : "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_done) : "memory");
          }
          __syncwarp();
        }
      }
    } else {
      for (uint32_t c0 = 0; c0 < n_s; c0 += 32, ++n) {
        uint32_t w[6];
        const uint4 ea = __ldg(ta + c0 + lane);
        w[0] = ea.x, w[1] = ea.y, w[2] = ea.z, w[3] = ea.w;
        if (P > 8) {
          const uint2 eb = __ldg(tb + c0 + lane);
          w[4] = eb.x, w[5] = eb.y;
        }
        if (!warp_wait(bar_done, n & 1u, s.spin_limit, abort_flag, err, 33)) {
          ok = false;
          break;
        }
        fence_after();
        float yh[32], yl[32];
        const uint32_t eb = exps[128 * (n & 1u)];
        const f2 q11 = pk(0x1p-11f, 0x1p-11f);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          float D[6][8];
#pragma unroll
          for (int g = 0; g < 6; ++g) tld8(tw + kColD + 32 * g + 8 * ch, D[g]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          // sum_g D_g 2^(-11 (g - 1)) as a pair: each step's rounding error is
          // exact and carried (the first four are integers below 2^24, so the sum
          // of the two of i + j = 4 is off by at most one)
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const f2 D1 = pk(D[0][i], D[0][i + 1]), D2 = pk(D[1][i], D[1][i + 1]);
            const f2 D4 = pk(D[2][i], D[2][i + 1]), D22 = pk(D[5][i], D[5][i + 1]), D3 = addp(D4, D22);
            const f2 off = subp(D22, subp(D3, D4));
            const f2 a = fma2(pk(D[4][i], D[4][i + 1]), q11, pk(D[3][i], D[3][i + 1]));
            const f2 bh = fma2(a, q11, D3), bl = addp(fma2(a, q11, subp(D3, bh)), off);
            const f2 ch2 = fma2(bh, q11, D2), cl = fma2(bl, q11, fma2(bh, q11, subp(D2, ch2)));
            const f2 dh = fma2(ch2, q11, D1), dl = fma2(cl, q11, fma2(ch2, q11, subp(D1, dh)));
            const f2 h = addp(dh, dl), l = subp(dl, subp(h, dh));
            up(h, yh[8 * ch + i], yh[8 * ch + i + 1]);
            up(l, yl[8 * ch + i], yl[8 * ch + i + 1]);
          }
        }
        fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_free) : "memory");
        const int e = static_cast<int>(eb) - 124 + kexp - 22;  // the pairs' unit
        {
          // own row, as float pairs: one orbital at a time no two sets meet
          const int e1 = e / 2;
          const float sc1 = __uint_as_float(static_cast<uint32_t>(127 + e1) << 23);
          const float sc2 = __uint_as_float(static_cast<uint32_t>(127 + e - e1) << 23);
#pragma unroll
          for (int o = 0; o < P; ++o) {
            const uint32_t a = ca + 2 * (o & 1 ? w[o >> 1] >> 16 : w[o >> 1] & 0xffffu);
            const float2 v = lds64(a);
            const ff t = ff(v.x, v.y) + ff(yh[o] * sc1 * sc2, yl[o] * sc1 * sc2);
            sts64(a, t.h, t.l);
            __syncwarp();
          }
        }
        double *yr = (DET ? slab : y) + c0 + lane;
        const uint32_t add = c0 + lane <= last ? holes : 0u;
        // a NaN or an infinity among the set's values makes every product NaN
        const uint32_t nan = yh[0] == yh[0] ? 0u : 0x7ff80000u;
#pragma unroll
        for (int b = 0; b < NR; b += 4) {
          const uint4 r = lds128(ra + 4 * b);
          const uint32_t st[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (b + i < NR && (holes & (1u << (b + i)))) {
              const double v = widen(yh[P + b + i], yl[P + b + i], e, nan);
              if (!DET) red64_if(yr + st[i], v, add & (1u << (b + i)));
              else if (add) yr[st[i]] = v;
            }
        }
      }
      __syncwarp();
      if (ok)
        for (uint32_t c = lane; c < n_own; c += 32) {
          const float2 v = cells[c];
          const uint32_t mag = __float_as_uint(v.x) & 0x7fffffffu;
          // renormalised; values out of the integer path's range through the FP64 units
          const float h = v.x + v.y, l = v.y - (h - v.x);
          const uint32_t mh = __float_as_uint(h) & 0x7fffffffu;
          const bool plain = mag < 0x7b800000u && (mh == 0 || mh > 0x1a800000u);
          const double t = plain ? widen(h, l, 0, 0u) : static_cast<double>(v.x) + static_cast<double>(v.y);
          if (DET) y[own + c] += t;
          else atomicAdd(y + own + c, t);
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

// sigma = diag x and x as float pairs
__global__ void init64_kernel(uint32_t D, const double *__restrict__ diag, const double *__restrict__ x,
                              double *__restrict__ y, ff *__restrict__ xf) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < D; t += gridDim.x * blockDim.x) {
    const double v = x[t];
    y[t] = diag[t] * v;
    xf[t] = ff_from(v);
  }
}

template <int P, bool DET>
int launch_p(const doci_ham *h, const PwShape &s, const ff *x, double *y, double *slab, cudaStream_t st) {
  const size_t smem = std::max(kMinSmem, static_cast<size_t>(kOffCells) + 8 * pw::cells(P) * (kThreads64 / 32));
  int per_sm = 1;
  const int r = kernel_blocks(reinterpret_cast<const void *>(sigma_pair_warp64_kernel<P, DET>), kThreads64, smem, &per_sm);
  if (r != DOCI_OK) return r;
  const int grid = std::min(device_sm_count(), (s.nquads + kSlots - 1) / kSlots);
  sigma_pair_warp64_kernel<P, DET><<<grid, kThreads64, smem, st>>>(
      s, h->d_wunits, h->d_wstart, static_cast<const uint4 *>(h->d_wtab_a), static_cast<const uint2 *>(h->d_wtab_b),
      h->d_kdig, h->kdig_exp, x, y, slab, h->d_tc_err);
  DOCI_CUDA(cudaGetLastError());
  return DOCI_OK;
}

}  // namespace

// K (mirrored orbitals) as five signed digits of eleven bits, below 1/4:
// K = 2^exp sum_j k_j 2^(-11 j), FP16, digit j at [j - 1][32][32].  The
// accumulators of i + j = 2, 3 and 4 (2 x 2 apart) have to hold their sums
// exactly whatever X: |x_1| <= 512, |x_2| <= 1024, |x_3| <= 1088 (the low part comes in
// there) over the L - N + 1 open slots of a set.  Where K's digits do not allow that,
// other digits are tried (a larger exponent, at a bit of K each); kdig_ok is false when
// none do.
//
// The digits keep K to 2^-56 of 2^exp, the float-pair kernel each element of K
// to itself, so small elements beside large ones have fewer bits here.  kdig_ok
// asks that 2^(exp - 2), which is the power of two above the largest element (or
// up to four bits more), be at most 18 times the smallest one that is not
// zero: up to there this form's products are as exact, element by element
// (largest error of a product with that smallest element, emulated, against
// float pairs: 16 times 1.1e-14 and 1.4e-14, 18 times 1.25e-14 and 1.3e-14, 20
// times 1.35e-14 and 1.2e-14; 1e4 times 3e-12).  A K that is graded more (core
// orbitals, separate fragments) runs the float-pair kernel.
int ham_build_kdigits(doci_ham *h) {
  const int L = h->L, open = L - h->N + 1;
  double big = 0, small = INFINITY;
  bool finite = true;
  for (double k : h->Kp) {
    big = std::max(big, std::fabs(k));
    if (k != 0) small = std::min(small, std::fabs(k));
    finite = finite && std::isfinite(k);
  }
  h->kdig_ok = false;
  if (!finite) return DOCI_OK;
  int ex = 0;
  std::frexp(big, &ex);  // big < 2^ex
  if (ex < -100 || ex > 100) return DOCI_OK;  // (the kernel's scale factors are floats)
  std::vector<uint16_t> dig(5 * 1024, 0);
  for (h->kdig_exp = ex + 2; !h->kdig_ok && h->kdig_exp <= ex + 6; ++h->kdig_exp) {
    if (big > 0 && std::ldexp(1.0, h->kdig_exp - 2) > 18 * small) break;
    double worst = 0;
    const double scale = std::ldexp(1.0, -h->kdig_exp);
    for (int a = 0; a < L; ++a) {
      double sums[3][kMaxOrbitals];
      for (int b = 0; b < L; ++b) {
        double v = h->Kp[(L - 1 - a) * L + (L - 1 - b)] * scale, k[5];
        for (int j = 0; j < 5; ++j) {
          v *= 2048;
          const double d = std::nearbyint(v);
          v -= d;
          k[j] = std::fabs(d);
          const __half hd = __float2half(static_cast<float>(d));
          dig[j * 1024 + a * 32 + b] = *reinterpret_cast<const uint16_t *>(&hd);
        }
        sums[0][b] = 1024 * k[0] + 512 * k[1];  // (i + j = 2, 512 k[0], is below it)
        sums[1][b] = 1088 * k[0] + 512 * k[2];
        sums[2][b] = 1024 * k[1];
      }
      const int n = std::min(open, L);
      for (auto &s : sums) {
        if (n < L) std::nth_element(s, s + n, s + L, std::greater<double>());
        worst = std::max(worst, std::accumulate(s, s + n, 0.0));
      }
    }
    // (a margin for the sum of the two of i + j = 4, formed from their rounded sum)
    h->kdig_ok = worst <= 16777216.0 - 1024.0;
  }
  if (!h->kdig_ok) return DOCI_OK;
  --h->kdig_exp;
  DOCI_CUDA(cudaMallocAsync(&h->d_kdig, dig.size() * sizeof(uint16_t), h->stream));
  DOCI_CUDA(cudaMemcpyAsync(h->d_kdig, dig.data(), dig.size() * sizeof(uint16_t), cudaMemcpyHostToDevice, h->stream));
  return DOCI_OK;
}

bool pair_warp64_fits(const doci_ham *h) { return pair_warp_fits(h) && h->kdig_ok; }

// A set's work here is the same whatever its open slots, a float pair's goes with
// their square: with up to eight slots (L - N + 1) the float-pair kernel is the faster,
// from nine on this one.  Measured (us, float pairs / here): 7 slots L=26 N=20 116
// / 162, L=32 N=26 632 / 714; 8 slots L=30 N=23 631 / 822, L=32 N=25 1,298 / 1,637,
// L=22 N=15 equal; 9 slots L=28 N=20 1.19 times, L=24 N=16 1.21 and L=22 N=14 1.28
// times faster here.  (The reproducible form runs here in any case.)
bool pair_warp64_wanted(const doci_ham *h) { return pair_warp64_fits(h) && h->L - h->N + 1 > 8; }

namespace {
template <bool DET>
int launch64(const doci_ham *h, const double *x, double *y, double *slab, cudaStream_t st) {
  if (!pair_warp64_fits(h)) return DOCI_ERR_INVALID;
  ff *xf = nullptr;
  DOCI_CUDA(cudaMallocAsync(&xf, sizeof(ff) * static_cast<size_t>(h->D), st));
  init64_kernel<<<static_cast<unsigned>(std::min<uint64_t>((static_cast<uint64_t>(h->D) + 255) / 256,
                                                           8ull * device_sm_count())),
                  256, 0, st>>>(h->D, h->d_diag, x, y, xf);
  int r = cuda_ok("init64_kernel");
  if (r == DOCI_OK) {
    const PwShape s = pair_warp_shape(h);
    r = h->wsplit == 12   ? launch_p<12, DET>(h, s, xf, y, slab, st)
        : h->wsplit == 10 ? launch_p<10, DET>(h, s, xf, y, slab, st)
                          : launch_p<8, DET>(h, s, xf, y, slab, st);
  }
  const cudaError_t ef = cudaFreeAsync(xf, st);
  if (r != DOCI_OK) return r;
  DOCI_CUDA(ef);
  return DOCI_OK;
}
}  // namespace

int launch_pair_warp64(const doci_ham *h, const double *x, double *y, cudaStream_t st) {
  return launch64<false>(h, x, y, nullptr, st);
}

int launch_pair_warp64_det(const doci_ham *h, const double *x, double *y, double *slab, cudaStream_t st) {
  const int r = launch64<true>(h, x, y, slab, st);
  return r == DOCI_OK ? launch_sum_slabs(h, slab, y, st) : r;
}

}  // namespace doci
