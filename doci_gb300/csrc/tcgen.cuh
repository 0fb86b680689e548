// tcgen.cuh -- PTX wrappers of the warp-per-unit pair kernels: shared-memory
// accesses, predicated global ones, mbarrier polls, tensor-memory loads and
// stores, the shared-memory operand descriptor.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace doci {
namespace {

__device__ __forceinline__ uint32_t su32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ float lds(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts(uint32_t a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
// *p where on, else 0; *p += v where on (predicated: `on` is the same in the whole warp or the lane is idle)
__device__ __forceinline__ float ldg_if(const float *p, uint32_t on) {
  float v;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}\n"
      : "=&f"(v)
      : "l"(p), "r"(on));
  return v;
}
__device__ __forceinline__ void red_if(float *p, float v, uint32_t on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q red.global.add.f32 [%0], %1;\n\t}\n" ::"l"(p), "f"(v),
               "r"(on)
               : "memory");
}
__device__ __forceinline__ void st_if(float *p, float v, uint32_t on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f32 [%0], %1;\n\t}\n" ::"l"(p), "f"(v),
               "r"(on)
               : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(a), "r"(parity), "r"(1000u)
      : "memory");
  return ok != 0;
}
// the four warps of warpgroup wg meet (named barrier wg + 1); true when any of them failed
__device__ __forceinline__ bool group_meet(int wg, bool fail) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, "
      "q;\n\t}\n"
      : "=r"(r)
      : "r"(static_cast<uint32_t>(fail)), "r"(wg + 1)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  // K-major, 128-byte swizzle: leading offset unused (16 B), 8-row groups 1024 B apart, version 1
  return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(1) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
         (static_cast<uint64_t>(2) << 61);
}
__device__ __forceinline__ void tst8(uint32_t t, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(t), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tld8(uint32_t t, float (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
               : "r"(t));
}
__device__ __forceinline__ void tst1(uint32_t t, uint32_t r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(t), "r"(r) : "memory");
}
__device__ __forceinline__ uint32_t tld1(uint32_t t) {
  uint32_t r;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(t));
  return r;
}
// bounded wait by a whole warp; false when it ran out or the slot was given up
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, long limit, volatile int *abort_flag, int *err,
                                          int code) {
  bool done = false;
  for (long k = 0; k < limit && !done; ++k) {
    done = mbar_try(bar, parity);
    if (!done && (k & 63) == 63 && *abort_flag) break;
  }
  done = __all_sync(0xffffffffu, done);
  if (!done && (threadIdx.x & 31) == 0) {
    *abort_flag = 1;
    atomicCAS(err, 0, code);
  }
  return done;
}
// byte offset of element (row r, column k) of a 128-byte-swizzled K-major tile of 32 FP32 per row
__host__ __device__ __forceinline__ uint32_t sw128(uint32_t r, uint32_t k) {
  return (r >> 3) * 1024u + (r & 7u) * 128u + ((((k >> 2) ^ r) & 7u) << 4) + (k & 3u) * 4u;
}

}  // namespace
}  // namespace doci
