// Tensor memory as a thread's own store (sm_100a).
//
// An SM's 256 KB of tensor memory is addressed by warps: warp w of a CTA
// reaches lanes 32 * (w % 4) .. + 31, one 32-bit word per column and lane, so
// a thread can put registers away in columns of its own and take them back
// without shared memory.  A CTA allocates columns (a power of two >= 32 of the
// SM's 512; the allocation waits while other CTAs of the SM hold too many) and
// frees them before it ends.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cuvhs {

// Warp 0 allocates COLS columns; the base address lands in *slot (shared).
// A __syncthreads() must follow before any thread reads it.
template <int COLS>
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, int warp) {
  static_assert(COLS >= 32 && COLS <= 512 && (COLS & (COLS - 1)) == 0, "columns: a power of two, 32..512");
  if (warp == 0) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(slot);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(a), "n"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
}
// After a __syncthreads() behind every thread's last load.  The warp frees as
// one (.aligned), whatever branches its threads took since.
template <int COLS>
__device__ __forceinline__ void tmem_free(uint32_t base, int warp) {
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(COLS));
  }
}
// The address of a warp's own columns: its lanes, `cols` columns a warp.
__device__ __forceinline__ uint32_t tmem_own(uint32_t base, int warp, int cols) {
  return base + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * cols);
}

// Eight words of this thread to / from columns [addr, addr + 8); whole warps.
__device__ __forceinline__ void tmem_st8(uint32_t addr, const float2 (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr),
               "r"(__float_as_uint(v[0].x)), "r"(__float_as_uint(v[0].y)), "r"(__float_as_uint(v[1].x)),
               "r"(__float_as_uint(v[1].y)), "r"(__float_as_uint(v[2].x)), "r"(__float_as_uint(v[2].y)),
               "r"(__float_as_uint(v[3].x)), "r"(__float_as_uint(v[3].y))
               : "memory");
}
// (The wait is part of the load: the registers hold nothing before it.)
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float2 (&v)[4]) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
// The 32 words stored at [addr, addr + 32).
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float2 (&v)[16]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
// After the thread's stores, before its loads of them.
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

}  // namespace cuvhs
