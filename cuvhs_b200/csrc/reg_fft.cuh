// Register-resident block FFT for T = N/16 threads (sm_100a): a CTA, or for N =
// 1024 a group of two warps.
//
// Thread t owns elements t + T*q, q = 0..15, of an N-point transform, both on
// entry (natural-order input) and on exit (natural-order output): radix-16
// passes (and one final radix 2/4/8 when N is not a power of 16) exchange data
// through a padded shared buffer between passes, but the first
// pass reads its inputs from registers and the last pass leaves its outputs in
// registers.  Since the output layout equals the input layout, a forward
// transform, a per-bin multiply and an inverse transform chain without any
// shared-memory round trip at the seams, and inputs/outputs move between HBM
// and registers with coalesced accesses (consecutive threads, consecutive
// elements).  Twiddles: the per-pass table of smem_fft.cuh (coalesced loads).
//
// The butterflies and twiddles are those of the Stockham passes of
// smem_fft.cuh, but a pass between the first and the last writes each output
// back where its butterfly read an input.  So a warp goes from its reads
// through the arithmetic to its writes without waiting for the others, one
// barrier a pass instead of two, and warps in different parts of a pass fill
// the FP32 pipe, the load/store unit and shared memory side by side.  (With a
// barrier between reads and writes all warps of a CTA met in the same unit:
// issue at 45-47% of cycles with every unit below 37%.)  The logical index i
// of pass p lies at: pass 2, i; pass 3, i with its two lowest base-16 digits'
// butterfly undone, and so on -- in each pass a constant stride for a
// butterfly's slots and 16 consecutive elements for 16 consecutive threads,
// hence no bank conflicts.
#pragma once
#include "smem_fft.cuh"

namespace cuvhs {

template <int N>
struct RegFFT {
  static_assert(N >= 1024 && N <= 16384 && (N & (N - 1)) == 0, "two radix-16 passes or three, and a smaller last one");
  static constexpr int T = N / 16;

  // Padded location of slot 0 of thread t's (first) butterfly in the pass of
  // span NS, and the strides from slot to slot and from butterfly to butterfly
  // (logical inputs t + T*b + r*N/R).
  template <int NS>
  __device__ __forceinline__ static int place(int t) {
    const int lo = t & 15, mid = ((t >> 4) & 15) * T, hi = t >> 8;
    if constexpr (NS == 16) return pidx(t);
    else if constexpr (N < 4096) return pidx(lo + (t >> 4) * T);
    else if constexpr (NS == 256) return pidx(hi * 16 + lo + mid);
    else return pidx(hi * (T / 16) + lo + mid);
  }
  template <int NS>
  __host__ __device__ static constexpr int slot_stride() {
    return NS == 16 ? fft_pad(T) : (NS == 256 && N >= 4096 ? fft_pad(T / 16) : 17);
  }
  template <int NS>
  __host__ __device__ static constexpr int butterfly_stride() {  // the last pass has several where N is no power of 16
    return N < 4096 ? fft_pad((T / 16) * T) : fft_pad((T / 256) * (T / 16));
  }

  // One pass of radix R at span NS (> 1).  LAST leaves the results in v in the
  // t + T*q layout.
  template <int NS, bool INV, bool LAST>
  __device__ __forceinline__ static void pass(float2 (&v)[16], float2* s, const float2* __restrict__ tw, int t) {
    constexpr int R = fft_radix(N, NS);
    constexpr int B = 16 / R;  // butterflies per thread
    static_assert(LAST || B == 1, "only the last pass has a smaller radix");
    float2* p = s + place<NS>(t);
    float2 w[B][R];
#pragma unroll
    for (int b = 0; b < B; b++) {
      const int k = (t + T * b) & (NS - 1);
      const float2* twp = tw + (NS - 16) + k;
      w[b][0] = p[b * butterfly_stride<NS>()];
#pragma unroll
      for (int r = 1; r < R; r++)
        w[b][r] = cmul_tw<INV>(p[b * butterfly_stride<NS>() + r * slot_stride<NS>()], __ldg(&twp[(r - 1) * NS]));
      dft<R, INV>(w[b]);
    }
    if constexpr (LAST) {
#pragma unroll
      for (int b = 0; b < B; b++)
#pragma unroll
        for (int r = 0; r < R; r++) v[b + B * r] = w[b][dft_slot<R>(r)];
    } else {
#pragma unroll
      for (int r = 0; r < R; r++) p[r * slot_stride<NS>()] = w[0][dft_slot<R>(r)];
      fft_sync<T>();
    }
  }

  template <int NS, bool INV>
  __device__ __forceinline__ static void rest(float2 (&v)[16], float2* s, const float2* __restrict__ tw, int t) {
    constexpr bool LAST = NS * fft_radix(N, NS) >= N;
    pass<NS, INV, LAST>(v, s, tw, t);
    if constexpr (!LAST) rest<NS * fft_radix(N, NS), INV>(v, s, tw, t);
  }

  // Transform v in place.  The buffer s (fft_pad(N) float2) may be in use by
  // the caller until this call: the first write waits on a barrier.  On return
  // other threads may still be reading s: a barrier comes before its next use.
  template <bool INV>
  __device__ __forceinline__ static void run(float2 (&v)[16], float2* s, const float2* __restrict__ tw, int t) {
    // pass NS = 1: butterfly t reads elements t + T*r, all held by this thread
    dft<16, INV>(v);
    after_first<INV>(v, s, tw, t);
  }

  // run() of an input whose upper half (slots 8..15) is zero; v[8..15] is not read.
  template <bool INV>
  __device__ __forceinline__ static void run_half(float2 (&v)[16], float2* s, const float2* __restrict__ tw, int t) {
    dft16_half<INV>(v);
    after_first<INV>(v, s, tw, t);
  }

  // run() of g[q] * v[q], real gains.
  template <bool INV>
  __device__ __forceinline__ static void run_gains(float2 (&v)[16], const float (&g)[16], float2* s,
                                                   const float2* __restrict__ tw, int t) {
    dft16_gains<INV>(v, g);
    after_first<INV>(v, s, tw, t);
  }

  // run() of an input that is zero but for slots 3, 4, 11 and 12.
  template <bool INV>
  __device__ __forceinline__ static void run_band(float2 (&v)[16], float2* s, const float2* __restrict__ tw, int t) {
    dft16_band<INV>(v);
    after_first<INV>(v, s, tw, t);
  }

  template <bool INV>
  __device__ __forceinline__ static void after_first(float2 (&v)[16], float2* s, const float2* __restrict__ tw,
                                                     int t) {
    fft_sync<T>();
#pragma unroll
    for (int r = 0; r < 16; r++) s[pidx(16 * t + r)] = v[dft_slot<16>(r)];
    fft_sync<T>();
    rest<16, INV>(v, s, tw, t);
  }
};

}  // namespace cuvhs
