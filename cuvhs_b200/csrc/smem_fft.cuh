// FP32 complex FFT parts (sm_100a): the butterflies and twiddles that every
// transform here is made of, and a transform in shared memory by two warps.
//
// Stockham auto-sort, radix-16 passes (plus one radix-2/4/8 pass for sizes that
// are not a power of 16).  Each thread holds its butterflies' inputs in
// registers, so one padded buffer serves as both source and destination of a
// pass (read all -> barrier -> write all -> barrier).  Index i lives at i + i/16
// so the stride-16 writes of the first pass do not collide on banks.
// Twiddles come from a per-pass table computed in FP64 on the host and
// rounded once to FP32: pass NS (>= 16) stores W_{NS*R}^{r*k} at
// (NS - 16) + (r - 1) * NS + k, so a warp's twiddle loads (consecutive k) are
// contiguous.  fft_twiddle_count(N) entries in all.
//
// Complex arithmetic is packed (packed.cuh): a complex value is one register
// pair, an addition one instruction, a product two.  The products' rounding is
// written out (fma(a, b, -(c*d)), fma(a, b, c*d)) instead of left to the
// compiler, so the same transform rounds alike in every kernel.
#pragma once
#include "packed.cuh"

namespace cuvhs {

__host__ __device__ constexpr int fft_pad(int n) { return n + (n >> 4); }

// The thread index as a value the compiler cannot prove equal to its source.
// Two transforms in one kernel compute the same shared-memory and twiddle
// offsets; given the plain index the compiler keeps the first transform's
// offsets live until the second uses them, which spills the transforms' data.
__device__ __forceinline__ int opaque_index(int t) {
  int r;
  asm volatile("mov.u32 %0, %1;" : "=r"(r) : "r"(t));
  return r;
}

// Radix of the pass that starts at span NS in an N-point transform.
__host__ __device__ constexpr int fft_radix(int N, int NS) { return NS * 16 <= N ? 16 : N / NS; }
// Entries of the per-pass twiddle table of an N-point transform.
__host__ __device__ constexpr int fft_twiddle_count(int N) {
  int n = 0;
  for (int ns = 16; ns < N; ns *= 16) n += (fft_radix(N, ns) - 1) * ns;
  return n;
}
__device__ __forceinline__ int pidx(int i) { return i + (i >> 4); }

// a * w (forward) or a * conj(w) (inverse)
template <bool INV>
__device__ __forceinline__ float2 cmul_tw(float2 a, float2 w) {
  if (INV) return parts(f2_fma(f2(a), f2(w.x, w.x), f2(a.y, a.x) * f2(w.y, -w.y)));
  return parts(f2_fma(f2(a.x, a.x), f2(w), f2(a.y, a.y) * f2(-w.y, w.x)));
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return parts(f2(a) + f2(b)); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return parts(f2(a) - f2(b)); }

// multiply by -i (forward) / +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 mul_mi(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// e^{-+2 pi i m / 16} constants
struct Root16 {
  static constexpr float c[16] = {1.0f, 0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f,
                                  0.0f, -0.38268343236508977f, -0.70710678118654752f, -0.92387953251128674f,
                                  -1.0f, -0.92387953251128674f, -0.70710678118654752f, -0.38268343236508977f,
                                  0.0f, 0.38268343236508977f, 0.70710678118654752f, 0.92387953251128674f};
  static constexpr float s[16] = {0.0f, 0.38268343236508977f, 0.70710678118654752f, 0.92387953251128674f,
                                  1.0f, 0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f,
                                  0.0f, -0.38268343236508977f, -0.70710678118654752f, -0.92387953251128674f,
                                  -1.0f, -0.92387953251128674f, -0.70710678118654752f, -0.38268343236508977f};
};

// v * W_R^m with R | 16 (m in units of 1/R turn)
template <int R, int M, bool INV>
__device__ __forceinline__ float2 rot(float2 v) {
  constexpr int m16 = (M * (16 / R)) & 15;
  if (m16 == 0) return v;
  if (m16 == 4) return mul_mi<INV>(v);
  if (m16 == 8) return make_float2(-v.x, -v.y);
  if (m16 == 12) return mul_mi<!INV>(v);
  const float c = Root16::c[m16];
  const float s = INV ? Root16::s[m16] : -Root16::s[m16];
  if (!INV && (m16 == 1 || m16 == 3)) return parts(f2_fma(f2(v), f2(c, c), f2(v.y, v.x) * f2(-s, s)));
  return parts(f2_fma(f2(v.x, v.x), f2(c, s), f2(v.y, v.y) * f2(-s, c)));
}

template <bool INV>
__device__ __forceinline__ void dft2(float2& a, float2& b) {
  float2 t = a;
  a = cadd(t, b);
  b = csub(t, b);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  float2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = mul_mi<INV>(csub(a1, a3));
  a0 = cadd(t0, t2);
  a2 = csub(t0, t2);
  a1 = cadd(t1, t3);
  a3 = csub(t1, t3);
}

// In-register DFT of size R, in place.  Output bin r ends up in v[dft_slot<R>(r)]
// (a compile-time permutation, free once the loops are unrolled).
template <int R>
__host__ __device__ constexpr int dft_slot(int r) {
  return R == 16 ? 4 * (r & 3) + (r >> 2) : (R == 8 ? 2 * (r & 3) + (r >> 2) : r);
}

// Second half of dft<16>: the inner turns and the dft4 over n2.
template <bool INV>
__device__ __forceinline__ void dft16_second(float2* v) {
  v[4 + 1] = rot<16, 1, INV>(v[4 + 1]);
  v[4 + 2] = rot<16, 2, INV>(v[4 + 2]);
  v[4 + 3] = rot<16, 3, INV>(v[4 + 3]);
  v[8 + 1] = rot<16, 2, INV>(v[8 + 1]);
  v[8 + 2] = rot<16, 4, INV>(v[8 + 2]);
  v[8 + 3] = rot<16, 6, INV>(v[8 + 3]);
  v[12 + 1] = rot<16, 3, INV>(v[12 + 1]);
  v[12 + 2] = rot<16, 6, INV>(v[12 + 2]);
  v[12 + 3] = rot<16, 9, INV>(v[12 + 3]);
#pragma unroll
  for (int k1 = 0; k1 < 4; k1++) dft4<INV>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2* v) {
  if constexpr (R == 2) {
    dft2<INV>(v[0], v[1]);
  } else if constexpr (R == 4) {
    dft4<INV>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    // 8 = 4 (n1) x 2 (n2): x[2 n1 + n2]; bin k1 + 4 k2 lands in v[2 k1 + k2]
    dft4<INV>(v[0], v[2], v[4], v[6]);
    dft4<INV>(v[1], v[3], v[5], v[7]);
    v[3] = rot<8, 1, INV>(v[3]);
    v[5] = rot<8, 2, INV>(v[5]);
    v[7] = rot<8, 3, INV>(v[7]);
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) dft2<INV>(v[2 * k1], v[2 * k1 + 1]);
  } else if constexpr (R == 16) {
    // 16 = 4 (n1) x 4 (n2): x[4 n1 + n2]; A[n2][k1] in v[4 k1 + n2];
    // bin k1 + 4 k2 lands in v[4 k1 + k2]
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) dft4<INV>(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
    dft16_second<INV>(v);
  }
}

// dft<16, INV> of g[i] * v[i] with real gains g, the products fused into the
// first additions.
template <bool INV>
__device__ __forceinline__ void dft16_gains(float2* v, const float* g) {
#pragma unroll
  for (int n2 = 0; n2 < 4; n2++) {
    const F2 g0 = f2(g[n2], g[n2]), g1 = f2(g[4 + n2], g[4 + n2]);
    const F2 g2 = f2(g[8 + n2], g[8 + n2]), g3 = f2(g[12 + n2], g[12 + n2]);
    const F2 a0 = f2(v[n2]), a1 = f2(v[4 + n2]), a2 = f2(v[8 + n2]), a3 = f2(v[12 + n2]);
    const F2 n2_ = f2(-v[8 + n2].x, -v[8 + n2].y), n3_ = f2(-v[12 + n2].x, -v[12 + n2].y);
    const F2 t0 = f2_fma(a0, g0, a2 * g2);
    const F2 t2 = f2_fma(a1, g1, a3 * g3);
    const F2 t1 = f2_fma(a0, g0, n2_ * g2);
    const F2 t3 = f2(mul_mi<INV>(parts(f2_fma(a1, g1, n3_ * g3))));
    v[n2] = parts(t0 + t2);
    v[8 + n2] = parts(t0 - t2);
    v[4 + n2] = parts(t1 + t3);
    v[12 + n2] = parts(t1 - t3);
  }
  dft16_second<INV>(v);
}

// dft<16, INV> of an input that is zero but for v[3], v[4], v[11] and v[12]
// (the others are not read): a band around a quarter of the sample rate and
// its mirror image.
template <bool INV>
__device__ __forceinline__ void dft16_band(float2* v) {
  // the dft4 over n1 of columns n2 = 0 and 3, for k1 = 0..3
  const float2 s0 = cadd(v[4], v[12]), d0 = mul_mi<INV>(csub(v[4], v[12]));
  const float2 s3 = cadd(v[3], v[11]), d3 = csub(v[3], v[11]);
  const float2 a0[4] = {s0, d0, make_float2(-s0.x, -s0.y), make_float2(-d0.x, -d0.y)};
  const float2 a3[4] = {s3, rot<16, 3, INV>(d3), rot<16, 6, INV>(s3), rot<16, 9, INV>(d3)};
#pragma unroll
  for (int k1 = 0; k1 < 4; k1++) {
    const float2 m = mul_mi<INV>(a3[k1]);
    v[4 * k1] = cadd(a0[k1], a3[k1]);
    v[4 * k1 + 2] = csub(a0[k1], a3[k1]);
    v[4 * k1 + 1] = csub(a0[k1], m);
    v[4 * k1 + 3] = cadd(a0[k1], m);
  }
}

// dft<16, INV> of an input whose upper half v[8..15] is zero (not read).
template <bool INV>
__device__ __forceinline__ void dft16_half(float2* v) {
#pragma unroll
  for (int n2 = 0; n2 < 4; n2++) {
    const float2 a = v[n2], b = v[4 + n2], c = mul_mi<INV>(b);
    v[n2] = cadd(a, b);
    v[4 + n2] = cadd(a, c);
    v[8 + n2] = csub(a, b);
    v[12 + n2] = csub(a, c);
  }
  dft16_second<INV>(v);
}

// Barrier of a transform's THREADS threads: a CTA, or one of the groups of 64 in
// a CTA, threads [64 g, 64 g + 64) on barrier 1 + g.
template <int THREADS>
__device__ __forceinline__ void fft_sync() {
  if constexpr (THREADS == 64) {
    // Immediate barrier ids: with a register id the compiler reserves all 16
    // barriers per CTA, which caps residency at 4 CTAs per SM.  The CTAs here
    // have two groups; a choice between two ids alone, as a branch or by
    // predicates, compiled to slower line kernels (40 fields and the trials
    // together 78 us: 79 and 83).
    const int g = threadIdx.x >> 6;
    if (g == 0) asm volatile("bar.sync 1, 64;" ::: "memory");
    else if (g == 1) asm volatile("bar.sync 2, 64;" ::: "memory");
    else if (g == 2) asm volatile("bar.sync 3, 64;" ::: "memory");
    else asm volatile("bar.sync 4, 64;" ::: "memory");
  } else {
    __syncthreads();
  }
}

// One Stockham pass of radix R on an N-point padded buffer, current span NS, by
// a group of 64 threads.
template <int N, int R, int NS, bool INV>
__device__ __forceinline__ void fft_pass(float2* s, const float2* __restrict__ tw, int tid) {
  constexpr int NB = N / R;
  constexpr int PER = NB / 64;
  static_assert(NB % 64 == 0, "whole butterflies a thread");
  float2 v[PER][R];
#pragma unroll
  for (int p = 0; p < PER; p++) {
    const int j = tid + p * 64;
#pragma unroll
    for (int r = 0; r < R; r++) v[p][r] = s[pidx(j + r * NB)];
    if constexpr (NS > 1) {
      const int k = j & (NS - 1);
      const float2* twp = tw + (NS - 16) + k;
#pragma unroll
      for (int r = 1; r < R; r++) v[p][r] = cmul_tw<INV>(v[p][r], __ldg(&twp[(r - 1) * NS]));
    }
    dft<R, INV>(v[p]);
  }
  fft_sync<64>();
#pragma unroll
  for (int p = 0; p < PER; p++) {
    const int j = tid + p * 64;
    const int k = j & (NS - 1);
    const int base = (j / NS) * NS * R + k;
#pragma unroll
    for (int r = 0; r < R; r++) s[pidx(base + r * NS)] = v[p][dft_slot<R>(r)];
  }
  fft_sync<64>();
}

// Full N-point transform by a group of 64 threads (N a power of two, at least
// 1024), natural order in and out, unnormalised.  The caller synchronises the
// group after filling s.  tid: this thread's index in its group.
template <int N, bool INV, int NS = 1>
__device__ __forceinline__ void smem_fft(float2* s, const float2* __restrict__ tw, int tid) {
  if constexpr (NS < N) {
    fft_pass<N, fft_radix(N, NS), NS, INV>(s, tw, tid);
    smem_fft<N, INV, NS * fft_radix(N, NS)>(s, tw, tid);
  }
}

}  // namespace cuvhs
