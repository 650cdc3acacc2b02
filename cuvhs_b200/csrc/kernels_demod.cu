// FM demodulation kernels (reference stage K1, src/pipeline/fm_demod.cu:396-485)
// and the sync-threshold edge finder (replaces the per-field serial scans of
// src/pipeline/vsync_discover.cu:5-45 and src/pipeline/sync_pulses.cu:10-58).
//
// Each tile f of the reference covers chunk samples [f*spp - 2048, f*spp - 2048 + tile)
// (clamped to the chunk) and is filtered circularly.  A CTA here computes two
// adjacent runs of one tile's outputs: gather both block windows (mod tile,
// clamped) as the real and imaginary parts of one input, forward FFT,
// separate and multiply by the block spectrum of the truncated kernel,
// inverse FFT per block, emit the valid middles.  HBM traffic is the stage interface only: K1a reads u8 and writes the
// FP32 demod and envelope; K1b reads the demod and writes video and sync.
#include <cuda_runtime.h>

#include "chain.cuh"
#include "cuvhs_internal.h"
#include "raw_input.cuh"
#include "reg_fft.cuh"
#include "tmem.cuh"

namespace cuvhs {
namespace {

constexpr int kThreadsA = Design::kNa / 16;
constexpr int kThreadsB = Design::kNb / 16;
// K1a: the exchange buffer and half a spectrum; K1b: the exchange buffer, with
// a spectrum of 32 words a thread in tensor memory
constexpr size_t kSmemA = sizeof(float2) * (fft_pad(Design::kNa) + Design::kNa / 2);
constexpr size_t kSmemB = sizeof(float2) * fft_pad(Design::kNb);
constexpr int kTmemColsB = 32 * (kThreadsB / 128);

__device__ __forceinline__ int wrap_tile(int q, int tile) {
  return q < 0 ? q + tile : (q >= tile ? q - tile : q);
}

// Both demod stages filter a real signal with a complex kernel g, so one CTA
// takes two adjacent blocks x1, x2 of a tile in one forward transform of
// u = x1 + i*x2.  With m = -k mod N, X1[k] = (U[k] + conj(U[m]))/2 and
// X2[k] = (U[k] - conj(U[m]))/2i, so Z1 = X1*g and Z2 = X2*g follow from U and
// its mirror (g is stored halved); each is inverted on its own.  Three
// transforms serve two blocks instead of four.  The analytic-signal kernel of
// K1a has no negative frequencies: its bins k >= N/2 are not formed and the
// inverse's first pass is that of a half-empty input.
//
// Bin k of both blocks: u = U[k], um = U[m], g = g[k].
__device__ __forceinline__ void split_bin(float2 u, float2 um, float2 g, float2& z1, float2& z2) {
  z1 = cmul_tw<false>(make_float2(u.x + um.x, u.y - um.y), g);
  z2 = cmul_tw<false>(make_float2(u.y + um.y, um.x - u.x), g);
}

// Angle of (x, y) in [-pi, pi], the phase step of K1a: octant reduction to
// t = min(|x|, |y|) / max(|x|, |y|) in [0, 1], then atan(t) = t + t^3 Q(t^2)
// with Q a degree-7 polynomial fitted for this kernel (least squares
// reweighted to minimax on [0, 1]; within 1.7 ulp of atan in FP32), and the
// octant restored.  About half the instructions of a library atan2 and within
// a few FP32 ulp of the angle: a few hundredths of a hertz of demodulated
// frequency, below the FP32 rounding of the stage.  Two angles at a time, the
// polynomial packed and everything branch-free, so that the work of several
// samples interleaves.
__device__ __forceinline__ float angle_ratio(float2 c) {
  const float ax = fabsf(c.x), ay = fabsf(c.y);
  float inv;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(fmaxf(ax, ay)));
  // 0/0 gives NaN, which fmaxf turns into the angle 0; no other divisor is
  // subnormal (the rotation scales the step up)
  return fmaxf(fminf(ax, ay) * inv, 0.0f);
}
__device__ __forceinline__ float angle_octant(float r, float2 c) {
  if (fabsf(c.y) > fabsf(c.x)) r = 1.57079632679489662f - r;
  if (c.x < 0.0f) r = 3.14159265358979324f - r;
  return copysignf(r, c.y);
}
// Angles of the complex values a and b.
__device__ __forceinline__ float2 phase_angle2(float2 a, float2 b) {
  const F2 t = f2(angle_ratio(a), angle_ratio(b));
  const F2 s = t * t;
  F2 q = f2(0.00262222f, 0.00262222f);
  q = f2_fma(q, s, f2(-0.01513242f, -0.01513242f));
  q = f2_fma(q, s, f2(0.04112168f, 0.04112168f));
  q = f2_fma(q, s, f2(-0.07366692f, -0.07366692f));
  q = f2_fma(q, s, f2(0.10573926f, 0.10573926f));
  q = f2_fma(q, s, f2(-0.14185974f, -0.14185974f));
  q = f2_fma(q, s, f2(0.19990396f, 0.19990396f));
  q = f2_fma(q, s, f2(-0.33332986f, -0.33332986f));
  const float2 r = parts(f2_fma(t * s, q, t));
  return make_float2(angle_octant(r.x, a), angle_octant(r.y, b));
}

// Predicated accesses: two words to global memory, a complex value from shared
// memory.  (Written as an if, each became a branch of its own.)
__device__ __forceinline__ void st_global_if(bool on, float* p, float x, float* q, float y) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p st.global.f32 [%1], %2;\n\t@p st.global.f32 [%3], %4;\n\t}" ::"r"(
          (int)on),
      "l"(p), "f"(x), "l"(q), "f"(y)
      : "memory");
}
__device__ __forceinline__ void ld_shared_if(int on, float2& v, uint32_t addr) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p ld.shared.v2.f32 {%0, %1}, [%3];\n\t}"
               : "+f"(v.x), "+f"(v.y)
               : "r"(on), "r"(addr)
               : "memory");
}

// K1a output stage for one block: phase step (FP32 Hz, relative to ire0) and
// envelope of outputs [j0, j0 + nout) of tile f, and the block's envelope sum.
// z (thread t, slot q) is block sample t + T*q; its predecessor is held by
// thread t-1 (same q), or for t = 0 by thread T-1 at q-1.
//
// Half of the kernel's instructions are here (64 an output with one sample at
// a time behind a range test).  Slots are taken two at a time in packed
// arithmetic, every slot computed and only the stores tested, so that the
// compiler interleaves them; the outermost slots, mostly or wholly outside
// the outputs, are paired with each other and skipped where both lie outside.
template <int T>
__device__ __forceinline__ void k1a_emit(const DemodArgs& a, const float2 (&z)[16], int f, int j0, int block,
                                         float2 (*warp_last)[18], double* red, int t) {
  const int lane = t & 31, warp = t >> 5;
  constexpr int W = T / 32;
  // row w of warp_last: the predecessors of warp w's first lane, slot q
  if (lane == 31) {
    float2* row = warp < W - 1 ? warp_last[warp + 1] : warp_last[0] + 1;
#pragma unroll
    for (int q = 0; q < 16; q++) row[q] = z[q];
  }
  __syncthreads();
  const int nout = min(a.a_out, kOverlap + a.spp - j0);
  const int i0 = t - (a.a_pos + 1);  // output index of slot 0
  float* dem_out = a.dem + (f * a.spp + (j0 - kOverlap)) + i0;
  float* env_out = a.env + (f * a.spp + (j0 - kOverlap)) + i0;
  const F2 rot = f2(a.rot_re, a.rot_im), rot_q = f2(-a.rot_im, a.rot_re);
  float e[16];
  const int first = lane == 0;
  const uint32_t prev = (uint32_t)__cvta_generic_to_shared(warp_last[warp]);
  // the step of slot q: z * conj(zp) rotated by the nominal step, so the angle is small (and scaled up)
  auto step = [&](int q) {
    float2 zp;
    zp.x = __shfl_up_sync(0xffffffffu, z[q].x, 1);
    zp.y = __shfl_up_sync(0xffffffffu, z[q].y, 1);
    ld_shared_if(first, zp, prev + 8 * q);
    const float2 zz = z[q];
    const float2 c = parts(f2_fma(f2(zz), f2(zp.x, zp.x), f2(zz.y, zz.x) * f2(zp.y, -zp.y)));
    return parts(f2_fma(f2(c.x, c.x), rot, f2(c.y, c.y) * rot_q));
  };
  auto power = [](float2 v) { return fmaf(v.x, v.x, v.y * v.y); };
  auto emit = [&](int qa, int qb) {
    float2 r = phase_angle2(step(qa), step(qb));
    // keep the un-rotated step in (-pi, pi] as the reference's wrap does
    if (r.x > a.wrap) r.x -= 6.28318530717959f;
    if (r.y > a.wrap) r.y -= 6.28318530717959f;
    const float2 hz = parts(f2_fma(f2(r), f2(a.demod_scale, a.demod_scale), f2(a.demod_offset, a.demod_offset)));
    // (CUDA's square root, correctly rounded for every power: 2 us more than an
    // estimate with one correction, which is not)
    const float2 m = make_float2(sqrtf(power(z[qa])), sqrtf(power(z[qb])));
    e[qa] = m.x;
    e[qb] = m.y;
    st_global_if((unsigned)(i0 + T * qa) < (unsigned)nout, dem_out + T * qa, hz.x, env_out + T * qa, m.x);
    st_global_if((unsigned)(i0 + T * qb) < (unsigned)nout, dem_out + T * qb, hz.y, env_out + T * qb, m.y);
  };
  const int lead = a.a_pos + 1;
#pragma unroll
  for (int p = 0; p < 2; p++) {
    e[p] = e[15 - p] = 0.0f;
    if (T * p + T - 1 >= lead || T * (15 - p) - lead < nout) emit(p, 15 - p);
  }
#pragma unroll
  for (int q = 2; q < 14; q += 2) emit(q, q + 1);
  // Deterministic per-block envelope partial sums (the dropout stage needs
  // the tile mean).
  double esum = 0.0;
#pragma unroll
  for (int q = 0; q < 16; q++)
    if ((unsigned)(i0 + T * q) < (unsigned)nout) esum += (double)e[q];
  for (int off = 16; off > 0; off >>= 1) esum += __shfl_down_sync(0xffffffffu, esum, off);
  if (lane == 0) red[warp] = esum;
  __syncthreads();
  if (t == 0) {
    double sacc = 0.0;
    for (int w = 0; w < W; w++) sacc += red[w];
    a.env_part[(size_t)f * a.env_blocks + block] = sacc;
  }
}

// K1a: u8 -> analytic signal -> phase step + envelope, blocks 2x and 2x+1 of
// the tile (the second may lie past the tile's end).
//
// Bound by an SM's units side by side, none of them full: FP32 pipe 49%,
// load/store 42%, issue 62% of cycles; DRAM 11%.  64 registers (16 bytes a
// thread spilled) and 51 KB of shared memory put four CTAs on an SM, in
// different parts of their transforms (three at 80 registers: 3% slower).  The
// second block's half spectrum waits in shared memory, and U is exchanged in
// the transform's own buffer.  40 fields at 28 MHz under ncu: 172 -> 134 us, 168
// MB of interface traffic at 978 -> 1,253 GB/s.  (Two pairs of blocks in the
// two lanes of packed arithmetic, four blocks a CTA at 128 registers and two
// CTAs an SM: 187 us.)
template <int FMT, class Src>
__global__ void __launch_bounds__(kThreadsA, 4) k1a_kernel(const __grid_constant__ Src src, int f_begin) {
  constexpr int N = Design::kNa, T = kThreadsA;
  const DemodArgs& a = src.get();
  if (f_begin + (int)blockIdx.y >= a.tiles) return;  // whole CTA: a batched capture with fewer tiles
  chain_wait();
  extern __shared__ float2 sm[];
  float2* z2 = sm + fft_pad(N);  // the second block's spectrum, each slot its own thread's
  __shared__ float2 warp_last[T / 32][18];
  __shared__ double red[T / 32];
  const int t = threadIdx.x;
  const int f = f_begin + blockIdx.y;
  const int blk0 = 2 * blockIdx.x;
  const int j0 = kOverlap + blk0 * a.a_out;  // first demod output of block 0 (tile position)
  // chunk positions fit in 32 bits (the batch is capped so T * spp < 2^31)
  const int tile0 = f * a.spp - kOverlap;    // chunk position of tile position 0
  const int last = (int)a.total - 1;
  const int base = j0 - 1 - a.a_pos;         // tile position of block-0 sample 0
  float2 v[16];
  // Interior windows (no wrap inside the tile, no clamp at the chunk ends)
  // take the direct addresses; the CTA-uniform test keeps the loop branch-free.
  const int span = a.a_out + N;  // tile positions [base, base + span) are read
  const float dc = a.dc ? *a.dc : 0.0f;
  if (base >= 0 && base + span <= a.tile && tile0 + base >= 0 && tile0 + base + span - 1 <= last &&
      tile0 + base + span <= a.n_read) {
    // one address a block, constant offsets from it
    const uint8_t* p0 = raw_at<FMT>(a.raw, tile0 + base + t);
    const uint8_t* p1 = raw_at<FMT>(p0, a.a_out);
#pragma unroll
    for (int q = 0; q < 16; q++)
      v[q] = make_float2(raw_convert<FMT>(p0, T * q) - dc, raw_convert<FMT>(p1, T * q) - dc);
  } else {
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const int q0 = base + t + T * q;
      const int p0 = min(max(tile0 + wrap_tile(q0, a.tile), 0), last);
      const int p1 = min(max(tile0 + wrap_tile(q0 + a.a_out, a.tile), 0), last);
      v[q] = make_float2(raw_sample<FMT>(a.raw, p0, a.n_read, dc), raw_sample<FMT>(a.raw, p1, a.n_read, dc));
    }
  }
  RegFFT<N>::run<false>(v, sm, a.tw_a, t);
  __syncthreads();  // the last pass's reads
#pragma unroll
  for (int q = 0; q < 16; q++) sm[pidx(t + T * q)] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int k = t + T * q;
    split_bin(v[q], sm[pidx((N - k) & (N - 1))], __ldg(&a.ga[k]), v[q], z2[k]);
  }
  // one copy of the inverse transform and output stage serves both blocks
  // (a rolled loop keeps the kernel body small for the instruction cache)
#pragma unroll 1
  for (int b = 0; b < 2; b++) {
    if (b == 1) {
      if (blk0 + 1 >= a.env_blocks) return;  // whole CTA
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = z2[t + T * q];
    }
    RegFFT<N>::run_half<true>(v, sm, a.tw_a_inv, t);
    k1a_emit<T>(a, v, f, j0 + b * a.a_out, blk0 + b, warp_last, red, t);
  }
}

// K1b output stage: video (real part) and sync (imaginary part) of one block.
// Sync samples within guard_hz of the pulse threshold are listed for the FP64
// re-evaluation (kernels_guard.cu); a handful per field, so the slot loop only
// notes that there is one.
template <int T>
__device__ __forceinline__ void k1b_emit(const DemodArgs& a, const float2 (&z)[16], int f, int j0, int t) {
  const int nout = min(a.b_out, kOverlap + a.spp - j0);
  const int i0 = t - a.b_pos;                        // output index of slot 0
  const int out0 = f * a.spp + (j0 - kOverlap) + i0;  // its chunk position
  float* video_out = a.video + out0;
  float* sync_out = a.sync + out0;
  const int lane = t & 31;
  // slot q's 32 consecutive positions (one per lane) as an in-pulse word:
  // lane q keeps slot q's ballot, and after the loop lanes 0..15 OR their
  // words into the (at most two) bit words each straddles, in parallel
  unsigned mine = 0;
  bool near = false;
  const F2 corr = f2(a.corr_video, a.corr_sync);
#pragma unroll
  for (int q = 0; q < 16; q++) {
    const float2 o = parts(f2(z[q]) + corr);
    const bool valid = (unsigned)(i0 + T * q) < (unsigned)nout;
    if (valid) {
      video_out[T * q] = o.x;
      sync_out[T * q] = o.y;
    }
    near = near || (valid && fabsf(o.y - a.thr_rel) < a.guard_hz);
    const unsigned m = __ballot_sync(0xffffffffu, valid && o.y <= a.thr_rel);
    mine = lane == q ? m : mine;
  }
  if (__any_sync(0xffffffffu, near) && a.guard_list) {
#pragma unroll 1
    for (int q = 0; q < 16; q++) {
      if ((unsigned)(i0 + T * q) < (unsigned)nout && fabsf(sync_out[T * q] - a.thr_rel) < a.guard_hz) {
        const int slot = atomicAdd(a.guard_count, 1);
        if (slot < a.guard_cap) a.guard_list[slot] = (unsigned)(out0 + T * q);
      }
    }
  }
  if (a.pulse_bits && mine) {  // only lanes 0..15 hold a word
    long long p0 = (long long)(out0 - lane) + (long long)T * lane;
    if (p0 < 0) {  // positions before the chunk start hold no bits
      mine >>= (int)(-p0);
      p0 = 0;
    }
    const long long w = p0 >> 5;
    const int sh = (int)(p0 & 31);
    atomicOr(&a.pulse_bits[w], mine << sh);
    if (sh && (mine >> (32 - sh))) atomicOr(&a.pulse_bits[w + 1], mine >> (32 - sh));
  }
}

// K1b: demod -> video + sync, blocks 2x and 2x+1 of the tile.
//
// One 8192-point exchange buffer (70 KB) and 64 registers a thread put two
// CTAs on an SM, one's arithmetic beside the other's exchanges: the second
// block's spectrum (64 KB, which shared memory does not hold twice more) waits
// in tensor memory, each thread's 32 words in columns of its own.  Both
// inverses in lockstep at 128 registers and one CTA an SM left every unit
// below 38% (issue 44%); now FP32 pipe 40%, load/store 36%, issue 51%, DRAM 15%
// (36 bytes a thread spilled).  40 fields at 28 MHz under ncu: 179 -> 149 us,
// 227 MB of interface traffic at 1,263 -> 1,517 GB/s.
template <class Src>
__global__ void __launch_bounds__(kThreadsB, 2) k1b_kernel(const __grid_constant__ Src src, int f_begin) {
  constexpr int N = Design::kNb, T = kThreadsB;
  const DemodArgs& a = src.get();
  if (f_begin + (int)blockIdx.y >= a.tiles) return;  // whole CTA
  extern __shared__ float2 sm[];
  __shared__ uint32_t tmem_base;
  const int t = threadIdx.x, warp = t >> 5;
  tmem_alloc<kTmemColsB>(&tmem_base, warp);
  chain_wait();
  const int f = f_begin + blockIdx.y;
  const int blk0 = 2 * blockIdx.x;
  const int j0 = kOverlap + blk0 * a.b_out;
  const int tile0 = f * a.spp - kOverlap;
  const int last = (int)a.total - 1;
  const int base = j0 - a.b_pos;
  float2 v[16];
  const int span = a.b_out + N;  // tile positions [base, base + span) are read
  if (base >= 0 && base + span <= a.tile && tile0 + base >= 0 && tile0 + base + span - 1 <= last) {
    // interior: no wrap inside the tile, no clamp at the chunk ends
    const float* p0 = a.dem + (tile0 + base + t);
    const float* p1 = p0 + a.b_out;
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = make_float2(__ldg(p0 + T * q), __ldg(p1 + T * q));
  } else {
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const int q0 = base + t + T * q;
      const int p0 = min(max(tile0 + wrap_tile(q0, a.tile), 0), last);
      const int p1 = min(max(tile0 + wrap_tile(q0 + a.b_out, a.tile), 0), last);
      v[q] = make_float2(__ldg(&a.dem[p0]), __ldg(&a.dem[p1]));
    }
  }
  RegFFT<N>::run<false>(v, sm, a.tw_b, t);
  __syncthreads();  // the last pass's reads
#pragma unroll
  for (int q = 0; q < 16; q++) sm[pidx(t + T * q)] = v[q];
  __syncthreads();
  // the second block's spectrum waits in tensor memory
  const uint32_t own = tmem_own(tmem_base, warp, 32);
#pragma unroll
  for (int c = 0; c < 4; c++) {
    float2 z2[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int q = 4 * c + i, k = t + T * q;
      split_bin(v[q], sm[pidx((N - k) & (N - 1))], __ldg(&a.gb[k]), v[q], z2[i]);
    }
    tmem_st8(own + 8 * c, z2);
  }
  tmem_wait_st();
  // one copy of the inverse transform and output stage serves both blocks
  const int nblk = kOverlap + (blk0 + 1) * a.b_out >= kOverlap + a.spp ? 1 : 2;  // the second may lie past the tile
#pragma unroll 1
  for (int b = 0; b < nblk; b++) {
    if (b == 1) {
      __syncwarp();
      tmem_ld32(own, v);
    }
    RegFFT<N>::run<true>(v, sm, a.tw_b_inv, opaque_index(t));
    k1b_emit<T>(a, v, f, j0 + b * a.b_out, t);
  }
  __syncthreads();
  tmem_free<kTmemColsB>(tmem_base, warp);
}

// Threshold edges in sample order.  Each thread owns 16 consecutive samples
// (one 64-byte line), a CTA 4096.  The count pass reads the signal once and
// keeps each thread's 16-bit falling / rising masks; one scan turns the
// per-CTA counts into offsets; the write pass reads only the masks and writes
// the positions in order, so the host receives sorted edge lists.
constexpr int kEdgeThreads = 256;
constexpr int kEdgePer = 16;
constexpr int kEdgeSeg = kEdgeThreads * kEdgePer;

__device__ __forceinline__ void edge_masks(const float* __restrict__ x, long long total, float thr, long long i0,
                                           unsigned& fm, unsigned& rm) {
  fm = 0;
  rm = 0;
  if (i0 >= total) return;
  float v[kEdgePer];
  // 16-byte loads where the signal is 16-byte aligned (a batched capture's
  // sync may start at any sample)
  if (i0 + kEdgePer <= total && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    const float4* p = reinterpret_cast<const float4*>(x + i0);
#pragma unroll
    for (int q = 0; q < kEdgePer / 4; q++) {
      const float4 t = __ldg(p + q);
      v[4 * q] = t.x;
      v[4 * q + 1] = t.y;
      v[4 * q + 2] = t.z;
      v[4 * q + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kEdgePer; j++) v[j] = (i0 + j < total) ? __ldg(&x[i0 + j]) : 0.0f;
  }
  bool prev_in = i0 > 0 ? (__ldg(&x[i0 - 1]) <= thr) : false;
#pragma unroll
  for (int j = 0; j < kEdgePer; j++) {
    if (i0 + j >= total) break;
    const bool in = v[j] <= thr;
    if (in && (i0 + j == 0 || !prev_in)) fm |= 1u << j;
    if (!in && i0 + j > 0 && prev_in) rm |= 1u << j;
    prev_in = in;
  }
}

// Block-wide exclusive scan of two counters; returns the block totals.
__device__ __forceinline__ int2 block_scan2(int a, int b, int& pa, int& pb) {
  __shared__ int2 warp_tot[kEdgeThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int sa = a, sb = b;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int ta = __shfl_up_sync(0xffffffffu, sa, off), tb = __shfl_up_sync(0xffffffffu, sb, off);
    if (lane >= off) {
      sa += ta;
      sb += tb;
    }
  }
  if (lane == 31) warp_tot[warp] = make_int2(sa, sb);
  __syncthreads();
  int ba = 0, bb = 0, ta = 0, tb = 0;
  for (int w = 0; w < kEdgeThreads / 32; w++) {
    if (w < warp) {
      ba += warp_tot[w].x;
      bb += warp_tot[w].y;
    }
    ta += warp_tot[w].x;
    tb += warp_tot[w].y;
  }
  pa = ba + sa - a;
  pb = bb + sb - b;
  return make_int2(ta, tb);
}

__global__ void __launch_bounds__(kEdgeThreads) edge_count_kernel(const float* __restrict__ x, long long total,
                                                                  float thr, int2* __restrict__ blk,
                                                                  unsigned* __restrict__ masks) {
  chain_wait();
  const long long i0 = (long long)blockIdx.x * kEdgeSeg + (long long)threadIdx.x * kEdgePer;
  unsigned fm, rm;
  edge_masks(x, total, thr, i0, fm, rm);
  masks[(size_t)blockIdx.x * kEdgeThreads + threadIdx.x] = fm | (rm << 16);
  int pa, pb;
  const int2 t = block_scan2(__popc(fm), __popc(rm), pa, pb);
  if (threadIdx.x == 0) blk[blockIdx.x] = t;
}

// One CTA: exclusive scan of the per-CTA counts in place, totals to
// counts[0..1].  Thread t sums a contiguous run of ceil(nblk / 1024) counts,
// the runs' totals are scanned with warp shuffles, then each thread writes its
// run's offsets.
constexpr int kScanThreads = 1024;
__device__ __forceinline__ void scan_blocks(int2* __restrict__ blk, int nblk, int* __restrict__ counts) {
  __shared__ int2 warp_tot[kScanThreads / 32];
  chain_wait();
  const int per = (nblk + kScanThreads - 1) / kScanThreads;
  const int b0 = min(nblk, (int)threadIdx.x * per), b1 = min(nblk, b0 + per);
  int sa = 0, sb = 0;
  for (int b = b0; b < b1; b++) {
    const int2 v = blk[b];
    sa += v.x;
    sb += v.y;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int ia = sa, ib = sb;  // inclusive within the warp
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int ta = __shfl_up_sync(0xffffffffu, ia, off), tb = __shfl_up_sync(0xffffffffu, ib, off);
    if (lane >= off) {
      ia += ta;
      ib += tb;
    }
  }
  if (lane == 31) warp_tot[warp] = make_int2(ia, ib);
  __syncthreads();
  if (warp == 0) {
    int wa = warp_tot[lane].x, wb = warp_tot[lane].y;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int ta = __shfl_up_sync(0xffffffffu, wa, off), tb = __shfl_up_sync(0xffffffffu, wb, off);
      if (lane >= off) {
        wa += ta;
        wb += tb;
      }
    }
    warp_tot[lane] = make_int2(wa, wb);  // inclusive over warps
  }
  __syncthreads();
  int ca = ia - sa, cb = ib - sb;  // exclusive start of this thread's run
  if (warp > 0) {
    ca += warp_tot[warp - 1].x;
    cb += warp_tot[warp - 1].y;
  }
  for (int b = b0; b < b1; b++) {
    const int2 v = blk[b];
    blk[b] = make_int2(ca, cb);
    ca += v.x;
    cb += v.y;
  }
  if (threadIdx.x == 0) {
    counts[0] = warp_tot[kScanThreads / 32 - 1].x;
    counts[1] = warp_tot[kScanThreads / 32 - 1].y;
  }
}


__global__ void __launch_bounds__(kScanThreads) edge_scan_kernel(int2* __restrict__ blk, int nblk,
                                                                 int* __restrict__ counts) {
  scan_blocks(blk, nblk, counts);
}

__global__ void __launch_bounds__(kEdgeThreads) edge_write_kernel(long long total, const unsigned* __restrict__ masks,
                                                                  const int2* __restrict__ blk,
                                                                  unsigned* __restrict__ fall,
                                                                  unsigned* __restrict__ rise, int cap) {
  chain_wait();
  const long long i0 = (long long)blockIdx.x * kEdgeSeg + (long long)threadIdx.x * kEdgePer;
  const unsigned m = __ldg(&masks[(size_t)blockIdx.x * kEdgeThreads + threadIdx.x]);
  unsigned fm = m & 0xFFFFu, rm = m >> 16;
  (void)total;
  int pa, pb;
  block_scan2(__popc(fm), __popc(rm), pa, pb);
  int kf = blk[blockIdx.x].x + pa, kr = blk[blockIdx.x].y + pb;
  while (fm) {
    const int j = __ffs(fm) - 1;
    fm &= fm - 1;
    if (kf < cap) fall[kf] = (unsigned)(i0 + j);
    kf++;
  }
  while (rm) {
    const int j = __ffs(rm) - 1;
    rm &= rm - 1;
    if (kr < cap) rise[kr] = (unsigned)(i0 + j);
    kr++;
  }
}

// Threshold edges from in-pulse bits: WPT consecutive 32-position words a
// thread (a CTA 8192 * WPT positions).  falling = in now and not before,
// rising = out now and in before; position 0 counts as preceded by "out" (a
// pulse open there falls there), positions at or past total hold no bits.
//
// A count pass, then a write pass that places each CTA's edges.  Where the
// CTAs are few (kDirectBlocks), each sums the counts before its own (32 KB from
// L2 at most); past that a scan kernel does it once.  Four words a thread
// (kWideEdges) once that still gives every SM two CTAs: a quarter of the CTAs,
// each with a quarter of the counts to sum (one word a thread, 2,460 CTAs for
// 40 fields at 28 MHz: 11 us in the write pass).  Latency bound.
constexpr int kDirectBlocks = 4096;
constexpr long long kWideEdges = 296ll * 4 * 8192;
template <int WPT>
__host__ __device__ constexpr long long bit_edge_seg() { return (long long)kEdgeThreads * WPT * 32; }

template <int WPT>
__device__ __forceinline__ void bit_edges(const unsigned* __restrict__ bits, long long total, long long w0,
                                          unsigned (&fm)[WPT], unsigned (&rm)[WPT]) {
  unsigned prev = w0 > 0 && w0 * 32 < total ? (__ldg(&bits[w0 - 1]) >> 31) : 0u;
#pragma unroll
  for (int q = 0; q < WPT; q++) {
    const long long w = w0 + q, p0 = w * 32;
    fm[q] = rm[q] = 0;
    if (p0 >= total) continue;
    const unsigned valid = total - p0 >= 32 ? 0xffffffffu : ((1u << (unsigned)(total - p0)) - 1u);
    const unsigned word = __ldg(&bits[w]), in = word & valid;
    const unsigned before = (in << 1) | prev;  // bit j: in at position j - 1
    fm[q] = in & ~before;
    rm[q] = ~in & before & valid;
    prev = word >> 31;
  }
}
template <int WPT>
__device__ __forceinline__ int bit_count(const unsigned (&m)[WPT]) {
  int n = 0;
#pragma unroll
  for (int q = 0; q < WPT; q++) n += __popc(m[q]);
  return n;
}

template <int WPT, class Src>
__global__ void __launch_bounds__(kEdgeThreads) edge_bits_count_kernel(const __grid_constant__ Src src) {
  const EdgeArgs& e = src.get();
  if ((long long)blockIdx.x * bit_edge_seg<WPT>() >= e.total) return;  // whole CTA
  chain_wait();
  const long long w = ((long long)blockIdx.x * kEdgeThreads + threadIdx.x) * WPT;
  unsigned fm[WPT], rm[WPT];
  bit_edges<WPT>(e.bits, e.total, w, fm, rm);
  int pa, pb;
  const int2 tot = block_scan2(bit_count(fm), bit_count(rm), pa, pb);
  if (threadIdx.x == 0) e.blk[blockIdx.x] = tot;
}

template <int WPT, class Src>
__global__ void __launch_bounds__(kScanThreads) edge_bits_scan_kernel(const __grid_constant__ Src src) {
  const EdgeArgs& e = src.get();
  scan_blocks(e.blk, (int)((e.total + bit_edge_seg<WPT>() - 1) / bit_edge_seg<WPT>()), e.counts);
}

// DIRECT: blk holds the count pass's counts and this CTA sums those before
// its own (the last CTA writes the totals); else blk holds offsets.
template <int WPT, bool DIRECT, class Src>
__global__ void __launch_bounds__(kEdgeThreads) edge_bits_write_kernel(const __grid_constant__ Src src) {
  const EdgeArgs& e = src.get();
  if ((long long)blockIdx.x * bit_edge_seg<WPT>() >= e.total) return;  // whole CTA
  chain_wait();
  const long long w = ((long long)blockIdx.x * kEdgeThreads + threadIdx.x) * WPT;
  unsigned fm[WPT], rm[WPT];
  bit_edges<WPT>(e.bits, e.total, w, fm, rm);
  int pa, pb;
  const int2 own = block_scan2(bit_count(fm), bit_count(rm), pa, pb);
  int2 at;
  if constexpr (DIRECT) {
    int sa = 0, sb = 0;
#pragma unroll 4
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += kEdgeThreads) {
      const int2 c = __ldcg(&e.blk[b]);
      sa += c.x;
      sb += c.y;
    }
    int ia, ib;
    __syncthreads();  // the first scan's totals
    at = block_scan2(sa, sb, ia, ib);
    if (threadIdx.x == 0 && (long long)(blockIdx.x + 1) * bit_edge_seg<WPT>() >= e.total) {
      e.counts[0] = at.x + own.x;
      e.counts[1] = at.y + own.y;
    }
  } else {
    at = e.blk[blockIdx.x];
  }
  int kf = at.x + pa, kr = at.y + pb;
#pragma unroll
  for (int q = 0; q < WPT; q++) {
    const long long p0 = (w + q) * 32;
    for (unsigned m = fm[q]; m; m &= m - 1) {
      if (kf < e.cap) e.fall[kf] = (unsigned)(p0 + __ffs(m) - 1);
      kf++;
    }
    for (unsigned m = rm[q]; m; m &= m - 1) {
      if (kr < e.cap) e.rise[kr] = (unsigned)(p0 + __ffs(m) - 1);
      kr++;
    }
  }
}

// The passes over `portions` captures of at most max_total positions.
template <int WPT, class S>
void edges_bits_launch(const S& e, int portions, long long max_total, cudaStream_t st) {
  const int nblk = (int)((max_total + bit_edge_seg<WPT>() - 1) / bit_edge_seg<WPT>());
  const dim3 grid(nblk, 1, portions);
  launch_chained(edge_bits_count_kernel<WPT, S>, grid, dim3(kEdgeThreads), 0, st, e);
  if constexpr (WPT > 1) {  // one word a thread: always few CTAs
    if (nblk > kDirectBlocks) {
      launch_chained(edge_bits_scan_kernel<WPT, S>, dim3(1, 1, portions), dim3(kScanThreads), 0, st, e);
      launch_chained(edge_bits_write_kernel<WPT, false, S>, grid, dim3(kEdgeThreads), 0, st, e);
      return;
    }
  }
  launch_chained(edge_bits_write_kernel<WPT, true, S>, grid, dim3(kEdgeThreads), 0, st, e);
}
template <class S>
int edges_bits_any(const S& e, int portions, long long max_total, cudaStream_t st) {
  static_assert(kWideEdges <= kDirectBlocks * bit_edge_seg<1>(), "narrow passes sum directly");
  if (max_total <= 0 || portions <= 0) return 0;
  if (max_total < kWideEdges) edges_bits_launch<1>(e, portions, max_total, st);
  else edges_bits_launch<4>(e, portions, max_total, st);
  return max_total <= kDirectBlocks * bit_edge_seg<4>() ? 2 : 3;
}

}  // namespace

size_t pulse_bit_words(long long total) { return (size_t)((total + 31) / 32) + 1; }

int launch_edges_bits(const unsigned* bits, long long total, unsigned* fall, unsigned* rise, int* counts, int cap,
                      int2* blk, cudaStream_t st) {
  ArgsOne<EdgeArgs> e;
  e.a[0].bits = bits;
  e.a[0].total = total;
  e.a[0].blk = blk;
  e.a[0].counts = counts;
  e.a[0].fall = fall;
  e.a[0].rise = rise;
  e.a[0].cap = cap;
  return edges_bits_any(e, 1, total, st);
}

int launch_edges_bits_many(const ArgsMany<EdgeArgs>& e, int portions, long long max_total, cudaStream_t st) {
  return edges_bits_any(e, portions, max_total, st);
}

void launch_k1a(const DemodArgs& a, int f0, int nf, cudaStream_t st) {
  if (nf <= 0) return;
  const size_t smem = kSmemA;
  const int blocks = (a.spp + a.a_out - 1) / a.a_out;  // = env_blocks
  dim3 grid((blocks + 1) / 2, nf);
  const ArgsOne<DemodArgs> src{a};
  auto go = [&](auto kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained(kernel, grid, dim3(kThreadsA), smem, st, src, f0);
  };
  using S = ArgsOne<DemodArgs>;
  if (a.in_fmt == kInS16) go(k1a_kernel<kInS16, S>);
  else if (a.in_fmt == kInU16) go(k1a_kernel<kInU16, S>);
  else go(k1a_kernel<kInU8, S>);
}

void launch_k1a_many(const ArgsMany<DemodArgs>& p, int portions, int max_tiles, cudaStream_t st) {
  if (portions <= 0 || max_tiles <= 0) return;
  const DemodArgs& a = p.a[0];  // the design constants every capture of a round shares
  const size_t smem = kSmemA;
  const int blocks = (a.spp + a.a_out - 1) / a.a_out;
  dim3 grid((blocks + 1) / 2, max_tiles, portions);
  auto go = [&](auto kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained(kernel, grid, dim3(kThreadsA), smem, st, p, 0);
  };
  using S = ArgsMany<DemodArgs>;
  if (a.in_fmt == kInS16) go(k1a_kernel<kInS16, S>);
  else if (a.in_fmt == kInU16) go(k1a_kernel<kInU16, S>);
  else go(k1a_kernel<kInU8, S>);
}

namespace {

// Sum of the converted samples as a 64-bit integer (every converted value is
// an integer, so the sum is exact and order-free).  Memory bounds it: 16 bytes
// a load, four loads of a thread in flight; the samples before the first
// 16-byte boundary and after the last go one at a time (2-byte loads
// throughout: 28 us for 24 tiles of 16-bit samples at 35.8 MHz, now 7.8).
template <int FMT>
__device__ __forceinline__ long long sum16(uint4 q) {
  const unsigned w[4] = {q.x, q.y, q.z, q.w};
  int acc = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if constexpr (FMT == kInU8) acc = (int)__dp4a(w[k], 0x01010101u, (unsigned)acc);
    else if constexpr (FMT == kInS16) acc += (int)(short)(w[k] & 0xffffu) + ((int)w[k] >> 16);
    else acc += (int)(w[k] & 0xffffu) + (int)(w[k] >> 16);
  }
  if constexpr (FMT == kInU8) return (long long)(acc - 16 * 128) * 256;
  if constexpr (FMT == kInS16) return acc;
  return acc - 8 * 32768;
}

template <int FMT>
__global__ void dc_sum_kernel(const uint8_t* raw, int n, unsigned long long* sum) {
  __shared__ long long part[8];
  constexpr int kPer = FMT == kInU8 ? 16 : 8;  // samples a load
  constexpr int kFlight = 4;
  const int t = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  // samples before the first 16-byte boundary (16-bit samples are 2-byte aligned)
  const int head = min(n, (int)(((16 - (reinterpret_cast<uintptr_t>(raw) & 15)) & 15) / (16 / kPer)));
  const int quads = (n - head) / kPer;
  const uint4* const body = reinterpret_cast<const uint4*>(raw_at<FMT>(raw, head));
  long long acc = 0;
  if (t < head) acc += (long long)raw_convert<FMT>(raw, t);
  const int tail = head + quads * kPer + t;
  if (tail < n) acc += (long long)raw_convert<FMT>(raw, tail);
  for (int i = t; i < quads; i += kFlight * stride) {
    uint4 q[kFlight];
#pragma unroll
    for (int k = 0; k < kFlight; k++)
      if (i + k * stride < quads) q[k] = __ldg(body + i + k * stride);
#pragma unroll
    for (int k = 0; k < kFlight; k++)
      if (i + k * stride < quads) acc += sum16<FMT>(q[k]);
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long s = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += part[w];
    atomicAdd(sum, (unsigned long long)s);
  }
}

__global__ void dc_mean_kernel(const unsigned long long* sum, int n, float* dc) {
  *dc = (float)((double)(long long)*sum / (double)n);
}

}  // namespace

void launch_dc_mean(const uint8_t* raw, int n, int in_fmt, unsigned long long* sum, float* dc, cudaStream_t st) {
  cudaMemsetAsync(sum, 0, sizeof(unsigned long long), st);
  const int threads = 256, blocks = 148 * 8;
  if (n > 0) {
    if (in_fmt == kInS16) dc_sum_kernel<kInS16><<<blocks, threads, 0, st>>>(raw, n, sum);
    else if (in_fmt == kInU16) dc_sum_kernel<kInU16><<<blocks, threads, 0, st>>>(raw, n, sum);
    else dc_sum_kernel<kInU8><<<blocks, threads, 0, st>>>(raw, n, sum);
  }
  dc_mean_kernel<<<1, 1, 0, st>>>(sum, n > 0 ? n : 1, dc);
}

void launch_k1b(const DemodArgs& a, int f0, int nf, cudaStream_t st) {
  if (nf <= 0) return;
  const size_t smem = kSmemB;
  using S = ArgsOne<DemodArgs>;
  cudaFuncSetAttribute(k1b_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int blocks = (a.spp + a.b_out - 1) / a.b_out;
  dim3 grid((blocks + 1) / 2, nf);
  const S src{a};
  launch_chained(k1b_kernel<S>, grid, dim3(kThreadsB), smem, st, src, f0);
}

void launch_k1b_many(const ArgsMany<DemodArgs>& p, int portions, int max_tiles, cudaStream_t st) {
  if (portions <= 0 || max_tiles <= 0) return;
  const DemodArgs& a = p.a[0];
  const size_t smem = kSmemB;
  using S = ArgsMany<DemodArgs>;
  cudaFuncSetAttribute(k1b_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int blocks = (a.spp + a.b_out - 1) / a.b_out;
  dim3 grid((blocks + 1) / 2, max_tiles, portions);
  launch_chained(k1b_kernel<S>, grid, dim3(kThreadsB), smem, st, p, 0);
}

int edge_blocks(long long total) { return (int)((total + kEdgeSeg - 1) / kEdgeSeg); }

size_t edge_mask_words(long long total) { return (size_t)edge_blocks(total) * kEdgeThreads; }

void launch_edges(const float* sync, long long total, float thr_rel, unsigned* fall, unsigned* rise, int* counts,
                  int cap, int2* blk, unsigned* masks, cudaStream_t st) {
  const int nblk = edge_blocks(total);
  if (nblk <= 0) return;
  launch_chained(edge_count_kernel, dim3(nblk), dim3(kEdgeThreads), 0, st, sync, total, thr_rel, blk, masks);
  launch_chained(edge_scan_kernel, dim3(1), dim3(kScanThreads), 0, st, blk, nblk, counts);
  launch_chained(edge_write_kernel, dim3(nblk), dim3(kEdgeThreads), 0, st, total, (const unsigned*)masks,
                 (const int2*)blk, fall, rise, cap);
}

}  // namespace cuvhs
