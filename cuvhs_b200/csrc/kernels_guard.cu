// Guard band of the sync threshold decisions.
//
// The reference decides in FP64 whether a sync sample lies at or below the
// pulse threshold (src/pipeline/sync_pulses.cu:35-55; the VSYNC widths of
// src/pipeline/vsync_discover.cu:5-45 and the threshold crossings of
// src/pipeline/hsync_refine.cu:21-65 make the same decision).  This decoder
// computes sync in FP32, within a few Hz of FP64.  K1b lists every sync sample
// it writes within kGuardHz of the threshold; guard_kernel re-evaluates each
// listed sample in FP64 straight from the raw capture and writes it back on the
// side of the FP32 threshold its FP64 value lies on, so every later threshold
// decision (edges, VSYNC widths, pulses, hsync crossings) is the FP64 one.
//
// The FP64 value follows the reference's tile arithmetic exactly, with the
// circular kernels truncated only where their taps fall below 1e-13 of the
// peak (Design::ga64 / hs64):
//   sync[s]  = sum_k hs[k] * dem[c(J - k)],   J = 2048 + s - f*spp, s in tile f,
//   dem[c]   = wrap(arg z(J') - arg z(J' - 1)) * fs / 2pi   (c in tile f', J' = 2048 + c - f'*spp),
//   z(j)     = sum_m g[m] * x_f'(j - m),
// where tile positions wrap mod the tile length and chunk positions clamp to
// the demodulated range (src/pipeline/fm_demod.cu:133-169, 396-485).
//
// Work: one CTA per listed sample.  The 2*hb + 1 demod positions the sample's
// sync sum reads split into a few runs -- consecutive chunk positions of one
// owning tile, or one clamped position repeated -- and each run's analytic
// signal is one FP64 overlap-save convolution: its raw window (tile wrap and
// chunk clamp applied per sample) goes through a 4096-point FP64 FFT (registers and shared
// memory), is multiplied by the FFT of the truncated taps and transformed back,
// giving every z of up to 4095 - 2*ha consecutive positions at once.  The
// phase differences fill a demod array indexed like the sync taps, and the
// sync sum is taken in a fixed order, so the result is deterministic.
#include <cuda_runtime.h>

#include <algorithm>

#include "chain.cuh"
#include "cuvhs_internal.h"
#include "raw_input.cuh"

namespace cuvhs {
namespace {

constexpr int kGT = 256;                  // threads per CTA: 16 points each (two CTAs per SM)
constexpr int kN = Design::kGuardN;       // FFT length
constexpr int kRow = 16 * 17 + 1;         // padded slots of 256 points: one after every 16 and every 256
constexpr int kSlots = 16 * kRow;         // the padded transform
constexpr int kTwQ = kN / 4;              // twiddles held in shared memory: exp(-2 pi i k / kN), k < kN / 4
constexpr int kTwPad = kTwQ + kTwQ / 8;   // one slot after every 8
constexpr double kPi64 = 3.14159265358979323846;
constexpr double kTau64 = 2.0 * kPi64;
static_assert(kN == 4096 && kGT == 256, "three passes of 16 points on 256 threads");

__device__ __forceinline__ int wrap_pos(int q, int tile) {
  return q < 0 ? q + tile : (q >= tile ? q - tile : q);
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a * (-i), conjugated for the inverse
template <bool kInverse>
__device__ __forceinline__ double2 turn(double2 a) {
  return kInverse ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// exp(-2 pi i j / kN) for j < kN from the quarter table: the quadrant
// q = j / (kN / 4) multiplies by (-i)^q.  The inverse conjugates.
template <bool kInverse>
__device__ __forceinline__ double2 twiddle(const double2* tq, int j) {
  const int m = j & (kTwQ - 1), q = j / kTwQ;
  const double2 w = tq[m + (m >> 3)];
  double2 r = (q & 1) ? make_double2(w.y, -w.x) : w;
  if (q & 2) r = make_double2(-r.x, -r.y);
  return kInverse ? make_double2(r.x, -r.y) : r;
}

// Four-point DFT of v[0], v[S], v[2S], v[3S] in place.
template <bool kInverse, int S>
__device__ __forceinline__ void dft4(double2* v) {
  const double2 s02 = cadd(v[0], v[2 * S]), d02 = csub(v[0], v[2 * S]);
  const double2 s13 = cadd(v[S], v[3 * S]), m = turn<kInverse>(csub(v[S], v[3 * S]));
  v[0] = cadd(s02, s13);
  v[S] = cadd(d02, m);
  v[2 * S] = csub(s02, s13);
  v[3 * S] = csub(d02, m);
}

// Sixteen-point DFT; output k is left in v[4 * (k & 3) + (k >> 2)] (slot16).
__device__ __forceinline__ constexpr int slot16(int k) { return 4 * (k & 3) + (k >> 2); }

template <bool kInverse>
__device__ __forceinline__ void dft16(double2 (&v)[16]) {
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;  // cos, sin of pi / 8
  constexpr double h = 0.70710678118654752440;
  constexpr double sg = kInverse ? 1.0 : -1.0;
#pragma unroll
  for (int c = 0; c < 4; c++) dft4<kInverse, 4>(v + c);  // v[4 r + c] -> r
  auto w8 = [](double2 a) {  // times exp(-+ i pi / 4)
    const double2 t = turn<kInverse>(a);
    return make_double2((a.x + t.x) * h, (a.y + t.y) * h);
  };
  v[5] = cmul(v[5], make_double2(c1, sg * s1));
  v[6] = w8(v[6]);
  v[7] = cmul(v[7], make_double2(s1, sg * c1));
  v[9] = w8(v[9]);
  v[10] = turn<kInverse>(v[10]);
  v[11] = turn<kInverse>(w8(v[11]));
  v[13] = cmul(v[13], make_double2(s1, sg * c1));
  v[14] = turn<kInverse>(w8(v[14]));
  v[15] = cmul(v[15], make_double2(-c1, -sg * s1));
#pragma unroll
  for (int r = 0; r < 4; r++) dft4<kInverse, 1>(v + 4 * r);
}

// The block's convolution: v[i] holds the real input at position t + 256 i;
// on return buf[t + 256 i] (padded: slot_of) holds the analytic signal there.
//
// FP64 multiply-adds and shared memory traffic bound a transform: three passes
// of 16 points in registers touch shared memory twice per transform (six
// radix-4 passes through it, on 512 threads, took the whole kernel from 36.2
// us to 26.4 for a 3-tile chunk, from 60.1 to 37.6 for 24 tiles at 35.8 MHz).
// A pass reads and writes its own slots, so one barrier per pass suffices; the
// spectrum leaves the third pass in the order the inverse's first pass takes,
// so the filter is applied in registers.  The padding keeps a warp's slots of
// every pass and of the first pass's twiddles (strides 0..15) on distinct banks
// (quarter warps of 16-byte accesses).
__device__ __forceinline__ int slot_of(int n) { return n + (n >> 4) + (n >> 8); }

__device__ __forceinline__ void convolve(double2 (&v)[16], double2* buf, const double2* tq, const double2* tw2,
                                         const double2* __restrict__ gfft) {
  const int t = threadIdx.x, lo = t & 15, hi = t >> 4;
  double2* const col = buf + t + hi;              // pass 1: position t + 256 i, i along kRow
  double2* const mid = buf + hi * kRow + lo;      // pass 2: row hi, position lo + 16 i, i along 17
  double2* const row = buf + lo * kRow + hi * 17; // pass 3: row lo, positions 16 hi + i
  dft16<false>(v);
#pragma unroll
  for (int k = 0; k < 16; k++) col[k * kRow] = k ? cmul(v[slot16(k)], twiddle<false>(tq, k * t)) : v[0];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = mid[i * 17];
  dft16<false>(v);
#pragma unroll
  for (int k = 0; k < 16; k++) mid[k * 17] = k ? cmul(v[slot16(k)], tw2[k * 16 + lo]) : v[0];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = row[i];
  dft16<false>(v);
  double2 g[16];
#pragma unroll
  for (int k = 0; k < 16; k++) g[k] = cmul(v[slot16(k)], __ldg(&gfft[t + 256 * k]));  // frequency lo + 16 hi + 256 k
  dft16<true>(g);
#pragma unroll
  for (int i = 0; i < 16; i++) {
    double2 w = tw2[hi * 16 + i];
    w.y = -w.y;
    row[i] = cmul(g[slot16(i)], w);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = mid[i * 17];
  dft16<true>(v);
#pragma unroll
  for (int i = 0; i < 16; i++) mid[i * 17] = cmul(v[slot16(i)], twiddle<true>(tq, hi * (lo + 16 * i)));
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = col[i * kRow];
  dft16<true>(v);
#pragma unroll
  for (int i = 0; i < 16; i++) col[i * kRow] = v[slot16(i)];
  __syncthreads();
}

// A run of the sample's demod positions: taps kk0..kk1 read chunk position
// c0 + step * (kk - kk0), step -1 (consecutive positions of one owning tile)
// or 0 (one clamped position).
struct Run {
  int kk0, kk1, step;
  long long c0;
};
constexpr int kMaxRuns = 8;

// Phase clocks for inspection (thread 0, first block of a sample only).
__device__ __forceinline__ void phase_clock(const GuardArgs& g, int y, int k) {
  if (g.dbg_clk && threadIdx.x == 0 && y < kGuardClockSamples) g.dbg_clk[(size_t)y * kPhaseSlots + k] = clock64();
}

template <int FMT, class Src>
__global__ void __launch_bounds__(kGT, 2) guard_kernel(const __grid_constant__ Src src) {
  const GuardArgs& g = src.get();
  extern __shared__ double2 gsm[];
  double2* buf = gsm;             // [kSlots]
  double2* tq = buf + kSlots;     // [kTwPad] exp(-2 pi i k / 4096), padded
  double2* tw2 = tq + kTwPad;     // [16][16] exp(-2 pi i k j / 256)
  double* dem = reinterpret_cast<double*>(tw2 + 256);  // [2 * hb + 1], indexed like the sync taps
  __shared__ Run runs[kMaxRuns];
  __shared__ int nruns, skip;
  __shared__ double red[kGT / 32];
  const int t = threadIdx.x;
  // the tables are the context's: staged before the wait for the launch ahead
  for (int k = t; k < kTwQ; k += kGT) tq[k + (k >> 3)] = __ldg(&g.tw[k]);
  tw2[t] = __ldg(&g.tw[16 * (t & 15) * (t >> 4)]);
  chain_wait();
  const int n_listed = min(*g.count, g.cap);
  const double dc = g.dc ? (double)*g.dc : 0.0;
  const long long last = g.total - 1;
  const int W = 2 * g.hb + 1;
  const int V = kN - 1 - 2 * g.ha;  // demod positions one FFT block yields
  if ((int)blockIdx.x >= n_listed) return;  // whole CTA
  for (int y = blockIdx.x; y < n_listed; y += gridDim.x) {
    const long long s = g.list[y];
    const long long f = (unsigned)s / (unsigned)g.spp;  // chunk positions fit 32 bits
    const long long J = kOverlap + (s - f * g.spp);
    phase_clock(g, y, 0);
    if (t == 0) {
      // tap kk reads tile position q = wrap(J + hb - kk), chunk position
      // clamp(f * spp - kOverlap + q): one or two runs of q (the tile wrap),
      // each cut where the clamp starts or the owning tile changes
      int n = 0;
      auto add_q_run = [&](int kk0, int kk1, long long q0) {
        const long long c0 = f * g.spp - kOverlap + q0;  // unclamped, falls by one per tap
        int kk = kk0;
        while (kk <= kk1 && n < kMaxRuns) {
          const long long c = c0 - (kk - kk0);
          int kend;
          if (c > last) {
            kend = (int)min((long long)kk1, kk0 + (c0 - last) - 1);
            runs[n++] = {kk, kend, 0, last};
          } else if (c < 0) {
            kend = kk1;
            runs[n++] = {kk, kend, 0, 0};
          } else {
            // the owning tile's first position
            const long long stop = (long long)((unsigned)c / (unsigned)g.spp) * g.spp;
            kend = (int)min((long long)kk1, kk + (c - stop));
            runs[n++] = {kk, kend, -1, c};
          }
          kk = kend + 1;
        }
      };
      const long long top = J + g.hb;  // q of tap 0 before the wrap
      if (top >= g.tile) {
        const int kw = (int)(top - g.tile);  // last tap whose q wraps
        add_q_run(0, kw, top - g.tile);
        add_q_run(kw + 1, W - 1, g.tile - 1);
      } else {
        add_q_run(0, W - 1, top);
      }
      nruns = n;
      // A window that reaches the zero fill past the samples read (the
      // capture's end) has analytic-signal values built from the taps' tails
      // alone, whose phase no FP64 evaluation fixes (the FFT's rounding, the
      // reference's included, exceeds them): such a sample keeps its FP32
      // value.
      int sk = 0;
      if (g.n_read < g.total) {
        for (int r = 0; r < n; r++) {
          const long long owner = (unsigned)runs[r].c0 / (unsigned)g.spp;
          const long long tile0 = owner * g.spp - kOverlap;
          const long long vmax = (kOverlap + runs[r].c0 - owner * g.spp) + g.ha;  // highest tile position read
          const long long pmax = min(tile0 + min(vmax, (long long)g.tile - 1), last);
          if (pmax >= g.n_read) sk = 1;
        }
      }
      skip = sk;
    }
    __syncthreads();
    if (skip) {
      if (t == 0 && g.values) g.values[y] = __longlong_as_double(0x7ff8000000000000LL);
      __syncthreads();  // runs and skip are rewritten for the next sample
      continue;
    }
    for (int r = 0; r < nruns; r++) {
      const Run run = runs[r];
      const long long c_hi = run.c0, c_lo = run.c0 + (long long)run.step * (run.kk1 - run.kk0);
      const long long owner = (unsigned)c_lo / (unsigned)g.spp;
      const long long tile0 = owner * g.spp - kOverlap;  // chunk position of the owner's tile position 0
      for (long long cb = c_lo; cb <= c_hi; cb += V) {
        const long long ce = min(cb + V - 1, c_hi);
        const int nz = (int)(ce - cb) + 2;             // z at tile positions J2(cb) - 1 .. J2(ce)
        const long long v0 = (kOverlap + cb - owner * g.spp) - 1 - g.ha;  // tile position of buf[0]
        const int L = nz + 2 * g.ha;
        // tile positions clamped to the chunk, and those read, as offsets from the tile's start
        const int q_lo = (int)max(-tile0, 0LL), q_hi = (int)min(last - tile0, (long long)g.tile - 1);
        const int q_read = (int)min((long long)g.n_read - tile0, (long long)g.tile);
        const uint8_t* const raw0 = g.raw + tile0 * (FMT == kInU8 ? 1 : 2);
        double2 v[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const int u = t + i * kGT;
          double x = 0.0;
          if (u < L) {
            const int q = min(max(wrap_pos((int)v0 + u, (int)g.tile), q_lo), q_hi);
            x = q < q_read ? (double)raw_convert<FMT>(raw0, q) - dc : 0.0;
          }
          v[i] = make_double2(x, 0.0);
        }
        const bool first_block = r == 0 && cb == c_lo;
        if (first_block) phase_clock(g, y, 1);
        convolve(v, buf, tq, tw2, g.gfft);
        if (first_block) phase_clock(g, y, 2);
        // phases of the block's z, in place
        for (int i = t; i < nz; i += kGT) {
          double2& z = buf[slot_of(g.ha + i)];
          z.x = atan2(z.y, z.x);
        }
        __syncthreads();
        if (first_block) phase_clock(g, y, 3);
        // k_unwrap_to_hz (fm_demod.cu:222-244) for chunk positions cb .. ce
        for (int i = t; i + 1 < nz; i += kGT) {
          double d = buf[slot_of(g.ha + i + 1)].x - buf[slot_of(g.ha + i)].x;
          if (d > kPi64) d -= kTau64;
          if (d < -kPi64) d += kTau64;
          const double hz = d * g.scale;
          if (run.step == 0) {
            for (int kk = run.kk0; kk <= run.kk1; kk++) dem[kk] = hz;  // one position, many taps
          } else {
            dem[run.kk0 + (int)(run.c0 - (cb + i))] = hz;
          }
        }
        __syncthreads();  // buf is refilled by the next block
        if (first_block) phase_clock(g, y, 4);
      }
    }
    phase_clock(g, y, 5);
    // sync sum in a fixed order: strided partials, warp tree, warps in order
    double acc = 0.0;
    for (int kk = t; kk < W; kk += kGT) acc += __ldg(&g.hs64[kk]) * dem[kk];
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if ((t & 31) == 0) red[t >> 5] = acc;
    __syncthreads();
    if (t == 0) {
      double x64 = 0.0;
      for (int w = 0; w < kGT / 32; w++) x64 += red[w];
      const bool in_pulse = x64 <= g.thr_hz;  // the reference's FP64 decision
      if (in_pulse != (g.sync[s] <= g.thr_rel)) {
        if (g.flips) atomicAdd(g.flips, 1);
        if (g.pulse_bits) atomicXor(&g.pulse_bits[s >> 5], 1u << (s & 31));
      }
      float r = (float)(x64 - g.ire0);
      if (in_pulse && !(r <= g.thr_rel)) r = g.thr_rel;
      if (!in_pulse && r <= g.thr_rel) r = nextafterf(g.thr_rel, 3.0e38f);
      g.sync[s] = r;
      if (g.values) g.values[y] = x64;
      if (g.dbg_clk && y < kGuardClockSamples) g.dbg_clk[(size_t)y * kPhaseSlots + 7] = nruns;
    }
    phase_clock(g, y, 6);
    __syncthreads();  // runs, dem and red are reused by the next sample
  }
}

}  // namespace

size_t guard_smem_bytes(int hb) {
  return (size_t)(kSlots + kTwPad + 256) * sizeof(double2) + (size_t)(2 * hb + 1) * sizeof(double);
}

bool guard_supported(int ha, int hb) {
  // one FFT block must yield at least one position, and the sync window must
  // not wrap below the tile start (J - hb >= 0 for every J >= kOverlap)
  return 2 * ha + 2 <= kN && hb < kOverlap && guard_smem_bytes(hb) <= (size_t)kMaxClassBytes;
}

namespace {
template <class S>
cudaError_t launch_guard(const S& src, const GuardArgs& g, int portions, int ctas, cudaStream_t st) {
  const size_t smem = guard_smem_bytes(g.hb);
  auto go = [&](auto kernel) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_chained(kernel, dim3(ctas, 1, portions), dim3(kGT), smem, st, src);
  };
  if (g.in_fmt == kInS16) return go(guard_kernel<kInS16, S>);
  if (g.in_fmt == kInU16) return go(guard_kernel<kInU16, S>);
  return go(guard_kernel<kInU8, S>);
}
}  // namespace

cudaError_t launch_sync_guard(const GuardArgs& g, cudaStream_t st) {
  if (!guard_supported(g.ha, g.hb) || g.cap <= 0) return cudaErrorInvalidValue;
  // a typical chunk lists a few dozen samples, each on its own SM; two CTAs fit an SM
  const int ctas = std::max(1, std::min(g.cap, 148 * 2));
  return launch_guard(ArgsOne<GuardArgs>{g}, g, 1, ctas, st);
}

cudaError_t launch_sync_guard_many(const ArgsMany<GuardArgs>& p, int portions, cudaStream_t st) {
  if (portions <= 0) return cudaSuccess;
  const GuardArgs& g = p.a[0];  // the design every capture of a round shares
  if (!guard_supported(g.ha, g.hb) || g.cap <= 0) return cudaErrorInvalidValue;
  const int ctas = std::max(1, std::min(g.cap, (148 * 2 + portions - 1) / portions));
  return launch_guard(p, g, portions, ctas, st);
}

}  // namespace cuvhs
