// Dropout detection, TBC mapping and concealment (reference K7,
// src/pipeline/dropout_detect.cu:17-339).
//
// The tile mean of the envelope comes from the per-CTA partial sums K1a
// already wrote.  Block means (16 samples) over the active range are
// classified into below-down / above-up / between; the two-state hysteresis
// over those classes is a "last decisive class" scan, so each segment's
// incoming state comes from one prefix pass instead of the reference's
// one-thread-per-field walk.  The short list of state changes is then merged,
// filtered and mapped to TBC lines in order by prefix sums, and the entries
// are concealed a thread per column, each pixel from where the reference's
// copy loop (column step by column step) would have taken it.
//
// Two forms share those steps:
//  * two-pass (the decoder): a wide class kernel (one thread per block, every
//    field at once, the envelope staged through shared memory with coalesced
//    loads) writes one class byte per block, and a per-field kernel reads the
//    bytes back from L2, scans, maps and conceals the luma.  The envelope read
//    -- the stage's HBM traffic -- runs on every SM.  Luma is final once the
//    luma resampler has run, so it is concealed (and can leave the device)
//    while chroma is still being decoded; chroma is concealed afterwards.
//  * fused (cuvhs_dropouts_noalloc): one CTA per field does everything, with
//    the classes in shared memory, so it needs no scratch beyond the partials.
#include <cuda_runtime.h>

#include "chain.cuh"
#include "cuvhs_internal.h"

namespace cuvhs {
namespace {

constexpr int kThreadsD = 256;       // fused kernel and class kernel
constexpr int kThreadsScan = 1024;   // two-pass scan kernel: a thread per column of an NTSC line
constexpr int kMaxEvents = 2048;
constexpr int kStage = kThreadsD * 16;  // envelope samples one class CTA stages
constexpr int kMaxEnvBlocks = 1024;     // envelope partials a class CTA holds in shared memory

// Index of the line holding pos among the n lines whose starts are ll[0..n].
__device__ int find_line(const double* ll, int n, double pos) {
  if (pos < ll[0] || pos >= ll[n]) return -1;
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (ll[mid] <= pos) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Active sample range [s0, s1) of field f (chunk sample indices).
__device__ __forceinline__ void active_range(const DropoutArgs& a, int f, int& s0, int& s1) {
  const double* ll = a.ll + (size_t)f * a.lines_per_frame;
  const int fstart = f * a.spp;
  s0 = max((int)ll[a.active_line_start], fstart);
  s1 = min((int)ll[a.active_line_start + a.out_h], fstart + a.spp);
}

// Lower threshold: 0.18 x the tile mean of the envelope, summed in partial order.
__device__ __forceinline__ double down_threshold(const DropoutArgs& a, int f) {
  double tot = 0.0;
  for (int b = 0; b < a.env_blocks; b++) tot += a.env_part[(size_t)f * a.env_blocks + b];
  return tot / (double)a.spp * 0.18;
}

__device__ __forceinline__ unsigned char block_class(double sum, int n, double down, double up) {
  const double m = sum / (double)n;
  return m <= down ? 0 : (m >= up ? 1 : 2);  // 0 = at/below down, 1 = at/above up, 2 = between
}

// Block-wide exclusive sum over THREADS threads (warp shuffles, then the warp
// totals).  wsh holds 32 ints; every thread must call.
template <int THREADS>
__device__ __forceinline__ int block_excl_sum(int v, int* wsh, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = THREADS / 32;
  int x = v;
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += o;
  }
  if (lane == 31) wsh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < NW ? wsh[lane] : 0;
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += o;
    }
    if (lane < NW) wsh[lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  const int res = x - v + (warp > 0 ? wsh[warp - 1] : 0);
  *total = wsh[NW - 1];
  __syncthreads();  // wsh free for the next scan
  return res;
}

struct MapScratch {
  double ll[kMaxFieldLines];  // the field's line starts from the first active line
  int rf_s[kMaxRfDropouts], rf_e[kMaxRfDropouts];
  int sl[kMaxRfDropouts], el[kMaxRfDropouts];  // lines each span touches
  int base[kMaxRfDropouts];                    // lines of the spans before it
  int wsh[32];
};

// The field's active line starts into shared memory (no barrier).
template <int THREADS>
__device__ __forceinline__ void load_lines(const DropoutArgs& a, int f, MapScratch& m) {
  const double* ll = a.ll + (size_t)f * a.lines_per_frame + a.active_line_start;
  for (int i = threadIdx.x; i <= a.out_h; i += THREADS) m.ll[i] = ll[i];
}

// Entries of one span: TBC line l of the lines [sl, el] it touches, columns
// [sx, ex).  False where the line gets no entry.
__device__ __forceinline__ bool span_entry(const double* ll, int l, int sl, int el, double sa, double ea, int W,
                                           int& sx, int& ex) {
  const double l0 = ll[l], len = ll[l + 1] - l0;
  if (len <= 0.0) return false;
  sx = (l == sl) ? max(0, (int)((sa - l0) / len * (double)W)) : 0;
  ex = (l == el) ? min(W, (int)((ea - l0) / len * (double)W + 0.999)) : W;
  return ex > sx;
}

// Step 4 (whole CTA): merge start/end events (<= 30 samples apart), keep <= 128
// spans, drop spans < 10 samples, map to TBC lines.  The state alternates from
// "no dropout", so events 2i and 2i + 1 are the start and end of run i (the
// last may lack its end: the range's end); a run joins the one before it when
// its start lies within 30 samples of that one's end, so the spans are the
// runs numbered by a prefix sum; the lines the spans touch, in the spans'
// order, are numbered by a second one and taken a thread each, their entries
// placed by a third.  Latency bound (a few hundred events at most, a few KB):
// one thread walking the events with each line search in global memory took
// 0.5 ms for a field that reaches past the capture's end, whose one span
// touches every line; with a thread per span walking its lines, and the
// concealment below testing every entry in every column, the dropout stage of
// 16 PAL fields took 154 us, now 79.
template <int THREADS>
__device__ void map_events(const DropoutArgs& a, int f, const int* events, int ne, int s0, int s1, MapScratch& m) {
  static_assert(THREADS >= kMaxRfDropouts, "a thread per span");
  const int tid = threadIdx.x, H = a.out_h, W = a.out_w;
  const int runs = (ne + 1) / 2;
  auto start = [&](int i) { return s0 + (events[2 * i] >> 1) * 16; };
  auto end = [&](int i) { return 2 * i + 1 < ne ? s0 + (events[2 * i + 1] >> 1) * 16 : s1; };
  int nrf = 0;
  for (int base = 0; base < runs; base += THREADS) {
    const int i = base + tid;
    const bool in = i < runs;
    const bool first = in && (i == 0 || start(i) - end(i - 1) > 30);
    int total;
    const int g = nrf + block_excl_sum<THREADS>(first ? 1 : 0, m.wsh, &total) + (first ? 1 : 0) - 1;
    if (in && g < kMaxRfDropouts) {
      if (first) m.rf_s[g] = start(i);
      if (i + 1 == runs || start(i + 1) - end(i) > 30) m.rf_e[g] = end(i);
    }
    nrf += total;
  }
  nrf = min(nrf, kMaxRfDropouts);
  __syncthreads();
  int sl = 0, el = -1;
  if (tid < nrf && m.rf_e[tid] - m.rf_s[tid] >= 10) {
    sl = find_line(m.ll, H, (double)m.rf_s[tid]);
    if (sl >= 0) {
      el = find_line(m.ll, H, (double)m.rf_e[tid] - 1.0);
      if (el < 0) el = H - 1;
    }
  }
  const int cnt = sl >= 0 ? max(el - sl + 1, 0) : 0;
  int lines;
  const int base = block_excl_sum<THREADS>(cnt, m.wsh, &lines);
  if (tid < nrf) {
    m.sl[tid] = sl;
    m.el[tid] = el;
    m.base[tid] = base;
  }
  __syncthreads();
  int* ol = a.do_lines + (size_t)f * kMaxDropouts;
  int* os = a.do_starts + (size_t)f * kMaxDropouts;
  int* oe = a.do_ends + (size_t)f * kMaxDropouts;
  int n = 0;
  for (int j0 = 0; j0 < lines && n < kMaxDropouts; j0 += THREADS) {
    const int j = j0 + tid;
    bool ok = false;
    int l = 0, sx = 0, ex = 0;
    if (j < lines) {
      // the last span whose lines start at or before j (one without lines shares the next one's base)
      int lo = 0, hi = nrf - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (m.base[mid] <= j) lo = mid;
        else hi = mid - 1;
      }
      l = m.sl[lo] + j - m.base[lo];
      ok = span_entry(m.ll, l, m.sl[lo], m.el[lo], (double)m.rf_s[lo], (double)m.rf_e[lo], W, sx, ex);
    }
    int total;
    const int k = n + block_excl_sum<THREADS>(ok ? 1 : 0, m.wsh, &total);
    if (ok && k < kMaxDropouts) {
      ol[k] = l;
      os[k] = sx;
      oe[k] = ex;
    }
    n += total;
  }
  if (tid == 0) a.do_count[f] = min(n, kMaxDropouts);
}

// Step 5: conceal from the line above (below for line 0).  The reference's
// copy loop takes the entries 32 at a time, one column step after another,
// every load of a step before its stores: entry d copies column c at step
// c - sx_d.  So, inside a group of 32, column c of entry d holds what its
// source row held at that step: the row's own pixel, or, where an entry e
// covers c on that row and started further right (sx_e > sx_d, an earlier
// step; the smallest such sx_e wrote last), what e's source row held at e's
// step.  Each pixel's origin therefore follows from the entries alone, and
// columns never mix: a thread takes a column through all groups in order,
// the group's loads all in flight before its stores.  A warp takes 32 columns:
// its lanes first look at the group's entries against those columns, so that
// entries elsewhere cost a test each, and one that covers them all with no
// other entry on its rows (a dropout of whole lines) a load and a store.
// Issue bound on the one SM of a field with many entries, latency bound
// otherwise; a warp stepping through the columns took 0.7 us a step, 1.4 ms
// for a field with 512 entries.
struct ConcealEntry {
  short line, src, sx, ex;
  unsigned before;  // entries of the group on row src with a larger sx
  unsigned after;   // entries of the group on the same line with a smaller sx (they write later)
};
static_assert(kMaxDropouts % 32 == 0, "whole groups");

// The field's n entries with their links into shared memory (ends with a barrier).
template <int THREADS>
__device__ void conceal_entries(const DropoutArgs& a, int f, int n, ConcealEntry* ent) {
  const int* ol = a.do_lines + (size_t)f * kMaxDropouts;
  const int* os = a.do_starts + (size_t)f * kMaxDropouts;
  const int* oe = a.do_ends + (size_t)f * kMaxDropouts;
  const int lane = threadIdx.x & 31;
  for (int g = (threadIdx.x >> 5) * 32; g < n; g += THREADS) {
    const int d = g + lane;
    int line = -1, src = -2, sx = 0, ex = 0;
    if (d < n) {
      line = ol[d];
      sx = os[d];
      ex = oe[d];
      src = line > 0 ? line - 1 : line + 1;
      if (src >= a.out_h) ex = sx;
    }
    unsigned before = 0, after = 0;
    for (int e = 0; e < 32; e++) {
      const int le = __shfl_sync(0xffffffffu, line, e), se = __shfl_sync(0xffffffffu, sx, e);
      if (le == src && se > sx) before |= 1u << e;
      if (le == line && se < sx) after |= 1u << e;
    }
    ent[d] = ConcealEntry{(short)line, (short)src, (short)sx, (short)ex, before, after};
  }
  __syncthreads();
}

__device__ __forceinline__ bool covers(const ConcealEntry& e, int c) { return c >= e.sx && c < e.ex; }

// Columns [c0, c0 + 32) of one plane through every group of entries (whole warp).
__device__ void conceal_columns(const ConcealEntry* ent, int n, uint16_t* plane, int W, int c0) {
  const int lane = threadIdx.x & 31;
  const int c = c0 + lane;
  const int c_end = min(c0 + 32, W);
  for (int g = 0; g < n; g += 32) {
    int src = 0, dst = 0;
    unsigned links = 0;
    bool touch = false, whole = false;
    if (g + lane < n) {
      const ConcealEntry e = ent[g + lane];
      touch = e.sx < c_end && e.ex > c0;
      whole = e.sx <= c0 && e.ex >= c_end;
      links = e.before | e.after;
      src = e.src * W;
      dst = e.line * W;
    }
    const unsigned any = __ballot_sync(0xffffffffu, touch);
    if (!any) continue;
    const unsigned plain = __ballot_sync(0xffffffffu, whole && (links & any) == 0);
    uint16_t v[32];
    unsigned act = 0;
#pragma unroll
    for (int d = 0; d < 32; d++) {
      v[d] = 0;
      if (!(any >> d & 1u)) continue;
      const int row_d = __shfl_sync(0xffffffffu, src, d);
      if (c >= W) continue;
      if (plain >> d & 1u) {
        act |= 1u << d;
        v[d] = plane[row_d + c];
        continue;
      }
      const ConcealEntry e = ent[g + d];
      if (!covers(e, c)) continue;
      bool last = true;  // no later write of the group to this pixel
      for (unsigned w = e.after & any; w; w &= w - 1) last = last && !covers(ent[g + __ffs(w) - 1], c);
      if (!last) continue;
      act |= 1u << d;
      int row = e.src;
      for (unsigned w = e.before & any; w;) {
        int best = -1, bsx = 1 << 30;
        for (; w; w &= w - 1) {
          const int k = __ffs(w) - 1;
          if (covers(ent[g + k], c) && ent[g + k].sx < bsx) {
            best = k;
            bsx = ent[g + k].sx;
          }
        }
        if (best >= 0) {
          row = ent[g + best].src;
          w = ent[g + best].before & any;
        }
      }
      v[d] = plane[row * W + c];
    }
#pragma unroll
    for (int d = 0; d < 32; d++) {
      if (!(any >> d & 1u)) continue;
      const int row_d = __shfl_sync(0xffffffffu, dst, d);
      if (act >> d & 1u) plane[row_d + c] = v[d];
    }
  }
}

// ------------------------------------------------------------------ fused form

__global__ void __launch_bounds__(kThreadsD) dropout_kernel(DropoutArgs a) {
  chain_wait();
  extern __shared__ unsigned char cls[];  // [a.max_blocks]
  __shared__ int last_cls[kThreadsD];
  __shared__ int state_in[kThreadsD];
  __shared__ int ev_count[kThreadsD];
  __shared__ int ev_off[kThreadsD];
  __shared__ int events[kMaxEvents];  // block index * 2 + (1 = start, 0 = end)
  __shared__ int n_events;
  __shared__ MapScratch map;
  __shared__ ConcealEntry ent[kMaxDropouts];
  __shared__ double down_s;
  const int f = blockIdx.x;
  const int tid = threadIdx.x;
  if (tid == 0) down_s = down_threshold(a, f);
  load_lines<kThreadsD>(a, f, map);
  int s0, s1;
  active_range(a, f, s0, s1);
  __syncthreads();
  if (s1 <= s0) {
    if (tid == 0) a.do_count[f] = 0;
    return;
  }
  const int nb = min((s1 - s0 + 15) / 16, a.max_blocks);
  const double down = down_s, up = down * 1.25;
  // 1. classify blocks
  for (int b = tid; b < nb; b += kThreadsD) {
    const int b0 = s0 + b * 16, b1 = min(b0 + 16, s1);
    double sum = 0.0;
    for (int i = b0; i < b1; i++) sum += (double)__ldg(&a.env[i]);
    cls[b] = block_class(sum, b1 - b0, down, up);
  }
  __syncthreads();
  // 2. per-segment last decisive class
  const int per = (nb + kThreadsD - 1) / kThreadsD;
  const int b_lo = min(nb, tid * per), b_hi = min(nb, b_lo + per);
  int lc = -1;
  for (int b = b_lo; b < b_hi; b++)
    if (cls[b] != 2) lc = cls[b];
  last_cls[tid] = lc;
  __syncthreads();
  if (tid == 0) {
    int st = 0;  // 0 = no dropout open
    for (int t = 0; t < kThreadsD; t++) {
      state_in[t] = st;
      if (last_cls[t] == 0) st = 1;
      else if (last_cls[t] == 1) st = 0;
    }
  }
  __syncthreads();
  // 3. state changes, counted then written in order
  int st = state_in[tid], cnt = 0;
  for (int b = b_lo; b < b_hi; b++) {
    if (cls[b] == 0 && !st) { st = 1; cnt++; }
    else if (cls[b] == 1 && st) { st = 0; cnt++; }
  }
  ev_count[tid] = cnt;
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int t = 0; t < kThreadsD; t++) { ev_off[t] = acc; acc += ev_count[t]; }
    n_events = acc;
  }
  __syncthreads();
  st = state_in[tid];
  int k = ev_off[tid];
  for (int b = b_lo; b < b_hi; b++) {
    if (cls[b] == 0 && !st) { st = 1; if (k < kMaxEvents) events[k] = b * 2 + 1; k++; }
    else if (cls[b] == 1 && st) { st = 0; if (k < kMaxEvents) events[k] = b * 2; k++; }
  }
  __syncthreads();
  map_events<kThreadsD>(a, f, events, min(n_events, kMaxEvents), s0, s1, map);
  __syncthreads();  // the entries and their count, written by this CTA
  const int n = a.do_count[f];
  if (n <= 0) return;  // whole CTA
  conceal_entries<kThreadsD>(a, f, n, ent);
  const size_t F = (size_t)a.out_h * a.out_w;
  for (int c0 = tid & ~31; c0 < a.out_w; c0 += kThreadsD) {
    conceal_columns(ent, n, a.luma + f * F, a.out_w, c0);
    conceal_columns(ent, n, a.chroma + f * F, a.out_w, c0);
  }
}

// --------------------------------------------------------------- two-pass form

// grid (ceil(max_blocks / kThreadsD), fields): CTA x classifies blocks
// [x*256, x*256 + 256) of field y.  The 4096 envelope samples behind them are
// staged with coalesced loads into rows of 17 floats (conflict-free column
// reads), then each thread sums its row in sample order.
template <class Src>
__global__ void __launch_bounds__(kThreadsD) dropout_class_kernel(const __grid_constant__ Src src) {
  const DropoutArgs& a = src.get();
  if ((int)blockIdx.y >= a.fields) return;  // whole CTA: a batched capture with fewer fields
  chain_wait();
  __shared__ float stage[kThreadsD * 17];
  __shared__ double part[kMaxEnvBlocks];
  __shared__ double down_s;
  const int f = blockIdx.y, tid = threadIdx.x;
  int s0, s1;
  active_range(a, f, s0, s1);
  const int nb = min((s1 - s0 + 15) / 16, a.max_blocks);
  const int b_first = blockIdx.x * kThreadsD;
  if (s1 <= s0 || b_first >= nb) return;  // whole CTA leaves together
  // the field's envelope partial sums, loaded in parallel with the stage
  const bool part_in_smem = a.env_blocks <= kMaxEnvBlocks;
  if (part_in_smem)
    for (int b = tid; b < a.env_blocks; b += kThreadsD) part[b] = a.env_part[(size_t)f * a.env_blocks + b];
  const int x0 = s0 + b_first * 16;
  const int nx = min(kStage, s1 - x0);
  // loads at a clamped index, so that all of a thread's loads are in flight
  // at once; samples past the range are zeroed afterwards
#pragma unroll
  for (int i = tid; i < kStage; i += kThreadsD) {
    const float e = __ldg(&a.env[x0 + min(i, nx - 1)]);
    stage[(i >> 4) * 17 + (i & 15)] = i < nx ? e : 0.0f;
  }
  __syncthreads();
  if (tid == 0) {
    // summed in partial order, as down_threshold
    double tot = 0.0;
    if (part_in_smem)
      for (int b = 0; b < a.env_blocks; b++) tot += part[b];
    else
      for (int b = 0; b < a.env_blocks; b++) tot += a.env_part[(size_t)f * a.env_blocks + b];
    down_s = tot / (double)a.spp * 0.18;
  }
  __syncthreads();
  const int b = b_first + tid;
  if (b >= nb) return;
  const int n = min(16, s1 - (s0 + b * 16));
  double sum = 0.0;
  for (int i = 0; i < n; i++) sum += (double)stage[tid * 17 + i];
  const double down = down_s;
  a.cls[(size_t)f * a.max_blocks + b] = block_class(sum, n, down, down * 1.25);
}

// "Last decisive class" prefix: combine(left, right) = right != -1 ? right : left.
// Block-wide over kThreadsScan threads; wsh holds 32 ints, every thread must call.
__device__ __forceinline__ int block_excl_last(int v, int* wsh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = kThreadsScan / 32;
  int x = v;
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off && x == -1) x = o;
  }
  if (lane == 31) wsh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < NW ? wsh[lane] : -1;
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off && w == -1) w = o;
    }
    if (lane < NW) wsh[lane] = w;
  }
  __syncthreads();
  int ex = __shfl_up_sync(0xffffffffu, x, 1);
  if (lane == 0) ex = -1;
  if (ex == -1 && warp > 0) ex = wsh[warp - 1];
  __syncthreads();
  return ex;
}

// One CTA per field: class bytes back from L2 into shared memory, then the
// hysteresis scan, event list, mapping and luma concealment (chroma is
// concealed by conceal_chroma_kernel once the chroma planes are final).  The
// luma is concealed here rather than in a kernel of its own: the chroma lines
// fill the SMs by then, and one more low-priority launch held the luma copy
// of a 40-field capture back by 18 us (1,617 -> 1,634 us a capture).
template <class Src>
__global__ void __launch_bounds__(kThreadsScan) dropout_scan_kernel(const __grid_constant__ Src src) {
  const DropoutArgs& a = src.get();
  if ((int)blockIdx.x >= a.fields) return;  // whole CTA
  chain_wait();
  extern __shared__ uint4 cls4[];  // [a.max_blocks / 16]
  __shared__ int wsh[32];
  __shared__ int events[kMaxEvents];
  __shared__ MapScratch map;
  __shared__ ConcealEntry ent[kMaxDropouts];
  const unsigned char* cls = reinterpret_cast<const unsigned char*>(cls4);
  const int f = blockIdx.x, tid = threadIdx.x;
  int s0, s1;
  active_range(a, f, s0, s1);
  if (s1 <= s0) {
    if (tid == 0) a.do_count[f] = 0;
    return;  // whole CTA leaves together
  }
  const int nb = min((s1 - s0 + 15) / 16, a.max_blocks);
  const uint4* cls_in = reinterpret_cast<const uint4*>(a.cls + (size_t)f * a.max_blocks);
  for (int i = tid; i < (nb + 15) / 16; i += kThreadsScan) cls4[i] = cls_in[i];
  load_lines<kThreadsScan>(a, f, map);
  __syncthreads();
  const int per = (nb + kThreadsScan - 1) / kThreadsScan;
  const int b_lo = min(nb, tid * per), b_hi = min(nb, b_lo + per);
  int lc = -1;
  for (int b = b_lo; b < b_hi; b++)
    if (cls[b] != 2) lc = cls[b];
  const int lc_in = block_excl_last(lc, wsh);
  const int st_in = lc_in == 0 ? 1 : 0;  // 1 = dropout open
  int st = st_in, cnt = 0;
  for (int b = b_lo; b < b_hi; b++) {
    if (cls[b] == 0 && !st) { st = 1; cnt++; }
    else if (cls[b] == 1 && st) { st = 0; cnt++; }
  }
  int n_events;
  int k = block_excl_sum<kThreadsScan>(cnt, wsh, &n_events);
  st = st_in;
  for (int b = b_lo; b < b_hi; b++) {
    if (cls[b] == 0 && !st) { st = 1; if (k < kMaxEvents) events[k] = b * 2 + 1; k++; }
    else if (cls[b] == 1 && st) { st = 0; if (k < kMaxEvents) events[k] = b * 2; k++; }
  }
  __syncthreads();
  if (n_events == 0) {
    if (tid == 0) a.do_count[f] = 0;
    return;  // whole CTA
  }
  map_events<kThreadsScan>(a, f, events, min(n_events, kMaxEvents), s0, s1, map);
  __syncthreads();  // the entries and their count, written by this CTA
  const int n = a.do_count[f];
  if (n <= 0) return;  // whole CTA
  conceal_entries<kThreadsScan>(a, f, n, ent);
  uint16_t* plane = a.luma + (size_t)f * a.out_h * a.out_w;
  for (int c0 = tid & ~31; c0 < a.out_w; c0 += kThreadsScan) conceal_columns(ent, n, plane, a.out_w, c0);
}

// Chroma concealment of fields [f0, f0 + nf) from the entries the scan kernel
// wrote: grid (fields, column strips), a thread per column, so that a field
// with many entries is spread over several SMs.
constexpr int kConcealThreads = 256;
template <class Src>
__global__ void __launch_bounds__(kConcealThreads) conceal_chroma_kernel(const __grid_constant__ Src src, int f0, int nf) {
  const DropoutArgs& a = src.get();
  const int f = f0 + blockIdx.x;
  if (f >= f0 + nf || f >= a.fields) return;  // whole CTA
  chain_wait();
  __shared__ ConcealEntry ent[kMaxDropouts];
  const int n = min(max(a.do_count[f], 0), kMaxDropouts);
  if (n == 0) return;  // whole CTA
  conceal_entries<kConcealThreads>(a, f, n, ent);
  const int c0 = blockIdx.y * kConcealThreads + (threadIdx.x & ~31);
  uint16_t* plane = a.chroma + (size_t)f * a.out_h * a.out_w;
  if (c0 < a.out_w) conceal_columns(ent, n, plane, a.out_w, c0);
}

}  // namespace

// The per-field class bytes live in dynamic shared memory.  Both kernels that
// hold them are given the same fixed cap (kMaxClassBytes, not the size one
// call needs), so contexts of different rates on different host threads never
// lower the cap between another thread's set and its launch.
cudaError_t launch_dropouts(const DropoutArgs& a, cudaStream_t st) {
  if (a.fields <= 0) return cudaSuccess;
  const size_t smem = (size_t)a.max_blocks;
  if (smem > (size_t)kMaxClassBytes) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(dropout_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxClassBytes);
  if (e != cudaSuccess) return e;
  return launch_chained(dropout_kernel, dim3(a.fields), dim3(kThreadsD), smem, st, a);
}

size_t dropout_class_bytes_per_field(int spp) { return (size_t)(((spp + 15) / 16 + 15) / 16 * 16); }

namespace {
template <class S>
void conceal_launch(const S& src, const DropoutArgs& a, int portions, int f0, int nf, cudaStream_t st) {
  const int strips = (a.out_w + kConcealThreads - 1) / kConcealThreads;
  launch_chained(conceal_chroma_kernel<S>, dim3(nf, strips, portions), dim3(kConcealThreads), 0, st, src, f0, nf);
}

template <class S>
void two_pass_launch(const S& src, const DropoutArgs& a, int portions, int max_fields, cudaStream_t st) {
  dim3 grid((a.max_blocks + kThreadsD - 1) / kThreadsD, max_fields, portions);
  launch_chained(dropout_class_kernel<S>, grid, dim3(kThreadsD), 0, st, src);
  const size_t smem = (size_t)a.max_blocks;
  cudaFuncSetAttribute(dropout_scan_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxClassBytes);
  launch_chained(dropout_scan_kernel<S>, dim3(max_fields, 1, portions), dim3(kThreadsScan), smem, st, src);
}

}  // namespace

void launch_dropouts_two_pass(const DropoutArgs& a, cudaStream_t st) {
  if (a.fields <= 0) return;
  two_pass_launch(ArgsOne<DropoutArgs>{a}, a, 1, a.fields, st);
}

void launch_dropout_conceal_chroma(const DropoutArgs& a, int f0, int nf, cudaStream_t st) {
  if (nf <= 0 || f0 < 0 || f0 >= a.fields) return;
  conceal_launch(ArgsOne<DropoutArgs>{a}, a, 1, f0, nf, st);
}

void launch_dropouts_two_pass_many(const ArgsMany<DropoutArgs>& p, int portions, int max_fields, cudaStream_t st) {
  if (portions > 0 && max_fields > 0) two_pass_launch(p, p.a[0], portions, max_fields, st);
}

void launch_dropout_conceal_chroma_many(const ArgsMany<DropoutArgs>& p, int portions, int max_fields,
                                        cudaStream_t st) {
  if (portions > 0 && max_fields > 0) conceal_launch(p, p.a[0], portions, 0, max_fields, st);
}

}  // namespace cuvhs
