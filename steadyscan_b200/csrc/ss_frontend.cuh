// Caller-side preparation of frames on the GPU: the part of the reference's MATLAB driver that
// turns raw frames into the block matrix the alignment reads (steady_scan.m:229-234), with
// prefilter_foralignment (steady_scan.m:625-643) and cropimage (steady_scan.m:830-834).
//
// Blur: the reference multiplies the frame's 2-D FFT on a grid padded by L rows and columns with
// the FFT of a periodic Gaussian, i.e. it convolves the zero-padded frame circularly (period H + L
// down a column, W + L along a row) with exp(-(dy^2 + dx^2) / (2 s^2)), dy and dx the circular
// distances, normalised to sum 1. The Gaussian is separable and its normalising sum is the product
// of the two axes' sums, so here the convolution runs as two 1-D circular passes in FP64 (down the
// columns, then along the rows), each over the taps within R = ceil(9.6 s) of the centre, where the
// weights fall below 1e-20 of the centre tap: the terms left out lie below FP64 rounding of the sum.
// Median normalisation divides each (blurred) frame by the median of its H x W samples, found
// exactly by narrowing a range of order-preserving 64-bit keys (NaN anywhere gives NaN, as MATLAB's
// median); the division happens as the samples are put in block order. Block reorder: entry (r, b) of
// a frame's block matrix is the cropped frame's pixel whose column-major index the caller's gather map
// holds there, or 0 where it holds -1 (image2blockmatrix, steady_scan.m:601-613).
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "ss_common.cuh"

namespace ss {

template <class T>
__device__ __forceinline__ double fe_load(const void* base, size_t i) {
  return to_double(reinterpret_cast<const T*>(base)[i]);
}

// One 1-D circular pass of the blur over frames of h x w column-major samples, n frames in a row, for
// windows wider than the tiled passes below hold (R > kBlurMaxR).
// axis 0: down each column (period h + L), axis 1: along each row (period w + L). taps[d], d in
// [0, R], are the normalised weights at circular distance d; `period` is the padded length.
// Grid: (ceil(h / blockDim.x), w, frames); a thread per output sample, lanes on consecutive rows, so
// every tap's loads are coalesced along the column. An output whose window lies inside the frame
// sums its taps in symmetric pairs; near the ends the window wraps over the period and skips the
// zero padding.
template <class InT, int AXIS>
__global__ void __launch_bounds__(256) k_blur_pass(const void* __restrict__ in, double* __restrict__ out, int h, int w,
                                                   int period, const double* __restrict__ taps, int R) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= h) return;
  const int j = blockIdx.y;
  const size_t base = (size_t)blockIdx.z * h * w;
  const int len = AXIS == 0 ? h : w;
  const int pos = AXIS == 0 ? i : j;
  const size_t stride = AXIS == 0 ? 1 : (size_t)h;
  const size_t at = base + (size_t)j * h + i;  // this output; the tap at offset d reads at + d stride
  double s;
  if (pos >= R && pos + R < len) {
    s = fe_load<InT>(in, at) * taps[0];
    for (int d = 1; d <= R; d++)
      s = fma(fe_load<InT>(in, at - d * stride) + fe_load<InT>(in, at + d * stride), taps[d], s);
  } else {
    s = 0.0;
    for (int d = -R; d <= R; d++) {
      int a = pos + d;
      if (a < 0) a += period;
      else if (a >= period) a -= period;
      if (a >= len) continue;  // the zero padding
      s = fma(fe_load<InT>(in, at + (ptrdiff_t)(a - pos) * (ptrdiff_t)stride), taps[d < 0 ? -d : d], s);
    }
  }
  out[at] = s;
}

// The tiled blur passes. Bound: the FP64 pipe (2 R + 1 operations per output and pass). A thread
// computes Q neighbouring outputs from two windows of Q samples that slide outwards one tap at a time,
// so a tap costs it two shared-memory loads and 2 Q FP64 operations in place of 2 Q cached global loads:
// 256 frames of 512 x 512 uint16, R = 10: the two passes 1240 us by k_blur_pass, 743 us here (the
// FP64 pipe 20-30% busy: staging and index work share the issue slots). Down a column the count is odd:
// lanes that many samples apart read different banks.
constexpr int kBlurDown = 9, kBlurAlong = 8;  // outputs of a thread: down the columns, along the rows
constexpr int kBlurMaxR = 320;  // the row pass stages (64 + 2 R) x 32 doubles in shared memory
constexpr int kBlurSeg = 32 * kBlurDown;    // outputs of a warp down a column
constexpr int kBlurCols = 8 * kBlurAlong;   // columns of a CTA of the row pass

// Sums of Q neighbouring outputs: x is the first output's sample, the others STRIDE apart.
template <int STRIDE, int Q>
__device__ __forceinline__ void blur_window(const double* x, const double* taps, int R, double (&acc)[Q]) {
  double lo[Q], hi[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) {
    lo[q] = hi[q] = x[q * STRIDE];
    acc[q] = lo[q] * taps[0];
  }
  // tap d0 + u: sample p of the window sits in slot p mod Q, the new ends replace the samples left behind
  const double* xl = x;
  const double* xh = x + (Q - 1) * STRIDE;
  auto tap = [&](int u) {
    lo[(2 * Q - u) % Q] = xl[-u * STRIDE];
    hi[(Q - 1 + u) % Q] = xh[u * STRIDE];
    const double t = taps[u];
#pragma unroll
    for (int q = 0; q < Q; q++) acc[q] = fma(lo[(q + 2 * Q - u) % Q] + hi[(q + u) % Q], t, acc[q]);
  };
  int left = R;
#pragma unroll 1
  for (; left >= Q; left -= Q) {
#pragma unroll
    for (int u = 1; u <= Q; u++) tap(u);
    xl -= Q * STRIDE;
    xh += Q * STRIDE;
    taps += Q;
  }
#pragma unroll
  for (int u = 1; u < Q; u++) {
    if (u > left) break;
    tap(u);
  }
}

// Position a of the padded axis of length `period`, of which the first len samples are the frame's:
// its sample index, or -1 in the zero padding.
__device__ __forceinline__ int blur_wrap(int a, int len, int period) {
  if (a < 0) a += period;
  else if (a >= period) a -= period;
  return a < len ? a : -1;
}

__host__ __device__ __forceinline__ size_t blur_cols_smem(int R) {
  return ((size_t)(R + 2) + 8 * (size_t)(kBlurSeg + 2 * R)) * sizeof(double);
}
__host__ __device__ __forceinline__ size_t blur_rows_smem(int R) {
  return ((size_t)(R + 2) + (size_t)(kBlurCols + 2 * R) * 32) * sizeof(double);
}
constexpr int kBlurBatch = 6;  // staging loads a thread keeps in flight

// Down the columns; a warp per kBlurSeg outputs of a column. Grid: (segments, ceil(w / 8), frames).
template <class InT>
__global__ void __launch_bounds__(256) k_blur_cols(const InT* __restrict__ in, double* __restrict__ out, int h, int w,
                                                   int period, const double* __restrict__ taps, int R) {
  extern __shared__ double fe_sh[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* s_taps = fe_sh;
  double* sv = fe_sh + (R + 2) + (size_t)warp * (kBlurSeg + 2 * R);
  for (int d = threadIdx.x; d <= R; d += 256) s_taps[d] = taps[d];
  const int j = blockIdx.y * 8 + warp, i0 = blockIdx.x * kBlurSeg, m = min(kBlurSeg, h - i0);
  const size_t at = (size_t)blockIdx.z * h * w + (size_t)j * h;
  if (j < w)
    for (int a0 = lane; a0 < m + 2 * R; a0 += 32 * kBlurBatch) {
      InT v[kBlurBatch];
      bool ok[kBlurBatch];
#pragma unroll
      for (int u = 0; u < kBlurBatch; u++) {
        const int a = a0 + 32 * u, p = a < m + 2 * R ? blur_wrap(i0 - R + a, h, period) : -1;
        ok[u] = p >= 0;
        v[u] = in[at + (ok[u] ? p : 0)];
      }
#pragma unroll
      for (int u = 0; u < kBlurBatch; u++)
        if (a0 + 32 * u < m + 2 * R) sv[a0 + 32 * u] = ok[u] ? to_double(v[u]) : 0.0;
    }
  __syncthreads();
  if (j >= w) return;
  double acc[kBlurDown];
  double* x = sv + R + kBlurDown * lane;
  blur_window<1>(x, s_taps, R, acc);
  __syncwarp();
#pragma unroll
  for (int q = 0; q < kBlurDown; q++) x[q] = acc[q];  // through shared memory: coalesced stores
  __syncwarp();
  for (int a = lane; a < m; a += 32) out[at + i0 + a] = sv[R + a];
}

// Order-preserving 64-bit key of a double and back.
__device__ __forceinline__ unsigned long long fe_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double fe_unkey(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
  return __longlong_as_double((long long)b);
}

// High word of a sample's key: the same order, to 32 bits.
__device__ __forceinline__ unsigned fe_key_hi(double v) {
  const int b = __double2hiint(v);
  return (unsigned)b ^ ((unsigned)(b >> 31) | 0x80000000u);
}

// What the median needs to know of a frame: {smallest high word of a key, ~largest, 0 where a sample
// is NaN}, all taken by minimum from a fill of ones.
constexpr int kFrameStats = 3;
struct KeyRange {
  unsigned lo = ~0u, hi = 0u;
  bool nan = false;
  __device__ __forceinline__ void add(double v) {
    const unsigned k = fe_key_hi(v);
    lo = min(lo, k);
    hi = max(hi, k);
    nan |= isnan(v);
  }
  // the CTA's range into the frame's stats (whole CTA; one atomic per entry and warp)
  __device__ __forceinline__ void commit(unsigned* stats) {
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    const bool any = __any_sync(0xffffffffu, nan);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(stats, lo);
      atomicMin(stats + 1, ~hi);
      if (any) atomicMin(stats + 2, 0u);
    }
  }
};

// Along the rows; lanes on 32 consecutive lines, a warp per kBlurAlong columns. With stats, also each
// frame's key range. Grid: (ceil(h / 32), ceil(w / kBlurCols), frames).
__global__ void __launch_bounds__(256) k_blur_rows(const double* __restrict__ in, double* __restrict__ out, int h, int w,
                                                   int period, const double* __restrict__ taps, int R,
                                                   unsigned* __restrict__ stats) {
  extern __shared__ double fe_sh[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* s_taps = fe_sh;
  double* sv = fe_sh + (R + 2);
  for (int d = threadIdx.x; d <= R; d += 256) s_taps[d] = taps[d];
  const int i = blockIdx.x * 32 + lane, j0 = blockIdx.y * kBlurCols, m = min(kBlurCols, w - j0);
  const size_t at = (size_t)blockIdx.z * h * w + i;
  const bool inside = j0 >= R && j0 + m + R <= w;  // the whole window lies in the frame
  for (int a0 = warp; a0 < m + 2 * R; a0 += 8 * kBlurBatch) {
    double v[kBlurBatch];
#pragma unroll
    for (int u = 0; u < kBlurBatch; u++) {
      const int a = a0 + 8 * u;
      int p = j0 - R + a;
      if (!inside) p = blur_wrap(p, w, period);
      v[u] = (a < m + 2 * R && p >= 0 && i < h) ? in[at + (size_t)p * h] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kBlurBatch; u++)
      if (a0 + 8 * u < m + 2 * R) sv[(a0 + 8 * u) * 32 + lane] = v[u];
  }
  __syncthreads();
  double acc[kBlurAlong];
  const int b = warp * kBlurAlong;
  KeyRange range;
  if (b < m) {
    blur_window<32>(sv + (b + R) * 32 + lane, s_taps, R, acc);
    double* o = out + at + (size_t)(j0 + b) * h;
    if (i < h) {
#pragma unroll
      for (int q = 0; q < kBlurAlong; q++)
        if (b + q < m) {
          o[(size_t)q * h] = acc[q];
          range.add(acc[q]);
        }
    }
  }
  if (stats) range.commit(stats + (size_t)kFrameStats * blockIdx.z);
}

// Key range of frames that are not blurred. Grid: (blocks, frames).
template <class T>
__global__ void __launch_bounds__(256) k_frame_range(const T* __restrict__ x, size_t per_frame,
                                                     unsigned* __restrict__ stats) {
  const T* fx = x + (size_t)blockIdx.y * per_frame;
  KeyRange range;
#pragma unroll 4
  for (size_t i = blockIdx.x * (size_t)256 + threadIdx.x; i < per_frame; i += (size_t)gridDim.x * 256)
    range.add(to_double(fx[i]));
  range.commit(stats + (size_t)kFrameStats * blockIdx.y);
}

// Median of each frame's samples: the middle sample, or the mean of the two middle samples for an even
// count; NaN when a sample is NaN. A cluster of kMedCtas CTAs per frame narrows the key range that
// holds the (lower) middle sample: a pass counts the samples of the range in kMedBins equal bins of
// keys (each CTA its part, combined over distributed shared memory), the bin that holds the middle
// becomes the range, until at most kMedCap samples are left (or one key); a last pass collects those
// (and, where the upper middle sample lies above them, the smallest key above), and the first CTA
// ranks them. Most samples are settled by the high words of their keys. Two passes for samples spread over a
// binade or a few, against nine of an 8-bit radix select by one CTA per frame; bound by memory latency
// between the cluster's barriers (256 frames of 512 x 512 FP64: 1410 us by radix select, 280 us here).
constexpr int kMedCtas = 8, kMedThreads = 512, kMedBins = kMedCtas * kMedThreads, kMedCap = 1024;
template <class T>
__global__ void __cluster_dims__(kMedCtas, 1, 1) __launch_bounds__(kMedThreads)
    k_frame_median(const T* __restrict__ x, size_t per_frame, const unsigned* __restrict__ stats,
                   double* __restrict__ med) {
  namespace cg = cooperative_groups;
  using u64 = unsigned long long;
  __shared__ unsigned hist[kMedBins];
  __shared__ u64 s_buf[kMedCap];
  __shared__ unsigned s_warp[kMedThreads / 32];
  __shared__ unsigned s_total, s_n;
  __shared__ u64 s_pick[3];  // bin, samples below it, samples in it
  __shared__ u64 s_min[kMedThreads / 32];  // per warp: the smallest key above the range
  __shared__ u64 s_ab[2];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const size_t f = blockIdx.x / kMedCtas;
  const unsigned* st = stats + kFrameStats * f;
  if (st[2] == 0) {  // a NaN; uniform over the cluster
    if (rank == 0 && t == 0) med[f] = NAN;
    return;
  }
  const T* fx = x + f * per_frame;
  constexpr int V = 16 / sizeof(T);  // samples of a 16-byte load
  const size_t part = ((per_frame + kMedCtas - 1) / kMedCtas + V - 1) / V * V, a = min(per_frame, rank * part),
               e = min(per_frame, a + part);
  // every sample of this CTA's part; 16-byte loads, four in flight, where the frame allows
  const bool wide = reinterpret_cast<uintptr_t>(fx) % 16 == 0;
  auto each = [&](auto&& use) {
    size_t i0 = a;
    if (wide) {
      const size_t nv = (e - a) / V;
      const uint4* q = reinterpret_cast<const uint4*>(fx + a);
      for (size_t i = t; i < nv; i += 4 * kMedThreads) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (i + u * kMedThreads < nv) v[u] = q[i + u * kMedThreads];
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (i + u * kMedThreads < nv) {
            const T* s = reinterpret_cast<const T*>(&v[u]);
#pragma unroll
            for (int c = 0; c < V; c++) use(to_double(s[c]));
          }
      }
      i0 = a + nv * V;
    }
#pragma unroll 4
    for (size_t i = i0 + t; i < e; i += kMedThreads) use(to_double(fx[i]));
  };
  // whole high words: with a shift of 32 or more a sample's bin follows from its key's high word
  u64 lo = (u64)st[0] << 32, hi = ((u64)~st[1] << 32) | 0xFFFFFFFFu, k = (per_frame - 1) / 2, cnt = per_frame;
  bool all = true;  // every sample lies in the range
  if (t == 0) s_n = 0;
  while (cnt > kMedCap && lo < hi) {
    const int shift = max(0, 64 - __clzll((long long)(hi - lo)) - 12);
    static_assert(kMedBins == 1 << 12, "bins of the narrowing");
    for (int b = t; b < kMedBins; b += kMedThreads) hist[b] = 0;
    __syncthreads();
    const unsigned lo_h = (unsigned)(lo >> 32), span_h = (unsigned)(hi >> 32) - lo_h;
    if (all && shift >= 32) {
      each([&](double v) { atomicAdd(&hist[(fe_key_hi(v) - lo_h) >> (shift - 32)], 1u); });
    } else {
      each([&](double v) {
        if (fe_key_hi(v) - lo_h > span_h) return;
        const u64 key = fe_key(v);
        if (key >= lo && key <= hi) atomicAdd(&hist[(key - lo) >> shift], 1u);
      });
    }
    all = false;
    cluster.sync();
    // this CTA's slice of the bins over all CTAs, and its exclusive scan
    unsigned v = 0;
#pragma unroll
    for (int q = 0; q < kMedCtas; q++) v += cluster.map_shared_rank(hist, q)[rank * kMedThreads + t];
    unsigned inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    unsigned before = 0;
    for (int q = 0; q < warp; q++) before += s_warp[q];
    if (t == kMedThreads - 1) s_total = before + inc;
    cluster.sync();
    u64 base = 0;
    int owner = -1;
    u64 mine = 0;
    for (int q = 0; q < kMedCtas; q++) {
      const u64 n = *cluster.map_shared_rank(&s_total, q);
      if (q == rank) mine = base;
      if (owner < 0 && k < base + n) owner = q;
      base += n;
    }
    const u64 first = mine + before + inc - v;
    if (rank == owner && k >= first && k < first + v) {
      s_pick[0] = (u64)(rank * kMedThreads + t);
      s_pick[1] = first;
      s_pick[2] = v;
    }
    cluster.sync();
    const u64* pick = cluster.map_shared_rank(s_pick, owner);
    const u64 bin = pick[0];
    k -= pick[1];
    cnt = pick[2];
    lo += bin << shift;
    hi = min(hi, lo + ((1ull << shift) - 1));
    cluster.sync();  // the bins, totals and picks are rewritten by the next round
  }
  const bool even = (per_frame & 1) == 0, single = lo == hi;
  // the upper middle sample is another sample of the range, or the smallest key above it
  const bool above = even && k + 1 >= cnt;
  cluster.sync();  // s_n is set
  if (!single || above) {
    u64 mn = ~0ull;
    unsigned* n0 = cluster.map_shared_rank(&s_n, 0);
    u64* buf0 = cluster.map_shared_rank(s_buf, 0);
    const unsigned lo_h = (unsigned)(lo >> 32), span_h = (unsigned)(hi >> 32) - lo_h;
    each([&](double v) {
      if (!above && fe_key_hi(v) - lo_h > span_h) return;
      const u64 key = fe_key(v);
      if (key > hi) mn = key < mn ? key : mn;
      else if (!single && key >= lo) buf0[atomicAdd(n0, 1u)] = key;
    });
    for (int o = 16; o > 0; o >>= 1) {
      const u64 m2 = __shfl_xor_sync(0xffffffffu, mn, o);
      mn = m2 < mn ? m2 : mn;
    }
    if (lane == 0) s_min[warp] = mn;
  }
  cluster.sync();
  if (rank == 0 && above && warp == 0) {  // the CTAs' minima (no 64-bit atomics on distributed shared memory)
    u64 mn = ~0ull;
    for (int q = lane; q < kMedCtas * (kMedThreads / 32); q += 32) {
      const u64 v = cluster.map_shared_rank(s_min, q / (kMedThreads / 32))[q % (kMedThreads / 32)];
      mn = v < mn ? v : mn;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const u64 m2 = __shfl_xor_sync(0xffffffffu, mn, o);
      mn = m2 < mn ? m2 : mn;
    }
    if (lane == 0) s_ab[1] = mn;
  }
  cluster.sync();  // no CTA leaves while the first may still read its minima
  if (rank != 0) return;
  if (!single) {
    for (int q = t; q < (int)cnt; q += kMedThreads) {
      const u64 key = s_buf[q];
      u64 r = 0;
      for (int i = 0; i < (int)cnt; i++) r += (s_buf[i] < key || (s_buf[i] == key && i < q)) ? 1 : 0;
      if (r == k) s_ab[0] = key;
      if (r == k + 1) s_ab[1] = key;  // (with `above` there is none)
    }
    __syncthreads();
  }
  if (t == 0) {
    const double m0 = fe_unkey(single ? lo : s_ab[0]);
    const double m1 = fe_unkey(single && !above ? lo : s_ab[1]);
    med[f] = even ? (m0 + m1) / 2.0 : m0;
  }
}

// A sample as an entry of the block matrix, divided by the frame's median m where `div`.
template <class InT, class OutT>
__device__ __forceinline__ OutT fe_convert(InT x, bool div, double m) {
  if constexpr (!std::is_same<OutT, uint16_t>::value) {  // (uint16 entries are only ever copied)
    if (div) return (OutT)(to_double(x) / m);
  }
  if constexpr (std::is_same<InT, OutT>::value) return x;
  else return (OutT)to_double(x);
}

// Block matrices of frames: out (Hb x nb * n) entry (r, b + f nb) = frame f's cropped pixel
// gather[r + b Hb] (column-major in the cropped hc x wc frame; -1: 0), the cropped frame being rows
// [r0, r0 + hc) and columns [c0, c0 + wc) of the h x w frame. For maps without row structure
// (k_block_rows); the reads follow the map, the writes are coalesced. With med, every sample is divided
// by its frame's median.
template <class InT, class OutT>
__global__ void __launch_bounds__(256) k_block_gather(const void* __restrict__ in, OutT* __restrict__ out, int h, int w,
                                                      int n, int r0, int c0, int hc, const int* __restrict__ gather,
                                                      int hb, int nb, const double* __restrict__ med) {
  const size_t per = (size_t)hb * nb, total = per * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const size_t f = e / per;
    const int g = gather[e - f * per];
    OutT v = OutT(0);
    if (g >= 0) {
      const int ci = g % hc, cj = g / hc;
      const size_t src = f * (size_t)h * w + (size_t)(cj + c0) * h + (ci + r0);
      v = fe_convert<InT, OutT>(reinterpret_cast<const InT*>(in)[src], med != nullptr, med ? med[f] : 1.0);
    }
    out[e] = v;
  }
}

// Block matrices of a map whose blocks are runs of whole lines: block b holds the cropped rows
// [start[b], start[b + 1]), entry r being row r mod k_b of column r div k_b (k_b = start[b+1] -
// start[b]), zeros past column wc - 1. That is the reference's map of a scan with a whole number of
// lines per knot, and a transpose in memory: the frame is column-major along the lines, a block along
// the pixels. Bound: HBM, with instruction issue close behind for 16-bit samples. A CTA moves a tile
// of bt consecutive blocks (at most kRowTile rows) by kRowTile columns through shared memory, so that
// reads run down the columns (VE samples, 16 bytes, per thread where every tile's first row and column
// is aligned) and writes along the blocks (VO entries, 16 bytes, per thread where hb is a multiple of
// VO); reading the map's strided pixels directly used 4 of the 32 bytes of each sector. Tile column j
// starts at word j * pitch + j / 4: the 4 columns of a thread's 8 entries (2 lines per block) then
// fall into different banks across the warp. K > 0: every block has K lines and the index arithmetic
// is shifts and constants (the default scan's 1, 2 and 4 lines per knot). With med, every sample is
// divided by its frame's median. Grid: (block tiles, column tiles, frames).
constexpr int kRowTile = 64;
constexpr int kRowMaxLines = 32;  // longer runs are coalesced already in k_block_gather
template <class InT, class OutT, int VE, int VO, int K>
__global__ void __launch_bounds__(256) k_block_rows(const InT* __restrict__ in, OutT* __restrict__ out, int h, int w,
                                                    int r0, int c0, int wc, const int* __restrict__ start, int hb,
                                                    int nb, int bt, int slots, unsigned slots_inv,
                                                    const double* __restrict__ med) {
  constexpr int kWord = sizeof(InT) < 4 ? 4 / sizeof(InT) : 1;  // samples of a tile word
  constexpr int kPitch = kRowTile + kWord;                      // an odd number of words
  __shared__ __align__(16) InT tile[kRowTile * kPitch + (kRowTile / 4) * kWord];
  __shared__ int s_k[kRowTile], s_m[kRowTile], s_off[kRowTile];
  auto col = [](int j) { return j * kPitch + (j >> 2) * kWord; };
  const int b0 = blockIdx.x * bt, nbt = min(bt, nb - b0);
  const int j0 = blockIdx.y * kRowTile, nc = min(kRowTile, wc - j0);
  const size_t f = blockIdx.z;
  const int row0 = start[b0], rows = start[b0 + nbt] - row0;
  const InT* src = in + f * (size_t)h * w + (size_t)(j0 + c0) * h + (row0 + r0);
  constexpr int kVecs = kRowTile / VE;  // vectors of a tile column
#pragma unroll 4
  for (int idx = threadIdx.x; idx < nc * kVecs; idx += 256) {
    const int j = idx / kVecs, i = (idx % kVecs) * VE;
    if (i >= rows) continue;
    if constexpr (VE == 1) {
      tile[col(j) + i] = src[(size_t)j * h + i];
    } else if constexpr (sizeof(InT) == 8) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + (size_t)j * h + i));
      const InT* e = reinterpret_cast<const InT*>(&v);
#pragma unroll
      for (int q = 0; q < VE; q++) tile[col(j) + i + q] = e[q];
    } else {  // whole words
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + (size_t)j * h + i));
      uint32_t* t = reinterpret_cast<uint32_t*>(tile + col(j) + i);
      t[0] = v.x; t[1] = v.y; t[2] = v.z; t[3] = v.w;
    }
  }
  if (K == 0 && (int)threadIdx.x < nbt) {
    const int s = start[b0 + threadIdx.x], k = start[b0 + threadIdx.x + 1] - s;
    s_k[threadIdx.x] = k;
    s_m[threadIdx.x] = (65536 + k - 1) / k;  // e / k == (e * m) >> 16 for e < 64 * 32, k <= 32
    s_off[threadIdx.x] = s - row0;
  }
  __syncthreads();
  OutT* const fo = out + f * (size_t)hb * nb;
  const bool div = med != nullptr;
  const double dm = div ? med[f] : 1.0;
  auto cvt = [&](InT x) -> OutT { return fe_convert<InT, OutT>(x, div, dm); };
  // `slots` runs of VO entries per block, the thread's block idx / slots (by its rounded-up reciprocal)
  const int ns = K ? kRowTile * K / VO : slots;
#pragma unroll 2
  for (int idx = threadIdx.x; idx < nbt * ns; idx += 256) {
    const int bl = K ? idx / ns : (int)__umulhi((unsigned)idx, slots_inv), e0 = (idx - bl * ns) * VO;
    const int k = K ? K : s_k[bl], off = K ? bl * K : s_off[bl], left = nc * k - e0;
    if (left <= 0) continue;
    const int m = K ? 0 : s_m[bl];
    auto col_of = [&](int e) { return K ? e / k : (e * m) >> 16; };
    struct alignas(VO * sizeof(OutT)) Run { OutT v[VO]; } run;
    if (kWord == 2 && VO > 1 && ((k | off) & 1) == 0) {  // both lines of a pair of entries in one word
#pragma unroll
      for (int q = 0; q < VO; q += 2) {
        const int e = e0 + q, j = col_of(e);  // past the columns: stale tile entries, not stored
        const uint32_t wd = *reinterpret_cast<const uint32_t*>(tile + col(j) + off + (e - j * k));
        if constexpr (std::is_same<InT, OutT>::value && VO > 1) {
          reinterpret_cast<uint32_t*>(&run)[q / 2] = wd;
        } else {
          const InT* x = reinterpret_cast<const InT*>(&wd);
          run.v[q] = cvt(x[0]);
          run.v[q + 1 < VO ? q + 1 : q] = cvt(x[1]);
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < VO; q++) {
        const int e = e0 + q, j = col_of(e);
        run.v[q] = cvt(tile[col(j) + off + (e - j * k)]);
      }
    }
    OutT* o = fo + (size_t)(b0 + bl) * hb + (size_t)j0 * k + e0;
    if (left >= VO) {
      *reinterpret_cast<Run*>(o) = run;
    } else {
#pragma unroll
      for (int q = 0; q < VO; q++)
        if (q < left) o[q] = run.v[q];
    }
  }
  if (j0 + kRowTile >= wc)  // the block's last column tile: zeros past its pixels
    for (int bl = threadIdx.x >> 5; bl < nbt; bl += 8)
      for (int r = (K ? K : s_k[bl]) * wc + (threadIdx.x & 31); r < hb; r += 32) fo[(size_t)(b0 + bl) * hb + r] = OutT(0);
}

}  // namespace ss
