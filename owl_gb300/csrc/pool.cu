// pool.cu -- max / average pooling, forward and backward, 2-D and 3-D,
// float32, float64, complex32 and complex64, with Owl's exact semantics
// (src/owl/core/owl_ndarray_pool_impl.h):
//   * window scan order: cols outer, rows, dpts inner; out-of-range taps
//     skipped (:60-77, :282-300);
//   * max: accumulator starts at -inf, replaced only when `acc < t`, so the
//     first maximum in scan order wins and NaN is never selected (:20-23 of
//     owl_ndarray_pool_stub.c); argmax is the flat index into the whole input
//     (batch offset included), -1 when nothing was selected (:516-527);
//   * avg: sum in the element type, in scan order, divided by the in-range
//     count (:71-79);
//   * backward: max routes dY to the recomputed argmax with max_idx
//     starting at 0 (:167); avg adds dY / count to every in-range element
//     (:189-191); contributions accumulate with += in output (window) order.
//
// Layout: channels innermost, so every thread works on a vector of V
// consecutive channels (16-byte loads and stores when the channel count
// allows) and a warp covers a contiguous run of channels and pixels.
//
// Every thread walks its window in chunks of eight taps, issuing the eight
// vector loads before reducing them in scan order, so each thread keeps
// several loads in flight (a pooling kernel is bound by HBM latency x
// parallelism, not by arithmetic).  The reduction axis is the window, not
// the contiguous channel axis, so no cross-lane shuffle is needed: a warp's
// loads of one tap are one contiguous run of channels.
//
// Backward has two forms, both equal to Owl's zero-initialised `+=` scatter
// bit for bit and without atomics:
//   * windows that do not overlap (stride >= kernel in every dimension):
//     one thread per window recomputes its winner and writes each element
//     of the window's cell once (read X and dY once, write dX once);
//   * overlapping windows: a block owns a tile of input elements, computes
//     each window that touches it once (winner and dY, or dY / count) into
//     shared memory, and every element then adds the windows that contain it
//     in output order, the order of Owl's `+=` sequence.
// A max window in which no element beats -inf routes its gradient to flat
// element 0 in Owl; such windows are detected on the device and element 0
// is then rebuilt by an ordered fix-up pass.
#include "common.cuh"

#include <algorithm>
#include <atomic>
#include <type_traits>

namespace owlgpu {
namespace {

struct PG {
  int64_t B, IC, IR, ID, Ch, KC, KR, KD, OC, OR, OD;
  int sc, sr, sd, pc, pr, pd;
};

PG to_pg(const PoolGeom &g) {
  PG p{g.B, g.IC, g.IR, g.ID, g.Ch, g.KC, g.KR, g.KD, g.OC, g.OR, g.OD,
       g.sc, g.sr, g.sd, g.pc, g.pr, g.pd};
  return p;
}

// Unsigned 32-bit division by a divisor fixed for the whole launch, by one
// multiply-high, an add and a shift (Granlund & Montgomery, "Division by
// invariant integers using multiplication", PLDI 1994, round-up variant):
// with l = ceil(log2 d), m = floor(2^32 (2^l - d) / d) + 1,
// n / d = (umulhi(m, n) + n) >> l for every n < 2^31.
struct FastDiv {
  uint32_t d, m, l;
};

FastDiv make_fastdiv(uint32_t d) {
  uint32_t l = 0;
  while ((1ull << l) < d) ++l;
  const uint64_t m = (((1ull << l) - d) << 32) / d + 1;
  return FastDiv{d, (uint32_t)m, l};
}

__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv &f) {
  return (__umulhi(f.m, n) + n) >> f.l;
}

// Output index -> (b, oc, or, od, channel vector) with channel vectors
// innermost; valid while the output has fewer than 2^31 vectors.
struct OutDecode {
  FastDiv cv, od, orr, oc;
};

OutDecode make_out_decode(const PG &g, int64_t cv) {
  return OutDecode{make_fastdiv((uint32_t)cv), make_fastdiv((uint32_t)g.OD),
                   make_fastdiv((uint32_t)g.OR), make_fastdiv((uint32_t)g.OC)};
}

struct OutPos {
  uint32_t p, cv;  // output pixel and channel vector
  int b, oc, orr, od;
};

__device__ __forceinline__ OutPos out_pos(const OutDecode &dec, uint32_t idx) {
  OutPos o;
  o.p = fdiv(idx, dec.cv);
  o.cv = idx - o.p * dec.cv.d;
  const uint32_t t1 = fdiv(o.p, dec.od);
  o.od = (int)(o.p - t1 * dec.od.d);
  const uint32_t t2 = fdiv(t1, dec.orr);
  o.orr = (int)(t1 - t2 * dec.orr.d);
  const uint32_t t3 = fdiv(t2, dec.oc);
  o.oc = (int)(t2 - t3 * dec.oc.d);
  o.b = (int)t3;
  return o;
}

template <typename T, int V>
struct Vec;
template <>
struct Vec<float, 4> { using type = float4; };
template <>
struct Vec<float, 2> { using type = float2; };
template <>
struct Vec<float, 1> { using type = float; };
template <>
struct Vec<double, 2> { using type = double2; };
template <>
struct Vec<double, 1> { using type = double; };
template <>
struct Vec<c32, 2> { using type = float4; };
template <>
struct Vec<c32, 1> { using type = float2; };
template <>
struct Vec<c64, 1> { using type = double2; };

template <typename T, int V>
__device__ __forceinline__ void load_vec(const T *p, T (&v)[V]) {
  using VT = typename Vec<T, V>::type;
  VT t = __ldg(reinterpret_cast<const VT *>(p));
  const T *e = reinterpret_cast<const T *>(&t);
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = e[i];
}

template <typename T, int V>
__device__ __forceinline__ void store_vec(T *p, const T (&v)[V]) {
  using VT = typename Vec<T, V>::type;
  VT t;
  T *e = reinterpret_cast<T *>(&t);
#pragma unroll
  for (int i = 0; i < V; ++i) e[i] = v[i];
  *reinterpret_cast<VT *>(p) = t;
}

// ---- window walking ------------------------------------------------------

// In-range part of one window: [c0,c1) x [r0,r1) x [d0,d1); n taps.
struct Box {
  int c0, c1, r0, r1, d0, d1, nr, nd, n;
};

__device__ __forceinline__ Box window_box(const PG &g, int oc, int orr, int od) {
  Box w;
  const int cs = oc * g.sc - g.pc, rs = orr * g.sr - g.pr, ds = od * g.sd - g.pd;
  w.c0 = max(cs, 0); w.c1 = min(cs + (int)g.KC, (int)g.IC);
  w.r0 = max(rs, 0); w.r1 = min(rs + (int)g.KR, (int)g.IR);
  w.d0 = max(ds, 0); w.d1 = min(ds + (int)g.KD, (int)g.ID);
  const int nc = max(w.c1 - w.c0, 0);
  w.nr = max(w.r1 - w.r0, 0);
  w.nd = max(w.d1 - w.d0, 0);
  w.n = nc * w.nr * w.nd;
  return w;
}

// Walks a window's taps in Owl's scan order (cols, rows, dpts) U at a time:
// all U loads of a chunk are issued before any is used, so a thread keeps U
// vector loads in flight instead of one.
struct Cursor {
  int a, b, c;
};

template <typename T, int V, int U>
__device__ __forceinline__ void load_chunk(const T *__restrict__ x, int64_t base, const PG &g,
                                           const Box &w, Cursor &cur, int left,
                                           T (&v)[U][V]) {
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (u < left) {
      load_vec<T, V>(x + base + (((int64_t)cur.a * g.IR + cur.b) * g.ID + cur.c) * g.Ch, v[u]);
      if (++cur.c == w.d1) {
        cur.c = w.d0;
        if (++cur.b == w.r1) { cur.b = w.r0; ++cur.a; }
      }
    }
  }
}

// Max over the window with Owl's strict `<` (first maximum wins, NaN never
// selected); bt = tap index of the winner in scan order, -1 if none.
template <typename T, int V, int U>
__device__ __forceinline__ void window_max(const T *__restrict__ x, int64_t base, const PG &g,
                                           const Box &w, T (&best)[V], int (&bt)[V]) {
#pragma unroll
  for (int i = 0; i < V; ++i) { best[i] = T(-INFINITY); bt[i] = -1; }
  Cursor cur{w.c0, w.r0, w.d0};
  for (int t0 = 0; t0 < w.n; t0 += U) {
    T v[U][V];
    load_chunk<T, V, U>(x, base, g, w, cur, w.n - t0, v);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < w.n - t0) {
#pragma unroll
        for (int i = 0; i < V; ++i)
          if (best[i] < v[u][i]) { best[i] = v[u][i]; bt[i] = t0 + u; }
      }
  }
}

// Sum over the window in scan order, in the element type.
template <typename T, int V, int U>
__device__ __forceinline__ void window_sum(const T *__restrict__ x, int64_t base, const PG &g,
                                           const Box &w, T (&acc)[V]) {
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = T(0);
  Cursor cur{w.c0, w.r0, w.d0};
  for (int t0 = 0; t0 < w.n; t0 += U) {
    T v[U][V];
    load_chunk<T, V, U>(x, base, g, w, cur, w.n - t0, v);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < w.n - t0) {
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] += v[u][i];
      }
  }
}

// Flat input offset (without the channel) of tap t of window w.
__device__ __forceinline__ int64_t tap_offset(const PG &g, int64_t xbase, const Box &w, int t) {
  const int per_c = w.nr * w.nd;
  const int a = w.c0 + t / per_c, rem = t % per_c;
  const int b = w.r0 + rem / w.nd, c = w.d0 + rem % w.nd;
  return xbase + (((int64_t)a * g.IR + b) * g.ID + c) * g.Ch;
}

constexpr int kChunk = 8;

// ---- forward --------------------------------------------------------------

template <typename T, int V, int MODE, bool ARG>
__global__ void __launch_bounds__(256) pool_fwd_kernel(PG g, const T *__restrict__ x,
                                                       T *__restrict__ y,
                                                       int64_t *__restrict__ argmax) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  const int64_t CV = g.Ch / V;
  const int64_t total = g.B * g.OC * g.OR * g.OD * CV;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t cv = idx % CV, p = idx / CV;
    const int od = (int)(p % g.OD);
    int64_t t = p / g.OD;
    const int orr = (int)(t % g.OR); t /= g.OR;
    const int oc = (int)(t % g.OC);
    const int64_t b = t / g.OC;
    const int64_t xbase = b * g.IC * g.IR * g.ID * g.Ch;
    const Box w = window_box(g, oc, orr, od);
    T out[V];
    if (MODE == POOL_MAX) {
      int bt[V];
      window_max<T, V, kChunk>(x, xbase + cv * V, g, w, out, bt);
      if (ARG) {
#pragma unroll
        for (int i = 0; i < V; ++i)
          argmax[p * g.Ch + cv * V + i] =
              bt[i] < 0 ? -1 : tap_offset(g, xbase, w, bt[i]) + cv * V + i;
      }
    } else {
      window_sum<T, V, kChunk>(x, xbase + cv * V, g, w, out);
#pragma unroll
      for (int i = 0; i < V; ++i) out[i] = div_count(out[i], w.n);
    }
    store_vec<T, V>(y + p * g.Ch + cv * V, out);
  }
}

// ---- degenerate max windows ------------------------------------------------

// A max window in which no element beats -inf (all -inf/NaN, or no in-range
// element) routes its gradient to flat element 0 in Owl.  Kernels that meet
// one raise this device-wide mark to their call's ticket with atomicMax; the
// fix-up kernel of a call runs when the mark is at or above its own ticket.
// Tickets grow monotonically, so a call never misses its own mark; a later
// call's mark can only make an earlier call redo the (always exact) ordered
// rebuild of dX[0].  No per-call memory is needed.
__device__ unsigned long long g_degenerate_mark = 0;
std::atomic<unsigned long long> g_ticket{0};

__device__ __forceinline__ void raise_mark(unsigned long long ticket) {
  atomicMax(&g_degenerate_mark, ticket);
}

// ---- backward, non-overlapping windows (scatter form) ---------------------

// Per-dimension part of the input owned by output position o when s >= k:
// [o*s - p, (o+1)*s - p) clipped to [0, I), the last position taking the
// tail up to I.  These ranges partition [0, I) and each contains its window.
__device__ __forceinline__ void cell_range(int o, int s, int p, int64_t O, int64_t I, int &lo,
                                           int &hi) {
  lo = min(max(o * s - p, 0), (int)I);
  hi = o == (int)O - 1 ? (int)I : min(max((o + 1) * s - p, 0), (int)I);
}

// One thread per (window, channel vector): recompute the window's maximum
// (or its count), then write every element of the window's cell exactly
// once: 0 + dY at the winner, 0 + dY/count for average, 0 elsewhere.  With
// s >= k every input element lies in at most one window, so this equals
// Owl's zero-initialised `+=` scatter bit for bit.
template <typename T, int V, int MODE>
__global__ void __launch_bounds__(256) pool_bwd_cell_kernel(PG g, const T *__restrict__ x,
                                                            const T *__restrict__ dy,
                                                            T *__restrict__ dx,
                                                            unsigned long long ticket) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  const int64_t CV = g.Ch / V;
  const int64_t total = g.B * g.OC * g.OR * g.OD * CV;
  bool degen = false;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t cv = idx % CV, p = idx / CV;
    const int od = (int)(p % g.OD);
    int64_t t = p / g.OD;
    const int orr = (int)(t % g.OR); t /= g.OR;
    const int oc = (int)(t % g.OC);
    const int64_t b = t / g.OC;
    const int64_t xbase = b * g.IC * g.IR * g.ID * g.Ch;
    const Box w = window_box(g, oc, orr, od);
    T gv[V];
    load_vec<T, V>(dy + p * g.Ch + cv * V, gv);
    int bt[V];
    if (MODE == POOL_MAX) {
      T best[V];
      window_max<T, V, kChunk>(x, xbase + cv * V, g, w, best, bt);
#pragma unroll
      for (int i = 0; i < V; ++i) degen |= bt[i] < 0;
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) gv[i] = div_count(gv[i], w.n);
    }
    int alo, ahi, blo, bhi, clo, chi;
    cell_range(oc, g.sc, g.pc, g.OC, g.IC, alo, ahi);
    cell_range(orr, g.sr, g.pr, g.OR, g.IR, blo, bhi);
    cell_range(od, g.sd, g.pd, g.OD, g.ID, clo, chi);
    for (int a = alo; a < ahi; ++a)
      for (int bb = blo; bb < bhi; ++bb)
        for (int c = clo; c < chi; ++c) {
          const bool in = a >= w.c0 && a < w.c1 && bb >= w.r0 && bb < w.r1 && c >= w.d0 &&
                          c < w.d1;
          const int tap = ((a - w.c0) * w.nr + (bb - w.r0)) * w.nd + (c - w.d0);
          T o[V];
#pragma unroll
          for (int i = 0; i < V; ++i) {
            if (MODE == POOL_MAX) o[i] = in && tap == bt[i] ? T(0) + gv[i] : T(0);
            else o[i] = in ? T(0) + gv[i] : T(0);
          }
          store_vec<T, V>(dx + xbase + (((int64_t)a * g.IR + bb) * g.ID + c) * g.Ch + cv * V, o);
        }
  }
  if (MODE == POOL_MAX && degen) raise_mark(ticket);
}

// ---- fixed-window fast paths ----------------------------------------------

// Windows of compile-time size KC x KR x KD: a window wholly inside the input
// has its taps constant strides apart and loads them all before the
// reduction; one that the border clips (SAME padding) walks its in-range taps
// as the general kernel does.  Same scan order and comparisons either way.
// HBM-bound.  3x3 stride 2 SAME on [16;112;112;64] (64 MB): 22.6 us when its
// clipped windows sent every window to the general kernel, 13.8 us here.
template <typename T, int V, int KC, int KR, int KD, int MODE, bool ARG>
__global__ void __launch_bounds__(256) pool_fwd_fixed_kernel(PG g, OutDecode dec,
                                                             const T *__restrict__ x,
                                                             T *__restrict__ y,
                                                             int64_t *__restrict__ argmax) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  constexpr int N = KC * KR * KD;
  const uint32_t total = (uint32_t)(g.B * g.OC * g.OR * g.OD * (g.Ch / V));
  const int64_t sd = g.Ch, sr = g.ID * g.Ch, sc = g.IR * g.ID * g.Ch;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += gridDim.x * blockDim.x) {
    const OutPos o = out_pos(dec, idx);
    const int64_t cv = o.cv, p = o.p;
    const int c0 = o.oc * g.sc - g.pc, r0 = o.orr * g.sr - g.pr, d0 = o.od * g.sd - g.pd;
    const int64_t xbase = (int64_t)o.b * g.IC * sc;
    T out[V];
    int bt[V];
    if (c0 >= 0 && c0 + KC <= g.IC && r0 >= 0 && r0 + KR <= g.IR && d0 >= 0 &&
        d0 + KD <= g.ID) {
      const int64_t base = xbase + c0 * sc + r0 * sr + d0 * sd + cv * V;
      T v[N][V];
#pragma unroll
      for (int a = 0; a < KC; ++a)
#pragma unroll
        for (int bb = 0; bb < KR; ++bb)
#pragma unroll
          for (int c = 0; c < KD; ++c)
            load_vec<T, V>(x + base + a * sc + bb * sr + c * sd, v[(a * KR + bb) * KD + c]);
      if (MODE == POOL_MAX) {
#pragma unroll
        for (int i = 0; i < V; ++i) { out[i] = T(-INFINITY); bt[i] = -1; }
#pragma unroll
        for (int u = 0; u < N; ++u)
#pragma unroll
          for (int i = 0; i < V; ++i)
            if (out[i] < v[u][i]) { out[i] = v[u][i]; bt[i] = u; }
        if (ARG) {
#pragma unroll
          for (int i = 0; i < V; ++i) {
            const int a = bt[i] / (KR * KD), bb = bt[i] / KD % KR, c = bt[i] % KD;
            argmax[p * g.Ch + cv * V + i] =
                bt[i] < 0 ? -1 : base + a * sc + bb * sr + c * sd + i;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < V; ++i) out[i] = T(0);
#pragma unroll
        for (int u = 0; u < N; ++u)
#pragma unroll
          for (int i = 0; i < V; ++i) out[i] += v[u][i];
#pragma unroll
        for (int i = 0; i < V; ++i) out[i] = div_count(out[i], N);
      }
    } else {
      const Box w = window_box(g, o.oc, o.orr, o.od);
      if (MODE == POOL_MAX) {
        window_max<T, V, 1>(x, xbase + cv * V, g, w, out, bt);
        if (ARG) {
#pragma unroll
          for (int i = 0; i < V; ++i)
            argmax[p * g.Ch + cv * V + i] =
                bt[i] < 0 ? -1 : tap_offset(g, xbase, w, bt[i]) + cv * V + i;
        }
      } else {
        window_sum<T, V, 1>(x, xbase + cv * V, g, w, out);
#pragma unroll
        for (int i = 0; i < V; ++i) out[i] = div_count(out[i], w.n);
      }
    }
    store_vec<T, V>(y + p * g.Ch + cv * V, out);
  }
}

// Backward for windows that tile the input exactly (stride = kernel, no
// padding, O*s = I): each window is its own cell.
template <typename T, int V, int KC, int KR, int KD, int MODE>
__global__ void __launch_bounds__(256) pool_bwd_tile_kernel(PG g, OutDecode dec,
                                                            const T *__restrict__ x,
                                                            const T *__restrict__ dy,
                                                            T *__restrict__ dx,
                                                            unsigned long long ticket) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  constexpr int N = KC * KR * KD;
  const uint32_t total = (uint32_t)(g.B * g.OC * g.OR * g.OD * (g.Ch / V));
  const int64_t sd = g.Ch, sr = g.ID * g.Ch, sc = g.IR * g.ID * g.Ch;
  bool degen = false;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += gridDim.x * blockDim.x) {
    const OutPos o = out_pos(dec, idx);
    const int64_t cv = o.cv, p = o.p;
    const int64_t base = (int64_t)o.b * g.IC * sc + (int64_t)o.oc * KC * sc +
                         (int64_t)o.orr * KR * sr + (int64_t)o.od * KD * sd + cv * V;
    T gv[V];
    load_vec<T, V>(dy + p * g.Ch + cv * V, gv);
    int bt[V];
    if (MODE == POOL_MAX) {
      T v[N][V];
#pragma unroll
      for (int a = 0; a < KC; ++a)
#pragma unroll
        for (int bb = 0; bb < KR; ++bb)
#pragma unroll
          for (int c = 0; c < KD; ++c)
            load_vec<T, V>(x + base + a * sc + bb * sr + c * sd, v[(a * KR + bb) * KD + c]);
      T best[V];
#pragma unroll
      for (int i = 0; i < V; ++i) { best[i] = T(-INFINITY); bt[i] = -1; }
#pragma unroll
      for (int u = 0; u < N; ++u)
#pragma unroll
        for (int i = 0; i < V; ++i)
          if (best[i] < v[u][i]) { best[i] = v[u][i]; bt[i] = u; }
#pragma unroll
      for (int i = 0; i < V; ++i) degen |= bt[i] < 0;
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) gv[i] = div_count(gv[i], N);
    }
#pragma unroll
    for (int a = 0; a < KC; ++a)
#pragma unroll
      for (int bb = 0; bb < KR; ++bb)
#pragma unroll
        for (int c = 0; c < KD; ++c) {
          const int u = (a * KR + bb) * KD + c;
          T o[V];
#pragma unroll
          for (int i = 0; i < V; ++i) {
            if (MODE == POOL_MAX) o[i] = bt[i] == u ? T(0) + gv[i] : T(0);
            else o[i] = T(0) + gv[i];
          }
          store_vec<T, V>(dx + base + a * sc + bb * sr + c * sd, o);
        }
  }
  if (MODE == POOL_MAX && degen) raise_mark(ticket);
}

// ---- backward, overlapping windows (gather form) ---------------------------

// Range of output positions o whose window [o*s - p, o*s - p + k) contains i.
__device__ __forceinline__ void win_range(int i, int s, int p, int k, int64_t O, int &lo,
                                          int &hi) {
  // o*s <= i + p  and  o*s > i + p - k
  int num = i + p - k + 1;  // o >= ceil(num / s)
  lo = num <= 0 ? 0 : (num + s - 1) / s;
  int top = i + p;  // o <= floor(top / s)
  hi = top < 0 ? -1 : top / s;
  if (hi > (int)O - 1) hi = (int)O - 1;
}

// One thread per input element (vector): visit the windows that contain it
// in output order, the order in which Owl's scatter loop adds their
// contributions, so the float sum is Owl's `+=` sequence without atomics.
template <typename T, int V, int MODE>
__global__ void __launch_bounds__(256) pool_bwd_gather_kernel(PG g, const T *__restrict__ x,
                                                              const T *__restrict__ dy,
                                                              T *__restrict__ dx,
                                                              unsigned long long ticket) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  const int64_t CV = g.Ch / V;
  const int64_t total = g.B * g.IC * g.IR * g.ID * CV;
  bool degen = false;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t cv = idx % CV, p = idx / CV;
    const int id = (int)(p % g.ID);
    int64_t t = p / g.ID;
    const int ir = (int)(t % g.IR); t /= g.IR;
    const int ic = (int)(t % g.IC);
    const int64_t b = t / g.IC;
    const int64_t xbase = b * g.IC * g.IR * g.ID * g.Ch;
    const int64_t ybase = b * g.OC * g.OR * g.OD * g.Ch;
    int oc0, oc1, or0, or1, od0, od1;
    win_range(ic, g.sc, g.pc, (int)g.KC, g.OC, oc0, oc1);
    win_range(ir, g.sr, g.pr, (int)g.KR, g.OR, or0, or1);
    win_range(id, g.sd, g.pd, (int)g.KD, g.OD, od0, od1);
    T acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = T(0);
    for (int oc = oc0; oc <= oc1; ++oc)
      for (int orr = or0; orr <= or1; ++orr)
        for (int od = od0; od <= od1; ++od) {
          const Box w = window_box(g, oc, orr, od);
          T gv[V];
          load_vec<T, V>(dy + ybase + (((int64_t)oc * g.OR + orr) * g.OD + od) * g.Ch + cv * V,
                         gv);
          if (MODE == POOL_AVG) {
#pragma unroll
            for (int i = 0; i < V; ++i) acc[i] += div_count(gv[i], w.n);
          } else {
            T best[V];
            int bt[V];
            window_max<T, V, kChunk>(x, xbase + cv * V, g, w, best, bt);
            const int mine = ((ic - w.c0) * w.nr + (ir - w.r0)) * w.nd + (id - w.d0);
#pragma unroll
            for (int i = 0; i < V; ++i) {
              if (bt[i] < 0) degen = true;
              else if (bt[i] == mine) acc[i] += gv[i];
            }
          }
        }
    store_vec<T, V>(dx + xbase + (((int64_t)ic * g.IR + ir) * g.ID + id) * g.Ch + cv * V, acc);
  }
  if (MODE == POOL_MAX && degen) raise_mark(ticket);
}

// The tile of an overlapping backward: TC x TR x TD input elements (powers of
// two) by CVB channel vectors; at most NWC x NWR x NWD windows touch it.
struct OverTile {
  int lc, lr, ld;          // log2 of the tile's extents
  int CVB, n_cb;           // channel vectors per block, blocks of them
  int n_c, n_r, n_d;       // tiles along each axis
  int NWR, NWD, NW;        // window box of a tile (rows, dpts; all)
  FastDiv nwr, nwd, cvb;
  FastDiv sc, sr, sd;      // strides
};

// First and last window (output position) of one axis that covers any input
// position of [i0, i1); s > 0.
__device__ __forceinline__ void tile_windows(int i0, int i1, const FastDiv &s, int p, int k,
                                             int O, int &lo, int &hi) {
  const int num = i0 + p - k + 1;
  lo = num <= 0 ? 0 : (int)fdiv((uint32_t)num + s.d - 1, s);
  const int top = i1 - 1 + p;
  hi = top < 0 ? -1 : min((int)fdiv((uint32_t)top, s), O - 1);
}

// Backward with overlapping windows.  One block owns a tile of input elements
// of one batch entry and a run of channel vectors.  Phase 1 computes every
// window that touches the tile once: its winning tap (one byte a channel) and
// dY for max, dY / count for average, both into shared memory.  Phase 2 visits
// for each element the windows that contain it in output order, as Owl's
// scatter loop adds them, so the float sum is Owl's `+=` sequence without
// atomics.  Bound: HBM (x, dy, dx once) plus L1 re-reads of x, k/s windows an
// axis.  Recomputing each window once per element it contains (one thread per
// element, no tile) took 315 us (max) and 80 us (average) for 3x3 stride 2 on
// [16;112;112;64]; with the tiles 65 and 43 us, and with the compile-time windows
// of the next kernel 31.5 and 16.0 us (HBM floor 17 and 9.5).
template <typename T, int V, int MODE>
__global__ void __launch_bounds__(256) pool_bwd_over_kernel(PG g, OverTile tl,
                                                            const T *__restrict__ x,
                                                            const T *__restrict__ dy,
                                                            T *__restrict__ dx,
                                                            unsigned long long ticket) {
  extern __shared__ __align__(16) unsigned char over_smem[];
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  T *gbuf = reinterpret_cast<T *>(over_smem);                  // [NW][CVB][V]
  uint8_t *code = over_smem + (size_t)tl.NW * tl.CVB * V * sizeof(T);  // [NW][CVB][V]
  // block -> (batch, tile, channel block); channel blocks innermost
  unsigned q = blockIdx.x;
  const int cb = (int)(q % tl.n_cb); q /= tl.n_cb;
  const int td = (int)(q % tl.n_d); q /= tl.n_d;
  const int tr = (int)(q % tl.n_r); q /= tl.n_r;
  const int tc = (int)(q % tl.n_c);
  const int64_t b = q / tl.n_c;
  const int i0c = tc << tl.lc, i0r = tr << tl.lr, i0d = td << tl.ld;
  const int i1c = min(i0c + (1 << tl.lc), (int)g.IC), i1r = min(i0r + (1 << tl.lr), (int)g.IR),
            i1d = min(i0d + (1 << tl.ld), (int)g.ID);
  const int CV = (int)(g.Ch / V);
  const int cv0 = cb * tl.CVB, ncv = min(tl.CVB, CV - cv0);
  const int64_t xbase = b * g.IC * g.IR * g.ID * g.Ch, ybase = b * g.OC * g.OR * g.OD * g.Ch;
  int wc0, wc1, wr0, wr1, wd0, wd1;
  tile_windows(i0c, i1c, tl.sc, g.pc, (int)g.KC, (int)g.OC, wc0, wc1);
  tile_windows(i0r, i1r, tl.sr, g.pr, (int)g.KR, (int)g.OR, wr0, wr1);
  tile_windows(i0d, i1d, tl.sd, g.pd, (int)g.KD, (int)g.OD, wd0, wd1);
  // threads: lane cv within the block's channel vectors, groups over windows
  const int grp = (int)fdiv(threadIdx.x, tl.cvb), cvl = (int)threadIdx.x - grp * tl.CVB;
  const int n_grp = (int)fdiv(blockDim.x, tl.cvb);
  const bool on = grp < n_grp && cvl < ncv;
  bool degen = false;
  if (on) {
    for (int w = grp; w < tl.NW; w += n_grp) {
      const int t = (int)fdiv((uint32_t)w, tl.nwd), kd = w - t * tl.NWD;
      const int kc = (int)fdiv((uint32_t)t, tl.nwr), kr = t - kc * tl.NWR;
      const int oc = wc0 + kc, orr = wr0 + kr, od = wd0 + kd;
      if (oc > wc1 || orr > wr1 || od > wd1) continue;
      const Box wb = window_box(g, oc, orr, od);
      T gv[V];
      load_vec<T, V>(dy + ybase + (((int64_t)oc * g.OR + orr) * g.OD + od) * g.Ch +
                         (int64_t)(cv0 + cvl) * V, gv);
      const int at = (w * tl.CVB + cvl) * V;
      if (MODE == POOL_MAX) {
        T best[V];
        int bt[V];
        window_max<T, V, kChunk + 1>(x, xbase + (int64_t)(cv0 + cvl) * V, g, wb, best, bt);
#pragma unroll
        for (int i = 0; i < V; ++i) {
          degen |= bt[i] < 0;
          code[at + i] = bt[i] < 0 ? 255 : (uint8_t)bt[i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < V; ++i) gv[i] = div_count(gv[i], wb.n);
      }
      store_vec<T, V>(gbuf + at, gv);
    }
  }
  if (MODE == POOL_MAX && degen) raise_mark(ticket);
  __syncthreads();
  if (!on) return;
  const int ne = 1 << (tl.lc + tl.lr + tl.ld);
  for (int e = grp; e < ne; e += n_grp) {
    const int id = i0d + (e & ((1 << tl.ld) - 1));
    const int ir = i0r + ((e >> tl.ld) & ((1 << tl.lr) - 1));
    const int ic = i0c + (e >> (tl.ld + tl.lr));
    if (ic >= i1c || ir >= i1r || id >= i1d) continue;
    int oc0, oc1, or0, or1, od0, od1;
    tile_windows(ic, ic + 1, tl.sc, g.pc, (int)g.KC, (int)g.OC, oc0, oc1);
    tile_windows(ir, ir + 1, tl.sr, g.pr, (int)g.KR, (int)g.OR, or0, or1);
    tile_windows(id, id + 1, tl.sd, g.pd, (int)g.KD, (int)g.OD, od0, od1);
    T acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = T(0);
    for (int oc = oc0; oc <= oc1; ++oc) {
      const int cs = max(oc * g.sc - g.pc, 0);
      for (int orr = or0; orr <= or1; ++orr) {
        const int rs = orr * g.sr - g.pr;
        const int r0 = max(rs, 0), nr = min(rs + (int)g.KR, (int)g.IR) - r0;
        for (int od = od0; od <= od1; ++od) {
          const int at = ((((oc - wc0) * tl.NWR + (orr - wr0)) * tl.NWD + (od - wd0)) * tl.CVB +
                          cvl) * V;
          T gv[V];
#pragma unroll
          for (int i = 0; i < V; ++i) gv[i] = gbuf[at + i];
          if (MODE == POOL_AVG) {
#pragma unroll
            for (int i = 0; i < V; ++i) acc[i] += gv[i];
          } else {
            const int ds = od * g.sd - g.pd;
            const int d0 = max(ds, 0), nd = min(ds + (int)g.KD, (int)g.ID) - d0;
            const int mine = ((ic - cs) * nr + (ir - r0)) * nd + (id - d0);
#pragma unroll
            for (int i = 0; i < V; ++i)
              if (code[at + i] == mine) acc[i] += gv[i];
          }
        }
      }
    }
    store_vec<T, V>(dx + xbase + (((int64_t)ic * g.IR + ir) * g.ID + id) * g.Ch +
                        (int64_t)(cv0 + cvl) * V, acc);
  }
}

// The same for compile-time windows K and strides S: input positions come in
// blocks of S an axis (i + p = a*S + j), and the D + 1 windows a-D .. a, D =
// (K-1)/S, are the ones that touch block a, element j lying in window a-d when
// j + d*S < K.  A thread of phase 2 reads its block's windows once from shared
// memory for all the block's elements, with no division and no per-element
// window range: 3x3 stride 2 on [16;112;112;64] 31.5 us (max) and 16.0 us (average)
// against 65 and 43 in the runtime-window kernel above.  Codes number the whole
// window's taps (clipped ones too).
template <typename T, int V, int KC, int KR, int KD, int SC, int SR, int SD, int MODE>
__global__ void __launch_bounds__(256) pool_bwd_over_fixed_kernel(PG g, OverTile tl,
                                                                  const T *__restrict__ x,
                                                                  const T *__restrict__ dy,
                                                                  T *__restrict__ dx,
                                                                  unsigned long long ticket) {
  extern __shared__ __align__(16) unsigned char over_smem[];
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  constexpr int DC = (KC - 1) / SC, DR = (KR - 1) / SR, DD = (KD - 1) / SD;
  constexpr int N = KC * KR * KD;
  static_assert(N < 255 && V == 4, "byte codes, four to a word");
  T *gbuf = reinterpret_cast<T *>(over_smem);  // [NW][CVB][V]
  uint32_t *code = reinterpret_cast<uint32_t *>(over_smem + (size_t)tl.NW * tl.CVB * V * sizeof(T));
  unsigned q = blockIdx.x;
  const int cb = (int)(q % tl.n_cb); q /= tl.n_cb;
  const int td = (int)(q % tl.n_d); q /= tl.n_d;
  const int tr = (int)(q % tl.n_r); q /= tl.n_r;
  const int tc = (int)(q % tl.n_c);
  const int64_t b = q / tl.n_c;
  const int a0c = tc << tl.lc, a0r = tr << tl.lr, a0d = td << tl.ld;  // first blocks of the tile
  const int cv0 = cb * tl.CVB, ncv = min(tl.CVB, (int)(g.Ch / V) - cv0);
  const int64_t sd = g.Ch, sr = g.ID * g.Ch, sc = g.IR * g.ID * g.Ch;
  const int64_t xbase = b * g.IC * sc, ybase = b * g.OC * g.OR * g.OD * g.Ch;
  const int grp = (int)fdiv(threadIdx.x, tl.cvb), cvl = (int)threadIdx.x - grp * tl.CVB;
  const int n_grp = (int)fdiv(blockDim.x, tl.cvb);
  const bool on = grp < n_grp && cvl < ncv;
  const int64_t ch = (int64_t)(cv0 + cvl) * V;
  bool degen = false;
  if (on) {
    for (int w = grp; w < tl.NW; w += n_grp) {
      const int t = (int)fdiv((uint32_t)w, tl.nwd), kd = w - t * tl.NWD;
      const int kc = (int)fdiv((uint32_t)t, tl.nwr), kr = t - kc * tl.NWR;
      const int oc = a0c - DC + kc, orr = a0r - DR + kr, od = a0d - DD + kd;
      const int at = w * tl.CVB + cvl;
      if ((unsigned)oc >= (unsigned)g.OC || (unsigned)orr >= (unsigned)g.OR ||
          (unsigned)od >= (unsigned)g.OD) {
        // no such window: a code that no tap has, and dY / count zero for
        // average (skipped in phase 2 by the same test)
        if (MODE == POOL_MAX) code[at] = 0xffffffffu;
        continue;
      }
      T gv[V];
      load_vec<T, V>(dy + ybase + (((int64_t)oc * g.OR + orr) * g.OD + od) * g.Ch + ch, gv);
      const int c0 = oc * SC - g.pc, r0 = orr * SR - g.pr, d0 = od * SD - g.pd;
      const bool full = c0 >= 0 && c0 + KC <= g.IC && r0 >= 0 && r0 + KR <= g.IR && d0 >= 0 &&
                        d0 + KD <= g.ID;
      if (MODE == POOL_MAX) {
        T best[V];
        int bt[V];
#pragma unroll
        for (int i = 0; i < V; ++i) { best[i] = T(-INFINITY); bt[i] = 255; }
        const T *xw = x + xbase + c0 * sc + r0 * sr + d0 * sd + ch;
        if (full) {
          T v[N][V];
#pragma unroll
          for (int a = 0; a < KC; ++a)
#pragma unroll
            for (int bb = 0; bb < KR; ++bb)
#pragma unroll
              for (int c = 0; c < KD; ++c)
                load_vec<T, V>(xw + a * sc + bb * sr + c * sd, v[(a * KR + bb) * KD + c]);
#pragma unroll
          for (int u = 0; u < N; ++u)
#pragma unroll
            for (int i = 0; i < V; ++i)
              if (best[i] < v[u][i]) { best[i] = v[u][i]; bt[i] = u; }
        } else {
          for (int a = 0; a < KC; ++a)
            for (int bb = 0; bb < KR; ++bb)
              for (int c = 0; c < KD; ++c) {
                if ((unsigned)(c0 + a) >= (unsigned)g.IC || (unsigned)(r0 + bb) >= (unsigned)g.IR ||
                    (unsigned)(d0 + c) >= (unsigned)g.ID)
                  continue;
                T v[V];
                load_vec<T, V>(xw + a * sc + bb * sr + c * sd, v);
#pragma unroll
                for (int i = 0; i < V; ++i)
                  if (best[i] < v[i]) { best[i] = v[i]; bt[i] = (a * KR + bb) * KD + c; }
              }
        }
        uint32_t word = 0;
#pragma unroll
        for (int i = 0; i < V; ++i) {
          degen |= bt[i] == 255;
          word |= (uint32_t)bt[i] << (8 * i);
        }
        code[at] = word;
      } else {
        int n = N;
        if (!full) n = window_box(g, oc, orr, od).n;
#pragma unroll
        for (int i = 0; i < V; ++i) gv[i] = div_count(gv[i], n);
      }
      store_vec<T, V>(gbuf + (size_t)at * V, gv);
    }
  }
  if (MODE == POOL_MAX && degen) raise_mark(ticket);
  __syncthreads();
  if (!on) return;
  const int nblk = 1 << (tl.lc + tl.lr + tl.ld);
  for (int e = grp; e < nblk; e += n_grp) {
    const int bd = e & ((1 << tl.ld) - 1), br = (e >> tl.ld) & ((1 << tl.lr) - 1),
              bc = e >> (tl.ld + tl.lr);
    const int ic0 = (a0c + bc) * SC - g.pc, ir0 = (a0r + br) * SR - g.pr,
              id0 = (a0d + bd) * SD - g.pd;
    if (ic0 >= g.IC || ir0 >= g.IR || id0 >= g.ID) continue;
    T acc[SC * SR * SD][V];
#pragma unroll
    for (int j = 0; j < SC * SR * SD; ++j)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[j][i] = T(0);
#pragma unroll
    for (int wc = 0; wc <= DC; ++wc)
#pragma unroll
      for (int wr = 0; wr <= DR; ++wr)
#pragma unroll
        for (int wd = 0; wd <= DD; ++wd) {  // window a - D + w: output order
          const int at = (((bc + wc) * tl.NWR + (br + wr)) * tl.NWD + (bd + wd)) * tl.CVB + cvl;
          if (MODE == POOL_AVG) {
            const int oc = a0c + bc + wc - DC, orr = a0r + br + wr - DR, od = a0d + bd + wd - DD;
            if ((unsigned)oc >= (unsigned)g.OC || (unsigned)orr >= (unsigned)g.OR ||
                (unsigned)od >= (unsigned)g.OD)
              continue;
          }
          const uint32_t word = MODE == POOL_MAX ? code[at] : 0u;
          T gv[V];
          // (a window that does not exist has codes that no element matches;
          // its dY slot is never added)
#pragma unroll
          for (int i = 0; i < V; ++i) gv[i] = gbuf[(size_t)at * V + i];
#pragma unroll
          for (int jc = 0; jc < SC; ++jc)
#pragma unroll
            for (int jr = 0; jr < SR; ++jr)
#pragma unroll
              for (int jd = 0; jd < SD; ++jd) {
                const int kc = jc + (DC - wc) * SC, kr = jr + (DR - wr) * SR,
                          kd = jd + (DD - wd) * SD;
                if (kc >= KC || kr >= KR || kd >= KD) continue;
                const int mine = (kc * KR + kr) * KD + kd;
                T(&o)[V] = acc[(jc * SR + jr) * SD + jd];
#pragma unroll
                for (int i = 0; i < V; ++i) {
                  if (MODE == POOL_AVG) o[i] += gv[i];
                  else if (((word >> (8 * i)) & 0xffu) == (uint32_t)mine) o[i] += gv[i];
                }
              }
        }
    T *out = dx + xbase + ic0 * sc + ir0 * sr + id0 * sd + ch;
#pragma unroll
    for (int jc = 0; jc < SC; ++jc)
#pragma unroll
      for (int jr = 0; jr < SR; ++jr)
#pragma unroll
        for (int jd = 0; jd < SD; ++jd)
          if ((unsigned)(ic0 + jc) < (unsigned)g.IC && (unsigned)(ir0 + jr) < (unsigned)g.IR &&
              (unsigned)(id0 + jd) < (unsigned)g.ID)
            store_vec<T, V>(out + jc * sc + jr * sr + jd * sd, acc[(jc * SR + jr) * SD + jd]);
  }
}

// The tile of an overlapping backward over V-element vectors of `es` bytes
// each; false when the window has too many taps for a one-byte code, an
// index does not fit 31 bits, or no tile fits shared memory (the per-element
// kernel then runs).  Larger tiles compute fewer windows twice; the tile is
// halved along its longest axis while fewer than two blocks an SM would run
// or its windows take more than 48 KB.
//
// `fixed`: the tile is counted in blocks of the stride (the compile-time
// kernel), and the blocks of an axis are the (I - 1 + p) / s + 1 that hold its
// positions; otherwise in single elements.
bool plan_over(const PG &g, int V, size_t es, bool fixed, OverTile &t, int64_t &blocks,
               size_t &smem) {
  const int64_t big = int64_t(1) << 30;
  if (g.KC * g.KR * g.KD > 254 || g.IC >= big || g.IR >= big || g.ID >= big || g.pc >= big ||
      g.pr >= big || g.pd >= big || g.KC >= big || g.KR >= big || g.KD >= big)
    return false;
  const int64_t CV = g.Ch / V;
  t.CVB = (int)std::min<int64_t>(CV, 16);
  t.n_cb = (int)ceil_div(CV, t.CVB);
  auto l2 = [](int64_t n, int most) {
    int l = 0;
    while (l < most && (int64_t(1) << l) < n) ++l;
    return l;
  };
  const int64_t EC = fixed ? (g.IC - 1 + g.pc) / g.sc + 1 : g.IC,
                ER = fixed ? (g.IR - 1 + g.pr) / g.sr + 1 : g.IR,
                ED = fixed ? (g.ID - 1 + g.pd) / g.sd + 1 : g.ID;
  const int most = fixed && std::max(g.sc, g.sr) > 1 ? 3 : 4;
  if (ED == 1) {
    t.ld = 0; t.lr = l2(ER, most); t.lc = l2(EC, most);
  } else {
    t.ld = l2(ED, most - 1); t.lr = l2(ER, most - 1); t.lc = l2(EC, most - 1);
  }
  auto wins = [fixed](int tile, int64_t k, int s, int64_t O) {
    return fixed ? tile + (k - 1) / s : std::min<int64_t>(O, (tile + k - 2) / s + 1);
  };
  while (true) {
    t.n_c = (int)ceil_div(EC, int64_t(1) << t.lc);
    t.n_r = (int)ceil_div(ER, int64_t(1) << t.lr);
    t.n_d = (int)ceil_div(ED, int64_t(1) << t.ld);
    const int64_t nwc = wins(1 << t.lc, g.KC, g.sc, g.OC), nwr = wins(1 << t.lr, g.KR, g.sr, g.OR),
                  nwd = wins(1 << t.ld, g.KD, g.sd, g.OD);
    blocks = g.B * t.n_c * t.n_r * t.n_d * t.n_cb;
    const int64_t need = nwc * nwr * nwd * t.CVB * V * (int64_t)(es + 1);
    const bool fits = need <= 48 * 1024;
    const int longest = std::max(t.lc, std::max(t.lr, t.ld));
    if (fits && (blocks >= 2 * 152 || t.lc + t.lr + t.ld <= 4 || longest == 0)) {
      if (blocks >= (int64_t(1) << 31)) return false;
      t.NWR = (int)nwr; t.NWD = (int)nwd; t.NW = (int)(nwc * nwr * nwd);
      smem = (size_t)need;
      break;
    }
    if (longest == 0) return false;
    if (t.lc == longest) --t.lc;
    else if (t.lr == longest) --t.lr;
    else --t.ld;
  }
  t.nwr = make_fastdiv((uint32_t)t.NWR);
  t.nwd = make_fastdiv((uint32_t)t.NWD);
  t.cvb = make_fastdiv((uint32_t)t.CVB);
  t.sc = make_fastdiv((uint32_t)g.sc);
  t.sr = make_fastdiv((uint32_t)g.sr);
  t.sd = make_fastdiv((uint32_t)g.sd);
  return true;
}

// Ordered rebuild of dX[0] for max-pool backward when some window selected
// nothing (Owl routes those windows to flat element 0, owl_ndarray_pool_impl.h
// :167).  One block walks all windows in Owl's loop order (b, oc, or, od,
// ch), 1024 at a time; contributions are summed by one thread in order.
// Runs only when this call's ticket is marked (or `force`: some window has
// no in-range element, which the gather form never visits).
template <typename T>
__global__ void __launch_bounds__(1024) pool_max_fix0_kernel(PG g, const T *__restrict__ x,
                                                             const T *__restrict__ dy,
                                                             T *__restrict__ dx,
                                                             unsigned long long ticket,
                                                             int force) {
  // Launched as a programmatic dependent of the backward kernel: wait for
  // that grid to finish and its writes to become visible.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!force && *(volatile unsigned long long *)&g_degenerate_mark < ticket) return;
  __shared__ T contrib[1024];
  __shared__ int hit[1024];
  const int64_t total = g.B * g.OC * g.OR * g.OD * g.Ch;
  T sum = T(0);
  for (int64_t base = 0; base < total; base += 1024) {
    int64_t w = base + threadIdx.x;
    hit[threadIdx.x] = 0;
    if (w < total) {
      int64_t ch = w % g.Ch, p = w / g.Ch;
      int64_t od = p % g.OD, t = p / g.OD;
      int64_t orr = t % g.OR; t /= g.OR;
      int64_t oc = t % g.OC, b = t / g.OC;
      const int64_t xbase = b * g.IC * g.IR * g.ID * g.Ch;
      const int cs = (int)(oc * g.sc) - g.pc, rs = (int)(orr * g.sr) - g.pr,
                ds = (int)(od * g.sd) - g.pd;
      T best = T(-INFINITY);
      int64_t bi = 0;
      for (int a = cs; a < cs + (int)g.KC; ++a)
        for (int bb = rs; bb < rs + (int)g.KR; ++bb)
          for (int c = ds; c < ds + (int)g.KD; ++c)
            if (a >= 0 && a < g.IC && bb >= 0 && bb < g.IR && c >= 0 && c < g.ID) {
              int64_t off = xbase + (((int64_t)a * g.IR + bb) * g.ID + c) * g.Ch + ch;
              T v = x[off];
              if (best < v) { best = v; bi = off; }
            }
      if (bi == 0) { hit[threadIdx.x] = 1; contrib[threadIdx.x] = dy[w]; }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int64_t rem = total - base;
      int n = rem < 1024 ? (int)rem : 1024;
      for (int i = 0; i < n; ++i)
        if (hit[i]) sum += contrib[i];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) dx[0] = sum;
}

int grid_for(int64_t work) {
  int64_t blocks = ceil_div(work, 256);
  return (int)std::max<int64_t>(1, std::min<int64_t>(blocks, 152 * 16));
}

// Elements per 16-byte vector: 4 floats, 2 doubles or complex32, 1 complex64.
template <typename T>
constexpr int kWide = (int)(16 / sizeof(T));

template <typename T>
int vec_width(int64_t ch, const void *a, const void *b, const void *c) {
  auto al = [](const void *p, int bytes) { return ((uintptr_t)p % bytes) == 0; };
  if (kWide<T> >= 4 && ch % 4 == 0 && al(a, 16) && al(b, 16) && al(c, 16)) return 4;
  if (kWide<T> >= 2 && ch % 2 == 0 && al(a, 2 * sizeof(T)) && al(b, 2 * sizeof(T)) &&
      al(c, 2 * sizeof(T)))
    return 2;
  return 1;
}

// Windows tile the input exactly: stride = kernel, no padding, O*s = I.
bool exact_tiling(const PG &g) {
  auto ok = [](int64_t I, int64_t K, int64_t O, int s, int p) {
    return p == 0 && s == K && O * s == I;
  };
  return ok(g.IC, g.KC, g.OC, g.sc, g.pc) && ok(g.IR, g.KR, g.OR, g.sr, g.pr) &&
         ok(g.ID, g.KD, g.OD, g.sd, g.pd);
}

bool window_is(const PG &g, int kc, int kr, int kd) {
  return g.KC == kc && g.KR == kr && g.KD == kd;
}

template <typename T, int V, int KC, int KR, int KD>
void fwd_fixed(const PG &g, PoolMode mode, const T *x, T *y, int64_t *arg, int grid,
               cudaStream_t s) {
  const OutDecode d = make_out_decode(g, g.Ch / V);
  int64_t *none = nullptr;
  if (mode == POOL_AVG)
    launch_pdl(pool_fwd_fixed_kernel<T, V, KC, KR, KD, POOL_AVG, false>, dim3(grid), dim3(256),
               0, s, g, d, x, y, none);
  else if (arg)
    launch_pdl(pool_fwd_fixed_kernel<T, V, KC, KR, KD, POOL_MAX, true>, dim3(grid), dim3(256), 0,
               s, g, d, x, y, arg);
  else
    launch_pdl(pool_fwd_fixed_kernel<T, V, KC, KR, KD, POOL_MAX, false>, dim3(grid), dim3(256),
               0, s, g, d, x, y, none);
}

// The fixed-window kernels index outputs with 32-bit fast division.
bool small_output(const PG &g, int V) {
  return g.B * g.OC * g.OR * g.OD * (g.Ch / V) < (int64_t(1) << 31);
}

// Fixed-window kernels exist for the widest vector of each type (16 bytes)
// and the common window shapes 2x2, 3x3, 2x2x2 and 3x3x3.

template <typename T, int V>
int fwd_launch(const PG &g, PoolMode mode, const T *x, T *y, int64_t *arg, cudaStream_t s) {
  int grid = grid_for(g.B * g.OC * g.OR * g.OD * (g.Ch / V));
  const bool fixed = V == kWide<T> && small_output(g, V);
  int64_t *none = nullptr;
  if (fixed && window_is(g, 2, 2, 1)) {
    fwd_fixed<T, V, 2, 2, 1>(g, mode, x, y, arg, grid, s);
  } else if (fixed && window_is(g, 3, 3, 1)) {
    fwd_fixed<T, V, 3, 3, 1>(g, mode, x, y, arg, grid, s);
  } else if (fixed && window_is(g, 2, 2, 2)) {
    fwd_fixed<T, V, 2, 2, 2>(g, mode, x, y, arg, grid, s);
  } else if (fixed && window_is(g, 3, 3, 3)) {
    fwd_fixed<T, V, 3, 3, 3>(g, mode, x, y, arg, grid, s);
  } else if (mode == POOL_AVG) {
    launch_pdl(pool_fwd_kernel<T, V, POOL_AVG, false>, dim3(grid), dim3(256), 0, s, g, x, y, none);
  } else if (arg) {
    launch_pdl(pool_fwd_kernel<T, V, POOL_MAX, true>, dim3(grid), dim3(256), 0, s, g, x, y, arg);
  } else {
    launch_pdl(pool_fwd_kernel<T, V, POOL_MAX, false>, dim3(grid), dim3(256), 0, s, g, x, y, none);
  }
  OWL_CHECK_LAUNCH("pool_fwd_kernel");
  return kOk;
}

template <typename T>
int fwd_t(const PoolGeom &pg, PoolMode mode, const T *x, T *y, int64_t *arg, cudaStream_t s) {
  PG g = to_pg(pg);
  if (pg.y_elems() == 0) return kOk;
  int v = vec_width<T>(g.Ch, x, y, y);
  if (v == 4) return fwd_launch<T, kWide<T>>(g, mode, x, y, arg, s);
  if constexpr (kWide<T> >= 2) {
    if (v == 2) return fwd_launch<T, 2>(g, mode, x, y, arg, s);
  }
  return fwd_launch<T, 1>(g, mode, x, y, arg, s);
}

// Windows overlap in no dimension: every input element lies in at most one.
bool non_overlapping(const PG &g) { return g.sc >= g.KC && g.sr >= g.KR && g.sd >= g.KD; }

template <typename T, int V, int KC, int KR, int KD>
void bwd_tile(const PG &g, PoolMode mode, const T *x, const T *dy, T *dx,
              unsigned long long ticket, int grid, cudaStream_t s) {
  const OutDecode d = make_out_decode(g, g.Ch / V);
  if (mode == POOL_AVG)
    launch_pdl(pool_bwd_tile_kernel<T, V, KC, KR, KD, POOL_AVG>, dim3(grid), dim3(256), 0, s, g,
               d, x, dy, dx, ticket);
  else
    launch_pdl(pool_bwd_tile_kernel<T, V, KC, KR, KD, POOL_MAX>, dim3(grid), dim3(256), 0, s, g,
               d, x, dy, dx, ticket);
}

template <typename T, int V, int KC, int KR, int KD, int SC, int SR, int SD>
bool bwd_over_fixed(const PG &g, PoolMode mode, const T *x, const T *dy, T *dx,
                    unsigned long long ticket, cudaStream_t s) {
  OverTile tl;
  int64_t blocks = 0;
  size_t smem = 0;
  if (!window_is(g, KC, KR, KD) || g.sc != SC || g.sr != SR || g.sd != SD ||
      !plan_over(g, V, sizeof(T), true, tl, blocks, smem))
    return false;
  if (mode == POOL_AVG)
    launch_pdl(pool_bwd_over_fixed_kernel<T, V, KC, KR, KD, SC, SR, SD, POOL_AVG>,
               dim3((unsigned)blocks), dim3(256), smem, s, g, tl, x, dy, dx, ticket);
  else
    launch_pdl(pool_bwd_over_fixed_kernel<T, V, KC, KR, KD, SC, SR, SD, POOL_MAX>,
               dim3((unsigned)blocks), dim3(256), smem, s, g, tl, x, dy, dx, ticket);
  return true;
}

// The overlapping windows that networks use, in float32 with 16-byte channel
// vectors: 3x3 stride 2 and 1, 2x2 stride 1, 3x3x3 stride 2.
template <typename T, int V>
bool bwd_over_common(const PG &g, PoolMode mode, const T *x, const T *dy, T *dx,
                     unsigned long long ticket, cudaStream_t s) {
  if constexpr (std::is_same_v<T, float> && V == 4) {
    return bwd_over_fixed<T, V, 3, 3, 1, 2, 2, 1>(g, mode, x, dy, dx, ticket, s) ||
           bwd_over_fixed<T, V, 3, 3, 1, 1, 1, 1>(g, mode, x, dy, dx, ticket, s) ||
           bwd_over_fixed<T, V, 2, 2, 1, 1, 1, 1>(g, mode, x, dy, dx, ticket, s) ||
           bwd_over_fixed<T, V, 3, 3, 3, 2, 2, 2>(g, mode, x, dy, dx, ticket, s);
  }
  return false;
}

template <typename T, int V>
int bwd_launch(const PG &g, PoolMode mode, const T *x, const T *dy, T *dx,
               unsigned long long ticket, cudaStream_t s) {
  if (non_overlapping(g)) {
    int grid = grid_for(g.B * g.OC * g.OR * g.OD * (g.Ch / V));
    const bool tile = V == kWide<T> && exact_tiling(g) && small_output(g, V);
    if (tile && window_is(g, 2, 2, 1))
      bwd_tile<T, V, 2, 2, 1>(g, mode, x, dy, dx, ticket, grid, s);
    else if (tile && window_is(g, 2, 2, 2))
      bwd_tile<T, V, 2, 2, 2>(g, mode, x, dy, dx, ticket, grid, s);
    else if (mode == POOL_AVG)
      launch_pdl(pool_bwd_cell_kernel<T, V, POOL_AVG>, dim3(grid), dim3(256), 0, s, g, x, dy, dx,
                 ticket);
    else
      launch_pdl(pool_bwd_cell_kernel<T, V, POOL_MAX>, dim3(grid), dim3(256), 0, s, g, x, dy, dx,
                 ticket);
    OWL_CHECK_LAUNCH("pool_bwd_cell_kernel");
  } else {
    OverTile tl;
    int64_t blocks = 0;
    size_t smem = 0;
    int grid = grid_for(g.B * g.IC * g.IR * g.ID * (g.Ch / V));
    if (bwd_over_common<T, V>(g, mode, x, dy, dx, ticket, s)) {
      // launched
    } else if (plan_over(g, V, sizeof(T), false, tl, blocks, smem)) {
      if (mode == POOL_AVG)
        launch_pdl(pool_bwd_over_kernel<T, V, POOL_AVG>, dim3((unsigned)blocks), dim3(256), smem,
                   s, g, tl, x, dy, dx, ticket);
      else
        launch_pdl(pool_bwd_over_kernel<T, V, POOL_MAX>, dim3((unsigned)blocks), dim3(256), smem,
                   s, g, tl, x, dy, dx, ticket);
    } else if (mode == POOL_AVG)
      launch_pdl(pool_bwd_gather_kernel<T, V, POOL_AVG>, dim3(grid), dim3(256), 0, s, g, x, dy,
                 dx, ticket);
    else
      launch_pdl(pool_bwd_gather_kernel<T, V, POOL_MAX>, dim3(grid), dim3(256), 0, s, g, x, dy,
                 dx, ticket);
    OWL_CHECK_LAUNCH("pool_bwd_gather_kernel");
  }
  return kOk;
}

// True when some window has no in-range element (possible only with
// inconsistent explicit pads); Owl then routes its max gradient to element 0.
bool has_empty_window(const PG &g) {
  auto dim_empty = [](int64_t I, int64_t K, int64_t O, int s, int p) {
    if (O <= 0) return false;
    int64_t first_end = -p + K;           // window 0 covers [-p, K - p)
    int64_t last_start = (O - 1) * s - p;  // last window start
    return first_end <= 0 || last_start >= I;
  };
  return dim_empty(g.IC, g.KC, g.OC, g.sc, g.pc) || dim_empty(g.IR, g.KR, g.OR, g.sr, g.pr) ||
         dim_empty(g.ID, g.KD, g.OD, g.sd, g.pd);
}

template <typename T>
int bwd_t(const PoolGeom &pg, PoolMode mode, const T *x, const T *dy, T *dx, cudaStream_t s) {
  PG g = to_pg(pg);
  if (pg.x_elems() == 0) return kOk;
  if (pg.y_elems() == 0) {
    OWL_CUDA(cudaMemsetAsync(dx, 0, sizeof(T) * pg.x_elems(), s));
    return kOk;
  }
  const unsigned long long ticket = ++g_ticket;
  int v = vec_width<T>(g.Ch, x ? (const void *)x : (const void *)dy, dy, dx);
  int rc;
  if (v == 4) rc = bwd_launch<T, kWide<T>>(g, mode, x, dy, dx, ticket, s);
  else if (v == 2) rc = bwd_launch<T, kWide<T> >= 2 ? 2 : 1>(g, mode, x, dy, dx, ticket, s);
  else rc = bwd_launch<T, 1>(g, mode, x, dy, dx, ticket, s);
  if (rc == kOk && mode == POOL_MAX) {
    const int force = has_empty_window(g) ? 1 : 0;
    // Programmatic dependent launch: the fix-up grid is scheduled while the
    // backward grid drains and waits on it with griddepcontrol.wait.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(1024);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, pool_max_fix0_kernel<T>, g, x, dy, dx, ticket, force);
    note_launch();
    if (e != cudaSuccess) rc = cuda_fail(e, "pool_max_fix0_kernel");
  }
  return rc;
}

}  // namespace

template <typename F>
static int by_dtype(Dtype dt, F f) {
  switch (dt) {
    case F32: return f((float *)nullptr);
    case F64: return f((double *)nullptr);
    case C32: return f((c32 *)nullptr);
    case C64: return f((c64 *)nullptr);
  }
  set_error("unknown element type");
  return kErrInvalid;
}

int pool_fwd(Dtype dt, PoolMode mode, const PoolGeom &g, const void *x, void *y,
             int64_t *argmax, cudaStream_t s) {
  return by_dtype(dt, [&](auto *tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    return fwd_t<T>(g, mode, (const T *)x, (T *)y, argmax, s);
  });
}

int pool_bwd(Dtype dt, PoolMode mode, const PoolGeom &g, const void *x, const void *dy,
             void *dx, cudaStream_t s) {
  return by_dtype(dt, [&](auto *tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    return bwd_t<T>(g, mode, (const T *)x, (const T *)dy, (T *)dx, s);
  });
}

}  // namespace owlgpu
