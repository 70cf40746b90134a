// conv_simt.cu -- CUDA-core implicit-GEMM convolutions (float32 "plain",
// float64, complex32 and complex64), forward / backward-input /
// backward-kernel, 2-D, 3-D, strided, dilated.  No im2col matrix is ever
// materialised: every GEMM operand element is gathered from the NHWC-style
// Owl array while the tile is staged into
// shared memory.
//
// GEMM views (k = ((kc*KR + kr)*KD + kd)*Ci + ci, Owl's im2col column order,
// owl_ndarray_conv_impl.h:315-325):
//   forward      Y[m][co]  = sum_k  X[gather(m, k)]           * W[k][co]
//                m = output pixel (b, oc, or, od)
//   bwd input    dX[m][ci] = sum_{tap,co} dY[scatter^-1(m,tap)][co] * W[tap][ci][co]
//                m = input pixel; only taps with (i + p - t*d) % s == 0 hit
//   bwd kernel   dW[tap*Ci+ci][co] = sum_m X[gather(m, tap)][ci] * dY[m][co]
//                reduction over output pixels, split across CTAs and summed
//                by a second kernel in a fixed order (deterministic).
#include "../../include/owlgpu.h"
#include "common.cuh"
#include "reduce.cuh"

#include <algorithm>
#include <type_traits>

namespace owlgpu {
namespace {

enum Mode { FWD = 0, BWDI = 1, BWDK = 2 };

struct Dev {
  int64_t B, IC, IR, ID, Ci, KC, KR, KD, OC, OR, OD, Co;
  int sc, sr, sd, dc, dr, dd, pc, pr, pd;
  int64_t M, N, K;  // GEMM view sizes
  // FWD only, ystrided: output pixel (b, oc, or, od) is written at pixel
  // yoff + b*ysb + oc*ysc + or*ysr + od*ysd of the output array (one
  // residue class of a backward_input); otherwise the output is dense.
  int ystrided;
  int64_t yoff, ysb, ysc, ysr, ysd;
  // FWD, float32 vector kernel only, ystrided == 2 (window scatter): column
  // n = t*s2d_ci + ci of row m goes to output pixel (row pixel of m) +
  // tc*s2d_tc + tr*s2d_tr + td, channel ci, for tap t = (tc*s2d_kr + tr)*s2d_kd
  // + td (a backward_input whose kernel equals its stride: every input pixel
  // receives exactly one tap)
  int64_t s2d_ci, s2d_tc, s2d_tr;
  int s2d_kr, s2d_kd;
  // FWD: y = act(conv + bias[n]) (bias of the element type, or null; act
  // OWLGPU_ACT_*), applied to the finished sum as a second pass would
  const void *bias;
  int act;
};

template <typename T>
__device__ __forceinline__ T with_bias_act(T v, const Dev &g, int64_t n) {
  if (g.bias) v += static_cast<const T *>(g.bias)[n];
  if constexpr (std::is_floating_point_v<T>) {
    if (g.act == OWLGPU_ACT_RELU) v = v > T(0) ? v : T(0);
  }
  return v;
}

template <typename T, int MODE, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
    conv_simt_kernel(Dev g, const T *__restrict__ A0, const T *__restrict__ B0,
                     T *__restrict__ C, int64_t k_per_split) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int A_PER = BM * BK / NT;
  constexpr int B_PER = BN * BK / NT;
  static_assert(BM * BK % NT == 0 && BN * BK % NT == 0, "tile/thread mismatch");

  static_assert(MODE != FWD || 256 % BK == 0, "the tap table holds whole slabs");
  __shared__ T As[2][BK][BM + 4];
  __shared__ T Bs[2][BK][BN + 4];
  // Per-row (FWD/BWDI) or per-k (BWDK) pixel decode cache.
  constexpr int PIX = (MODE == BWDK) ? BK : BM;
  __shared__ int64_t s_base[2][PIX];
  __shared__ int s_c[2][PIX], s_r[2][PIX], s_d[2][PIX];
  // FWD: where k's tap and channel lie relative to a window's origin (element
  // offset, and the tap's position for the bounds), for KT consecutive k: one
  // 64-bit division per k and CTA instead of several per k slab and thread.
  constexpr int KT = MODE == FWD ? (sizeof(T) < 16 ? 512 : 256) : 1;
  __shared__ int64_t s_koff[KT];
  __shared__ int s_kc[KT], s_kr[KT], s_kd[KT];
  int64_t kt_begin = -KT;  // k of the table's first entry

  const int tid = threadIdx.x;
  // Pixels and taps are decoded in 32 bits where the sizes allow: the decode of a
  // slab is a serial chain of divisions that every thread waits for.
  const bool narrow = g.M < (1LL << 31) && g.K < (1LL << 31);
  auto split = [&](int64_t &p, int64_t d) -> int64_t {  // p / d in place; the remainder
    if (narrow) {
      const uint32_t a = (uint32_t)p, q = a / (uint32_t)d;
      p = q;
      return a - q * (uint32_t)d;
    }
    const int64_t q = p / d, r = p - q * d;
    p = q;
    return r;
  };
  const int64_t m0 = (int64_t)blockIdx.x * BM;
  // BWDK: a thread's A elements all sit in row m0 + tid % BM (NT is a
  // multiple of BM), so its tap and channel are decoded once.
  static_assert(MODE != BWDK || NT % BM == 0, "BWDK row decode needs NT % BM == 0");
  int a_dc = 0, a_dr = 0, a_dd = 0, a_ci = 0;
  bool a_mval = false;
  if (MODE == BWDK) {
    const int64_t m = m0 + tid % BM;
    a_mval = m < g.M;
    if (a_mval) {
      int64_t kc = m;
      a_ci = (int)split(kc, g.Ci);
      const int kd = (int)split(kc, g.KD), kr = (int)split(kc, g.KR);
      a_dc = (int)kc * g.dc;
      a_dr = kr * g.dr;
      a_dd = kd * g.dd;
    }
  }
  const int64_t n0 = (int64_t)blockIdx.y * BN;
  const int64_t k_begin = (int64_t)blockIdx.z * k_per_split;
  const int64_t k_end = min(g.K, k_begin + k_per_split);

  // ---- pixel decode helpers ------------------------------------------
  // FWD: row m is an output pixel; store batch base of X and window origin.
  // BWDI: row m is an input pixel; store batch base of dY and (i + pad).
  // BWDK: k index is an output pixel; store batch base of X and origin.
  auto decode_pixel = [&](int64_t p, int slot, int buf) {
    if (MODE == BWDI) {
      if (p < g.M) {
        int64_t b = p;
        const int64_t id = split(b, g.ID), ir = split(b, g.IR), ic = split(b, g.IC);
        s_base[buf][slot] = b * g.OC * g.OR * g.OD;
        s_c[buf][slot] = (int)ic + g.pc;
        s_r[buf][slot] = (int)ir + g.pr;
        s_d[buf][slot] = (int)id + g.pd;
      } else {
        s_base[buf][slot] = -1;
      }
    } else {
      int64_t lim = (MODE == FWD) ? g.M : g.K;
      if (p < lim) {
        int64_t b = p;
        const int64_t od = split(b, g.OD), orr = split(b, g.OR), oc = split(b, g.OC);
        s_base[buf][slot] = b * g.IC * g.IR * g.ID;
        s_c[buf][slot] = (int)(oc * g.sc) - g.pc;
        s_r[buf][slot] = (int)(orr * g.sr) - g.pr;
        s_d[buf][slot] = (int)(od * g.sd) - g.pd;
      } else {
        s_base[buf][slot] = -1;
      }
    }
  };

  if (MODE != BWDK) {
    for (int i = tid; i < BM; i += NT) decode_pixel(m0 + i, i, 0);
    for (int i = tid; i < BM; i += NT) {
      s_base[1][i] = s_base[0][i];
      s_c[1][i] = s_c[0][i]; s_r[1][i] = s_r[0][i]; s_d[1][i] = s_d[0][i];
    }
    __syncthreads();  // rows decoded by one thread are gathered by others
    if (MODE == FWD) {
      // a window's origin as an element offset
      for (int i = tid; i < BM; i += NT)
        if (s_base[0][i] >= 0)
          s_base[1][i] =
              (s_base[0][i] + ((int64_t)s_c[0][i] * g.IR + s_r[0][i]) * g.ID + s_d[0][i]) * g.Ci;
      __syncthreads();
    }
  }

  T a_reg[A_PER], b_reg[B_PER];

  // Gather one BK-slab of A and B into registers.
  auto load_tiles = [&](int64_t k0, int buf) {
    if (MODE == FWD) {
      // A[m][k]: thread owns a fixed k column, several rows.
      if (k0 >= kt_begin + KT) {  // (the same for every thread; KT is whole slabs)
        kt_begin = k0;
        __syncthreads();
        for (int i = tid; i < KT; i += NT) {
          const int64_t k = k0 + i;
          if (k >= k_end) break;
          int64_t kc = k;
          const int64_t ci = split(kc, g.Ci), kd = split(kc, g.KD), kr = split(kc, g.KR);
          s_kc[i] = (int)(kc * g.dc);
          s_kr[i] = (int)(kr * g.dr);
          s_kd[i] = (int)(kd * g.dd);
          s_koff[i] = ((kc * g.dc * g.IR + kr * g.dr) * g.ID + kd * g.dd) * g.Ci + ci;
        }
        __syncthreads();
      }
      const int kk = tid % BK;
      const int ki = (int)(k0 - kt_begin) + kk;
      const bool kval = k0 + kk < k_end;
      int64_t koff = 0;
      int tc = 0, tr = 0, td = 0;
      if (kval) {
        koff = s_koff[ki];
        tc = s_kc[ki]; tr = s_kr[ki]; td = s_kd[ki];
      }
#pragma unroll
      for (int i = 0; i < A_PER; ++i) {
        int mm = tid / BK + i * (NT / BK);
        T v = T(0);
        if (kval && s_base[0][mm] >= 0) {
          const int c = s_c[0][mm] + tc, r = s_r[0][mm] + tr, d = s_d[0][mm] + td;
          if (c >= 0 && c < g.IC && r >= 0 && r < g.IR && d >= 0 && d < g.ID)
            v = A0[s_base[1][mm] + koff];
        }
        a_reg[i] = v;
      }
      // B[k][n] = W[k][n], n fastest.
#pragma unroll
      for (int i = 0; i < B_PER; ++i) {
        int e = tid + i * NT;
        int kk2 = e / BN, nn = e % BN;
        int64_t kq = k0 + kk2, n = n0 + nn;
        b_reg[i] = (kq < k_end && n < g.N) ? B0[kq * g.N + n] : T(0);
      }
    } else if (MODE == BWDI) {
      // A[m][k], k = tap*Co + co: thread owns fixed k, several rows.
      const int kk = tid % BK;
      const int64_t k = k0 + kk;
      int kc = 0, kr = 0, kd = 0, co = 0;
      bool kval = k < k_end;
      if (kval) {
        int64_t t = k;
        co = (int)split(t, g.Co);
        kd = (int)split(t, g.KD);
        kr = (int)split(t, g.KR);
        kc = (int)t;
      }
#pragma unroll
      for (int i = 0; i < A_PER; ++i) {
        int mm = tid / BK + i * (NT / BK);
        T v = T(0);
        int64_t base = s_base[buf][mm];
        if (kval && base >= 0) {
          int tc = s_c[buf][mm] - kc * g.dc, tr = s_r[buf][mm] - kr * g.dr,
              td = s_d[buf][mm] - kd * g.dd;
          if (tc >= 0 && tr >= 0 && td >= 0 && tc % g.sc == 0 && tr % g.sr == 0 &&
              td % g.sd == 0) {
            int oc = tc / g.sc, orr = tr / g.sr, od = td / g.sd;
            if (oc < g.OC && orr < g.OR && od < g.OD)
              v = A0[((base + ((int64_t)oc * g.OR + orr) * g.OD + od) * g.Co) + co];
          }
        }
        a_reg[i] = v;
      }
      // B[k][n] = W[tap][n=ci][co]: co fastest across threads for coalescing.
#pragma unroll
      for (int i = 0; i < B_PER; ++i) {
        int e = tid + i * NT;
        int kk2 = e % BK, nn = e / BK;
        int64_t kq = k0 + kk2, n = n0 + nn;
        T v = T(0);
        if (kq < k_end && n < g.N) {
          int64_t tap = kq;
          const int64_t co = split(tap, g.Co);
          v = B0[(tap * g.Ci + n) * g.Co + co];
        }
        b_reg[i] = v;
      }
    } else {
      // BWDK: A[m=(tap,ci)][k=pixel] = X[gather], m fastest across threads.
#pragma unroll
      for (int i = 0; i < A_PER; ++i) {
        const int kk = (tid + i * NT) / BM;
        T v = T(0);
        const int64_t base = s_base[buf][kk];
        if (a_mval && base >= 0) {
          const int c = s_c[buf][kk] + a_dc, r = s_r[buf][kk] + a_dr, d = s_d[buf][kk] + a_dd;
          if (c >= 0 && c < g.IC && r >= 0 && r < g.IR && d >= 0 && d < g.ID)
            v = A0[((base + ((int64_t)c * g.IR + r) * g.ID + d) * g.Ci) + a_ci];
        }
        a_reg[i] = v;
      }
      // B[k=pixel][n=co] = dY[pixel][co].
#pragma unroll
      for (int i = 0; i < B_PER; ++i) {
        int e = tid + i * NT;
        int kk2 = e / BN, nn = e % BN;
        int64_t kq = k0 + kk2, n = n0 + nn;
        b_reg[i] = (kq < k_end && n < g.N) ? B0[kq * g.N + n] : T(0);
      }
    }
  };

  auto store_tiles = [&](int buf) {
    if (MODE == BWDK) {
#pragma unroll
      for (int i = 0; i < A_PER; ++i) {
        int e = tid + i * NT;
        As[buf][e / BM][e % BM] = a_reg[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < A_PER; ++i) {
        int mm = tid / BK + i * (NT / BK);
        As[buf][tid % BK][mm] = a_reg[i];
      }
    }
    if (MODE == BWDI) {
#pragma unroll
      for (int i = 0; i < B_PER; ++i) {
        int e = tid + i * NT;
        Bs[buf][e % BK][e / BK] = b_reg[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < B_PER; ++i) {
        int e = tid + i * NT;
        Bs[buf][e / BN][e % BN] = b_reg[i];
      }
    }
  };

  T acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = T(0);

  const int tx = tid % (BN / TN), ty = tid / (BN / TN);

  if (k_begin < k_end) {
    int buf = 0;
    if (MODE == BWDK) {
      for (int i = tid; i < BK; i += NT) decode_pixel(k_begin + i, i, 0);
      __syncthreads();
    }
    load_tiles(k_begin, 0);
    store_tiles(0);
    __syncthreads();
    for (int64_t k0 = k_begin; k0 < k_end; k0 += BK) {
      const int64_t kn = k0 + BK;
      const bool more = kn < k_end;
      if (more) {
        if (MODE == BWDK) {
          for (int i = tid; i < BK; i += NT) decode_pixel(kn + i, i, buf ^ 1);
          __syncthreads();
        }
        load_tiles(kn, buf ^ 1);
      }
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        T a[TM], b[TN];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = As[buf][kk][ty * TM + i];
#pragma unroll
        for (int j = 0; j < TN; ++j) b[j] = Bs[buf][kk][tx * TN + j];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
      }
      if (more) store_tiles(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }

  // ---- epilogue --------------------------------------------------------
  // split z of a split-K launch writes its own partial (z = 0 otherwise)
  T *Cz = C + (int64_t)blockIdx.z * g.M * g.N;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int64_t m = m0 + ty * TM + i;
    if (m >= g.M) continue;
    int64_t row = m;
    if (MODE == FWD && g.ystrided) {
      int64_t t = m;
      const int64_t od = t % g.OD;
      t /= g.OD;
      const int64_t orr = t % g.OR;
      t /= g.OR;
      const int64_t oc = t % g.OC, b = t / g.OC;
      row = g.yoff + b * g.ysb + oc * g.ysc + orr * g.ysr + od * g.ysd;
    }
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int64_t n = n0 + tx * TN + j;
      if (n < g.N) Cz[row * g.N + n] = MODE == FWD ? with_bias_act(acc[i][j], g, n) : acc[i][j];
    }
  }
}

// ---- float32 vector path ----------------------------------------------------
// The same GEMM views in float32 with 16-byte operand gathers and packed
// multiply-adds: BM x BN tiles, 16-deep k slabs, a thread TM x TN outputs in
// 4 x 4 quadrants (rows ty*4 + q*BM*4/TM, columns tx*4 + q*BN*4/TN, so every
// shared-memory fragment is one 16-byte load without bank conflicts).
//   FWD : a slab is 16 consecutive input channels of one tap (Ci % 16 == 0);
//         four threads read one pixel's 64 bytes, and each thread's output
//         pixels and the taps inside X are decoded once per CTA.  A is stored k-major with
//         its row index XOR-swizzled by the channel quad (k / 4) * 8, so the
//         four threads of a pixel write four different bank groups.  BT: the
//         kernel operand is [n][k] (a dense layer's x w^T), staged like A.
//   BWDK: a slab is 16 consecutive output pixels; a thread reads four
//         consecutive (tap, ci) rows of one pixel (Ci % 4 == 0), a warp one
//         pixel's rows; the slab's pixels are decoded by 16 threads into
//         shared memory one slab ahead.
// The k order of every output's sum is the same as the scalar kernel's
// (ascending, one fused multiply-add per k), whatever the tile, so a float32
// result has the same bits on either path.
//
// Bound: the FMA pipe and the latency that two or three warps a scheduler leave
// open.  A loop of nothing but fmaf reaches 60 TFLOP/s on this chip, one of
// fma.rn.f32x2 (two multiply-adds an instruction, each rounded as fmaf) 68, so
// the accumulators are pairs of neighbouring rows: A's fragments are read as
// pairs, B's values duplicated into both halves.  Blocks of 128 threads (three an
// SM) instead of 256 (one) let one block's barrier and loads overlap another's
// arithmetic: [32;56;56;128] x [3;3;128;128] 43 -> 48 TFLOP/s.
//
// WIDE: the column tiles lie along grid.x and the row tiles along grid.y, for
// products of more columns than 65535 tiles hold.
constexpr int kVBK = 16;
constexpr int64_t kMaxGridY = 65535;

__device__ __forceinline__ float4 ldg4(const float *p) {
  return __ldg(reinterpret_cast<const float4 *>(p));
}

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void ffma2(uint64_t &d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int MODE, int BM, int BN, int TM, int TN, bool BT, bool WIDE>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
    conv_f32v_kernel(Dev g, const float *__restrict__ A0, const float *__restrict__ B0,
                     float *__restrict__ C, int64_t k_per_split) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  static_assert(MODE == FWD || !BT, "transposed B: FWD only");
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int NI = TM / 4, NJ = TN / 4;            // row and column quads per thread
  constexpr int RSTEP = BM / NI, CSTEP = BN / NJ;    // between them
  __shared__ __align__(16) float As[2][kVBK][BM];
  __shared__ __align__(16) float Bs[2][kVBK][BN];
  // BWDK: the slab's pixels: window origin (c, r, d; w = 0 past the end) and
  // the origin's pixel index in X
  __shared__ int4 s_pix[2][kVBK];
  __shared__ int64_t s_lin[2][kVBK];

  const int tid = threadIdx.x;
  // A warp covers 8 row threads x 4 column threads: its 16-byte fragment
  // loads touch one contiguous run of A and one of B per k (one shared-memory
  // wavefront each).
  constexpr int CW = BN / TN / 4;  // warps along the columns
  const int lane = tid & 31, warp = tid >> 5;
  const int ty = (warp / CW) * 8 + (lane >> 2), tx = (warp % CW) * 4 + (lane & 3);
  const int64_t m0 = (int64_t)(WIDE ? blockIdx.y : blockIdx.x) * BM,
                n0 = (int64_t)(WIDE ? blockIdx.x : blockIdx.y) * BN;
  const int64_t k_begin = (int64_t)blockIdx.z * k_per_split;
  const int64_t k_end = min(g.K, k_begin + k_per_split);
  const int64_t img = g.IC * g.IR * g.ID;  // pixels per batch image of X

  // ---- FWD: this thread's RQ output pixels and its channel quad -----------
  constexpr int RQ = BM * 4 / NT;
  const int aq = tid & 3;  // FWD: channel quad within the slab
  // MASKS: a pixel's window origin in X (at this thread's channel quad) and a
  // bit for each of 32 taps, set when the tap lies inside X, rebuilt every 32
  // taps: a slab costs a pixel one bit test and one add.  Otherwise its image
  // and origin coordinates, tested per slab.  The masks pay in the 128 x 32 tile
  // ([16;57;43;96] x [3;3;96;160] 282 -> 254 us); in the 8 x 8-output tile their
  // registers cost more than they save (617 -> 637 us on [32;56;56;128] x
  // [3;3;128;128]), and in the small tile, for short reductions, their set-up.
  constexpr bool MASKS = MODE == FWD && TM == 8 && TN == 4;
  const float *arow[RQ];
  uint32_t amask[RQ];
  int64_t abase[RQ];
  int ac[RQ], ar[RQ], ad[RQ];
  // ---- BWDK: this thread's four (tap, ci) rows, its pixels ak + AKS*h
  constexpr int MQ = BM / 4;   // row quads per k row
  constexpr int AKS = NT / MQ > kVBK ? kVBK : NT / MQ;  // k rows per pass
  const int mq = (tid % MQ) * 4;
  const int ak = tid / MQ;
  bool mval = false;
  int t_dc = 0, t_dr = 0, t_dd = 0;
  const float *a_tap = A0;  // BWDK: the rows' channel at their tap from a window's origin
  // FWD: decode this thread's pixels (MASKS: with the masks of the 32 taps from
  // t0 on)
  auto row_masks = [&](int t0, bool first) {
#pragma unroll
    for (int h = 0; h < RQ; ++h) {
      const int64_t m = m0 + (tid >> 2) + NT / 4 * h;
      amask[h] = 0;
      abase[h] = -1;
      ac[h] = ar[h] = ad[h] = 0;
      if (first) arow[h] = A0;
      if (m < g.M) {
        int64_t t = m;
        const int64_t od = t % g.OD;
        t /= g.OD;
        const int64_t orr = t % g.OR;
        t /= g.OR;
        const int64_t oc = t % g.OC, b = t / g.OC;
        const int c = (int)(oc * g.sc) - g.pc, r = (int)(orr * g.sr) - g.pr,
                  d = (int)(od * g.sd) - g.pd;
        if (!MASKS) {
          abase[h] = b * img;
          ac[h] = c; ar[h] = r; ad[h] = d;
          continue;
        }
        if (first)
          arow[h] = A0 + (b * img + ((int64_t)c * g.IR + r) * g.ID + d) * g.Ci + aq * 4;
        const int krd = (int)(g.KR * g.KD);
        int kc = t0 / krd, rem = t0 - kc * krd;
        int kr = rem / (int)g.KD, kd = rem - kr * (int)g.KD;
        const int n = (int)min((int64_t)32, g.KC * g.KR * g.KD - t0);
        uint32_t mask = 0;
        for (int q = 0; q < n; ++q) {
          mask |= (uint32_t)((unsigned)(c + kc * g.dc) < (unsigned)g.IC &&
                             (unsigned)(r + kr * g.dr) < (unsigned)g.IR &&
                             (unsigned)(d + kd * g.dd) < (unsigned)g.ID)
                  << q;
          if (++kd == g.KD) {
            kd = 0;
            if (++kr == g.KR) {
              kr = 0;
              ++kc;
            }
          }
        }
        amask[h] = mask;
      }
    }
  };
  if (MODE == FWD) {
    row_masks(0, true);
  } else {
    const int64_t m = m0 + mq;
    if (m < g.M) {
      mval = true;
      int64_t tap = m / g.Ci;
      const int64_t mci = m - tap * g.Ci;
      const int kd = (int)(tap % g.KD);
      tap /= g.KD;
      const int kr = (int)(tap % g.KR), kc = (int)(tap / g.KR);
      t_dc = kc * g.dc;
      t_dr = kr * g.dr;
      t_dd = kd * g.dd;
      a_tap = A0 + (((int64_t)t_dc * g.IR + t_dr) * g.ID + t_dd) * g.Ci + mci;
    }
  }
  // BWDK: decode pixel p into slot `slot` of buffer `buf` (-1 past k_end)
  auto put_pixel = [&](int64_t b, int64_t oc, int64_t orr, int64_t od, int slot, int buf) {
    const int c = (int)(oc * g.sc) - g.pc, r = (int)(orr * g.sr) - g.pr,
              d = (int)(od * g.sd) - g.pd;
    s_pix[buf][slot] = make_int4(c, r, d, 1);
    s_lin[buf][slot] = b * img + ((int64_t)c * g.IR + r) * g.ID + d;
  };
  auto decode = [&](int64_t p, int slot, int buf) {
    if (p < k_end) {
      int64_t t = p;
      const int64_t od = t % g.OD;
      t /= g.OD;
      const int64_t orr = t % g.OR;
      t /= g.OR;
      put_pixel(t / g.OC, t % g.OC, orr, od, slot, buf);
    } else {
      s_pix[buf][slot] = make_int4(0, 0, 0, 0);
    }
  };

  // BWDK: in the loop, decode thread tid (< 16) decodes pixel dp = (slab j +
  // 2)'s pixel tid, one slab further each step: (b, oc, orr*OD + od) advance
  // by adding 16 to the last with carries, no division per slab
  int64_t dp = 0, db = 0, doc = 0, dq = 0;
  const int64_t ORD = g.OR * g.OD;
  if (MODE == BWDK && tid < kVBK) {
    dp = k_begin + 2 * kVBK + tid;
    int64_t t = dp;
    dq = t % ORD;
    t /= ORD;
    doc = t % g.OC;
    db = t / g.OC;
  }
  auto decode_next = [&](int slot, int buf) {
    if (dp < k_end) {
      const int64_t orr = g.OD == 1 ? dq : dq / g.OD, od = dq - orr * g.OD;
      put_pixel(db, doc, orr, od, slot, buf);
    } else {
      s_pix[buf][slot] = make_int4(0, 0, 0, 0);
    }
    dp += kVBK;
    dq += kVBK;
    while (dq >= ORD) {
      dq -= ORD;
      if (++doc == g.OC) {
        doc = 0;
        ++db;
      }
    }
  };

  // FWD slab position: tap (kc, kr, kd) = number `tap`, first channel ci0 of
  // slab k0, and their offset soff from a window's origin
  int kc = 0, kr = 0, kd = 0, tap = 0;
  int64_t ci0 = 0, soff = 0;
  auto tap_offset = [&]() {
    soff = (((int64_t)kc * g.dc * g.IR + (int64_t)kr * g.dr) * g.ID + (int64_t)kd * g.dd) * g.Ci;
  };
  if (MODE == FWD) {
    int64_t t = k_begin / g.Ci;
    ci0 = k_begin - t * g.Ci;
    tap = (int)t;
    kd = (int)(t % g.KD);
    t /= g.KD;
    kr = (int)(t % g.KR);
    kc = (int)(t / g.KR);
    tap_offset();
    soff += ci0;
    if (MASKS && tap >= 32) row_masks(tap & ~31, false);
  }

  // A: FWD RQ float4 (pixels), BWDK 16/AKS float4 (k rows)
  constexpr int AH = MODE == FWD ? RQ : kVBK / AKS;
  // B: float4 column bcol of k rows bk + BKS*h, or (BT) k quad aq of rows n
  constexpr int BQ = BN / 4;  // float4 per k row of B
  constexpr int BKS = NT / BQ > kVBK ? kVBK : NT / BQ;
  constexpr int BH = BT ? (BN * 4 + NT - 1) / NT : kVBK / BKS;
  const int bcol = (tid % BQ) * 4;
  const int bk = tid / BQ;
  const bool bval = bk < BKS && n0 + bcol < g.N;
  float4 va[AH], vb[BH];

  // global -> registers for slab k0 (FWD: at tap kc/kr/kd, channels ci0..)
  auto load = [&](int64_t k0, int buf) {
    if (MODE == FWD) {
#pragma unroll
      for (int h = 0; h < AH; ++h) {
        va[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (MASKS) {
          if ((amask[h] >> (tap & 31)) & 1u) va[h] = ldg4(arow[h] + soff);
        } else {
          const int c = ac[h] + kc * g.dc, r = ar[h] + kr * g.dr, d = ad[h] + kd * g.dd;
          if (abase[h] >= 0 && (unsigned)c < (unsigned)g.IC && (unsigned)r < (unsigned)g.IR &&
              (unsigned)d < (unsigned)g.ID)
            va[h] = ldg4(A0 + (abase[h] + ((int64_t)c * g.IR + r) * g.ID + d) * g.Ci + ci0 + aq * 4);
        }
      }
    } else {
#pragma unroll
      for (int h = 0; h < AH; ++h) {
        va[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (mval && ak < AKS) {
          const int kl = ak + AKS * h;
          const int4 px = s_pix[buf][kl];
          if (px.w && (unsigned)(px.x + t_dc) < (unsigned)g.IC &&
              (unsigned)(px.y + t_dr) < (unsigned)g.IR && (unsigned)(px.z + t_dd) < (unsigned)g.ID)
            va[h] = ldg4(a_tap + s_lin[buf][kl] * g.Ci);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < BH; ++h) {
      vb[h] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (BT) {
        const int n = (tid >> 2) + NT / 4 * h;
        if (n < BN && n0 + n < g.N) vb[h] = ldg4(B0 + (n0 + n) * g.K + k0 + aq * 4);
      } else {
        const int64_t kq = k0 + bk + BKS * h;
        if (bval && kq < k_end) vb[h] = ldg4(B0 + kq * g.N + n0 + bcol);
      }
    }
  };
  auto store = [&](int buf) {
    if (MODE == FWD) {
#pragma unroll
      for (int h = 0; h < AH; ++h) {
        const int row = ((tid >> 2) + NT / 4 * h) ^ (aq << 3);
        As[buf][aq * 4 + 0][row] = va[h].x;
        As[buf][aq * 4 + 1][row] = va[h].y;
        As[buf][aq * 4 + 2][row] = va[h].z;
        As[buf][aq * 4 + 3][row] = va[h].w;
      }
    } else if (ak < AKS) {
#pragma unroll
      for (int h = 0; h < AH; ++h)
        *reinterpret_cast<float4 *>(&As[buf][ak + AKS * h][mq]) = va[h];
    }
    if (BT) {
#pragma unroll
      for (int h = 0; h < BH; ++h) {
        const int n = (tid >> 2) + NT / 4 * h, col = n ^ (aq << 3);
        if (n < BN) {
          Bs[buf][aq * 4 + 0][col] = vb[h].x;
          Bs[buf][aq * 4 + 1][col] = vb[h].y;
          Bs[buf][aq * 4 + 2][col] = vb[h].z;
          Bs[buf][aq * 4 + 3][col] = vb[h].w;
        }
      }
    } else if (bk < BKS) {
#pragma unroll
      for (int h = 0; h < BH; ++h)
        *reinterpret_cast<float4 *>(&Bs[buf][bk + BKS * h][bcol]) = vb[h];
    }
  };
  auto next_tap = [&]() {
    ci0 += kVBK;
    soff += kVBK;
    if (ci0 == g.Ci) {
      ci0 = 0;
      if (++kd == g.KD) {
        kd = 0;
        if (++kr == g.KR) {
          kr = 0;
          ++kc;
        }
      }
      tap_offset();
      if (MASKS && (++tap & 31) == 0) row_masks(tap, false);
    }
  };

  uint64_t acc[TM / 2][TN];  // rows 2i, 2i + 1 of the thread's TM
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0;

  if (k_begin < k_end) {
    if (MODE == BWDK) {
      if (tid < kVBK) decode(k_begin + tid, tid, 0);
      if (tid >= kVBK && tid < 2 * kVBK) decode(k_begin + kVBK + tid - kVBK, tid - kVBK, 1);
      __syncthreads();
    }
    load(k_begin, 0);
    store(0);
    if (MODE == FWD) next_tap();
    __syncthreads();
    int buf = 0;
    for (int64_t k0 = k_begin; k0 < k_end; k0 += kVBK) {
      const int64_t kn = k0 + kVBK;
      const bool more = kn < k_end;
      if (more) load(kn, buf ^ 1);  // BWDK: slab kn's pixels sit in buffer buf ^ 1
      // BWDK: decode slab kn + 16 into this slab's (now unused) buffer
      if (MODE == BWDK && tid < kVBK) decode_next(tid, buf);  // pixel kn + 16 + tid
#pragma unroll
      for (int k = 0; k < kVBK; ++k) {
        const int sw = MODE == FWD ? ((k >> 2) << 3) : 0, swb = BT ? ((k >> 2) << 3) : 0;
        uint64_t a[TM / 2];
#pragma unroll
        for (int q = 0; q < NI; ++q) {
          const ulonglong2 f =
              *reinterpret_cast<const ulonglong2 *>(&As[buf][k][(RSTEP * q + ty * 4) ^ sw]);
          a[2 * q] = f.x;
          a[2 * q + 1] = f.y;
        }
#pragma unroll
        for (int q = 0; q < NJ; ++q) {
          const float4 f =
              *reinterpret_cast<const float4 *>(&Bs[buf][k][(CSTEP * q + tx * 4) ^ swb]);
          const uint64_t b[4] = {pack2(f.x, f.x), pack2(f.y, f.y), pack2(f.z, f.z),
                                 pack2(f.w, f.w)};
#pragma unroll
          for (int i = 0; i < TM / 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) ffma2(acc[i][4 * q + j], a[i], b[j]);
        }
      }
      if (more) {
        store(buf ^ 1);
        if (MODE == FWD) next_tap();
      }
      __syncthreads();
      buf ^= 1;
    }
  }

  float *Cz = C + (int64_t)blockIdx.z * g.M * g.N;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int64_t m = m0 + RSTEP * (i >> 2) + ty * 4 + (i & 3);
    if (m >= g.M) continue;
    int64_t row = m;
    if (MODE == FWD && g.ystrided) {
      int64_t t = m;
      const int64_t od = t % g.OD;
      t /= g.OD;
      const int64_t orr = t % g.OR;
      t /= g.OR;
      const int64_t oc = t % g.OC, b = t / g.OC;
      row = g.yoff + b * g.ysb + oc * g.ysc + orr * g.ysr + od * g.ysd;
    }
#pragma unroll
    for (int q = 0; q < NJ; ++q) {
      const int64_t n = n0 + q * CSTEP + tx * 4;
      if (n >= g.N) continue;
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float lo, hi;
        unpack2(acc[i >> 1][4 * q + j], lo, hi);
        v[j] = (i & 1) ? hi : lo;
        if (MODE == FWD) v[j] = with_bias_act(v[j], g, n + j);
      }
      float *dst = Cz + row * g.N + n;
      if (MODE == FWD && g.ystrided == 2) {
        const int64_t t = n / g.s2d_ci, ci = n - t * g.s2d_ci;
        const int64_t tc = t / (g.s2d_kr * g.s2d_kd), tr = (t / g.s2d_kd) % g.s2d_kr,
                      td = t % g.s2d_kd;
        dst = Cz + (row + tc * g.s2d_tc + tr * g.s2d_tr + td) * g.s2d_ci + ci;
      }
      *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
}

// Whether the float32 vector path takes a launch: 16-byte aligned operands,
// N a multiple of 4, FWD slabs inside one tap (Ci % 16, whole slabs per
// split), BWDK rows in quads of one tap (Ci % 4); BWDI only as the product
// x w^T of a 1x1 geometry (simt_gemm), with whole slabs of K = Co.
bool f32v_ok(int mode, const Dev &d, const void *A, const void *B, const void *C,
             int64_t kps) {
  auto al = [](const void *p) { return ((uintptr_t)p & 15) == 0; };
  if (!al(A) || !al(B) || !al(C) || d.N % 4 != 0 || d.N == 0) return false;
  if (d.IC >= (1 << 30) || d.IR >= (1 << 30) || d.ID >= (1 << 30)) return false;
  if (mode == FWD) return d.Ci % kVBK == 0 && kps % kVBK == 0;
  if (mode == BWDK) return d.Ci % 4 == 0;
  return d.KC * d.KR * d.KD == 1 && d.sc == 1 && d.sr == 1 && d.sd == 1 && d.pc == 0 &&
         d.pr == 0 && d.pd == 0 && d.IC == d.OC && d.IR == d.OR && d.ID == d.OD &&
         d.Co % kVBK == 0 && kps % kVBK == 0;
}

template <int MODE, int BM, int BN, int TM, int TN, bool BT, bool WIDE = false>
cudaError_t launch_f32v_tile(const Dev &d, const float *A, const float *B, float *C, int splits,
                             int64_t kps, cudaStream_t s) {
  const unsigned mt = (unsigned)ceil_div(d.M, BM), nt = (unsigned)ceil_div(d.N, BN);
  const dim3 grid(WIDE ? nt : mt, WIDE ? mt : nt, (unsigned)splits);
  return launch_pdl(conv_f32v_kernel<MODE, BM, BN, TM, TN, BT, WIDE>, grid,
                    dim3((BM / TM) * (BN / TN)), 0, s, d, A, B, C, kps);
}

// The tile of a launch: the one whose busiest SM takes the least time: n * BM *
// BN outputs (n whole tiles while they are resident together, else the average
// plus half a tile of tail), at the tile's cost per output with the GPU full
// (measured on [32;56;56;128] x [3;3;128;128]: 617, 699 and 790 us), over the
// share of the FMA pipe that the resident tiles keep busy, about w / (w + 3) for
// w warps (by registers 3 blocks of 128 x 64 fit, 4 of 128 x 32, 6 of 64 x 32).
// Measured against each tile forced: it takes the fastest on wide, ragged (N =
// 160, 96), 5x5x32x64, 3-D and [8;32;32;16] x [3;3;16;32] layers in all three passes,
// or one within 3 %.  Where the 32-column tiles are more than a grid's y axis takes,
// the 64-column one; where those are too, that one with its grid turned (3: a kernel of
// its own, for choosing the axis in the kernel cost the ragged float32 layers 2 %).
int pick_f32v(const Dev &d, int splits) {
  static const struct { int bm, bn, most; double cost; } t[] = {
      {128, 64, 3, 1.0}, {128, 32, 4, 1.13}, {64, 32, 6, 1.33}};
  if (ceil_div(d.N, 64) > kMaxGridY) return 3;
  if (ceil_div(d.N, 32) > kMaxGridY) return 0;
  int best = 0;
  double least = 0;
  for (int i = 0; i < 3; ++i) {
    const int64_t tiles = ceil_div(d.M, t[i].bm) * ceil_div(d.N, t[i].bn) * splits;
    const int64_t whole = ceil_div(tiles, 152);
    const double n = whole <= t[i].most ? (double)whole : (double)tiles / 152 + 0.5;
    const double w = 4.0 * std::min<double>(n, t[i].most);
    const double c = n * t[i].bm * t[i].bn * t[i].cost * (w + 3) / w;
    if (i == 0 || c < least) { least = c; best = i; }
  }
  return best;
}

template <int MODE, bool BT = false>
int launch_f32v(const Dev &d, const float *A, const float *B, float *C, int splits, int64_t kps,
                cudaStream_t s) {
  cudaError_t e;
  switch (pick_f32v(d, splits)) {
    case 0: e = launch_f32v_tile<MODE, 128, 64, 8, 8, BT>(d, A, B, C, splits, kps, s); break;
    case 1: e = launch_f32v_tile<MODE, 128, 32, 8, 4, BT>(d, A, B, C, splits, kps, s); break;
    case 2: e = launch_f32v_tile<MODE, 64, 32, 4, 4, BT>(d, A, B, C, splits, kps, s); break;
    default: e = launch_f32v_tile<MODE, 128, 64, 8, 8, BT, true>(d, A, B, C, splits, kps, s);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  note_launch();
  return e == cudaSuccess ? kOk : cuda_fail(e, "conv_f32v_kernel");
}

Dev make_dev(const ConvGeom &g, int mode) {
  Dev d{};
  d.B = g.B; d.IC = g.IC; d.IR = g.IR; d.ID = g.ID; d.Ci = g.Ci;
  d.KC = g.KC; d.KR = g.KR; d.KD = g.KD;
  d.OC = g.OC; d.OR = g.OR; d.OD = g.OD; d.Co = g.Co;
  d.sc = g.sc; d.sr = g.sr; d.sd = g.sd;
  d.dc = g.dc; d.dr = g.dr; d.dd = g.dd;
  d.pc = g.pc; d.pr = g.pr; d.pd = g.pd;
  d.ystrided = 0;
  d.yoff = 0;
  d.ysb = g.OC * g.OR * g.OD; d.ysc = g.OR * g.OD; d.ysr = g.OD; d.ysd = 1;
  if (mode == FWD) { d.M = g.out_pixels(); d.N = g.Co; d.K = g.taps() * g.Ci; }
  else if (mode == BWDI) { d.M = g.in_pixels(); d.N = g.Ci; d.K = g.taps() * g.Co; }
  else { d.M = g.taps() * g.Ci; d.N = g.Co; d.K = g.out_pixels(); }
  return d;
}

template <typename T, int MODE, int BM, int BN, int BK, int TM, int TN>
int launch_cfg(const Dev &d, const T *A, const T *B, T *C, int splits, int64_t kps,
               cudaStream_t s) {
  constexpr int NT = (BM / TM) * (BN / TN);
  dim3 grid((unsigned)ceil_div(d.M, BM), (unsigned)ceil_div(d.N, BN), (unsigned)splits);
  cudaError_t e = launch_pdl(conv_simt_kernel<T, MODE, BM, BN, BK, TM, TN>, grid, dim3(NT), 0, s,
                             d, A, B, C, kps);
  if (e == cudaSuccess) e = cudaGetLastError();
  note_launch();
  return e == cudaSuccess ? kOk : cuda_fail(e, "conv_simt_kernel");
}

// The scalar kernel's tile.  4-byte elements: by the GEMM's N (output channels
// for FWD, input channels for BWDI, Co for BWDK), and 32 rows for a
// backward_kernel of at most 32 (tap, channel) rows (a one-channel image),
// with slabs of 32 pixels: each slab costs a pixel decode and two barriers.
// 8- and 16-byte elements: the FP64 pipe is slow enough that any tile feeds
// it, so the smallest busiest SM wins, ceil(tiles / SMs) tiles of BM x BN, the
// larger tile on a tie ([8;28;28;32] x [5;5;32;64]: 98 tiles of 64 x 64 leave a
// third of the SMs idle, 883 us; 392 of 32 x 32, 625 us).  No tile of 32 columns where
// N has more of them than a grid's y axis takes.
template <typename T, int MODE>
int launch_any(const Dev &d, const T *A, const T *B, T *C, int splits, int64_t kps,
               cudaStream_t s) {
  if constexpr (std::is_same_v<T, float>) {
    if (f32v_ok(MODE, d, A, B, C, kps)) {
      if (MODE != BWDI) return launch_f32v<MODE == BWDK ? BWDK : FWD>(d, A, B, C, splits, kps, s);
      // dX = dY w^T of a 1x1 geometry: a forward product with w read as [n][k]
      Dev f = d;
      f.Ci = d.Co;
      f.Co = d.Ci;
      return launch_f32v<FWD, true>(f, A, B, C, splits, kps, s);
    }
  }
  const bool wide = ceil_div(d.N, 32) > kMaxGridY;
  if constexpr (sizeof(T) == 4) {
    if constexpr (MODE == BWDK) {
      if (d.M <= 32 && !wide) return launch_cfg<T, MODE, 32, 32, 32, 2, 2>(d, A, B, C, splits, kps, s);
    }
    if (d.N > 64) return launch_cfg<T, MODE, 128, 128, 8, 8, 8>(d, A, B, C, splits, kps, s);
    if (d.N > 32) return launch_cfg<T, MODE, 128, 64, 8, 8, 4>(d, A, B, C, splits, kps, s);
    return launch_cfg<T, MODE, 128, 32, 8, 4, 4>(d, A, B, C, splits, kps, s);
  } else {
    auto busiest = [&](int bm, int bn) {
      return ceil_div(ceil_div(d.M, bm) * ceil_div(d.N, bn) * splits, 152) * bm * bn;
    };
    const int64_t big = d.N > 32 ? busiest(64, 64) : busiest(64, 32), mid = busiest(32, 32);
    if (!wide && busiest(16, 32) < std::min(big, mid))
      return launch_cfg<T, MODE, 16, 32, 16, 1, 2>(d, A, B, C, splits, kps, s);
    if (!wide && mid < big) return launch_cfg<T, MODE, 32, 32, 8, 2, 2>(d, A, B, C, splits, kps, s);
    if (d.N > 32) return launch_cfg<T, MODE, 64, 64, 8, 4, 4>(d, A, B, C, splits, kps, s);
    return launch_cfg<T, MODE, 64, 32, 8, 4, 2>(d, A, B, C, splits, kps, s);
  }
}

// The tile that the split count of a reduction is planned for, not one that is
// launched: the vector kernel's are smaller, several to an SM (four waves of these are
// enough of those), and the FP64 ones follow the split count.
template <typename T>
int tile_m(const Dev &d) { return sizeof(T) == 4 ? (d.N <= 32 ? 256 : 128) : 64; }
template <typename T>
int tile_n(const Dev &d) {
  if (sizeof(T) == 4) return d.N > 64 ? 128 : (d.N > 32 ? 64 : 32);
  return d.N > 32 ? 64 : 32;
}

template <typename T>
int fwd_t(const ConvGeom &g, const T *x, const T *w, T *y, cudaStream_t s, const void *bias,
          int act) {
  Dev d = make_dev(g, FWD);
  d.bias = bias;
  d.act = act;
  if (d.M == 0 || d.N == 0) return kOk;
  if (d.K == 0) {
    OWL_CUDA(cudaMemsetAsync(y, 0, sizeof(T) * d.M * d.N, s));
    return kOk;
  }
  return launch_any<T, FWD>(d, x, w, y, 1, d.K, s);
}

// The kernel of one residue class of backward_input, laid out as the kernel
// of a forward convolution of dY: w2[t'][co][ci] = w[orig(t')][ci][co], t' =
// (a, b, c) over the class's taps, orig = (base + mul * t') per axis.
template <typename T>
__global__ void bwdi_class_weights(const T *__restrict__ w, T *__restrict__ w2, int Ka, int Kb,
                                   int Kc, int base_a, int base_b, int base_c, int mul_a,
                                   int mul_b, int mul_c, int KR, int KD, int64_t Ci,
                                   int64_t Co) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  const int64_t total = (int64_t)Ka * Kb * Kc * Co * Ci;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ci = i % Ci;
    int64_t r = i / Ci;
    const int64_t co = r % Co;
    r /= Co;
    const int c = (int)(r % Kc), b = (int)((r / Kc) % Kb), a = (int)(r / ((int64_t)Kc * Kb));
    const int64_t orig = ((int64_t)(base_a + mul_a * a) * KR + (base_b + mul_b * b)) * KD +
                         (base_c + mul_c * c);
    w2[i] = w[(orig * Ci + ci) * Co + co];
  }
}

// The kernel of a kernel = stride backward_input as one GEMM operand:
// w2[co][t*Ci + ci] = w[t][ci][co].
__global__ void window_weights(const float *__restrict__ w, float *__restrict__ w2, int64_t T,
                               int64_t Ci, int64_t Co) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  const int64_t total = T * Ci * Co;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ci = i % Ci;
    const int64_t r = i / Ci;
    const int64_t t = r % T, co = r / T;
    w2[i] = w[(t * Ci + ci) * Co + co];
  }
}

// float32 backward_input of a convolution whose kernel equals its stride
// (no dilation, no padding, the windows tiling the input exactly): every
// input pixel takes exactly one tap of one output pixel, so dX is one GEMM,
// dY [pixels][Co] x w2 [Co][taps*Ci], scattered window by window
// (depth-to-space) in its epilogue.  One launch reads dY once, where the
// residue classes (one tap each) read it once per class.  Returns 1 when the
// geometry or the operands do not qualify.
int bwdi_window_f32(const ConvGeom &g, float *dx, const float *w, const float *dy,
                    cudaStream_t s) {
  const bool win = g.KC == g.sc && g.KR == g.sr && g.KD == g.sd && g.dc == 1 && g.dr == 1 &&
                   g.dd == 1 && g.pc == 0 && g.pr == 0 && g.pd == 0 &&
                   g.IC == g.OC * g.sc && g.IR == g.OR * g.sr && g.ID == g.OD * g.sd &&
                   g.taps() > 1;
  if (!win) return 1;
  ConvGeom gc{};
  gc.B = g.B;
  gc.IC = g.OC; gc.IR = g.OR; gc.ID = g.OD; gc.Ci = g.Co;
  gc.KC = gc.KR = gc.KD = 1;
  gc.OC = g.OC; gc.OR = g.OR; gc.OD = g.OD; gc.Co = g.taps() * g.Ci;
  gc.sc = gc.sr = gc.sd = 1;
  gc.dc = gc.dr = gc.dd = 1;
  Dev d = make_dev(gc, FWD);
  d.ystrided = 2;
  d.yoff = 0;
  d.ysb = g.IC * g.IR * g.ID;
  d.ysc = (int64_t)g.sc * g.IR * g.ID;
  d.ysr = (int64_t)g.sr * g.ID;
  d.ysd = g.sd;
  d.s2d_ci = g.Ci;
  d.s2d_tc = g.IR * g.ID;
  d.s2d_tr = g.ID;
  d.s2d_kr = (int)g.KR;
  d.s2d_kd = (int)g.KD;
  if (g.Ci % 4 != 0 || !f32v_ok(FWD, d, dy, dy, dx, d.K)) return 1;  // w2 is fresh scratch
  float *w2 = nullptr;
  int rc = scratch_alloc((void **)&w2, sizeof(float) * (size_t)g.w_elems(), s);
  if (rc) return rc;
  const int64_t nw = g.w_elems();
  const dim3 wgrid((unsigned)std::min<int64_t>(ceil_div(nw, 256), 1024));
  cudaError_t e = launch_pdl(window_weights, wgrid, dim3(256), 0, s, w, w2, (int64_t)g.taps(),
                             (int64_t)g.Ci, (int64_t)g.Co);
  if (e == cudaSuccess) e = cudaGetLastError();
  note_launch();
  if (e != cudaSuccess) rc = cuda_fail(e, "window_weights");
  if (rc == kOk) rc = launch_f32v<FWD>(d, dy, w2, dx, 1, d.K, s);
  scratch_free(w2, s);
  return rc;
}

// backward_input as forward convolutions over the residue classes of dX.
// With forward index s*o - p + t*d, element i = s*a + r of dX receives
// dY[o] W[t] for the taps with (r + p - t*d) divisible by s, at
// o = a + (r + p - t*d)/s.  Those taps, largest first, spaced s/g apart
// (g = gcd(s, d)), form a stride-1 convolution of dY with dilation d/g and
// leading pad -(r + p - tmax*d)/s, whose output is the sub-grid i = s*a + r
// of dX: every multiply-add is a useful one (no tap is tested and masked).
// Classes that no tap reaches are zero; dX is cleared first when there are
// any.  Stride 1 is one class: dY against the flipped, channel-exchanged
// kernel.
template <typename T>
int bwdi_t(const ConvGeom &g, T *dx, const T *w, const T *dy, cudaStream_t s) {
  if (g.in_pixels() == 0 || g.Ci == 0) return kOk;
  if constexpr (std::is_same_v<T, float>) {
    if (g.Co > 0 && g.out_pixels() > 0) {
      const int rc = bwdi_window_f32(g, dx, w, dy, s);
      if (rc != 1) return rc;
    }
  }
  const int S[3] = {g.sc, g.sr, g.sd}, D[3] = {g.dc, g.dr, g.dd}, P[3] = {g.pc, g.pr, g.pd};
  const int64_t K[3] = {g.KC, g.KR, g.KD}, I[3] = {g.IC, g.IR, g.ID};
  struct Axis {
    int n, base, mul, dil, pad;
    int64_t out;
  };
  auto axis_class = [&](int ax, int r) {
    Axis a{0, 0, 0, 1, 0, 0};
    int tmax = -1;
    for (int t = 0; t < (int)K[ax]; ++t)
      if ((((r + P[ax] - t * D[ax]) % S[ax]) + S[ax]) % S[ax] == 0) {
        tmax = t > tmax ? t : tmax;
        ++a.n;
      }
    int gg = S[ax], dd = D[ax];
    while (dd) { const int t = gg % dd; gg = dd; dd = t; }
    a.base = tmax;
    a.mul = -(S[ax] / gg);
    a.dil = D[ax] / gg;
    a.pad = a.n ? -((r + P[ax] - tmax * D[ax]) / S[ax]) : 0;
    a.out = I[ax] > r ? (I[ax] - r + S[ax] - 1) / S[ax] : 0;
    return a;
  };
  bool any_empty = g.Co == 0 || g.out_pixels() == 0;
  for (int ax = 0; ax < 3; ++ax)
    for (int r = 0; r < S[ax]; ++r) {
      const Axis a = axis_class(ax, r);
      if (a.n == 0 && a.out > 0) any_empty = true;
    }
  if (any_empty) OWL_CUDA(cudaMemsetAsync(dx, 0, sizeof(T) * (size_t)g.x_elems(), s));
  if (g.Co == 0 || g.out_pixels() == 0) return kOk;
  T *w2 = nullptr;
  int rc = scratch_alloc((void **)&w2, sizeof(T) * (size_t)g.w_elems(), s);
  if (rc) return rc;
  for (int r0 = 0; r0 < S[0] && rc == kOk; ++r0)
    for (int r1 = 0; r1 < S[1] && rc == kOk; ++r1)
      for (int r2 = 0; r2 < S[2] && rc == kOk; ++r2) {
        const Axis a = axis_class(0, r0), b = axis_class(1, r1), c = axis_class(2, r2);
        if (a.n == 0 || b.n == 0 || c.n == 0 || a.out * b.out * c.out == 0) continue;
        const int64_t nw = (int64_t)a.n * b.n * c.n * g.Co * g.Ci;
        cudaError_t e = launch_pdl(
            bwdi_class_weights<T>, dim3((unsigned)std::min<int64_t>(ceil_div(nw, 256), 1024)),
            dim3(256), 0, s, w, w2, a.n, b.n, c.n, a.base, b.base, c.base, a.mul, b.mul, c.mul,
            (int)g.KR, (int)g.KD, (int64_t)g.Ci, (int64_t)g.Co);
        if (e == cudaSuccess) e = cudaGetLastError();
        note_launch();
        if (e != cudaSuccess) {
          rc = cuda_fail(e, "bwdi_class_weights");
          break;
        }
        ConvGeom gc{};
        gc.B = g.B;
        gc.IC = g.OC; gc.IR = g.OR; gc.ID = g.OD; gc.Ci = g.Co;
        gc.KC = a.n; gc.KR = b.n; gc.KD = c.n;
        gc.OC = a.out; gc.OR = b.out; gc.OD = c.out; gc.Co = g.Ci;
        gc.sc = gc.sr = gc.sd = 1;
        gc.dc = a.dil; gc.dr = b.dil; gc.dd = c.dil;
        gc.pc = a.pad; gc.pr = b.pad; gc.pd = c.pad;
        Dev d = make_dev(gc, FWD);
        d.ystrided = 1;
        d.ysb = g.IC * g.IR * g.ID;
        d.ysc = (int64_t)S[0] * g.IR * g.ID;
        d.ysr = (int64_t)S[1] * g.ID;
        d.ysd = S[2];
        d.yoff = ((int64_t)r0 * g.IR + r1) * g.ID + r2;
        rc = launch_any<T, FWD>(d, dy, w2, dx, 1, d.K, s);
      }
  scratch_free(w2, s);
  return rc;
}

// The GEMM view of one pass with its reduction split across CTAs: each
// split writes a partial, summed in split order by a second kernel
// (deterministic).  A/B are the pass's operands in launch_any's order.
// A bias (per column) and activation, if any, are applied to the finished sums.
template <typename T, int MODE>
int splitk_t(Dtype dt, const ConvGeom &g, const T *A, const T *B, T *C, cudaStream_t s,
             const void *bias = nullptr, int act = 0) {
  Dev d = make_dev(g, MODE);
  if (d.M == 0 || d.N == 0) return kOk;
  if (d.K == 0) {
    OWL_CUDA(cudaMemsetAsync(C, 0, sizeof(T) * d.M * d.N, s));
    return kOk;
  }
  // Split the reduction so that ~4 waves of CTAs cover 152 SMs, with
  // each split at least 8 K-tiles deep.  A small result is worth more splits (one
  // tile's CTAs are all there are: [256;28;28;1] x [5;5;1;32] 55 us with 256 of them,
  // 40 with 598, their sums 5.5 and 10).
  int64_t tiles = ceil_div(d.M, tile_m<T>(d)) * ceil_div(d.N, tile_n<T>(d));
  int64_t want = ceil_div(4 * 152, tiles);
  int64_t max_by_k = ceil_div(d.K, 64);
  const int64_t most = d.M * d.N <= 4096 ? 4 * 152 : 256;
  int splits = (int)std::max<int64_t>(1, std::min<int64_t>(want, std::min<int64_t>(max_by_k, most)));
  int64_t kps = ceil_div(ceil_div(d.K, splits), 16) * 16;
  splits = (int)ceil_div(d.K, kps);
  if (splits == 1) {
    if (MODE == FWD) {
      d.bias = bias;
      d.act = act;
    }
    int rc = launch_any<T, MODE>(d, A, B, C, 1, kps, s);
    if (rc || MODE == FWD || (!bias && act == OWLGPU_ACT_NONE)) return rc;
    return bias_act_inplace(dt, C, bias, d.M * d.N, d.N, act, s);
  }
  void *ws = nullptr;
  size_t bytes = sizeof(T) * (size_t)splits * d.M * d.N;
  int rc = scratch_alloc(&ws, bytes, s);
  if (rc) return rc;
  rc = launch_any<T, MODE>(d, A, B, (T *)ws, splits, kps, s);
  if (rc == kOk) {
    rc = sum_splits<T>((const T *)ws, C, d.M * d.N, splits, (const T *)bias, d.N, act, s);
  }
  scratch_free(ws, s);
  return rc;
}

template <typename T>
int bwdk_t(Dtype dt, const ConvGeom &g, const T *x, T *dw, const T *dy, cudaStream_t s) {
  return splitk_t<T, BWDK>(dt, g, x, dy, dw, s);
}

// backward_kernel, float32, with the split-K partials written into a
// caller-provided workspace of `ws_elems` floats instead of an allocation.
// The split count is capped so that splits * |dW| fits the workspace; every
// partial element is written before it is read, so the workspace needs no
// clearing between calls.
int bwdk_f32_into(const ConvGeom &g, const float *x, float *dw, const float *dy, float *ws,
                  int64_t ws_elems, cudaStream_t s) {
  Dev d = make_dev(g, BWDK);
  if (d.M == 0 || d.N == 0) return kOk;
  if (d.K == 0) {
    OWL_CUDA(cudaMemsetAsync(dw, 0, sizeof(float) * d.M * d.N, s));
    return kOk;
  }
  int64_t tiles = ceil_div(d.M, tile_m<float>(d)) * ceil_div(d.N, tile_n<float>(d));
  int64_t want = ceil_div(4 * 152, tiles);
  int64_t max_by_k = ceil_div(d.K, 64);
  int64_t max_by_ws = ws_elems / (d.M * d.N);
  int splits = (int)std::max<int64_t>(
      1, std::min<int64_t>(std::min<int64_t>(want, max_by_ws), std::min<int64_t>(max_by_k, 256)));
  int64_t kps = ceil_div(ceil_div(d.K, splits), 16) * 16;
  splits = (int)ceil_div(d.K, kps);
  if (splits == 1) return launch_any<float, BWDK>(d, x, dy, dw, 1, kps, s);
  int rc = launch_any<float, BWDK>(d, x, dy, ws, splits, kps, s);
  if (rc != kOk) return rc;
  return sum_splits<float>(ws, dw, d.M * d.N, splits, nullptr, d.N, 0, s);
}

}  // namespace

int simt_conv_bwd_kernel_f32_into(const ConvGeom &g, const float *x, float *dw,
                                  const float *dy, float *ws, int64_t ws_elems,
                                  cudaStream_t s) {
  return bwdk_f32_into(g, x, dw, dy, ws, ws_elems, s);
}

// Element type of each Dtype: float, double, and the complex pairs (whose
// tiles are those of double: 8- and 16-byte elements).
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

int simt_conv_fwd(Dtype dt, const ConvGeom &g, const void *x, const void *w, void *y,
                  cudaStream_t s, const void *bias, int act) {
  if (g.taps() * g.Ci == 0 && g.y_elems() > 0 && (bias || act != OWLGPU_ACT_NONE)) {
    const int rc = simt_conv_fwd(dt, g, x, w, y, s, nullptr, OWLGPU_ACT_NONE);
    return rc ? rc : bias_act_inplace(dt, y, bias, g.y_elems(), g.Co, act, s);
  }
  return by_dtype(dt, [&](auto *tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    return fwd_t<T>(g, (const T *)x, (const T *)w, (T *)y, s, bias, act);
  });
}

int simt_conv_bwd_input(Dtype dt, const ConvGeom &g, void *dx, const void *w, const void *dy,
                        cudaStream_t s) {
  return by_dtype(dt, [&](auto *tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    return bwdi_t<T>(g, (T *)dx, (const T *)w, (const T *)dy, s);
  });
}

// A pass of a 1x1 geometry as a split-K GEMM (the dense layer's products on
// the CUDA cores): mode 0 forward (a = x, b = w, c = y), 1 backward_input
// (a = dy, b = w, c = dx), 2 backward_kernel (a = x, b = dy, c = dw).
// `bias` (per column of c, or null) and `act` are applied to the product.
int simt_gemm(Dtype dt, int mode, const ConvGeom &g, const void *a, const void *b, void *c,
              cudaStream_t s, const void *bias, int act) {
  if (dt != F32 && dt != F64) {
    set_error("simt_gemm: real element kinds only");
    return kErrInvalid;
  }
  return by_dtype(dt, [&](auto *tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    if (mode == FWD)
      return splitk_t<T, FWD>(dt, g, (const T *)a, (const T *)b, (T *)c, s, bias, act);
    if (mode == BWDI)
      return splitk_t<T, BWDI>(dt, g, (const T *)a, (const T *)b, (T *)c, s, bias, act);
    return splitk_t<T, BWDK>(dt, g, (const T *)a, (const T *)b, (T *)c, s, bias, act);
  });
}

int simt_conv_bwd_kernel(Dtype dt, const ConvGeom &g, const void *x, void *dw, const void *dy,
                         cudaStream_t s) {
  return by_dtype(dt, [&](auto *tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    return bwdk_t<T>(dt, g, (const T *)x, (T *)dw, (const T *)dy, s);
  });
}

}  // namespace owlgpu
