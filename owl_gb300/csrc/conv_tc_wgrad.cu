// conv_tc_wgrad.cu -- tcgen05 backward-kernel (weight gradient) for float32
// data in BF16 or split-BF16 precision (a TF32 request runs split-BF16),
// strides up to 8, any dilation, 2-D/3-D.
//
//   dW[t][ci][co] = sum over output pixels p of X[p + off(t)][ci] * dY[p][co]
//
// Per tap this is a GEMM with M = ci (128 per MMA), N = co (BN <= 256), and the
// reduction K running over output pixels.  Both operands are staged from the
// float32 activations by producer warps in the same [16-byte channel chunk]
// [pixel][16 B] layout as the forward kernel's halo.  Read MN-major, 8
// consecutive pixels x 8 channels of that layout form one core matrix, so
// every tap of a tap group reads the same X halo through a shifted descriptor
// and all of them share one staged dY tile.  Taps are grouped by phase
// (k*d mod s per dimension), so a strided convolution's halo holds only the
// input rows and columns its group reads: a quarter of the footprint at
// stride 2 in 2-D.
//
// Work split: a CTA owns (tap group, ci block, co block, pixel range).  It
// accumulates the group's taps in TMEM (TG * BN columns) over all the pixel
// tiles of its range, then writes the partial dW of its range.  A second
// kernel sums the ranges in a fixed order, so the result is deterministic.
// CTAs that share a pixel range are launched next to each other, so the
// activations they re-read come from L2.
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "../../include/owlgpu.h"
#include "common.cuh"
#include "reduce.cuh"
#include "tc_ptx.cuh"
#include "tc_stage.cuh"

namespace owlgpu {
namespace {

using namespace ptx;

// Warp roles.  The accumulator is drained once per CTA, after the last
// pixel tile, so every warp but the MMA issuer (warp 0) stages operands;
// warps 4-15, three per TMEM lane quadrant, then drain the accumulator (8.7 us
// of [64;56;56;128]x[3;3;128;128] with one per quadrant).
// (Measured on GB300: 15 producer warps beat 9 or 12 here even though three
// of them share the MMA warp's scheduler.)
constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kMmaWarp = 0;
constexpr int kEpiWarp0 = 4, kEpiParts = (kWarps - kEpiWarp0) / 4;
constexpr int kProducerWarps = kWarps - 1;
__device__ __forceinline__ int producer_index(int warp) { return warp - 1; }
constexpr int kSmemMax = 232448;
// Taps are grouped through a table in the launch parameters when the
// convolution is strided (and, up to this many taps, always).
constexpr int kMaxOrderedTaps = 256;
constexpr long long kSpinLimit = 4000000000LL;

enum Kind { K_BF16 = 0, K_TF32 = 1, K_BF16X3 = 2 };

struct WgParams {
  const float *x, *dy;
  float *out;
  int *status;
  int B, IW, IU, IV, OW, OU, OV, KW, KU, KV, dw, du, dv, pw, pu, pv, sw, su, sv;
  long long xsb, xsw, xsu, xsv, ysb, ysw, ysu, ysv;
  int Ci, Co, T, TG, n_tg, BN, n_nb, n_mb, R;
  int TU, TP;             // reduction tile: TU output rows (u) x 8 columns (v) = TP pixels
  int YPS;                // dY plane stride in pixels: TP + 1, so that the 16-byte chunks
                          // of one pixel fall in different shared-memory banks
  int u_tiles, v_tiles;
  long long total_tiles, tiles_per_range;
  int n_tab;              // pixels of the largest X halo and the dY tile (the LANES tables)
  int PS;                 // X halo plane stride in pixels (max over groups)
  unsigned x_bytes, y_bytes;  // per stage, per precision part
  int NS;
  unsigned idesc, tmem_cols;
  unsigned small_off;  // BF16X3: TMEM column of the cross-term accumulators
  // Accumulator sets, set_cols = TG * BN TMEM columns each: the pixel tiles go to them in
  // turn and the epilogue adds them.  The tensor core rounds an accumulator toward zero at
  // every MMA, so the error of a sum grows with its length, and sets shorten it for
  // nothing.  (BF16X3's cross terms hold 2^-8 of a sum and have one set, the last.)
  int sets;
  unsigned set_cols;
  int vec_x, vec_y;
  int pk_nch;  // PACK: chunk rows of a halo row (a power of two), else 16
  // LANES: floats from a tile's first pixel to the next tile's along v; from there
  // to the next row of tiles; and so on along w and b
  long long x_dv, x_du, x_dw, x_db, y_dv, y_du, y_dw, y_db;
  // Tap groups.  ordered: group g holds taps tap_order[gstart[g] ..
  // gstart[g+1]); else group g holds taps g*TG .. min(T, (g+1)*TG) - 1.
  // Every group is phase-uniform: all its taps have the same k*d mod s in
  // each dimension, so its X halo needs only input rows and columns of
  // that phase (every s-th one).
  long long spin_limit;  // cycles a pipeline wait polls before the CTA gives up
  int ordered;
  unsigned short tap_order[kMaxOrderedTaps];
  unsigned short gstart[kMaxOrderedTaps + 1];
};

__device__ int g_tc_status_wg;

__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                         int *status, long long limit) {
  if (mbar_try_wait(bar, parity)) return true;
  long long t0 = clock64();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > limit) {
      *abort_flag = 1;
      atomicExch(status, 1);
      return false;
    }
  }
}

// A producer warp's: the same answer for all its lanes (they arrive together).
__device__ __forceinline__ bool wait_bar_warp(uint32_t bar, uint32_t parity,
                                              volatile int *abort_flag, int *status,
                                              long long limit) {
  return __all_sync(0xffffffffu, wait_bar(bar, parity, abort_flag, status, limit));
}

// The MMA warp's: polled by the whole warp.
__device__ __forceinline__ bool poll_bar(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                         int *status, long long limit) {
  if (mbar_test_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_test_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > limit) {
      *abort_flag = 1;
      atomicExch(status, 1);
      return false;
    }
  }
  return true;
}

// Pixels from one chunk row of a packed X stage to the next: as many as a halo row
// has, or the few more that put the 16-byte chunks that eight lanes store together
// into different banks.
__host__ __device__ inline int chunk_row(int hvr, int nch) {
  const int step = 8 / nch > 0 ? 8 / nch : 1;  // nch rows x step pixels
  while (nch > 1 && (hvr % (2 * step)) != step) ++hvr;
  return hvr;
}

// LANES: the operands are staged as whole 32-byte chunks (both arrays 32-byte
// aligned, their channels multiples of 8), else element by element where needed.
// PACK: at most 64 input channels, of which an MMA's 128 rows hold
// those of several taps, ku, ku + su, ..: the X stage keeps, halo row after halo row,
// `pk` chunk rows of PSR pixels, so that one stride of PSR pixels walks the chunks of
// a halo row and on into the next one's, the next tap's operand.  With a tap to an
// MMA, 32 channels used a quarter of each: [4;32;32;32;32]x[3;3;3;32;64] took 77 us.
// SETS: several accumulator sets may be in use (a kernel of its own for whole chunks,
// where the choice in the loops cost layers with one set 1 to 3 %).
template <int KIND, bool LANES, bool PACK, bool SETS>
__global__ void __launch_bounds__(kThreads, 1) wgrad_tc_kernel(const __grid_constant__ WgParams p) {
  constexpr int EB = (KIND == K_TF32) ? 4 : 2;
  constexpr int EPC = 16 / EB;
  constexpr int PARTS = (KIND == K_BF16X3) ? 2 : 1;
  constexpr int XPL = 128 * EB / 16;  // planes for 128 input channels
  constexpr int KSTEP_PIX = 32 / EB;  // pixels per MMA (K = 16 bf16 / 8 tf32)
  // BF16X3: the cross terms (hi*lo + lo*hi) accumulate apart from the hi*hi
  // sums and are added in the epilogue.  The tensor core rounds its FP32
  // accumulator toward zero after every MMA; with all three MMAs of a K step
  // in one accumulator that rounding is three times that of the hi*hi sums.
  constexpr bool SEP = (KIND == K_BF16X3);
  extern __shared__ __align__(1024) uint8_t smem[];
  // a programmatic dependent of the work before it: wait for that work (X
  // and dY may be its output) before any global access
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // (the shuffle shows the compiler that a warp takes one side of the role branches
  // as a whole: the MMA loop keeps its descriptors in uniform registers)
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int YPL = p.BN * EB / 16;

  // ---- work unit of this CTA ----
  unsigned u = blockIdx.x;
  const int tg = (int)(u % (unsigned)p.n_tg); u /= (unsigned)p.n_tg;
  const int nb = (int)(u % (unsigned)p.n_nb); u /= (unsigned)p.n_nb;
  const int mb = (int)(u % (unsigned)p.n_mb);
  const int r = (int)(u / (unsigned)p.n_mb);
  const long long t_begin = (long long)r * p.tiles_per_range;
  const long long t_end = min(p.total_tiles, t_begin + p.tiles_per_range);
  const int gbeg = p.ordered ? (int)p.gstart[tg] : tg * p.TG;
  const int ntap = p.ordered ? (int)p.gstart[tg + 1] - gbeg : min(p.TG, p.T - gbeg);
  // (PACK: the first tap of each pack)
  auto tap_of = [&](int i) { return p.ordered ? (int)p.tap_order[gbeg + i] : gbeg + i; };
  const int pk = p.pk_nch, pk_taps = PACK ? XPL / pk : 1;

  // bounding box of this group's tap offsets -> halo extents
  int minw = 1 << 30, minu = 1 << 30, minv = 1 << 30, maxw = -1, maxu = -1, maxv = -1;
  for (int i = 0; i < ntap; ++i) {
    const int t = tap_of(i);
    const int kv = t % p.KV, ku = (t / p.KV) % p.KU, kw = t / (p.KV * p.KU);
    minw = min(minw, kw * p.dw); maxw = max(maxw, kw * p.dw);
    minu = min(minu, ku * p.du);
    maxu = max(maxu, (PACK ? ku + min(pk_taps - 1, (p.KU - 1 - ku) / p.su) * p.su : ku) * p.du);
    minv = min(minv, kv * p.dv); maxv = max(maxv, kv * p.dv);
  }
  // X halo of a phase-uniform group: input rows and columns of the group's
  // phase only, so halo row (hw, hu) is input (minw + hw*sw, minu + hu*su)
  // relative to the tile origin, and its HVR pixels are every sv-th input
  // column: 8 consecutive output columns are 8 consecutive stored pixels.
  const int HW = (maxw - minw) / p.sw + 1, HU = p.TU + (maxu - minu) / p.su;
  const int HVR = 8 + (maxv - minv) / p.sv;
  // PACK: pixels from a chunk row to the next, and from a halo row to the next; else
  // pixels from one chunk plane to the next, and the halo rows lie in one plane
  const int PSR = PACK ? chunk_row(HVR, pk) : p.PS, row_px = PACK ? pk * PSR : HVR;
  // X halo rows; when both operand tiles have at most one row per producer
  // warp, each warp stages its X row and dY row together in a single pass
  const int xrows = HW * HU;
  const int nch = PACK ? pk : XPL;  // chunks of X staged element by element
  const bool paired = xrows <= kProducerWarps && p.TU <= kProducerWarps &&
                      HVR * nch <= 32 * 5 && 8 * YPL <= 32 * 4;

  uint8_t *xs = smem;
  uint8_t *ys = smem + (size_t)p.NS * PARTS * p.x_bytes;
  uint64_t *bars = reinterpret_cast<uint64_t *>(ys + (size_t)p.NS * PARTS * p.y_bytes);
  uint64_t *full = bars;
  uint64_t *empty = full + p.NS;
  uint64_t *acc_full = empty + p.NS;
  uint64_t *drain = acc_full + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  uint32_t *tap_off = tmem_slot + 2;  // per-tap start pixel in the X halo (16-byte units)

  for (int i = threadIdx.x; i < ntap; i += blockDim.x) {
    const int tt = tap_of(i);
    const int kv = tt % p.KV, ku = (tt / p.KV) % p.KU, kw = tt / (p.KV * p.KU);
    tap_off[i] =
        (uint32_t)((((kw * p.dw - minw) / p.sw) * HU + (ku * p.du - minu) / p.su) * row_px +
                   (kv * p.dv - minv) / p.sv);
  }

  // LANES: where the tile's pixels lie, X's then dY's: {offset in floats from the
  // tile's first pixel, position}, and one past the end that is outside any bounds
  int2 *xtab = reinterpret_cast<int2 *>((reinterpret_cast<uintptr_t>(tap_off + p.TG) + 7) &
                                        ~(uintptr_t)7);
  int2 *ytab = xtab + xrows * HVR + 1;
  uint16_t *xdst = reinterpret_cast<uint16_t *>(ytab + p.TP + 1);  // PACK: places in the stage
  if (LANES) {
    const int n = xrows * HVR, out = (int)(stage::position(stage::kMaxV + 1, 0, 0) | stage::kGuard);
    for (int i = threadIdx.x; i <= n; i += blockDim.x) {
      const int hv = i % HVR, hu = (i / HVR) % HU, hw = i / (HVR * HU);
      if (PACK && i < n) xdst[i] = (uint16_t)(i / HVR * row_px + hv);
      xtab[i] =
          i < n ? make_int2((int)((hw * p.sw * p.xsw + hu * p.su * p.xsu + hv * p.sv * p.xsv) * p.Ci),
                            (int)(stage::position(hv * p.sv, hu * p.su, hw * p.sw) | stage::kGuard))
                : make_int2(0, out);
    }
    for (int i = threadIdx.x; i <= p.TP; i += blockDim.x)
      ytab[i] = i < p.TP ? make_int2((int)((i / 8 * p.ysu + i % 8 * p.ysv) * p.Co),
                                     (int)(stage::position(i % 8, i / 8, 0) | stage::kGuard))
                         : make_int2(0, out);
  }

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.NS; ++i) {
      mbar_init(smem_u32(&full[i]), kProducerWarps);
      mbar_init(smem_u32(&empty[i]), 1);
    }
    mbar_init(smem_u32(acc_full), 1);
    mbar_init(smem_u32(drain), 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int pidx = producer_index(warp);
  if (warp != kMmaWarp) {
    // ===================== producers: X halo + dY tile =====================
    bool staged = true;
    // The tile's position and the ring's stage advance by counting: every warp
    // decodes every tile, and the 64-bit divisions there took 14 of 128 us on
    // [64;56;56;128] x [3;3;128;128].
    int v0, u0, ow, b;
    {
      long long q = t_begin;
      v0 = (int)(q % p.v_tiles) * 8; q /= p.v_tiles;
      u0 = (int)(q % p.u_tiles) * p.TU; q /= p.u_tiles;
      ow = (int)(q % p.OW);
      b = (int)(q / p.OW);
    }
    const int v_end = p.v_tiles * 8, u_end = p.u_tiles * p.TU;
    auto next_tile = [&]() {
      if ((v0 += 8) == v_end) {
        v0 = 0;
        if ((u0 += p.TU) == u_end) {
          u0 = 0;
          if (++ow == p.OW) {
            ow = 0;
            ++b;
          }
        }
      }
    };
    int st = 0;
    uint32_t ph = 1;
    if constexpr (LANES) {
      // The chunks that exist are staged (the planes past the channels stay as they
      // are: they only reach accumulator rows and columns that are not stored): a
      // lane keeps one chunk of each operand and takes every lanes/chunks-th pixel of
      // the tile, QX of X and QY of dY a round (one round for most tiles).  Where a
      // pixel lies relative to its tile comes from a table, the tile's pointers
      // advance by constant steps and only tiles at the array's edge test their
      // pixels: with row and pixel arithmetic in the loop it took 610 instructions a
      // warp and tile (54% of the issue slots), with conversion and stores some 80 of
      // them.  The loads of one operand are in flight while the other is converted
      // and stored, the next round's (or tile's) X while this one's dY: issued
      // together and then waited for they cost a round trip, in all warps at once.
      const int id = pidx * 32 + lane;
      const int nchx = min(XPL, (p.Ci - mb * 128 + 7) / 8), nchy = min(YPL, (p.Co - nb * p.BN + 7) / 8);
      const int lgx = 32 - __clz(nchx - 1), lgy = 32 - __clz(nchy - 1);  // (clz(0) = 32)
      const int jx = id & ((1 << lgx) - 1), jy = id & ((1 << lgy) - 1);
      const int px = id >> lgx, dpx = (kProducerWarps * 32) >> lgx, npx = xrows * HVR;
      const int py = id >> lgy, dpy = (kProducerWarps * 32) >> lgy, npy = p.TP;
      const bool onx = jx < nchx, ony = jy < nchy;  // (others load chunk 0 and store nothing)
      const int rounds_x = (npx + dpx - 1) / dpx, rounds_y = (npy + dpy - 1) / dpy;
      const uint32_t lane_x = (uint32_t)(jx * PSR + (PACK ? 0 : px)) * 16u, lane_y = (uint32_t)(jy * p.YPS + py) * 16u;
      int iw0 = ow * p.sw - p.pw + minw, iu0 = u0 * p.su - p.pu + minu, iv0 = v0 * p.sv - p.pv + minv;
      const float *xt = p.x + ((long long)b * p.xsb + (long long)iw0 * p.xsw + (long long)iu0 * p.xsu +
                               (long long)iv0 * p.xsv) * p.Ci + mb * 128 + (onx ? jx * 8 : 0);
      const float *yt = p.dy + ((long long)b * p.ysb + (long long)ow * p.ysw + (long long)u0 * p.ysu +
                                (long long)v0 * p.ysv) * p.Co + nb * p.BN + (ony ? jy * 8 : 0);
      // the parts of the tile that lie inside the arrays: along u and w, then along v too
      unsigned x_lo, x_hi, y_lo, y_hi;
      auto rows_in = [&] {
        unsigned l, h;
        stage::field(iu0, p.IU, stage::kMaxU, l, h);
        x_lo = l << 11;
        x_hi = h << 11;
        stage::field(iw0, p.IW, stage::kMaxW, l, h);
        x_lo |= l << 22;
        x_hi |= h << 22;
        stage::field(u0, p.OU, stage::kMaxU, l, h);
        y_lo = l << 11;
        y_hi = h << 11;
      };
      rows_in();
      auto stage_tiles = [&](auto qx, auto qy) {
        constexpr int QX = qx.value, QY = qy.value;
        float vx[QX][8], vy[QY][8];
        long long left = t_end - t_begin;
        int k = 0;
        auto load_x = [&] {
          unsigned l, h;
          stage::field(iv0, left > 0 ? p.IV : -p.IV, stage::kMaxV, l, h);
          stage::table_load<QX>(xtab, px + k * dpx * QX, dpx, npx, xt, x_lo | l, x_hi | h, vx);
        };
        load_x();
        while (left > 0) {
          {
            unsigned l, h;
            stage::field(v0, p.OV, stage::kMaxV, l, h);
            stage::table_load<QY>(ytab, py + k * dpy * QY, dpy, npy, yt, y_lo | l, y_hi | h, vy);
          }
          if (k == 0 &&
              !wait_bar_warp(smem_u32(&empty[st]), ph, abort_flag, p.status, p.spin_limit)) {
            staged = false;
            break;
          }
          const int kx = k * dpx * QX, ky = k * dpy * QY;
          uint8_t *yd = ys + (uint32_t)st * PARTS * p.y_bytes + lane_y + (uint32_t)ky * 16u;
          const int ny = ony ? npy - py - ky : 0;
          uint8_t *xd = xs + (uint32_t)st * PARTS * p.x_bytes + lane_x;
          const int nx = onx ? npx - px - kx : 0;
          if (PACK)
            stage::table_store_at<KIND, QX>(xd, xdst + px + kx, dpx, p.x_bytes, nx, vx);
          else
            stage::table_store<KIND, QX>(xd + (uint32_t)kx * 16u, dpx, p.x_bytes, nx, vx);
          ++k;
          const bool last = k * QX >= rounds_x && k * QY >= rounds_y;  // the tile's last round
          if (last) {
            k = 0;
            --left;
            v0 += 8;
            iv0 += 8 * p.sv;
            xt += p.x_dv;
            yt += p.y_dv;
            if (v0 == v_end) {
              v0 = 0;
              u0 += p.TU;
              xt += p.x_du;
              yt += p.y_du;
              if (u0 == u_end) {
                u0 = 0;
                xt += p.x_dw;
                yt += p.y_dw;
                if (++ow == p.OW) {
                  ow = 0;
                  xt += p.x_db;
                  yt += p.y_db;
                }
              }
              iw0 = ow * p.sw - p.pw + minw;
              iu0 = u0 * p.su - p.pu + minu;
              iv0 = minv - p.pv;
              rows_in();
            }
          }
          load_x();
          stage::table_store<KIND, QY>(yd, dpy, p.y_bytes, ny, vy);
          if (last) {
            fence_proxy_async();
            mbar_arrive_warp(smem_u32(&full[st]), lane);
            if (++st == p.NS) { st = 0; ph ^= 1; }
          }
        }
      };
      // tiles of few pixels (or channels): fewer slots, each of which costs its
      // instructions whether the tile has a pixel for it or not
      if (rounds_x <= 3 && rounds_y <= 3)
        stage_tiles(std::integral_constant<int, 3>{}, std::integral_constant<int, 3>{});
      else
        stage_tiles(std::integral_constant<int, 5>{}, std::integral_constant<int, 4>{});
    } else {
      for (long long t = t_begin; t < t_end; ++t, next_tile()) {
        if (!wait_bar_warp(smem_u32(&empty[st]), ph, abort_flag, p.status, p.spin_limit)) {
          staged = false;
          break;
        }
        uint8_t *xd = xs + (size_t)st * PARTS * p.x_bytes;
        uint8_t *yd = ys + (size_t)st * PARTS * p.y_bytes;
        // X halo: rows (w, u) of HVR pixels x 128 channels of ci block mb;
        // dY tile: TU rows (u) of 8 output pixels x BN channels of co block nb.
        const int xcb = mb * 128, ycb = nb * p.BN;
        auto xrow = [&](int r) {
          const int hu = r % HU, hw = r / HU;
          const int iw = ow * p.sw - p.pw + minw + hw * p.sw;
          const int iu = u0 * p.su - p.pu + minu + hu * p.su;
          const int ivs = v0 * p.sv - p.pv + minv;
          stage::Row row;
          row.ok = iw >= 0 && iw < p.IW && iu >= 0 && iu < p.IU;
          row.rowp = p.x + ((long long)b * p.xsb + (long long)iw * p.xsw + (long long)iu * p.xsu +
                            (long long)ivs * p.xsv) * p.Ci + xcb;
          row.pstep = (long long)p.sv * p.xsv * p.Ci;
          row.vfirst = ivs;
          row.vstride = p.sv;
          row.vlim = p.IV;
          return row;
        };
        auto yrow = [&](int r) {
          const int ou = u0 + r;
          stage::Row row;
          row.ok = ou < p.OU;
          row.rowp = p.dy + ((long long)b * p.ysb + (long long)ow * p.ysw + (long long)ou * p.ysu +
                             (long long)v0 * p.ysv) * p.Co + ycb;
          row.pstep = p.ysv * p.Co;
          row.vfirst = v0;
          row.vstride = 1;
          row.vlim = p.OV;
          return row;
        };
        if (paired) {
          // at most one row of each per warp: both rows in one pass
          stage::RowSet sx{xd, p.x_bytes, (uint32_t)PSR * 16, xrows, HVR, row_px, nch, p.Ci - xcb};
          stage::RowSet sy{yd, p.y_bytes, (uint32_t)p.YPS * 16, p.TU, 8, 8, YPL, p.Co - ycb};
          stage::stage_rows2<KIND, EPC, 5, 4>(sx, xrow, sy, yrow, min(p.vec_x, p.vec_y),
                                              pidx, kProducerWarps, lane);
        } else {
          stage::stage_rows<KIND, EPC, 6>(xd, p.x_bytes, (uint32_t)PSR * 16, xrows, HVR, row_px, nch,
                                          p.Ci - xcb, p.vec_x, pidx, kProducerWarps, lane,
                                          xrow);
          stage::stage_rows<KIND, EPC, 4>(yd, p.y_bytes, (uint32_t)p.YPS * 16, p.TU, 8, 8, YPL,
                                          p.Co - ycb, p.vec_y, pidx, kProducerWarps, lane,
                                          yrow);
        }
        fence_proxy_async();
        mbar_arrive_warp(smem_u32(&full[st]), lane);
        if (++st == p.NS) { st = 0; ph ^= 1; }
      }
    }
    if (staged && warp >= kEpiWarp0) {
      // ===================== epilogue: TMEM -> partial dW =====================
      // (a warp reaches the TMEM lanes of its quadrant, warp % 4; the quadrant's
      // warps take every kEpiParts-th 16 columns)
      const int q = warp & 3;
      const int n_sets = (int)min((long long)p.sets, t_end - t_begin);
      int mine = (warp - kEpiWarp0) >> 2;
      const int row = q * 32 + lane, pt = PACK ? row / (pk * 8) : 0;  // tap of the pack
      const int ci = PACK ? row - pt * pk * 8 : mb * 128 + row;
      if (wait_bar(smem_u32(acc_full), 0, abort_flag, p.status, p.spin_limit)) {
        tc_fence_after();
        for (int i = 0; i < ntap; ++i) {
          const int tt = tap_of(i) + pt * p.su * p.KV;
          const bool real =
              ci < p.Ci && (!PACK || tap_of(i) / p.KV % p.KU + pt * p.su < p.KU);
          float *out = p.out + (((long long)r * p.T + tt) * p.Ci + ci) * p.Co + nb * p.BN;
          const uint32_t tcol = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(i * p.BN);
          for (int c0 = 0; c0 < p.BN; c0 += 16) {
            if (mine != 0) {
              --mine;
              continue;
            }
            mine = kEpiParts - 1;
            uint32_t rr[16], r2[16];
            auto add = [](uint32_t(&a)[16], const uint32_t(&b)[16]) {
#pragma unroll
              for (int e = 0; e < 16; ++e)
                a[e] = __float_as_uint(__uint_as_float(a[e]) + __uint_as_float(b[e]));
            };
            tmem_ld16(tcol + (uint32_t)c0, rr);
            if (SEP) tmem_ld16(tcol + p.small_off + (uint32_t)c0, r2);
            tmem_ld_wait();
            for (int k = 1; SETS && k < n_sets; ++k) {
              uint32_t more[16];
              tmem_ld16(tcol + (uint32_t)k * p.set_cols + (uint32_t)c0, more);
              tmem_ld_wait();
              add(rr, more);
            }
            if (SEP) add(rr, r2);
            if (real) {
              const int n0 = nb * p.BN + c0;
              if (p.vec_y == 2 && n0 + 16 <= p.Co && ((uintptr_t)(out + c0) % 32 == 0)) {
                stage::st8(out + c0, rr);
                stage::st8(out + c0 + 8, rr + 8);
              } else if (p.vec_y && n0 + 16 <= p.Co && ((uintptr_t)(out + c0) % 16 == 0)) {
#pragma unroll
                for (int e = 0; e < 16; e += 4)
                  *reinterpret_cast<float4 *>(out + c0 + e) =
                      make_float4(__uint_as_float(rr[e]), __uint_as_float(rr[e + 1]),
                                  __uint_as_float(rr[e + 2]), __uint_as_float(rr[e + 3]));
              } else {
#pragma unroll
                for (int e = 0; e < 16; ++e)
                  if (n0 + e < p.Co) out[c0 + e] = __uint_as_float(rr[e]);
              }
            }
          }
        }
        tc_fence_before();
      }
    }
  } else {
    // ===================== MMA issuer =====================
    {
      const uint32_t lead = elect_one();
      const uint32_t x0 = smem_u32(xs), y0 = smem_u32(ys);
      const uint32_t a_lbo = (uint32_t)row_px * 16, a_sbo = (uint32_t)PSR * 16;
      const uint32_t b_lbo = 128, b_sbo = (uint32_t)p.YPS * 16;
      const uint32_t xlo16 = p.x_bytes >> 4, ylo16 = p.y_bytes >> 4;
      // per K step: 16 pixels = two halo rows further into the X halo, 16
      // pixels further into the dY tile (16-byte units)
      const uint32_t xk16 = (uint32_t)(KSTEP_PIX / 8) * (uint32_t)row_px;
      const int nks = p.TP / KSTEP_PIX;
      // up to four taps' A offsets in registers (the common tap groups)
      const bool few = ntap <= 4;
      uint32_t to[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) to[i] = i < ntap ? tap_off[i] : 0u;
      int st = 0;
      uint32_t ph = 0;
      uint32_t acc = 0, acc_s = 0;
      bool ok = true;
      int set = 0;
      const uint32_t small0 = tmem_base + p.small_off;
      for (long long t = t_begin; t < t_end; ++t) {
        uint32_t d0 = tmem_base;
        if (SETS) {
          acc = t - t_begin >= p.sets;  // the first tile of a set overwrites it
          d0 += (uint32_t)set * p.set_cols;
          if (++set == p.sets) set = 0;
        }
        uint32_t dc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) dc[i] = d0 + (uint32_t)(i * p.BN);
        if (!poll_bar(smem_u32(&full[st]), ph, abort_flag, p.status, p.spin_limit)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // descriptors advance by adds of 16-byte units (start-address field)
        const uint64_t xd_st = smem_desc(x0 + (uint32_t)st * PARTS * p.x_bytes, a_lbo, a_sbo);
        const uint64_t yd_st = smem_desc(y0 + (uint32_t)st * PARTS * p.y_bytes, b_lbo, b_sbo);
#pragma unroll 2
        for (int s = 0; s < nks; ++s) {
          const uint64_t bd = yd_st + (uint64_t)(s * KSTEP_PIX);
          const uint64_t xs_ = xd_st + (uint64_t)(s * xk16);
          if (few) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (i < ntap) {
                const uint64_t ad = xs_ + (uint64_t)to[i];
                if (KIND == K_TF32) {
                  mma_tf32(lead, dc[i], ad, bd, p.idesc, acc);
                } else {
                  mma_bf16(lead, dc[i], ad, bd, p.idesc, acc);
                  if (KIND == K_BF16X3) {
                    const uint32_t ds = SETS ? small0 + (uint32_t)(i * p.BN) : dc[i] + p.small_off;
                    mma_bf16(lead, ds, ad, bd + (uint64_t)ylo16, p.idesc, SETS ? acc_s : acc);
                    mma_bf16(lead, ds, ad + (uint64_t)xlo16, bd, p.idesc, 1);
                  }
                }
              }
            }
          } else {
            for (int i = 0; i < ntap; ++i) {
              const uint64_t ad = xs_ + (uint64_t)tap_off[i];
              const uint32_t d = d0 + (uint32_t)(i * p.BN);
              if (KIND == K_TF32) {
                mma_tf32(lead, d, ad, bd, p.idesc, acc);
              } else {
                mma_bf16(lead, d, ad, bd, p.idesc, acc);
                if (KIND == K_BF16X3) {
                  const uint32_t ds = SETS ? small0 + (uint32_t)(i * p.BN) : d + p.small_off;
                  mma_bf16(lead, ds, ad, bd + (uint64_t)ylo16, p.idesc, SETS ? acc_s : acc);
                  mma_bf16(lead, ds, ad + (uint64_t)xlo16, bd, p.idesc, 1);
                }
              }
            }
          }
          acc = acc_s = 1;
        }
        mma_commit(lead, smem_u32(&empty[st]));
        if (++st == p.NS) { st = 0; ph ^= 1; }
      }
      if (ok) mma_commit(lead, smem_u32(acc_full));
      mma_commit(lead, smem_u32(drain));
      long long t0 = clock64();
      while (!mbar_try_wait(smem_u32(drain), 0) && clock64() - t0 < kSpinLimit) {
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

// Estimated time of a plan in cycles, from a fit to 950 plans of twelve layers on
// GB300 (3% off on average; the choice needs the ratios only).  A tile costs its
// rounds of staging slots, its bytes and its MMAs, which overlap little; each wave
// of CTAs a start and an epilogue; the partial sums their writing and reading.
double estimate(const WgParams &p, int halo_pixels, int parts, long long ctas, int sms) {
  auto pow2 = [](int n) {
    int q = 1;
    while (q < n) q *= 2;
    return q;
  };
  const int nx = std::min(16, (p.Ci + 7) / 8), ny = std::min(p.BN / 8, (p.Co + 7) / 8);
  const int lanes = kProducerWarps * 32;
  const int rx = (halo_pixels * pow2(nx) + lanes - 1) / lanes,
            ry = (p.TP * pow2(ny) + lanes - 1) / lanes;
  const bool few = rx <= 3 && ry <= 3;
  const int rounds = few ? 1 : std::max((rx + 4) / 5, (ry + 3) / 4);
  const double mma = p.TG <= 4 ? 23 : 45;
  const double tile = rounds * (390 + (few ? 6 : 9) * (parts == 2 ? 135 : 132)) +
                      (halo_pixels * nx + p.TP * ny) * 32 / 115.0 +
                      p.TP / 16 * p.TG * (parts == 2 ? 3 : 1) * std::max(mma, 0.26 * p.BN);
  const double waves = (double)((ctas + sms - 1) / sms);
  const double sums = p.R > 1 ? 1.3e-3 * p.T * p.Ci * (double)p.Co * p.R : 0.0;
  return waves * ((double)p.tiles_per_range * tile + 25.0 * p.TG * p.BN * parts + 8e3) + sums;
}

int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 148;
}

int *status_word() {
  static int *p[64] = {nullptr};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return nullptr;
  if (!p[dev]) {
    void *q = nullptr;
    if (cudaGetSymbolAddress(&q, g_tc_status_wg) != cudaSuccess) return nullptr;
    p[dev] = static_cast<int *>(q);
  }
  return p[dev];
}

template <int KIND, bool LANES, bool PACK, bool SETS>
int launch(const WgParams &p, size_t smem, int grid, cudaStream_t s) {
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr[dev]) {
    OWL_CUDA(cudaFuncSetAttribute(wgrad_tc_kernel<KIND, LANES, PACK, SETS>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    attr[dev] = true;
  }
  cudaError_t e = launch_pdl(wgrad_tc_kernel<KIND, LANES, PACK, SETS>, dim3(grid), dim3(kThreads),
                             smem, s, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  note_launch();
  note_tc_launch();
  if (e != cudaSuccess) return cuda_fail(e, "wgrad_tc_kernel");
  return kOk;
}

}  // namespace

int *tc_wgrad_status_word() { return status_word(); }

// out[i] = sum_r part[r][i] for r = 0 .. R-1 in order (deterministic).
int sum_partials_f32(const float *part, float *out, long long n, int R, cudaStream_t s) {
  return sum_splits<float>(part, out, n, R, nullptr, 1, 0, s);
}

int tc_conv_bwd_kernel(int prec, const ConvGeom &g, const float *x, float *dw, const float *dy,
                       cudaStream_t s) {
  if (g.sc > 8 || g.sr > 8 || g.sd > 8) return kErrUnsupported;
  // The weight gradient reads both operands MN-major, which the TF32 MMA
  // kind does not accept here; a TF32 request runs the split-BF16 kernel,
  // whose error (~1e-5) is below TF32's (~1e-3).
  const int kind = (prec == OWLGPU_PREC_TF32 || prec == OWLGPU_PREC_BF16X3) ? K_BF16X3 : K_BF16;
  const int EB = kind == K_TF32 ? 4 : 2;
  const int parts = kind == K_BF16X3 ? 2 : 1;
  if (g.Ci == 0 || g.Co == 0 || g.taps() == 0) return kErrUnsupported;
  if (g.out_pixels() == 0) return kErrUnsupported;
  WgParams p{};
  p.x = x; p.dy = dy;
  p.B = (int)g.B;
  p.Ci = (int)g.Ci; p.Co = (int)g.Co;
  const bool flat = (g.ID == 1 && g.OD == 1 && g.KD == 1);
  if (flat) {
    p.IW = 1; p.IU = (int)g.IC; p.IV = (int)g.IR; p.OW = 1; p.OU = (int)g.OC; p.OV = (int)g.OR;
    p.KW = 1; p.KU = (int)g.KC; p.KV = (int)g.KR; p.dw = 1; p.du = g.dc; p.dv = g.dr;
    p.pw = 0; p.pu = g.pc; p.pv = g.pr;
    p.sw = 1; p.su = g.sc; p.sv = g.sr;
    p.xsw = 1; p.xsu = g.IR; p.xsv = 1; p.ysw = 1; p.ysu = g.OR; p.ysv = 1;
  } else {
    p.IW = (int)g.IC; p.IU = (int)g.IR; p.IV = (int)g.ID;
    p.OW = (int)g.OC; p.OU = (int)g.OR; p.OV = (int)g.OD;
    p.KW = (int)g.KC; p.KU = (int)g.KR; p.KV = (int)g.KD;
    p.dw = g.dc; p.du = g.dr; p.dv = g.dd; p.pw = g.pc; p.pu = g.pr; p.pv = g.pd;
    p.sw = g.sc; p.su = g.sr; p.sv = g.sd;
    p.xsw = g.IR * g.ID; p.xsu = g.ID; p.xsv = 1;
    p.ysw = g.OR * g.OD; p.ysu = g.OD; p.ysv = 1;
  }
  p.xsb = g.IC * g.IR * g.ID;
  p.ysb = g.OC * g.OR * g.OD;
  p.T = (int)g.taps();
  p.n_mb = (p.Ci + 127) / 128;
  // Tap order: taps sorted by phase class (k*d mod s in each dimension), in
  // tap order within a class, so that every group of consecutive taps of a
  // class reads only input rows and columns of one phase.  Unstrided
  // convolutions have a single class (the identity order).
  const bool strided = p.sw > 1 || p.su > 1 || p.sv > 1;
  if (strided && p.T > kMaxOrderedTaps) return kErrUnsupported;
  p.ordered = p.T <= kMaxOrderedTaps;
  int order[kMaxOrderedTaps], cls_begin[kMaxOrderedTaps + 1], n_cls = 0;
  if (p.ordered) {
    auto phase = [&](int t) {
      const int kv = t % p.KV, ku = (t / p.KV) % p.KU, kw = t / (p.KV * p.KU);
      return ((kw * p.dw % p.sw) * p.su + ku * p.du % p.su) * p.sv + kv * p.dv % p.sv;
    };
    for (int t = 0; t < p.T; ++t) order[t] = t;
    std::stable_sort(order, order + p.T, [&](int a, int b) { return phase(a) < phase(b); });
    for (int i = 0; i < p.T; ++i)
      if (i == 0 || phase(order[i]) != phase(order[i - 1])) cls_begin[n_cls++] = i;
    cls_begin[n_cls] = p.T;
    for (int i = 0; i < p.T; ++i) p.tap_order[i] = (unsigned short)order[i];
  }
  // 1: 16-byte vector loads; 2: 32-byte aligned chunks (one load per chunk)
  auto vec_of = [](const float *a, long long ch) {
    if ((uintptr_t)a % 32 == 0 && ch % 8 == 0) return 2;
    return ((uintptr_t)a % 16 == 0 && ch % 4 == 0) ? 1 : 0;
  };
  p.vec_x = vec_of(x, p.Ci);
  p.vec_y = vec_of(dy, p.Co);
  // (the tables' offsets are 32-bit, their positions' fields 10, 10 and 9 bits; tiles
  // have at most 16 rows)
  const long long fw = (long long)p.KW * p.dw + p.sw, fu = 16LL * p.su + (long long)p.KU * p.du,
                  fv = 8LL * p.sv + (long long)p.KV * p.dv;
  const bool lanes = p.vec_x == 2 && p.vec_y == 2 && fw <= stage::kMaxW && fu <= stage::kMaxU &&
                     fv <= stage::kMaxV &&
                     (fw * p.xsw + fu * p.xsu + fv * p.xsv) * p.Ci < (1LL << 31) &&
                     (16 * p.ysu + 8 * p.ysv) * p.Co < (1LL << 31);
  // Packs of taps along u where the channels leave room for them in an MMA's 128
  // rows; from here on a "tap" of a group is a pack.
  p.pk_nch = 16;
  int n_ent = p.T;
  if (p.ordered && p.Ci <= 64 && p.du == 1 && p.KU > p.su) {
    p.pk_nch = 1;
    while (p.pk_nch * 8 < p.Ci) p.pk_nch *= 2;
    const int taps = 16 / p.pk_nch;
    int n = 0, begin = 0;
    for (int c = 0; c < n_cls; ++c) {
      const int end = cls_begin[c + 1];
      cls_begin[c] = n;
      for (int i = begin; i < end; ++i)
        if (order[i] / p.KV % p.KU / p.su % taps == 0) p.tap_order[n++] = (unsigned short)order[i];
      begin = end;
    }
    cls_begin[n_cls] = n_ent = n;
  }
  const bool pack = p.pk_nch < 16;
  // Groups of at most tg taps: each class split into the fewest groups,
  // sizes as even as possible.  Returns the number of groups and fills
  // gstart (ordered) or sets the contiguous split (unordered).
  auto make_groups = [&](int tg) {
    if (!p.ordered) {
      const int n = (p.T + tg - 1) / tg;
      p.TG = (p.T + n - 1) / n;
      return (p.T + p.TG - 1) / p.TG;
    }
    int n = 0, widest = 0;
    for (int c = 0; c < n_cls; ++c) {
      const int nc = cls_begin[c + 1] - cls_begin[c];
      const int ng = (nc + tg - 1) / tg;
      for (int g = 0, at = cls_begin[c]; g < ng; ++g) {
        const int sz = nc / ng + (g < nc % ng ? 1 : 0);
        p.gstart[n++] = (unsigned short)at;
        at += sz;
        widest = std::max(widest, sz);
      }
    }
    p.gstart[n] = (unsigned short)n_ent;
    p.TG = widest;
    return n;
  };
  // The groupings by at most 16 taps and their groups' halos beyond a tile, those that
  // lie within another left out.
  struct Halo {
    int w, u, v;
  };
  constexpr int kMaxHalos = 32;
  struct Grouping {
    int tg, n, widest, nh;  // asked for, groups, taps of the widest, halos
    Halo halo[kMaxHalos];
  } grouping[16];
  int n_grouping = 0;
  struct Reach {
    int w, u, v, u1;  // a tap's offsets; PACK: the u offset of its pack's last tap
  };
  Reach few_taps[kMaxOrderedTaps];
  std::vector<Reach> many_taps(p.T > kMaxOrderedTaps ? p.T : 0);
  Reach *reach = p.T > kMaxOrderedTaps ? many_taps.data() : few_taps;
  for (int t = 0; t < p.T; ++t) {
    const int tu = t / p.KV, kv = t - tu * p.KV, kw = tu / p.KU, ku = tu - kw * p.KU;
    const int last = pack ? ku + std::min(16 / p.pk_nch - 1, (p.KU - 1 - ku) / p.su) * p.su : ku;
    reach[t] = {kw * p.dw, ku * p.du, kv * p.dv, last * p.du};
  }
  for (int tg = std::min(n_ent, 16); tg >= 1; --tg) {
    const int n = make_groups(tg);
    if (n_grouping > 0 && n == grouping[n_grouping - 1].n) continue;
    Grouping &gr = grouping[n_grouping++];
    gr.tg = tg;
    gr.n = n;
    gr.widest = p.TG;
    gr.nh = 0;
    for (int gi = 0; gi < n; ++gi) {
      const int b0 = p.ordered ? p.gstart[gi] : gi * p.TG;
      const int b1 = p.ordered ? p.gstart[gi + 1] : std::min(p.T, b0 + p.TG);
      int mnw = 1 << 30, mnu = 1 << 30, mnv = 1 << 30, mxw = -1, mxu = -1, mxv = -1;
      for (int i = b0; i < b1; ++i) {
        const Reach &o = reach[p.ordered ? p.tap_order[i] : i];
        mnw = std::min(mnw, o.w); mxw = std::max(mxw, o.w);
        mnu = std::min(mnu, o.u); mxu = std::max(mxu, o.u1);
        mnv = std::min(mnv, o.v); mxv = std::max(mxv, o.v);
      }
      const Halo h{(mxw - mnw) / p.sw + 1, (mxu - mnu) / p.su, (mxv - mnv) / p.sv};
      bool seen = false;
      for (int i = 0; i < gr.nh && !seen; ++i)
        seen = gr.halo[i].w >= h.w && gr.halo[i].u >= h.u && gr.halo[i].v >= h.v;
      if (seen) continue;
      if (gr.nh < kMaxHalos) {
        gr.halo[gr.nh++] = h;
      } else {  // one that holds both
        Halo &l = gr.halo[gr.nh - 1];
        l = {std::max(l.w, h.w), std::max(l.u, h.u), std::max(l.v, h.v)};
      }
    }
  }
  // Plan: BN output channels and TG taps per CTA (TG*BN <= 512 TMEM columns, or
  // 2*TG*BN with split-BF16's separate cross-term accumulators) and tiles of TU (even,
  // so that TU*8 pixels fill whole 16-pixel K steps) rows, two stages of which fit
  // shared memory: those with the least estimated time.  Fewer, wider groups stage
  // the activations less often, smaller ones fill the SMs with longer pixel ranges
  // and leave fewer partial sums: with the widest block and the tallest tile first
  // [16;14;14;256]x[3;3;256;256] took 27.6 us where 128 channels a CTA take 22, 64 x
  // 7x7x512 72 where they take 46, and [64;56;56;128]x[3;3;128;128] at rate 2 in
  // split BF16, one tap per CTA, 250 where TU = 8 and two taps take 194.
  const int sms = sm_count();
  // heights, tallest first: those that leave the fewest rows past the output, the least
  // even ones that some number of tiles needs
  int tus[8], ntu = 0;
  for (int tu = 16; tu >= 2 && ntu < 5; tu -= 2) {
    const int tiles = (p.OU + tu - 1) / tu;
    if (std::max(2, (p.OU + tiles - 1) / tiles + 1) / 2 * 2 == tu) tus[ntu++] = tu;
  }
  const long long rows = (long long)p.B * p.OW;
  int HP = 0;  // pixels of the largest halo
  // the sizes of one configuration, one wave of pixel ranges; false when it does not fit
  auto fit = [&](const Grouping &gr, int bn, int tu, bool tables = true) {
    p.n_tg = gr.n;
    p.TG = gr.widest;
    p.BN = std::min(bn, (p.Co + 15) / 16 * 16);
    p.set_cols = (unsigned)(p.TG * p.BN);
    if (parts * p.set_cols > 512) return false;
    HP = 0;
    int packed = 0;  // PACK: pixels of the largest halo's stage
    for (int i = 0; i < gr.nh; ++i) {
      const int hvr = 8 + gr.halo[i].v, hu = tu + gr.halo[i].u;
      HP = std::max(HP, gr.halo[i].w * hu * hvr);
      // (an MMA reads on past the last halo row, into rows of no tap)
      if (pack)
        packed = std::max(packed, (gr.halo[i].w * hu + 16 / p.pk_nch - 1) * p.pk_nch *
                                          chunk_row(hvr, p.pk_nch) + 8);
    }
    p.TU = tu;
    p.TP = tu * 8;
    p.YPS = p.TP + 1;
    p.PS = HP + (((1 - HP) % 8) + 8) % 8;
    if (p.PS >= 16384) return false;
    if (packed >= 16384 || (packed > 0 && HP >= 65536)) return false;
    p.x_bytes = pack ? (unsigned)((packed + 15) / 16 * 16) * 16u
                     : (unsigned)(128 * EB / 16) * (unsigned)p.PS * 16u;
    p.y_bytes = (unsigned)(p.BN * EB / 16) * (unsigned)p.YPS * 16u;
    p.NS = 2;
    p.n_tab = HP + p.TP;
    const size_t need = (size_t)p.NS * parts * (p.x_bytes + p.y_bytes) + 256 +
                        (tables ? 8 * (size_t)(p.n_tab + 3) + 2 * (size_t)p.n_tab : 0);
    if (need > (size_t)kSmemMax) return false;
    p.u_tiles = (p.OU + tu - 1) / tu;
    p.v_tiles = (p.OV + 7) / 8;
    p.total_tiles = rows * p.u_tiles * p.v_tiles;
    p.n_nb = (p.Co + p.BN - 1) / p.BN;
    return true;
  };
  auto set_ranges = [&](long long R) {
    R = std::max<long long>(1, std::min(R, p.total_tiles));
    p.tiles_per_range = (p.total_tiles + R - 1) / R;
    p.R = (int)((p.total_tiles + p.tiles_per_range - 1) / p.tiles_per_range);
  };
  auto units = [&] { return (long long)p.n_tg * p.n_nb * p.n_mb; };
  // MMAs that follow one another in an accumulator
  auto chain = [&](int sets) {
    const long long tiles =
        sets == 1 ? p.tiles_per_range : (p.tiles_per_range + sets - 1) / sets;
    return tiles * (p.TP / 16);
  };
  // The longest accumulation that is allowed, in MMAs: that of the widest block, the
  // height that stages the fewest rows (a tile counts as four more) and the fewest
  // groups (PACK: those of single taps), whose CTAs have about the most pixel ranges that
  // fill the GPU once.  Plans by time alone took 1.3 to 4 times as many for split BF16,
  // and its error, which is theirs, grew as much (64 x 7x7x512: 4.9e-6 to 6.7e-6 of the
  // largest element, with values of one sign 3.3e-6 to 7.2e-6).  What does not show is
  // allowed: beside what split BF16 leaves out (4e-6) 16 MMAs, or an eighth more than the
  // bound up to 128; beside the rounding of BF16's operands to 2^-9 144 MMAs, or a
  // quarter more up to 512 ([53;68;11;144]x[3;3;144;192]: 315 instead of 252 in a row give
  // 2.65e-5 instead of 2.62e-5 rms with values of one sign, the same with both).  Held to
  // the bound itself [15;15;101;112]x[3;3;112;208] in split BF16 took 61 us instead of
  // 43, for 100 MMAs instead of 104.
  long long bound = -1;
  int heights[8] = {14, 12, 10, 16, 8, 6, 4, 2};
  long long staged[8];
  for (int i = 0; i < 8; ++i) {  // sorted by the rows they stage
    const int tu = heights[i];
    const long long n =
        (p.OU + tu - 1) / tu * (tu + 4LL) + (tu > kProducerWarps ? 1LL << 40 : 0);
    int k = i;
    for (; k > 0 && staged[k - 1] > n; --k) {
      staged[k] = staged[k - 1];
      heights[k] = heights[k - 1];
    }
    staged[k] = n;
    heights[k] = tu;
  }
  for (int bn = 256; bn >= 16 && bound < 0; bn /= 2)
    for (int ti = 0; ti < 8 && bound < 0; ++ti)
      for (int gi = 0; gi < n_grouping && bound < 0; ++gi)
        if (fit(grouping[gi], bn, heights[ti], false)) {
          const int tg = std::min(16, 512 / (parts * p.BN));
          const long long groups = pack ? std::max(p.n_tg, (p.T + tg - 1) / tg) : p.n_tg;
          set_ranges(sms / (groups * p.n_nb * p.n_mb));
          bound = chain(1);
        }
  bound = kind == K_BF16X3 ? std::max({bound, std::min(bound * 9 / 8, 128LL), 16LL})
                           : std::max({bound, std::min(bound * 5 / 4, 512LL), 144LL});
  double least = -1;
  int best_tg = 0;
  WgParams best = p;
  for (int gi = 0; gi < n_grouping; ++gi) {
    int last_bn = 0;
    for (int bn : {256, 128, 64, 32, 16}) {
      if (std::min(bn, (p.Co + 15) / 16 * 16) == last_bn) continue;
      if (bn < 64 && least >= 0) continue;  // (narrow blocks waste the tensor core)
      for (int ti = 0; ti < ntu; ++ti) {
        if (!fit(grouping[gi], bn, tus[ti])) continue;
        last_bn = p.BN;
        // pixel ranges: enough CTAs to fill the GPU once; accumulator sets, which cost
        // nothing, and beyond them ranges for several waves of CTAs where an accumulation
        // is too long (each wave an epilogue more)
        set_ranges(sms / units());
        const long long most = std::min(512LL / p.set_cols - parts + 1, p.tiles_per_range);
        p.sets = 1;
        while (chain(p.sets) > bound && p.sets < most) ++p.sets;
        for (int waves = 2; chain(p.sets) > bound && p.tiles_per_range > p.sets; ++waves)
          set_ranges(std::max<long long>(waves, waves * sms / units()));
        const double t = estimate(p, HP, parts, units() * p.R, sms);
        if (least < 0 || t < least) {
          least = t;
          best = p;
          best_tg = grouping[gi].tg;
        }
      }
    }
  }
  if (least < 0) return kErrUnsupported;
  p = best;
  p.n_tg = make_groups(best_tg);
  p.small_off = p.set_cols * (unsigned)p.sets;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.set_cols * (unsigned)(p.sets + parts - 1)) p.tmem_cols <<= 1;
  uint32_t idesc = instr_desc(kind == K_TF32 ? 2u : 1u, (uint32_t)p.BN);
  idesc |= (1u << 15) | (1u << 16);  // A and B MN-major
  p.idesc = idesc;
  p.spin_limit = wait_limit();
  p.status = status_word();
  if (!p.status) {
    set_error("wgrad_tc: cannot locate device status word");
    return kErrCuda;
  }
  const long long welems = (long long)p.T * p.Ci * p.Co;
  float *part = nullptr;
  if (p.R > 1) {
    int rc = scratch_alloc((void **)&part, sizeof(float) * (size_t)welems * p.R, s);
    if (rc) return rc;
    p.out = part;
  } else {
    p.out = dw;
  }
  const size_t smem =
      (size_t)p.NS * parts * (p.x_bytes + p.y_bytes) + (2 * p.NS + 2) * 8 + 16 + 4 * (size_t)p.TG +
      8 * (size_t)(p.n_tab + 3) + 2 * (size_t)p.n_tab;
  const int grid = (int)(units() * p.R);
  int rc;
  p.x_dv = 8LL * p.sv * p.xsv * p.Ci;
  p.x_du = (long long)p.TU * p.su * p.xsu * p.Ci - p.v_tiles * p.x_dv;
  p.x_dw = p.sw * p.xsw * p.Ci - (long long)p.u_tiles * p.TU * p.su * p.xsu * p.Ci;
  p.x_db = p.xsb * p.Ci - (long long)p.OW * p.sw * p.xsw * p.Ci;
  p.y_dv = 8LL * p.ysv * p.Co;
  p.y_du = (long long)p.TU * p.ysu * p.Co - p.v_tiles * p.y_dv;
  p.y_dw = p.ysw * p.Co - (long long)p.u_tiles * p.TU * p.ysu * p.Co;
  p.y_db = p.ysb * p.Co - (long long)p.OW * p.ysw * p.Co;
  auto go = [&](auto k, auto packed) {
    constexpr int KIND = decltype(k)::value;
    constexpr bool PACK = decltype(packed)::value;
    if (!lanes) return launch<KIND, false, PACK, true>(p, smem, grid, s);
    return p.sets > 1 ? launch<KIND, true, PACK, true>(p, smem, grid, s)
                      : launch<KIND, true, PACK, false>(p, smem, grid, s);
  };
  using X3 = std::integral_constant<int, K_BF16X3>;
  using B1 = std::integral_constant<int, K_BF16>;
  if (kind == K_BF16X3) rc = pack ? go(X3{}, std::true_type{}) : go(X3{}, std::false_type{});
  else rc = pack ? go(B1{}, std::true_type{}) : go(B1{}, std::false_type{});
  if (rc == kOk && p.R > 1) rc = sum_partials_f32(part, dw, welems, p.R, s);
  if (part) scratch_free(part, s);
  return rc;
}

}  // namespace owlgpu
