// Motion-compensation interpolation on 16-bit planes (8..12-bit samples):
// 1/16-pel 8-tap luma and 1/32-pel 4-tap chroma, uni-prediction output or
// 14-bit bi-prediction intermediates, and the BCW weighted bi average.
// Follows interpolate_luma_block_16 (inter.rs:2010-2134),
// interpolate_chroma_block_format_16 (:2543-2672) and weighted_average_bi_16
// (:2676-2698) of the reference, including the uni-prediction second-stage
// shift `12 - bd` for 2-D fractional positions (inter.rs:2051 / :2583); and
// the 8-bit functions interpolate_luma_block (inter.rs:896-1051) and
// interpolate_chroma_block_420 (:1056-1182), which read 8-bit planes and use
// the second stage (sum + 2^11) >> 12 for 2-D uni-prediction.
//
// Each warp takes tiles of 32x16 outputs by itself: the tile's
// reference window is staged as int16 in shared memory, a lane filters runs
// of eight outputs along a row, then two columns by four rows, both with dp2a
// on packed sample pairs. The horizontal outputs fit 16 bits because the taps
// sum to at most 128 in absolute value and the shift is bd - 8.
#pragma once
#include "vvcg_device.cuh"
#include "vvcg_tables_dev.cuh"

namespace vvcg {

constexpr int kMcW = 32, kMcH = 16;  // a warp's tile
constexpr int kMcWarps = 4;
constexpr int kMcPitch = 48;         // window row: 3 + 32 + 7 samples, padded

struct McParams {
  const uint16_t* ref;
  const uint8_t* ref8;  // 8-bit plane of the 8-bit functions (then ref is unused and bd is 8)
  int32_t w, h, stride, bd;
  int32_t chroma;   // 0 = luma (8 taps), else chroma format (4 taps)
};

// A block's interpolation: integer offset, fractions, packed taps, shifts.
struct McFilter {
  int dx, dy, fx, fy;
  uint32_t th0, th1, tv0, tv1;  // taps 0..3 and 4..7 as int8, horizontal and vertical
  int head, shift1, shift2, add2, offs, maxv;
  bool bi, eight;
};

// One output of a 2-D, 1-D or copied position from its sums.
__device__ __forceinline__ int mc_copy(const McFilter& F, int s) { return F.bi ? (s << F.head) - F.offs : s; }
__device__ __forceinline__ int mc_1d(const McFilter& F, int s) {
  return F.bi ? (s >> F.shift1) - F.offs : clampi((s + 32) >> 6, 0, F.maxv);
}
__device__ __forceinline__ int mc_2d(const McFilter& F, int s) {
  // 8-bit functions: (sum of taps x (tmp - 2^13) + 2^11 + 2^13 x 64) >> 12,
  // which is (s + 2^11) >> 12 because every filter's taps sum to 64
  return F.bi ? (s >> F.shift2) - F.offs
              : (F.eight ? clampi((s + 2048) >> 12, 0, 255)
                         : clampi((int)((unsigned)s + (unsigned)F.add2) >> F.shift2, 0, F.maxv));
}

__device__ __forceinline__ int mc_tap(uint32_t t0, uint32_t t1, int k) {
  return (int8_t)((k < 4 ? t0 : t1) >> (8 * (k & 3)));
}

// a / n for 0 <= a < 32 and 1 <= n <= 32 (exact: the quotient's distance from a
// whole number is at least 1 / 64).
__device__ __forceinline__ int div_lane(int a, int n) { return (int)(((float)a + 0.5f) * __frcp_rn((float)n)); }
__device__ __forceinline__ int per_warp(int n) { return (int)(32.5f * __frcp_rn((float)n)); }  // 32 / n

// Eight sums of kTaps products along a row, from sample j of `row`.
template <int kTaps>
__device__ __forceinline__ void mc_row8(const int16_t* row, int j, uint32_t t0, uint32_t t1, int (&v)[8]) {
  constexpr int kPairs = (8 + kTaps) / 2;  // sample pairs the run needs
  const uint32_t* q = reinterpret_cast<const uint32_t*>(row) + (j >> 1);
  uint32_t e[kPairs];
  const uint32_t sh = (j & 1) * 16;
  uint32_t c = q[0];
#pragma unroll
  for (int k = 0; k < kPairs; k++) {
    const uint32_t n = q[k + 1];
    e[k] = __funnelshift_r(c, n, sh);
    c = n;
  }
  uint32_t f[kPairs - 1];  // pairs starting at odd samples
#pragma unroll
  for (int k = 0; k < kPairs - 1; k++) f[k] = __byte_perm(e[k], e[k + 1], 0x5432);
#pragma unroll
  for (int i = 0; i < 8; i++) {
    auto p = [&](int q) -> int { return (int)((i & 1) ? f[(i >> 1) + q] : e[(i >> 1) + q]); };
    int s = __dp2a_hi(p(1), (int)t0, __dp2a_lo(p(0), (int)t0, 0));
    if (kTaps == 8) s = __dp2a_hi(p(3), (int)t1, __dp2a_lo(p(2), (int)t1, s));
    v[i] = s;
  }
}

struct McWs {
  __align__(16) int16_t win[(kMcH + 7) * kMcPitch + 16];
  __align__(16) int16_t tmp[(kMcH + 7) * kMcW];
};

// One tile of a block by one warp: outputs tw x th at o (row pitch bw), whose
// window starts at plane position (wx0, wy0). False, with nothing written,
// when a sample of the window lies above the bit depth.
// Out: int32_t (the interpolation calls) or int16_t (predictions kept in
// shared memory).
template <int kTaps, bool kEight, class Out>
__device__ __forceinline__ bool mc_tile(const McParams& Pm, const McFilter& F, int wx0, int wy0, int tw, int th,
                                        Out* o, int bw, McWs& S, int lane) {
  constexpr int half = kTaps / 2 - 1;
  const int ww = tw + kTaps - 1, wh = th + kTaps - 1;
  // the window, at column `xo` of its rows; groups of four samples where the
  // plane's rows are aligned for it and the window lies inside
  int xo = 0;
  uint32_t high = 0;
  const uint32_t mask = ~(uint32_t)F.maxv & 0xFFFFu;
  const bool inside = wx0 >= 0 && wy0 >= 0 && wx0 + ww <= Pm.w && wy0 + wh <= Pm.h;
  const uintptr_t base = kEight ? reinterpret_cast<uintptr_t>(Pm.ref8) : reinterpret_cast<uintptr_t>(Pm.ref);
  // a group may reach past the window's last sample, but not past the plane's row
  if (inside && (Pm.stride & 3) == 0 && (base & (kEight ? 3 : 7)) == 0 && ((wx0 + ww + 3) & ~3) <= Pm.w) {
    xo = wx0 & 3;
    const int ng = (xo + ww + 3) >> 2;  // groups a row, at most 11
    const int rows = per_warp(ng), r0 = div_lane(lane, ng), c0 = lane - r0 * ng;
    // six loads in flight a lane: their latency, not their number, is the cost
    constexpr int kBatch = 6;
    const size_t at = (size_t)wy0 * Pm.stride + (wx0 & ~3) + 4 * c0;
    for (int y0 = r0 < rows ? r0 : wh; y0 < wh; y0 += kBatch * rows) {
      uint2 v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        const int y = y0 + k * rows;
        v[k] = make_uint2(0, 0);
        if (y < wh) {
          const size_t i = at + (size_t)y * Pm.stride;
          if (kEight)
            v[k].x = __ldg(reinterpret_cast<const uint32_t*>(Pm.ref8 + i));
          else
            v[k] = __ldg(reinterpret_cast<const uint2*>(Pm.ref + i));
        }
      }
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        const int y = y0 + k * rows;
        if (kEight) v[k] = make_uint2(__byte_perm(v[k].x, 0, 0x4140), __byte_perm(v[k].x, 0, 0x4342));
        high |= v[k].x | v[k].y;
        if (y < wh) *reinterpret_cast<uint2*>(&S.win[y * kMcPitch + 4 * c0]) = v[k];
      }
    }
    high = (high | high >> 16) & mask;
  } else {
    for (int x = lane; x < ww; x += 32) {
      const int cx = clampi(wx0 + x, 0, Pm.w - 1);
#pragma unroll 4
      for (int y = 0; y < wh; y++) {
        const size_t i = (size_t)clampi(wy0 + y, 0, Pm.h - 1) * Pm.stride + cx;
        const uint32_t v = kEight ? (uint32_t)__ldg(Pm.ref8 + i) : (uint32_t)__ldg(Pm.ref + i);
        high |= v & mask;
        S.win[y * kMcPitch + x] = (int16_t)v;
      }
    }
  }
  if (__any_sync(0xffffffffu, high != 0)) return false;
  __syncwarp();
  // lane -> (row, run) of a step
  const int runs = (tw + 7) >> 3, rrows = per_warp(runs), ry = div_lane(lane, runs), x0 = 8 * (lane - ry * runs);
  if (F.fy == 0) {  // rows only, or a copy
    for (int y = ry < rrows ? ry : th; y < th; y += rrows) {
      const int16_t* row = S.win + (y + half) * kMcPitch;
      int v[8];
      if (F.fx == 0) {
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = mc_copy(F, row[xo + x0 + half + k]);
      } else {
        mc_row8<kTaps>(row, xo + x0, F.th0, F.th1, v);
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = mc_1d(F, v[k]);
      }
      Out* d = o + (size_t)y * bw + x0;
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (x0 + k < tw) d[k] = (Out)v[k];
    }
    __syncwarp();
    return true;
  }
  for (int y = ry < rrows ? ry : wh; y < wh; y += rrows) {
    const int16_t* row = S.win + y * kMcPitch;
    int v[8];
    if (F.fx == 0) {
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = row[xo + x0 + half + k];
    } else {
      mc_row8<kTaps>(row, xo + x0, F.th0, F.th1, v);
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] >>= F.shift1;
    }
    *reinterpret_cast<uint4*>(&S.tmp[y * kMcW + x0]) =
        make_uint4(__byte_perm((uint32_t)v[0], (uint32_t)v[1], 0x5410), __byte_perm((uint32_t)v[2], (uint32_t)v[3], 0x5410),
                   __byte_perm((uint32_t)v[4], (uint32_t)v[5], 0x5410), __byte_perm((uint32_t)v[6], (uint32_t)v[7], 0x5410));
  }
  __syncwarp();
  // columns: two by four outputs a lane and step
  const int cp = (tw + 1) >> 1;
  const bool pair = ((reinterpret_cast<uintptr_t>(o) & (2 * sizeof(Out) - 1)) | (bw & 1)) == 0;
  const int crows = per_warp(cp), cy = div_lane(lane, cp), x = 2 * (lane - cy * cp);
  for (int y0 = cy < crows ? 4 * cy : th; y0 < th; y0 += 4 * crows) {
    constexpr int kRows = kTaps + 3;
    uint32_t r[kRows];
#pragma unroll
    for (int k = 0; k < kRows; k++) r[k] = *reinterpret_cast<const uint32_t*>(&S.tmp[(y0 + k) * kMcW + x]);
    int a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k + 1 < kRows; k++) {
      const uint32_t lo = __byte_perm(r[k], r[k + 1], 0x5410), hi = __byte_perm(r[k], r[k + 1], 0x7632);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int tap = k - q;  // the pair's first tap of output q
        if (tap < 0 || tap >= kTaps || (tap & 1)) continue;
        const int t = (int)(tap < 4 ? F.tv0 : F.tv1);
        if (tap & 2) {
          a[q] = __dp2a_hi((int)lo, t, a[q]);
          b[q] = __dp2a_hi((int)hi, t, b[q]);
        } else {
          a[q] = __dp2a_lo((int)lo, t, a[q]);
          b[q] = __dp2a_lo((int)hi, t, b[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (y0 + q >= th) continue;
      const int va = F.fx == 0 ? mc_1d(F, a[q]) : mc_2d(F, a[q]), vb = F.fx == 0 ? mc_1d(F, b[q]) : mc_2d(F, b[q]);
      Out* d = o + (size_t)(y0 + q) * bw + x;
      if (pair && x + 1 < tw) {
        if constexpr (sizeof(Out) == 4)
          *reinterpret_cast<int2*>(d) = make_int2(va, vb);
        else
          *reinterpret_cast<uint32_t*>(d) = __byte_perm((uint32_t)va, (uint32_t)vb, 0x5410);
      } else {
        d[0] = (Out)va;
        if (x + 1 < tw) d[1] = (Out)vb;
      }
    }
  }
  __syncwarp();
  return true;
}

// The filter of one block.
template <bool kEight>
__device__ __forceinline__ McFilter mc_filter(const McParams& Pm, const vvcg_mc_block& B) {
  const int bd = clampi(Pm.bd, 8, 12);
  McFilter F;
  F.bi = (B.flags & VVCG_MC_BI) != 0;
  F.eight = kEight;
  F.maxv = (1 << bd) - 1;
  if (Pm.chroma == 0) {
    F.dx = B.mv_x >> 4;
    F.dy = B.mv_y >> 4;
    F.fx = B.mv_x & 15;
    F.fy = B.mv_y & 15;
    const uint32_t* tab = reinterpret_cast<const uint32_t*>((B.flags & VVCG_MC_AFFINE) ? c_affine_taps8 : c_luma_taps8);
    F.th0 = tab[F.fx * 2];
    F.th1 = tab[F.fx * 2 + 1];
    F.tv0 = tab[F.fy * 2];
    F.tv1 = tab[F.fy * 2 + 1];
    if ((B.flags & (VVCG_MC_AFFINE | VVCG_MC_ALT_HPEL)) == VVCG_MC_ALT_HPEL) {
      uint32_t a0 = 0, a1 = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        a0 |= (uint32_t)(uint8_t)c_luma_alt_hpel[k] << (8 * k);
        a1 |= (uint32_t)(uint8_t)c_luma_alt_hpel[4 + k] << (8 * k);
      }
      if (F.fx == 8) F.th0 = a0, F.th1 = a1;
      if (F.fy == 8) F.tv0 = a0, F.tv1 = a1;
    }
  } else {
    const int sw = (Pm.chroma == 1 || Pm.chroma == 2) ? 2 : 1, shh = Pm.chroma == 1 ? 2 : 1;
    const int mx = B.mv_x * (sw == 1 ? 2 : 1), my = B.mv_y * (shh == 1 ? 2 : 1);
    F.dx = mx >> 5;
    F.dy = my >> 5;
    F.fx = mx & 31;
    F.fy = my & 31;
    const uint32_t* tab = reinterpret_cast<const uint32_t*>(c_chroma_taps4);
    F.th0 = tab[F.fx];
    F.tv0 = tab[F.fy];
    F.th1 = F.tv1 = 0;
  }
  F.head = max(14 - bd, 2);
  F.shift1 = 6 - F.head;
  F.shift2 = F.bi ? 6 : 12 - bd;
  // The reference's release build masks the shift count to 5 bits (1 << 31 at
  // 12 bit, where shift2 is 0) and wraps the addition.
  F.add2 = F.bi ? 0 : (int)(1u << ((unsigned)(F.shift2 - 1) & 31));
  F.offs = 1 << (bd + F.head - 1);
  return F;
}

// A tile with samples above the bit depth (nothing rejects them), in 32 bits
// straight from the plane.
template <int kTaps, bool kEight>
__device__ __noinline__ void mc_tile_wide(const McParams* params, const vvcg_mc_block* block, int x0, int y0,
                                          int32_t* out) {
  const McParams Pm = *params;
  const vvcg_mc_block B = *block;
  const McFilter F = mc_filter<kEight>(Pm, B);
  const int lane = threadIdx.x & 31, bw = B.w, tw = min(kMcW, B.w - x0), th = min(kMcH, B.h - y0);
  constexpr int half = kTaps / 2 - 1;
  const int wx0 = B.x + x0 + F.dx - half, wy0 = B.y + y0 + F.dy - half;
  int32_t* o = out + B.out_offset + (size_t)y0 * bw + x0;
  auto at = [&](int x, int y) -> int {
    const size_t i = (size_t)clampi(wy0 + y, 0, Pm.h - 1) * Pm.stride + clampi(wx0 + x, 0, Pm.w - 1);
    return Pm.ref8 ? (int)Pm.ref8[i] : (int)Pm.ref[i];
  };
  for (int i = lane; i < tw * th; i += 32) {
    const int x = i % tw, y = i / tw;
    int v;
    if (F.fx == 0 && F.fy == 0) {
      v = mc_copy(F, at(x + half, y + half));
    } else if (F.fy == 0) {
      int s = 0;
      for (int k = 0; k < kTaps; k++) s += mc_tap(F.th0, F.th1, k) * at(x + k, y + half);
      v = mc_1d(F, s);
    } else if (F.fx == 0) {
      int s = 0;
      for (int k = 0; k < kTaps; k++) s += mc_tap(F.tv0, F.tv1, k) * at(x + half, y + k);
      v = mc_1d(F, s);
    } else {
      int s = 0;
      for (int j = 0; j < kTaps; j++) {
        int t = 0;
        for (int k = 0; k < kTaps; k++) t += mc_tap(F.th0, F.th1, k) * at(x + k, y + j);
        s += mc_tap(F.tv0, F.tv1, j) * (t >> F.shift1);
      }
      v = mc_2d(F, s);
    }
    o[(size_t)y * bw + x] = v;
  }
}

// Grid: (blocks / kMcWarps, kMcSplit). A warp takes the tiles y, y + kMcSplit,
// ... of its block: most of a picture's blocks are one tile, whose other warps
// exit at once, and a 64x64 block's eight tiles are spread, so that no warp's
// chain is much longer than the rest. What bounds it is the latency of that
// chain (record, window, two passes, stores) and the blocks in flight: 7,400
// blocks of 8..64 samples a side of a 1920x1080 picture take 23 us for luma
// and 13 us a chroma plane. With one CTA of 256 threads per block, 32-bit
// tiles and a multiply per tap they took 37 and 18 us; with the window loaded
// a row group at a time instead of six in flight 36 and 18 us.
constexpr int kMcSplit = 4;
template <int kTaps, bool kEight>
__global__ void __launch_bounds__(kMcWarps * 32, 8) k_mc(const __grid_constant__ McParams Pm,
                                                        const vvcg_mc_block* __restrict__ blocks, uint32_t n,
                                                        int32_t* __restrict__ out) {
  __shared__ McWs ws[kMcWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t b = blockIdx.x * kMcWarps + wid;
  if (b >= n) return;
  const vvcg_mc_block B = blocks[b];
  const int tx = (B.w + kMcW - 1) / kMcW, tiles = tx * ((B.h + kMcH - 1) / kMcH);
  if ((int)blockIdx.y >= tiles) return;
  constexpr int half = kTaps / 2 - 1;
  const McFilter F = mc_filter<kEight>(Pm, B);
  bool fits = true;
  for (int t = blockIdx.y; t < tiles; t += kMcSplit) {
    const int ty = t / tx, x0 = (t - ty * tx) * kMcW, y0 = ty * kMcH;
    fits &= mc_tile<kTaps, kEight>(Pm, F, B.x + x0 + F.dx - half, B.y + y0 + F.dy - half, min(kMcW, B.w - x0),
                                   min(kMcH, B.h - y0), out + B.out_offset + (size_t)y0 * B.w + x0, B.w, ws[wid], lane);
  }
  if (!fits)  // after the loop, where the call costs it no registers
    for (int t = blockIdx.y; t < tiles; t += kMcSplit)
      mc_tile_wide<kTaps, kEight>(&Pm, &blocks[b], (t % tx) * kMcW, (t / tx) * kMcH, out);
}

// weighted_average_bi_16 (inter.rs:2676-2698), four samples a thread where
// the arrays are aligned for it.
__global__ void k_bi_average(const int32_t* __restrict__ p0, const int32_t* __restrict__ p1,
                             uint64_t n, int bcw, int bd, uint16_t* __restrict__ out) {
  bd = clampi(bd, 8, 12);
  const int maxv = (1 << bd) - 1;
  const int w1 = c_bcw_weights[min(bcw, 4)], w0 = 8 - w1;
  const int head = max(14 - bd, 2), sn = head + 3;
  const int off = (1 << (sn - 1)) + ((1 << (bd + head - 1)) << 3);
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
  auto avg = [&](int a, int b) -> uint32_t { return (uint32_t)clampi((a * w0 + b * w1 + off) >> sn, 0, maxv); };
  uint64_t done = 0;
  if (((reinterpret_cast<uintptr_t>(p0) | reinterpret_cast<uintptr_t>(p1)) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(out) & 7) == 0) {
    for (uint64_t i = t; i < n / 4; i += step) {
      const int4 a = __ldcs(reinterpret_cast<const int4*>(p0) + i), b = __ldcs(reinterpret_cast<const int4*>(p1) + i);
      reinterpret_cast<uint2*>(out)[i] =
          make_uint2(avg(a.x, b.x) | avg(a.y, b.y) << 16, avg(a.z, b.z) | avg(a.w, b.w) << 16);
    }
    done = n & ~3ull;
  }
  for (uint64_t i = done + t; i < n; i += step) out[i] = (uint16_t)avg(p0[i], p1[i]);
}

}  // namespace vvcg
