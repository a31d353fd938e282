// Function-level transform-unit kernels of libvvcg (sm_100a): levels ->
// residual (dequantisation, inverse LFNST, inverse DCT-2 / DST-7 / DCT-8,
// BDPCM) and residual -> levels (forward transform, forward LFNST,
// quantisation). One warp per transform unit; the host bins units by size so
// each warp's shared tiles fit the largest unit of its bin.
//
// The matrix products are dp2a (pairs of 16-bit samples x 8-bit matrix
// entries): each lane keeps its output's matrix row in registers and reads the
// lines of the tile as broadcast 16-byte words. Every sum is exact: inverse
// stages and the forward first stage stay below 2^31 (int16 inputs, |matrix|
// <= 90, at most 64 terms). The forward second stage's inputs are not clipped;
// where one of a unit's leaves 16 bits (residuals far beyond its bit depth) the
// stage is summed in two 16-bit halves and 64 bits. With one 32-bit sample and
// one matrix byte loaded per product before, 16,000 mixed units took 523 us
// forward and 458 us inverse; now 129 us and 106 us (the 64-point bins 405 ->
// 62 and 329 -> 53 us).
//
// The 32-bit tile functions (tu_*) below serve the luma transform search,
// which quantises and reconstructs in place.
#pragma once
#include <stdint.h>

#include "vvcg_device.cuh"
#include "vvcg_tables_dev.cuh"

namespace vvcg {

// Grouped diagonal scans of every (log2 w, log2 h) in 0..6, raster indices of
// the top-left min(w,32) x min(h,32) (transform.rs:43-80 CoeffScan::new).
constexpr int kTuScanTotal = 95 * 95;
__device__ int16_t g_tu_scan[kTuScanTotal];
__device__ int32_t g_tu_scan_off[49];
// Inverse of g_tu_scan (same offsets): the scan position of sample (x, y) at
// index y * min(w, 32) + x.
__device__ int16_t g_tu_scan_pos[kTuScanTotal];
// Transform matrices as rows of packed int8 words (tu_mat_row): offsets by
// direction (forward, inverse), type (DCT-2, DST-7, DCT-8) and log2 length.
constexpr int kTmWords = 4096;
__device__ __align__(16) uint32_t g_tm[kTmWords];
__constant__ uint16_t c_tm_off[2][3][7];
// LFNST kernels (tr_tables.rs LFNST_8X8 / LFNST_4X4 / LFNST_LUT).
__device__ int8_t g_lfnst8[4 * 2 * 16 * 48];
__device__ int8_t g_lfnst4[4 * 2 * 16 * 16];
__device__ uint8_t g_lfnst_lut[95];

constexpr int kTuPad = 64;   // tiles are padded by one sample per row or column

// Transform types and zero-out of a unit (decode_general.rs:4165-4198 with
// mts_types :4205, primary_skips :4216, lfnst_skips :4233).
struct TuShape {
  int w, h, lw, lh, n;
  int th, tv;  // 0 DCT-2, 1 DST-7, 2 DCT-8
  int sw, sh;  // zero-out width / height (at least the default of the types)
};

__host__ __device__ __forceinline__ int tu_default_skip(int tr, int n) {
  return (tr != 0 && n == 32) ? 16 : (n > 32 ? n - 32 : 0);
}

__host__ __device__ __forceinline__ void tu_shape(const vvcg_tu_rec& r, TuShape& s) {
  s.lw = r.log2_w;
  s.lh = r.log2_h;
  s.w = 1 << s.lw;
  s.h = 1 << s.lh;
  s.n = s.w * s.h;
  const bool mts = r.mts_idx != 0;
  if (mts) {
    s.th = (r.mts_idx == 1 || r.mts_idx == 3) ? 1 : 2;
    s.tv = (r.mts_idx == 1 || r.mts_idx == 2) ? 1 : 2;
  } else if ((r.flags & VVCG_TU_IMPLICIT_MTS) && r.lfnst_idx == 0) {
    s.th = (s.w >= 4 && s.w <= 16) ? 1 : 0;
    s.tv = (s.h >= 4 && s.h <= 16) ? 1 : 0;
  } else {
    s.th = s.tv = 0;
  }
  int sw, sh;
  if (r.lfnst_idx > 0 && !mts) {
    const int nz = (s.w == 4 || s.h == 4) ? 4 : 8;
    sw = s.w - (nz < s.w ? nz : s.w);
    sh = s.h - (nz < s.h ? nz : s.h);
  } else {
    sw = tu_default_skip(s.th, s.w);
    sh = tu_default_skip(s.tv, s.h);
  }
  const int dw = tu_default_skip(s.th, s.w), dh = tu_default_skip(s.tv, s.h);
  s.sw = sw > dw ? sw : dw;
  s.sh = sh > dh ? sh : dh;
}

__device__ __forceinline__ const int8_t* tu_matrix(int tr, int log2n) {
  if (tr == 0) return g_dct2_m[log2n - 1];
  return tr == 1 ? g_dst7_m[log2n - 2] : g_dct8_m[log2n - 2];
}

__device__ __forceinline__ const int16_t* tu_scan(int lw, int lh) { return g_tu_scan + g_tu_scan_off[lw * 7 + lh]; }

// dct.rs:828-830 transform shift with the sqrt(2) flag of the quantisers.
__device__ __forceinline__ int tu_tr_shift(int lw, int lh, int bd, bool* s2) {
  *s2 = ((lw + lh) & 1) != 0;
  return 15 - bd - ((lw + lh) >> 1) - (*s2 ? 1 : 0);
}

// transform.rs:229-246 dequantize_ts (with the reference's `as i32` truncation)
__device__ __forceinline__ int tu_dequant_ts(int level, int qp) {
  qp = max(4, qp);
  const int qp_per = qp / 6, rs = 6 - qp_per;
  const long long v = (long long)level * c_inv_quant_scale[0][qp % 6];
  const long long s = rs > 0 ? (v + (1ll << (rs - 1))) >> rs : v << (-rs);
  return clip16i((int32_t)(uint32_t)(unsigned long long)s);
}

// transform.rs:214-226 quantize_ts
__device__ __forceinline__ int tu_quant_ts(int res, int qp) {
  qp = max(4, qp);
  const int qbits = 14 + qp / 6;
  const long long add = 171ll << (qbits - 9);
  const long long a = ((long long)abs(res) * c_quant_scale[0][qp % 6] + add) >> qbits;
  const int sign = (res > 0) - (res < 0);
  return clip16((long long)sign * a);
}

// Splits scan positions [0, last] into 32 chunks walked from the end: lane 0
// takes the highest positions. Returns this lane's chunk [lo, hi].
__device__ __forceinline__ void dq_chunk(int last, int lane, int& lo, int& hi) {
  const int cs = (last + 32) >> 5;
  hi = last - lane * cs;
  lo = max(hi - cs + 1, 0);
}

// Entry state of each lane's chunk from per-lane state maps (2 bits per
// state): an inclusive warp scan of map compositions, shifted by one lane.
__device__ __forceinline__ int dq_entry_state(uint32_t map, int lane) {
  uint32_t pre = map;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t other = __shfl_up_sync(0xffffffffu, pre, o);
    if (lane >= o) {
      uint32_t comp = 0;
      for (int s = 0; s < 4; s++) comp |= ((pre >> (2 * ((other >> (2 * s)) & 3))) & 3) << (2 * s);
      pre = comp;
    }
  }
  const uint32_t excl = __shfl_up_sync(0xffffffffu, pre, 1);
  return lane == 0 ? 0 : (int)(excl & 3);
}

// Position (row, column) in the unit of LFNST element j (lfnst.rs:253-292):
// the non-transposed layout fills rows of sb (first 4 rows) then 4; the
// transposed one fills columns.
__device__ __forceinline__ int lfnst_pos(int j, int sb, bool transposed, int w) {
  int y, x;
  if (!transposed) {
    if (sb == 4) {
      y = j >> 2;
      x = j & 3;
    } else if (j < 32) {
      y = j >> 3;
      x = j & 7;
    } else {
      y = 4 + ((j - 32) >> 2);
      x = (j - 32) & 3;
    }
  } else {
    if (sb == 4) {
      y = j & 3;
      x = j >> 2;
    } else if (j < 32) {
      y = j & 7;
      x = j >> 3;
    } else {
      y = (j - 32) & 3;
      x = 4 + ((j - 32) >> 2);
    }
  }
  return y * w + x;
}

struct LfnstParams {
  int sb, tr, zo;
  const int8_t* m;  // [16][tr] rows of the selected kernel
  bool transposed;
};

__device__ __forceinline__ LfnstParams lfnst_params(const TuShape& S, int idx, int mode) {
  LfnstParams p;
  p.sb = (S.w >= 8 && S.h >= 8) ? 8 : 4;
  const bool small = (S.w == 4 && S.h == 4) || (S.w == 8 && S.h == 8);
  p.tr = p.sb == 4 ? 16 : 48;
  p.zo = small ? 8 : 16;
  const int set = g_lfnst_lut[mode];
  p.m = p.sb == 4 ? g_lfnst4 + (set * 2 + idx - 1) * 16 * 16 : g_lfnst8 + (set * 2 + idx - 1) * 16 * 48;
  p.transposed = (mode >= 35 && mode < 67) || mode >= 81;
  return p;
}

// lfnst.rs:219-294 inverse_lfnst_rect, in place on A (raster, stride w).
__device__ void tu_lfnst_inverse(int32_t* A, const TuShape& S, int idx, int mode, int lane) {
  const LfnstParams p = lfnst_params(S, idx, mode);
  const int16_t* scan8 = tu_scan(3, 3);
  int src[16];
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const int r = scan8[i];
    src[i] = A[(r >> 3) * S.w + (r & 7)];
  }
  int o[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int j = lane + 32 * q;
    int s = 0;
    if (j < p.tr)
      for (int i = 0; i < p.zo; i++) s += src[i] * (int)p.m[i * p.tr + j];
    o[q] = clip16i((s + 64) >> 7);
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int j = lane + 32 * q;
    if (j < p.tr) A[lfnst_pos(j, p.sb, p.transposed, S.w)] = o[q];
  }
  __syncwarp();
}

// lfnst.rs:131-205 forward_lfnst_rect, in place on A (raster, stride w).
__device__ void tu_lfnst_forward(int32_t* A, const TuShape& S, int idx, int mode, int lane) {
  const LfnstParams p = lfnst_params(S, idx, mode);
  const int16_t* scan8 = tu_scan(3, 3);
  // lane j holds src[j] and src[j + 32]
  int s0 = lane < p.tr ? A[lfnst_pos(lane, p.sb, p.transposed, S.w)] : 0;
  int s1 = lane + 32 < p.tr ? A[lfnst_pos(lane + 32, p.sb, p.transposed, S.w)] : 0;
  int out = 0;  // lane j < zo: output j
  for (int i = 0; i < p.tr; i++) {
    const int v = __shfl_sync(0xffffffffu, i < 32 ? s0 : s1, i & 31);
    if (lane < p.zo) out += v * (int)p.m[lane * p.tr + i];
  }
  out = (out + 64) >> 7;
  __syncwarp();
  if (lane < p.tr) {
    const int r = scan8[lane];
    A[(r >> 3) * S.w + (r & 7)] = lane < p.zo ? out : 0;
  }
  if (lane + 32 < p.tr) {
    const int r = scan8[lane + 32];
    A[(r >> 3) * S.w + (r & 7)] = 0;
  }
  __syncwarp();
}

// dct.rs:996-1109 inverse_transform_rect_bd: A (dequantised, raster) -> A
// (residual, raster), B as the transposed intermediate (stride h + 1).
__device__ void tu_inverse_transform(int32_t* A, int32_t* B, const TuShape& S, int bd, int lane) {
  if (S.w == 1 || S.h == 1) {
    const bool col = S.w == 1;
    const int len = col ? S.h : S.w, lg = col ? S.lh : S.lw;
    const int8_t* m = tu_matrix(col ? S.tv : S.th, lg);
    const int cut = len - (col ? S.sh : S.sw);
    const int shift = 21 - bd, add = 1 << (shift - 1);
    int r[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int j = lane + 32 * q;
      int s = 0;
      if (j < len)
        for (int k = 0; k < cut; k++) s += (int)m[k * len + j] * A[k];
      r[q] = clip16i((s + add) >> shift);
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; q++)
      if (lane + 32 * q < len) A[lane + 32 * q] = r[q];
    __syncwarp();
    return;
  }
  const int8_t* mv = tu_matrix(S.tv, S.lh);
  const int8_t* mh = tu_matrix(S.th, S.lw);
  const int cw = S.w - S.sw, ch = S.h - S.sh;
  const int hs = S.h + 1;
  for (int id = lane; id < cw * S.h; id += 32) {
    const int i = id >> S.lh, j = id & (S.h - 1);
    int s = 0;
    for (int k = 0; k < ch; k++) s += (int)mv[k * S.h + j] * A[k * S.w + i];
    B[i * hs + j] = clip16i((s + 64) >> 7);
  }
  __syncwarp();
  const int sh2 = 20 - bd, add2 = 1 << (sh2 - 1);
  for (int id = lane; id < S.n; id += 32) {
    const int y = id >> S.lw, x = id & (S.w - 1);
    int s = 0;
    for (int k = 0; k < cw; k++) s += (int)mh[k * S.w + x] * B[k * hs + y];
    A[id] = clip16i((s + add2) >> sh2);
  }
  __syncwarp();
}

// dct.rs:865-991 forward_transform_rect_bd: A (residual, row stride w + 1)
// -> A (coefficients, raster, zero outside the kept region), B intermediate.
__device__ void tu_forward_transform(int32_t* A, int32_t* B, const TuShape& S, int bd, int lane) {
  const int ws = S.w + 1;
  if (S.w == 1 || S.h == 1) {
    const bool col = S.w == 1;
    const int len = col ? S.h : S.w, lg = col ? S.lh : S.lw;
    const int8_t* m = tu_matrix(col ? S.tv : S.th, lg);
    const int cut = len - (col ? S.sh : S.sw);
    const int shift = lg + bd + 6 - 15;
    const int add = shift > 0 ? 1 << (shift - 1) : 0;
    int r[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int v = lane + 32 * q;
      int s = 0;
      if (v < cut)
        for (int k = 0; k < len; k++) s += (int)m[v * len + k] * A[col ? k * ws : k];
      r[q] = v < cut ? clip16(shift >= 0 ? (long long)((s + add) >> shift) : (long long)s << (-shift)) : 0;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; q++)
      if (lane + 32 * q < len) A[lane + 32 * q] = r[q];
    __syncwarp();
    return;
  }
  const int8_t* mh = tu_matrix(S.th, S.lw);
  const int8_t* mv = tu_matrix(S.tv, S.lh);
  const int cw = S.w - S.sw, ch = S.h - S.sh;
  const int hs = S.h + 1;
  const int sh1 = S.lw + bd + 6 - 15;
  const int add1 = sh1 > 0 ? 1 << (sh1 - 1) : 0;
  for (int id = lane; id < cw * S.h; id += 32) {
    const int k = id >> S.lh, y = id & (S.h - 1);
    int s = 0;
    for (int x = 0; x < S.w; x++) s += (int)mh[k * S.w + x] * A[y * ws + x];
    B[k * hs + y] = (s + add1) >> sh1;  // not clipped (dct.rs:963)
  }
  __syncwarp();
  for (int i = lane; i < S.n; i += 32) A[i] = 0;
  __syncwarp();
  const int sh2 = S.lh + 6;
  const long long add2 = 1ll << (sh2 - 1);
  for (int id = lane; id < ch * cw; id += 32) {
    const int v = id / cw, k = id - v * cw;
    long long s = 0;
    for (int y = 0; y < S.h; y++) s += (long long)mv[v * S.h + y] * B[k * hs + y];
    A[v * S.w + k] = clip16((s + add2) >> sh2);
  }
  __syncwarp();
}

// ------------------------------------------------------- 16-bit warp path --

// Tile pitch (int16) of rows of up to n samples: whole 16-byte words and 8
// more, so that stores of one column spread over the banks.
__host__ __device__ constexpr int tu_pitch(int n) { return ((n + 7) & ~7) + 8; }

// Tile sizes (int16) of a unit with at most kMax coefficients, maximised over
// the shapes of the bin: inverse, coefficients transposed (<= 32x32) and the
// intermediate; forward, the residual (later the coefficients) and the
// intermediate. Transform skip with BDPCM uses the inverse's sum as one raster
// tile of w + 2 columns (units below 64x64).
struct TuTiles {
  int c, t, a, b;
};
__host__ __device__ constexpr TuTiles tu_tiles(int max_coeffs) {
  TuTiles r{0, 0, 0, 0};
  for (int lw = 0; lw <= 6; lw++)
    for (int lh = 0; lh <= 6; lh++) {
      const int w = 1 << lw, h = 1 << lh, cw = w < 32 ? w : 32, ch = h < 32 ? h : 32;
      if (w * h > max_coeffs) continue;
      const int c = cw * tu_pitch(ch), t = h * tu_pitch(cw), a = h * tu_pitch(w), b = cw * tu_pitch(h);
      r.c = c > r.c ? c : r.c;
      r.t = t > r.t ? t : r.t;
      r.a = a > r.a ? a : r.a;
      r.b = b > r.b ? b : r.b;
    }
  return r;
}
// int16 entries of a warp's workspace.
__host__ __device__ constexpr int tu_inv_ws(int max_coeffs) { return tu_tiles(max_coeffs).c + tu_tiles(max_coeffs).t; }
__host__ __device__ constexpr int tu_fwd_ws(int max_coeffs) { return tu_tiles(max_coeffs).a + tu_tiles(max_coeffs).b; }

// Row o of a transform's matrix as packed int8 words (padded to whole words):
// basis function o (forward) or every basis function's sample o (inverse).
__device__ __forceinline__ const uint32_t* tu_mat_row(bool inverse, int type, int log2n, int o) {
  return g_tm + c_tm_off[inverse ? 1 : 0][type][log2n] + o * (log2n <= 2 ? 1 : 1 << (log2n - 2));
}

// Where a pass puts output o of line l.
struct TuStore {
  int16_t* p;
  int so, sl;  // strides of outputs and lines
};

// One transform pass of a warp: for every output o < n_out of L lines,
// (sum_{k < 4 KW} M[o][k] in[l][k] + add) >> sh, clipped to 16 bits; returns
// whether any sum was outside them. Lines past the unit's last nonzero input
// may be cut to 4 KW < the transform's length by the caller, with zeros kept
// up to there.
template <int KW>
__device__ __forceinline__ bool tu_pass(const uint32_t* rows, int row_words, int lg_out, int L, const int16_t* in,
                                        int pin, const TuStore st, int add, int sh, int lane) {
  const int n = min(1 << lg_out, 32), lgn = min(lg_out, 5);
  bool wide = false;
  for (int o0 = 0; o0 < (1 << lg_out); o0 += 32) {
    const int o = o0 + (lane & (n - 1));
    const uint32_t* row = rows + o * row_words;
    uint32_t m[KW];
    if (KW >= 4) {
#pragma unroll
      for (int k = 0; k < KW; k += 4) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(row + k));
        m[k] = v.x;
        m[k + 1] = v.y;
        m[k + 2] = v.z;
        m[k + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < KW; k++) m[k] = __ldg(row + k);
    }
    int16_t* out = st.p + o * st.so;
#pragma unroll 2
    for (int l = lane >> lgn; l < L; l += 32 >> lgn) {
      const int16_t* r = in + l * pin;
      int s = add;
      if (KW == 1) {
        const uint2 v = *reinterpret_cast<const uint2*>(r);
        s = __dp2a_hi((int)v.y, (int)m[0], __dp2a_lo((int)v.x, (int)m[0], s));
      } else {
#pragma unroll
        for (int k = 0; k < KW / 2; k++) {
          const uint4 v = reinterpret_cast<const uint4*>(r)[k];
          s = __dp2a_hi((int)v.y, (int)m[2 * k], __dp2a_lo((int)v.x, (int)m[2 * k], s));
          s = __dp2a_hi((int)v.w, (int)m[2 * k + 1], __dp2a_lo((int)v.z, (int)m[2 * k + 1], s));
        }
      }
      s >>= sh;
      const int c = clip16i(s);
      wide |= c != s;
      out[l * st.sl] = (int16_t)c;
    }
  }
  return wide;
}

// tu_pass with kw (>= 1) input groups of four, rounded up to a power of two.
__device__ __noinline__ bool tu_pass_n(int kw, const uint32_t* rows, int row_words, int lg_out, int L,
                                       const int16_t* in, int pin, const TuStore st, int add, int sh, int lane) {
  if (kw <= 1) return tu_pass<1>(rows, row_words, lg_out, L, in, pin, st, add, sh, lane);
  if (kw <= 2) return tu_pass<2>(rows, row_words, lg_out, L, in, pin, st, add, sh, lane);
  if (kw <= 4) return tu_pass<4>(rows, row_words, lg_out, L, in, pin, st, add, sh, lane);
  if (kw <= 8) return tu_pass<8>(rows, row_words, lg_out, L, in, pin, st, add, sh, lane);
  return tu_pass<16>(rows, row_words, lg_out, L, in, pin, st, add, sh, lane);
}
__device__ __forceinline__ int tu_pow2_groups(int n) {  // inputs covered by tu_pass_n for n inputs
  return 4 << (n <= 4 ? 0 : 32 - __clz((n - 1) >> 2));
}

// Entry maps of the dependent quantiser's four states, two bits each: an even
// level swaps a state's bits (0 1 2 3 -> 0 2 1 3), an odd one also flips the
// high bit (-> 2 0 3 1; dct.rs:1238, table 32040).
__device__ __forceinline__ int dq_step(int st, int level) {
  return (((st & 1) << 1) | (st >> 1)) ^ ((level & 1) << 1);
}

// predict.rs:4224-4240: saturating running sums along rows or down columns,
// one lane a line, in place.
__device__ __noinline__ void tu_bdpcm(int16_t* p, int stride, const TuShape& S, bool vert, int lane) {
  const int lines = vert ? S.w : S.h, len = vert ? S.h : S.w;
  const int step = vert ? stride : 1, lstep = vert ? 1 : stride;
  for (int l = lane; l < lines; l += 32) {
    int16_t* q = p + (size_t)l * lstep;
    int acc = *q;
    for (int k = 1; k < len; k++) {
      q += step;
      acc = clip16i(*q + acc);
      *q = (int16_t)acc;
    }
  }
  __syncwarp();
}

// One warp: levels -> residual of one unit (decode_general.rs:4100-4199 and
// the BDPCM of :4055-4060). The residual goes to `out` with row stride
// `ostride` (0: the unit's width). ws: tu_inv_ws int16 entries, 16-byte
// aligned. Rows and columns past the last nonzero coefficient hold zeros and
// are left out of the sums. The levels are raster, or with npairs >= 0 the
// sparse form: `in` holds npairs (raster index, level) pairs, 4-byte aligned,
// with rising indices (units of at most 32x32); false when an index is outside
// the unit or not above the one before it (that entry is left out).
__device__ bool warp_tu_inverse(const vvcg_tu_rec& r, const int16_t* __restrict__ in,
                                int16_t* __restrict__ out, int16_t* ws, int lane, int ostride = 0, int npairs = -1) {
  TuShape S;
  tu_shape(r, S);
  const int bd = r.bit_depth, qp = r.qp;
  const int os = ostride ? ostride : S.w;
  const bool sparse = npairs >= 0;
  const bool vec = !sparse && (reinterpret_cast<uintptr_t>(in) & 15) == 0 && S.n >= 256;  // 8 levels a lane and load
  bool ok = true;
  // calls put(index, level) for this lane's sparse entries, each index checked
  // against the entry before it, so that no two land on one coefficient
  auto for_pairs = [&](auto&& put) {
    const uint32_t* pr = reinterpret_cast<const uint32_t*>(in);
    int prev_last = -1;
    for (int base = 0; base < npairs; base += 32) {
      const int i = base + lane;
      const bool have = i < npairs;
      const uint32_t e = have ? pr[i] : (uint32_t)S.n;
      const int pos = (int)(e & 0xFFFFu), L = (int)(int16_t)(e >> 16);
      int prev = __shfl_up_sync(0xffffffffu, pos, 1);
      if (lane == 0) prev = prev_last;
      if (have) {
        if (pos >= S.n || pos <= prev)
          ok = false;
        else if (L != 0)
          put(pos, L);
      }
      prev_last = __shfl_sync(0xffffffffu, pos, 31);
    }
    ok = __all_sync(0xffffffffu, ok);
  };
  const bool bdpcm = (r.flags & (VVCG_TU_BDPCM_HOR | VVCG_TU_BDPCM_VER)) != 0;
  if (r.flags & VVCG_TU_TRANSFORM_SKIP) {
    // BDPCM sums in the workspace, except for 64x64, which does not fit
    const bool tile = bdpcm && S.n < 4096;
    int16_t* d = tile ? ws : out;
    const int ds = tile ? S.w + 2 : os;
    if (sparse) {
      for (int i = lane; i < S.n; i += 32) d[(size_t)(i >> S.lw) * ds + (i & (S.w - 1))] = 0;
      __syncwarp();
      for_pairs([&](int i, int L) { d[(size_t)(i >> S.lw) * ds + (i & (S.w - 1))] = (int16_t)tu_dequant_ts(L, qp); });
    } else {
      for (int i = lane; i < S.n; i += 32)
        d[(size_t)(i >> S.lw) * ds + (i & (S.w - 1))] = (int16_t)tu_dequant_ts(in[i], qp);
    }
    __syncwarp();
    if (bdpcm) tu_bdpcm(d, ds, S, (r.flags & VVCG_TU_BDPCM_VER) != 0, lane);
    if (tile)
      for (int i = lane; i < S.n; i += 32)
        out[(size_t)(i >> S.lw) * os + (i & (S.w - 1))] = ws[(i >> S.lw) * ds + (i & (S.w - 1))];
    __syncwarp();
    return ok;
  }
  // coefficients transposed: C[x][y], x < 32, y < 32
  const int tw = min(S.w, 32), th = min(S.h, 32);
  const int pc = tu_pitch(th), pt = tu_pitch(tw);
  int16_t* C = ws;
  int16_t* T = ws + tw * pc;
  const bool dq = (r.flags & VVCG_TU_DEP_QUANT) != 0;
  const bool lfnst = r.lfnst_idx > 0 && r.mts_idx == 0;
  bool s2;
  const int tr_shift = tu_tr_shift(S.lw, S.lh, bd, &s2);
  const int q4 = max(4, qp);
  const int rs = 6 - (tr_shift + q4 / 6);
  const long long scale = c_inv_quant_scale[s2 ? 1 : 0][q4 % 6];
  const int scan_at = g_tu_scan_off[S.lw * 7 + S.lh];
  int maxr = -1, maxc = -1, lastpos = -1;
  uint4 buf[4];
  if (vec) {
#pragma unroll
    for (int v = 0; v < 4; v++)
      if (8 * (lane + 32 * v) < S.n) buf[v] = reinterpret_cast<const uint4*>(in)[lane + 32 * v];
  }
  for (int i = lane; i < (tw * pc) / 8; i += 32) reinterpret_cast<uint4*>(C)[i] = make_uint4(0, 0, 0, 0);
  __syncwarp();
  auto put = [&](int i, int L) {
    const int y = i >> S.lw, x = i & (S.w - 1);
    if (x >= tw || y >= th) return;  // outside the scan and the kept coefficients of 64-point units
    maxr = max(maxr, y);
    maxc = max(maxc, x);
    int v = L;
    if (dq) {
      lastpos = max(lastpos, (int)g_tu_scan_pos[scan_at + y * tw + x]);
    } else {  // dct.rs:1151-1187 dequantize_rect_bd
      const long long p = (long long)L * scale;
      v = clip16(rs > 0 ? (p + (1ll << (rs - 1))) >> rs : p << (-rs));
    }
    C[x * pc + y] = (int16_t)v;
  };
  if (sparse) {
    for_pairs(put);
  } else if (vec) {
    for (int v0 = 0; v0 < S.n; v0 += 1024) {
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const int at = v0 + 8 * (lane + 32 * v);
        if (at >= S.n) continue;
        uint32_t x0 = buf[v].x, x1 = buf[v].y, x2 = buf[v].z, x3 = buf[v].w;
        if (at + 1024 < S.n) buf[v] = *reinterpret_cast<const uint4*>(in + at + 1024);
        if ((x0 | x1 | x2 | x3) == 0) continue;  // 8 zero levels (most of a unit)
#pragma unroll 1
        for (int e = 0; e < 8; e++) {
          const int L = (int)(int16_t)(x0 & 0xFFFFu);
          if (L != 0) put(at + e, L);
          x0 = __funnelshift_r(x0, x1, 16);
          x1 = __funnelshift_r(x1, x2, 16);
          x2 = __funnelshift_r(x2, x3, 16);
          x3 >>= 16;
        }
      }
    }
  } else {
    for (int i = lane; i < S.n; i += 32) {
      const int L = in[i];
      if (L != 0) put(i, L);
    }
  }
  if (dq) {
    // dequantize_dep_quant_bd (dct.rs:1191-1248): the scan is walked backwards
    // from the last nonzero level, 32 chunks at once (dq_entry_state)
    __syncwarp();
    const int16_t* scan = g_tu_scan + scan_at;
    const int last = __reduce_max_sync(0xffffffffu, lastpos);
    if (last >= 0) {
      int lo, hi;
      dq_chunk(last, lane, lo, hi);
      uint32_t map = 0xE4u;
      for (int s = hi; s >= lo; s--) {
        const int i = scan[s];
        const int L = C[(i & (S.w - 1)) * pc + (i >> S.lw)];
        map = (((map & 0x55u) << 1) | ((map >> 1) & 0x55u)) ^ ((L & 1) ? 0xAAu : 0u);
      }
      int st = dq_entry_state(map, lane);
      const int qp_dq = q4 + 1;
      const int shift = 7 - qp_dq / 6 - tr_shift;
      long long inv_q = c_inv_quant_scale[s2 ? 1 : 0][qp_dq % 6];
      if (shift < 0) inv_q <<= -shift;
      const long long add = shift > 0 ? (1ll << (shift - 1)) : 0;
      const int rsh = max(0, shift);
      __syncwarp();
      for (int s = hi; s >= lo; s--) {
        const int i = scan[s];
        int16_t* p = &C[(i & (S.w - 1)) * pc + (i >> S.lw)];
        const int L = *p;
        if (L != 0) {
          const long long q = (long long)(2 * L + (L > 0 ? -(st >> 1) : (st >> 1)));
          *p = (int16_t)clip16((q * inv_q + add) >> rsh);
        }
        st = dq_step(st, L);
      }
    }
  }
  maxr = __reduce_max_sync(0xffffffffu, maxr);
  maxc = __reduce_max_sync(0xffffffffu, maxc);
  __syncwarp();
  if (lfnst) {  // lfnst.rs:219-294 inverse_lfnst_rect
    const LfnstParams p = lfnst_params(S, r.lfnst_idx, r.lfnst_mode);
    const int16_t* scan8 = tu_scan(3, 3);
    int o[2] = {0, 0};
    for (int i = 0; i < p.zo; i++) {
      const int k = scan8[i];
      const int v = C[(k & 7) * pc + (k >> 3)];
      if (lane < p.tr) o[0] += v * (int)p.m[i * p.tr + lane];
      if (lane + 32 < p.tr) o[1] += v * (int)p.m[i * p.tr + lane + 32];
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int j = lane + 32 * q;
      if (j < p.tr) {
        const int at = lfnst_pos(j, p.sb, p.transposed, 8);
        C[(at & 7) * pc + (at >> 3)] = (int16_t)clip16i((o[q] + 64) >> 7);
      }
    }
    maxr = max(maxr, p.sb - 1);
    maxc = max(maxc, p.sb - 1);
    __syncwarp();
  }
  // dct.rs:996-1109 inverse_transform_rect_bd
  if (S.w == 1 || S.h == 1) {
    const bool col = S.w == 1;
    const int len = col ? S.h : S.w, lg = col ? S.lh : S.lw;
    const int8_t* m = tu_matrix(col ? S.tv : S.th, lg);
    const int cut = min(len - (col ? S.sh : S.sw), max(maxr, maxc) + 1);
    const int shift = 21 - bd, add = 1 << (shift - 1), stride = col ? 1 : pc;
    for (int j = lane; j < len; j += 32) {
      int s = 0;
      for (int k = 0; k < cut; k++) s += (int)m[k * len + j] * C[k * stride];
      out[(size_t)j * (col ? os : 1)] = (int16_t)clip16i((s + add) >> shift);
    }
    __syncwarp();
    if (bdpcm) tu_bdpcm(out, os, S, (r.flags & VVCG_TU_BDPCM_VER) != 0, lane);
    return ok;
  }
  const int nc = min(S.w - S.sw, maxc + 1), nr = min(S.h - S.sh, maxr + 1);
  if (nc <= 0 || nr <= 0) {
    for (int i = lane; i < S.n; i += 32) out[(size_t)(i >> S.lw) * os + (i & (S.w - 1))] = 0;
    __syncwarp();
    return ok;
  }
  // coefficients the zero-out drops inside the last group (the other rows
  // and columns up to the groups read are zero already or not read)
  const int kr = tu_pow2_groups(nr), kc = tu_pow2_groups(nc);
  if (nr <= maxr && (S.h - S.sh) < kr)
    for (int i = lane; i < nc * (kr - nr); i += 32) C[(i / (kr - nr)) * pc + nr + i % (kr - nr)] = 0;
  for (int i = lane; i < S.h * (kc - nc); i += 32) T[(i / (kc - nc)) * pt + nc + i % (kc - nc)] = 0;
  __syncwarp();
  tu_pass_n(kr >> 2, tu_mat_row(true, S.tv, S.lh, 0), S.lh <= 2 ? 1 : 1 << (S.lh - 2), S.lh, nc, C, pc,
            TuStore{T, pt, 1}, 64, 7, lane);
  __syncwarp();
  tu_pass_n(kc >> 2, tu_mat_row(true, S.th, S.lw, 0), S.lw <= 2 ? 1 : 1 << (S.lw - 2), S.lw, S.h, T, pt,
            TuStore{out, 1, os}, 1 << (19 - bd), 20 - bd, lane);
  __syncwarp();
  if (bdpcm) tu_bdpcm(out, os, S, (r.flags & VVCG_TU_BDPCM_VER) != 0, lane);
  return ok;
}

// One warp: residual -> levels of one unit (slice.rs:690-760, level side).
// ws: tu_fwd_ws int16 entries, 16-byte aligned; low: 16 int32 entries.
__device__ void warp_tu_forward(const vvcg_tu_rec& r, const int16_t* __restrict__ in,
                                int16_t* __restrict__ out, int16_t* ws, int32_t* low, int lane) {
  TuShape S;
  tu_shape(r, S);
  const int bd = r.bit_depth, qp = r.qp;
  if (r.flags & VVCG_TU_TRANSFORM_SKIP) {
    for (int i = lane; i < S.n; i += 32) out[i] = (int16_t)tu_quant_ts(in[i], qp);
    return;
  }
  const int pa = tu_pitch(S.w), tw = min(S.w, 32), th = min(S.h, 32);
  int16_t* A = ws;                // residual rows, then the coefficients (raster, pitch pc)
  int16_t* B = ws + S.h * pa;
  const int cw = S.w - S.sw, ch = S.h - S.sh;
  const int pc = S.w == 1 || S.h == 1 ? S.w : tw + 2;
  if ((reinterpret_cast<uintptr_t>(in) & 15) == 0 && S.w >= 8) {
    for (int i = lane; i < S.n >> 3; i += 32) {
      const int e = 8 * i;
      *reinterpret_cast<uint4*>(A + (e >> S.lw) * pa + (e & (S.w - 1))) =
          __ldcs(reinterpret_cast<const uint4*>(in) + i);
    }
  } else {
    for (int i = lane; i < S.n; i += 32) A[(i >> S.lw) * pa + (i & (S.w - 1))] = in[i];
    if (S.w < 4)  // the packed product reads four samples a row
      for (int i = lane; i < S.h * (4 - S.w); i += 32) A[(i / (4 - S.w)) * pa + S.w + i % (4 - S.w)] = 0;
  }
  __syncwarp();
  // dct.rs:865-991 forward_transform_rect_bd
  int16_t* C = A;
  if (S.w == 1 || S.h == 1) {
    const bool col = S.w == 1;
    const int len = col ? S.h : S.w, lg = col ? S.lh : S.lw;
    const int8_t* m = tu_matrix(col ? S.tv : S.th, lg);
    const int cut = len - (col ? S.sh : S.sw);
    const int shift = lg + bd + 6 - 15;
    const int add = shift > 0 ? 1 << (shift - 1) : 0;
    int v[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int o = lane + 32 * q;
      int s = 0;
      if (o < cut)
        for (int k = 0; k < len; k++) s += (int)m[o * len + k] * A[col ? k * pa : k];
      v[q] = o < cut ? clip16(shift >= 0 ? (long long)((s + add) >> shift) : (long long)s << (-shift)) : 0;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; q++)
      if (lane + 32 * q < len) C[lane + 32 * q] = (int16_t)v[q];
    __syncwarp();
  } else {
    const int pb = tu_pitch(S.h);
    const int sh1 = S.lw + bd + 6 - 15, add1 = sh1 > 0 ? 1 << (sh1 - 1) : 0;
    const int lcw = ilog2(cw);
    if (S.h < 4) {
      for (int i = lane; i < cw * (4 - S.h); i += 32) B[(i / (4 - S.h)) * pb + S.h + i % (4 - S.h)] = 0;
      __syncwarp();
    }
    bool wide = tu_pass_n(max(1, S.w >> 2), tu_mat_row(false, S.th, S.lw, 0), S.lw <= 2 ? 1 : 1 << (S.lw - 2), lcw,
                          S.h, A, pa, TuStore{B, pb, 1}, add1, sh1, lane);
    wide = __any_sync(0xffffffffu, wide);
    __syncwarp();
    const int sh2 = S.lh + 6;
    if (!wide) {
      for (int i = lane; i < th * pc; i += 32) C[i] = 0;
      __syncwarp();
      tu_pass_n(max(1, S.h >> 2), tu_mat_row(false, S.tv, S.lh, 0), S.lh <= 2 ? 1 : 1 << (S.lh - 2), ilog2(ch), cw, B,
                pb, TuStore{C, pc, 1}, 1 << (sh2 - 1), sh2, lane);
    } else {
      // the first stage's outputs as low 15 bits (B) and the rest (in `out`,
      // which is written last), summed in 64 bits
      const int8_t* mh = tu_matrix(S.th, S.lw);
      const int8_t* mv = tu_matrix(S.tv, S.lh);
      for (int id = lane; id < cw * S.h; id += 32) {
        const int k = id >> S.lh, y = id & (S.h - 1);
        int s = 0;
        for (int x = 0; x < S.w; x++) s += (int)mh[k * S.w + x] * A[y * pa + x];
        s = (s + add1) >> sh1;
        B[k * pb + y] = (int16_t)(s & 0x7FFF);
        out[id] = (int16_t)(s >> 15);
      }
      __threadfence_block();
      __syncwarp();
      for (int i = lane; i < th * pc; i += 32) C[i] = 0;
      __syncwarp();
      for (int id = lane; id < ch * cw; id += 32) {
        const int v = id / cw, k = id - v * cw;
        long long s = 1ll << (sh2 - 1);
        for (int y = 0; y < S.h; y++)
          s += (long long)mv[v * S.h + y] * (((long long)out[k * S.h + y] << 15) + B[k * pb + y]);
        C[v * pc + k] = (int16_t)clip16(s >> sh2);
      }
    }
    __syncwarp();
  }
  const bool lfnst = r.lfnst_idx > 0;
  if (lfnst) {
    // lfnst.rs:131-205 forward_lfnst_rect; its outputs are not clipped: the
    // first 16 positions of the 8x8 scan (all inside the top-left 4x4) are
    // kept in 32 bits, the other positions it covers become zero
    const LfnstParams p = lfnst_params(S, r.lfnst_idx, r.lfnst_mode);
    const int16_t* scan8 = tu_scan(3, 3);
    auto src = [&](int j) -> int {
      const int at = lfnst_pos(j, p.sb, p.transposed, 8);
      return C[(at >> 3) * pc + (at & 7)];
    };
    const int s0 = lane < p.tr ? src(lane) : 0, s1 = lane + 32 < p.tr ? src(lane + 32) : 0;
    int o = 0;
    for (int i = 0; i < p.tr; i++) {
      const int v = __shfl_sync(0xffffffffu, i < 32 ? s0 : s1, i & 31);
      if (lane < p.zo) o += v * (int)p.m[lane * p.tr + i];
    }
    __syncwarp();
    for (int j = lane; j < p.tr; j += 32) {
      const int k = scan8[j];
      C[(k >> 3) * pc + (k & 7)] = 0;
      if (j < 16) low[(k >> 3) * 4 + (k & 7)] = j < p.zo ? (o + 64) >> 7 : 0;
    }
    __syncwarp();
  }
  // coefficient at (x, y); the levels replace the coefficients in C
  auto coeff = [&](int x, int y) -> int { return lfnst && x < 4 && y < 4 ? low[y * 4 + x] : C[y * pc + x]; };
  bool s2;
  const int tr_shift = tu_tr_shift(S.lw, S.lh, bd, &s2);
  const int ns = tw * th;
  if (r.flags & VVCG_TU_DEP_QUANT) {
    // dct.rs:1252-1301 quantize_dep_quant_bd: a level depends on the state
    // only through its high bit, so a position maps the four states
    const int16_t* scan = tu_scan(S.lw, S.lh);
    const int qp_dq = max(4, qp) + 1;
    const int q_shift = 13 + qp_dq / 6 + tr_shift;
    const long long q_scale = c_quant_scale[s2 ? 1 : 0][qp_dq % 6];
    const long long half = 1ll << max(0, q_shift - 1);
    auto qest = [&](int c) -> long long { return ((long long)abs(c) * q_scale + half) >> max(0, q_shift); };
    auto level_of = [&](long long est, int c, int off) -> int {
      const int a = est <= off ? 0 : (int)((est + off + 1) >> 1);
      return clampi(c < 0 ? -a : a, -32768, 32767);
    };
    int lo, hi;
    dq_chunk(ns - 1, lane, lo, hi);
    uint32_t map = 0xE4u;
    for (int s = hi; s >= lo; s--) {
      const int i = scan[s];
      const int c = coeff(i & (S.w - 1), i >> S.lw);
      const long long est = qest(c);
      uint32_t step = 0xD8u;
      if (est > 0) {
        if (level_of(est, c, 0) & 1) step ^= 0x0Au;
        if (level_of(est, c, 1) & 1) step ^= 0xA0u;
      }
      uint32_t next = 0;
#pragma unroll
      for (int q = 0; q < 4; q++) next |= ((step >> (2 * ((map >> (2 * q)) & 3))) & 3) << (2 * q);
      map = next;
    }
    int st = dq_entry_state(map, lane);
    for (int s = hi; s >= lo; s--) {
      const int i = scan[s], x = i & (S.w - 1), y = i >> S.lw;
      const int c = coeff(x, y);
      const int L = level_of(qest(c), c, st >> 1);
      C[y * pc + x] = (int16_t)L;
      st = dq_step(st, L);
    }
  } else {
    // dct.rs:1113-1147 quantize_rect_bd
    const int q = max(4, qp);
    const int qbits = 14 + q / 6 + tr_shift;
    const long long add = (long long)((r.flags & VVCG_TU_INTER) ? 85 : 171) << max(0, qbits - 9);
    const long long scale = c_quant_scale[s2 ? 1 : 0][q % 6];
    const int ltw = ilog2(tw);
    for (int i = lane; i < ns; i += 32) {
      const int x = i & (tw - 1), y = i >> ltw;
      const int c = coeff(x, y);
      const long long lv = ((long long)abs(c) * scale + add) >> max(0, qbits);
      C[y * pc + x] = (int16_t)clip16(c < 0 ? -lv : lv);
    }
  }
  __syncwarp();
  for (int i = lane; i < S.n; i += 32) {
    const int y = i >> S.lw, x = i & (S.w - 1);
    out[i] = x < tw && y < th ? C[y * pc + x] : (int16_t)0;
  }
}

// Grid: ceil(units / warps); each warp takes idx[blockIdx.x * warps + warp].
template <int kMax, int kWarps, bool kForward>
__global__ void __launch_bounds__(kWarps * 32)
k_tu(const vvcg_tu_rec* __restrict__ recs, const uint32_t* __restrict__ idx, uint32_t n,
     const int16_t* __restrict__ in, int16_t* __restrict__ out) {
  extern __shared__ __align__(16) int16_t tu_smem[];
  __shared__ int32_t low[kWarps][16];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t t = blockIdx.x * kWarps + wid;
  if (t >= n) return;
  constexpr int kWs = kForward ? tu_fwd_ws(kMax) : tu_inv_ws(kMax);
  static_assert(kWs % 8 == 0, "16-byte aligned workspaces");
  int16_t* ws = tu_smem + wid * kWs;
  const vvcg_tu_rec r = recs[idx[t]];
  if (kForward)
    warp_tu_forward(r, in + r.in_off, out + r.out_off, ws, low[wid], lane);
  else
    warp_tu_inverse(r, in + r.in_off, out + r.out_off, ws, lane);
}

template <int kMax, int kWarps>
constexpr size_t tu_smem_bytes(bool forward) {
  return (size_t)kWarps * (forward ? tu_fwd_ws(kMax) : tu_inv_ws(kMax)) * sizeof(int16_t);
}

// True when TB c of a coding unit with tu_tools `t` leaves the frame path's
// DCT-2 residual kernel: transform skip, or (luma) explicit MTS / LFNST.
__host__ __device__ __forceinline__ bool tb_uses_tu_tools(uint32_t t, int c) {
  return ((t >> c) & 1) || (c == 0 && (t >> VVCG_CU_MTS_SHIFT) != 0);
}

constexpr int kResToolWarps = 4;

// The frame path's TBs with per-TB transform choices (pictures with
// VVCG_TOOL_TU_TOOLS; slice.rs:1050-1097 reconstruct_block, residual part):
// one warp per coding unit runs each such coded TB through the TU path above
// (transform-skip dequantisation, or dequantisation, inverse LFNST with the
// CU's luma mode, inverse DCT-2 / DST-7 / DCT-8 with the zero-out) into the
// scratch planes, where the reconstruction adds it to the prediction.
// Records outside the ranges of vvcg_cu_rec.tu_tools, or with levels past the
// pool, set the bad-record status and are skipped.
// Grid: (ceil(max CUs per picture / kResToolWarps), pictures).
__global__ void __launch_bounds__(kResToolWarps * 32)
k_residual_tools(const DevPic* __restrict__ pics, const int16_t* __restrict__ levels, uint64_t n_levels,
                 uint32_t* status) {
  __shared__ __align__(16) int16_t ws[kResToolWarps][tu_inv_ws(1024)];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const DevPic& P = pics[blockIdx.y];
  if (!(P.tools & VVCG_TOOL_TU_TOOLS)) return;
  const int cu = blockIdx.x * kResToolWarps + wid;
  if (cu >= P.grid_w * P.grid_h) return;
  const vvcg_cu_rec rec = P.cus[cu];
  const uint32_t t = rec.tu_tools;
  if (!t) return;
  const int mts = (t >> VVCG_CU_MTS_SHIFT) & 7, lfnst = t >> VVCG_CU_LFNST_SHIFT;
  const bool bad_tools = mts > 4 || lfnst > 2 || (mts && lfnst) || ((t & VVCG_CU_TS_Y) && (mts || lfnst));
  const bool sparse = (P.tools & VVCG_TOOL_SPARSE_LEVELS) != 0;
  const int gx = cu % P.grid_w, gy = cu / P.grid_w;
  for (int c = 0; c < (P.cf ? 3 : 1); c++) {
    if (!tb_uses_tu_tools(t, c) || !((rec.cbf >> c) & 1)) continue;
    const int off = rec.level_off[c];
    if (off < 0) continue;
    const int w = c ? P.tb_cw : P.tb, h = c ? P.tb_ch : P.tb;
    int cnt = -1;
    bool ok = !bad_tools;
    if (sparse) {  // count at levels[off], pairs from off + 2 (off even)
      cnt = (off & 1) || (uint64_t)off + 2 > n_levels ? -1 : levels[off];
      ok = ok && cnt >= 0 && cnt <= w * h && (uint64_t)off + 2 + 2 * (uint64_t)cnt <= n_levels;
    } else {
      ok = ok && (uint64_t)off + (uint64_t)(w * h) <= n_levels;
    }
    if (!ok) {
      if (lane == 0) atomicOr(status, kStatusBadRecord);
      continue;
    }
    const bool ts = (t >> c) & 1;
    const int q = c ? P.cqp : P.lqp;
    vvcg_tu_rec r;
    r.log2_w = (uint8_t)ilog2(w);
    r.log2_h = (uint8_t)ilog2(h);
    r.bit_depth = (uint8_t)P.bd;
    r.qp = (uint8_t)(ts ? max(4, q) : q);
    r.flags = ts ? VVCG_TU_TRANSFORM_SKIP : ((P.tools & VVCG_TOOL_DEP_QUANT) ? VVCG_TU_DEP_QUANT : 0);
    r.mts_idx = (uint8_t)(c ? 0 : mts);
    r.lfnst_idx = (uint8_t)(c ? 0 : lfnst);
    r.lfnst_mode = rec.luma_mode;
    r.in_off = r.out_off = 0;
    const int x0 = c ? gx * P.tb / P.sub_w : gx * P.tb, y0 = c ? gy * P.tb / P.sub_h : gy * P.tb;
    int16_t* out = reinterpret_cast<int16_t*>(P.scratch[c]) + (size_t)y0 * P.stride[c] + x0;
    if (!warp_tu_inverse(r, levels + off + (sparse ? 2 : 0), out, ws[wid], lane, P.stride[c], cnt) && lane == 0)
      atomicOr(status, kStatusBadRecord);
  }
}

}  // namespace vvcg
