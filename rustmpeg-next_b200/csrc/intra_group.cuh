// Intra prediction of the 8..12-bit frame path by a group of threads: the
// reference gather, the mode's reference arrays, the prediction of runs of
// eight samples, and the CCLM models. The wavefront kernels give each colour
// component of a coding unit such a group, so that a coding unit takes one L2
// round trip and a few barriers instead of one warp's serial walk over 1,536
// samples. The arithmetic is that of the reference functions named beside
// each part (crates/rustmpeg-video/src/vvc/predict.rs), bit for bit.
//
// Layout: a block's w x h samples (w, h in {16, 32}) are cut into runs of
// eight samples along the prediction's main direction: along x for planar,
// DC, CCLM and the vertical angular modes, along y for the horizontal ones.
// Along a run the slope's offset and taps are constants, so eight outputs need
// eleven reference samples: packed pairs and dp2a (16-bit samples x 8-bit
// taps) make that about 12 instructions a sample instead of 50 for one sample
// at a time. The runs go through a shared tile, which transposes the
// horizontal modes and gives every store 16 bytes.
#pragma once
#include "intra.cuh"

namespace vvcg {

// A group: `n` threads (a multiple of 32, whole warps) with named barrier
// `bar` (1..3); one warp alone needs no barrier. The barrier numbers are
// constants in the code: a number in a register makes a kernel reserve all 16
// hardware barriers, which leaves room for only 4 CTAs on an SM.
struct Grp {
  int tid, n, bar;
  __device__ __forceinline__ void sync() const {
    if (n == 32)
      __syncwarp();
    else if (bar == 1)
      asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
    else if (bar == 2)
      asm volatile("bar.sync 2, %0;" ::"r"(n) : "memory");
    else
      asm volatile("bar.sync 3, %0;" ::"r"(n) : "memory");
  }
};

// A block's references: a[0] = l[0] the corner, a[1 + i] the row above
// (2w samples), l[1 + j] the column to the left (2h samples).
struct RawRefs {
  int16_t a[72], l[72];
};

// The arrays a mode predicts from: main[kMainBase + k], k = -32..2n+2, the
// reference along the main direction (k = 0 the corner, k < 0 the projected
// side of negative slopes), and side[k], k = 0..2n. The extremes of k over all
// modes and block shapes of the frame path (32x32, 16x16, 16x32) are -32,
// 2n + 2 and 2n; loads of whole words reach at most 4 entries further.
constexpr int kMainBase = 34;
struct ModeRefs {
  int16_t main[112];
  int16_t side[80];
};

// A component's prediction mode with what the group's threads need of it.
struct ModeInfo {
  int16_t mode;     // 0..66, larger: predicts zeros
  int16_t angle;
  int16_t abs_inv;
  int8_t scale;     // PDPC scale (non-negative where pdpc is set)
  uint8_t flags;    // kMode*
};
enum : uint8_t { kModeVer = 1, kModeFilter = 2, kModeInterp = 4, kModePdpc = 8, kModeLuma = 16 };

// The parameters of a mode for a w x h block (one thread; the group reads the
// result from shared memory).
__device__ __forceinline__ ModeInfo mode_info(int mode, int w, int h, bool is_luma) {
  ModeInfo m{(int16_t)mode, 0, 0, 0, (uint8_t)((is_luma ? kModeLuma : 0) | kModeVer)};
  if (mode >= 2 && mode <= 66) {
    const AngP p = angular_params(mode, w, h, is_luma);
    const int ww = p.is_ver ? w : h, wh = p.is_ver ? h : w;
    m.angle = (int16_t)p.angle;
    m.abs_inv = (int16_t)(p.angle == 0 ? 0 : p.abs_inv);
    m.scale = (int8_t)(p.angle == 0 ? (ilog2(ww) + ilog2(wh) - 2) >> 2 : p.scale);
    m.flags = (uint8_t)((is_luma ? kModeLuma : 0) | (p.is_ver ? kModeVer : 0) | (p.ref_filter ? kModeFilter : 0) |
                        (p.interp ? kModeInterp : 0) | (p.pdpc ? kModePdpc : 0));
  } else if (mode == 0 && is_luma) {
    m.flags |= kModeFilter;  // luma blocks are 32x32: planar filters blocks above 32 samples
  }
  return m;
}

// The reference entries of a block, one after another: 2w above, 2h left, the
// corner, then (luma of a CCLM unit) the samples of the CclmRefs below.
// gather_references_16 (predict.rs:3016-3076) with the coded-unit
// substitution of predict_coded_block_16 (:3101-3135).
struct RefGeo {
  const uint16_t* at;   // the block's first sample
  int st, w, h, def;
  bool ha, hl, ar, bl;  // row above, column left, above-right and below-left samples exist
};

// Entry e < 2 (w + h) + 1: its value into the raw references.
__device__ __forceinline__ int ref_offset(const RefGeo& G, int e) {
  const int nw = 2 * G.w;
  int o;
  if (e < nw) {
    o = (e >= G.w && !G.ar ? G.w - 1 : e) - G.st;
    if (!G.ha) o = -1;  // filled with the first left sample
  } else {
    const int j = e - nw;
    const bool corner = j == 2 * G.h;
    o = (corner ? -1 : (j >= G.h && !G.bl ? G.h - 1 : j)) * G.st - 1;
    if (corner && !G.ha) o = -1;
    if (!G.hl) o = -G.st;  // filled with the first above sample
  }
  return o;
}

__device__ __forceinline__ void ref_put(int w, int h, int e, int v, RawRefs& R) {
  if (e < 2 * w)
    R.a[1 + e] = (int16_t)v;
  else if (e < 2 * (w + h))
    R.l[1 + e - 2 * w] = (int16_t)v;
  else
    R.a[0] = R.l[0] = (int16_t)v;
}

// One entry of a reference array: sample k of r (o: the other side), with the
// [1 2 1] filter of ReferenceSamples16::filtered (predict.rs:2970-3005).
__device__ __forceinline__ int ref_value(const int16_t* r, const int16_t* o, int k, int n, bool filt) {
  const int v = r[k];
  if (!filt || k == 2 * n) return v;
  const int prev = k == 0 ? o[1] : r[k - 1];
  return (prev + 2 * v + r[k + 1] + 2) >> 2;
}

// The mode's arrays from the raw references (planar: predict_from_refs_16;
// angular: predict_angular_16, predict.rs:3240-3305): entries 1..2n of the main
// side, then 1..2n of the other side, or the projected entries of a negative
// slope. The caller syncs after.
__device__ __forceinline__ void group_prep(int tid, int n, const ModeInfo& m, int w, int h, const RawRefs& R,
                                           ModeRefs& S) {
  if (m.mode == 1 || m.mode > 66) return;
  const bool ver = (m.flags & kModeVer) != 0, filt = (m.flags & kModeFilter) != 0;
  const int16_t* rm = ver ? R.a : R.l;
  const int16_t* ro = ver ? R.l : R.a;
  const int ww = ver ? w : h, wh = ver ? h : w;
  const bool neg = m.angle < 0;
  for (int e = tid; e < 2 * (ww + wh); e += n) {
    if (e < 2 * ww) {
      const int v = ref_value(rm, ro, e + 1, ww, filt);
      S.main[kMainBase + 1 + e] = (int16_t)v;
      if (e == 0) S.main[kMainBase] = (int16_t)ref_value(rm, ro, 0, ww, filt);
      if (e == 2 * ww - 1) S.main[kMainBase + 2 + e] = S.main[kMainBase + 3 + e] = (int16_t)v;
    } else {
      const int k = e - 2 * ww + 1;
      if (!neg)
        S.side[k] = (int16_t)ref_value(ro, rm, k, wh, filt);
      else if (k <= wh)
        S.main[kMainBase - k] = (int16_t)ref_value(ro, rm, min((k * m.abs_inv + 256) >> 9, wh), wh, filt);
    }
  }
}

// The DC value (predict.rs:3150-3180), by one whole warp.
__device__ __forceinline__ int warp_dc(const RawRefs& R, int w, int h, int maxv) {
  const int lane = threadIdx.x & 31;
  const int lw = ilog2(w), lh = ilog2(h);
  const unsigned st = __reduce_add_sync(0xffffffffu, lane < w ? (unsigned)R.a[1 + lane] : 0u);
  const unsigned sl = __reduce_add_sync(0xffffffffu, lane < h ? (unsigned)R.l[1 + lane] : 0u);
  const unsigned v = w == h ? (st + sl + (unsigned)w) >> (lw + 1)
                            : (w > h ? (st + ((unsigned)w >> 1)) >> lw : (sl + ((unsigned)h >> 1)) >> lh);
  return (int)min(v & 0xFFFFu, (unsigned)maxv);
}

// Tiles of predictions: raster rows of up to 32 samples at a pitch of 40, so
// that 16-byte accesses of eight rows in one column touch all banks once.
constexpr int kTilePitch = 40;

// Predicts run r of a block into its tile: planar / DC with apply_pdpc_16
// (predict.rs:3138-3215), angular with its PDPC (:3305-3410), zeros for other
// mode values (:3194). Neighbouring lanes take neighbouring lines, so the PDPC
// of a line's first samples stays in the warps that hold them. The reference
// clips planar, DC and positive-slope PDPC values too; those are weighted
// means of samples and cannot leave the range.
__device__ __forceinline__ void predict_run(int r, const ModeInfo& m, int w, int h, int bd, int dc, const RawRefs& R,
                                            const ModeRefs& S, int16_t* tile) {
  const bool ver = (m.flags & kModeVer) != 0;
  const int lw = ilog2(w), lh = ilog2(h);
  const int lwh = ver ? lh : lw;
  const int x0 = 8 * (r >> lwh), yy = r & ((1 << lwh) - 1);
  int v[8];
  if (m.mode >= 2 && m.mode <= 66) {
    // One 4-tap filter over main[j..j+3], j = di + x, covers every slope:
    // whole-sample slopes take main[j + 1] (taps 0 64 0 0), chroma's linear
    // interpolation is taps 0, 2 (32 - f), 2 f, 0, luma takes the Gaussian or
    // cubic taps.
    const int dp = m.angle * (yy + 1);
    const int di = dp >> 5, fr = dp & 31;
    uint32_t taps;
    if ((m.angle & 0x1F) == 0)
      taps = 64u << 8;
    else if (!(m.flags & kModeLuma))
      taps = (uint32_t)(2 * (32 - fr)) << 8 | (uint32_t)(2 * fr) << 16;
    else if (m.flags & kModeInterp)
      taps = (uint32_t)(16 - (fr >> 1)) | (uint32_t)(32 - (fr >> 1)) << 8 | (uint32_t)(16 + (fr >> 1)) << 16 |
             (uint32_t)(fr >> 1) << 24;
    else
      taps = s_cubic_taps[fr];
    const int j = kMainBase + di + x0;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(S.main) + (j >> 1);
    uint32_t e[6];  // sample pairs (2k, 2k + 1) of the run
    {
      uint32_t c = q[0];
      const uint32_t sh = (j & 1) * 16;
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const uint32_t n = q[k + 1];
        e[k] = __funnelshift_r(c, n, sh);
        c = n;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int k = i >> 1;
      const uint32_t lo = (i & 1) ? __byte_perm(e[k], e[k + 1], 0x5432) : e[k];
      const uint32_t hi = (i & 1) ? __byte_perm(e[k + 1], e[k + 2], 0x5432) : e[k + 1];
      v[i] = __dp2a_hi((int)hi, (int)taps, __dp2a_lo((int)lo, (int)taps, 32)) >> 6;
    }
    // PDPC of the first samples of each line; a zero slope weighs the side's
    // difference to the corner, others to the prediction
    const int lim = (m.flags & kModePdpc) ? min(3 << m.scale, ver ? w : h) : 0;
    if (x0 < lim) {
      const bool zero = m.angle == 0;
      const int corner = S.main[kMainBase], maxv = (1 << bd) - 1;
      int inv = 256 + (x0 + 1) * m.abs_inv;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (x0 + i < lim) {
          const int wl = 32 >> ((2 * (x0 + i)) >> m.scale);
          const int c = zero ? v[i] : clampi(v[i], 0, maxv);
          v[i] = c + ((wl * (S.side[yy + (inv >> 9) + 1] - (zero ? corner : c)) + 32) >> 6);
        }
        inv += m.abs_inv;
      }
    }
  } else if (m.mode == 0) {
    const int16_t* A = S.main + kMainBase + 1;
    const int16_t* L = S.side + 1;
    const int shift = lw + lh + 1, sc = (lw + lh - 2) >> 2;
    const int tr = A[w], bl = L[h], left = L[yy];
    const int wt = 32 >> min(31, (yy * 2) >> sc);
    const int vb = (yy + 1) * bl, vm = h - 1 - yy;
    int hor = ((w - 1 - x0) * left + (x0 + 1) * tr) << lh;
    const int hstep = (tr - left) << lh;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int x = x0 + i, a = A[x];
      const int val = (((vm * a + vb) << lw) + hor + (1 << (shift - 1))) >> shift;
      const int wl = 32 >> min(31, (x * 2) >> sc);
      v[i] = val + ((wl * (left - val) + wt * (a - val) + 32) >> 6);
      hor += hstep;
    }
  } else if (m.mode == 1) {
    const int sc = (lw + lh - 2) >> 2;
    const int wt = 32 >> min(31, (yy * 2) >> sc);
    const int dl = R.l[1 + yy] - dc;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int x = x0 + i;
      const int wl = 32 >> min(31, (x * 2) >> sc);
      v[i] = dc + ((wl * dl + wt * (R.a[1 + x] - dc) + 32) >> 6);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = 0;
  }
  const uint32_t maxv = (1u << bd) - 1, max2 = maxv | maxv << 16;
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; i++)
    o[i] = __vmins2(__vmaxs2(__byte_perm((uint32_t)v[2 * i], (uint32_t)v[2 * i + 1], 0x5410), 0u), max2);
  if (ver) {
    *reinterpret_cast<uint4*>(tile + yy * kTilePitch + x0) = make_uint4(o[0], o[1], o[2], o[3]);
  } else {
    int16_t* t = tile + x0 * kTilePitch + yy;
#pragma unroll
    for (int i = 0; i < 8; i++) t[i * kTilePitch] = (int16_t)(o[i >> 1] >> (16 * (i & 1)));
  }
}

// clip(prediction + residual) of a pair of samples, for predictions of 0..4095
// (what the intra predictors and 8-bit references give): the residual is
// clamped to +-4096 first, which changes no clipped sum of such predictions
// and keeps the packed addition inside 16 bits.
__device__ __forceinline__ uint32_t add_clip2(uint32_t pred, uint32_t res, uint32_t max2) {
  res = __vmaxs2(__vmins2(res, 0x10001000u), 0xF000F000u);
  return __vmins2(__vmaxs2(__vadd2(pred, res), 0u), max2);
}

// ---------------------------------------------------------------------- CCLM --

// The luma samples beside a coding unit that the CCLM templates read besides
// its raw references: the row two above (from one left of the unit) and the
// columns two and three to the left.
struct CclmRefs {
  int16_t row2[36], c2[32], c3[32];
};
constexpr int kCclmExtra = 33 + 32 + 32;

// Offset of extra entry e from the unit's first luma sample, or 0 (no
// entry's offset) where the templates do not read it.
__device__ __forceinline__ int cclm_offset(const RefGeo& G, int cf, bool ctu_top, int e) {
  if (e < 33) return cf != 1 || ctu_top || (!G.hl && e == 0) ? 0 : e - 1 - 2 * G.st;
  if (!G.hl || cf == 3) return 0;
  return ((e - 33) & 31) * G.st - (e < 65 ? 2 : 3);
}

__device__ __forceinline__ void cclm_put(int e, int v, CclmRefs& C) {
  if (e < 33)
    C.row2[e] = (int16_t)v;
  else if (e < 65)
    C.c2[e - 33] = (int16_t)v;
  else
    C.c3[e - 65] = (int16_t)v;
}

struct CclmModel {
  int a, b, shift;
};

// One component's model by one whole warp (every lane returns it): templates
// of downsample_luma_for_cclm_format_16 (predict.rs:3869-3990) at the
// positions predict_cclm_with_format_16 (:3996-4066) takes, and
// derive_cclm_params_from_4_samples (:2088-2177). L: the luma references,
// Cr: the component's own.
__device__ __forceinline__ CclmModel warp_cclm_model(const DevPic& P, int bx, int by, int cw, int ch, int cclm_mode,
                                                     const RawRefs& L, const CclmRefs& X, const RawRefs& Cr) {
  const int lane = threadIdx.x & 31;
  const int bd = P.bd, mid = 1 << (bd - 1);
  const bool has_top = by > 0 && cclm_mode != 1;
  const bool has_left = bx > 0 && cclm_mode != 2;
  const int cnt = has_top || has_left ? 4 : 0;  // blocks are at least 16 wide and high
  // this lane's template sample (lanes 0..3 hold them)
  const int i = lane & 3;
  bool top;
  int k;
  if (has_top && has_left) {
    top = i < 2;
    const int n = top ? cw : ch;
    k = (i & 1) ? (3 * n) / 4 : n / 4;
  } else {
    top = has_top;
    const int n = top ? cw : ch;
    k = min(((2 * i + 1) * n) / 8, n - 1);
  }
  int vl = mid, vc = mid;
  if (cnt) {
    if (top) {
      vc = Cr.a[1 + k];
      if (P.cf == 3) {
        vl = L.a[1 + k];
      } else {
        const int x = 2 * k;
        const int xl = k == 0 && bx == 0 ? 0 : x - 1;  // sample left of x, relative to the unit
        const int r1 = 2 * L.a[1 + x] + L.a[1 + xl] + L.a[2 + x];
        if (P.cf == 2 || (by & (P.ctu - 1)) == 0)
          vl = (r1 + 2) >> 2;
        else
          vl = (2 * X.row2[1 + x] + X.row2[1 + xl] + X.row2[2 + x] + r1 + 4) >> 3;
      }
    } else {
      vc = Cr.l[1 + k];
      if (P.cf == 3) {
        vl = L.l[1 + k];
      } else if (P.cf == 2) {
        vl = (2 * X.c2[k] + X.c3[k] + L.l[1 + k] + 2) >> 2;
      } else {
        const int y = 2 * k;
        vl = (2 * X.c2[y] + X.c3[y] + L.l[1 + y] + 2 * X.c2[y + 1] + X.c3[y + 1] + L.l[2 + y] + 4) >> 3;
      }
    }
  }
  CclmModel M{0, mid, 0};
  if (cnt) {
    int l0 = __shfl_sync(0xffffffffu, vl, 0), l1 = __shfl_sync(0xffffffffu, vl, 1);
    int l2 = __shfl_sync(0xffffffffu, vl, 2), l3 = __shfl_sync(0xffffffffu, vl, 3);
    int c0 = __shfl_sync(0xffffffffu, vc, 0), c1 = __shfl_sync(0xffffffffu, vc, 1);
    int c2 = __shfl_sync(0xffffffffu, vc, 2), c3 = __shfl_sync(0xffffffffu, vc, 3);
    // minimum pair (0, 2), maximum pair (1, 3), ordered by luma
    auto swap = [](int& a, int& b) {
      const int t = a;
      a = b;
      b = t;
    };
    if (l0 > l2) swap(l0, l2), swap(c0, c2);
    if (l1 > l3) swap(l1, l3), swap(c1, c3);
    if (l0 > l3) swap(l0, l1), swap(c0, c1), swap(l2, l3), swap(c2, c3);
    if (l2 > l1) swap(l2, l1), swap(c2, c1);
    const int min_l = (l0 + l2 + 1) >> 1, min_c = (c0 + c2 + 1) >> 1;
    const int max_l = (l1 + l3 + 1) >> 1, max_c = (c1 + c3 + 1) >> 1;
    const int diff = max_l - min_l;
    M.b = min_c;
    if (diff > 0) {
      const int diff_c = max_c - min_c;
      int xx = floor_log2((unsigned)diff);
      const int norm = ((diff << 4) >> xx) & 15;
      const int vv = (int)c_cclm_div_sig[norm] | 8;
      if (norm != 0) xx += 1;
      const int yy = diff_c == 0 ? 1 : floor_log2((unsigned)abs(diff_c)) + 1;
      const int add = (1 << yy) >> 1;
      M.a = (diff_c * vv + add) >> yy;
      M.shift = 3 + xx - yy;
      if (M.shift < 1) {
        M.shift = 1;
        M.a = M.a == 0 ? 0 : (M.a < 0 ? -15 : 15);
      }
      M.b = min_c - ((M.a * min_l) >> M.shift);
    }
  }
  return M;
}

// Predicts run r (eight samples of a row) of a chroma block of width 1 << lw from the unit's reconstructed luma
// (`luma`, a tile, and the column left of it in L.l) into the block's
// tile, with the downsampling of downsample_luma_for_cclm_format_16.
__device__ __forceinline__ void cclm_run(int r, int cf, int bd, int bx, int lw, const CclmModel& M,
                                         const int16_t* luma, const RawRefs& L, int16_t* tile) {
  const int maxv = (1 << bd) - 1;
  const int x0 = 8 * (r & ((1 << (lw - 3)) - 1)), y = r >> (lw - 3);
  int v[8];
  if (cf == 3) {
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = luma[y * kTilePitch + x0 + i];
  } else {
    const int rows = cf == 1 ? 2 : 1;
    const int ly = y * rows;
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = cf == 1 ? 4 : 2;
#pragma unroll 1
    for (int t = 0; t < rows; t++) {
      const int16_t* row = luma + (ly + t) * kTilePitch + 2 * x0;
      int prev = x0 > 0 ? row[-1] : (bx > 0 ? L.l[1 + ly + t] : row[0]);
      const uint4 w0 = *reinterpret_cast<const uint4*>(row), w1 = *reinterpret_cast<const uint4*>(row + 8);
      const uint32_t q[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int i = 0; i < 8; i++) {
        v[i] += prev + 2 * (int)(q[i] & 0xFFFFu) + (int)(q[i] >> 16);
        prev = (int)(q[i] >> 16);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] >>= rows + 1;
  }
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int p0 = clampi(((v[2 * i] * M.a) >> M.shift) + M.b, 0, maxv);
    const int p1 = clampi(((v[2 * i + 1] * M.a) >> M.shift) + M.b, 0, maxv);
    o[i] = (uint32_t)p0 | (uint32_t)p1 << 16;
  }
  *reinterpret_cast<uint4*>(tile + y * kTilePitch + x0) = make_uint4(o[0], o[1], o[2], o[3]);
}

}  // namespace vvcg
