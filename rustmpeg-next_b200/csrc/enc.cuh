// The frame-path encoder of libvvcg (sm_100a): slice::encode_vvc_frame_picture
// (crates/rustmpeg-video/src/vvc/slice.rs:4171-4634) without its CABAC writes.
// A CTA walks a CTU row in the same wavefront as the reconstruction. Each
// coding unit: the 7-mode luma SAD decision (two warps a candidate), forward
// DCT-2, regular or dependent quantisation and the encoder's own
// reconstruction by all 16 warps, then the chroma mode decision (DM or CCLM by
// SAD, a warp a candidate) and the same chain for Cb and Cr, eight warps each.
// The reconstruction feeds the next units' predictions, exactly as the
// reference's sequential CTU loop does.
//
// What bounds it is the serial chain of a picture's units (see k_recon_rows):
// one warp per row took 184 us a unit, this takes 14 us (four 1920x1088 10-bit
// 4:2:0 pictures: 23.1 -> 1.77 ms).
#pragma once
#include "recon.cuh"
#include "tu.cuh"

namespace vvcg {

constexpr int kEncMain = 512;                // 16 warps of samples
constexpr int kEncThreads = kEncMain + 64;   // and the pilot and the publisher
constexpr int kEncCands = 7;

// Tiles of the workspace: the luma candidates' predictions (the winner's
// becomes the reconstructed luma), the transforms' work tiles (Cb and luma
// share the first two), which hold the chroma candidates' predictions before
// that, the chroma predictions, and the source.
enum { kTileCand = 0, kTileWork = 7, kTilePredC = 11, kTileSrc = 13, kEncTiles = 16 };

struct EncUnit {
  int16_t gx, gy;
  uint8_t ar, bl;
};

struct __align__(16) EncWs {
  int16_t tile[kEncTiles][32 * kTilePitch];
  int16_t lv[3][1024];            // levels, raster
  int32_t wide[2][1024 + kTuPad]; // tiles of wide_forward
  uint32_t mat[4][256];           // DCT-2 matrices of int8: 16-point rows, columns, 32-point rows, columns
  DevPic P;
  RawRefs raw[3], plain[2];       // references (coded-unit rules); the mode decisions' where they differ
  ModeRefs refs[kEncCands];       // a candidate's arrays, then the final predictions'
  CclmRefs cclm;
  ModeInfo cand[kEncCands], cand_c[kEncCands];
  EncUnit unit[4];
  uint32_t sad[2 * kEncCands];
  uint32_t sad_c[4];
  uint32_t cbf[3];
  uint32_t maps[3][16];           // dependent quantisation: each warp's state transitions
  uint32_t item;
};

// Luma candidates of choose_intra_mode_16 (predict.rs:4069-4105), in order:
// a later candidate wins only with a strictly lower SAD.
__device__ __forceinline__ int enc_candidate(int c) {
  return c == 0 ? 0 : c == 1 ? 1 : c == 2 ? 18 : c == 3 ? 50 : c == 4 ? 2 : c == 5 ? 34 : 66;
}

// Named barrier of a part of the CTA, ids 7.. (constants, see Grp).
template <int kId>
__device__ __forceinline__ void enc_sync(int n) {
  asm volatile("bar.sync %0, %1;" ::"n"(kId), "r"(n) : "memory");
}
__device__ __forceinline__ void pair_sync(int cand) {  // the two warps of a luma candidate
  switch (cand) {
    case 0: enc_sync<7>(64); break;
    case 1: enc_sync<8>(64); break;
    case 2: enc_sync<9>(64); break;
    case 3: enc_sync<10>(64); break;
    case 4: enc_sync<11>(64); break;
    case 5: enc_sync<12>(64); break;
    default: enc_sync<13>(64); break;
  }
}

// Barrier 1 of the 16 sample warps; whether any thread's flag is set.
__device__ __forceinline__ bool any_main(bool flag) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred p, 1, %2, q;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)flag), "n"(kEncMain)
      : "memory");
  return r != 0;
}

// Sum of absolute differences of one run (eight samples) of two tiles.
__device__ __forceinline__ uint32_t run_sad(const int16_t* a, const int16_t* b) {
  const uint4 x = *reinterpret_cast<const uint4*>(a), y = *reinterpret_cast<const uint4*>(b);
  const uint32_t p[4] = {x.x, x.y, x.z, x.w}, q[4] = {y.x, y.y, y.z, y.w};
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t d = __vsub2(__vmaxu2(p[k], q[k]), __vminu2(p[k], q[k]));
    s += (d & 0xFFFFu) + (d >> 16);
  }
  return s;
}

// One pass of a transform by a group: out = clip16((sum_i M[o][i] in[l][i] +
// add) >> sh) for N outputs o of L lines l, pairs of i multiplied by dp2a.
// kTrans stores out[o][l], else out[l][o]. The frame path's sums fit 32 bits
// and the forward first stage's outputs (which the reference leaves
// unclipped, dct.rs:963) fit 16: a row of the DCT-2 matrix has at most
// 64 N in absolute sum, so |out| <= 2^bd 64 N >> (log2 N + bd - 9) <= 2^15.
template <int N, bool kTrans>
__device__ __forceinline__ void xform_pass(const Grp& g, const uint32_t* M, int L, const int16_t* in, int16_t* out,
                                           int add, int sh) {
  const int o = g.tid & (N - 1);
  const int lpt = (N * L) / g.n, l0 = (g.tid / N) * lpt;
  uint32_t m[N / 4];
#pragma unroll
  for (int k = 0; k < N / 4; k += 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(M + o * (N / 4) + k);
    m[k] = v.x;
    m[k + 1] = v.y;
    m[k + 2] = v.z;
    m[k + 3] = v.w;
  }
  for (int l = l0; l < l0 + lpt; l++) {
    const uint4* r = reinterpret_cast<const uint4*>(in + l * kTilePitch);
    int s = add;
#pragma unroll
    for (int k = 0; k < N / 8; k++) {
      const uint4 v = r[k];
      s = __dp2a_lo((int)v.x, (int)m[2 * k], s);
      s = __dp2a_hi((int)v.y, (int)m[2 * k], s);
      s = __dp2a_lo((int)v.z, (int)m[2 * k + 1], s);
      s = __dp2a_hi((int)v.w, (int)m[2 * k + 1], s);
    }
    out[kTrans ? o * kTilePitch + l : l * kTilePitch + o] = (int16_t)clip16i(s >> sh);
  }
}

template <bool kTrans>
__device__ __forceinline__ void xform(const Grp& g, const uint32_t (*mat)[256], bool inverse, int N, int L,
                                      const int16_t* in, int16_t* out, int add, int sh) {
  if (N == 32)
    xform_pass<32, kTrans>(g, mat[inverse ? 3 : 2], L, in, out, add, sh);
  else
    xform_pass<16, kTrans>(g, mat[inverse ? 1 : 0], L, in, out, add, sh);
}

// The forward transform of a unit whose source leaves the bit depth, by one
// warp in 32-bit tiles (tu.cuh): transposed coefficients into X.
__device__ __noinline__ void wide_forward(const int16_t* src, const int16_t* pred, int w, int h, int bd, int32_t* A,
                                          int32_t* B, int16_t* X) {
  const int lane = threadIdx.x & 31;
  TuShape S;
  S.w = w;
  S.h = h;
  S.lw = ilog2(w);
  S.lh = ilog2(h);
  S.n = w * h;
  S.th = S.tv = S.sw = S.sh = 0;
  for (int i = lane; i < S.n; i += 32) {
    const int y = i >> S.lw, x = i & (w - 1), o = y * kTilePitch + x;
    A[y * (w + 1) + x] = (int)(uint16_t)src[o] - (int)(uint16_t)pred[o];
  }
  __syncwarp();
  tu_forward_transform(A, B, S, bd, lane);
  for (int i = lane; i < S.n; i += 32) X[(i & (w - 1)) * kTilePitch + (i >> S.lw)] = (int16_t)A[i];
  __syncwarp();
}

// Forward transform, quantisation and the encoder's own reconstruction of one
// TB by a group (slice.rs:4298-4346 for luma, :4442-4553 for chroma): DCT-2
// both ways, no zero-out at these sizes, intra rounding offset. Writes the
// levels to lv_out when any is nonzero and the reconstruction to the plane at
// `at` and into the prediction's tile. X, Y: work tiles; with `wide` X holds
// the coefficients already. Returns the cbf.
//
// Dependent quantisation (dct.rs:1252-1301, :1191-1248) is a four-state
// machine over the scan from its end. A position's level depends on the state
// only through one bit, so its effect is a map of the four states; every
// thread composes the maps of its positions, a scan over the group gives each
// its entry state, and because leading zero levels keep the state at 0, these
// are also the states of the dequantisation, which is done in the same pass.
__device__ __forceinline__ bool code_tb(const Grp& g, EncWs& W, int comp, int w, int h, int qp, int bd, bool dq,
                                        const int16_t* src, int16_t* pred, int16_t* X, int16_t* Y, int16_t* lv_out,
                                        uint16_t* at, int st, bool wide) {
  const int lane = g.tid & 31, wid = g.tid >> 5, lw = ilog2(w), lh = ilog2(h), n = w * h;
  if (g.tid == 0) W.cbf[comp] = 0;
  if (!wide) {
    for (int r = g.tid; r < n >> 3; r += g.n) {  // residual
      const int o = (r >> (lw - 3)) * kTilePitch + 8 * (r & ((w >> 3) - 1));
      const uint4 a = *reinterpret_cast<const uint4*>(src + o), b = *reinterpret_cast<const uint4*>(pred + o);
      *reinterpret_cast<uint4*>(X + o) =
          make_uint4(__vsub2(a.x, b.x), __vsub2(a.y, b.y), __vsub2(a.z, b.z), __vsub2(a.w, b.w));
    }
    g.sync();
    const int sh1 = lw + bd + 6 - 15;
    xform<true>(g, W.mat, false, w, h, X, Y, sh1 > 0 ? 1 << (sh1 - 1) : 0, sh1);
    g.sync();
    // coefficients transposed: X[column][row]
    xform<false>(g, W.mat, false, h, w, Y, X, 1 << (lh + 5), lh + 6);
  }
  g.sync();
  bool s2;
  const int tr_shift = tu_tr_shift(lw, lh, bd, &s2);
  int16_t* lv = W.lv[comp];
  bool nz = false;
  if (dq) {
    const int16_t* scan = tu_scan(lw, lh);
    const int qp_dq = max(4, qp) + 1;
    const int q_shift = 13 + qp_dq / 6 + tr_shift;
    const long long q_scale = c_quant_scale[s2 ? 1 : 0][qp_dq % 6];
    const long long half = 1ll << max(0, q_shift - 1);
    auto level_of = [&](int c, int off) -> int {  // off: the state's high bit
      const long long est = ((long long)abs(c) * q_scale + half) >> max(0, q_shift);
      const int a = est <= off ? 0 : (int)((est + off + 1) >> 1);
      return clampi(c < 0 ? -a : a, -32768, 32767);
    };
    const int per = n / g.n;  // 1, 2 or 4 positions a thread
    const int s_hi = n - 1 - g.tid * per;
    // map: entry state s -> field s; 0xD8 swaps a state's bits, an odd level
    // also flips the high bit
    uint32_t map = 0xE4u;
    auto compose = [](uint32_t f, uint32_t then) -> uint32_t {
      uint32_t r = 0;
#pragma unroll
      for (int s = 0; s < 4; s++) r |= ((then >> (2 * ((f >> (2 * s)) & 3))) & 3) << (2 * s);
      return r;
    };
    for (int k = 0; k < per; k++) {
      const int r = scan[s_hi - k];
      const int c = X[(r & (w - 1)) * kTilePitch + (r >> lw)];
      const uint32_t step = 0xD8u ^ ((level_of(c, 0) & 1) ? 0x0Au : 0u) ^ ((level_of(c, 1) & 1) ? 0xA0u : 0u);
      map = compose(map, step);
    }
    uint32_t pre = map;  // inclusive over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t other = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre = compose(other, pre);
    }
    if (lane == 31) W.maps[comp][wid] = pre;
    uint32_t excl = __shfl_up_sync(0xffffffffu, pre, 1);
    if (lane == 0) excl = 0xE4u;
    g.sync();
    int state = 0;
    for (int k = 0; k < wid; k++) state = (int)((W.maps[comp][k] >> (2 * state)) & 3);
    state = (int)((excl >> (2 * state)) & 3);
    const int shift = 7 - qp_dq / 6 - tr_shift;
    long long inv_q = c_inv_quant_scale[s2 ? 1 : 0][qp_dq % 6];
    if (shift < 0) inv_q <<= -shift;
    const long long add = shift > 0 ? (1ll << (shift - 1)) : 0;
    const int rsh = max(0, shift);
    for (int k = 0; k < per; k++) {
      const int r = scan[s_hi - k];
      int16_t* p = &X[(r & (w - 1)) * kTilePitch + (r >> lw)];
      const int L = level_of(*p, state >> 1);
      lv[r] = (int16_t)L;
      int v = 0;
      if (L != 0) {
        nz = true;
        v = clip16(((long long)(2 * L + (L > 0 ? -(state >> 1) : (state >> 1))) * inv_q + add) >> rsh);
      }
      *p = (int16_t)v;
      state = (((state & 1) << 1) | (state >> 1)) ^ ((L & 1) << 1);
    }
  } else {
    // quantize_rect_bd (dct.rs:1113-1147, intra offset), dequantize_rect_bd (:1151-1187)
    const int q = max(4, qp);
    const int qbits = max(0, 14 + q / 6 + tr_shift);
    const long long qadd = 171ll << max(0, 14 + q / 6 + tr_shift - 9);
    const long long scale = c_quant_scale[s2 ? 1 : 0][q % 6];
    const int rs = 6 - (tr_shift + q / 6);
    const long long inv = c_inv_quant_scale[s2 ? 1 : 0][q % 6];
    for (int r = g.tid; r < n; r += g.n) {
      int16_t* p = &X[(r & (w - 1)) * kTilePitch + (r >> lw)];
      const int c = *p;
      const long long a = ((long long)abs(c) * scale + qadd) >> qbits;
      const int L = clip16(c < 0 ? -a : a);
      nz |= L != 0;
      lv[r] = (int16_t)L;
      const long long v = (long long)L * inv;
      *p = (int16_t)clip16(rs > 0 ? (v + (1ll << (rs - 1))) >> rs : v << (-rs));
    }
  }
  if (__any_sync(0xffffffffu, nz) && lane == 0) atomicOr(&W.cbf[comp], 1u);
  g.sync();
  const bool cbf = W.cbf[comp] != 0;
  if (cbf) {
    for (int r = g.tid; r < n >> 3; r += g.n)
      *reinterpret_cast<uint4*>(lv_out + 8 * r) = *reinterpret_cast<const uint4*>(lv + 8 * r);
    xform<true>(g, W.mat, true, h, w, X, Y, 64, 7);
    g.sync();
    xform<false>(g, W.mat, true, w, h, Y, X, 1 << (19 - bd), 20 - bd);
    g.sync();
  }
  const uint32_t max2 = ((1u << bd) - 1) * 0x10001u;
  for (int r = g.tid; r < n >> 3; r += g.n) {
    const int o = (r >> (lw - 3)) * kTilePitch + 8 * (r & ((w >> 3) - 1));
    const uint4 res = cbf ? *reinterpret_cast<const uint4*>(X + o) : make_uint4(0, 0, 0, 0);
    store_run(at, st, lw, max2, r, res, pred, true);
  }
  return cbf;
}

// Gathers a block's references by threads tid of n.
__device__ __forceinline__ void enc_gather(int tid, int n, const RefGeo& G, RawRefs& R) {
  const int nref = 2 * (G.w + G.h) + 1;
  int v[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int e = tid + k * n;
    v[k] = e < nref && (G.ha || G.hl) ? ldp(G.at + ref_offset(G, e)) : G.def;
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int e = tid + k * n;
    if (e < nref) ref_put(G.w, G.h, e, v[k], R);
  }
}

// Encoder wavefront over the batch's CTU rows.
__global__ void __launch_bounds__(kEncThreads, 2)
k_encode_rows(const DevPic* __restrict__ pics, const RowItem* __restrict__ rows, uint32_t n_rows,
              uint32_t* counter, uint32_t epoch, uint32_t spin_limit, uint32_t* status) {
  extern __shared__ __align__(16) unsigned char enc_smem[];
  EncWs& W = *reinterpret_cast<EncWs*>(enc_smem);
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  load_cubic_taps();
  for (int i = t; i < 1024; i += kEncThreads) {
    int8_t* m = reinterpret_cast<int8_t*>(W.mat);
    m[2048 + i] = g_dct2_m[4][i];
    m[3072 + (i & 31) * 32 + (i >> 5)] = g_dct2_m[4][i];
    if (i < 256) {
      m[i] = g_dct2_m[3][i];
      m[1024 + (i & 15) * 16 + (i >> 4)] = g_dct2_m[3][i];
    }
  }
  for (;;) {
    __syncthreads();
    if (t == 0) W.item = atomicAdd(counter, 1u);
    __syncthreads();
    if (W.item >= n_rows) break;
    const RowItem item = rows[W.item];
    for (int i = t; i < (int)(sizeof(DevPic) / 4); i += kEncThreads)
      reinterpret_cast<uint32_t*>(&W.P)[i] = reinterpret_cast<const uint32_t*>(&pics[item.pic])[i];
    __syncthreads();
    const DevPic& P = W.P;
    if (t < 2 * kEncCands) {
      const int c = t >> 1, mode = enc_candidate(c);
      if (t & 1)
        W.cand_c[c] = mode_info(mode, max(P.tb_cw, 2), max(P.tb_ch, 2), false);
      else
        W.cand[c] = mode_info(mode, 32, 32, true);
    }
    __syncthreads();
    const int cy = (int)item.cy;
    const int sh = P.ctu_log2 - 5;
    const int ncu = 1 << (2 * sh);
    const int steps = P.ctu_w << (2 * sh);
    if (wid == kEncMain / 32 + 1) {
      // ---- publisher
      uint64_t* mine = P.row_done + (size_t)cy * kRowFlagStride;
      for (int s = 0; s < steps; s++) {
        part_sync<5>(kEncMain + 32);
        if (lane == 0 && (s & (ncu - 1)) == ncu - 1) {
          __threadfence();
          st_release64(mine, ((uint64_t)epoch << 32) | (uint32_t)((s >> (2 * sh)) + 1));
        }
        __syncwarp();
      }
    } else if (wid == kEncMain / 32) {
      // ---- pilot: positions a step ahead, and the wait
      const uint64_t* above = cy > 0 ? P.row_done + (size_t)(cy - 1) * kRowFlagStride : nullptr;
      uint32_t have = 0;
      for (int s = -1; s < steps; s++) {
        if (lane == 0) {
          if (s + 1 < steps) {
            int gx, gy;
            bool ar, bl;
            row_step(s + 1, sh, cy, gx, gy);
            unit_edges(P, gx, gy, sh, ar, bl);
            W.unit[(s + 1) & 3] = EncUnit{(int16_t)gx, (int16_t)gy, ar, bl};
          }
          if (s >= 0 && above && (s & (ncu - 1)) == 0)
            pilot_wait(above, epoch, min((s >> (2 * sh)) + 2, P.ctu_w), P.ctu_w, spin_limit, status, have);
        }
        __syncwarp();
        part_sync<4>(kEncMain + 32);
      }
    } else {
      // ---- the unit's samples
      const int cf = P.cf, bd = P.bd, cw = P.tb_cw, ch = P.tb_ch, lcw = ilog2(max(cw, 8));
      const int def = 1 << (bd - 1);
      const bool dq = (P.tools & VVCG_TOOL_DEP_QUANT) != 0;
      const bool use_cclm = cf && (P.tools & VVCG_TOOL_ENC_CCLM);
      const int n_lv = 1024 + 2 * cw * ch;
      const Grp all{t, kEncMain, 1};
      const Grp half{t & 255, 256, 2 + (t >> 8)};  // Cb: warps 0..7, Cr: 8..15
      // source: one run of eight samples a thread, luma first
      const int nrc = (cw * ch) >> 3;
      const int sc = t < 128 ? 0 : (t < 128 + nrc ? 1 : (t < 128 + 2 * nrc ? 2 : 3));
      const int sr = t - (sc == 0 ? 0 : (sc == 1 ? 128 : 128 + nrc));
      const int slw = sc ? lcw : 5, sx = 8 * (sr & ((1 << (slw - 3)) - 1)), sy = sr >> (slw - 3);
      auto load_src = [&](const EncUnit& U) -> uint4 {
        if (sc == 3) return make_uint4(0, 0, 0, 0);
        const int uw = sc ? cw : 32, uh = sc ? ch : 32;
        return __ldcs(reinterpret_cast<const uint4*>(P.scratch[sc] + (size_t)(U.gy * uh + sy) * P.stride[sc] +
                                                     U.gx * uw + sx));
      };
      part_sync<4>(kEncMain + 32);
      uint4 src = load_src(W.unit[0]);
      for (int s = 0; s < steps; s++) {
        const EncUnit U = W.unit[s & 3];
        const int gx = U.gx, gy = U.gy;
        const int k = gy * P.grid_w + gx;
        // the mode decisions' references: no coded-unit substitution
        // (predict_block_16), equal to the others in CTUs of one unit
        const bool plain_ar = gy > 0 && gx + 1 < P.grid_w;
        const bool same = (U.ar != 0) == plain_ar && !U.bl;
        uint16_t* at[3];
#pragma unroll
        for (int c = 0; c < 3; c++)
          at[c] = P.plane[c] + (size_t)(gy * (c ? ch : 32)) * P.stride[c] + gx * (c ? cw : 32);
        if (sc < 3) *reinterpret_cast<uint4*>(W.tile[kTileSrc + sc] + sy * kTilePitch + sx) = src;
        const uint32_t top2 = __vmaxu2(__vmaxu2(src.x, src.y), __vmaxu2(src.z, src.w));
        const bool high = max(top2 & 0xFFFFu, top2 >> 16) > (1u << bd) - 1;
        part_sync<4>(kEncMain + 32);
        if (s + 1 < steps) src = load_src(W.unit[(s + 1) & 3]);
        // references: luma (and the CCLM templates' samples) by warps 0..7, Cb 8..11, Cr 12..15
        {
          const bool ha = gy > 0, hl = gx > 0;
          const RefGeo GY{at[0], P.stride[0], 32, 32, def, ha, hl, U.ar != 0, U.bl != 0};
          if (wid < 8) {
            int o = 0;
            const int e = t - 129;
            if (t >= 129 && e < kCclmExtra && use_cclm) o = cclm_offset(GY, cf, (gy & ((1 << sh) - 1)) == 0, e);
            const int v = o ? ldp(at[0] + o) : 0;
            enc_gather(t, 256, GY, W.raw[0]);
            if (t >= 129 && e < kCclmExtra) cclm_put(e, v, W.cclm);
            if (!same) {
              RefGeo GP = GY;
              GP.ar = plain_ar;
              GP.bl = false;
              enc_gather(t, 256, GP, W.plain[0]);
            }
          } else if (cf) {
            const int c = wid < 12 ? 1 : 2;
            RefGeo G{at[c], P.stride[c], cw, ch, def, ha, hl, U.ar != 0, U.bl != 0};
            enc_gather(t & 127, 128, G, W.raw[c]);
            if (c == 1 && !same) {
              G.ar = plain_ar;
              G.bl = false;
              enc_gather(t & 127, 128, G, W.plain[1]);
            }
          }
        }
        // source samples above the bit depth (which nothing rejects) do not fit
        // the packed transforms: such units take the 32-bit forward transform
        const bool wide = any_main(high);
        // slice.rs:4264-4274: luma mode by SAD of the plain prediction against the source
        const RawRefs& RL = same ? W.raw[0] : W.plain[0];
        if (wid < 2 * kEncCands) {
          const int c = wid >> 1, pt = t & 63;
          const ModeInfo m = W.cand[c];
          int16_t* tile = W.tile[kTileCand + c];
          group_prep(pt, 64, m, 32, 32, RL, W.refs[c]);
          pair_sync(c);
          const int dc = m.mode == 1 ? warp_dc(RL, 32, 32, (1 << bd) - 1) : 0;
#pragma unroll 1
          for (int r = pt; r < 128; r += 64) predict_run(r, m, 32, 32, bd, dc, RL, W.refs[c], tile);
          pair_sync(c);
          uint32_t sad = 0;
#pragma unroll
          for (int r = pt; r < 128; r += 64) {
            const int o = (r >> 2) * kTilePitch + 8 * (r & 3);
            sad += run_sad(W.tile[kTileSrc] + o, tile + o);
          }
          sad = __reduce_add_sync(0xffffffffu, sad);
          if (lane == 0) W.sad[wid] = sad;
        }
        all.sync();
        int best = 0;
        {
          uint32_t best_sad = 0xffffffffu;
#pragma unroll
          for (int c = 0; c < kEncCands; c++) {
            const uint32_t v = W.sad[2 * c] + W.sad[2 * c + 1];
            if (v < best_sad) {
              best_sad = v;
              best = c;
            }
          }
          if (!(P.tools & VVCG_TOOL_ENC_FULL_INTRA) && best > 1) best = 0;
        }
        int16_t* luma = W.tile[kTileCand + best];
        if (!same) {  // the chosen mode from the coded units' references
          const ModeInfo m = W.cand[best];
          all.sync();  // every thread has read the SADs; the arrays are free
          group_prep(t, kEncMain, m, 32, 32, W.raw[0], W.refs[best]);
          all.sync();
          const int dc = m.mode == 1 ? warp_dc(W.raw[0], 32, 32, (1 << bd) - 1) : 0;
          if (t < 128) predict_run(t, m, 32, 32, bd, dc, W.raw[0], W.refs[best], luma);
          all.sync();
        }
        const int32_t off0 = P.lv_base + k * n_lv;
        int16_t* lv = P.lv_pool + off0;
        if (wide) {
          all.sync();
          if (wid == 0)
            wide_forward(W.tile[kTileSrc], luma, 32, 32, bd, W.wide[0], W.wide[1], W.tile[kTileWork]);
        }
        const bool cbf_y = code_tb(all, W, 0, 32, 32, P.lqp, bd, dq, W.tile[kTileSrc], luma, W.tile[kTileWork],
                                   W.tile[kTileWork + 1], lv, at[0], P.stride[0], wide);
        int chroma_mode = enc_candidate(best);
        if (cf) {
          all.sync();  // the reconstructed luma is complete, the work tiles are free
          if (use_cclm) {
            // slice.rs:4362-4397: DM (plain prediction) against LM / LM-L / LM-T on Cb, a warp each
            if (wid < 4) {
              int16_t* tile = W.tile[kTileWork + wid];
              if (wid == 0) {
                const RawRefs& RC = same ? W.raw[1] : W.plain[1];
                const ModeInfo m = W.cand_c[best];
                group_prep(lane, 32, m, cw, ch, RC, W.refs[0]);
                __syncwarp();
                const int dc = m.mode == 1 ? warp_dc(RC, cw, ch, (1 << bd) - 1) : 0;
                for (int r = lane; r < nrc; r += 32) predict_run(r, m, cw, ch, bd, dc, RC, W.refs[0], tile);
              } else {
                const CclmModel M = warp_cclm_model(P, gx * 32, gy * 32, cw, ch, wid - 1, W.raw[0], W.cclm, W.raw[1]);
                for (int r = lane; r < nrc; r += 32) cclm_run(r, cf, bd, gx, lcw, M, luma, W.raw[0], tile);
              }
              __syncwarp();
              uint32_t sad = 0;
              for (int r = lane; r < nrc; r += 32) {
                const int o = (r >> (lcw - 3)) * kTilePitch + 8 * (r & ((cw >> 3) - 1));
                sad += run_sad(W.tile[kTileSrc + 1] + o, tile + o);
              }
              sad = __reduce_add_sync(0xffffffffu, sad);
              if (lane == 0) W.sad_c[wid] = sad;
            }
            all.sync();
            uint32_t bsad = W.sad_c[0];
#pragma unroll
            for (int m = 0; m < 3; m++)
              if (W.sad_c[1 + m] < bsad) {
                bsad = W.sad_c[1 + m];
                chroma_mode = 81 + m;
              }
          }
          const int c = 1 + (t >> 8);
          int16_t* pred = W.tile[kTilePredC + c - 1];
          if (chroma_mode >= 81) {
            const CclmModel M =
                warp_cclm_model(P, gx * 32, gy * 32, cw, ch, chroma_mode - 81, W.raw[0], W.cclm, W.raw[c]);
            for (int r = half.tid; r < nrc; r += half.n) cclm_run(r, cf, bd, gx, lcw, M, luma, W.raw[0], pred);
          } else {
            const ModeInfo m = W.cand_c[best];
            group_prep(half.tid, half.n, m, cw, ch, W.raw[c], W.refs[c]);
            half.sync();
            const int dc = m.mode == 1 ? warp_dc(W.raw[c], cw, ch, (1 << bd) - 1) : 0;
            for (int r = half.tid; r < nrc; r += half.n)
              predict_run(r, m, cw, ch, bd, dc, W.raw[c], W.refs[c], pred);
          }
          half.sync();
          int16_t* X = W.tile[kTileWork + 2 * (c - 1)];
          if (wide) {
            all.sync();
            if (wid == 0)
              for (int q = 0; q < 2; q++)
                wide_forward(W.tile[kTileSrc + 1 + q], W.tile[kTilePredC + q], cw, ch, bd, W.wide[0], W.wide[1],
                             W.tile[kTileWork + 2 * q]);
            all.sync();
          }
          code_tb(half, W, c, cw, ch, P.cqp, bd, dq, W.tile[kTileSrc + c], pred, X,
                          W.tile[kTileWork + 2 * (c - 1) + 1], lv + 1024 + (c - 1) * cw * ch, at[c], P.stride[c], wide);
        }
        part_sync<5>(kEncMain + 32);
        if (t == 0) {  // the next unit's chroma clears the flags only after its luma
          const bool cb = cf && W.cbf[1], cr = cf && W.cbf[2];
          vvcg_cu_rec r;
          r.luma_mode = (uint8_t)enc_candidate(best);
          r.chroma_mode = (uint8_t)chroma_mode;
          r.cbf = (uint8_t)((cbf_y ? 1 : 0) | (cb ? 2 : 0) | (cr ? 4 : 0));
          r.tu_tools = 0;
          r.level_off[0] = cbf_y ? off0 : -1;
          r.level_off[1] = cb ? off0 + 1024 : -1;
          r.level_off[2] = cr ? off0 + 1024 + cw * ch : -1;
          const_cast<vvcg_cu_rec*>(P.cus)[k] = r;
        }
      }
    }
  }
}

}  // namespace vvcg
