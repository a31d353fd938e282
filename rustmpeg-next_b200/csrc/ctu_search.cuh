// CTU full search of the GPU encoder: every block of the six split types of a
// 32x32 CTU, each over the 67 luma modes (or a candidate list), on 8..12-bit
// samples, open loop from the source, with the predictors of predict_block_16
// (crates/rustmpeg-video/src/vvc/predict.rs:3079-3410): cost = 8x8 Hadamard SATD
// + lambda * mode bits, the first candidate with the lowest cost wins.
//
// One CTA per CTU and split type: all six cover the CTU's 16 tiles of 8x8
// once, so each has 16 tiles x 67 modes to predict and transform. A lane takes
// one (tile, angular mode) and keeps the tile's 64 residuals in 32 registers:
// a line of eight predictions is 16 dp2a on packed sample pairs; a horizontal
// mode is evaluated on the transposed source (the Hadamard sum does not change),
// so lanes differ in data only. Two residuals share a word as sum + difference
// * 2^16, which is the transform's first stage; the words then add and
// subtract as plain 32-bit numbers, and the last stage is left out
// (|a + b| + |a - b| = 2 max(|a|, |b|)), which keeps 10-bit samples inside 16
// bits. Nothing but the references passes through shared memory.
// Planar and DC, bit depths above 10 and sources above their bit depth take a
// lane per line with 32-bit arithmetic.
//
// 1,980 CTUs at 10 bits take 1.07 ms, bound by instruction issue (0.6 a cycle and
// scheduler, 62,000 warp instructions a CTA). With a warp per candidate, one
// prediction at a time into shared memory and a 16-bit Hadamard from there they
// took 3.41 ms; with the tile's eight lines unrolled and tasks tile by tile
// instead of mode by mode 1.81 ms (instruction-cache misses).
#pragma once
#include "vvcg_device.cuh"
#include "vvcg_tables_dev.cuh"

namespace vvcg {

constexpr int kCtsWarps = 7;  // 33 warps of angular tasks and 8 of planar / DC in six rounds
constexpr int kCtsModes = 67;
constexpr int kCtsRef = 72;   // a reference row: corner, 2n samples, two repeats, padding

// Bits a block is charged in the search cost: a header of 8 bits (split
// flags, cbf and the like) plus its mode, ordered by the default MPM list
// (derive_intra_mpms with no neighbours, predict.rs): MPM i costs 2 + i bits,
// any other mode 7.
__device__ __forceinline__ int search_mode_bits(int m) {
  return 8 + (m == 0 ? 2 : m == 1 ? 3 : m == 50 ? 4 : m == 18 ? 5 : m == 46 ? 6 : 7);
}

// Blocks of a 32x32 CTU by slot (x, y, log2 w, log2 h), the slots of each split
// type (none, quad, binary and ternary, horizontal then vertical) and its bits.
__constant__ uint8_t c_search_blocks[15][4] = {
    {0, 0, 5, 5},  {0, 0, 4, 4},  {16, 0, 4, 4}, {0, 16, 4, 4}, {16, 16, 4, 4}, {0, 0, 5, 4},  {0, 16, 5, 4}, {0, 0, 4, 5},
    {16, 0, 4, 5}, {0, 0, 5, 3},  {0, 8, 5, 4},  {0, 24, 5, 3}, {0, 0, 3, 5},   {8, 0, 4, 5},  {24, 0, 3, 5}};
__constant__ uint8_t c_split_first[6] = {0, 1, 5, 7, 9, 12};
__constant__ uint8_t c_split_count[6] = {1, 4, 2, 2, 3, 3};
__constant__ uint8_t c_split_bits[6] = {1, 2, 3, 3, 4, 4};


struct CtsArgs {
  const uint16_t* src;
  int64_t stride;
  int32_t width, height, bd;
  uint32_t lambda_q8;
  const vvcg_ctu_search_req* reqs;
  uint32_t* block_cost;  // [ctu][15]
  uint8_t* block_mode;   // [ctu][15]
  uint32_t* mode_costs;  // optional [ctu][67]: every mode's cost of the unsplit CU (full set)
};

// One candidate of one block: init_angular_params (predict.rs:1608-1685) and
// where its reference arrays lie (int16 indexes of sample k = 0).
struct __align__(16) CtsMode {
  int16_t angle, inv;
  uint16_t main, side;
  uint8_t tab;    // taps: 0 Gaussian, 1 cubic, 2 whole samples
  int8_t scale;   // PDPC scale
  uint8_t lim;    // PDPC: samples of a line it changes
  uint8_t flags;  // kCts*
  int32_t mode;
};
enum : uint8_t { kCtsVer = 1, kCtsZero = 2 };

struct CtsWs {
  __align__(16) uint32_t src[2][32][20];  // sum-difference words of the CTU's samples, raster and transposed
  uint16_t px[33][68];                    // samples x - 1 .. x + 63 (columns clamped) of rows y - 1 .. y + 31
  // reference rows [block][unfiltered / filtered][above / left], then the
  // extended rows of the negative slopes: the projected side, the corner, n + 1 samples
  __align__(16) int16_t ref[4 * 4 * kCtsRef + 4464 + 16];
  CtsMode mode[4 * kCtsModes];            // [block][candidate]
  uint32_t cost[4 * kCtsModes];
  uint32_t taps[3][32];
  int32_t dc[4];
  uint8_t cand[kCtsModes];                // modes by candidate
  uint8_t ang[kCtsModes], flat[kCtsModes];  // the angular candidates, and planar / DC
  int32_t n_ang, n_flat;
  uint32_t wide;                          // bit 0: bit depth above 10, bit 1: samples above the bit depth
};

// [1 2 1] filtered sample k of row r (o: the other row's first sample), 2n samples.
__device__ __forceinline__ int cts_filtered(const int16_t* r, int o1, int k, int n) {
  if (k == 2 * n) return r[k];
  return ((k == 0 ? o1 : r[k - 1]) + 2 * r[k] + r[k + 1] + 2) >> 2;
}

// The block of split type s that covers tile (tx, ty).
__device__ __forceinline__ int cts_block(int s, int tx, int ty) {
  switch (s) {
    case 0: return 0;
    case 1: return (ty >> 1) * 2 + (tx >> 1);
    case 2: return ty >> 1;
    case 3: return tx >> 1;
    case 4: return (ty + 1) >> 1;
    default: return (tx + 1) >> 1;
  }
}

// SATD of one tile for one angular candidate by one lane (10-bit samples or
// less, all within the bit depth). row: the tile's sum-difference words, line
// pitch 20; x0, y0: the tile's position along and across the mode's direction.
__device__ __forceinline__ uint32_t cts_tile(const CtsWs& S, const CtsMode& m, const uint32_t* row, int x0, int y0,
                                             int maxv) {
  const uint32_t* ref = reinterpret_cast<const uint32_t*>(S.ref);
  const bool pdpc = x0 < m.lim;
  uint32_t w[4][4], top[4][4];
  // two halves of four lines, rolled: unrolled over all eight, the code left
  // the instruction cache
#pragma unroll 1
  for (int half = 0; half < 2; half++, y0 += 4, row += 80) {
    if (half) {
#pragma unroll
      for (int r = 0; r < 4; r++)
#pragma unroll
        for (int k = 0; k < 4; k++) top[r][k] = w[r][k];
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int y = y0 + r;
      const int dp = m.angle * (y + 1);
      const uint32_t taps = S.taps[m.tab][dp & 31];
      const int j = m.main + (dp >> 5) + x0;
      const uint32_t* q = ref + (j >> 1);
      uint32_t e[6], c = q[0];
      const uint32_t sh = (j & 1) * 16;
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const uint32_t n = q[k + 1];
        e[k] = __funnelshift_r(c, n, sh);
        c = n;
      }
      int v[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int k = i >> 1;
        const uint32_t lo = (i & 1) ? __byte_perm(e[k], e[k + 1], 0x5432) : e[k];
        const uint32_t hi = (i & 1) ? __byte_perm(e[k + 1], e[k + 2], 0x5432) : e[k + 1];
        v[i] = __dp2a_hi((int)hi, (int)taps, __dp2a_lo((int)lo, (int)taps, 32)) >> 6;
      }
      if (m.tab == 1) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = clampi(v[i], 0, maxv);
      }
      if (pdpc) {
        const bool zero = (m.flags & kCtsZero) != 0;
        const int corner = S.ref[m.main];
        int inv = 256 + (x0 + 1) * m.inv;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          if (x0 + i < m.lim) {
            const int wl = 32 >> ((2 * (x0 + i)) >> m.scale);
            v[i] = clampi(v[i] + ((wl * (S.ref[m.side + y + (inv >> 9) + 1] - (zero ? corner : v[i])) + 32) >> 6), 0, maxv);
          }
          inv += m.inv;
        }
      }
      const uint4 s = *reinterpret_cast<const uint4*>(row + r * 20);
      const uint32_t sv[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
      for (int k = 0; k < 4; k++)  // (v0 + v1) + (v0 - v1) * 2^16 - source
        w[r][k] = (uint32_t)v[2 * k] * 0x10001u + ((uint32_t)v[2 * k + 1] * 0xFFFF0001u - sv[k]);
      // two stages along the line
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const uint32_t a = w[r][k], b = w[r][k + 2];
        w[r][k] = a + b;
        w[r][k + 2] = a - b;
      }
#pragma unroll
      for (int k = 0; k < 4; k += 2) {
        const uint32_t a = w[r][k], b = w[r][k + 1];
        w[r][k] = a + b;
        w[r][k + 1] = a - b;
      }
    }
    // two stages down the lines
#pragma unroll
    for (int st = 1; st < 4; st <<= 1)
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (!(r & st)) {
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const uint32_t a = w[r][k], b = w[r + st][k];
            w[r][k] = a + b;
            w[r + st][k] = a - b;
          }
        }
  }
  // the last stage: 2 max(|a|, |b|) of lines r and r + 4
  int sum = 0;
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int k = 0; k < 4; k++) {
      // halves as two 16-bit numbers: a negative low half borrowed from the high one
      uint32_t a = top[r][k], b = w[r][k];
      a += (a & 0x8000u) << 1;
      b += (b & 0x8000u) << 1;
      const uint32_t x = __vmaxs2(__vmaxs2(a, b), __vneg2(__vmins2(a, b)));
      sum = __dp2a_lo((int)x, 0x0202, sum);
    }
  return ((uint32_t)sum + 2) >> 2;
}

// Prediction of eight samples of a line, 32-bit and one sample at a time.
__device__ __forceinline__ void cts_line(const CtsWs& S, const CtsMode& m, int b, int lw, int lh, int x0, int y,
                                         int maxv, int (&v)[8]) {
  const int w = 1 << lw, h = 1 << lh;
  if (m.mode <= 1) {
    // planar (predict.rs:1688-1719, filtered: every block has over 32 samples)
    // or DC (:1722-1736) with PDPC (:1739-1754)
    const int16_t* top = S.ref + m.main + 1;
    const int16_t* left = S.ref + m.side + 1;
    const int sc = (lw + lh - 2) >> 2;
    const int tr = top[w], bl = left[h], lf = left[y], wt = 32 >> min((y * 2) >> sc, 31);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int x = x0 + i;
      int p = S.dc[b];
      if (m.mode == 0) {
        const int hor = (lf << lw) + (x + 1) * (tr - lf);
        const int vert = (top[x] << lh) + (y + 1) * (bl - top[x]);
        p = ((hor << lh) + (vert << lw) + (1 << (lw + lh))) >> (1 + lw + lh);
      }
      const int wl = 32 >> min((x * 2) >> sc, 31);
      v[i] = p + ((wl * (lf - p) + wt * (top[x] - p) + 32) >> 6);
    }
    return;
  }
  const int dp = m.angle * (y + 1);
  const uint32_t t = S.taps[m.tab][dp & 31];
  const int16_t* rm = S.ref + m.main + (dp >> 5) + x0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    int p = rm[i + 1];
    if (m.tab != 2)
      p = clampi(((int8_t)t * rm[i] + (int8_t)(t >> 8) * rm[i + 1] + (int8_t)(t >> 16) * rm[i + 2] +
                  (int8_t)(t >> 24) * rm[i + 3] + 32) >> 6, 0, maxv);
    const int x = x0 + i;
    if (x < m.lim) {
      const int wl = 32 >> ((2 * x) >> m.scale);
      const int sv = S.ref[m.side + y + ((256 + (x + 1) * m.inv) >> 9) + 1];
      p = clampi(p + ((wl * (sv - ((m.flags & kCtsZero) ? S.ref[m.main] : p)) + 32) >> 6), 0, maxv);
    }
    v[i] = p;
  }
}

// SATD of four tiles by one warp, a lane per line of the mode's direction. The
// transform runs along the samples' rows first, whose sums are 16-bit numbers;
// only with sources above the bit depth do they wrap. For those (kRows) the
// rows of a horizontal mode, which lie across the lanes, come first; for all
// others the order does not change a sum, and the lane's own line comes first
// (keeping to the rows there cost 1.7% of a 10-bit search, 4% at 12 bits; as a
// function called where it is needed 0.6% and nothing).
template <bool kRows>
__device__ __forceinline__ uint32_t cts_lines(const CtsWs& S, const CtsMode& m, int b, int lw, int lh, int tx, int ty,
                                              int bx, int by, int maxv) {
  const int r = threadIdx.x & 7;
  const bool ver = (m.flags & kCtsVer) != 0;
  const int x0 = 8 * (ver ? tx : ty) - (ver ? bx : by), y = 8 * (ver ? ty : tx) - (ver ? by : bx) + r;
  int v[8];
  cts_line(S, m, b, lw, lh, x0, y, maxv, v);
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int line = 8 * (ver ? ty : tx) + r, at = 8 * (ver ? tx : ty) + i;
    const int s = ver ? S.px[1 + line][1 + at] : S.px[1 + at][1 + line];
    v[i] = (int16_t)(s - v[i]);
  }
  auto along = [&] {
#pragma unroll
    for (int st = 1; st < 8; st <<= 1)
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (!(k & st)) {
          const int a = v[k], c = v[k + st];
          v[k] = a + c;
          v[k + st] = a - c;
        }
  };
  if (!kRows || ver) {
    along();
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = (int16_t)v[k];
  }
  if (kRows) __syncwarp();
#pragma unroll
  for (int st = 1; st < 8; st <<= 1)
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int o = __shfl_xor_sync(0xffffffffu, v[k], st);
      v[k] = (r & st) ? o - v[k] : v[k] + o;
    }
  if (kRows && !ver) {
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = (int16_t)v[k];
    along();
  }
  if (kRows) __syncwarp();
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) sum += (uint32_t)abs(v[k]);
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  sum += __shfl_xor_sync(0xffffffffu, sum, 4);
  return (sum + 2) >> 2;
}

// Adds the costs of `n` candidates, all or the flat ones, a lane per line.
template <bool kRows>
__device__ __forceinline__ void cts_by_lines(CtsWs& S, int split, int n, bool all, int maxv) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, first = c_split_first[split];
  for (int i = kCtsWarps - 1 - warp; i < 4 * n; i += kCtsWarps) {
    const int c = all ? i >> 2 : S.flat[i >> 2], tile = 4 * (i & 3) + (lane >> 3);
    const int tx = tile & 3, ty = tile >> 2, b = cts_block(split, tx, ty);
    const CtsMode m = S.mode[b * kCtsModes + c];
    const uint8_t* g = c_search_blocks[first + b];
    const uint32_t s = cts_lines<kRows>(S, m, b, g[2], g[3], tx, ty, g[0], g[1], maxv);
    if ((lane & 7) == 0) atomicAdd(&S.cost[b * kCtsModes + c], s);
  }
}
__device__ __noinline__ void cts_rows(CtsWs& S, int split, int n, int maxv) {
  cts_by_lines<true>(S, split, n, true, maxv);
}

// Grid: CTUs x 6 split types.
__global__ void __launch_bounds__(kCtsWarps * 32, 3) k_ctu_costs(const __grid_constant__ CtsArgs A) {
  __shared__ CtsWs S;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  constexpr int kThreads = kCtsWarps * 32;
  const uint32_t ctu = blockIdx.x / 6;
  const int split = (int)(blockIdx.x - ctu * 6);
  const vvcg_ctu_search_req R = A.reqs[ctu];
  if (!((R.split_mask >> split) & 1)) return;
  const int maxv = (1 << A.bd) - 1, mid = 1 << (A.bd - 1);
  const int n_cand = R.n_cand ? R.n_cand : kCtsModes;
  const int first = c_split_first[split], nb = c_split_count[split];
  const int cx = (int)R.x, cy = (int)R.y;
  // samples around the CTU; the candidates
  if (t == 0) S.wide = A.bd > 10;
  __syncthreads();
  uint32_t over = 0;
#pragma unroll
  for (int q = 0; q < (33 + kCtsWarps - 1) / kCtsWarps; q++) {
    const int y = warp + q * kCtsWarps, py = cy - 1 + y;
    if (y > 32) break;
    const uint16_t* row = A.src + (int64_t)py * A.stride;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int x = lane + 32 * k, px = cx - 1 + x;
      uint32_t v = 0;
      if (x < 65 && px >= 0 && py >= 0) v = __ldg(row + min(px, A.width - 1));
      over |= v > (uint32_t)maxv;
      if (x < 65) S.px[y][x] = (uint16_t)v;
    }
  }
  if (over) atomicOr(&S.wide, 2u);
  for (int i = t; i < 4 * kCtsModes; i += kThreads) S.cost[i] = 0;
  for (int i = t; i < n_cand; i += kThreads) S.cand[i] = R.n_cand ? R.cand[i] : (uint8_t)i;
  if (t < 32) {
    S.taps[0][t] = (uint32_t)(16 - (t >> 1)) | (uint32_t)(32 - (t >> 1)) << 8 | (uint32_t)(16 + (t >> 1)) << 16 |
                   (uint32_t)(t >> 1) << 24;
    S.taps[1][t] = reinterpret_cast<const uint32_t*>(c_chroma_taps4)[t];
    S.taps[2][t] = 64u << 8;
  }
  __syncthreads();
  if (t == 0) {  // angular candidates apart from planar and DC
    int a = 0, f = 0;
    for (int c = 0; c < n_cand; c++)
      if (S.cand[c] >= 2)
        S.ang[a++] = (uint8_t)c;
      else
        S.flat[f++] = (uint8_t)c;
    S.n_ang = a;
    S.n_flat = f;
  }
  // raw reference rows (gather_references_16, predict.rs:3016-3076)
  for (int i = t; i < nb * 2 * kCtsRef; i += kThreads) {
    const int b = i / (2 * kCtsRef), k = i % kCtsRef;
    const bool above = (i / kCtsRef) % 2 == 0;
    const int x = c_search_blocks[first + b][0], y = c_search_blocks[first + b][1];
    const int w = 1 << c_search_blocks[first + b][2], h = 1 << c_search_blocks[first + b][3];
    const bool ha = cy + y > 0, hl = cx + x > 0;
    int v = mid;
    if (k == 0)
      v = ha && hl ? S.px[y][x] : (ha ? S.px[y][x + 1] : (hl ? S.px[y + 1][x] : mid));
    else if (above)
      v = ha ? S.px[y][x + min(k, 2 * w)] : (hl ? S.px[y + 1][x] : mid);
    else
      v = hl ? S.px[y + min(k, h)][x] : (ha ? S.px[y][x + 1] : mid);
    S.ref[((b * 2) * 2 + (above ? 0 : 1)) * kCtsRef + k] = (int16_t)v;
  }
  // the CTU's samples as sum-difference words
  for (int i = t; i < 32 * 16; i += kThreads) {
    const int y = i >> 4, k = i & 15;
    const uint32_t a = S.px[1 + y][1 + 2 * k], b = S.px[1 + y][2 + 2 * k];
    S.src[0][y][k] = a * 0x10001u + b * 0xFFFF0001u;
    const uint32_t c = S.px[1 + 2 * k][1 + y], d = S.px[2 + 2 * k][1 + y];
    S.src[1][y][k] = c * 0x10001u + d * 0xFFFF0001u;
  }
  __syncthreads();
  // filtered rows; the DC values
  for (int i = t; i < nb * 2 * kCtsRef; i += kThreads) {
    const int b = i / (2 * kCtsRef), k = i % kCtsRef, side = (i / kCtsRef) % 2;
    const int n = 1 << c_search_blocks[first + b][side ? 3 : 2];
    const int16_t* r = S.ref + (b * 4 + side) * kCtsRef;
    const int16_t* o = S.ref + (b * 4 + 1 - side) * kCtsRef;
    S.ref[(b * 4 + 2 + side) * kCtsRef + k] = (int16_t)cts_filtered(r, o[1], min(k, 2 * n), n);
  }
  if (warp < nb) {
    const int lw = c_search_blocks[first + warp][2], lh = c_search_blocks[first + warp][3];
    const int16_t* a = S.ref + warp * 4 * kCtsRef;
    const int16_t* l = a + kCtsRef;
    const int st = __reduce_add_sync(0xffffffffu, lane < (1 << lw) ? (int)a[1 + lane] : 0);
    const int sl = __reduce_add_sync(0xffffffffu, lane < (1 << lh) ? (int)l[1 + lane] : 0);
    const int denom = lw == lh ? 2 << lw : max(1 << lw, 1 << lh);
    const int sum = (lw >= lh ? st : 0) + (lw <= lh ? sl : 0);
    if (lane == 0) S.dc[warp] = (sum + (denom >> 1)) >> floor_log2((unsigned)denom);
  }
  // the candidates' parameters (init_angular_params, predict.rs:1608-1685)
  for (int i = t; i < nb * n_cand; i += kThreads) {
    const int b = i / n_cand, c = i - b * n_cand, dir = S.cand[c];
    const int lw = c_search_blocks[first + b][2], lh = c_search_blocks[first + b][3], w = 1 << lw, h = 1 << lh;
    const int rows = b * 4 * kCtsRef;
    CtsMode m;
    m.mode = dir;
    if (dir <= 1) {
      const int at = rows + (dir == 0 ? 2 * kCtsRef : 0);
      m = CtsMode{0, 0, (uint16_t)at, (uint16_t)(at + kCtsRef), 0, 0, 0, kCtsVer, dir};
    } else {
      int mode = dir;
      const int delta = abs(lw - lh), s = delta == 0 ? 0 : (delta == 1 ? 6 : 10);  // blocks are at most 1:4
      if (w > h && dir < 2 + s)
        mode = dir + 65;
      else if (h > w && dir > 66 - s)
        mode = dir - 65;
      const bool ver = mode >= 34;
      const int am = ver ? mode - 50 : -(mode - 18), absm = min(31, abs(am));
      const int ang = c_ang_table[absm], inv = c_inv_ang_table[absm];
      const int ww = ver ? w : h, wh = ver ? h : w;
      int scale = 0, lim = 0;
      if (am == 0) {
        scale = (lw + lh - 2) >> 2;
        lim = min(3 << scale, ww);
      } else if (am > 0) {
        scale = min(2, floor_log2((unsigned)wh) - (floor_log2((unsigned)max(1, 3 * inv - 2)) - 8));
        lim = scale >= 0 ? min(3 << scale, ww) : 0;
      }
      const bool integer = (ang & 31) == 0;
      const bool far = min(abs(mode - 18), abs(mode - 50)) > c_intra_filter_thr[min(7, (lw + lh) >> 1)];
      const int at = rows + (far && integer ? 2 * kCtsRef : 0);  // the filtered rows
      const int n_neg = w + h + 2 + 2;  // extended row of a negative slope
      int neg_at = 4 * 4 * kCtsRef;
      for (int q = 0; q < b; q++)
        neg_at += 31 * ((1 << c_search_blocks[first + q][2]) + (1 << c_search_blocks[first + q][3]) + 4);
      m.angle = (int16_t)(am < 0 ? -ang : ang);
      m.inv = (int16_t)(am == 0 ? 0 : inv);
      m.main = (uint16_t)(am < 0 ? neg_at + (dir - 19) * n_neg + wh : at + (ver ? 0 : kCtsRef));
      m.side = (uint16_t)(at + (ver ? kCtsRef : 0));
      m.tab = integer ? 2 : (far ? 0 : 1);
      m.scale = (int8_t)max(scale, 0);
      m.lim = (uint8_t)lim;
      m.flags = (uint8_t)((ver ? kCtsVer : 0) | (am == 0 ? kCtsZero : 0));
    }
    S.mode[b * kCtsModes + c] = m;
  }
  __syncthreads();
  // extended rows of the negative slopes (modes 19..49, predict.rs:3260-3290), a warp each
  for (int b = 0; b < nb; b++) {
    const int w = 1 << c_search_blocks[first + b][2], h = 1 << c_search_blocks[first + b][3];
    // (the full set holds the modes at their own numbers)
    for (int c = warp + (R.n_cand ? 0 : 19); c < (R.n_cand ? n_cand : 50); c += kCtsWarps) {
      const CtsMode& m = S.mode[b * kCtsModes + c];
      if (m.angle >= 0) continue;  // planar and DC among them
      const bool ver = (m.flags & kCtsVer) != 0;
      const int ww = ver ? w : h, wh = ver ? h : w, inv = m.inv;
      const int16_t* so = S.ref + m.side;
      const int16_t* mo = ver ? so - kCtsRef : so + kCtsRef;
      int16_t* d = S.ref + m.main;
      if (lane < wh) d[-1 - lane] = so[min(((lane + 1) * inv + 256) >> 9, wh)];
      if (lane <= ww + 1) d[lane] = mo[lane];
      if (lane + 32 <= ww + 1) d[lane + 32] = mo[lane + 32];
    }
  }
  __syncthreads();
  const bool wide = S.wide != 0;
  const int n_ang = S.n_ang, n_flat = S.n_flat;
  if (!wide) {
    // two candidates' tiles a warp: negative slopes have no PDPC, the others agree on its extent
    for (int i = t; i < 16 * n_ang; i += kThreads) {
      const int tile = i & 15, c = S.ang[i >> 4];
      const int tx = tile & 3, ty = tile >> 2, b = cts_block(split, tx, ty);
      const CtsMode m = S.mode[b * kCtsModes + c];
      const int bx = c_search_blocks[first + b][0], by = c_search_blocks[first + b][1];
      const bool ver = (m.flags & kCtsVer) != 0;
      const int at = 8 * (ver ? tx : ty), line = 8 * (ver ? ty : tx);
      const uint32_t s = cts_tile(S, m, &S.src[ver ? 0 : 1][line][at >> 1], at - (ver ? bx : by), line - (ver ? by : bx), maxv);
      atomicAdd(&S.cost[b * kCtsModes + c], s);
    }
  }
  // a lane per line: planar and DC, or everything
  if (S.wide & 2)
    cts_rows(S, split, n_cand, maxv);
  else
    cts_by_lines<false>(S, split, wide ? n_cand : n_flat, wide, maxv);
  __syncthreads();
  // the first candidate with the lowest cost
  if (warp < nb) {
    uint32_t best = 0xFFFFFFFFu;
    int bc = 0;
    for (int c = lane; c < n_cand; c += 32) {
      const uint32_t v = S.cost[warp * kCtsModes + c] +
                         (uint32_t)(((uint64_t)A.lambda_q8 * search_mode_bits(S.cand[c])) >> 8);
      if (A.mode_costs && first + warp == 0 && R.n_cand == 0) A.mode_costs[(size_t)ctu * kCtsModes + c] = v;
      if (v < best) {
        best = v;
        bc = c;
      }
    }
    const uint32_t low = __reduce_min_sync(0xffffffffu, best);
    const int win = __reduce_min_sync(0xffffffffu, best == low ? bc : 0x7fffffff);
    if (lane == 0) {
      A.block_cost[(size_t)ctu * 15 + first + warp] = low;
      A.block_mode[(size_t)ctu * 15 + first + warp] = low == 0xFFFFFFFFu ? 0 : S.cand[win];
    }
  }
}

// Per CTU: each evaluated split's cost (its blocks' costs + lambda * split
// bits), the first lowest wins.
__global__ void k_ctu_search_combine(const vvcg_ctu_search_req* reqs, int n, uint32_t lambda_q8,
                                     const uint32_t* block_cost, const uint8_t* block_mode,
                                     vvcg_ctu_search_res* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t mask = reqs[i].split_mask;
  vvcg_ctu_search_res o;
  o.cost = 0xFFFFFFFFu;
  o.split = 0xFF;
  o.cu_mode = 0xFF;
  for (int k = 0; k < 4; k++) o.modes[k] = 0xFF;
  o.reserved[0] = o.reserved[1] = 0;
  for (int s = 0; s < 6; s++) {
    o.split_cost[s] = 0xFFFFFFFFu;
    if (!(mask & (1u << s))) continue;
    uint64_t c = ((uint64_t)lambda_q8 * c_split_bits[s]) >> 8;
    for (int k = 0; k < c_split_count[s]; k++) c += block_cost[(size_t)i * 15 + c_split_first[s] + k];
    o.split_cost[s] = c < 0xFFFFFFFEull ? (uint32_t)c : 0xFFFFFFFEu;
    if (o.split_cost[s] < o.cost) {
      o.cost = o.split_cost[s];
      o.split = (uint8_t)s;
      for (int k = 0; k < 4; k++)
        o.modes[k] = k < c_split_count[s] ? block_mode[(size_t)i * 15 + c_split_first[s] + k] : 0xFF;
    }
  }
  if (mask & 1u) o.cu_mode = block_mode[(size_t)i * 15];
  out[i] = o;
}

}  // namespace vvcg
