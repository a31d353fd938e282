// The CNN pruner of the GPU encoder: 32x32 luma blocks (samples / max value,
// rounded to bf16) with a second, constant input plane QP / 63 (the split
// decision depends on lambda) -> conv 3x3 2->32 + ReLU -> 3 x (conv 3x3
// 32->32 + ReLU) -> global average -> 67 intra-mode logits and 6 split logits.
//
// Forward: two blocks at a time per CTA, each with its own half of the
// threads, image and TMEM (k_cnn_forward). A block's activations stay in
// shared memory as one image of 34 x 34 pixels (a zero halo around 32 x 32)
// in four planes of 8 channels, 16 bytes per pixel, so each layer's 3x3
// convolution is 144 tcgen05 MMAs (M = 128 pixels, N = 32 output channels,
// K = 16 input channels of one tap) whose A operand points straight into the
// image: the 8 rows of a core matrix are 8 neighbouring pixels of an image
// row (16 B apart), SBO steps one image row, LBO one channel plane, and a tap
// is an address offset. The 8 tiles of a layer accumulate in 256 TMEM
// columns; 8 warps read them back, add the bias, apply ReLU and write the
// image again (or the average): the layer's MMAs are done with it by then.
// The first layer (two input channels) runs on the CUDA cores.
#pragma once
#include "umma.cuh"

namespace vvcg {

constexpr int kCnnCh = 32, kCnnModes = 67, kCnnSplits = 6, kCnnOut = kCnnModes + kCnnSplits;
constexpr int kCnnConvW = kCnnCh * kCnnCh * 9;  // 9216
// fp32 parameter vector: W1 [co][2 inputs][tap], b1, then per layer 2..4
// W [co][ci][tap] and b, then the heads W [out][ch] and b.
constexpr int kOffW1 = 0, kOffB1 = 576;
__host__ __device__ constexpr int cnn_off_w(int layer) { return 608 + (layer - 2) * (kCnnConvW + kCnnCh); }
__host__ __device__ constexpr int cnn_off_b(int layer) { return cnn_off_w(layer) + kCnnConvW; }
constexpr int kOffWi = cnn_off_w(5), kOffBi = kOffWi + kCnnModes * kCnnCh;
constexpr int kOffWs = kOffBi + kCnnModes, kOffBs = kOffWs + kCnnSplits * kCnnCh;
constexpr int kCnnParams = kOffBs + kCnnSplits;  // 30761

constexpr int kImgW = 34;                 // 32 + halo
// One plane of 8 channels, bytes. The 16 bytes of padding spread the four
// planes over the banks: layer 1 stores 4 bytes of every plane in two rows at
// once (four-way conflicts without them).
constexpr int kPlane = kImgW * kImgW * 16 + 16;
constexpr int kImg = 4 * kPlane;
constexpr int kPackL = 36 * 32 * 16;        // packed bf16 weights of one layer: [tap*4 + ci/8][co][ci%8]
constexpr int kCnnThreads = 256;
constexpr uint32_t kCnnIdesc = umma_idesc_bf16(128, 32);
constexpr int kCnnGroups = 2;                   // blocks in flight per CTA of the forward pass
constexpr int kHeadPitch = kCnnCh + 1;          // head weights by row, one bank apart
constexpr int kXPad = 34 * 34;                  // the input zero-padded by one pixel
constexpr int kCnnGroupF = kXPad + 8 * 32 + 32;  // floats of one group: input, partial averages, average
constexpr int kCnnMisc = (576 + 32 + 96 + kCnnOut * kHeadPitch + 76 - kCnnOut % 4 + kCnnGroups * kCnnGroupF) * 4;
constexpr int kCnnSmem = kCnnGroups * kImg + 3 * kPackL + kCnnMisc + 64;
static_assert(kCnnSmem <= 227 * 1024, "forward shared memory");

__device__ __forceinline__ uint16_t f2bf(float f) {  // round to nearest even
  const uint32_t u = __float_as_uint(f);
  return (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
}
__device__ __forceinline__ float bf2f(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }
// Two values to bf16, round to nearest even: the first in the low half. Equal
// to f2bf for all but NaN.
__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// Two fp32 values in a register pair, and their fused multiply-adds (each
// half rounds as fmaf does).
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// Sums v[c] over the warp for kN channels c, into the lanes of number
// c * 32 / kN on: each step halves the channels that a lane carries (31
// shuffles for 32 channels instead of 160; the additions pair the same lanes,
// at distances 16, 8, 4, 2, 1, as a butterfly per channel).
template <int kN>
__device__ __forceinline__ float warp_sum(float* v, int lane) {
#pragma unroll
  for (int o = 16, n = kN / 2; o > 0; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int c = 0; c < n; c++) {
      const float send = up ? v[c] : v[c + n], keep = up ? v[c + n] : v[c];
      v[c] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
    }
    if (n == 0) v[0] += __shfl_xor_sync(0xFFFFFFFFu, v[0], o);
  }
  return v[0];
}
// Barriers of one group of kCnnThreads threads (the id in a register takes
// all 16 barriers, which the one CTA of an SM can have).
__device__ __forceinline__ void cnn_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kCnnThreads) : "memory");
}
__device__ __forceinline__ bool cnn_sync_and(int id, bool v) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(id), "n"(kCnnThreads)
      : "memory");
  return r != 0;
}

// pack[layer][tap*4 + ci/8][co][ci%8] = bf16(W[co][ci][tap]) (forward), or with
// flip the weights of the transposed convolution: [tap*4 + co/8][ci][co%8] =
// bf16(W[co][ci][8 - tap]).
__global__ void k_cnn_pack(const float* __restrict__ params, uint16_t* __restrict__ pack, bool flip) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * kCnnConvW) return;
  const int l = i / kCnnConvW, r = i % kCnnConvW;
  const int kg = r / 256, n = (r / 8) % 32, j = r % 8;
  const int tap = kg / 4, g = kg % 4;
  const float* W = params + cnn_off_w(2 + l);
  float v;
  if (!flip)
    v = W[(n * kCnnCh + g * 8 + j) * 9 + tap];  // n = co, input channel g*8+j
  else
    v = W[((g * 8 + j) * kCnnCh + n) * 9 + (8 - tap)];  // n = ci, output channel g*8+j
  pack[i] = f2bf(v);
}

struct CnnFwdArgs {
  const uint16_t* plane;
  int64_t stride;
  int32_t width, height, maxv, n;
  float qp_in;             // the QP plane's value, QP / 63 rounded to bf16
  const uint32_t* ctu_xy;  // n (x, y) pairs
  const float* params;
  const uint16_t* pack;
  float* logits;     // n x 73
  float* gap_out;    // n x 32, or null
  uint16_t* acts;    // n x 4 x 1024 x 32 bf16 (layer, pixel, channel), or null
  uint32_t* status;  // bit 0: a completion wait gave up; bit 1: a block outside the plane
};

// Issues the 144 MMAs of one 3x3 32->32 layer reading image `xin` with the
// packed weights `w` into TMEM columns tile * 32, then (with commit) commits
// to mbar; called behind elect_one(). The start address is the descriptor's
// low field in 16-byte units (one pixel, and it never carries out of its 14
// bits): every operand is a base descriptor plus an offset. Bound by the
// operands' shared-memory reads, 4 KB of A and 1 KB of B per MMA at 128 B per
// cycle (40 cycles; 41 measured).
__device__ __forceinline__ void cnn_issue_layer(uint32_t tmem, uint32_t xin, uint32_t w, uint64_t* mbar,
                                                bool commit = true) {
  constexpr uint64_t kA = umma_desc(0, kPlane, kImgW * 16), kB = umma_desc(0, 512, 128);
  const uint32_t a0 = (uint32_t)kA + (xin >> 4), b0 = (uint32_t)kB + (w >> 4);
#pragma unroll 1
  for (int tile = 0; tile < 8; tile++) {
    const uint32_t at = a0 + (tile >> 2) * 16 * kImgW + (tile & 3) * 8;
#pragma unroll
    for (int tap = 0; tap < 9; tap++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        umma_bf16(tmem + tile * 32, (kA >> 32 << 32) | (at + (tap / 3) * kImgW + tap % 3 + h * (2 * kPlane / 16)),
                  (kB >> 32 << 32) | (b0 + (tap * 4 + 2 * h) * 32), kCnnIdesc, (tap | h) != 0);
  }
  if (commit) umma_commit(mbar);
}

// The four input samples of thread t of a group (rows t / 32 + 8 k) of block
// blk; false, with nothing read, for a block outside the plane.
__device__ __forceinline__ bool cnn_load_px(const uint16_t* plane, int64_t stride, int width, int height,
                                            const uint32_t* ctu_xy, int blk, int t, uint16_t* px) {
  const uint32_t ux = ctu_xy[2 * blk], uy = ctu_xy[2 * blk + 1];
  if (ux > (uint32_t)width - 32 || uy > (uint32_t)height - 32 || width < 32 || height < 32) return false;
#pragma unroll
  for (int k = 0; k < 4; k++) px[k] = plane[(int64_t)((int)uy + (t >> 5) + 8 * k) * stride + (int)ux + (t & 31)];
  return true;
}

// Layer 1 of one block on the CUDA cores: 16 lanes take a pair of channels
// each (both in one packed fp32 operation) and the warp's halves two image
// rows each, so the 36 weights of a thread stay in registers and a step of two
// columns reads eight new samples for 72 packed operations. Sums run in tap
// order, the input's first, then the QP plane's, zero in the halo. xt is the
// zero-padded input by columns. Bound by the fp32 pipe: 590 k multiply-adds
// are 4.6 k cycles (a thread per pixel and all channels read each weight from
// shared memory again: 16 k cycles, the load path's rate).
__device__ __forceinline__ void cnn_layer1(const float* xt, const float2* w1, const float2* b1, float qp_in,
                                           uint8_t* img, uint16_t* acts, int warp, int lane) {
  const int c2 = lane & 15, y0 = 4 * warp + 2 * (lane >> 4);
  uint64_t wx[9], wq[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    wx[k] = ((const uint64_t*)w1)[k * 16 + c2];
    wq[k] = ((const uint64_t*)w1)[(9 + k) * 16 + c2];
  }
  const uint64_t bias = ((const uint64_t*)b1)[c2];
  const uint64_t q = f2_pack(qp_in, qp_in), q0 = y0 == 0 ? 0ull : q, q3 = y0 == 30 ? 0ull : q;
  const float* xp = xt + y0;
  float2 na[2], nb[2];  // rows y0 - 1 .. y0 + 2 of the next two columns
  auto load = [&](int x) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      na[i] = *(const float2*)(xp + (x + i) * kImgW);
      nb[i] = *(const float2*)(xp + (x + i) * kImgW + 2);
    }
  };
  uint64_t in[4][4];  // columns x - 1 .. x + 2 (a ring), the four rows
  auto put = [&](int i, uint64_t* v) {
    v[0] = f2_pack(na[i].x, na[i].x);
    v[1] = f2_pack(na[i].y, na[i].y);
    v[2] = f2_pack(nb[i].x, nb[i].x);
    v[3] = f2_pack(nb[i].y, nb[i].y);
  };
  load(0);
  put(0, in[0]);
  put(1, in[1]);
  load(2);
  put(0, in[2]);
  put(1, in[3]);
  uint8_t* dst = img + (c2 >> 2) * kPlane + ((y0 + 1) * kImgW + 1) * 16 + (c2 & 3) * 4;
  uint32_t* ga = acts ? (uint32_t*)acts + y0 * 32 * 16 + c2 : nullptr;
  // two columns by two rows at a time: four independent sums
#pragma unroll 1
  for (int x0 = 0; x0 < 32; x0 += 4)
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      const int x = x0 + j;
      if (x < 30) load(x + 4);
      uint64_t s[4] = {bias, bias, bias, bias};
#pragma unroll
      for (int k = 0; k < 9; k++)
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = f2_fma(wx[k], in[(j + (i & 1) + k % 3) & 3][(i >> 1) + k / 3], s[i]);
#pragma unroll
      for (int k = 0; k < 9; k++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int row = (i >> 1) + k / 3;
          uint64_t v = row == 0 ? q0 : row == 3 ? q3 : q;
          if (j == 0 && (i & 1) == 0 && k % 3 == 0 && x0 == 0) v = 0ull;
          if (j == 2 && (i & 1) == 1 && k % 3 == 2 && x0 == 28) v = 0ull;
          s[i] = f2_fma(wq[k], v, s[i]);
        }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float2 o = f2_unpack(s[i]);
        const uint32_t pk = pack_bf2(fmaxf(o.x, 0.0f), fmaxf(o.y, 0.0f));
        *(uint32_t*)(dst + ((i >> 1) * kImgW + x + (i & 1)) * 16) = pk;
        if (ga) ga[((i >> 1) * 32 + x + (i & 1)) * 16] = pk;
      }
      put(0, in[j & 3]);
      put(1, in[(j + 1) & 3]);
    }
}

// Takes one of the turns of a CTA's two groups, given back by atomicExch. One
// group at a time is in layer 1 and one at a time issues MMAs: side by side
// both would take twice as long and then do the next part side by side too,
// block after block. The turns are only for speed: after some tens of
// microseconds a group goes on without.
__device__ __forceinline__ void cnn_take(uint32_t* turn) {
  for (int i = 0; i < 1024 && atomicCAS(turn, 0u, 1u) != 0u; i++) __nanosleep(32);
}

// Persistent, one CTA per SM with two groups of 8 warps that work on blocks
// of their own, independently: while one group's MMAs run, the other adds
// biases, packs and stores, and the tensor core idles only where both do
// (one block at a time: MMAs 24 k of a block's 64 k cycles, serial with the
// rest). Each group's image is written in place, so two images and the
// weights fill the shared memory as two ping-pong images of one block would;
// 2 x 256 columns fill the TMEM. The next block's samples are loaded while the
// current block's layers run. 1980 blocks: 414 us
// -> 199 us (the tensor core busy for 35 k of the 42 k cycles that two blocks
// take); without the turns 244 us.
__global__ void __launch_bounds__(kCnnGroups* kCnnThreads, 1) k_cnn_forward(const __grid_constant__ CnnFwdArgs A) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int grp = __shfl_sync(0xFFFFFFFFu, (int)threadIdx.x / kCnnThreads, 0);
  const int t = threadIdx.x % kCnnThreads, warp = __shfl_sync(0xFFFFFFFFu, t >> 5, 0), lane = t & 31;
  uint8_t* W = smem + kCnnGroups * kImg;
  float* w1 = (float*)(W + 3 * kPackL);  // [18][32]
  float* b1 = w1 + 576;
  float* bias = b1 + 32;                         // [3][32]
  float* xt = bias + 96 + grp * kCnnGroupF;      // the group's padded input, by columns
  float* gpart = xt + kXPad;                     // [8 warps][32]
  float* gap = gpart + 256;                      // [32]
  float* heads = bias + 96 + kCnnGroups * kCnnGroupF;  // [73][kHeadPitch], then the 73 biases
  uint64_t* mbars = (uint64_t*)(W + 3 * kPackL + kCnnMisc);
  uint32_t* tslot = (uint32_t*)(mbars + kCnnGroups);
  uint32_t* turn = tslot + 1;  // taken: [0] layer 1, [1] the tensor core
  uint8_t* X = smem + grp * kImg;
  uint64_t* mbar = mbars + grp;

  // weights, zero images (the halos stay zero), TMEM, barriers
  constexpr int kAll = kCnnGroups * kCnnThreads;
  for (int i = threadIdx.x; i < 3 * kPackL / 16; i += kAll) ((uint4*)W)[i] = ((const uint4*)A.pack)[i];
  for (int i = threadIdx.x; i < kCnnGroups * kImg / 16; i += kAll) ((uint4*)smem)[i] = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < 576; i += kAll) w1[(i % 18) * 32 + i / 18] = A.params[kOffW1 + i];
  for (int i = threadIdx.x; i < kCnnOut * 32; i += kAll)
    heads[(i >> 5) * kHeadPitch + (i & 31)] =
        A.params[(i >> 5) < kCnnModes ? kOffWi + i : kOffWs + i - kCnnModes * 32];
  if (threadIdx.x < kCnnOut)
    heads[kCnnOut * kHeadPitch + threadIdx.x] =
        A.params[threadIdx.x < kCnnModes ? kOffBi + threadIdx.x : kOffBs + threadIdx.x - kCnnModes];
  for (int i = t; i < kXPad; i += kCnnThreads) xt[i] = 0.0f;
  if (threadIdx.x < 32) b1[t] = A.params[kOffB1 + t];
  if (threadIdx.x < 96) bias[t] = A.params[cnn_off_b(2 + t / 32) + t % 32];
  if (threadIdx.x < 32) {
    tmem_alloc(tslot, kCnnGroups * 256);
    tmem_relinquish();
  }
  if (t == 0) {
    mbar_init(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    turn[0] = turn[1] = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot + grp * 256;
  const float inv = 1.0f / (float)A.maxv;
  const int bar = 1 + grp;
  uint32_t phase = 0;
  bool ok = true;

  const int step = kCnnGroups * gridDim.x;
  int blk = blockIdx.x + grp * gridDim.x;
  uint16_t px[4];
  bool inside = blk < A.n && cnn_load_px(A.plane, A.stride, A.width, A.height, A.ctu_xy, blk, t, px);
  while (blk < A.n) {
    const int next = blk + step;
    if (!inside) {
      // a block outside the plane: NaN logits, flagged, nothing read
      if (t < kCnnOut) A.logits[(size_t)blk * kCnnOut + t] = __int_as_float(0x7FC00000);
      if (t == 0) atomicOr(A.status, 2u);
      blk = next;
      inside = blk < A.n && cnn_load_px(A.plane, A.stride, A.width, A.height, A.ctu_xy, blk, t, px);
      continue;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      xt[((t & 31) + 1) * kImgW + (t >> 5) + 8 * k + 1] = bf2f(f2bf((float)px[k] * inv));
    if (t == 0) cnn_take(turn);
    cnn_sync(bar);
    uint16_t* acts = A.acts ? A.acts + (size_t)blk * 4 * 1024 * 32 : nullptr;
    cnn_layer1(xt, (const float2*)w1, (const float2*)b1, A.qp_in, X, acts, warp, lane);
    inside = next < A.n && cnn_load_px(A.plane, A.stride, A.width, A.height, A.ctu_xy, next, t, px);
    float acc[32];
#pragma unroll
    for (int c = 0; c < 32; c++) acc[c] = 0.0f;
#pragma unroll 1
    for (int l = 0; l < 3; l++) {
      fence_async_smem();
      tc_fence_before();
      cnn_sync(bar);
      tc_fence_after();
      if (warp == 0 && elect_one()) {
        if (l == 0) atomicExch(turn, 0u);
        cnn_take(turn + 1);
        cnn_issue_layer(tmem, smem_u32(X), smem_u32(W) + l * kPackL, mbar);
        atomicExch(turn + 1, 0u);
      }
      __syncwarp();
      ok = cnn_sync_and(bar, mbar_wait(mbar, phase, 1u << 26));
      phase ^= 1;
      tc_fence_after();
      if (!ok) break;
      const int q = warp & 3;
#pragma unroll 1
      for (int k = 0; k < 4; k++) {
        const int tile = (warp >> 2) + 2 * k;
        const int m = 32 * q + lane, j = m >> 3, r = m & 7;
        const int iy = 16 * (tile >> 2) + j, ix = 8 * (tile & 3) + r;
        float v[32];
        tmem_ld32(tmem + ((uint32_t)(32 * q) << 16) + tile * 32, v);
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          const float4 b = *(const float4*)(bias + l * 32 + c);
          v[c] = fmaxf(v[c] + b.x, 0.0f);
          v[c + 1] = fmaxf(v[c + 1] + b.y, 0.0f);
          v[c + 2] = fmaxf(v[c + 2] + b.z, 0.0f);
          v[c + 3] = fmaxf(v[c + 3] + b.w, 0.0f);
        }
        if (l < 2 || acts) {
          const int off = ((iy + 1) * kImgW + ix + 1) * 16;
          uint4* dst = acts ? (uint4*)(acts + ((size_t)(l + 1) * 1024 + iy * 32 + ix) * 32) : nullptr;
#pragma unroll
          for (int g = 0; g < 4; g++) {
            const uint4 pk = make_uint4(pack_bf2(v[8 * g], v[8 * g + 1]), pack_bf2(v[8 * g + 2], v[8 * g + 3]),
                                        pack_bf2(v[8 * g + 4], v[8 * g + 5]), pack_bf2(v[8 * g + 6], v[8 * g + 7]));
            if (l < 2) *(uint4*)(X + g * kPlane + off) = pk;
            if (dst) dst[g] = pk;
          }
        }
        if (l == 2) {
#pragma unroll
          for (int c = 0; c < 32; c++) acc[c] += v[c];
        }
      }
    }
    if (!ok) break;
    // global average: the warp's 128 pixels, then the 8 warps
    gpart[warp * 32 + lane] = warp_sum<32>(acc, lane);
    tc_fence_before();
    cnn_sync(bar);
    if (t < 32) {
      float s = 0.0f;
      for (int w = 0; w < 8; w++) s += gpart[w * 32 + t];
      gap[t] = s * (1.0f / 1024.0f);
      if (A.gap_out) A.gap_out[(size_t)blk * 32 + t] = gap[t];
    }
    cnn_sync(bar);
    if (t < kCnnOut) {
      const float* Wh = heads + t * kHeadPitch;
      float s = heads[kCnnOut * kHeadPitch + t];
      for (int c = 0; c < 32; c++) s = fmaf(Wh[c], gap[c], s);
      A.logits[(size_t)blk * kCnnOut + t] = s;
    }
    blk = next;
  }
  if (!ok && t == 0) atomicOr(A.status, 1u);
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(*tslot, kCnnGroups * 256);
}

}  // namespace vvcg

namespace vvcg {

// ---------------------------------------------------------------- backward --
//
// One CTA of 16 warps per block (persistent). From the forward's activations
// a1..a4, gap and logits: the head gradients, then per layer l = 4, 3, 2 the
// gradient dZ_l (w.r.t. the layer's pre-activation) held as a bf16 image:
//  * its input gradient dA_{l-1} = conv(dZ_l, flipped W_l) is 144 tcgen05
//    MMAs exactly as in the forward pass (the taps of the transposed
//    convolution are the mirrored address offsets);
//  * behind them, the weight gradient
//    dW_l[co][ci][tap] = sum_p dZ_l[p][co] a_{l-1}[p + tap][ci] is 576 more
//    MMAs (cnn_issue_dw): the 1024 pixels are the K dimension and both
//    images are MN-major operands as they lie;
//  * the epilogue masks dA_{l-1} by a_{l-1} > 0 into dZ_{l-1}, in place of
//    a_{l-1}.
// Layer 1's weight gradient uses the bf16 input. Gradients and the loss
// accumulate in the CTA's own slice of `partial` (no atomics), laid out as
// the threads hold them; a second kernel sums the slices into the parameter
// order.
//
// The two halves of the warps take 16 channels each of the same pixels, so
// every sum keeps one order whatever the number of warps. Beside the MMAs:
// the activations come by cp.async, the next layer's (or block's) into the
// buffer that the layer has done with, during its epilogue; a layer's weight
// gradient is read out of TMEM while the next input gradient's MMAs run.
// 1024 blocks: 958 -> 442 us, the 432 + 1728 MMAs of a block 62 k of 106 k cycles
// at the rate of their operand reads.
struct CnnBwdArgs {
  const uint16_t* plane;
  int64_t stride;
  int32_t width, height, maxv, n;
  float qp_in;
  const uint32_t* ctu_xy;
  const uint8_t* labels;  // n x (mode, split)
  const float* params;
  const float* soft;       // optional n x kCnnModes target distribution of the mode head (else the label)
  const uint16_t* packT;  // flipped packed weights of layers 2..4
  const float* logits;
  const float* gap;
  const uint16_t* acts;
  float* partial;  // [gridDim.x][kCnnSlice]: each CTA's slice of gradients and loss (kSl*)
  float inv_batch;
  uint32_t* status;
};
constexpr int kCnnBwdThreads = 512;
constexpr int kCnnBwdRed = 8 * 32 * 18;  // layer 1's partial weight gradients
constexpr int kCnnBwdMisc = (kXPad + 32 + 32 * 8 + 96 + kCnnBwdRed) * 4;
// A CTA's slice of the partial sums, in floats: per layer 2..4, tap pair and
// column the 64 values of one TMEM column (cnn_slice_w), then W1 and b1, the
// three biases, the heads and the loss.
constexpr int kSlW1 = 3 * 5 * 32 * 64, kSlB = kSlW1 + 608, kSlHeads = kSlB + 96;
constexpr int kSlLoss = kSlHeads + kCnnParams - kOffWi, kCnnSlice = (kSlLoss + 1 + 3) / 4 * 4;
// M = 64, N = 32, both operands MN-major
constexpr uint32_t kCnnIdescW = umma_idesc_bf16(64, 32) | (1u << 15) | (1u << 16);
constexpr int kCnnBwdCols = 512;  // dA_{l-1}: columns 0..255; dW_l: 256..415

// Issues the weight-gradient MMAs of one 3x3 32->32 layer and returns
// without committing. Per tap t, D_t (M = 64, N = 32) += L * H_t^T over the
// 1024 pixels, 16 of one image row per MMA (K), with L the image at `lo`
// and H the one at `hi`: as MN-major operands without swizzle a core matrix
// is 8 pixels (K, 16 B apart) x 8 channels (16 B), LBO = 128 B steps the
// next 8 pixels and SBO = one channel plane the next 8 channels. Only L's
// 32 channels are rows of interest: rows 32..63 read the 4 planes that
// follow L, which must be the other image (lo is the lower of the two
// buffers), and are never read back. The tap's pixel offset applies to the
// activation image: to L when lo_tap, else to H. D_t sits in the TMEM lanes
// 16 (t & 1) + {0..15, 32..47} of columns (t >> 1) * 32 + 0..31 (two M = 64
// accumulators share columns in the two half sub-partitions).
__device__ __forceinline__ void cnn_issue_dw(uint32_t tmem, uint32_t lo, uint32_t hi, bool lo_tap) {
  // Bound by the operands' shared-memory reads, 2 KB of L and 1 KB of H per MMA
  // at 128 B per cycle (24 cycles, as measured).
  constexpr uint64_t kD = umma_desc(0, 128, kPlane);
  const uint32_t a0 = (uint32_t)kD + (lo >> 4), b0 = (uint32_t)kD + (hi >> 4), ma = lo_tap ? 0xFFFFFFFFu : 0u;
#pragma unroll 1
  for (int y = 0; y < 32; y++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t base = (y + 1) * kImgW + 1 + 16 * h;
#pragma unroll
      for (int tap = 0; tap < 9; tap++) {
        const uint32_t sh = (uint32_t)((tap / 3 - 1) * kImgW + tap % 3 - 1);
        umma_bf16(tmem + ((uint32_t)(16 * (tap & 1)) << 16) + (tap >> 1) * 32,
                  (kD >> 32 << 32) | (a0 + base + (sh & ma)), (kD >> 32 << 32) | (b0 + base + (sh & ~ma)),
                  kCnnIdescW, (y | h) != 0);
      }
    }
}
constexpr int kCnnBwdSmem = 2 * kImg + 3 * kPackL + kCnnBwdMisc + 64;
static_assert(kCnnBwdSmem <= 227 * 1024, "backward shared memory");

// Starts the copy of activation image `layer` (0..3) of block blk from global
// into an image buffer (interior only; the halo stays zero) as one cp.async
// group of every thread.
__device__ __forceinline__ void cnn_load_act(uint8_t* img, const uint16_t* acts, int blk, int layer) {
  const uint4* src = (const uint4*)(acts + ((size_t)blk * 4 + layer) * 1024 * 32);
#pragma unroll
  for (int k = 0; k < 1024 * 4 / kCnnBwdThreads; k++) {
    const int i = threadIdx.x + k * kCnnBwdThreads, p = i >> 2, g = i & 3;
    const uint32_t dst = smem_u32(img + g * kPlane + (((p >> 5) + 1) * kImgW + (p & 31) + 1) * 16);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + i) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int kPending>
__device__ __forceinline__ void cnn_load_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// The first block from blk on (in steps of the grid) that lies inside the
// plane with labels in range; flags the skipped ones.
__device__ __forceinline__ int cnn_next_block(const CnnBwdArgs& A, int blk) {
  for (; blk < A.n; blk += gridDim.x) {
    const uint32_t ux = A.ctu_xy[2 * blk], uy = A.ctu_xy[2 * blk + 1];
    if (!(ux > (uint32_t)A.width - 32 || uy > (uint32_t)A.height - 32 || A.width < 32 || A.height < 32 ||
          A.labels[2 * blk] >= kCnnModes || A.labels[2 * blk + 1] >= kCnnSplits))
      break;
    if (threadIdx.x == 0) atomicOr(A.status, 2u);
  }
  return blk;
}

// Adds the weight gradient in TMEM to the slice of layer li: lane quarters 0
// and 1 hold rows 0..31 (the channels of the image at P), a lane tap
// 2 g + lane / 16 of row 16 q + lane % 16, a column the other image's channel.
// kWarps warps, numbered from 0, take part.
template <int kWarps>
__device__ __forceinline__ void cnn_drain_dw(float* part, uint32_t tmem, int li, int warp, int lane) {
  const int q = warp & 3;
  if (q >= 2) return;
#pragma unroll 1
  for (int u = warp >> 2; u < 10; u += kWarps / 4) {
    const int g = u >> 1;
    float v[16], o[16];
    tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + u * 16, v);
    if (2 * g + (lane >> 4) < 9) {  // the loads first, then the stores
      float* d = part + ((li * 5 + g) * 32 + (u & 1) * 16) * 64 + q * 32 + lane;
#pragma unroll
      for (int n = 0; n < 16; n++) o[n] = d[n * 64];
#pragma unroll
      for (int n = 0; n < 16; n++) d[n * 64] = o[n] + v[n];
    }
  }
}

__global__ void __launch_bounds__(kCnnBwdThreads, 1) k_cnn_backward(const __grid_constant__ CnnBwdArgs A) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* P = smem;
  uint8_t* Q = smem + kImg;
  uint8_t* Wt = smem + 2 * kImg;
  // (bf16 normalised input, bf16 1) inside the block, (0, 0) in the halo
  uint32_t* xpad = (uint32_t*)(Wt + 3 * kPackL);
  float* dgap = (float*)(xpad + kXPad);
  float* dbp = dgap + 32;   // [8 warps][32] bias-gradient partials
  float* dlog = dbp + 256;  // [73] logit gradients (+ pad)
  float* red = dlog + 96;   // [8 row groups][32 channels][18]
  uint64_t* mbar = (uint64_t*)(Wt + 3 * kPackL + kCnnBwdMisc);
  uint32_t* tslot = (uint32_t*)(mbar + 1);
  const int t = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, t >> 5, 0), lane = t & 31;
  const int hw = warp >> 3, w8 = warp & 7;  // channel half, warp within it
  float* part = A.partial + (size_t)blockIdx.x * kCnnSlice;
  int blk = cnn_next_block(A, blockIdx.x);
  for (int i = t; i < kCnnSlice / 4; i += kCnnBwdThreads) ((float4*)part)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int i = t; i < 2 * kImg / 16; i += kCnnBwdThreads) ((uint4*)P)[i] = make_uint4(0, 0, 0, 0);
  for (int i = t; i < 3 * kPackL / 16; i += kCnnBwdThreads) ((uint4*)Wt)[i] = ((const uint4*)A.packT)[i];
  for (int i = t; i < kXPad; i += kCnnBwdThreads) xpad[i] = 0;
  if (warp == 0) {
    tmem_alloc(tslot, kCnnBwdCols);
    tmem_relinquish();
  }
  if (t == 0) {
    mbar_init(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  uint32_t phase = 0;
  bool ok = true;

  if (blk < A.n) cnn_load_act(P, A.acts, blk, 3);
  while (blk < A.n) {
    cnn_load_act(Q, A.acts, blk, 2);
    const int bx = (int)A.ctu_xy[2 * blk], by = (int)A.ctu_xy[2 * blk + 1];
    float hwt[kCnnOut];  // warp 2: its channel's head weights, loaded beside the softmax
    // heads: softmax cross-entropy of both heads, mean over the batch
    if (warp == 0 || warp == 1) {
      const float* lg = A.logits + (size_t)blk * kCnnOut;
      const int n_out = warp == 0 ? kCnnModes : kCnnSplits, base = warp == 0 ? 0 : kCnnModes;
      const int label = A.labels[2 * blk + warp];
      float mx = -INFINITY;
      for (int j = lane; j < n_out; j += 32) mx = fmaxf(mx, lg[base + j]);
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
      float se = 0.0f;
      for (int j = lane; j < n_out; j += 32) se += __expf(lg[base + j] - mx);
      for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xFFFFFFFFu, se, o);
      // soft targets of the mode head: cross-entropy against the given
      // distribution, the loss summed in a fixed order (shuffles of lanes)
      const float* tg = (warp == 0 && A.soft) ? A.soft + (size_t)blk * kCnnModes : nullptr;
      float ce = 0.0f;
      for (int j = lane; j < n_out; j += 32) {
        const float pj = __expf(lg[base + j] - mx) / se;
        const float yj = tg ? tg[j] : (j == label ? 1.0f : 0.0f);
        dlog[base + j] = (pj - yj) * A.inv_batch;
        if (tg) ce += yj * (logf(se) + mx - lg[base + j]);
      }
      if (tg)
        for (int o = 16; o > 0; o >>= 1) ce += __shfl_xor_sync(0xFFFFFFFFu, ce, o);
      if (lane == 0) dlog[kCnnOut + warp] = (tg ? ce : (logf(se) + mx - lg[base + label])) * A.inv_batch;
    } else if (warp == 2) {
#pragma unroll
      for (int j = 0; j < kCnnOut; j++)
        hwt[j] = A.params[(j < kCnnModes ? kOffWi : kOffWs - kCnnModes * 32) + j * 32 + lane];
    } else if (warp >= 8) {
      const float inv = 1.0f / (float)A.maxv;
      uint16_t pv[4];  // the loads first, then the stores
#pragma unroll
      for (int u = 0; u < 4; u++) pv[u] = A.plane[(int64_t)(by + w8 + 8 * u) * A.stride + bx + lane];
#pragma unroll
      for (int u = 0; u < 4; u++)
        xpad[(w8 + 8 * u + 1) * 34 + lane + 1] = (uint32_t)f2bf((float)pv[u] * inv) | 0x3F800000u;
    }
    __syncthreads();
    // the two heads' losses, added in a fixed order (training is deterministic)
    if (t == 0) part[kSlLoss] += dlog[kCnnOut] + dlog[kCnnOut + 1];
    if (warp == 2) {
      float s = 0.0f;
#pragma unroll
      for (int j = 0; j < kCnnOut; j++) s = fmaf(hwt[j], dlog[j], s);
      dgap[lane] = s;
    } else if (warp > 2) {
      const float* gp = A.gap + (size_t)blk * 32;
      const float gv = gp[lane];
      constexpr int kR = (kCnnOut + 12) / 13;  // rows of the head weights per warp
      float* ph = part + kSlHeads;             // both heads' rows, 67 biases between them
      float o[kR];                             // the loads first, then the stores
#pragma unroll
      for (int k = 0; k < kR; k++) {
        const int j = warp - 3 + 13 * k;
        if (j < kCnnOut) o[k] = ph[(j < kCnnModes ? 0 : kCnnModes) + j * 32 + lane];
      }
#pragma unroll
      for (int k = 0; k < kR; k++) {
        const int j = warp - 3 + 13 * k;
        if (j < kCnnOut) ph[(j < kCnnModes ? 0 : kCnnModes) + j * 32 + lane] = o[k] + dlog[j] * gv;
      }
    } else {  // the head biases
      for (int j = t; j < kCnnOut; j += 64)
        part[kSlHeads + (j < kCnnModes ? kOffBi - kOffWi + j : kOffBs - kOffWi + j - kCnnModes)] += dlog[j];
    }
    cnn_load_wait<1>();
    __syncthreads();
    // dZ4 in place of a4 (a4 > 0 passes dgap / 1024): four channels of every
    // 64th pixel, a3 on its way into Q
    {
      const int t8 = t & 255, g = t8 & 3;
      const float* dg = dgap + g * 8 + hw * 4;
      const float d[4] = {dg[0] * (1.0f / 1024.0f), dg[1] * (1.0f / 1024.0f), dg[2] * (1.0f / 1024.0f),
                          dg[3] * (1.0f / 1024.0f)};
      float dbs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
      for (int u = 0; u < 16; u++) {
        const int p = (t8 >> 2) + 64 * u;
        uint2* a = (uint2*)(P + g * kPlane + (((p >> 5) + 1) * kImgW + (p & 31) + 1) * 16 + hw * 8);
        const uint2 av = *a;
        const uint32_t aw[2] = {av.x, av.y};
        uint32_t o[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const float d0 = (aw[k] & 0xFFFFu) && !(aw[k] & 0x8000u) ? d[2 * k] : 0.0f;
          const float d1 = (aw[k] >> 16) && !(aw[k] & 0x80000000u) ? d[2 * k + 1] : 0.0f;
          dbs[2 * k] += d0;
          dbs[2 * k + 1] += d1;
          o[k] = pack_bf2(d0, d1);
        }
        *a = make_uint2(o[0], o[1]);
      }
      // the 64 threads with the same g hold that plane's sums: reduced over
      // the warp's lanes of equal g, then over the warps in a fixed order
#pragma unroll
      for (int k = 0; k < 4; k++) {
        float s2 = dbs[k];
#pragma unroll
        for (int o2 = 4; o2 < 32; o2 <<= 1) s2 += __shfl_xor_sync(0xFFFFFFFFu, s2, o2);
        if (lane < 4) dbp[w8 * 32 + lane * 8 + hw * 4 + k] = s2;
      }
    }
    const int next = cnn_next_block(A, blk + gridDim.x);
    uint8_t* dz = P;  // dZ_l
    uint8_t* act = Q; // a_{l-1}, becomes dZ_{l-1}
#pragma unroll 1
    for (int layer = 4; layer >= 2; layer--) {
      const int li = layer - 2;
      cnn_load_wait<0>();
      fence_async_smem();
      tc_fence_before();
      __syncthreads();
      tc_fence_after();
      if (warp == 2) {
        if (elect_one()) cnn_issue_layer(tmem, smem_u32(dz), smem_u32(Wt) + li * kPackL, mbar, false);
        __syncwarp();
      } else if (layer < 4) {
        cnn_drain_dw<16>(part, tmem + 256, li + 1, warp, lane);
      }
      if (warp == 3) {  // the bias gradient of this layer
        float s = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; w++) s += dbp[w * 32 + lane];
        part[kSlB + li * 32 + lane] += s;
      }
      tc_fence_before();
      __syncthreads();
      tc_fence_after();
      if (warp == 2) {
        if (elect_one()) {
          cnn_issue_dw(tmem + 256, smem_u32(P), smem_u32(Q), act == P);
          umma_commit(mbar);
        }
        __syncwarp();
      }
      ok = __syncthreads_and(mbar_wait(mbar, phase, 1u << 26));
      phase ^= 1;
      tc_fence_after();
      if (!ok) break;
      // the old dZ_l buffer takes a_{l-2}, or the next block's a4
      if (layer > 2)
        cnn_load_act(dz, A.acts, blk, layer - 3);
      else if (next < A.n)
        cnn_load_act(dz, A.acts, next, 3);
      // epilogue: dZ_{l-1} = dA_{l-1} where a_{l-1} > 0, in place of a_{l-1}
      float dbs[16];
#pragma unroll
      for (int c = 0; c < 16; c++) dbs[c] = 0.0f;
      const int q = warp & 3;
#pragma unroll 2
      for (int k = 0; k < 4; k++) {
        const int tile = (w8 >> 2) + 2 * k;
        const int m = 32 * q + lane, j = m >> 3, r = m & 7;
        const int iy = 16 * (tile >> 2) + j, ix = 8 * (tile & 3) + r;
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + tile * 32 + hw * 16, v);
        uint8_t* ap = act + 2 * hw * kPlane + ((iy + 1) * kImgW + ix + 1) * 16;
#pragma unroll
        for (int g = 0; g < 2; g++) {
          const uint4 av = *(const uint4*)(ap + g * kPlane);
          const uint32_t aw[4] = {av.x, av.y, av.z, av.w};
          uint32_t o[4];
#pragma unroll
          for (int k2 = 0; k2 < 4; k2++) {
            const int c = g * 8 + 2 * k2;
            const float d0 = ((aw[k2] & 0xFFFFu) && !(aw[k2] & 0x8000u)) ? v[c] : 0.0f;
            const float d1 = ((aw[k2] >> 16) && !(aw[k2] & 0x80000000u)) ? v[c + 1] : 0.0f;
            dbs[c] += d0;
            dbs[c + 1] += d1;
            o[k2] = pack_bf2(d0, d1);
          }
          *(uint4*)(ap + g * kPlane) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      // a lane ends with channel lane / 2 of its half
      const float s = warp_sum<16>(dbs, lane);
      if (!(lane & 1)) dbp[w8 * 32 + hw * 16 + (lane >> 1)] = s;
      uint8_t* tmp = dz;
      dz = act;
      act = tmp;
    }
    if (!ok) break;
    __syncthreads();
    // layer 1: dW1[co][input][tap] = sum_p dZ1[p][co] in[p + tap] (dZ1 is in
    // dz; the second input is the constant QP plane, zero in the halo). Warp
    // w of the first half takes rows 4w..4w+3, a lane a pair of channels and
    // one of the two input planes, over a sliding 3x3 window in packed fp32;
    // the 8 row groups' sums meet in shared memory and are added in a fixed
    // order. Meanwhile the second half takes layer 2's weight gradient.
    if (hw == 1) {
      cnn_drain_dw<8>(part, tmem + 256, 0, warp - 8, lane);
      if (warp == 11) {
        float s = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; w++) s += dbp[w * 32 + lane];
        part[kSlW1 + kOffB1 + lane] += s;
      }
      tc_fence_before();
    } else {
      const int c2 = lane & 15, in = lane >> 4;
      const uint8_t* zp = dz + (c2 >> 2) * kPlane + (c2 & 3) * 4;
      const uint16_t* xp = (const uint16_t*)xpad + in;
      auto window = [&](int i) {
        const float f = bf2f(xp[2 * i]);
        return f2_pack(f, f);
      };
      uint64_t sx[9];
#pragma unroll
      for (int k = 0; k < 9; k++) sx[k] = 0ull;
#pragma unroll 1
      for (int y = 4 * w8; y < 4 * w8 + 4; y++) {
        uint64_t w[3][3];
#pragma unroll
        for (int dy = 0; dy < 3; dy++)
#pragma unroll
          for (int dx = 0; dx < 2; dx++) w[dy][dx + 1] = window((y + dy) * 34 + dx);
#pragma unroll 8
        for (int x = 0; x < 32; x++) {
#pragma unroll
          for (int dy = 0; dy < 3; dy++) {
            w[dy][0] = w[dy][1];
            w[dy][1] = w[dy][2];
            w[dy][2] = window((y + dy) * 34 + x + 2);
          }
          const uint32_t zz = *(const uint32_t*)(zp + ((y + 1) * kImgW + x + 1) * 16);
          const uint64_t z = f2_pack(__uint_as_float(zz << 16), __uint_as_float(zz & 0xFFFF0000u));
#pragma unroll
          for (int k = 0; k < 9; k++) sx[k] = f2_fma(z, w[k / 3][k % 3], sx[k]);
        }
      }
#pragma unroll
      for (int k = 0; k < 9; k++) {
        const float2 v = f2_unpack(sx[k]);
        red[(w8 * 32 + 2 * c2) * 18 + in * 9 + k] = v.x;
        red[(w8 * 32 + 2 * c2 + 1) * 18 + in * 9 + k] = v.y;
      }
    }
    {
      __syncthreads();
      for (int o = t; o < 32 * 18; o += kCnnBwdThreads) {
        float v = 0.0f;
#pragma unroll
        for (int g = 0; g < 8; g++) v += red[g * 32 * 18 + o];
        part[kSlW1 + o] += (o % 18) < 9 ? v : v * A.qp_in;
      }
    }
    blk = next;
  }
  if (!ok && t == 0) atomicOr(A.status, 1u);
  cnn_load_wait<0>();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kCnnBwdCols);
}

// grads = the sum over the CTA slices in their order, a thread per value of a
// slice (taps 9 of the last tap pair are no values); loss[0] = that of the
// loss slots.
__global__ void k_cnn_reduce(const float* __restrict__ partial, int slices, float* __restrict__ grads,
                             float* __restrict__ loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > kSlLoss) return;
  float* dst;
  if (i < kSlW1) {
    const int l = i / (5 * 2048), r = i % (5 * 2048), lane = r & 31;
    const int tap = 2 * (r / 2048) + (lane >> 4), row = 16 * ((r >> 5) & 1) + (lane & 15), col = (r >> 6) & 31;
    if (tap > 8) return;
    // the rows are the channels of the image at P: dZ in layers 4 and 2, the activation in layer 3
    const int co = l == 1 ? col : row, ci = l == 1 ? row : col;
    dst = grads + cnn_off_w(2 + l) + (co * kCnnCh + ci) * 9 + tap;
  } else if (i < kSlB) {
    dst = grads + i - kSlW1;
  } else if (i < kSlHeads) {
    dst = grads + cnn_off_b(2 + (i - kSlB) / 32) + (i - kSlB) % 32;
  } else if (i < kSlLoss) {
    dst = grads + kOffWi + i - kSlHeads;
  } else {
    dst = loss;
  }
  float s = 0.0f;
#pragma unroll 16
  for (int k = 0; k < slices; k++) s += partial[(size_t)k * kCnnSlice + i];
  *dst = s;
}

// Adam (bias-corrected) on the fp32 parameter vector.
__global__ void k_cnn_adam(float* __restrict__ params, const float* __restrict__ grads, float* __restrict__ m,
                           float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kCnnParams) return;
  const float g = grads[i];
  const float mi = b1 * m[i] + (1.0f - b1) * g, vi = b2 * v[i] + (1.0f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  params[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace vvcg
