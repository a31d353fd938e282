// Parameters of the intra prediction of the 8..12-bit frame path: coding order
// of the units, angular parameters and interpolation taps. Integer arithmetic
// only; each function follows the reference function named beside it
// (crates/rustmpeg-video/src/vvc/predict.rs, slice.rs), bit for bit.
#pragma once
#include "vvcg_device.cuh"
#include "vvcg_tables_dev.cuh"

namespace vvcg {

// 4-tap cubic intra interpolation taps, one packed word per 1/32 position,
// staged in shared memory by the kernels that predict (lane-divergent indices
// would serialise constant-memory reads).
__shared__ uint32_t s_cubic_taps[32];
__device__ __forceinline__ void load_cubic_taps() {
  for (int i = threadIdx.x; i < 32; i += blockDim.x)
    s_cubic_taps[i] = (uint32_t)(uint8_t)c_chroma_taps4[4 * i] | ((uint32_t)(uint8_t)c_chroma_taps4[4 * i + 1] << 8) |
                      ((uint32_t)(uint8_t)c_chroma_taps4[4 * i + 2] << 16) |
                      ((uint32_t)(uint8_t)c_chroma_taps4[4 * i + 3] << 24);
  __syncthreads();
}

// Position of the CU at tb-grid cell (gx, gy) in the coding order of the
// frame path: CTU raster scan, quadtree z-order inside a CTU (slice.rs:164-187).
__device__ __forceinline__ uint32_t cu_order(const DevPic& P, int gx, int gy) {
  int sh = P.ctu_log2 - ilog2(P.tb);
  int cx = gx >> sh, cy = gy >> sh;
  int lx = gx & ((1 << sh) - 1), ly = gy & ((1 << sh) - 1);
  uint32_t z = 0;
  for (int b = 0; b < sh; b++) z |= (((lx >> b) & 1) << (2 * b)) | (((ly >> b) & 1) << (2 * b + 1));
  return ((uint32_t)(cy * P.ctu_w + cx) << (2 * sh)) | z;
}

// AngularParams of predict.rs:1608-1685 (no ISP, no MRL).
struct AngP {
  int pred_mode, angle, abs_inv, scale;
  bool is_ver, ref_filter, interp, pdpc;
};
__device__ __forceinline__ AngP angular_params(int dir, int w, int h, bool is_luma) {
  AngP p;
  int mode = dir;
  // predict.rs:1405-1422 get_modified_wide_angle
  if (dir > 1 && dir <= 66) {
    int delta = abs(floor_log2(w) - floor_log2(h));
    if (delta < 6) {
      const int shifts[6] = {0, 6, 10, 12, 14, 15};
      int s = shifts[delta];
      if (w > h && dir < 2 + s)
        mode = dir + 65;
      else if (h > w && dir > 66 - s)
        mode = dir - 65;
    }
  }
  p.pred_mode = mode;
  p.is_ver = mode >= 34;
  p.pdpc = w >= 4 && h >= 4;
  int am = p.is_ver ? mode - 50 : -(mode - 18);
  int absm = min(31, abs(am));
  int abs_ang = c_ang_table[absm];
  p.abs_inv = c_inv_ang_table[absm];
  p.angle = (am < 0 ? -1 : 1) * abs_ang;
  p.scale = 0;
  if (am < 0) {
    p.pdpc = false;
  } else if (am > 0) {
    int side = p.is_ver ? h : w;
    int inv_term = floor_log2((unsigned)max(1, 3 * p.abs_inv - 2)) - 8;
    p.scale = min(2, floor_log2((unsigned)side) - inv_term);
    if (p.scale < 0) p.pdpc = false;
  }
  p.ref_filter = false;
  p.interp = false;
  if (is_luma && dir != 1 && dir != 0) {
    int diff = min(abs(mode - 18), abs(mode - 50));
    int l2 = (floor_log2(w) + floor_log2(h)) >> 1;
    if (diff > c_intra_filter_thr[min(7, l2)]) {
      bool integer = (abs_ang & 0x1F) == 0;
      p.ref_filter = integer;
      p.interp = !integer;
    }
  }
  return p;
}


__device__ __forceinline__ int ldp(const uint16_t* p) { return __ldcg(p); }

}  // namespace vvcg
