// P pictures of the multi-tool stream on the GPU (vvcg_decode_p_batch) and
// the context's picture buffer (vvcg_dpb_*). Included at the end of vvcg.cu.
//
// decode_inter_picture (slice.rs:3677-3834) reconstructs every CTU as one
// coding unit: the inter prediction of its motion (predict_inter_pu,
// inter.rs:1734: 8-bit uni-prediction with the luma 8-tap / chroma 4-tap
// filters of interpolate_luma_block :896 and interpolate_chroma_block_420
// :1056, reference reads clamped to the picture), each component's residual
// (reconstruct_component_full, slice.rs:1920: DCT-2 or transform skip,
// regular or dependent dequantisation) and the clipped sum. Every CTU of a
// picture depends only on the reference pictures, so one CTA per CTU runs
// them all at once: the TU path's warp_tu_inverse turns the levels into
// residuals and the interpolation's tiles (mc.cuh) predict into shared memory;
// all four warps then store the clipped sums
// into the picture's buffer slot. apply_inter_loop_filters'
// CTU-boundary deblocking (slice.rs:2291) follows for pictures that enable
// it. Pictures are grouped into levels by their slots (a picture waits for
// the pictures before it that write a slot it reads or writes, or read the
// slot it writes); one launch runs a level.

namespace vvcg {

constexpr int kPWarps = 4;

struct PPicDev {
  const vvcg_inter_cu* cus;
  uint16_t* out[3];
  const uint16_t* ref[4][3];
  int32_t stride[3];
  int32_t w, h, gw, gh, lqp, cqp, num_refs;
  uint32_t flags;  // bit0 dependent quantisation, bit1 sparse levels
};

// A component's reference plane and the unit's filter for it (the 8-bit
// functions' rounding on 16-bit planes).
template <bool kLuma>
__device__ __forceinline__ McParams p_params(const PPicDev& P, const vvcg_inter_cu& rec, int comp) {
  return McParams{P.ref[min((int)rec.ref_idx[0], P.num_refs - 1)][comp], nullptr, kLuma ? P.w : P.w / 2,
                  kLuma ? P.h : P.h / 2, P.stride[comp], 8, kLuma ? 0 : 1};
}
template <bool kLuma>
__device__ __forceinline__ McFilter p_filter(const McParams& Pm, const vvcg_inter_cu& rec) {
  vvcg_mc_block B;
  B.mv_x = rec.mv[0][0];
  B.mv_y = rec.mv[0][1];
  B.flags = kLuma && (rec.flags & VVCG_INTER_CU_ALT_HPEL) ? VVCG_MC_ALT_HPEL : 0;
  return mc_filter<true>(Pm, B);
}

// A prediction tile whose reference window holds samples above 8 bits (a
// picture-buffer upload does not reject them), one output at a time with the
// 16-bit window and intermediate the filters then wrap in.
template <bool kLuma>
__device__ __noinline__ void p_tile_wide(const PPicDev* pic, const vvcg_inter_cu* unit, int comp, int bx, int by,
                                         int16_t* o) {
  constexpr int tw = kLuma ? 32 : 16, ntap = kLuma ? 8 : 4, half = ntap / 2 - 1;
  const int lane = threadIdx.x & 31;
  const McParams Pm = p_params<kLuma>(*pic, *unit, comp);
  const McFilter F = p_filter<kLuma>(Pm, *unit);
  const int wx0 = bx + F.dx - half, wy0 = by + F.dy - half;
  auto at = [&](int x, int y) -> int {
    return (int16_t)Pm.ref[(size_t)clampi(wy0 + y, 0, Pm.h - 1) * Pm.stride + clampi(wx0 + x, 0, Pm.w - 1)];
  };
  for (int i = lane; i < tw * 16; i += 32) {
    const int x = i % tw, y = i / tw;
    int s = 0;
    if (F.fx == 0 && F.fy == 0) {
      s = at(x + half, y + half);
    } else if (F.fy == 0) {
      for (int k = 0; k < ntap; k++) s += mc_tap(F.th0, F.th1, k) * at(x + k, y + half);
      s = clampi((s + 32) >> 6, 0, 255);
    } else if (F.fx == 0) {
      for (int k = 0; k < ntap; k++) s += mc_tap(F.tv0, F.tv1, k) * at(x + half, y + k);
      s = clampi((s + 32) >> 6, 0, 255);
    } else {
      for (int j = 0; j < ntap; j++) {
        int t = 0;
        for (int k = 0; k < ntap; k++) t += mc_tap(F.th0, F.th1, k) * at(x + k, y + j);
        s += mc_tap(F.tv0, F.tv1, j) * (int16_t)t;
      }
      s = clampi((s + 2048) >> 12, 0, 255);
    }
    o[y * tw + x] = (int16_t)s;
  }
}

// The inter prediction of one 16-row tile (luma 32x16, chroma 16x16) of a
// coding unit by one warp, raster into `pred`. (bx, by): the tile's position in
// the component's plane.
template <bool kLuma>
__device__ __forceinline__ void p_predict_tile(const PPicDev& P, const vvcg_inter_cu& rec, int cu, int comp, int bx,
                                               int by, int16_t* pred, McWs& S, int lane) {
  constexpr int tw = kLuma ? 32 : 16, ntap = kLuma ? 8 : 4, half = ntap / 2 - 1;
  if (!((rec.inter_dir & 1) && rec.ref_idx[0] >= 0)) {  // predict_inter_pu without a usable list: 128
    for (int i = lane; i < tw * 8; i += 32) reinterpret_cast<uint32_t*>(pred)[i] = 128u | 128u << 16;
    return;
  }
  const McParams Pm = p_params<kLuma>(P, rec, comp);
  const McFilter F = p_filter<kLuma>(Pm, rec);
  if (!mc_tile<ntap, false>(Pm, F, bx + F.dx - half, by + F.dy - half, tw, 16, pred, tw, S, lane))
    p_tile_wide<kLuma>(&P, &P.cus[cu], comp, bx, by, pred);
}

// clip(prediction + residual) to 8 bits of a pair of 16-bit numbers, in 32
// bits: whole-sample motion copies reference samples above 8 bits as they
// are, outside the range in which add_clip2 is exact.
__device__ __forceinline__ uint32_t p_add_wide2(uint32_t pred, uint32_t res) {
  const int lo = (int)(int16_t)pred + (int)(int16_t)res, hi = ((int)pred >> 16) + ((int)res >> 16);
  return (uint32_t)clampi(lo, 0, 255) | (uint32_t)clampi(hi, 0, 255) << 16;
}

// Grid: (CTUs of the largest picture of the level, pictures of the level).
// The unit's work is cut into near-equal parts: warp 0 turns the luma levels
// into the residual, warps 1 and 2 a chroma component's and then predict half
// of the luma, warp 3 predicts Cb and Cr; then all four add, clip and store.
// Which warp is which rotates with the unit, because a warp's place decides
// its scheduler: fixed, 298 us for eight 1920x1088 pictures; rotated, 265; with
// sparse levels read straight into the transform tile, 218 (27 us a picture).
// Before the 16-bit transforms and packed filters it took 644 us. What bounds it
// now is instruction fetch and the wait for the slowest part.
__global__ void __launch_bounds__(kPWarps * 32, 8)
k_p_cu(const PPicDev* __restrict__ pics, const int16_t* __restrict__ levels, uint64_t n_levels, uint32_t* status) {
  constexpr int kWs = sizeof(McWs) > tu_inv_ws(256) * 2 ? sizeof(McWs) : tu_inv_ws(256) * 2;
  __shared__ __align__(16) int16_t ws_luma[tu_inv_ws(1024)];
  __shared__ __align__(16) unsigned char ws[3][kWs];  // warps 1..3: transform tiles, then prediction window
  __shared__ __align__(16) int16_t res[1024 + 2 * 256];
  __shared__ __align__(16) int16_t pred[1024 + 2 * 256];
  const PPicDev& P = pics[blockIdx.y];
  const int cu = blockIdx.x;
  if (cu >= P.gw * P.gh) return;
  const vvcg_inter_cu rec = P.cus[cu];
  const int bx = (cu % P.gw) * 32, by = (cu / P.gw) * 32;
  const int lane = threadIdx.x & 31, wid = ((threadIdx.x >> 5) + cu) & 3;
  if (wid < 3) {
    const int c = wid, n = c ? 256 : 1024, off_res = c == 0 ? 0 : (c == 1 ? 1024 : 1280);
    int16_t* r = res + off_res;
    bool coded = (rec.cbf >> c) & 1;
    if (coded) {
      const int off = rec.level_off[c];
      bool ok = off >= 0 && !(rec.tu_tools >> 3);
      int cnt = -1;
      if (ok && (P.flags & 2)) {  // sparse: count, unused word, (index, level) pairs
        cnt = (off & 1) || (uint64_t)off + 2 > n_levels ? -1 : levels[off];
        ok = cnt >= 0 && cnt <= n && (uint64_t)off + 2 + 2 * (uint64_t)cnt <= n_levels;
      } else if (ok) {
        ok = (uint64_t)off + (uint64_t)n <= n_levels;
      }
      if (!ok) {
        if (lane == 0) atomicOr(status, kStatusBadRecord);
        coded = false;
      } else {
        const bool ts = (rec.tu_tools >> c) & 1;
        const int q = c ? P.cqp : P.lqp;
        vvcg_tu_rec t;
        t.log2_w = t.log2_h = (uint8_t)(c ? 4 : 5);
        t.bit_depth = 8;
        t.qp = (uint8_t)(ts ? max(4, q) : q);
        t.flags = ts ? VVCG_TU_TRANSFORM_SKIP : ((P.flags & 1) ? VVCG_TU_DEP_QUANT : 0);
        t.mts_idx = t.lfnst_idx = t.lfnst_mode = 0;
        t.in_off = t.out_off = 0;
        if (!warp_tu_inverse(t, levels + off + (cnt >= 0 ? 2 : 0), r,
                             c ? reinterpret_cast<int16_t*>(ws[c - 1]) : ws_luma, lane, 0, cnt) &&
            lane == 0)
          atomicOr(status, kStatusBadRecord);
      }
    }
    if (!coded)
      for (int i = lane; i < n / 2; i += 32) reinterpret_cast<uint32_t*>(r)[i] = 0;
    __syncwarp();
  }
  if (wid >= 1) {
    McWs& S = *reinterpret_cast<McWs*>(ws[wid - 1]);
    if (wid < 3) {
      p_predict_tile<true>(P, rec, cu, 0, bx, by + 16 * (wid - 1), pred + 512 * (wid - 1), S, lane);
    } else {
#pragma unroll 1
      for (int c = 1; c <= 2; c++) {
        p_predict_tile<false>(P, rec, cu, c, bx / 2, by / 2, pred + 768 + 256 * c, S, lane);
        __syncwarp();
      }
    }
  }
  __syncthreads();
  // reconstruction: clip(prediction + residual), eight samples a step
  for (int r = threadIdx.x; r < (1024 + 512) / 8; r += blockDim.x) {
    const int comp = r < 128 ? 0 : (r < 160 ? 1 : 2);
    const int k = comp == 0 ? r : (comp == 1 ? r - 128 : r - 160);
    const int x = comp ? 8 * (k & 1) : 8 * (k & 3), y = comp ? k >> 1 : k >> 2;
    const uint4 p = *reinterpret_cast<const uint4*>(&pred[8 * r]), d = *reinterpret_cast<const uint4*>(&res[8 * r]);
    uint16_t* const at = P.out[comp] + (size_t)((comp ? by / 2 : by) + y) * P.stride[comp] + (comp ? bx / 2 : bx) + x;
    constexpr uint32_t top = 0x00FF00FFu;
    const bool wide = ((p.x | p.y | p.z | p.w) & ~top) != 0;
    *reinterpret_cast<uint4*>(at) =
        wide ? make_uint4(p_add_wide2(p.x, d.x), p_add_wide2(p.y, d.y), p_add_wide2(p.z, d.z), p_add_wide2(p.w, d.w))
             : make_uint4(add_clip2(p.x, d.x, top), add_clip2(p.y, d.y, top), add_clip2(p.z, d.z, top),
                          add_clip2(p.w, d.w, top));
  }
}

// The CTU-boundary deblocking's cells: each CTU's own L0 motion and cbfs
// (slice.rs:2319-2326, :2438-2444), one thread per record.
__global__ void k_p_cells(const vvcg_inter_cu* __restrict__ cus, uint32_t n, vvcg_ctu_motion* __restrict__ cells) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const vvcg_inter_cu& r = cus[i];
  vvcg_ctu_motion m;
  for (int j = 0; j < 3; j++) {
    m.mv[j][0] = r.mv[0][0];
    m.mv[j][1] = r.mv[0][1];
    m.ref[j] = r.ref_idx[0];
    m.reserved[j] = 0;
  }
  m.cbf = r.cbf & 7;
  cells[i] = m;
}

}  // namespace vvcg

// ---------------------------------------------------------------------------
// Picture buffer and P-picture state of a context.
// ---------------------------------------------------------------------------
struct PState {
  uint32_t slots = 0, w = 0, h = 0, stride[3] = {0, 0, 0};
  uint64_t slot_samples = 0;
  DevBuf arena, d_cus, d_levels, d_cells, d_pics, d_status;
  uint16_t* plane(uint32_t slot, int comp) const {
    uint16_t* base = (uint16_t*)arena.p + slot * slot_samples;
    if (comp == 0) return base;
    return base + (uint64_t)stride[0] * h + (comp == 2 ? (uint64_t)stride[1] * (h / 2) : 0);
  }
};

void p_state_free(PState* s) {
  if (!s) return;
  for (DevBuf* b : {&s->arena, &s->d_cus, &s->d_levels, &s->d_cells, &s->d_pics, &s->d_status}) b->release();
  delete s;
}

static_assert(sizeof(vvcg_inter_cu) == 48, "inter CU layout");
static_assert(sizeof(vvcg_p_pic) == 36, "P picture layout");

extern "C" vvcg_status vvcg_dpb_reserve(vvcg_ctx* ctx, uint32_t slots, uint32_t width, uint32_t height) {
  if (!ctx) return VVCG_INVALID_INPUT;
  if (!slots || slots > 1024 || !width || !height || (width & 1) || (height & 1))
    return fail(ctx, VVCG_INVALID_INPUT, "picture buffer: 1..1024 slots of a nonzero even size");
  if ((uint64_t)width * height > kMaxLumaSamples) return fail(ctx, VVCG_LIMIT_EXCEEDED, "picture too large");
  CK(cudaSetDevice(ctx->device), "cudaSetDevice");
  CK(cudaStreamSynchronize(ctx->stream), "sync");
  if (!ctx->p) ctx->p = new PState();
  PState& s = *ctx->p;
  s.w = width;
  s.h = height;
  s.stride[0] = (width + 63) & ~63u;
  s.stride[1] = s.stride[2] = ((width / 2) + 63) & ~63u;
  s.slot_samples = (uint64_t)s.stride[0] * height + 2ull * s.stride[1] * (height / 2);
  s.slots = 0;
  CK(s.arena.reserve(slots * s.slot_samples * sizeof(uint16_t)), "cudaMalloc");
  s.slots = slots;
  return VVCG_OK;
}

extern "C" vvcg_status vvcg_dpb_plane(vvcg_ctx* ctx, uint32_t slot, uint32_t comp, void** dev_ptr, uint32_t* stride) {
  if (!ctx || !dev_ptr || !ctx->p || slot >= ctx->p->slots || comp > 2) return VVCG_INVALID_INPUT;
  *dev_ptr = ctx->p->plane(slot, (int)comp);
  if (stride) *stride = ctx->p->stride[comp];
  return VVCG_OK;
}

extern "C" vvcg_status vvcg_dpb_store(vvcg_ctx* ctx, uint32_t pic, uint32_t slot) {
  if (!ctx) return VVCG_INVALID_INPUT;
  if (!ctx->p || slot >= ctx->p->slots) return fail(ctx, VVCG_INVALID_INPUT, "no such picture-buffer slot");
  if (!ctx->prepared || pic >= ctx->num_pics) return fail(ctx, VVCG_INVALID_INPUT, "no such batch picture");
  const PicLayout& L = ctx->layout[pic];
  const DevPic& D = ctx->pics[pic];
  PState& s = *ctx->p;
  if (D.bd != 8 || D.cf != 1 || (uint32_t)L.pw[0] != s.w || (uint32_t)L.ph[0] != s.h)
    return fail(ctx, VVCG_INVALID_INPUT, "batch picture %u is not an 8-bit 4:2:0 picture of the buffer's size", pic);
  CK(cudaSetDevice(ctx->device), "cudaSetDevice");
  for (int c = 0; c < 3; c++) {
    void* src = nullptr;
    uint32_t sstride = 0;
    vvcg_batch_plane(ctx, pic, (uint32_t)c, &src, &sstride);
    CK(cudaMemcpy2DAsync(s.plane(slot, c), s.stride[c] * 2, src, (size_t)sstride * 2, (size_t)L.pw[c] * 2, L.ph[c],
                         cudaMemcpyDeviceToDevice, ctx->stream),
       "copy");
  }
  return VVCG_OK;
}

static vvcg_status dpb_copy(vvcg_ctx* ctx, uint32_t slot, const void* const* ptr, const uint32_t* strides, bool in) {
  if (!ctx) return VVCG_INVALID_INPUT;
  if (!ctx->p || slot >= ctx->p->slots) return fail(ctx, VVCG_INVALID_INPUT, "no such picture-buffer slot");
  PState& s = *ctx->p;
  for (int c = 0; c < 3; c++)
    if (!ptr[c] || strides[c] < (c ? s.w / 2 : s.w)) return fail(ctx, VVCG_INVALID_INPUT, "plane %d", c);
  CK(cudaSetDevice(ctx->device), "cudaSetDevice");
  for (int c = 0; c < 3; c++) {
    const uint32_t pw = c ? s.w / 2 : s.w, ph = c ? s.h / 2 : s.h;
    if (in)
      CK(cudaMemcpy2DAsync(s.plane(slot, c), s.stride[c] * 2, ptr[c], (size_t)strides[c] * 2, (size_t)pw * 2, ph,
                           cudaMemcpyDefault, ctx->stream),
         "upload");
    else
      CK(cudaMemcpy2DAsync(const_cast<void*>(ptr[c]), (size_t)strides[c] * 2, s.plane(slot, c), s.stride[c] * 2,
                           (size_t)pw * 2, ph, cudaMemcpyDefault, ctx->stream),
         "download");
  }
  CK(cudaStreamSynchronize(ctx->stream), "sync");
  return VVCG_OK;
}

extern "C" vvcg_status vvcg_dpb_upload(vvcg_ctx* ctx, uint32_t slot, const vvcg_plane_in planes[3]) {
  if (!ctx || !planes) return VVCG_INVALID_INPUT;
  const void* p[3] = {planes[0].data, planes[1].data, planes[2].data};
  const uint32_t st[3] = {planes[0].stride, planes[1].stride, planes[2].stride};
  return dpb_copy(ctx, slot, p, st, true);
}

extern "C" vvcg_status vvcg_dpb_download(vvcg_ctx* ctx, uint32_t slot, const vvcg_plane_out planes[3]) {
  if (!ctx || !planes) return VVCG_INVALID_INPUT;
  const void* p[3] = {planes[0].data, planes[1].data, planes[2].data};
  const uint32_t st[3] = {planes[0].stride, planes[1].stride, planes[2].stride};
  return dpb_copy(ctx, slot, p, st, false);
}

extern "C" vvcg_status vvcg_decode_p_batch(vvcg_ctx* ctx, const vvcg_p_pic* pics, uint32_t num_pics,
                                           const vvcg_inter_cu* cus, uint32_t num_cus, const int16_t* levels,
                                           uint64_t num_levels) {
  if (!ctx) return VVCG_INVALID_INPUT;
  if (!num_pics) return VVCG_OK;
  if (!pics || !cus || (!levels && num_levels)) return fail(ctx, VVCG_INVALID_INPUT, "missing arguments");
  if (num_pics > 65535) return fail(ctx, VVCG_LIMIT_EXCEEDED, "more than 65535 pictures in one call");
  if (!ctx->p || !ctx->p->slots) return fail(ctx, VVCG_INVALID_INPUT, "no picture buffer (vvcg_dpb_reserve)");
  PState& s = *ctx->p;
  const uint32_t gw = s.w / 32, gh = s.h / 32;
  if (s.w % 32 || s.h % 32) return fail(ctx, VVCG_INVALID_INPUT, "picture buffer size is not a multiple of 32");
  // validation of pictures and records, and the dependency level of each picture
  std::vector<int> level(num_pics, 0);
  int num_levels_dep = 0;
  for (uint32_t i = 0; i < num_pics; i++) {
    const vvcg_p_pic& p = pics[i];
    if (p.width != s.w || p.height != s.h) return fail(ctx, VVCG_INVALID_INPUT, "picture %u: size", i);
    if (p.qp > 63 || (p.options & ~(uint32_t)(VVCG_SLICE_DEP_QUANT | VVCG_SLICE_DEBLOCK | VVCG_SLICE_SIGN_HIDING)))
      return fail(ctx, VVCG_INVALID_INPUT, "picture %u: QP or options", i);
    if (p.num_refs < 1 || p.num_refs > 4 || p.out_slot < 0 || (uint32_t)p.out_slot >= s.slots)
      return fail(ctx, VVCG_INVALID_INPUT, "picture %u: reference count or output slot", i);
    for (int r = 0; r < p.num_refs; r++)
      if (p.ref_slot[r] < 0 || (uint32_t)p.ref_slot[r] >= s.slots || p.ref_slot[r] == p.out_slot)
        return fail(ctx, VVCG_INVALID_INPUT, "picture %u: reference slot %d", i, r);
    if ((uint64_t)p.cu_offset + (uint64_t)gw * gh > num_cus)
      return fail(ctx, VVCG_INVALID_INPUT, "picture %u: records past the array", i);
    for (uint32_t k = 0; k < gw * gh; k++) {
      const vvcg_inter_cu& r = cus[p.cu_offset + k];
      if (r.tu_tools >> 3 || (r.cbf >> 3)) return fail(ctx, VVCG_INVALID_INPUT, "picture %u CU %u: flags", i, k);
      for (int c = 0; c < 3; c++)
        if (((r.cbf >> c) & 1) &&
            (r.level_off[c] < 0 ||
             !tb_level_extent(levels, num_levels, (uint64_t)r.level_off[c], c ? 256 : 1024, p.sparse != 0)))
          return fail(ctx, VVCG_INVALID_INPUT, "picture %u CU %u: levels of component %d", i, k, c);
    }
    auto reads = [&](const vvcg_p_pic& q, int32_t slot) {
      for (int r = 0; r < q.num_refs; r++)
        if (q.ref_slot[r] == slot) return true;
      return false;
    };
    for (uint32_t j = 0; j < i; j++)
      if (reads(p, pics[j].out_slot) || pics[j].out_slot == p.out_slot || reads(pics[j], p.out_slot))
        level[i] = std::max(level[i], level[j] + 1);
    num_levels_dep = std::max(num_levels_dep, level[i] + 1);
  }
  CK(cudaSetDevice(ctx->device), "cudaSetDevice");
  // uploads: records, levels, deblocking cells, the per-picture descriptors
  const uint64_t ncu = (uint64_t)num_cus;
  CK(s.d_cus.reserve(ncu * sizeof(vvcg_inter_cu)), "cudaMalloc");
  CK(s.d_levels.reserve(std::max<uint64_t>(num_levels, 1) * sizeof(int16_t)), "cudaMalloc");
  CK(s.d_cells.reserve(ncu * sizeof(vvcg_ctu_motion)), "cudaMalloc");
  CK(s.d_pics.reserve(num_pics * sizeof(vvcg::PPicDev)), "cudaMalloc");
  CK(s.d_status.reserve(sizeof(uint32_t)), "cudaMalloc");
  CK(cudaMemcpyAsync(s.d_cus.p, cus, ncu * sizeof(vvcg_inter_cu), cudaMemcpyHostToDevice, ctx->stream), "upload");
  if (num_levels)
    CK(cudaMemcpyAsync(s.d_levels.p, levels, num_levels * sizeof(int16_t), cudaMemcpyHostToDevice, ctx->stream),
       "upload");
  CK(cudaMemsetAsync(s.d_status.p, 0, sizeof(uint32_t), ctx->stream), "memset");
  std::vector<std::vector<vvcg::PPicDev>> by_level(num_levels_dep);
  for (uint32_t i = 0; i < num_pics; i++) {
    const vvcg_p_pic& p = pics[i];
    vvcg::PPicDev d{};
    d.cus = (const vvcg_inter_cu*)s.d_cus.p + p.cu_offset;
    for (int c = 0; c < 3; c++) {
      d.out[c] = s.plane((uint32_t)p.out_slot, c);
      d.stride[c] = (int32_t)s.stride[c];
      for (int r = 0; r < 4; r++) d.ref[r][c] = s.plane((uint32_t)p.ref_slot[std::min(r, p.num_refs - 1)], c);
    }
    d.w = (int32_t)s.w;
    d.h = (int32_t)s.h;
    d.gw = (int32_t)gw;
    d.gh = (int32_t)gh;
    // slice.rs:3568-3569: max(SliceQpY, 4) and max(derived_chroma_qp, 4) (hls.rs:778)
    d.lqp = std::max<int>(p.qp, 4);
    d.cqp = std::max(4, p.qp <= 26 ? (int)p.qp : (int)p.qp - 1);
    d.num_refs = p.num_refs;
    d.flags = ((p.options & VVCG_SLICE_DEP_QUANT) ? 1u : 0u) | (p.sparse ? 2u : 0u);
    by_level[level[i]].push_back(d);
  }
  std::vector<vvcg::PPicDev> flat;
  std::vector<size_t> start;
  for (auto& L : by_level) {
    start.push_back(flat.size());
    flat.insert(flat.end(), L.begin(), L.end());
  }
  CK(cudaMemcpyAsync(s.d_pics.p, flat.data(), flat.size() * sizeof(vvcg::PPicDev), cudaMemcpyHostToDevice,
                     ctx->stream),
     "upload");
  // deblocking passes of the pictures that enable it, level by level: luma V,
  // chroma V, luma H, chroma H; the cells of all records
  std::vector<DbfPass>& passes = ctx->dbf_ctu;
  passes.clear();
  struct LevelPasses {
    size_t at[4];
    uint32_t pics;
  };
  std::vector<LevelPasses> dbf(num_levels_dep, LevelPasses{{0, 0, 0, 0}, 0});
  for (int L = 0; L < num_levels_dep; L++) {
    std::vector<DbfPass> kind[4];
    for (uint32_t i = 0; i < num_pics; i++) {
      if (level[i] != L || !(pics[i].options & VVCG_SLICE_DEBLOCK)) continue;
      uint16_t* planes[3] = {s.plane((uint32_t)pics[i].out_slot, 0), s.plane((uint32_t)pics[i].out_slot, 1),
                             s.plane((uint32_t)pics[i].out_slot, 2)};
      DbfPass six[6];
      ctu_edge_passes(planes, s.stride, s.w, s.h, 32, pics[i].qp,
                      (const vvcg_ctu_motion*)s.d_cells.p + pics[i].cu_offset, six);
      kind[0].push_back(six[0]);
      kind[1].insert(kind[1].end(), six + 1, six + 3);
      kind[2].push_back(six[3]);
      kind[3].insert(kind[3].end(), six + 4, six + 6);
      dbf[L].pics++;
    }
    for (int k = 0; k < 4; k++) {
      dbf[L].at[k] = passes.size();
      passes.insert(passes.end(), kind[k].begin(), kind[k].end());
    }
  }
  if (!passes.empty()) {
    CK(ctx->d_dbf_ctu.reserve(sizeof(DbfPass) * passes.size()), "cudaMalloc");
    CK(cudaMemcpyAsync(ctx->d_dbf_ctu.p, passes.data(), sizeof(DbfPass) * passes.size(), cudaMemcpyHostToDevice,
                       ctx->stream),
       "upload");
    vvcg::k_p_cells<<<(num_cus + 255) / 256, 256, 0, ctx->stream>>>((const vvcg_inter_cu*)s.d_cus.p, num_cus,
                                                                     (vvcg_ctu_motion*)s.d_cells.p);
    CK(cudaGetLastError(), "cells launch");
    ctx->launches++;
  }
  const vvcg::PPicDev* dp = (const vvcg::PPicDev*)s.d_pics.p;
  for (int L = 0; L < num_levels_dep; L++) {
    vvcg::k_p_cu<<<dim3(gw * gh, (unsigned)by_level[L].size()), vvcg::kPWarps * 32, 0, ctx->stream>>>(
        dp + start[L], (const int16_t*)s.d_levels.p, num_levels, (uint32_t*)s.d_status.p);
    ctx->launches++;
    CK(cudaGetLastError(), "P-picture launch");
    if (dbf[L].pics) {
      const DbfPass* d = (const DbfPass*)ctx->d_dbf_ctu.p;
      const vvcg_status st = launch_ctu_edges(ctx, d + dbf[L].at[0], d + dbf[L].at[1], d + dbf[L].at[2],
                                              d + dbf[L].at[3], &passes[dbf[L].at[0]], &passes[dbf[L].at[1]],
                                              &passes[dbf[L].at[2]], &passes[dbf[L].at[3]], dbf[L].pics);
      if (st != VVCG_OK) return st;
    }
  }
  uint32_t status = 0;
  CK(cudaMemcpyAsync(&status, s.d_status.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream), "status");
  CK(cudaStreamSynchronize(ctx->stream), "sync");
  if (status) return fail(ctx, VVCG_INVALID_INPUT, "malformed records or levels (status 0x%x)", status);
  return VVCG_OK;
}
