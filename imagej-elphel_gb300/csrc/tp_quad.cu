// tp_quad.cu -- the forward of standard quads (4 sensors, the six pairs of Correlation2d.PAIRS, mono or
// Bayer, all images of one type): the shape of nearly every scene, so it has its own kernels.
//
// A warp carries a tile through all stages, as in the general warp-per-tile schedule, with three
// differences: the image windows are staged in shared memory one item ahead (tp_forward.cuh), the
// six pairs are taken together two values per instruction (tp_pairs.cuh), and the extraction's serial
// half runs as a pass of its own (extract_kernel).  u16 Bayer tiles with short strips are shared by three warps
// (quad3_kernel).
//
// Measured (kernel and extraction together, general schedule -> now): 4x2592x1936 u16 Bayer with kernel
// tables, 78,408 tiles: 0.922 -> 0.756 ms; 4x1304x984 float Bayer, 7,018 tiles: 129 -> 80 us; 16 batched
// 4x512x384 float mono scenes, 49,152 tiles: 452 -> 316 us.  What bounds it now: latency at 16 warps
// an SM (128 registers a thread).  Issue slots and shared-memory pipe in use: 41 and 36 % at 3,072 mono tiles, 51
// and 47 % at 7,018 float Bayer tiles, 51 and 59 % over the 16 batched scenes.
//
// Shared memory of a warp (floats): CLT [C][4 sensors][QP_CLT] first; the windows of colour item c at
// 4 QP_CLT c (where that item's CLT goes once they are read); the pairs' spectra over the CLT
// (QP_SURF floats), then the surfaces; transpose buffers behind the CLT.
#include "tp_forward.cuh"
#include "tp_pairs.cuh"
#include "tp_launch.h"

namespace {

__host__ __device__ constexpr int quad_warp_floats(int C) { return C == 3 ? 12 * QP_CLT + SCR : QP_FLOATS; }
__host__ __device__ constexpr int quad_tbuf(int C) { return C == 3 ? 12 * QP_CLT : 4 * Stage<false>::WIN; }

__device__ __forceinline__ SubtilePlan quad_plan(const SceneDev &sc, int C, int task, int s, int c) {
  return sc.plan[((size_t)task * 4 + s) * C + c];
}

// lane q * 8 + r copies its share of sensor q's window of colour item c
template <bool U16>
__device__ __forceinline__ void quad_stage(const SceneDev &sc, const SubtilePlan &p, int c, float *ws, int q, int r) {
  stage_window<U16>(sc, sc.images[q], p.tlx, p.tly, ws + c * 4 * QP_CLT + q * Stage<U16>::WIN, r);
  cp_async_commit();
}

// phase A of a tile: p is the plan of (sensor q, colour 0), whose windows are staged
template <int C, bool U16>
__device__ __forceinline__ void quad_clt(const SceneDev &sc, int task, SubtilePlan p, float *ws, int lane) {
  const int q = lane >> 3, r = lane & 7;
  const int rr = sc.bayer_red_row, rc = sc.bayer_red_col;
  float *tbuf = ws + quad_tbuf(C) + q * 72;
#pragma unroll 1
  for (int c = 0; c < C; c++) {
    const SubtilePlan pn = (c + 1 < C) ? quad_plan(sc, C, task, q, c + 1) : p;
    SWin<U16> w;
    w.base = (const typename Stage<U16>::T *)(ws + c * 4 * QP_CLT + q * Stage<U16>::WIN);
    w.sx = p.tlx & (Stage<U16>::CH - 1);
    w.scale = sc.color_scale[c];
    cp_async_wait_all();  // this item's windows, copied by every lane
    __syncwarp();
    float o[4][8];
    if (C == 1) {
      subtile_clt<0>(w, p.rx, p.ry, 0, 0, 0, r, tbuf, o);
    } else if (c < 2) {
      const int pc = ((c == 0 ? rc : 1 - rc) - p.tlx) & 1, pr = ((c == 0 ? rr : 1 - rr) - p.tly) & 1;
      subtile_clt<1>(w, p.rx, p.ry, pc, pr, 0, r, tbuf, o);
    } else {
      const int pg = (p.tlx + p.tly + rc + rr + 1) & 1;
      subtile_clt<2>(w, p.rx, p.ry, 0, 0, pg, r, tbuf, o);
    }
    // every lane has read this item's windows (the transposes in subtile_clt synchronise the warp)
    if (c + 1 < C) quad_stage<U16>(sc, pn, c + 1, ws, q, r);
    const float *kp = (p.kidx >= 0) ? sc.kernels[q] + (size_t)p.kidx * TP_CLT : nullptr;
    conv_shift(o, kp, p.rx, p.ry, r);
    float *sdst = ws + (c * 4 + q) * QP_CLT + r * 8 + (r & 4) * ((QP_HALF - 32) / 4);
#pragma unroll
    for (int m = 0; m < 4; m++) {
      *(float4 *)(sdst + m * QP_QUAD) = make_float4(o[m][0], o[m][1], o[m][2], o[m][3]);
      *(float4 *)(sdst + m * QP_QUAD + 4) = make_float4(o[m][4], o[m][5], o[m][6], o[m][7]);
    }
    p = pn;
  }
  __syncwarp();
}

// the products the extraction pass starts from
template <int NT>
__device__ __forceinline__ void store_products(const SceneDev &sc, size_t task, int RE, int lane, const float cmb[8],
                                               const float oprod[8]) {
#pragma unroll
  for (int t = 0; t < NT; t++) {
    const int e = lane + 32 * t;
    if (e < RE) sc.sprod[task * RE + e] = cmb[t];
  }
  float4 *ob = (float4 *)(sc.osum + (task * 32 + lane) * 8);
  ob[0] = make_float4(oprod[0], oprod[1], oprod[2], oprod[3]);
  ob[1] = make_float4(oprod[4], oprod[5], oprod[6], oprod[7]);
}

__device__ __forceinline__ size_t tile_of(const SceneDev &sc, int task) {
  const int txy = sc.task_txy[task];
  return (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
}

}  // namespace

template <int C, bool U16, int NT>
__global__ void __launch_bounds__(128, 4) quad_kernel(const __grid_constant__ SceneDev sc,
                                                      const __grid_constant__ CorrConst cfg, int RE) {
  extern __shared__ float sm[];
  __shared__ float s_lpf[64];  // the correlation LPF, read per lane
  for (int i = threadIdx.x; i < 64; i += blockDim.x) s_lpf[i] = cfg.lpf[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3, r = lane & 7, NW = blockDim.x >> 5;
  float *ws = sm + warp * quad_warp_floats(C);
  const short *strip_code = &sc.corr_cfg->strip_code[0][0][0];
  const int stride = gridDim.x * NW;
  int task = blockIdx.x * NW + warp;
  SubtilePlan p;
  size_t tile = 0;
  if (task < sc.num_tasks) {
    p = quad_plan(sc, C, task, q, 0);
    tile = tile_of(sc, task);
    quad_stage<U16>(sc, p, 0, ws, q, r);
  }
  for (; task < sc.num_tasks; task += stride) {
    quad_clt<C, U16>(sc, task, p, ws, lane);
    const size_t cur = tile;
    const int next = task + stride;
    if (next < sc.num_tasks) {
      p = quad_plan(sc, C, next, q, 0);
      tile = tile_of(sc, next);
    }
    const float *surf = quad_surfaces<C>(sc, cfg, s_lpf, cur, ws, lane);
    if (next < sc.num_tasks) quad_stage<U16>(sc, p, 0, ws, q, r);  // the next tile's first windows
    float cmb[8], oprod[8];
    quad_strips<NT>(sc, cfg, surf, cur, RE, strip_code, lane, cmb, oprod);
    store_products<NT>(sc, task, RE, lane, cmb, oprod);
    if (C > 1) {  // the next tile's windows and CLT go over the surfaces
      if (lane == 0) bulk_read_done();
      __syncwarp();
    }
  }
  cp_async_wait_all();
  if (lane == 0) bulk_done();
}

// conv_shift (tp_forward.cuh) on two neighbouring values v, v + 1 at a time, the same bits.  buf: 16 floats per
// eight lanes, where the row's cosines and sines are exchanged.
__device__ __forceinline__ void conv_shift_pairs(float o[4][8], const float *kp, float rx, float ry, int r, float *buf) {
  float ch, shh, cvr, svr;
  __sincosf(CUDART_PI_F * 0.0625f * (2 * r + 1) * rx, &shh, &ch);
  __sincosf(CUDART_PI_F * 0.0625f * (2 * r + 1) * ry, &svr, &cvr);
  buf[r] = cvr;
  buf[8 + r] = svr;
  __syncwarp();
  const float2 ch2 = dup2(ch), sh2 = dup2(shh), ns2 = dup2(-shh);
#pragma unroll
  for (int w = 0; w < 2; w++) {
    float4 k[4];
    if (kp) {
#pragma unroll
      for (int m = 0; m < 4; m++) k[m] = __ldg((const float4 *)(kp + m * 64 + r * 8 + 4 * w));
    }
    const float4 cq = *(const float4 *)(buf + 4 * w), sq = *(const float4 *)(buf + 8 + 4 * w);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int v = 4 * w + 2 * u;
      float2 d[4];
#pragma unroll
      for (int m = 0; m < 4; m++) d[m] = make_float2(o[m][v], o[m][v + 1]);
      if (kp) {
        float2 kk[4], n[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
          kk[m] = u ? make_float2(k[m].z, k[m].w) : make_float2(k[m].x, k[m].y);
          n[m] = neg2(kk[m]);
        }
        const float2 e0 = fma2(d[3], kk[3], fma2(d[2], n[2], fma2(d[0], kk[0], mul2(d[1], n[1]))));
        const float2 e1 = fma2(d[2], n[3], fma2(d[3], n[2], fma2(d[1], kk[0], mul2(d[0], kk[1]))));
        const float2 e2 = fma2(d[1], n[3], fma2(d[0], kk[2], fma2(d[2], kk[0], mul2(d[3], n[1]))));
        const float2 e3 = fma2(d[0], kk[3], fma2(d[1], kk[2], fma2(d[3], kk[0], mul2(d[2], kk[1]))));
        d[0] = e0; d[1] = e1; d[2] = e2; d[3] = e3;
      }
      const float2 cv = u ? make_float2(cq.z, cq.w) : make_float2(cq.x, cq.y);
      const float2 sv = u ? make_float2(sq.z, sq.w) : make_float2(sq.x, sq.y);
      const float2 nv = neg2(sv);
      const float2 t0 = fma2(d[0], ch2, mul2(d[1], ns2)), t1 = fma2(d[1], ch2, mul2(d[0], sh2));
      const float2 t2 = fma2(d[2], ch2, mul2(d[3], ns2)), t3 = fma2(d[3], ch2, mul2(d[2], sh2));
      const float2 f[4] = {fma2(t0, cv, mul2(t2, nv)), fma2(t1, cv, mul2(t3, nv)), fma2(t0, sv, mul2(t2, cv)),
                           fma2(t1, sv, mul2(t3, cv))};
#pragma unroll
      for (int m = 0; m < 4; m++) {
        o[m][v] = f[m].x;
        o[m][v + 1] = f[m].y;
      }
    }
  }
  __syncwarp();
}

// u16 Bayer quads with strips of up to 32 entries: three warps per tile.  Phase A: warp k folds colour item k of the
// four sensors; phase B: warp k carries pairs 2k and 2k + 1 over the three colours to their surfaces and strip
// values.  A warp needs a third of the registers' and shared memory's contents that it does with a tile to
// itself, so 24 warps share an SM at 80 registers (warp per tile: 16 at 128).  Two barriers per tile: A, every warp
// has read the last tile's CLT and written its strip values; B, the CLT is complete.  A warp's own scratch (floats):
// the staged windows, a tile ahead, then a couple's spectra; behind them its two surfaces, where the folds'
// transposes go too.
// 4 x 2592x1936 with kernel tables, 78,408 tiles: warp per tile 729 us, this 728, with conv_shift_pairs
// 693 (packed, the warp per tile spills: 746); 4 x 648x488, 4,941 tiles: 52 -> 46.  The price is that each warp
// reads the whole CLT (288 shared-memory accesses a tile instead of 96), so that pipe is at 69 % and the issue
// slots at 59 % (4 x 1296x968); float windows are too large for eight CTAs an SM (7,018 tiles: 73 us warp per tile, 75 here), so
// they stay with a warp per tile.
constexpr int Q3_SURF = 4 * Stage<true>::WIN;       // first surface (+ 0 or 2 floats)
constexpr int Q3_WS = Q3_SURF + 456;                // scratch of a warp
// 29,152 bytes with the 1 KB a CTA costs: eight in 228 KB, with 32 bytes left for each (static shared memory, of which
// the kernel has none, is not in the assertion)
constexpr int Q3_FLOATS = 12 * QP_CLT + 3 * Q3_WS;
static_assert(Q3_SURF >= QP_BUF && 8 * (4 * Q3_FLOATS + 1024) <= 228 * 1024, "spectra over the windows, eight CTAs");
// strip value e of pair p: [6][32] in the 4 unused floats of each of the 48 quadrants
__device__ __forceinline__ int q3_strip(int p, int e) { return (p * 8 + (e >> 2)) * QP_QUAD + 32 + (e & 3); }

__global__ void __launch_bounds__(96, 8) quad3_kernel(const __grid_constant__ SceneDev sc,
                                                      const __grid_constant__ CorrConst cfg, int RE) {
  extern __shared__ float sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3, r = lane & 7;
  float *ws = sm + 12 * QP_CLT + warp * Q3_WS;
  const float2 lpf = make_float2(0.25f * cfg.lpf[lane], 0.25f * cfg.lpf[lane + 32]);
  const int rr = sc.bayer_red_row, rc = sc.bayer_red_col;
  // the couple's sensors: 0-1 and 2-3, 0-2 and 1-3, 0-3 and 2-1
  const int f1 = warp == 1 ? 1 : 2, g0 = warp + 1, g1 = warp == 2 ? 1 : 3;
  // the strip products of a task: the values are 1 for pairs that are not combined
  auto products = [&](size_t t) {
    if (lane < RE) {
      float v = sm[q3_strip(0, lane)];
#pragma unroll
      for (int p = 1; p < 6; p++) v *= sm[q3_strip(p, lane)];
      sc.sprod[t * RE + lane] = v;
    }
  };
  int task = blockIdx.x;
  if (task >= sc.num_tasks) return;
  SubtilePlan p = quad_plan(sc, 3, task, q, warp);
  size_t tile = tile_of(sc, task), prev = 0;
  stage_window<true>(sc, sc.images[q], p.tlx, p.tly, ws + q * Stage<true>::WIN, r);
  cp_async_commit();
#pragma unroll 1
  for (;;) {
    SWin<true> w;
    w.base = (const Stage<true>::T *)(ws + q * Stage<true>::WIN);
    w.sx = p.tlx & (Stage<true>::CH - 1);
    w.scale = sc.color_scale[warp];
    cp_async_wait_all();
    __syncwarp();
    float o[4][8];
    float *tbuf = ws + Q3_SURF + q * 72;
    if (warp < 2) {
      const int pc = ((warp == 0 ? rc : 1 - rc) - p.tlx) & 1, pr = ((warp == 0 ? rr : 1 - rr) - p.tly) & 1;
      subtile_clt<1>(w, p.rx, p.ry, pc, pr, 0, r, tbuf, o);
    } else {
      const int pg = (p.tlx + p.tly + rc + rr + 1) & 1;
      subtile_clt<2>(w, p.rx, p.ry, 0, 0, pg, r, tbuf, o);
    }
    conv_shift_pairs(o, (p.kidx >= 0) ? sc.kernels[q] + (size_t)p.kidx * TP_CLT : nullptr, p.rx, p.ry, r, tbuf);
    __syncthreads();  // A
    float *sdst = sm + (warp * 4 + q) * QP_CLT + r * 8 + (r & 4) * ((QP_HALF - 32) / 4);
#pragma unroll
    for (int m = 0; m < 4; m++) {
      *(float4 *)(sdst + m * QP_QUAD) = make_float4(o[m][0], o[m][1], o[m][2], o[m][3]);
      *(float4 *)(sdst + m * QP_QUAD + 4) = make_float4(o[m][4], o[m][5], o[m][6], o[m][7]);
    }
    if (warp == 2 && task >= (int)gridDim.x) products(task - gridDim.x);  // the last task's
    prev = tile;
    const int next = task + gridDim.x;
    const bool more = next < sc.num_tasks;
    if (more) {
      p = quad_plan(sc, 3, next, q, warp);
      tile = tile_of(sc, next);
    }
    __syncthreads();  // B
    couple_of_quad<3>(sc, cfg, lpf, sm, prev, warp, 0, g0, f1, g1, (float2 *)ws, lane);
    // 1800 bytes from a couple to the next: 0 or 8 past a 16-byte boundary, in shared memory too; the two floats
    // before or after the aligned 1792 bytes go out by plain stores
    const int odd = (int)((prev + warp) & 1);
    float *surf = ws + Q3_SURF + 2 * odd;
    couple_surfaces((float2 *)ws, surf, surf + 225, lane);
    bulk_fence();
    __syncwarp();
    float *g = sc.corr + prev * 1350 + warp * 450;
    if (lane == 0) bulk_store(g + 2 * odd, surf + 2 * odd, 1792);
    if (lane < 2) g[odd ? lane : 448 + lane] = surf[odd ? lane : 448 + lane];
    if (more) {
      stage_window<true>(sc, sc.images[q], p.tlx, p.tly, ws + q * Stage<true>::WIN, r);
      cp_async_commit();
    }
    if (warp < 2) {
      // getMaxXSOrtho profiles of the horizontal (warp 0) and the vertical pairs, as quad_strips: lane j of each
      // half one column or row, rows 4 half .. 4 half + 3
      const int half = lane >> 4, j = lane & 15, stride = warp ? 1 : 15;
      if (j < 15) {
        const float *lo = surf + (warp ? j * 15 : j) + 4 * half * stride, *hi = lo + (14 - 8 * half) * stride;
        float pr[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          pr[i] = (0.5f * (lo[0] + hi[0]) + cfg.corr_offset) * (0.5f * (lo[225] + hi[225]) + cfg.corr_offset);
          lo += stride;
          hi -= stride;
        }
        *(float4 *)(sc.osum + ((size_t)task * 32 + warp * 16 + j) * 8 + half * 4) = make_float4(pr[0], pr[1], pr[2], pr[3]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int pi = 2 * warp + h;
      float v = 1.f;
      if (cfg.pairs[pi].in_combo && lane < RE) {
        const float d = strip_of(surf + 225 * h, quad_code(&sc.corr_cfg->strip_code[0][0][0], pi < 4 ? pi >> 1 : pi - 2, lane), lane);
        if (sc.strips) sc.strips[(prev * 6 + pi) * RE + lane] = d;  // kept for the adjoint
        v = d + cfg.corr_offset;
        if (v < 0.0f) v = 0.0f;
        if (cfg.twice_diagonal) v *= v;
      }
      sm[q3_strip(pi, lane)] = v;
    }
    if (!more) break;
    if (lane == 0) bulk_read_done();  // the surfaces are out of shared memory
    __syncwarp();
    task = next;
  }
  __syncthreads();
  if (warp == 2) products(task);
  if (lane == 0) bulk_done();
}

// The same over many mono scenes, a unit of four tiles (of one scene) per CTA and step, as
// fused_batch_kernel.
template <bool U16, int NT>
__global__ void __launch_bounds__(128, 4)
    quad_batch_kernel(const SceneDev *__restrict__ scenes, const int *__restrict__ unit_off, int nscenes,
                      int total_units, int cfg_floats) {
  extern __shared__ float smem[];
  __shared__ int s_off[TP_BATCH_MAX + 1];
  __shared__ SceneDev s_sc;
  CorrConst *s_cfg = (CorrConst *)smem;  // header and the six pairs of the current scene
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3, r = lane & 7;
  float *ws = smem + cfg_floats + warp * quad_warp_floats(1);
  for (int i = threadIdx.x; i <= nscenes; i += blockDim.x) s_off[i] = unit_off[i];
  int cur = -1;
  bool staged = false;
  SubtilePlan p;
  __syncthreads();
  for (int u = blockIdx.x; u < total_units; u += gridDim.x) {
    int lo = 0, hi = nscenes - 1;  // last scene whose first unit is <= u
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_off[mid] <= u) lo = mid;
      else hi = mid - 1;
    }
    if (lo != cur) {
      __syncthreads();
      const int *src = (const int *)(scenes + lo);
      for (int i = threadIdx.x; i < (int)(sizeof(SceneDev) / sizeof(int)); i += blockDim.x) ((int *)&s_sc)[i] = src[i];
      const int cfg_words = (int)((offsetof(CorrConst, pairs) + 6 * sizeof(PairDev)) / sizeof(int));
      const int *csrc = (const int *)scenes[lo].corr_cfg;
      for (int i = threadIdx.x; i < cfg_words; i += blockDim.x) ((int *)s_cfg)[i] = csrc[i];
      cur = lo;
      __syncthreads();
    }
    const SceneDev &sc = s_sc;
    const CorrConst &cfg = *s_cfg;
    const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
    const int task = (u - s_off[lo]) * 4 + warp;
    const int nu = u + gridDim.x, next = (nu < s_off[lo + 1]) ? (nu - s_off[lo]) * 4 + warp : sc.num_tasks;
    if (task < sc.num_tasks) {
      if (!staged) {
        p = quad_plan(sc, 1, task, q, 0);
        quad_stage<U16>(sc, p, 0, ws, q, r);
      }
      const size_t tile = tile_of(sc, task);
      quad_clt<1, U16>(sc, task, p, ws, lane);
      staged = next < sc.num_tasks;  // the next unit's windows, where it is of the same scene
      if (staged) p = quad_plan(sc, 1, next, q, 0);
      const float *surf = quad_surfaces<1>(sc, cfg, cfg.lpf, tile, ws, lane);
      if (staged) quad_stage<U16>(sc, p, 0, ws, q, r);
      float cmb[8], oprod[8];
      quad_strips<NT>(sc, cfg, surf, tile, RE, &sc.corr_cfg->strip_code[0][0][0], lane, cmb, oprod);
      store_products<NT>(sc, task, RE, lane, cmb, oprod);
    }
  }
  cp_async_wait_all();
  if (lane == 0) bulk_done();
}

// Phase C for the tiles of a fused forward that left it out: warp per task, from the strip
// products (sc.sprod) and the ortho profile products (sc.osum) the forward wrote.  Both lie by task and the
// combined strip goes to another buffer (sc.combo), so a tile that the task list names twice is finished twice
// from unchanged products.  Phase C is short chains of dependent shuffles, divides and powers; the
// fused kernel's 16 warps per SM cannot hide their latency, while this kernel's few registers
// and no CLT buffer let 64 warps share an SM.
template <int NT>
__device__ __forceinline__ void extract_task(const SceneDev &sc, const CorrConst &cfg, int quad, int RE, int task,
                                             float *combo, int lane) {
  const size_t tile = tile_of(sc, task);
  float cmb[8], oprod[8];
#pragma unroll
  for (int t = 0; t < NT; t++) {
    const int e = lane + 32 * t;
    cmb[t] = (e < RE) ? sc.sprod[(size_t)task * RE + e] : 0.f;
  }
  if (quad) {  // other layouts have no ortho profiles
    const float4 *ob = (const float4 *)(sc.osum + ((size_t)task * 32 + lane) * 8);
    const float4 o0 = ob[0], o1 = ob[1];
    oprod[0] = o0.x; oprod[1] = o0.y; oprod[2] = o0.z; oprod[3] = o0.w;
    oprod[4] = o1.x; oprod[5] = o1.y; oprod[6] = o1.z; oprod[7] = o1.w;
  }
  const int ncomb = cfg.twice_diagonal ? 2 * cfg.num_combo : cfg.num_combo;
  const float sum = fwd_extract_values<NT, true>(sc, cfg, quad, sc.num_pairs, RE, cfg.log_combine, ncomb, tile, combo,
                                                 lane, cmb, oprod);
  fwd_extract_finish(sc, cfg, quad, tile, combo, sum, lane);
}

template <int NT>
__global__ void __launch_bounds__(128) extract_kernel(const __grid_constant__ SceneDev sc,
                                                      const __grid_constant__ CorrConst cfg, int quad, int RE) {
  __shared__ float s_combo[4][TP_MAX_STRIP * 15];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int task = blockIdx.x * 4 + warp;
  if (task >= sc.num_tasks) return;  // whole warps
  extract_task<NT>(sc, cfg, quad, RE, task, s_combo[warp], lane);
}

// the extraction of every scene of a batch: a block per unit of four tiles
template <int NT>
__global__ void __launch_bounds__(128) extract_batch_kernel(const SceneDev *__restrict__ scenes,
                                                            const int *__restrict__ unit_off, int nscenes) {
  __shared__ float s_combo[4][TP_MAX_STRIP * 15];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, u = blockIdx.x;
  int lo = 0, hi = nscenes - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (unit_off[mid] <= u) lo = mid;
    else hi = mid - 1;
  }
  const SceneDev &sc = scenes[lo];
  const int task = (u - unit_off[lo]) * 4 + warp;
  if (task >= sc.num_tasks) return;  // whole warps
  const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  extract_task<NT>(sc, *sc.corr_cfg, 1, RE, task, s_combo[warp], lane);
}

cudaError_t upload_quad_constants() { return upload_dtt_constants(); }

static bool one_type(const SceneDev &sc) {
  for (int i = 1; i < sc.num_sensors; i++)
    if (sc.img_dtype[i] != sc.img_dtype[0]) return false;
  return true;
}

// a standard quad with images of one type and room for the products between the two passes
bool quad_forward_ok(const SceneDev &sc) { return sc.quad_std && sc.sprod && sc.osum && one_type(sc); }

// a batch's mono scenes, all standard quads of the same image type
bool quad_batch_ok(const SceneDev *h, int n) {
  for (int i = 0; i < n; i++)
    if (!quad_forward_ok(h[i]) || h[i].num_colors != 1 || h[i].img_dtype[0] != h[0].img_dtype[0]) return false;
  return n > 0;
}

cudaError_t launch_extract_pass(const SceneDev &sc, const CorrConst &cc, int quad, int RE, cudaStream_t st) {
  if (RE <= 32) extract_kernel<1><<<(sc.num_tasks + 3) / 4, 128, 0, st>>>(sc, cc, quad, RE);
  else extract_kernel<8><<<(sc.num_tasks + 3) / 4, 128, 0, st>>>(sc, cc, quad, RE);
  return cudaGetLastError();
}

static int strip_entries(const SceneDev &sc) {
  return (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
}

template <typename K>
static cudaError_t go_quad(K kernel, int nw, const SceneDev &sc, const CorrConst &cc, int RE, cudaStream_t st) {
  const int bytes = quad_warp_floats(sc.num_colors) * nw * 4, units = (sc.num_tasks + nw - 1) / nw;
  int res = 0;
  const cudaError_t e = kernel_residency((const void *)kernel, nw * 32, bytes, &res);
  if (e != cudaSuccess) return e;
  if (res < 1) return cudaErrorInvalidConfiguration;
  kernel<<<units < res ? units : res, nw * 32, bytes, st>>>(sc, cc, RE);
  return cudaGetLastError();
}

static cudaError_t go_quad3(const SceneDev &sc, const CorrConst &cc, int RE, cudaStream_t st) {
  const int bytes = Q3_FLOATS * 4;
  int res = 0;
  const cudaError_t e = kernel_residency((const void *)quad3_kernel, 96, bytes, &res);
  if (e != cudaSuccess) return e;
  if (res < 1) return cudaErrorInvalidConfiguration;
  quad3_kernel<<<sc.num_tasks < res ? sc.num_tasks : res, 96, bytes, st>>>(sc, cc, RE);
  return cudaGetLastError();
}

cudaError_t launch_quad_forward(const SceneDev &sc, const CorrConst &cc, int nw, cudaStream_t st) {
  const int RE = strip_entries(sc);
  const bool one = RE <= 32, u16 = sc.img_dtype[0] == 1;
  cudaError_t e;
  if (sc.num_colors == 3) {
    if (u16 && one) e = go_quad3(sc, cc, RE, st);
    else if (one) e = go_quad(quad_kernel<3, false, 1>, nw, sc, cc, RE, st);
    else e = u16 ? go_quad(quad_kernel<3, true, 8>, nw, sc, cc, RE, st) : go_quad(quad_kernel<3, false, 8>, nw, sc, cc, RE, st);
  } else {
    if (u16) e = one ? go_quad(quad_kernel<1, true, 1>, nw, sc, cc, RE, st) : go_quad(quad_kernel<1, true, 8>, nw, sc, cc, RE, st);
    else e = one ? go_quad(quad_kernel<1, false, 1>, nw, sc, cc, RE, st) : go_quad(quad_kernel<1, false, 8>, nw, sc, cc, RE, st);
  }
  return e != cudaSuccess ? e : launch_extract_pass(sc, cc, 1, RE, st);
}

cudaError_t launch_quad_batch(const SceneDev *h, const SceneDev *scenes_dev, const int *unit_off_dev, int n,
                              int total_units, cudaStream_t st) {
  const int cf = (int)((offsetof(CorrConst, pairs) + 6 * sizeof(PairDev) + 15) / 16 * 4);
  const int bytes = (cf + 4 * quad_warp_floats(1)) * 4;
  bool one = true;
  for (int i = 0; i < n; i++) one = one && strip_entries(h[i]) <= 32;
  auto go = [&](auto kernel) -> cudaError_t {
    int res = 0;
    const cudaError_t e = kernel_residency((const void *)kernel, 128, bytes, &res);
    if (e != cudaSuccess) return e;
    if (res < 1) return cudaErrorInvalidConfiguration;
    kernel<<<total_units < res ? total_units : res, 128, bytes, st>>>(scenes_dev, unit_off_dev, n, total_units, cf);
    return cudaGetLastError();
  };
  cudaError_t e;
  if (h[0].img_dtype[0] == 1) e = one ? go(quad_batch_kernel<true, 1>) : go(quad_batch_kernel<true, 8>);
  else e = one ? go(quad_batch_kernel<false, 1>) : go(quad_batch_kernel<false, 8>);
  if (e != cudaSuccess) return e;
  if (one) extract_batch_kernel<1><<<total_units, 128, 0, st>>>(scenes_dev, unit_off_dev, n);
  else extract_batch_kernel<8><<<total_units, 128, 0, st>>>(scenes_dev, unit_off_dev, n);
  return cudaGetLastError();
}
