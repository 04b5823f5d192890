// tp_fused.cu -- fused forward tile kernel: convert+correct -> pair correlation
// -> strip combination -> disparity extraction, one CTA per group of tiles, for the scenes that
// tp_quad.cu (standard quads) and tp_many.cu (many general pairs) do not take; the choice between
// them (launch_fused_forward); the rig's inter-camera correlation; IMCLT.
//
// Same arithmetic as the stage kernels (ImageDtt.extract_correct_tile,
// convolve_tile, fract_shift; Correlation2d.correlateCompositeFD,
// scaleRotateInterpoateSingleCorrelation, combineInterpolatedCorrelations,
// getMaxXYInt, getMaxXCm, getMaxXSOrtho) but organised for GB300:
//
//  phase A  one warp = one colour of 4 sensors of a tile; lanes 8q..8q+7 own
//           sensor q, lane r owns folded row r.  The fold reads each needed
//           pixel once (L1-cached __ldg); 8-point DCT-IV/DST-IV run in
//           registers (Plonka-Tasche recursion, DttRad2.java:1107-1146, scale
//           folded into the first stage); the 8x8 transpose goes through a
//           9-padded shared buffer.  For Bayer planes only the transforms that
//           are not symmetric images of another are computed: a red/blue
//           window is sparse on a 2x2 lattice, so SC/CS/SS are index reversals
//           of CC with window-phase signs; a green window is a checkerboard, so
//           CS and SS are reversals of SC and CC.  That is 4 instead of 12 2D
//           transforms per sensor.  CLT goes to shared memory (for phase B) and
//           to HBM (a declared output); per-frequency amplitudes are cached.
//  phase B  one warp = one (tile, pair): the correlation product, fat-zero
//           normalisation, colour mix and LPF on 2 CLT indices per lane, the
//           four 2D DCT-IIe/DST-IIe in registers, the 15x15 unfold, the surface
//           to HBM, and that pair's strip folded into a per-warp running product.
//  phase C  one warp = one tile: combine the per-warp strip products, integer
//           argmax on the disparity axis, windowed centroid, hor/vert maxima.
#include "tp_forward.cuh"
#include "tp_pairs.cuh"
#include "tp_launch.h"

// ---------------------------------------------------------------------------
// warp-per-tile schedule: one warp carries a tile through all stages, no CTA barriers
// ---------------------------------------------------------------------------
template <int C, int NT>  // colours: 1 (mono) or 3 (Bayer R, B, G); strip entries per lane / 32
__global__ void __launch_bounds__(128, 4) fused_forward_kernel(const __grid_constant__ SceneDev sc,
                                                               const __grid_constant__ FwdShape fs,
                                                               const __grid_constant__ CorrConst cfg) {
  extern __shared__ float sm[];
  __shared__ float s_lpf[64];  // the correlation LPF, read per lane by fwd_pair
  for (int i = threadIdx.x; i < 64; i += blockDim.x) s_lpf[i] = cfg.lpf[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = fs.S, P = fs.P, RE = fs.RE, NW = fs.nw;
  // per-warp shared memory: CLT of the tile [S][C][4][64] and a 288-float scratch buffer
  float *s_clt = sm + warp * fs.per_warp;
  float *scr = s_clt + fs.clt_floats;
  const short *strip_code = &sc.corr_cfg->strip_code[0][0][0];
  const int groups = (S + 3) >> 2;
  const bool log_mode = cfg.log_combine;
  const int ncomb = cfg.twice_diagonal ? 2 * cfg.num_combo : cfg.num_combo;
  for (int task = blockIdx.x * NW + warp; task < sc.num_tasks; task += gridDim.x * NW) {
    const int txy = sc.task_txy[task];
    const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
    for (int gt = 0; gt < C * groups; gt++) fwd_clt_item<C>(sc, S, task, tile, gt, groups, s_clt, scr, lane);
    __syncwarp();
    float cmb[8];
#pragma unroll
    for (int t = 0; t < NT; t++) cmb[t] = log_mode ? 0.f : 1.f;
    float oprod[8];  // hor / vert profile products of this lane's column (row), filled by phase B
#pragma unroll
    for (int i = 0; i < 8; i++) oprod[i] = 1.f;
    for (int pi = 0; pi < P; pi++)
      fwd_pair<C, NT, true>(sc, cfg, s_lpf, tile, P, pi, RE, log_mode, strip_code, s_clt, scr, lane, cmb, nullptr,
                            oprod);
    fwd_extract<NT, true>(sc, cfg, fs.quad, P, RE, log_mode, ncomb, tile, scr, lane, cmb, oprod);
  }
}

// ---------------------------------------------------------------------------
// Warp per tile with staged image windows: scenes of 4 (or fewer) u16 Bayer sensors.
// The image reads of phase A are its main cost (the warp waits on them once per
// colour item), so each item's four 16x16 sensor windows are copied into shared
// memory one item ahead, while the warp computes the previous item: 16 rows x 24
// u16 from the 16-byte boundary below the window corner, three 16-byte cp.async
// chunks per row, into the CLT slot of (sensor, colour) -- that slot holds nothing
// until the item writes its CLT there, after its last window read.  The next
// tile's first windows go in after its correlation phase has read the CLT slots.
// Windows that cross the image border are gathered with the edge mirroring.
// ---------------------------------------------------------------------------
__device__ __forceinline__ SubtilePlan load_plan(const SceneDev &sc, int task, int s, int c) {
  return sc.plan[((size_t)task * sc.num_sensors + s) * 3 + c];
}

// phase A item c (colour) of a staged tile: the window of (sensor q, c) is in its CLT slot; pn is
// the plan of item c + 1, whose windows are staged once this item's are read
__device__ __forceinline__ void fwd_clt_item_win(const SceneDev &sc, const uint16_t *img, int S, size_t tile, int c,
                                                 const SubtilePlan &p, const SubtilePlan &pn, float *s_clt,
                                                 float *scr, int lane) {
  const int q = lane >> 3, r = lane & 7;
  const int rr = sc.bayer_red_row, rc = sc.bayer_red_col;
  const bool act = q < S;
  const int sidx = act ? q : S - 1;
  SWin<true> w;
  w.base = (const uint16_t *)(s_clt + ((size_t)sidx * 3 + c) * TP_CLT);
  w.sx = p.tlx - (p.tlx & ~7);
  w.scale = sc.color_scale[c];
  cp_async_wait_all();  // this item's windows, copied by every lane
  __syncwarp();
  float o[4][8];
  float *tbuf = scr + q * 72;
  if (c < 2) {
    const int pc = ((c == 0 ? rc : 1 - rc) - p.tlx) & 1, pr = ((c == 0 ? rr : 1 - rr) - p.tly) & 1;
    subtile_clt<1>(w, p.rx, p.ry, pc, pr, 0, r, tbuf, o);
  } else {
    const int pg = (p.tlx + p.tly + rc + rr + 1) & 1;
    subtile_clt<2>(w, p.rx, p.ry, 0, 0, pg, r, tbuf, o);
  }
  // every lane has read this item's windows (the transposes in subtile_clt synchronise the warp)
  if (c < 2) {
    if (act) stage_window<true>(sc, img, pn.tlx, pn.tly, s_clt + ((size_t)q * 3 + c + 1) * TP_CLT, r);
    cp_async_commit();
  }
  const float *kp = (p.kidx >= 0) ? sc.kernels[sidx] + (size_t)p.kidx * TP_CLT : nullptr;
  conv_shift(o, kp, p.rx, p.ry, r);
  if (act) {
    float *sdst = s_clt + ((size_t)q * 3 + c) * TP_CLT + r * 8;
#pragma unroll
    for (int m = 0; m < 4; m++) {
      *(float4 *)(sdst + m * 64) = make_float4(o[m][0], o[m][1], o[m][2], o[m][3]);
      *(float4 *)(sdst + m * 64 + 4) = make_float4(o[m][4], o[m][5], o[m][6], o[m][7]);
    }
    store_clt(sc, c, r, sc.clt + ((tile * S + q) * 3 + c) * TP_CLT + r * 8, o);
  }
}

template <int NT>
__global__ void __launch_bounds__(128, 4) fused_forward_win_kernel(const __grid_constant__ SceneDev sc,
                                                                   const __grid_constant__ FwdShape fs,
                                                                   const __grid_constant__ CorrConst cfg) {
  extern __shared__ float sm[];
  __shared__ float s_lpf[64];  // the correlation LPF, read per lane by fwd_pair
  for (int i = threadIdx.x; i < 64; i += blockDim.x) s_lpf[i] = cfg.lpf[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3, r = lane & 7;
  const int S = fs.S, P = fs.P, RE = fs.RE, NW = fs.nw;
  float *s_clt = sm + warp * fs.per_warp;
  float *scr = s_clt + fs.clt_floats;
  const short *strip_code = &sc.corr_cfg->strip_code[0][0][0];
  const bool log_mode = cfg.log_combine;
  const bool act = q < S;
  const int sidx = act ? q : S - 1;
  const uint16_t *img = (const uint16_t *)sc.images[sidx];
  const int stride = gridDim.x * NW;
  SubtilePlan pc;
  int task = blockIdx.x * NW + warp;
  if (task < sc.num_tasks) {
    pc = load_plan(sc, task, sidx, 0);
    if (act) stage_window<true>(sc, img, pc.tlx, pc.tly, s_clt + (size_t)q * 3 * TP_CLT, r);
    cp_async_commit();
  }
  for (; task < sc.num_tasks; task += stride) {
    const int txy = sc.task_txy[task];
    const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
#pragma unroll 1
    for (int c = 0; c < 3; c++) {
      const SubtilePlan pn = load_plan(sc, task, sidx, c < 2 ? c + 1 : c);
      fwd_clt_item_win(sc, img, S, tile, c, pc, pn, s_clt, scr, lane);
      pc = pn;
    }
    __syncwarp();
    const int next = task + stride;
    if (next < sc.num_tasks) pc = load_plan(sc, next, sidx, 0);
    float cmb[8];
#pragma unroll
    for (int t = 0; t < NT; t++) cmb[t] = log_mode ? 0.f : 1.f;
    float oprod[8];
#pragma unroll
    for (int i = 0; i < 8; i++) oprod[i] = 1.f;
    for (int pi = 0; pi < P; pi++)
      fwd_pair<3, NT, true>(sc, cfg, s_lpf, tile, P, pi, RE, log_mode, strip_code, s_clt, scr, lane, cmb, nullptr,
                            oprod);
    if (next < sc.num_tasks) {  // the CLT slots are read (fwd_pair ends with __syncwarp): next tile's windows
      if (act) stage_window<true>(sc, img, pc.tlx, pc.tly, s_clt + (size_t)q * 3 * TP_CLT, r);
      cp_async_commit();
    }
    // phase C in extract_kernel: the strip products and ortho profile products go out as they are
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const int e = lane + 32 * t;
      if (e < RE) sc.sprod[(size_t)task * RE + e] = cmb[t];
    }
    float4 *ob = (float4 *)(sc.osum + ((size_t)task * 32 + lane) * 8);
    ob[0] = make_float4(oprod[0], oprod[1], oprod[2], oprod[3]);
    ob[1] = make_float4(oprod[4], oprod[5], oprod[6], oprod[7]);
  }
  cp_async_wait_all();
}

// ---------------------------------------------------------------------------
// pair-per-warp schedule: a CTA of nw warps per tile shares the tile's CLT; the
// warps split the (colour, sensor-group) items, then the pairs, and warp 0
// combines their partial strip products for the extraction.  For many pairs
// (16 sensors, 120 pairs) this holds one CLT per CTA instead of one per warp.
// MAXT / MINB: the launch bounds.  With 3 warps for a quad colour scene (one colour
// item, then two pairs per warp) and 8 CTAs per SM the register budget is 85 per
// thread, for 24 resident warps sharing 8 tile CLTs.
// ---------------------------------------------------------------------------
template <int C, int NT, int MAXT = 128, int MINB = 4>
__global__ void __launch_bounds__(MAXT, MINB) fused_split_kernel(const __grid_constant__ SceneDev sc,
                                                          const __grid_constant__ FwdShape fs,
                                                          const __grid_constant__ CorrConst cfg) {
  extern __shared__ float sm[];
  __shared__ float s_lpf[64];  // the correlation LPF, read per lane by fwd_pair
  for (int i = threadIdx.x; i < 64; i += blockDim.x) s_lpf[i] = cfg.lpf[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = fs.S, P = fs.P, RE = fs.RE, NW = fs.nw;
  float *s_clt = sm;
  float *scr = sm + fs.clt_floats + warp * SCR;
  float *part = sm + fs.clt_floats + NW * SCR;  // [NW][240] partial strip combinations
  const short *strip_code = &sc.corr_cfg->strip_code[0][0][0];
  const int groups = (S + 3) >> 2;
  const bool log_mode = cfg.log_combine;
  const int ncomb = cfg.twice_diagonal ? 2 * cfg.num_combo : cfg.num_combo;
  for (int task = blockIdx.x; task < sc.num_tasks; task += gridDim.x) {
    const int txy = sc.task_txy[task];
    const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
    for (int gt = warp; gt < C * groups; gt += NW) fwd_clt_item<C>(sc, S, task, tile, gt, groups, s_clt, scr, lane);
    __syncthreads();
    float cmb[8];
#pragma unroll
    for (int t = 0; t < NT; t++) cmb[t] = log_mode ? 0.f : 1.f;
    for (int pi = warp; pi < P; pi += NW)
      fwd_pair<C, NT>(sc, cfg, s_lpf, tile, P, pi, RE, log_mode, strip_code, s_clt, scr, lane, cmb);
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const int e = lane + 32 * t;
      if (e < RE) part[warp * 240 + e] = cmb[t];
    }
    __syncthreads();  // also makes the surfaces every warp wrote visible to warp 0
    if (warp == 0) {
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const int e = lane + 32 * t;
        if (e < RE) {
          float v = part[e];
          for (int w2 = 1; w2 < NW; w2++) v = log_mode ? v + part[w2 * 240 + e] : v * part[w2 * 240 + e];
          cmb[t] = v;
        }
      }
      fwd_extract<NT>(sc, cfg, fs.quad, P, RE, log_mode, ncomb, tile, scr, lane, cmb);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Batched persistent forward over many scenes of different sensor counts,
// colours, pair sets and sizes.  Scenes are grouped in three classes by the
// schedule their tiles take (colour warp-per-tile, mono warp-per-tile, mono
// pair-per-warp); each class is one persistent launch over a queue of units in
// scene order (NW tiles per unit for warp-per-tile, 1 tile per unit for
// pair-per-warp).  CTAs take units grid-stride, find the unit's scene by
// binary search over the unit offsets and keep the current scene's SceneDev in
// shared memory (reloaded only when the scene changes); the scene's
// correlation set-up is read through its device pointer.
// ---------------------------------------------------------------------------
static cudaError_t init_records(const SceneDev &sc, cudaStream_t st);

int batch_class(const SceneDev &sc) {
  if (sc.num_colors == 3) return 0;
  return sc.num_pairs > 8 ? 2 : 1;
}

static int class_warps(int cls) { return cls == 0 ? 1 : 4; }

int batch_units(const SceneDev &sc) {
  const int nw = batch_class(sc) == 2 ? 1 : class_warps(batch_class(sc));
  return (sc.num_tasks + nw - 1) / nw;
}

template <int C, bool SPLIT, int NW, int NT>
__global__ void __launch_bounds__(NW * 32, (NW == 1) ? 16 : 4)
    fused_batch_kernel(const SceneDev *__restrict__ scenes, const int *__restrict__ unit_off, int nscenes,
                       int total_units, int warp_floats, int cfg_floats) {
  extern __shared__ float smem[];
  __shared__ int s_off[TP_BATCH_MAX + 1];
  __shared__ SceneDev s_sc;
  // the current scene's correlation set-up (header and its pairs) leads the dynamic shared memory
  CorrConst *s_cfg = (CorrConst *)smem;
  float *sm = smem + cfg_floats;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i <= nscenes; i += blockDim.x) s_off[i] = unit_off[i];
  int cur = -1;
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
      int *dst = (int *)&s_sc;
      for (int i = threadIdx.x; i < (int)(sizeof(SceneDev) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
      const int cfg_words = (int)((offsetof(CorrConst, pairs) + scenes[lo].num_pairs * sizeof(PairDev)) / sizeof(int));
      const int *csrc = (const int *)scenes[lo].corr_cfg;
      for (int i = threadIdx.x; i < cfg_words; i += blockDim.x) ((int *)s_cfg)[i] = csrc[i];
      cur = lo;
      __syncthreads();
    }
    const SceneDev &sc = s_sc;
    const CorrConst &cfg = *s_cfg;
    const int S = sc.num_sensors, P = sc.num_pairs;
    const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
    const short *strip_code = &sc.corr_cfg->strip_code[0][0][0];
    const int groups = (S + 3) >> 2;
    const bool log_mode = cfg.log_combine;
    const int ncomb = cfg.twice_diagonal ? 2 * cfg.num_combo : cfg.num_combo;
    const int lu = u - s_off[lo];
    if (SPLIT) {
      float *s_clt = sm;
      float *scr = sm + S * TP_CLT + warp * SCR;
      float *part = sm + S * TP_CLT + NW * SCR;
      const int task = lu;
      const int txy = sc.task_txy[task];
      const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
      for (int gt = warp; gt < groups; gt += NW) fwd_clt_item<C>(sc, S, task, tile, gt, groups, s_clt, scr, lane);
      __syncthreads();
      float cmb[8];
#pragma unroll
      for (int t = 0; t < NT; t++) cmb[t] = log_mode ? 0.f : 1.f;
      for (int pi = warp; pi < P; pi += NW)
        fwd_pair<C, NT>(sc, cfg, cfg.lpf, tile, P, pi, RE, log_mode, strip_code, s_clt, scr, lane, cmb);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const int e = lane + 32 * t;
        if (e < RE) part[warp * 240 + e] = cmb[t];
      }
      __syncthreads();
      if (warp == 0) {
#pragma unroll
        for (int t = 0; t < NT; t++) {
          const int e = lane + 32 * t;
          if (e < RE) {
            float v = part[e];
            for (int w2 = 1; w2 < NW; w2++) v = log_mode ? v + part[w2 * 240 + e] : v * part[w2 * 240 + e];
            cmb[t] = v;
          }
        }
        fwd_extract<NT>(sc, cfg, P <= 8, P, RE, log_mode, ncomb, tile, scr, lane, cmb);
      }
      __syncthreads();
    } else {
      const int task = lu * NW + warp;
      if (task < sc.num_tasks) {
        float *s_clt = sm + warp * warp_floats;
        float *scr = s_clt + S * C * TP_CLT;
        const int txy = sc.task_txy[task];
        const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
        for (int gt = 0; gt < C * groups; gt++) fwd_clt_item<C>(sc, S, task, tile, gt, groups, s_clt, scr, lane);
        __syncwarp();
        float cmb[8];
#pragma unroll
        for (int t = 0; t < NT; t++) cmb[t] = log_mode ? 0.f : 1.f;
        for (int pi = 0; pi < P; pi++)
          fwd_pair<C, NT>(sc, cfg, cfg.lpf, tile, P, pi, RE, log_mode, strip_code, s_clt, scr, lane, cmb);
        fwd_extract<NT>(sc, cfg, P <= 8, P, RE, log_mode, ncomb, tile, scr, lane, cmb);
      }
    }
  }
}

template <typename K>
static cudaError_t launch_batch_k(K kernel, int threads, int bytes, int total_units, const SceneDev *scenes_dev,
                                  const int *unit_off_dev, int n, int warp_floats, int cfg_floats, cudaStream_t st) {
  int res = 0;
  const cudaError_t e = kernel_residency((const void *)kernel, threads, bytes, &res);
  if (e != cudaSuccess) return e;
  if (res < 1) return cudaErrorInvalidConfiguration;
  const int grid = total_units < res ? total_units : res;
  kernel<<<grid, threads, bytes, st>>>(scenes_dev, unit_off_dev, n, total_units, warp_floats, cfg_floats);
  return cudaGetLastError();
}

// one class: scenes_host / scenes_dev hold only that class's scenes, unit_off_dev their unit offsets
cudaError_t launch_fused_batch(int cls, const SceneDev *scenes_host, const SceneDev *scenes_dev,
                               const int *unit_off_dev, int n, int total_units, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (n > TP_BATCH_MAX) return cudaErrorInvalidValue;
  int wf = 0, sp = 0, maxp = 0, maxre = 0;
  for (int i = 0; i < n; i++) {
    maxp = scenes_host[i].num_pairs > maxp ? scenes_host[i].num_pairs : maxp;
    const int re = (scenes_host[i].strip_rows < scenes_host[i].wndy_size ? scenes_host[i].strip_rows
                                                                         : scenes_host[i].wndy_size) * 15;
    maxre = re > maxre ? re : maxre;
    const SceneDev &sc = scenes_host[i];
    if (batch_class(sc) != cls || sc.strip_rows * 15 > 8 * 32) return cudaErrorInvalidValue;
    const cudaError_t ei = init_records(sc, st);
    if (ei != cudaSuccess) return ei;
    const int f = ((sc.num_sensors * sc.num_colors * TP_CLT + SCR) + 3) & ~3;
    wf = f > wf ? f : wf;
    const int g = sc.num_sensors * TP_CLT + 4 * SCR + 4 * 240;
    sp = g > sp ? g : sp;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || total_units <= 0) return e;
  if (quad_batch_ok(scenes_host, n)) return launch_quad_batch(scenes_host, scenes_dev, unit_off_dev, n, total_units, st);
  const int cf = (int)(((offsetof(CorrConst, pairs) + maxp * sizeof(PairDev)) + 15) / 16 * 4);
  auto go = [&](auto kernel, int threads, int floats) {
    return launch_batch_k(kernel, threads, (cf + floats) * 4, total_units, scenes_dev, unit_off_dev, n, wf, cf, st);
  };
  const bool one = maxre <= 32;
  if (cls == 0) return one ? go(fused_batch_kernel<3, false, 1, 1>, 32, wf) : go(fused_batch_kernel<3, false, 1, 8>, 32, wf);
  if (cls == 1)
    return one ? go(fused_batch_kernel<1, false, 4, 1>, 128, 4 * wf) : go(fused_batch_kernel<1, false, 4, 8>, 128, 4 * wf);
  return one ? go(fused_batch_kernel<1, true, 4, 1>, 128, sp) : go(fused_batch_kernel<1, true, 4, 8>, 128, sp);
}

// ---------------------------------------------------------------------------
// Rig (two quad cameras): inter-camera correlation of the sensor-averaged CLT
// of each camera (Correlation2d.correlateInterCamerasFD / cltMixCameras,
// Correlation2d.java:401-448) and its disparity along the horizontal rig
// baseline (ImageDtt.tileInterCamCorrs, ImageDtt.java:7370-7560, without the
// LMA branch).  Warp per tile of the main camera's task list; the correlation
// is the forward kernel's pair phase run on the two averaged CLTs.
// ---------------------------------------------------------------------------
template <int C, int NT>
__global__ void __launch_bounds__(128, 4) rig_kernel(const __grid_constant__ SceneDev mn,
                                                     const __grid_constant__ SceneDev ax,
                                                     const __grid_constant__ CorrConst cfg, float *rig_corr,
                                                     float *rig_rec, float cm_norm, int no_int_x0, int per_warp) {
  extern __shared__ float sm[];
  __shared__ float s_lpf[64];  // the correlation LPF, read per lane by fwd_pair
  for (int i = threadIdx.x; i < 64; i += blockDim.x) s_lpf[i] = cfg.lpf[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, NW = blockDim.x >> 5;
  float *mix = sm + warp * per_warp;  // [2][C][256]
  float *scr = mix + 2 * C * TP_CLT;
  const int RE = (cfg.strip_rows < cfg.wndy_size ? cfg.strip_rows : cfg.wndy_size) * 15;
  const short *strip_code = &mn.corr_cfg->strip_code[0][0][0];
  const int ncomb = cfg.twice_diagonal ? 2 : 1;
  for (int task = blockIdx.x * NW + warp; task < mn.num_tasks; task += gridDim.x * NW) {
    const int txy = mn.task_txy[task];
    const size_t tile = (size_t)(txy >> 16) * mn.tilesX + (txy & 0xffff);
    float *rec = rig_rec + tile * 4;
    if (ax.tile_task[tile] < 0) {
      if (lane < 4) rec[lane] = (lane == 1) ? 0.f : CUDART_NAN_F;
      continue;
    }
    for (int i = lane; i < C * TP_CLT; i += 32) {
      float a = 0.f, b = 0.f;
      for (int s = 0; s < mn.num_sensors; s++) a += mn.clt[(tile * mn.num_sensors + s) * C * TP_CLT + i];
      for (int s = 0; s < ax.num_sensors; s++) b += ax.clt[(tile * ax.num_sensors + s) * C * TP_CLT + i];
      mix[i] = a * (1.0f / mn.num_sensors);
      mix[C * TP_CLT + i] = b * (1.0f / ax.num_sensors);
    }
    __syncwarp();
    float cmb[8];
#pragma unroll
    for (int t = 0; t < NT; t++) cmb[t] = 1.f;
    fwd_pair<C, NT>(mn, cfg, s_lpf, tile, 1, 0, RE, false, strip_code, mix, scr, lane, cmb, rig_corr + tile * TP_CORR);
    float *combo = scr;
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const int e = lane + 32 * t;
      if (e < RE) {
        float v = cmb[t];
        if (v > 0.0f) v = powf(v, 1.0f / ncomb) - cfg.corr_offset;
        combo[e] = v;
      }
    }
    __syncwarp();
    float r0 = CUDART_NAN_F, r1 = 0.f;
    const float v = (lane < 15) ? combo[lane] : CUDART_NAN_F;
    float best = isnan(v) ? -CUDART_INF_F : v;
    int bi = lane < 15 ? lane : 99;
#pragma unroll
    for (int o2 = 16; o2 > 0; o2 >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o2);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o2);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    const unsigned finite = __ballot_sync(0xffffffffu, lane < 15 && !isnan(v));
    const int imx = finite ? bi : 14;
    const float vmax = combo[imx];
    if (vmax >= (no_int_x0 ? 0.5f : 1.0f) * cfg.min_corr) {
      const int ix = imx - 7;
      r0 = (float)(-ix);
      r1 = vmax;
      int dh = cfg.strip_rows;
      float wys = 1.0f;
      if (dh > cfg.wndy_size) dh = cfg.wndy_size;
      else if (dh < cfg.wndy_size) {
        float swy = cfg.wndy[0];
        for (int i = 1; i < dh; i++) swy += cfg.wndy[i];
        wys = 1.0f / swy;
      }
      const int ixc = no_int_x0 ? 0 : ix;
      const int x0 = 7 + ixc, nk = dh * 2 * cfg.wndx_size;
      float s0 = 0.f, sx = 0.f, sx2 = 0.f;
      for (int k = lane; k < nk; k += 32) {  // getMaxXCm with the second moment
        const int dy = k / (2 * cfg.wndx_size), rest = k - dy * 2 * cfg.wndx_size;
        const int adx = rest >> 1, dir = (rest & 1) ? 1 : -1, odd = dy & 1;
        if (((adx - odd) & 1) || (adx == 0 && dir < 0)) continue;
        const int idx = (adx * dir) >> 1, xx = 2 * idx + odd, x1 = x0 + idx;
        if (x1 < 0 || x1 >= 15) continue;
        float d = combo[dy * 15 + x1];
        if (isnan(d) || !(d > 0.0f)) continue;
        d *= (((dy == 0) ? wys : 2.0f * wys) * cfg.wndy[dy]) * cfg.wndx[adx];
        s0 += d;
        sx += d * xx;
        sx2 += d * xx * xx;
      }
      s0 = warp_sum(s0);
      sx = warp_sum(sx);
      sx2 = warp_sum(sx2);
      if (s0 != 0.0f) {
        r0 = -(ixc + sx / s0 / 2);
        const float sigma = sqrtf(s0 * sx2 - sx * sx) / s0 / 2, eff = sigma * cm_norm;
        r1 = s0 / (eff * eff);
      }
    }
    if (lane < 4) rec[lane] = (lane == 0) ? r0 : ((lane == 1) ? r1 : CUDART_NAN_F);
    __syncwarp();
  }
}

// tiles without a main-camera task keep {NaN, 0, NaN, NaN}
__global__ void rig_init_kernel(float *rig_rec, int ntiles) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ntiles * 4) rig_rec[i] = ((i & 3) == 1) ? 0.f : CUDART_NAN_F;
}

cudaError_t launch_rig(const SceneDev &mn, const SceneDev &ax, const CorrConst &cc, float *rig_corr, float *rig_rec,
                       float cm_norm, int no_int_x0, cudaStream_t st) {
  const int ntiles = mn.tilesX * mn.tilesY;
  rig_init_kernel<<<(ntiles * 4 + 255) / 256, 256, 0, st>>>(rig_rec, ntiles);
  if (mn.num_tasks <= 0) return cudaGetLastError();
  const int C = mn.num_colors;
  const int RE = (cc.strip_rows < cc.wndy_size ? cc.strip_rows : cc.wndy_size) * 15;
  const int per_warp = ((2 * C * TP_CLT + SCR) + 3) & ~3, nw = 4, bytes = per_warp * nw * 4;
  const int units = (mn.num_tasks + nw - 1) / nw;
  auto go = [&](auto kernel) -> cudaError_t {
    int res = 0;
    const cudaError_t e = kernel_residency((const void *)kernel, nw * 32, bytes, &res);
    if (e != cudaSuccess) return e;
    if (res < 1) return cudaErrorInvalidConfiguration;
    const int grid = units < res ? units : res;
    kernel<<<grid, nw * 32, bytes, st>>>(mn, ax, cc, rig_corr, rig_rec, cm_norm, no_int_x0, per_warp);
    return cudaGetLastError();
  };
  if (RE <= 32) return C == 3 ? go(rig_kernel<3, 1>) : go(rig_kernel<1, 1>);
  return C == 3 ? go(rig_kernel<3, 8>) : go(rig_kernel<1, 8>);
}

// ---------------------------------------------------------------------------
// IMCLT (ImageDtt.iclt_2d, the reference GPU imclt_rbg) with overlap-add into the
// padded colour frames.  CTA = one region of IR x IR blocks of 8x8 pixels of one (sensor, colour)
// plane; the (IR + 1)^2 tiles touching it are processed in the four tile-parity phases
// (tiles of one phase never overlap), so the region accumulates in shared memory
// without atomics and in a fixed order.  A warp carries 4 tiles at once, one per
// 8-lane group, lane r owning row r of each quadrant; the transforms carry quadrants m and m + 2
// two values per instruction.
// 12 planes of 1296x968 and of 640x480: 113 and 38.6 us with scalar transforms, 14 x 14 blocks and nine warps, 108
// and 33.7 with these; 12 and seven 107 and 32.6, 10 and five 105 and 30.7, 8 and seven 116 and 32.0.  What bounds
// it: the phases' barriers and the latency of each phase's first loads.
// ---------------------------------------------------------------------------
// dct4_fast (tp_dtt.cuh) of two rows, the same operations
__device__ __forceinline__ void dct4_two(const float2 x[8], float2 y[8]) {
  const float2 C18 = dup2(1.3065629648763766f), C38 = dup2(0.5411961001461970f), N18 = dup2(-1.3065629648763766f),
               SQ2 = dup2(1.4142135623730951f);
  float2 u0[4], u1[4], v0[4], v1[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    u0[j] = fma2(dup2(k_d4c[j]), x[j], mul2(dup2(k_d4s[j]), x[7 - j]));
    // the odd ones negated in their factors
    const float sg = (j & 1) ? -1.f : 1.f;
    u1[j] = fma2(dup2(sg * k_d4c[3 - j]), x[4 + j], mul2(dup2(-sg * k_d4s[3 - j]), x[3 - j]));
  }
  {
    const float2 a0 = add2(u0[0], u0[3]), a1 = add2(u0[1], u0[2]), b0 = sub2(u0[0], u0[3]), b1 = sub2(u0[1], u0[2]);
    v0[0] = add2(a0, a1); v0[2] = sub2(a0, a1);
    v0[1] = fma2(C18, b0, mul2(C38, b1)); v0[3] = fma2(C38, b0, mul2(N18, b1));
  }
  {
    const float2 a0 = add2(u1[0], u1[3]), a1 = add2(u1[1], u1[2]), b0 = sub2(u1[0], u1[3]), b1 = sub2(u1[1], u1[2]);
    v1[0] = add2(a0, a1); v1[2] = sub2(a0, a1);
    v1[1] = fma2(C18, b0, mul2(C38, b1)); v1[3] = fma2(C38, b0, mul2(N18, b1));
  }
  y[0] = mul2(SQ2, v0[0]);
  y[7] = mul2(SQ2, v1[0]);
  y[2] = add2(v0[1], v1[3]);
  y[4] = sub2(v0[2], v1[2]);
  y[6] = add2(v0[3], v1[1]);
  y[1] = sub2(v0[1], v1[3]);
  y[3] = add2(v0[2], v1[2]);
  y[5] = sub2(v0[3], v1[1]);
}

constexpr int IMCLT_IR = 10;      // region = IR x IR blocks of 8x8 pixels
constexpr int IMCLT_WARPS = 5;    // the four parity phases (25, 30, 30, 36 tiles), four tiles a warp, in two rounds each
constexpr int IMCLT_SMALL = 152;  // regions for a region on each of the chip's SMs

template <int IR, int NW>
__global__ void __launch_bounds__(32 * NW) imclt_fast_kernel(const __grid_constant__ SceneDev sc) {
  constexpr int IPX = IR * 8, ISTR = IPX + 1;
  extern __shared__ float acc[];  // [IPX][ISTR]
  __shared__ float2 tbuf_all[NW][4 * 72];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3, r = lane & 7;
  const int S = sc.num_sensors, C = sc.num_colors;
  const int plane = blockIdx.z, s = plane / C, c = plane - s * C;
  const int bx0 = blockIdx.x * IR, by0 = blockIdx.y * IR;
  const int fw = sc.width + 8, fh = sc.height + 8;
  for (int i = threadIdx.x; i < IPX * ISTR; i += 32 * NW) acc[i] = 0.f;
  __syncthreads();
  float2 *tbuf = tbuf_all[warp] + q * 72;
  // (a stored CLT that already carries the LPF, clt_lpf_mask, is not filtered again)
  const float *lpf = (sc.lpf_rbg && !((sc.clt_lpf_mask >> c) & 1)) ? sc.lpf_rbg + c * 64 : nullptr;
  // unfold rows fed by source row r (DttRad2.get_unfold_index_signs, 392-404)
  const int i1 = (r >= 4) ? r - 4 : 11 - r, i2 = (r >= 4) ? 11 - r : r + 12;
  const float sa1 = (r >= 4) ? 1.f : -1.f, sb1 = 1.f;    // signs (cos, sin branch) of row i1
  const float sa2 = -1.f, sb2 = (r >= 4) ? 1.f : -1.f;   // signs of row i2
  const float w1 = k_hwin[i1 < 8 ? i1 : 15 - i1], w2 = k_hwin[i2 < 8 ? i2 : 15 - i2];
  // the DST-IV of quadrants 2 and 3 in the first pass leaves the odd rows negative: sg
  const float sg = (r & 1) ? -1.f : 1.f;
  const float kc1 = sa1 * w1, ks1 = sg * sb1 * w1, kc2 = sa2 * w2, ks2 = sg * sb2 * w2;
  float lk[8];  // 0.25 x the colour's LPF for row r (the iclt_2d scale)
#pragma unroll
  for (int v = 0; v < 8; v++) lk[v] = 0.25f * (lpf ? lpf[r * 8 + v] : 1.0f);
#pragma unroll 1
  for (int ph = 0; ph < 4; ph++) {
    const int pxp = ph & 1, pyp = ph >> 1;
    int tx0 = bx0 - 1, ty0 = by0 - 1;
    if ((tx0 & 1) != pxp) tx0++;
    if ((ty0 & 1) != pyp) ty0++;
    const int ntx = (bx0 + IR - 1 - tx0) / 2 + 1, nty = (by0 + IR - 1 - ty0) / 2 + 1;
#pragma unroll 1
    for (int k0 = warp * 4; k0 < ntx * nty; k0 += 4 * NW) {
      const int k = k0 + q;
      const int tx = tx0 + 2 * (k % ntx), ty = ty0 + 2 * (k / ntx);
      bool act = k < ntx * nty && tx >= 0 && ty >= 0 && tx < sc.tilesX && ty < sc.tilesY;
      const size_t tile = act ? (size_t)ty * sc.tilesX + tx : 0;
      if (act && sc.tile_task[tile] < 0) act = false;
      const float *src = sc.clt + ((tile * S + s) * C + c) * TP_CLT + r * 8;
      // inverse 2D DCT-IV/DST-IV with the swapped mode (ImageDtt.java:3628): rows (vertical frequency) first,
      // then columns; DST-IV(x)[k] = (-1)^k DCT-IV(reversed x)[k]
      float2 p[2][8];  // quadrants (0, 2) and (1, 3): vertical position r, horizontal positions
#pragma unroll
      for (int m = 0; m < 2; m++) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, d = a, e = a;
        if (act) {
          a = __ldg((const float4 *)(src + m * 64));
          b = __ldg((const float4 *)(src + m * 64 + 4));
          d = __ldg((const float4 *)(src + m * 64 + 128));
          e = __ldg((const float4 *)(src + m * 64 + 132));
        }
        p[m][0] = make_float2(a.x * lk[0], e.w * lk[7]);
        p[m][1] = make_float2(a.y * lk[1], e.z * lk[6]);
        p[m][2] = make_float2(a.z * lk[2], e.y * lk[5]);
        p[m][3] = make_float2(a.w * lk[3], e.x * lk[4]);
        p[m][4] = make_float2(b.x * lk[4], d.w * lk[3]);
        p[m][5] = make_float2(b.y * lk[5], d.z * lk[2]);
        p[m][6] = make_float2(b.z * lk[6], d.y * lk[1]);
        p[m][7] = make_float2(b.w * lk[7], d.x * lk[0]);
      }
#pragma unroll
      for (int m = 0; m < 2; m++) {
        float2 z[8];
        dct4_two(p[m], z);
#pragma unroll
        for (int j = 0; j < 8; j++) tbuf[j * 9 + r] = z[j];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; j++) z[j] = tbuf[r * 9 + (m ? 7 - j : j)];
        __syncwarp();
        dct4_two(z, p[m]);  // quadrants 1 and 3: the odd positions are negative
      }
      // unfold (DttRad2.unfold_tile) into rows i1, i2 and accumulate
      const int gx0 = (tx - bx0) * 8, gy1 = (ty - by0) * 8 + i1, gy2 = (ty - by0) * 8 + i2;
      const bool left = act && gx0 >= 0, right = act && gx0 + 8 < IPX;  // the tile's halves lie in the region
      const bool r1 = gy1 >= 0 && gy1 < IPX, r2 = gy2 >= 0 && gy2 < IPX;
      float *a1 = acc + gy1 * ISTR + gx0, *a2 = acc + gy2 * ISTR + gx0;
#pragma unroll
      for (int jj = 0; jj < 16; jj++) {
        const int seg = jj >> 2, xx = jj & 3;
        const int ih = (seg == 0) ? xx + 4 : ((seg == 1) ? 7 - xx : ((seg == 2) ? 3 - xx : xx));
        const float hs1 = (seg == 0) ? 1.f : -1.f, hs2 = ((seg == 3) != ((ih & 1) != 0)) ? -1.f : 1.f;
        const float wh = k_hwin[jj < 8 ? jj : 15 - jj];
        const float2 ab = fma2(dup2(hs2 * wh), p[1][ih], mul2(dup2(hs1 * wh), p[0][ih]));
        const bool in = jj < 8 ? left : right;
        if (in && r1) a1[jj] += fmaf(ks1, ab.y, kc1 * ab.x);
        if (in && r2) a2[jj] += fmaf(ks2, ab.y, kc2 * ab.x);
      }
    }
    __syncthreads();
  }
  float *dst = sc.rbg + (size_t)plane * fw * fh + bx0 * 8;
  for (int ly = warp; ly < IPX && by0 * 8 + ly < fh; ly += NW) {
    float *row = dst + (size_t)(by0 * 8 + ly) * fw;
    for (int lx = lane; lx < IPX && bx0 * 8 + lx < fw; lx += 32) row[lx] = acc[ly * ISTR + lx];
  }
}

template <int IR, int NW>
static cudaError_t go_imclt(const SceneDev &sc, cudaStream_t st) {
  const int bytes = IR * 8 * (IR * 8 + 1) * 4;
  const cudaError_t e = cudaFuncSetAttribute(imclt_fast_kernel<IR, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  const dim3 grid((sc.tilesX + 1 + IR - 1) / IR, (sc.tilesY + 1 + IR - 1) / IR, sc.num_sensors * sc.num_colors);
  imclt_fast_kernel<IR, NW><<<grid, 32 * NW, bytes, st>>>(sc);
  return cudaGetLastError();
}

cudaError_t launch_imclt_fast(const SceneDev &sc, cudaStream_t st) {
  // Regions of 10 x 10 blocks need the fewest repeated tiles among the sizes with enough warps an SM; where they
  // would leave SMs without one, 6 x 6 (four mono planes of 128x96: 14 us and 9 us; 12 planes of 1296x968: 105 us
  // and 109 us).
  const int regions = ((sc.tilesX + IMCLT_IR) / IMCLT_IR) * ((sc.tilesY + IMCLT_IR) / IMCLT_IR) * sc.num_sensors * sc.num_colors;
  return regions < IMCLT_SMALL ? go_imclt<6, 4>(sc, st) : go_imclt<IMCLT_IR, IMCLT_WARPS>(sc, st);
}

__global__ void disp_init_kernel(float *disp, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n * TP_NDISP) {
    int k = i % TP_NDISP;
    disp[i] = (k == 2 || k == 4 || k == 6) ? 0.0f : CUDART_NAN_F;
  }
}

// The records of tiles outside the task list; a forward writes all of its tasks' records, so where a
// task list made from tile ops (no tile twice) holds every tile there is nothing to do.
static cudaError_t init_records(const SceneDev &sc, cudaStream_t st) {
  const int ntiles = sc.tilesX * sc.tilesY;
  if (sc.ports_from_geometry && sc.num_tasks == ntiles) return cudaSuccess;
  disp_init_kernel<<<(ntiles * TP_NDISP + 255) / 256, 256, 0, st>>>(sc.disp, ntiles);
  return cudaGetLastError();
}

cudaError_t upload_fused_constants() { return upload_dtt_constants(); }

// GPU_DTT24_DRV (dtt8x8.cuh:100-158): every 8x8 block of a float image through the 2D transform of
// one mode, rows first (bit 0: DST), then columns (bit 1); modes 0-3 DCT-IV / DST-IV, 4-7 the
// orthonormal DCT-II / DST-II (the DCT-IIe butterflies with the constant term scaled by 1/sqrt 2).
// An 8-lane group per block, lane r holding row r, then column r after the transpose.
__device__ __forceinline__ void dtt8_mode(const float x[8], float y[8], int mode, bool sine) {
  if (mode < 4) {
    dtt4_fast(x, y, sine);
  } else {
    dtt2e_fast(x, y, sine);
    if (sine) y[7] *= 0.70710678118654752f;
    else y[0] *= 0.70710678118654752f;
  }
}

__global__ void __launch_bounds__(128) dtt8x8_kernel(float *dst, const float *src, int stride, int bw, int nblocks,
                                                     int mode) {
  __shared__ float tb[16][72];
  const int g = threadIdx.x >> 3, r = threadIdx.x & 7;
  const int blk = blockIdx.x * 16 + g;
  const bool act = blk < nblocks;
  const int b = act ? blk : nblocks - 1;  // every group takes part in the warp's transposes
  const int by = b / bw, bx = b - by * bw;
  const float *s = src + (size_t)(by * 8 + r) * stride + bx * 8;
  float x[8], y[8];
#pragma unroll
  for (int c = 0; c < 8; c++) x[c] = s[c];
  dtt8_mode(x, y, mode, mode & 1);
  group_transpose(y, tb[g], r);
  dtt8_mode(y, x, mode, (mode >> 1) & 1);
  group_transpose(x, tb[g], r);
  if (act) {
    float *d = dst + (size_t)(by * 8 + r) * stride + bx * 8;
#pragma unroll
    for (int c = 0; c < 8; c++) d[c] = x[c];
  }
}

cudaError_t launch_dtt8x8(float *dst, const float *src, int stride, int width, int height, int mode,
                          cudaStream_t st) {
  const int bw = width / 8, nblocks = bw * (height / 8);
  if (nblocks <= 0) return cudaSuccess;
  dtt8x8_kernel<<<(nblocks + 15) / 16, 128, 0, st>>>(dst, src, stride, bw, nblocks, mode);
  return cudaGetLastError();
}

static FwdShape make_shape(const SceneDev &sc, int nw) {
  FwdShape f;
  f.S = sc.num_sensors;
  f.C = sc.num_colors;
  f.P = sc.num_pairs;
  // only the strip rows the extraction reads are built: getMaxXYInt uses row 0 and
  // getMaxXCm clips the strip to the y-window (Correlation2d.java:944-951)
  f.RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  f.quad = (sc.num_pairs <= 8) ? 1 : 0;
  f.nw = nw > 0 ? nw : 4;  // the autotuner's pick on 4x2592x1936 Bayer and 4x512x384 mono
  f.clt_floats = f.S * f.C * TP_CLT;
  f.per_warp = f.clt_floats + SCR;
  f.per_warp = (f.per_warp + 3) & ~3;
  return f;
}

static int split_smem_floats(const FwdShape &f) { return f.clt_floats + f.nw * SCR + f.nw * 240; }

template <typename K>
static cudaError_t launch_persistent(K kernel, int threads, int bytes, int units, const SceneDev &sc,
                                     const FwdShape &f, const CorrConst &cc, cudaStream_t st) {
  int res = 0;
  const cudaError_t e = kernel_residency((const void *)kernel, threads, bytes, &res);
  if (e != cudaSuccess) return e;
  if (res < 1) return cudaErrorInvalidConfiguration;
  const int grid = units < res ? units : res;
  kernel<<<grid, threads, bytes, st>>>(sc, f, cc);
  return cudaGetLastError();
}

// Schedules: tiles_per_block == warps_per_block (<= 4): warp per tile;
// tiles_per_block == 1 with warps_per_block 2, 3 or 4: pair per warp (CTA per tile).
cudaError_t launch_fused_forward(const SceneDev &sc, const CorrConst &cc, int tpb, int nw, cudaStream_t st) {
  cudaError_t e = init_records(sc, st);
  if (e != cudaSuccess || sc.num_tasks <= 0) return e;
  if (sc.strip_rows * 15 > 8 * 32) return cudaErrorInvalidConfiguration;
  if (tpb <= 0 && nw <= 0 && sc.num_pairs > 8) {  // default for many pairs: four warps share a tile
    tpb = 1;
    nw = 4;
  }
  FwdShape f = make_shape(sc, nw);
  if (f.nw > 4) return cudaErrorInvalidConfiguration;
  if (tpb == 1 && f.nw == 4 && many_forward_ok(sc)) return launch_many_forward(sc, cc, st);
  if (tpb == 1 && f.nw > 1) {
    const int bytes = split_smem_floats(f) * 4;
    if (f.nw == 3) {  // quad colour scenes: one colour item per warp, 8 CTAs per SM
      if (f.RE <= 32)
        return sc.num_colors == 3
                   ? launch_persistent(fused_split_kernel<3, 1, 96, 8>, 96, bytes, sc.num_tasks, sc, f, cc, st)
                   : launch_persistent(fused_split_kernel<1, 1, 96, 8>, 96, bytes, sc.num_tasks, sc, f, cc, st);
      return sc.num_colors == 3
                 ? launch_persistent(fused_split_kernel<3, 8, 96, 8>, 96, bytes, sc.num_tasks, sc, f, cc, st)
                 : launch_persistent(fused_split_kernel<1, 8, 96, 8>, 96, bytes, sc.num_tasks, sc, f, cc, st);
    }
    if (f.RE <= 32)
      return sc.num_colors == 3
                 ? launch_persistent(fused_split_kernel<3, 1>, f.nw * 32, bytes, sc.num_tasks, sc, f, cc, st)
                 : launch_persistent(fused_split_kernel<1, 1>, f.nw * 32, bytes, sc.num_tasks, sc, f, cc, st);
    return sc.num_colors == 3
               ? launch_persistent(fused_split_kernel<3, 8>, f.nw * 32, bytes, sc.num_tasks, sc, f, cc, st)
               : launch_persistent(fused_split_kernel<1, 8>, f.nw * 32, bytes, sc.num_tasks, sc, f, cc, st);
  }
  if (quad_forward_ok(sc)) return launch_quad_forward(sc, cc, f.nw, st);
  const int bytes = f.per_warp * f.nw * 4;
  const int units = (sc.num_tasks + f.nw - 1) / f.nw;
  bool all16 = true;
  for (int i = 0; i < sc.num_sensors; i++) all16 = all16 && sc.img_dtype[i] == 1;
  auto go = [&](auto kernel) { return launch_persistent(kernel, f.nw * 32, bytes, units, sc, f, cc, st); };
  const bool one = f.RE <= 32;
  if (sc.num_colors == 3 && sc.num_sensors <= 4 && all16 && sc.sprod && sc.osum) {  // staged windows
    // the extraction's serial half in its own pass
    e = one ? go(fused_forward_win_kernel<1>) : go(fused_forward_win_kernel<8>);
    return e != cudaSuccess ? e : launch_extract_pass(sc, cc, f.quad, f.RE, st);
  }
  if (sc.num_colors == 3) return one ? go(fused_forward_kernel<3, 1>) : go(fused_forward_kernel<3, 8>);
  return one ? go(fused_forward_kernel<1, 1>) : go(fused_forward_kernel<1, 8>);
}
