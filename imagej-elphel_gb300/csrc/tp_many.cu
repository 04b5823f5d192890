// tp_many.cu -- the forward of mono scenes with many general pairs (16 sensors, 120 pairs).
//
// A CTA of four warps shares one tile's CLT, as fused_split_kernel's: the warps take a group of four
// sensors each, then every fourth pair.  Nearly all the time is the pair phase, which is bound by
// instruction issue and the shared-memory pipe, so here a warp takes two of its pairs at once, one in
// each half of the packed FP32 registers (tp_pairs.cuh); a surface goes to HBM by a bulk copy instead
// of eight loads and stores; the strip taps, the same for every tile, are read from a table instead of
// computed (CorrDev::gen_tap); the image windows are staged (tp_forward.cuh); and the extraction is a
// pass of its own, where here three warps would wait for the fourth.
// Results are the same bits: every warp's pairs are summed in the same order.
// Measured on 16x640x512 (5,120 tiles): 500 -> 380 us; 480 warp instructions a pair (677 before), the
// surfaces' 553 MB alone take 81 us; 375 with the windows 8 banks apart, 370 with a first sensor that both pairs
// share (more than half of the couples) read once.  What bounds it now: the shared-memory pipe (78 %).
#include "tp_forward.cuh"
#include "tp_launch.h"
#include "tp_pairs.cuh"

namespace {

constexpr int MANY_NW = 4;
// CTAs per SM: the pairs are chains of shared-memory reads, shuffles and dependent arithmetic, so warps
// count more than registers (16x640x512: 4 CTAs of 118 registers 462 us, 6 of 80 380 us; the windows
// share the pair buffers' space so that six fit)
constexpr int MANY_CTAS = 6;
constexpr int MANY_SURF = 228;                            // a surface and up to 3 floats of misalignment
constexpr int MANY_WIN = 4 * Stage<false>::WIN;           // floats of a warp's four windows
constexpr int MANY_WARP = MANY_WIN;                       // a warp's space: windows, then pair buffers
static_assert(QP_BUF + 2 * MANY_SURF <= MANY_WARP, "pair buffers");
__host__ __device__ constexpr int many_floats(int S) {    // CLT, the warps' space, partial strips
  return ((S + 3) / 4) * 4 * TP_CLT + MANY_NW * (MANY_WARP + 32);
}

// a 15x15 surface (in shared memory at its global address modulo 16) to HBM
__device__ __forceinline__ void store_surface(float *g, const float *s, int mis, int lane) {
  const int head = (4 - mis) & 3, body = (225 - head) & ~3;
  if (lane == 0) bulk_store(g + head, s + head, body * 4);
  const int i = lane < 4 ? lane : head + body + lane - 4;  // lanes 0-3 the head, 4-7 the tail
  if (lane < 4 ? i < head : (lane < 8 && i < 225)) g[i] = s[i];
}

// the normalised, filtered spectra of two pairs into b (interleaved [4][8][9]); the pairs are numbered by their first
// sensor, which two that lie four apart mostly share
__device__ __forceinline__ void couple_spectra(const CorrConst &cfg, const PairDev &pa, const PairDev &pb, float2 l0,
                                               float2 l1, const float *s_clt, float2 *b, int lane) {
  const float *a1 = s_clt + pa.cam1 * TP_CLT + lane, *a2 = s_clt + pa.cam2 * TP_CLT + lane;
  const float *b1 = s_clt + pb.cam1 * TP_CLT + lane, *b2 = s_clt + pb.cam2 * TP_CLT + lane;
  float2 d1[2][4], d2[2][4], amp[2];
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int o = m * 64 + 32 * h;
      d1[h][m] = dup2(a1[o]);
      d2[h][m] = make_float2(a2[o], b2[o]);
    }
  if (pa.cam1 != pb.cam1) {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int m = 0; m < 4; m++) d1[h][m].y = b1[m * 64 + 32 * h];
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    float2 s1 = mul2(d1[h][0], d1[h][0]), s2 = mul2(d2[h][0], d2[h][0]);
#pragma unroll
    for (int m = 1; m < 4; m++) {
      s1 = fma2(d1[h][m], d1[h][m], s1);
      s2 = fma2(d2[h][m], d2[h][m], s2);
    }
    const float2 pr = mul2(s1, s2);
    amp[h] = make_float2(amp_of(pr.x), amp_of(pr.y));
  }
  const float2 fzs = warp_sum2(add2(amp[0], amp[1]), lane, 1.0f / 64, cfg.fat_zero);
  const int off = (lane >> 3) * 9 + (lane & 7);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const float2 den = fma2(fzs, dup2(cfg.fat_zero), amp[h]);
    const float2 sw = make_float2(__fdividef(1.0f, den.x), __fdividef(1.0f, den.y));
    float2 n[4], t[4];
#pragma unroll
    for (int m = 1; m < 4; m++) n[m] = neg2(d1[h][m]);
    clt_products(d1[h], n, d2[h], t);
#pragma unroll
    for (int m = 0; m < 4; m++) b[m * 72 + 36 * h + off] = mul2(mul2(t[m], sw), h ? l1 : l0);
  }
  __syncwarp();
}

}  // namespace

// U16: image type of every sensor.  RE <= 32.
template <bool U16>
__global__ void __launch_bounds__(32 * MANY_NW, MANY_CTAS) many_kernel(const __grid_constant__ SceneDev sc,
                                                               const __grid_constant__ CorrConst cfg, int RE) {
  extern __shared__ float sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3, r = lane & 7;
  const int S = sc.num_sensors, P = sc.num_pairs, groups = (S + 3) >> 2;
  float *s_clt = sm;
  float *wb = sm + groups * 4 * TP_CLT + warp * MANY_WARP;
  float2 *buf = (float2 *)wb;
  float *part = sm + groups * 4 * TP_CLT + MANY_NW * MANY_WARP;  // [4][32] log sums of the warps' pairs
  const float2 l0 = dup2(0.25f * cfg.lpf[lane]), l1 = dup2(0.25f * cfg.lpf[lane + 32]);
  const int s = min(warp * 4 + q, S - 1);  // the sensor whose window and CLT this lane works on
  const bool act = warp * 4 + q < S, has_group = warp < groups;
  // where the task's products go, carried along: worked out at the store it cost 4 us in 16x640x512 (422.7 and
  // 419.6 us a pass; by tile as the surfaces 419.0)
  float *out = sc.sprod + (size_t)blockIdx.x * RE + lane;
  for (int task = blockIdx.x; task < sc.num_tasks; task += gridDim.x, out += (size_t)gridDim.x * RE) {
    const int txy = sc.task_txy[task];
    const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
    if (has_group) {
      const SubtilePlan p = sc.plan[(size_t)task * S + s];
      if (lane == 0) bulk_read_done();  // the windows go over the last surfaces
      __syncwarp();
      stage_window<U16>(sc, sc.images[s], p.tlx, p.tly, wb + q * Stage<U16>::WIN, r);
      cp_async_commit();
      SWin<U16> w;
      w.base = (const typename Stage<U16>::T *)(wb + q * Stage<U16>::WIN);
      w.sx = p.tlx & (Stage<U16>::CH - 1);
      w.scale = sc.color_scale[0];
      cp_async_wait_all();
      __syncwarp();
      float o[4][8];
      subtile_clt<0>(w, p.rx, p.ry, 0, 0, 0, r, wb + q * 72, o);
      conv_shift(o, (p.kidx >= 0) ? sc.kernels[s] + (size_t)p.kidx * TP_CLT : nullptr, p.rx, p.ry, r);
      if (act) {
        float *sdst = s_clt + s * TP_CLT + r * 8;
#pragma unroll
        for (int m = 0; m < 4; m++) {
          *(float4 *)(sdst + m * 64) = make_float4(o[m][0], o[m][1], o[m][2], o[m][3]);
          *(float4 *)(sdst + m * 64 + 4) = make_float4(o[m][4], o[m][5], o[m][6], o[m][7]);
        }
        store_clt(sc, 0, r, sc.clt + (tile * S + s) * TP_CLT + r * 8, o);
      }
    }
    __syncthreads();
    float cmb = 0.f;
#pragma unroll 1
    for (int pi = warp; pi < P; pi += 2 * MANY_NW) {
      // pairs pi and pi + 4 (the last one alone: taken twice, used once)
      const bool two = pi + MANY_NW < P;
      const int pj = two ? pi + MANY_NW : pi;
      // their taps are read ahead of the arithmetic
      const float4 ta = __ldg((const float4 *)sc.corr_cfg->gen_tap[pi] + lane), tb = __ldg((const float4 *)sc.corr_cfg->gen_tap[pj] + lane);
      const int ca = __ldg(sc.corr_cfg->gen_cell[pi] + lane), cb = __ldg(sc.corr_cfg->gen_cell[pj] + lane);
      couple_spectra(cfg, cfg.pairs[pi], cfg.pairs[pj], l0, l1, s_clt, buf, lane);
      if (lane == 0) bulk_read_done();  // the surfaces before these are out
      const size_t ga = tile * P + pi, gb = tile * P + pj;
      float *sa = wb + QP_BUF + (ga & 3), *sb = wb + QP_BUF + MANY_SURF + (gb & 3);
      couple_surfaces(buf, sa, sb, lane);
      bulk_fence();
      __syncwarp();
      store_surface(sc.corr + ga * TP_CORR, sa, (int)(ga & 3), lane);
      if (two) store_surface(sc.corr + gb * TP_CORR, sb, (int)(gb & 3), lane);
      const bool both = lane >= 15;  // strip rows below the first average two sides
      const float da = tap_strip(sa, ta, ca, both), db = tap_strip(sb, tb, cb, both);
      float va = da + cfg.corr_offset, vb = db + cfg.corr_offset;
      if (va < 0.0f) va = 0.0f;
      if (vb < 0.0f) vb = 0.0f;
      const float ga_log = logf(va), gb_log = logf(vb);
      if (cfg.pairs[pi].in_combo) {
        if (sc.strips && lane < RE) sc.strips[ga * RE + lane] = da;  // kept for the adjoint
        cmb += ga_log;
      }
      if (two && cfg.pairs[pj].in_combo) {
        if (sc.strips && lane < RE) sc.strips[gb * RE + lane] = db;
        cmb += gb_log;
      }
      __syncwarp();
    }
    part[warp * 32 + lane] = cmb;
    __syncthreads();  // also: every warp has read the CLT
    if (warp == 0 && lane < RE) {
      float v = part[lane];
      for (int w2 = 1; w2 < MANY_NW; w2++) v += part[w2 * 32 + lane];
      *out = v;
    }
  }
  if (lane == 0) bulk_done();
}

cudaError_t upload_many_constants() { return upload_dtt_constants(); }

// mono, more than 8 pairs, all of kind 4, images of one type, a strip of at most 32 entries
bool many_forward_ok(const SceneDev &sc) {
  const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  for (int i = 1; i < sc.num_sensors; i++)
    if (sc.img_dtype[i] != sc.img_dtype[0]) return false;
  return sc.num_colors == 1 && sc.num_pairs > 8 && sc.all_general && RE <= 32 && sc.sprod;
}

cudaError_t launch_many_forward(const SceneDev &sc, const CorrConst &cc, cudaStream_t st) {
  const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  const int bytes = many_floats(sc.num_sensors) * 4;
  auto go = [&](auto kernel) -> cudaError_t {
    int res = 0;
    const cudaError_t e = kernel_residency((const void *)kernel, 32 * MANY_NW, bytes, &res);
    if (e != cudaSuccess) return e;
    if (res < 1) return cudaErrorInvalidConfiguration;
    kernel<<<sc.num_tasks < res ? sc.num_tasks : res, 32 * MANY_NW, bytes, st>>>(sc, cc, RE);
    return cudaGetLastError();
  };
  const cudaError_t e = sc.img_dtype[0] == 1 ? go(many_kernel<true>) : go(many_kernel<false>);
  return e != cudaSuccess ? e : launch_extract_pass(sc, cc, 0, RE, st);
}
