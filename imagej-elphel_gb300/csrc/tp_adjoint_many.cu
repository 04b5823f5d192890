// tp_adjoint_many.cu -- the adjoint's per-tile kernel for mono scenes with many general pairs.
//
// The same chain as adjoint_kernel (tp_adjoint.cu), whose time is the pairs: about 900 warp instructions
// a pair, in chains of shared-memory accesses and dependent arithmetic at 16 warps an SM.  Here a warp
// takes two pairs at once, one in each half of the packed FP32 registers, so a round holds up to eight
// pairs on distinct sensors (16 sensors: 15 rounds of 8); the strip taps come from the forward's table;
// and the windows of the shift derivatives are staged (tp_forward.cuh).
// Needs the forward's strip samples (SceneDev::strips, recorded or sampled again) and a strip of at most 32 entries.
// Measured on 16x640x512 (5,120 tiles, 120 pairs): 992 -> 640 us; 617 with the windows over a group's CLT once it is
// read, which leaves room for a fifth CTA an SM (96 registers; with 128 and four CTAs 643).  What bounds it
// now: the shared-memory pipe (about 70 %: the pairs' CLT reads and gradient updates are 96 of some 350 accesses a
// couple) and the latency of those accesses at 20 warps an SM (32 KB of CLT and gradient a tile).
#include "tp_adjoint_pairs.cuh"
#include "tp_launch.h"

namespace {

constexpr int AM_WARP = QP_BUF;  // a warp's space: the gradients of its two pairs' surfaces, over them the spectra
static_assert(2 * AM_SURF <= AM_WARP, "a warp's space");
// at the end a group's windows: three over its CLT, the last one in the warp's space
static_assert(3 * Stage<false>::WIN <= 4 * TP_CLT && Stage<false>::WIN <= AM_WARP, "a group's windows");
__host__ __device__ constexpr int am_floats(int S) {  // CLT and its gradient, strip, the warps' space
  return ((S + 3) / 4) * 8 * TP_CLT + 64 + AD_NW * AM_WARP;
}

// The strip gradients of two pairs (lanes 0-14 the first's, lanes 16-30 the second's) spread into the
// pairs' surface gradients g[2][228]: the first row's entries (f0), then the second row's (f1) two sides.
__device__ __forceinline__ void scatter_strips(float *g, float f0, float f1, const CorrDev &cd, int pair, int lane) {
  const int j = min(lane & 15, 14);
  float *gp = g + (lane >> 4) * AM_SURF;
  const float4 t0 = __ldg((const float4 *)cd.gen_tap[pair] + j), t1 = __ldg((const float4 *)cd.gen_tap[pair] + 15 + j);
  const int c0 = __ldg(cd.gen_cell[pair] + j), c1 = __ldg(cd.gen_cell[pair] + 15 + j);
  const int last = max((c0 >> 26) & 15, __shfl_xor_sync(0xffffffffu, (c0 >> 26) & 15, 16));  // over both pairs
  add_entry(gp + (c0 & 255), f0, f0 != 0.f && !(c0 & 0x10000), t0.x, t0.y, (c0 >> 18) & 15, last);
  const float h = 0.5f * f1;
  add_entry(gp + (c1 & 255), h, f1 != 0.f && !(c1 & 0x10000), t1.x, t1.y, (c1 >> 18) & 15, last);
  add_entry(gp + ((c1 >> 8) & 255), h, f1 != 0.f && !(c1 & 0x20000), t1.z, t1.w, (c1 >> 22) & 15, last);
}

}  // namespace

template <bool U16>
__global__ void __launch_bounds__(32 * AD_NW, 5) adjoint_many_kernel(const __grid_constant__ SceneDev sc,
                                                                     const __grid_constant__ CorrConst cfg, int RE,
                                                                     float *sens, float *dval) {
  extern __shared__ float sm[];
  __shared__ float s_d;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 3, r = lane & 7;
  const int S = sc.num_sensors, P = sc.num_pairs, groups = (S + 3) >> 2;
  float *s_clt = sm;                              // [groups * 4][256]
  float *s_g = s_clt + groups * 4 * TP_CLT;       // the same, dd/dCLT
  float *gcmb = s_g + groups * 4 * TP_CLT;        // [32] dd/dcombo
  float *gG = gcmb + 32;                          // [32] combo, then combo + offset
  float *wb = gG + 32 + warp * AM_WARP;
  float2 *buf = (float2 *)wb;
  const float inv_n = 1.0f / cfg.num_combo;
  const float l0 = cfg.lpf[lane], l1 = cfg.lpf[lane + 32];
  const short *sched = &sc.corr_cfg->adj_round8[0][0];
  const int rounds = sc.corr_cfg->adj_rounds8;

  for (int task = blockIdx.x; task < sc.num_tasks; task += gridDim.x) {
    const int txy = sc.task_txy[task];
    const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
    {
      const float4 *src = (const float4 *)(sc.clt + tile * S * TP_CLT);
      for (int i = tid; i < S * 64; i += 32 * AD_NW) {
        ((float4 *)s_clt)[i] = __ldg(src + i);
        ((float4 *)s_g)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    if (warp == 0) {
      gG[lane] = lane < RE ? sc.combo[tile * RE + lane] : 0.f;
      gcmb[lane] = 0.f;
      __syncwarp();
      const float dres = strip_centroid(cfg, gG, gcmb, lane);
      if (lane < RE) gG[lane] = gG[lane] + cfg.corr_offset;  // the geometric mean the strip entries enter
      if (lane == 0) s_d = dres;
    }
    __syncthreads();
    const float dres = s_d;
    if (isnan(dres)) {
      if (tid == 0) dval[tile] = CUDART_NAN_F;
      for (int i = tid; i < 2 * S; i += 32 * AD_NW) sens[tile * 2 * S + i] = 0.f;
      __syncthreads();
      continue;
    }
    // dd/d(strip entry) of a pair = w / v: d combo / d v_p = G / (n v_p) for the geometric mean of n pairs;
    // lanes 0-14 and 16-30: entries j of the first and the second strip row
    const int j = lane & 15;
    const bool on0 = j < 15 && j < RE && gcmb[j] != 0.f, on1 = j < 15 && 15 + j < RE && gcmb[15 + j] != 0.f;
    const float w0 = on0 ? gcmb[j] * gG[j] * inv_n : 0.f, w1 = on1 ? gcmb[15 + j] * gG[15 + j] * inv_n : 0.f;
    // ---------------- reverse pass over the pairs, one round at a time ----------------
    // a warp's two pairs: lanes 0-15 load the first's strip samples, lanes 16-31 the second's, a round ahead
    short2 pn = rounds > 0 ? *(const short2 *)&sched[warp * 2] : make_short2(-1, -1);
    float n0 = 0.f, n1 = 0.f;
    auto samples = [&]() {
      const int pk = lane < 16 ? pn.x : pn.y;
      if (pk >= 0 && on0) n0 = sc.strips[(tile * P + pk) * RE + j];
      if (pk >= 0 && on1) n1 = sc.strips[(tile * P + pk) * RE + 15 + j];
    };
    samples();
#pragma unroll 1
    for (int rd = 0; rd < rounds; rd++) {
      const int pi = pn.x, pj = pn.y >= 0 ? pn.y : pn.x;
      const bool mine = lane < 16 || pn.y >= 0;
      const float v0 = n0 + cfg.corr_offset, v1 = n1 + cfg.corr_offset;
      if (rd + 1 < rounds) {
        pn = *(const short2 *)&sched[(rd + 1) * 8 + warp * 2];
        samples();
      }
      if (pi >= 0) {
        const float f0 = mine && on0 && v0 > 0.0f ? __fdividef(w0, v0) : 0.f;
        const float f1 = mine && on1 && v1 > 0.0f ? __fdividef(w1, v1) : 0.f;
        const unsigned any = __ballot_sync(0xffffffffu, f0 != 0.f || f1 != 0.f);
        if (any) {
          for (int i = lane; i < AM_SURF / 2; i += 32) ((float4 *)wb)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          __syncwarp();
          scatter_strips(wb, f0, f1, *sc.corr_cfg, lane < 16 ? pi : pj, lane);
          couple_unsurface(wb, buf, lane);
          const PairDev &pa = cfg.pairs[pi], &pb = cfg.pairs[pj];
          const int oa1 = pa.cam1 * TP_CLT + lane, oa2 = pa.cam2 * TP_CLT + lane;
          const int ob1 = pb.cam1 * TP_CLT + lane, ob2 = pb.cam2 * TP_CLT + lane;
          const bool one = any & 0xffffu, two = any >> 16;
          couple_products_grad(cfg, 1.0f, s_clt + oa1, s_clt + oa2, s_clt + ob1, s_clt + ob2, l0, l1, buf, lane,
                               [&](int h, int m, float2 x, float2 y) {  // no other pair adds to these sensors in this round
                                 const int o = m * 64 + 32 * h;
                                 if (one) {
                                   s_g[oa1 + o] += x.x;
                                   s_g[oa2 + o] += y.x;
                                 }
                                 if (two) {
                                   s_g[ob1 + o] += x.y;
                                   s_g[ob2 + o] += y.y;
                                 }
                               });
          __syncwarp();  // the spectra are read
        }
      }
      __syncthreads();
    }
    // ---------------- dd/drx, dd/dry per sensor (forward mode on the CLT) ----------------
    for (int g = warp; g < groups; g += AD_NW) {
      const int s = g * 4 + q;
      const bool act = s < S;
      const int sidx = act ? s : S - 1;
      const SubtilePlan p = sc.plan[(size_t)task * S + sidx];
      float *wq = q < 3 ? s_clt + g * 4 * TP_CLT + q * Stage<U16>::WIN : wb;
      SWin<U16> win;
      win.base = (const typename Stage<U16>::T *)wq;
      win.sx = p.tlx & (Stage<U16>::CH - 1);
      win.scale = sc.color_scale[0];
      // the group's transposes go through the sensor's CLT once it is read; a lane group beyond the last
      // sensor works on copies of the last one's slots, in slots of its own
      if (!act) {
        float4 *d = (float4 *)(s_clt + s * TP_CLT), *e = (float4 *)(s_g + s * TP_CLT);
        for (int i = r; i < 64; i += 8) {
          d[i] = ((const float4 *)(s_clt + sidx * TP_CLT))[i];
          e[i] = ((const float4 *)(s_g + sidx * TP_CLT))[i];
        }
      }
      __syncwarp();
      float gxy[2];
      shift_sens(sc, win, p, sidx, s_clt + (size_t)s * TP_CLT, s_g + (size_t)s * TP_CLT, s_clt + (size_t)s * TP_CLT, r,
                 true, gxy, [&]() {
                   stage_window<U16>(sc, sc.images[sidx], p.tlx, p.tly, wq, r);
                   cp_async_commit();
                 });
      if (r == 0 && act) {
        sens[(tile * S + s) * 2] = gxy[0];
        sens[(tile * S + s) * 2 + 1] = gxy[1];
      }
    }
    if (tid == 0) dval[tile] = dres;
    __syncthreads();
  }
}

cudaError_t upload_adjoint_many_constants() { return upload_dtt_constants(); }

// mono, more than 8 pairs, all of kind 4, images of one type, a strip of at most 32 entries, the stored CLT
bool adjoint_many_ok(const SceneDev &sc, int recompute) {
  const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  for (int i = 1; i < sc.num_sensors; i++)
    if (sc.img_dtype[i] != sc.img_dtype[0]) return false;
  return !recompute && sc.num_colors == 1 && sc.num_pairs > 8 && sc.all_general && RE <= 32;
}

cudaError_t launch_adjoint_many(const SceneDev &sc, const CorrConst &cc, float *sens, float *dval, cudaStream_t st) {
  const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  const int bytes = am_floats(sc.num_sensors) * 4;
  auto go = [&](auto kernel) -> cudaError_t {
    int res = 0;
    const cudaError_t e = kernel_residency((const void *)kernel, 32 * AD_NW, bytes, &res);
    if (e != cudaSuccess) return e;
    if (res < 1) return cudaErrorInvalidConfiguration;
    kernel<<<sc.num_tasks < res ? sc.num_tasks : res, 32 * AD_NW, bytes, st>>>(sc, cc, RE, sens, dval);
    return cudaGetLastError();
  };
  return sc.img_dtype[0] == 1 ? go(adjoint_many_kernel<true>) : go(adjoint_many_kernel<false>);
}
