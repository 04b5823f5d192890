// tp_adjoint_many.cu -- the adjoint's per-tile kernel for mono scenes with many general pairs.
//
// The same chain as adjoint_kernel (tp_adjoint.cu), whose time is the pairs: about 900 warp instructions
// a pair, in chains of shared-memory accesses and dependent arithmetic at 16 warps an SM.  Here a warp
// takes two pairs at once, one in each half of the packed FP32 registers, so a round holds up to eight
// pairs on distinct sensors (16 sensors: 15 rounds of 8); the strip taps come from the forward's table;
// and the windows of the shift derivatives are staged (tp_forward.cuh).
// Needs the forward's strip samples (SceneDev::strips) and a strip of at most 32 entries.
// Measured on 16x640x512 (5,120 tiles, 120 pairs): 992 -> 638 us.  What bounds it now: the shared-memory
// pipe (about 65 %: the pairs' CLT reads and gradient updates are 96 of some 350 accesses a couple) and
// the latency of those accesses at 16 warps an SM (32 KB of CLT and gradient a tile).
#include "tp_adjoint.cuh"
#include "tp_launch.h"
#include "tp_pairs.cuh"

namespace {

constexpr int AM_SURF = 228;                       // a pair's surface gradient (rounded to 16 bytes)
constexpr int AM_WARP = 4 * Stage<false>::WIN;     // a warp's space: the gradients of its two pairs' surfaces, over them
                                                   // the spectra; at the end its four windows
static_assert(QP_BUF <= AM_WARP && 2 * AM_SURF <= AM_WARP, "a warp's space");
__host__ __device__ constexpr int am_floats(int S) {  // CLT and its gradient, strip, the warps' space
  return ((S + 3) / 4) * 8 * TP_CLT + 64 + AD_NW * AM_WARP;
}

// x = T^T y of two rows for the DCT-IIe (sg = 1) / DST-IIe (sg = -1, y given in reverse order):
// dtt2e_transposed
__device__ __forceinline__ void dtt2e_transposed_pair(const float2 t[8], float2 x[8], float2 sg) {
  const float S = 0.5f;
  const float C4 = 0.7071067811865476f, C8 = 0.9238795325112867f, C38 = 0.3826834323650898f;
  float2 u1[4];
#pragma unroll
  for (int j = 0; j < 4; j++)
    u1[j] = fma2(dup2(k_dct2e[8 + j]), t[1],
                 fma2(dup2(k_dct2e[24 + j]), t[3], fma2(dup2(k_dct2e[40 + j]), t[5], mul2(dup2(k_dct2e[56 + j]), t[7]))));
  const float2 c4 = mul2(dup2(S * C4), t[4]);
  const float2 a0 = fma2(dup2(S), t[0], c4), a1 = fma2(dup2(S), t[0], neg2(c4));
  const float2 b0 = mul2(dup2(S), fma2(dup2(C8), t[2], mul2(dup2(C38), t[6])));
  const float2 b1 = mul2(dup2(S), fma2(dup2(C38), t[2], mul2(dup2(-C8), t[6])));
  const float2 u0[4] = {add2(a0, b0), add2(a1, b1), sub2(a1, b1), sub2(a0, b0)};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float2 p = add2(u0[j], u1[j]), m = sub2(u0[j], u1[j]);
    x[j] = (j & 1) ? mul2(p, sg) : p;
    x[7 - j] = (j & 1) ? m : mul2(m, sg);
  }
}

// One strip entry's gradient f into its four cells: the lanes in the order of their place among the lanes
// of the same cell, tap by tap, so that no two lanes meet (shared-memory float atomics are
// compare-and-swap loops: with them the kernel took 788 us on 16x640x512).  last: the largest place.
__device__ __forceinline__ void add_entry(volatile float *g, float f, bool on, float dx, float dy, int place, int last) {
  const float v[4] = {f * ((1.0f - dx) * (1.0f - dy)), f * (dx * (1.0f - dy)), f * ((1.0f - dx) * dy), f * (dx * dy)};
  constexpr int o[4] = {0, 1, 15, 16};
#pragma unroll 1
  for (int n = 0; n <= last; n++) {
    const bool now = on && place == n;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (now) g[o[k]] = g[o[k]] + v[k];
      __syncwarp();
    }
  }
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

// surface gradients of two pairs (g[2][228]) -> gradients of their filtered spectra in b
// ([4][8][9] float2, over the same space): the 15x15 unfold and both transform passes transposed
__device__ __forceinline__ void couple_unsurface(const float *g, float2 *b, int lane) {
  const int q = lane >> 3, r = lane & 7;
  float2 gi[2][4];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int a = (lane >> 3) + 4 * k, c = lane & 7;
    const int i1 = (7 + a) * 15 + 7 + c, i2 = i1 - 2 * c, i3 = (7 - a) * 15 + 7 + c, i4 = i3 - 2 * c;
    auto cell = [&](int i, bool on) { return on ? make_float2(g[i], g[AM_SURF + i]) : make_float2(0.f, 0.f); };
    gi[k][0] = cell(i1, true);
    gi[k][1] = cell(i2, c != 0);
    gi[k][2] = cell(i3, a != 0);
    gi[k][3] = cell(i4, a && c);
  }
  __syncwarp();  // the gradients are read
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int a = (lane >> 3) + 4 * k, c = lane & 7;
    const float2 z = make_float2(0.f, 0.f);
    const float2 g1 = gi[k][0], g2 = gi[k][1], g3 = gi[k][2], g4 = gi[k][3];
    const float2 p = add2(g1, g2), m = sub2(g1, g2), f = dup2(0.25f);
    // rows of quadrants 2 and 3 in reverse order, for the DST; row or column 7 of the quadrants without a
    // zero frequency is 0
    b[a * 9 + c] = mul2(f, add2(add2(p, g3), g4));
    b[72 + a * 9 + (c ? c - 1 : 7)] = c ? mul2(f, sub2(add2(m, g3), g4)) : z;
    b[144 + (a ? 8 - a : 0) * 9 + c] = a ? mul2(f, sub2(sub2(p, g3), g4)) : z;
    b[216 + (a ? 8 - a : 0) * 9 + (c ? c - 1 : 7)] = (a && c) ? mul2(f, add2(sub2(m, g3), g4)) : z;
  }
  __syncwarp();
  float2 z8[8], v[8];
  float2 *col = b + q * 72 + r;
#pragma unroll
  for (int k = 0; k < 8; k++) z8[k] = col[k * 9];
  dtt2e_transposed_pair(z8, v, dup2((q & 2) ? -1.f : 1.f));
  __syncwarp();
  float2 *row = b + q * 72 + ((q & 1) ? 7 - r : r) * 9;  // in reverse order for the second DST
#pragma unroll
  for (int n = 0; n < 8; n++) row[n] = v[n];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; k++) z8[k] = col[k * 9];
  dtt2e_transposed_pair(z8, v, dup2((q & 1) ? -1.f : 1.f));
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; k++) col[k * 9] = v[k];
  __syncwarp();
}

// The gradients of two pairs' normalised products, added to their sensors' CLT gradients (a round's
// pairs are on distinct sensors); two: the second pair counts.
__device__ __forceinline__ void couple_products_grad(const CorrConst &cfg, const PairDev &pa, const PairDev &pb, bool one,
                                                     bool two, float l0, float l1, const float *s_clt, float *s_g,
                                                     const float2 *b, int lane) {
  const int oa1 = pa.cam1 * TP_CLT + lane, oa2 = pa.cam2 * TP_CLT + lane;
  const int ob1 = pb.cam1 * TP_CLT + lane, ob2 = pb.cam2 * TP_CLT + lane;
  const int off = (lane >> 3) * 9 + (lane & 7);
  const float fzz = cfg.fat_zero * cfg.fat_zero;
  float2 d1[2][4], d2[2][4], a2[2], ia2[2], s1v[2], s2v[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int o = m * 64 + 32 * h;
      d1[h][m] = make_float2(s_clt[oa1 + o], s_clt[ob1 + o]);
      d2[h][m] = make_float2(s_clt[oa2 + o], s_clt[ob2 + o]);
    }
    float2 s1 = mul2(d1[h][0], d1[h][0]), s2 = mul2(d2[h][0], d2[h][0]);
#pragma unroll
    for (int m = 1; m < 4; m++) {
      s1 = fma2(d1[h][m], d1[h][m], s1);
      s2 = fma2(d2[h][m], d2[h][m], s2);
    }
    // |d1| |d2| with the forward's approximate square root; ia2 = 1 / a2 (0 where a2 = 0)
    const float2 pr = mul2(s1, s2);
    ia2[h] = make_float2(pr.x > 0.0f ? rsqrtf(pr.x) : 0.0f, pr.y > 0.0f ? rsqrtf(pr.y) : 0.0f);
    a2[h] = mul2(pr, ia2[h]);
    s1v[h] = s1;
    s2v[h] = s2;
  }
  const float2 fz2 = warp_sum2(add2(a2[0], a2[1]), lane, 1.0f / 64, fzz);
  float2 tg[2][4], dbar[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const float2 den = add2(a2[h], fz2);
    const float2 u = make_float2(__fdividef(1.0f, den.x), __fdividef(1.0f, den.y));
    float2 n[4], t[4], gq[4];
#pragma unroll
    for (int m = 1; m < 4; m++) n[m] = neg2(d1[h][m]);
    clt_products(d1[h], n, d2[h], t);
    const float2 l = dup2(h ? l1 : l0);
#pragma unroll
    for (int m = 0; m < 4; m++) gq[m] = mul2(b[m * 72 + 36 * h + off], l);
    const float2 sw = fma2(gq[3], t[3], fma2(gq[2], t[2], fma2(gq[0], t[0], mul2(gq[1], t[1]))));
    dbar[h] = mul2(mul2(neg2(sw), u), u);
#pragma unroll
    for (int m = 0; m < 4; m++) tg[h][m] = mul2(gq[m], u);
  }
  const float2 dsum = warp_sum2(add2(dbar[0], dbar[1]), lane, 1.0f / 64, fzz);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const float2 a2bar = add2(dbar[h], dsum);
    const float2 *e = d2[h], *d = d1[h];
    const float2 T0 = tg[h][0], T1 = tg[h][1], T2 = tg[h][2], T3 = tg[h][3];
    const float2 n1 = neg2(T1), n2 = neg2(T2), n3 = neg2(T3);
    float2 g1[4], g2[4];
    g1[0] = fma2(T3, e[3], fma2(T2, e[2], fma2(T0, e[0], mul2(T1, e[1]))));
    g1[1] = fma2(n3, e[2], fma2(T2, e[3], fma2(T0, e[1], mul2(n1, e[0]))));
    g1[2] = fma2(n3, e[1], fma2(n2, e[0], fma2(T0, e[2], mul2(T1, e[3]))));
    g1[3] = fma2(T3, e[0], fma2(n2, e[1], fma2(T0, e[3], mul2(n1, e[2]))));
    g2[0] = fma2(T3, d[3], fma2(n2, d[2], fma2(T0, d[0], mul2(n1, d[1]))));
    g2[1] = fma2(n3, d[2], fma2(n2, d[3], fma2(T0, d[1], mul2(T1, d[0]))));
    g2[2] = fma2(n3, d[1], fma2(T2, d[0], fma2(T0, d[2], mul2(n1, d[3]))));
    g2[3] = fma2(T3, d[0], fma2(T2, d[1], fma2(T0, d[3], mul2(T1, d[2]))));
    // a2 = sqrt(s1 s2): d a2 / d d1[m] = d1[m] s2 / a2
    const float2 k1 = mul2(mul2(a2bar, s2v[h]), ia2[h]), k2 = mul2(mul2(a2bar, s1v[h]), ia2[h]);
#pragma unroll
    for (int m = 0; m < 4; m++) {  // no other pair adds to these sensors in this round
      const int o = m * 64 + 32 * h;
      const float2 x = fma2(k1, d[m], g1[m]), y = fma2(k2, e[m], g2[m]);
      if (one) {
        s_g[oa1 + o] += x.x;
        s_g[oa2 + o] += y.x;
      }
      if (two) {
        s_g[ob1 + o] += x.y;
        s_g[ob2 + o] += y.y;
      }
    }
  }
}

}  // namespace

template <bool U16>
__global__ void __launch_bounds__(32 * AD_NW, 4) adjoint_many_kernel(const __grid_constant__ SceneDev sc,
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
          couple_products_grad(cfg, cfg.pairs[pi], cfg.pairs[pj], any & 0xffffu, any >> 16, l0, l1, s_clt, s_g, buf, lane);
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
      stage_window<U16>(sc, sc.images[sidx], p.tlx, p.tly, wb + q * Stage<U16>::WIN, r);
      cp_async_commit();
      SWin<U16> win;
      win.base = (const typename Stage<U16>::T *)(wb + q * Stage<U16>::WIN);
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
      shift_sens<true>(sc, win, p, sidx, s_clt + (size_t)s * TP_CLT, s_g + (size_t)s * TP_CLT,
                       s_clt + (size_t)s * TP_CLT, r, true, gxy);
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
