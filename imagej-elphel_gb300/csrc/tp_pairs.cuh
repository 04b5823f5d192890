// tp_pairs.cuh -- the pair phase of the forward with two values per instruction.
//
// The scalar pair phase (fwd_pair) issues about 870 warp instructions per pair and is bound by
// that, not by memory or FP32 rate.  GB300 has packed FP32 arithmetic (two independent,
// IEEE-rounded operations per instruction), so here every arithmetic step carries two values:
// the products carry CLT indices l and l + 32 of one pair, the transforms and the unfold carry two
// pairs.  The operation order and the fused multiply-adds are the scalar code's, so the results
// are the same bits.
#pragma once
#include "tp_dtt.cuh"

namespace {

__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }

// DCT-IIe of two rows (dtt2e_fast): sg = -1 gives the DST-IIe with its outputs in reverse order
// (the reader indexes them backwards), +1 the DCT-IIe.  The sign of the odd inputs goes into the
// first butterflies as an exact product.
__device__ __forceinline__ void dtt2e_pair(const float2 x[8], float2 t[8], float2 sg) {
  const float S = 0.5f, C4 = 0.7071067811865476f, C8 = 0.9238795325112867f, C38 = 0.3826834323650898f;
  const float2 ng = neg2(sg);
  float2 u0[4], u1[4];
  u0[0] = fma2(sg, x[7], x[0]); u1[0] = fma2(ng, x[7], x[0]);
  u0[1] = fma2(sg, x[1], x[6]); u1[1] = fma2(sg, x[1], neg2(x[6]));
  u0[2] = fma2(sg, x[5], x[2]); u1[2] = fma2(ng, x[5], x[2]);
  u0[3] = fma2(sg, x[3], x[4]); u1[3] = fma2(sg, x[3], neg2(x[4]));
  const float2 a0 = add2(u0[0], u0[3]), a1 = add2(u0[1], u0[2]);
  const float2 b0 = sub2(u0[0], u0[3]), b1 = sub2(u0[1], u0[2]);
  t[0] = mul2(dup2(S), add2(a0, a1));
  t[4] = mul2(dup2(S * C4), sub2(a0, a1));
  t[2] = mul2(dup2(S), fma2(dup2(C8), b0, mul2(dup2(C38), b1)));
  t[6] = mul2(dup2(S), fma2(dup2(C38), b0, mul2(dup2(-C8), b1)));
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int k = 2 * j + 1;
    t[k] = fma2(dup2(k_dct2e[k * 8 + 0]), u1[0],
                fma2(dup2(k_dct2e[k * 8 + 1]), u1[1],
                     fma2(dup2(k_dct2e[k * 8 + 2]), u1[2], mul2(dup2(k_dct2e[k * 8 + 3]), u1[3]))));
  }
}

// |d1| |d2| from the product of the squared amplitudes (approximate square root, ~2 ulp)
__device__ __forceinline__ float amp_of(float pr) { return (pr > 0.0f) ? pr * rsqrtf(pr) : 0.0f; }

// warp sums of six values at once, times k0 and fz: the butterfly tree of warp_sum (strides 16, 8, 4, 2, 1),
// each exchange halving the values a lane keeps, then one broadcast per value: 14 shuffles
// instead of 30
__device__ __forceinline__ void warp_sum6(const float v[6], int lane, float k0, float fz, float out[6]) {
  const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
  float r[3];
#pragma unroll
  for (int i = 0; i < 3; i++)
    r[i] = (h16 ? v[3 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, h16 ? v[i] : v[3 + i], 16);
  const float s0 = (h8 ? r[2] : r[0]) + __shfl_xor_sync(0xffffffffu, h8 ? r[0] : r[2], 8);
  const float s1 = r[1] + __shfl_xor_sync(0xffffffffu, r[1], 8);
  const bool odd = h4 && !h8;
  float t = (odd ? s1 : s0) + __shfl_xor_sync(0xffffffffu, (h8 || h4) ? s0 : s1, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  t = t * k0 * fz;
#pragma unroll
  for (int p = 0; p < 6; p++) out[p] = __shfl_sync(0xffffffffu, t, (p / 3) * 16 + ((p % 3) == 0 ? 0 : ((p % 3) == 1 ? 4 : 8)));
}

// the same for two values: sums of a over lanes and of b over lanes, each times k0 and fz
__device__ __forceinline__ float2 warp_sum2(float2 v, int lane, float k0, float fz) {
  const bool h16 = lane & 16;
  float t = (h16 ? v.y : v.x) + __shfl_xor_sync(0xffffffffu, h16 ? v.x : v.y, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  t = t * k0 * fz;
  return make_float2(__shfl_sync(0xffffffffu, t, 0), __shfl_sync(0xffffffffu, t, 16));
}

// the normalised products of a pair (Correlation2d.correlateSingleColorFD, the ZI table) on two
// CLT indices: t[0..3] from a (first sensor), its negatives n[1..3] and b (second sensor)
__device__ __forceinline__ void clt_products(const float2 a[4], const float2 n[4], const float2 b[4], float2 t[4]) {
  t[0] = fma2(a[3], b[3], fma2(a[2], b[2], fma2(a[0], b[0], mul2(a[1], b[1]))));
  t[1] = fma2(a[2], b[3], fma2(n[3], b[2], fma2(a[0], b[1], mul2(n[1], b[0]))));
  t[2] = fma2(a[1], b[3], fma2(a[0], b[2], fma2(n[2], b[0], mul2(n[3], b[1]))));
  t[3] = fma2(a[0], b[3], fma2(n[1], b[2], fma2(a[3], b[0], mul2(n[2], b[1]))));
}

// asynchronous copy of a shared-memory range to global memory (both 16-byte aligned, bytes a
// multiple of 16) by one lane, after the warp's writes were fenced; bulk_read_done() before the
// range is written again
__device__ __forceinline__ void bulk_store(void *gdst, const void *ssrc, int bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(gdst),
               "r"((unsigned)__cvta_generic_to_shared(ssrc)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void bulk_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_read_done() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_done() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

// ---------------------------------------------------------------------------
// All six pairs of the standard quad (Correlation2d.PAIRS: cameras 0-1, 2-3, 0-2, 1-3, 0-3, 2-1)
// of one tile by one warp.  Each sensor's coefficients are read once for the six pairs (the scalar
// phase reads them three times) and squared once; then the six spectra are kept as three
// interleaved couples [4][8][9] of float2 over the space of the CLT, which is no longer needed.
// ws: the warp's region of QP_FLOATS or more floats, the CLT [C][4][QP_CLT] first; it is stored to HBM here too.
// surfaces (15x15, six in a row) go to `surf` and from there to HBM in one asynchronous copy.
// ---------------------------------------------------------------------------
// The CLT of a (colour, sensor) here: four quadrants of two half quadrants (rows 0-3, rows 4-7), each 32 values
// and then 4 unused ones, so that eight lanes that store a row each, 16 bytes at a time, reach different banks.
constexpr int QP_HALF = 36, QP_QUAD = 68, QP_CLT = 4 * QP_QUAD;  // floats to the second half, the next quadrant, sensor
constexpr int QP_BUF = 576;                       // floats of one couple's spectra
constexpr int QP_SURF = 3 * QP_BUF;               // first surface (+ 2 floats for odd tiles)
constexpr int QP_FLOATS = QP_SURF + 2 + 6 * 225 + 4;  // rounded to 16 bytes: 3084

// store_clt for a sensor of colour c, from the lanes' values of CLT indices l and l + 32: 128 contiguous bytes a store
// (a row a lane, 16 bytes at a time, each store touches half of 32 sectors)
template <int C>
__device__ __forceinline__ void store_clt_lanes(const SceneDev &sc, int c, size_t tile, int cam, const float2 d[4],
                                                int lane) {
  float *g = sc.clt + ((tile * 4 + cam) * C + c) * TP_CLT + lane;
  float2 l = make_float2(1.f, 1.f);  // exact
  if (sc.lpf_rbg && ((sc.clt_lpf_mask >> c) & 1))
    l = make_float2(__ldg(sc.lpf_rbg + c * 64 + lane), __ldg(sc.lpf_rbg + c * 64 + 32 + lane));
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const float2 v = mul2(d[m], l);
    g[m * 64] = v.x;
    g[m * 64 + 32] = v.y;
  }
}

template <int C>
__device__ __forceinline__ void quad_spectra(const SceneDev &sc, const CorrConst &cfg, const float *lpf, size_t tile,
                                             float *ws, int lane) {
  // The loops over colours and couples stay loops: unrolled, a tile's straight-line code misses the
  // instruction cache (the 16 warps of an SM are all at different places of it).
  float2 acc[6][4];
#pragma unroll
  for (int p = 0; p < 6; p++)
#pragma unroll
    for (int m = 0; m < 4; m++) acc[p][m] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int c = 0; c < C; c++) {
    float2 d[4][4], s[4];
#pragma unroll
    for (int cam = 0; cam < 4; cam++) {
      const float *p = ws + (c * 4 + cam) * QP_CLT + lane;
#pragma unroll
      for (int m = 0; m < 4; m++) d[cam][m] = make_float2(p[m * QP_QUAD], p[m * QP_QUAD + QP_HALF]);
      s[cam] = mul2(d[cam][0], d[cam][0]);
#pragma unroll
      for (int m = 1; m < 4; m++) s[cam] = fma2(d[cam][m], d[cam][m], s[cam]);
    }
#pragma unroll
    for (int cam = 0; cam < 4; cam++) store_clt_lanes<C>(sc, c, tile, cam, d[cam], lane);
    constexpr int c1[6] = {0, 2, 0, 1, 0, 2}, c2[6] = {1, 3, 2, 3, 3, 1};
    float2 a2[6];
    float v[6], fzs[6];
#pragma unroll
    for (int p = 0; p < 6; p++) {
      const float2 pr = mul2(s[c1[p]], s[c2[p]]);
      a2[p] = make_float2(amp_of(pr.x), amp_of(pr.y));
      v[p] = a2[p].x + a2[p].y;
    }
    warp_sum6(v, lane, 1.0f / 64, cfg.fat_zero, fzs);
    const float wgt = (C == 1) ? 1.0f : cfg.col_weights[c];
    constexpr int order[6] = {0, 2, 4, 1, 5, 3};  // by first sensor, whose negatives are formed once
    float2 n[4];
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const int p = order[i];
      if (i == 0 || i == 3 || i == 5) {
#pragma unroll
        for (int m = 1; m < 4; m++) n[m] = neg2(d[c1[p]][m]);
      }
      const float2 den = fma2(dup2(fzs[p]), dup2(cfg.fat_zero), a2[p]);  // |d1||d2| + its mean x fat_zero^2
      const float2 sw = make_float2(__fdividef(wgt, den.x), __fdividef(wgt, den.y));
      float2 t[4];
      clt_products(d[c1[p]], n, d[c2[p]], t);
#pragma unroll
      for (int m = 0; m < 4; m++) acc[p][m] = fma2(t[m], sw, acc[p][m]);
    }
  }
  // LPF; the unfold's factor 1/4 goes in here (a power of two: the same bits)
  const float2 l = make_float2(0.25f * lpf[lane], 0.25f * lpf[lane + 32]);
  __syncwarp();  // the whole CLT is read
  const int off = (lane >> 3) * 9 + (lane & 7);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float2 *b = (float2 *)(ws + k * QP_BUF) + off;
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const float2 x = mul2(acc[2 * k][m], l), y = mul2(acc[2 * k + 1][m], l);
      b[m * 72] = make_float2(x.x, y.x);
      b[m * 72 + 36] = make_float2(x.y, y.y);
    }
  }
  __syncwarp();
}

// the two transform passes and the 15x15 unfold of one couple's spectra b ([4][72] float2) into the
// surfaces s0, s1 of its two pairs
__device__ __forceinline__ void couple_surfaces(float2 *b, float *s0, float *s1, int lane) {
  const int q = lane >> 3, r = lane & 7;
  const float2 sg1 = dup2((q & 2) ? -1.f : 1.f), sg2 = dup2((q & 1) ? -1.f : 1.f);
  float2 x[8], t[8];
  const float2 *row = b + q * 72 + r * 9;
#pragma unroll
  for (int e = 0; e < 8; e++) x[e] = row[e];
  dtt2e_pair(x, t, sg1);
  __syncwarp();
  float2 *col = b + q * 72 + r;
#pragma unroll
  for (int j = 0; j < 8; j++) col[j * 9] = t[j];
  __syncwarp();
  const float2 *row2 = b + q * 72 + ((q & 2) ? 7 - r : r) * 9;  // the DST's rows come in reverse order
#pragma unroll
  for (int e = 0; e < 8; e++) x[e] = row2[e];
  dtt2e_pair(x, t, sg2);
  __syncwarp();
  float2 *out = b + q * 72 + r * 9;
#pragma unroll
  for (int e = 0; e < 8; e++) out[e] = t[e];
  __syncwarp();
  // unfold (DttRad2.corr_unfold_tile): cells (a, b) and their mirror images; quadrants 1 and 3 hold
  // their columns in reverse order.  Where a or b is 0 the mirror image is the cell itself.
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int a = (lane >> 3) + 4 * k, bb = lane & 7;
    const float2 z = make_float2(0.f, 0.f);
    const float2 A = b[a * 9 + bb];
    const float2 B = bb ? b[72 + a * 9 + 8 - bb] : z;
    const float2 Cc = a ? b[144 + (a - 1) * 9 + bb] : z;
    const float2 D = (a && bb) ? b[216 + (a - 1) * 9 + 8 - bb] : z;
    const float2 p = add2(A, B), m = sub2(A, B);
    const float2 o1 = add2(add2(p, Cc), D), o2 = sub2(add2(m, Cc), D), o3 = sub2(sub2(p, Cc), D),
                 o4 = add2(sub2(m, Cc), D);
    const int i1 = (7 + a) * 15 + 7 + bb, i2 = i1 - 2 * bb, i3 = (7 - a) * 15 + 7 + bb, i4 = i3 - 2 * bb;
    s0[i1] = o1.x; s1[i1] = o1.y;
    s0[i2] = o2.x; s1[i2] = o2.y;
    s0[i3] = o3.x; s1[i3] = o3.y;
    s0[i4] = o4.x; s1[i4] = o4.y;
  }
}

// One couple of a standard quad's pairs over C colours: spectra of pairs 2k and 2k + 1 into b ([4][72] float2).
// clt: [C][4][QP_CLT]; the couple's sensors f0, g0 and f1, g1.  The CLT of colour `keep` is stored to HBM.  l: the
// LPF at l and l + 32, over four (the unfold's factor).
template <int C>
__device__ __forceinline__ void couple_of_quad(const SceneDev &sc, const CorrConst &cfg, float2 l, const float *clt,
                                               size_t tile, int keep, int f0, int g0, int f1, int g1, float2 *b, int lane) {
  float2 acc[2][4];
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int m = 0; m < 4; m++) acc[h][m] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int c = 0; c < C; c++) {
    const float *cc = clt + c * 4 * QP_CLT + lane;
    float2 t[2][4], a2[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int sf = h ? f1 : f0, sg = h ? g1 : g0;
      const float *pf = cc + sf * QP_CLT, *pg = cc + sg * QP_CLT;
      float2 x[4], y[4], n[4];
#pragma unroll
      for (int m = 0; m < 4; m++) {
        x[m] = make_float2(pf[m * QP_QUAD], pf[m * QP_QUAD + QP_HALF]);
        y[m] = make_float2(pg[m * QP_QUAD], pg[m * QP_QUAD + QP_HALF]);
      }
      if (c == keep) {
        store_clt_lanes<C>(sc, c, tile, sf, x, lane);
        store_clt_lanes<C>(sc, c, tile, sg, y, lane);
      }
      float2 sx = mul2(x[0], x[0]), sy = mul2(y[0], y[0]);
#pragma unroll
      for (int m = 1; m < 4; m++) {
        sx = fma2(x[m], x[m], sx);
        sy = fma2(y[m], y[m], sy);
        n[m] = neg2(x[m]);
      }
      const float2 pr = mul2(sx, sy);
      a2[h] = make_float2(amp_of(pr.x), amp_of(pr.y));
      clt_products(x, n, y, t[h]);
    }
    const float2 fzs = warp_sum2(make_float2(a2[0].x + a2[0].y, a2[1].x + a2[1].y), lane, 1.0f / 64, cfg.fat_zero);
    const float wgt = (C == 1) ? 1.0f : cfg.col_weights[c];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const float2 den = fma2(dup2(h ? fzs.y : fzs.x), dup2(cfg.fat_zero), a2[h]);
      const float2 sw = make_float2(__fdividef(wgt, den.x), __fdividef(wgt, den.y));
#pragma unroll
      for (int m = 0; m < 4; m++) acc[h][m] = fma2(t[h][m], sw, acc[h][m]);
    }
  }
  b += (lane >> 3) * 9 + (lane & 7);
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const float2 x = mul2(acc[0][m], l), y = mul2(acc[1][m], l);
    b[m * 72] = make_float2(x.x, y.x);
    b[m * 72 + 36] = make_float2(x.y, y.y);
  }
  __syncwarp();
}

// sample of a strip entry: sample_code of the two sides, averaged below the first row
__device__ __forceinline__ float strip_of(const float *c, short2 code, int e) {
  float d = sample_code(c, code.x);
  if (e >= 15) {
    const float d2 = sample_code(c, code.y);
    d = (isnan(d) || isnan(d2)) ? CUDART_NAN_F : (0.5f * d + 0.5f * d2);
  }
  return d;
}

__device__ __forceinline__ short2 quad_code(const short *strip_code, int kind, int e) {
  return *(const short2 *)&strip_code[(kind * TP_MAX_STRIP * 15 + e) * 2];
}

// one strip entry of a general pair from its taps (CorrDev::gen_tap; strip_sample, both sides below the first row)
__device__ __forceinline__ float tap_sample(const float *c, float dx, float dy) {
  const float w00 = (1.0f - dx) * (1.0f - dy), w10 = dx * (1.0f - dy), w01 = (1.0f - dx) * dy, w11 = dx * dy;
  return fmaf(w11, c[16], fmaf(w01, c[15], fmaf(w00, c[0], w10 * c[1])));
}
__device__ __forceinline__ float tap_strip(const float *c, float4 tap, int cells, bool both) {
  const float d = tap_sample(c + (cells & 255), tap.x, tap.y), d2 = tap_sample(c + ((cells >> 8) & 255), tap.z, tap.w);
  const bool out = (cells & 0x10000) || (both && (cells & 0x20000));
  return out ? CUDART_NAN_F : (both ? 0.5f * d + 0.5f * d2 : d);
}

// First half of a standard quad's pair phase: the six surfaces to ws + QP_SURF and, asynchronously, to
// HBM; returns where they are.  The spectra's space (up to QP_SURF) is then free; the caller waits
// (bulk_read_done by lane 0, then __syncwarp) before it writes the surfaces' space again.
template <int C>
__device__ __forceinline__ const float *quad_surfaces(const SceneDev &sc, const CorrConst &cfg, const float *lpf,
                                                      size_t tile, float *ws, int lane) {
  quad_spectra<C>(sc, cfg, lpf, tile, ws, lane);
  if (C == 1) {  // the last tile's surfaces are out (with colours the caller has waited already)
    if (lane == 0) bulk_read_done();
    __syncwarp();
  }
  // a tile's six surfaces are 5400 bytes, so odd tiles start 8 past a 16-byte boundary; in shared
  // memory they start at the same remainder, and the two floats before or after the aligned 5392
  // bytes go out by plain stores
  const int odd = (int)(tile & 1);
  float *surf = ws + QP_SURF + 2 * odd;
#pragma unroll 1
  for (int k = 0; k < 3; k++)
    couple_surfaces((float2 *)(ws + k * QP_BUF), surf + 450 * k, surf + 450 * k + 225, lane);
  bulk_fence();
  __syncwarp();
  float *g = sc.corr + tile * 1350;
  if (lane == 0) bulk_store(g + 2 * odd, surf + 2 * odd, 5392);
  if (lane < 2) g[odd ? lane : 1348 + lane] = surf[odd ? lane : 1348 + lane];
  return surf;
}

// Second half: strip products cmb and ortho profile products oprod (the same as six calls of
// fwd_pair)
template <int NT>
__device__ __forceinline__ void quad_strips(const SceneDev &sc, const CorrConst &cfg, const float *surf, size_t tile,
                                            int RE, const short *strip_code, int lane, float cmb[8], float oprod[8]) {
  {
    // getMaxXSOrtho profiles: lanes 0-14 the horizontal pairs' columns, lanes 16-30 the vertical pairs'
    // rows, symmetrised (even in i, so rows 0..7 carry it) and multiplied over the two pairs
    const int half = lane >> 4, j = lane & 15, stride = half ? 1 : 15;
    const float *lo = surf + half * 450 + (half ? j * 15 : j), *hi = lo + 14 * stride;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      oprod[i] = (0.5f * (lo[0] + hi[0]) + cfg.corr_offset) * (0.5f * (lo[225] + hi[225]) + cfg.corr_offset);
      lo += stride;
      hi -= stride;
    }
  }
#pragma unroll
  for (int t = 0; t < NT; t++) cmb[t] = 1.f;
#pragma unroll 1
  for (int p = 0; p < 6; p++) {
    if (!cfg.pairs[p].in_combo) continue;
    const int kind = (p < 4) ? p >> 1 : p - 2;
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const int e = lane + 32 * t;
      if (e < RE) {
        const float d = strip_of(surf + 225 * p, quad_code(strip_code, kind, e), e);
        if (sc.strips) sc.strips[(tile * 6 + p) * RE + e] = d;  // kept for the adjoint
        float v = d + cfg.corr_offset;
        if (v < 0.0f) v = 0.0f;
        cmb[t] *= cfg.twice_diagonal ? v * v : v;
      }
    }
  }
}

}  // namespace
