// tp_adjoint.cuh -- device functions of the adjoint shared by its kernels: the transposed steps of the
// pair chain and of the CLT, a sub-tile's sensitivity to its residual shift, the strip's centroid.
#pragma once
#include "tp_forward.cuh"

namespace {

// a compile-time index as a type
template <int N>
struct Int {
  static constexpr int value = N;
};

constexpr float K16 = 0.19634954084936207f;  // pi / 16

struct AdjShape {
  int S, C, P, RE;
  int per_warp;   // floats of shared memory per warp
  int recompute;  // 1: recompute the CLT from the image instead of reading it back
  int use_strips; // 1: the forward recorded its per-pair strip samples in sc.strips
};

__device__ __forceinline__ void convolve(float o[4][8], const float *kp, int r) {
  if (!kp) return;
  float k[4][8];
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const float4 *p = (const float4 *)(kp + m * 64 + r * 8);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    k[m][0] = a.x; k[m][1] = a.y; k[m][2] = a.z; k[m][3] = a.w;
    k[m][4] = b.x; k[m][5] = b.y; k[m][6] = b.z; k[m][7] = b.w;
  }
#pragma unroll
  for (int v = 0; v < 8; v++) {
    const float d0 = o[0][v], d1 = o[1][v], d2 = o[2][v], d3 = o[3][v];
    const float k0 = k[0][v], k1 = k[1][v], k2 = k[2][v], k3 = k[3][v];
    o[0][v] = d0 * k0 - d1 * k1 - d2 * k2 + d3 * k3;
    o[1][v] = d1 * k0 + d0 * k1 - d3 * k2 - d2 * k3;
    o[2][v] = d2 * k0 - d3 * k1 + d0 * k2 - d1 * k3;
    o[3][v] = d3 * k0 + d2 * k1 + d1 * k2 + d0 * k3;
  }
}

// the phase rotation of fract_shift (same angles as the forward kernel)
__device__ __forceinline__ void rotate(float o[4][8], float rx, float ry, int r) {
  float ch, shh, cvr, svr;
  __sincosf(CUDART_PI_F * 0.0625f * (2 * r + 1) * rx, &shh, &ch);
  __sincosf(CUDART_PI_F * 0.0625f * (2 * r + 1) * ry, &svr, &cvr);
  const int base = threadIdx.x & 24;
#pragma unroll
  for (int v = 0; v < 8; v++) {
    const float cv = __shfl_sync(0xffffffffu, cvr, base + v), sv = __shfl_sync(0xffffffffu, svr, base + v);
    const float t0 = o[0][v] * ch - o[1][v] * shh, t1 = o[1][v] * ch + o[0][v] * shh;
    const float t2 = o[2][v] * ch - o[3][v] * shh, t3 = o[3][v] * ch + o[2][v] * shh;
    o[0][v] = t0 * cv - t2 * sv;
    o[2][v] = t2 * cv + t0 * sv;
    o[1][v] = t1 * cv - t3 * sv;
    o[3][v] = t3 * cv + t1 * sv;
  }
}

// transpose of rotate (both turns are orthogonal: undone in reverse order)
__device__ __forceinline__ void rotate_t(float o[4][8], float rx, float ry, int r) {
  float ch, shh, cvr, svr;
  __sincosf(CUDART_PI_F * 0.0625f * (2 * r + 1) * rx, &shh, &ch);
  __sincosf(CUDART_PI_F * 0.0625f * (2 * r + 1) * ry, &svr, &cvr);
  const int base = threadIdx.x & 24;
#pragma unroll
  for (int v = 0; v < 8; v++) {
    const float cv = __shfl_sync(0xffffffffu, cvr, base + v), sv = __shfl_sync(0xffffffffu, svr, base + v);
    const float t0 = o[0][v] * cv + o[2][v] * sv, t2 = o[2][v] * cv - o[0][v] * sv;
    const float t1 = o[1][v] * cv + o[3][v] * sv, t3 = o[3][v] * cv - o[1][v] * sv;
    o[0][v] = t0 * ch + t1 * shh;
    o[1][v] = t1 * ch - t0 * shh;
    o[2][v] = t2 * ch + t3 * shh;
    o[3][v] = t3 * ch - t2 * shh;
  }
}

// row r (8 values) of each of the four quadrants at p, by 16-byte accesses (row by row the eight lanes
// of a group would meet on the same banks)
__device__ __forceinline__ void load_rows(const float *p, int r, float o[4][8]) {
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const float4 a = *(const float4 *)(p + m * 64 + r * 8), b = *(const float4 *)(p + m * 64 + r * 8 + 4);
    o[m][0] = a.x; o[m][1] = a.y; o[m][2] = a.z; o[m][3] = a.w;
    o[m][4] = b.x; o[m][5] = b.y; o[m][6] = b.z; o[m][7] = b.w;
  }
}

// transpose of convolve (the per-frequency 4x4 sign matrix of the kernel, transposed)
__device__ __forceinline__ void convolve_t(float o[4][8], const float *kp, int r) {
  if (!kp) return;
  float k[4][8];
  load_rows(kp, r, k);
#pragma unroll
  for (int v = 0; v < 8; v++) {
    const float k0 = k[0][v], k1 = k[1][v], k2 = k[2][v], k3 = k[3][v];
    const float g0 = o[0][v], g1 = o[1][v], g2 = o[2][v], g3 = o[3][v];
    o[0][v] = k0 * g0 + k1 * g1 + k2 * g2 + k3 * g3;
    o[1][v] = -k1 * g0 + k0 * g1 - k3 * g2 + k2 * g3;
    o[2][v] = -k2 * g0 - k3 * g1 + k0 * g2 + k1 * g3;
    o[3][v] = k3 * g0 - k2 * g1 - k1 * g2 + k0 * g3;
  }
}

__device__ __forceinline__ Win make_win(const SceneDev &sc, const SubtilePlan &p, int s, int c = 0) {
  Win w;
  w.img = sc.images[s];
  w.pitch = sc.img_pitch;
  w.tlx = p.tlx; w.tly = p.tly; w.W = sc.width; w.H = sc.height;
  w.u16 = sc.img_dtype[s];
  w.inside = (p.tlx >= 0) && (p.tly >= 0) && (p.tlx <= sc.width - 16) && (p.tly <= sc.height - 16);
  w.scale = sc.color_scale[c];
  return w;
}

// one colour plane of a Bayer mosaic seen through a window: the mosaic's pixels of colour c
// (0 red, 1 blue, 2 green, on the Bayer phase (red row, red column)), zero elsewhere -- the
// sparse plane the forward transforms (the mirrored border keeps the pixel parity)
struct BayerWin {
  Win w;
  int c, rr, rc;
  __device__ __forceinline__ float at(int row, int col) const {
    const bool ry = ((w.tly + row) & 1) == rr, rx = ((w.tlx + col) & 1) == rc;
    const bool keep = (c == 0) ? (ry && rx) : ((c == 1) ? (!ry && !rx) : (ry != rx));
    return keep ? w.at(row, col) : 0.f;
  }
};

// taps of one strip sample (sample_code / strip_sample): returns the tap count
__device__ __forceinline__ int code_taps(int code, int idx[4], float wt[4]) {
  if (code < 0) return 0;
  const int i = code & 255, cs = code >> 8;
  idx[0] = i;
  if (cs == 0) { wt[0] = 1.f; return 1; }
  if (cs == 1) { wt[0] = 0.5f; idx[1] = i + 1; wt[1] = 0.5f; return 2; }
  if (cs == 2) { wt[0] = 0.5f; idx[1] = i + 15; wt[1] = 0.5f; return 2; }
  idx[1] = i + 1; idx[2] = i + 15; idx[3] = i + 16;
  wt[0] = wt[1] = wt[2] = wt[3] = 0.25f;
  return 4;
}
__device__ __forceinline__ int general_taps(float bx, float by, int row, int scol, int down, int idx[4],
                                            float wt[4]) {
  const float a = scol + 0.5f * (row & 1), pp = 0.5f * down * row;
  const float x = a * bx - pp * by, y = a * by + pp * bx;
  if (x > 7.f || x < -7.f || y > 7.f || y < -7.f) return 0;
  const float fx = x + 7.f, fy = y + 7.f;
  const int ix0 = min((int)floorf(fx), 13), iy0 = min((int)floorf(fy), 13);
  const float dx = fx - ix0, dy = fy - iy0;
  idx[0] = iy0 * 15 + ix0; wt[0] = (1.0f - dx) * (1.0f - dy);
  idx[1] = idx[0] + 1;     wt[1] = dx * (1.0f - dy);
  idx[2] = idx[0] + 15;    wt[2] = (1.0f - dx) * dy;
  idx[3] = idx[0] + 16;    wt[3] = dx * dy;
  return 4;
}

// one strip entry of a pair exactly as the forward kernel computes it
__device__ __forceinline__ float strip_entry(const float *c, const short *strip_code, const PairDev &pd, int e) {
  const int row = e / 15;
  float d;
  if (pd.kind <= 3) {
    const short2 code = *(const short2 *)&strip_code[(pd.kind * TP_MAX_STRIP * 15 + e) * 2];
    d = sample_code(c, code.x);
    if (row > 0) {
      const float d2 = sample_code(c, code.y);
      d = (isnan(d) || isnan(d2)) ? CUDART_NAN_F : (0.5f * d + 0.5f * d2);
    }
  } else {
    const int scol = e - row * 15 - 7;
    d = strip_sample(c, 4, pd.bx, pd.by, row, scol, -1);
    if (row > 0) {
      const float d2 = strip_sample(c, 4, pd.bx, pd.by, row, scol, 1);
      d = (isnan(d) || isnan(d2)) ? CUDART_NAN_F : (0.5f * d + 0.5f * d2);
    }
  }
  return d;
}

constexpr int AD_NW = 4;  // warps per tile

// First part of a sub-tile's sensitivity to its residual shift, 8-lane group (lane r holds row r): the
// rotation's own derivative dotted with the dd/dCLT gl (gdir, this lane's part), and gl taken back through the
// phase rotation, the kernel convolution and the 2D DCT-IV/DST-IV (symmetric transforms: the transpose runs
// through the same butterflies) to the folded tile (gf, row r).  tbq may lie over clt.
__device__ __forceinline__ void shift_grad(const SubtilePlan &p, const float *kp, const float *clt, const float *gl, float *tbq,
                                           int r, float gdir[2], float gf[4][8]) {
  // the rotation's own derivative (pi/16 (2k+1) x the CLT turned by 90 degrees) dotted with dd/dCLT
  gdir[0] = gdir[1] = 0.f;
  load_rows(gl, r, gf);
#pragma unroll
  for (int w4 = 0; w4 < 2; w4++) {
    float4 c4[4];
#pragma unroll
    for (int m = 0; m < 4; m++) c4[m] = *(const float4 *)(clt + m * 64 + r * 8 + 4 * w4);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int v = 4 * w4 + u;
      auto at = [&](int m) { return u == 0 ? c4[m].x : (u == 1 ? c4[m].y : (u == 2 ? c4[m].z : c4[m].w)); };
      const float c0 = at(0), c1 = at(1), c2 = at(2), c3 = at(3);
      const float g0 = gf[0][v], g1 = gf[1][v], g2 = gf[2][v], g3 = gf[3][v];
      const float fx = K16 * (2 * r + 1), fy = K16 * (2 * v + 1);
      gdir[0] = fmaf(fx, (g1 * c0 - g0 * c1) + (g3 * c2 - g2 * c3), gdir[0]);
      gdir[1] = fmaf(fy, (g2 * c0 - g0 * c2) + (g3 * c1 - g1 * c3), gdir[1]);
    }
  }
  __syncwarp();  // the CLT is read
  rotate_t(gf, p.rx, p.ry, r);
  convolve_t(gf, kp, r);
#pragma unroll
  for (int m = 0; m < 4; m++) {
    float u[8];
    dtt4_fast(gf[m], u, (m >> 1) & 1);
    group_transpose(u, tbq, r);
    dtt4_fast(u, gf[m], m & 1);
  }
}

// Last part: the lanes' parts summed, then dd/d(port x, port y) in every lane.
// residual = TL - px: dd/dpx = -dd/drx; the kernel-centre offsets add the dependence of px, py
// on the port through kdx, kdy (ImageDtt.java:4930-4939)
__device__ __forceinline__ void shift_out(const SceneDev &sc, const SubtilePlan &p, int s, float gdir[2], float out[2]) {
#pragma unroll
  for (int dir = 0; dir < 2; dir++) {
    gdir[dir] += __shfl_xor_sync(0xffffffffu, gdir[dir], 1);
    gdir[dir] += __shfl_xor_sync(0xffffffffu, gdir[dir], 2);
    gdir[dir] += __shfl_xor_sync(0xffffffffu, gdir[dir], 4);
  }
  const float gpx = -gdir[0], gpy = -gdir[1];
  out[0] = gpx;
  out[1] = gpy;
  if (p.kidx >= 0) {
    const float4 e1 = __ldg((const float4 *)(sc.kext[s] + (size_t)p.kidx * 8) + 1);
    out[0] = gpx * (1.0f - e1.x) - gpy * e1.z;
    out[1] = -gpx * e1.y + gpy * (1.0f - e1.w);
  }
}

// dd/d(port x, port y) of one (sensor, colour) sub-tile, 8-lane group: its dd/dCLT gl taken back to the folded
// tile, which is dotted with the fold of the pixels under the derivative window, one fold per direction,
// plus the rotation's own derivative.  gl is overwritten (with the folded gradient) where `own` is set.
// stage() is called by the whole warp once clt is no longer needed: it may copy the windows over it,
// asynchronously.
struct NoStage {
  __device__ __forceinline__ void operator()() const {}
};
template <typename PIX, typename STAGE = NoStage>
__device__ __forceinline__ void shift_sens(const SceneDev &sc, const PIX &w, const SubtilePlan &p, int s,
                                           const float *clt, float *gl_all, float *tbq, int r, bool own,
                                           float out[2], STAGE stage = STAGE()) {
  const float *kp = (p.kidx >= 0) ? sc.kernels[s] + (size_t)p.kidx * TP_CLT : nullptr;
  float ahs, ahc, avs, avc;
  __sincosf(CUDART_PI_F * 0.0625f * p.rx, &ahs, &ahc);
  __sincosf(CUDART_PI_F * 0.0625f * p.ry, &avs, &avc);
  const FoldIdx fv = fold_idx(r);
  float gdir[2];
  float *gfs = gl_all + r * 8;  // gfs[m * 64 + j] for folded row r
  {
    float gf[4][8];
    shift_grad(p, kp, clt, gl_all, tbq, r, gdir, gf);
    if (own) {
#pragma unroll
      for (int m = 0; m < 4; m++) {
        *(float4 *)(gfs + m * 64) = make_float4(gf[m][0], gf[m][1], gf[m][2], gf[m][3]);
        *(float4 *)(gfs + m * 64 + 4) = make_float4(gf[m][4], gf[m][5], gf[m][6], gf[m][7]);
      }
    }
  }
  __syncwarp();
  stage();
  cp_async_wait_all();
  __syncwarp();
  // the lane's two source rows of the window, read once for both directions and both vertical
  // variants
  float p0[16], p1[16];
#pragma unroll
  for (int cix = 0; cix < 16; cix++) {
    p0[cix] = w.at(fv.src0, cix);
    p1[cix] = w.at(fv.src1, cix);
  }
  // per direction: the fold with the derivative window dotted with the folded gradient
#pragma unroll
  for (int dir = 0; dir < 2; dir++) {
    float vw0, vw1, hw0[8], hw1[8];
    if (dir == 0) fold_weights(-K16 * ahs, K16 * ahc, avc, avs, fv, vw0, vw1, hw0, hw1);
    else fold_weights(ahc, ahs, -K16 * avs, K16 * avc, fv, vw0, vw1, hw0, hw1);
    float acc = 0.f;
#pragma unroll
    for (int vb = 0; vb < 2; vb++) {
      const float k0 = (vb ? fv.ss0 : fv.sc0) * vw0, k1 = (vb ? fv.ss1 : fv.sc1) * vw1;
      float vc[16];
#pragma unroll
      for (int cix = 0; cix < 16; cix++) vc[cix] = fmaf(k1, p1[cix], k0 * p0[cix]);
#pragma unroll
      for (int hb = 0; hb < 2; hb++) {
        const float4 ga = *(const float4 *)(gfs + (vb * 2 + hb) * 64), gb = *(const float4 *)(gfs + (vb * 2 + hb) * 64 + 4);
        const float g[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
        for (int j2 = 0; j2 < 8; j2++) {
          const FoldIdx fh = fold_idx(j2);
          const float h0 = (hb ? fh.ss0 : fh.sc0) * hw0[j2], h1 = (hb ? fh.ss1 : fh.sc1) * hw1[j2];
          acc = fmaf(fmaf(h1, vc[fh.src1], h0 * vc[fh.src0]), g[j2], acc);
        }
      }
    }
    gdir[dir] += acc;
  }
  shift_out(sc, p, s, gdir, out);
}

// x = T^T y for the DCT-IIe / DST-IIe of dtt2e_fast (its transposed data flow)
__device__ __forceinline__ void dtt2e_transposed(const float y[8], float x[8], bool sine) {
  const float S = 0.5f;
  const float C4 = 0.7071067811865476f, C8 = 0.9238795325112867f, C38 = 0.3826834323650898f;
  float t[8];
#pragma unroll
  for (int k = 0; k < 8; k++) t[k] = sine ? y[7 - k] : y[k];
  float u1[4];
#pragma unroll
  for (int j = 0; j < 4; j++)
    u1[j] = fmaf(k_dct2e[8 + j], t[1], fmaf(k_dct2e[24 + j], t[3], fmaf(k_dct2e[40 + j], t[5], k_dct2e[56 + j] * t[7])));
  const float a0 = S * t[0] + (S * C4) * t[4], a1 = S * t[0] - (S * C4) * t[4];
  const float b0 = S * fmaf(C8, t[2], C38 * t[6]), b1 = S * fmaf(C38, t[2], -C8 * t[6]);
  const float u0[4] = {a0 + b0, a1 + b1, a1 - b1, a0 - b0};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    x[j] = u0[j] + u1[j];
    x[7 - j] = u0[j] - u1[j];
  }
  if (sine) {
#pragma unroll
    for (int n = 1; n < 8; n += 2) x[n] = -x[n];
  }
}

// centroid of a combined strip (gG, one warp) and its derivatives by the strip's entries (gcmb, zero on
// entry); NaN where the tile has no peak
__device__ __forceinline__ float strip_centroid(const CorrConst &cfg, const float *gG, float *gcmb, int lane) {
  float dres = CUDART_NAN_F;
  const float v = (lane < 15) ? gG[lane] : CUDART_NAN_F;
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
  const float vmax = gG[imx];
  if (vmax >= cfg.min_corr) {
    const int ix = imx - 7;
    int dh = cfg.strip_rows;
    float wys = 1.0f;
    if (dh > cfg.wndy_size) dh = cfg.wndy_size;
    else if (dh < cfg.wndy_size) {
      float swy = cfg.wndy[0];
      for (int i = 1; i < dh; i++) swy += cfg.wndy[i];
      wys = 1.0f / swy;
    }
    const int x0 = 7 + ix, nk = dh * 2 * cfg.wndx_size;
    float s0 = 0.f, sx = 0.f;
    for (int pass = 0; pass < 2; pass++) {
      const float xm = (pass == 1) ? sx / s0 : 0.f;
      for (int k = lane; k < nk; k += 32) {
        const int dy = k / (2 * cfg.wndx_size), rest = k - dy * 2 * cfg.wndx_size;
        const int adx = rest >> 1, dir = (rest & 1) ? 1 : -1, odd = dy & 1;
        if (((adx - odd) & 1) || (adx == 0 && dir < 0)) continue;
        const int idx = (adx * dir) >> 1, xx = 2 * idx + odd, x1 = x0 + idx;
        if (x1 < 0 || x1 >= 15) continue;
        const float d = gG[dy * 15 + x1];
        if (isnan(d) || !(d > 0.0f)) continue;
        const float wk = (((dy == 0) ? wys : 2.0f * wys) * cfg.wndy[dy]) * cfg.wndx[adx];
        if (pass == 0) {
          s0 += d * wk;
          sx += d * wk * xx;
        } else {
          // d(-(ix + sx/s0/2)) / d(combo): -(wk / (2 s0)) (xx - sx/s0)
          gcmb[dy * 15 + x1] = -(wk / (2.0f * s0)) * (xx - xm);
        }
      }
      if (pass == 0) {
        s0 = warp_sum(s0);
        sx = warp_sum(sx);
        if (s0 == 0.0f) break;
        dres = -(ix + sx / s0 / 2);
      }
    }
  }
  __syncwarp();
  return dres;
}

}  // namespace
