// tp_forward.cuh -- device functions of the forward shared by its schedules: a sub-tile's CLT
// (fold, DTT, kernel convolution, shift), the scalar pair phase, the extraction, window staging.
#pragma once
#include "tp_dtt.cuh"

#include <cstddef>

namespace {

constexpr int SCR = 288;           // per-warp scratch floats: [4][8][9] transpose / surface buffer

// ---------------------------------------------------------------------------
// phase A: CLT of one sub-tile, lane r of the 8-lane group holds row r
// (= horizontal frequency r) of each quadrant on return: o[m][v].
// ---------------------------------------------------------------------------
template <int KIND, typename PIX = Win>  // 0 mono, 1 Bayer red/blue, 2 Bayer green; PIX: at(row, col)
__device__ __forceinline__ void subtile_clt(const PIX &w, float rx, float ry, int pc, int pr, int pg, int r,
                                            float *tbuf, float o[4][8]) {
  float ahs, ahc, avs, avc;
  __sincosf(CUDART_PI_F * 0.0625f * rx, &ahs, &ahc);
  __sincosf(CUDART_PI_F * 0.0625f * ry, &avs, &avc);
  const FoldIdx fv = fold_idx(r);
  float vw0, vw1, hw0[8], hw1[8];
  fold_weights(ahc, ahs, avc, avs, fv, vw0, vw1, hw0, hw1);
  if constexpr (KIND == 1) {
    // one nonzero pixel per folded value: the term whose source row/column has the colour's parity
    const bool a1 = (fv.src0 & 1) != pr;
    const int srow = a1 ? fv.src1 : fv.src0;
    const float vk = a1 ? fv.sc1 * vw1 : fv.sc0 * vw0;
    float y[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const FoldIdx fh = fold_idx(j);
      const bool b1 = (fh.src0 & 1) != pc;
      const int scol = b1 ? fh.src1 : fh.src0;
      const float hk = b1 ? fh.sc1 * hw1[j] : fh.sc0 * hw0[j];
      y[j] = (vk * hk) * w.at(srow, scol);
    }
    __syncwarp();  // every window is read: the transpose buffers may lie over them
    float z[8];
    dct4_fast(y, z);
    group_transpose(z, tbuf, r);
    dct4_fast(z, o[0]);
    // SC[h][v] = sh CC[7-h][v], CS[h][v] = sv CC[h][7-v], SS = sh sv CC[7-h][7-v]
    const float sh = pc ? -1.f : 1.f, sv = pr ? -1.f : 1.f;
#pragma unroll
    for (int v = 0; v < 8; v++) o[1][v] = sh * __shfl_xor_sync(0xffffffffu, o[0][v], 7);
#pragma unroll
    for (int v = 0; v < 8; v++) {
      o[2][v] = sv * o[0][7 - v];
      o[3][v] = sv * o[1][7 - v];
    }
  } else if constexpr (KIND == 2) {
    // two nonzero pixels per folded value (checkerboard): CC and SC folds
    float ycc[8], ysc[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const FoldIdx fh = fold_idx(j);
      float cc = 0.f, sc = 0.f;
#pragma unroll
      for (int a = 0; a < 2; a++) {
        const int srow = a ? fv.src1 : fv.src0;
        const float vk = a ? fv.sc1 * vw1 : fv.sc0 * vw0;
        const bool b1 = ((fh.src0 + srow) & 1) != pg;  // column term with (row + col) parity pg
        const int scol = b1 ? fh.src1 : fh.src0;
        const float x = vk * w.at(srow, scol);
        cc = fmaf(b1 ? fh.sc1 * hw1[j] : fh.sc0 * hw0[j], x, cc);
        sc = fmaf(b1 ? fh.ss1 * hw1[j] : fh.ss0 * hw0[j], x, sc);
      }
      ycc[j] = cc;
      ysc[j] = sc;
    }
    __syncwarp();  // every window is read: the transpose buffers may lie over them
    float z[8];
    dct4_fast(ycc, z);
    group_transpose(z, tbuf, r);
    dct4_fast(z, o[0]);
    dtt4_fast(ysc, z, true);
    group_transpose(z, tbuf, r);
    dct4_fast(z, o[1]);
    // CS[h][v] = sg SC[7-h][7-v], SS[h][v] = sg CC[7-h][7-v]
    const float sg = pg ? -1.f : 1.f;
#pragma unroll
    for (int v = 0; v < 8; v++) {
      o[2][7 - v] = sg * __shfl_xor_sync(0xffffffffu, o[1][v], 7);
      o[3][7 - v] = sg * __shfl_xor_sync(0xffffffffu, o[0][v], 7);
    }
  } else {
    fold_dtt_dense(w, fv, vw0, vw1, hw0, hw1, r, tbuf, o);
  }
}

// convolution with the kernel tile and the phase-rotation shift, in place on o[m][v]
__device__ __forceinline__ void conv_shift(float o[4][8], const float *kp, float rx, float ry, int r) {
  if (kp) {
    float k[4][8];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const float4 *p = (const float4 *)(kp + m * 64 + r * 8);
      float4 a = __ldg(p), b = __ldg(p + 1);
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
  float ch, shh, cvr, svr;
  __sincosf(CUDART_PI_F * 0.0625f * (2 * r + 1) * rx, &shh, &ch);
  __sincosf(CUDART_PI_F * 0.0625f * (2 * r + 1) * ry, &svr, &cvr);
  const int base = threadIdx.x & 24;  // first lane of this 8-lane group
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

// the stored CLT of row r (horizontal frequency r) of the four quadrants; with the colour's bit
// in clt_lpf_mask multiplied by the LPF (in place), as the reference GPU stores it (lpf_mask,
// TileProcessor.cuh:1037-1061, GPUTileProcessor.java:547); the correlation keeps the unfiltered copy
__device__ __forceinline__ void store_clt(const SceneDev &sc, int c, int r, float *gdst, float o[4][8]) {
  if (sc.lpf_rbg && ((sc.clt_lpf_mask >> c) & 1)) {
    const float4 *lp = (const float4 *)(sc.lpf_rbg + c * 64 + r * 8);
    const float4 la = __ldg(lp), lb = __ldg(lp + 1);
    const float l[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
      for (int v = 0; v < 8; v++) o[m][v] *= l[v];
  }
#pragma unroll
  for (int m = 0; m < 4; m++) {
    *(float4 *)(gdst + m * 64) = make_float4(o[m][0], o[m][1], o[m][2], o[m][3]);
    *(float4 *)(gdst + m * 64 + 4) = make_float4(o[m][4], o[m][5], o[m][6], o[m][7]);
  }
}

struct FwdShape {
  int nw;                 // warps per CTA (each warp owns whole tiles)
  int S, C, P, RE, quad;  // sensors, colours, pairs, strip entries, quad layout
  int clt_floats, per_warp;
};

// ---------------------------------------------------------------------------
// the three phases of the forward for one tile, shared by the schedules
// ---------------------------------------------------------------------------
// phase A item gt = (colour, group of 4 sensors): lanes 8q..8q+7 own sensor 4g+q
template <int C>
__device__ __forceinline__ void fwd_clt_item(const SceneDev &sc, int S, int task, size_t tile, int gt, int groups,
                                             float *s_clt, float *scr, int lane) {
  const int q = lane >> 3, r = lane & 7;
  const int rr = sc.bayer_red_row, rc = sc.bayer_red_col;
  const int c = gt / groups, g = gt - c * groups;
  const int s = g * 4 + q;
  const bool act = s < S;
  const int sidx = act ? s : S - 1;
  const SubtilePlan p = sc.plan[((size_t)task * S + sidx) * C + c];
  Win w;
  w.img = sc.images[sidx];
  w.pitch = sc.img_pitch;
  w.tlx = p.tlx; w.tly = p.tly; w.W = sc.width; w.H = sc.height;
  w.u16 = sc.img_dtype[sidx];
  w.inside = (p.tlx >= 0) && (p.tly >= 0) && (p.tlx <= sc.width - 16) && (p.tly <= sc.height - 16);
  w.scale = sc.color_scale[c];
  float o[4][8];
  float *tbuf = scr + q * 72;
  if (C == 1) {
    subtile_clt<0>(w, p.rx, p.ry, 0, 0, 0, r, tbuf, o);
  } else if (c < 2) {
    const int pc = ((c == 0 ? rc : 1 - rc) - p.tlx) & 1, pr = ((c == 0 ? rr : 1 - rr) - p.tly) & 1;
    subtile_clt<1>(w, p.rx, p.ry, pc, pr, 0, r, tbuf, o);
  } else {
    const int pg = (p.tlx + p.tly + rc + rr + 1) & 1;
    subtile_clt<2>(w, p.rx, p.ry, 0, 0, pg, r, tbuf, o);
  }
  const float *kp = (p.kidx >= 0) ? sc.kernels[sidx] + (size_t)p.kidx * TP_CLT : nullptr;
  conv_shift(o, kp, p.rx, p.ry, r);
  if (act) {
    // all four quadrants: after the convolution and the shift the Bayer symmetries no longer hold
    float *sdst = s_clt + ((size_t)s * C + c) * TP_CLT + r * 8;
#pragma unroll
    for (int m = 0; m < 4; m++) {
      *(float4 *)(sdst + m * 64) = make_float4(o[m][0], o[m][1], o[m][2], o[m][3]);
      *(float4 *)(sdst + m * 64 + 4) = make_float4(o[m][4], o[m][5], o[m][6], o[m][7]);
    }
    store_clt(sc, c, r, sc.clt + ((tile * S + s) * C + c) * TP_CLT + r * 8, o);
  }
}

// phase B for pair pi: correlation surface to HBM, strip entries folded into cmb
// (NT = strip entries per lane / 32 rounded up: 1 when the extraction reads <= 32 entries)
// lpf: the correlation LPF (64 floats) in shared memory: each lane reads its own two entries,
// which from the kernel's parameter space would take one constant-cache access per lane
template <int C, int NT, bool OACC = false>
__device__ __forceinline__ void fwd_pair(const SceneDev &sc, const CorrConst &cfg, const float *lpf, size_t tile,
                                         int P, int pi, int RE, bool log_mode, const short *strip_code,
                                         const float *s_clt, float *scr, int lane, float cmb[8],
                                         float *corr_out = nullptr, float *oprod = nullptr) {
  const int q = lane >> 3, r = lane & 7;
  float *qb = scr;
  const PairDev pd = cfg.pairs[pi];
  const float *c1 = s_clt + (size_t)pd.cam1 * C * TP_CLT, *c2 = s_clt + (size_t)pd.cam2 * C * TP_CLT;
  // with one strip entry per lane its sample code is read ahead of the correlation arithmetic
  short2 code1 = make_short2(-1, -1);
  if (NT == 1 && pd.in_combo && pd.kind <= 3 && lane < RE)
    code1 = *(const short2 *)&strip_code[(pd.kind * TP_MAX_STRIP * 15 + lane) * 2];
  float acc[4][2];
#pragma unroll
  for (int c = 0; c < C; c++) {
    float d1[4][2], d2[4][2], a2[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int m = 0; m < 4; m++) {
        d1[m][h] = c1[c * TP_CLT + m * 64 + lane + 32 * h];
        d2[m][h] = c2[c * TP_CLT + m * 64 + lane + 32 * h];
        s1 = fmaf(d1[m][h], d1[m][h], s1);
        s2 = fmaf(d2[m][h], d2[m][h], s2);
      }
      const float pr = s1 * s2;
      a2[h] = (pr > 0.0f) ? pr * rsqrtf(pr) : 0.0f;  // |d1| |d2|; approximate square root (~2 ulp)
    }
    const float fz2 = warp_sum(a2[0] + a2[1]) * (1.0f / 64) * cfg.fat_zero * cfg.fat_zero;
    const float wgt = (C == 1) ? 1.0f : cfg.col_weights[c];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const float sw = __fdividef(wgt, a2[h] + fz2);
      const float t0 = d1[0][h] * d2[0][h] + d1[1][h] * d2[1][h] + d1[2][h] * d2[2][h] + d1[3][h] * d2[3][h];
      const float t1 = -d1[1][h] * d2[0][h] + d1[0][h] * d2[1][h] - d1[3][h] * d2[2][h] + d1[2][h] * d2[3][h];
      const float t2 = -d1[2][h] * d2[0][h] - d1[3][h] * d2[1][h] + d1[0][h] * d2[2][h] + d1[1][h] * d2[3][h];
      const float t3 = d1[3][h] * d2[0][h] - d1[2][h] * d2[1][h] - d1[1][h] * d2[2][h] + d1[0][h] * d2[3][h];
      if (c == 0) {
        acc[0][h] = t0 * sw; acc[1][h] = t1 * sw; acc[2][h] = t2 * sw; acc[3][h] = t3 * sw;
      } else {
        acc[0][h] = fmaf(t0, sw, acc[0][h]); acc[1][h] = fmaf(t1, sw, acc[1][h]);
        acc[2][h] = fmaf(t2, sw, acc[2][h]); acc[3][h] = fmaf(t3, sw, acc[3][h]);
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int idx = lane + 32 * h;
    const float l = lpf[idx];
    const int off = (idx >> 3) * 9 + (idx & 7);
#pragma unroll
    for (int qq = 0; qq < 4; qq++) qb[qq * 72 + off] = acc[qq][h] * l;
  }
  __syncwarp();
  {
    // both passes transpose in place: every row is read into registers before any is overwritten
    float x[8], y[8];
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = qb[q * 72 + r * 9 + e];
    dtt2e_fast(x, y, (q >> 1) & 1);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; j++) qb[q * 72 + j * 9 + r] = y[j];
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = qb[q * 72 + r * 9 + e];
    dtt2e_fast(x, y, q & 1);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; e++) qb[q * 72 + r * 9 + e] = y[e];
  }
  __syncwarp();
  // 15x15 unfold (DttRad2.corr_unfold_tile): each lane owns 2 cells (a, b) and writes their mirror
  // images; the quadrants are read into registers first, the surface then overwrites them
  float uA[2], uB[2], uC[2], uD[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int a = (lane >> 3) + 4 * k, b = lane & 7;
    uA[k] = qb[a * 9 + b];
    uB[k] = b ? qb[72 + a * 9 + b - 1] : 0.f;
    uC[k] = a ? qb[144 + (a - 1) * 9 + b] : 0.f;
    uD[k] = (a && b) ? qb[216 + (a - 1) * 9 + b - 1] : 0.f;
  }
  __syncwarp();
  float *cs = qb;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int a = (lane >> 3) + 4 * k, b = lane & 7;
    const float A = uA[k], B = uB[k], Cc = uC[k], D = uD[k];
    cs[(7 + a) * 15 + 7 + b] = 0.25f * (((A + B) + Cc) + D);
    if (b) cs[(7 + a) * 15 + 7 - b] = 0.25f * (((A - B) + Cc) - D);
    if (a) cs[(7 - a) * 15 + 7 + b] = 0.25f * (((A + B) - Cc) - D);
    if (a && b) cs[(7 - a) * 15 + 7 - b] = 0.25f * (((A - B) - Cc) + D);
  }
  __syncwarp();
  if (OACC && (pd.kind == 0 || pd.kind == 1) && !cfg.log_combine) {
    // getMaxXSOrtho profile of a horizontal (lanes 0-14, columns) or vertical (lanes 16-30, rows)
    // pair, symmetrised (even in i, so rows 0..7 carry it) and multiplied into this lane's oprod
    const int half = lane >> 4, j = lane & 15;
    if (half == pd.kind && j < 15) {
      const int stride = half ? 1 : 15, base = half ? j * 15 : j;
#pragma unroll
      for (int i = 0; i < 8; i++)
        oprod[i] *= 0.5f * (cs[base + i * stride] + cs[base + (14 - i) * stride]) + cfg.corr_offset;
    }
  }
  float *gc = corr_out ? corr_out : sc.corr + (tile * P + pi) * TP_CORR;
  for (int o2 = lane; o2 < TP_CORR; o2 += 32) gc[o2] = cs[o2];
  if (pd.in_combo) {
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const int e = lane + 32 * t;
      if (e < RE) {
        const int row = e / 15;
        float d;
        if (pd.kind <= 3) {
          const short2 code = (NT == 1) ? code1 : *(const short2 *)&strip_code[(pd.kind * TP_MAX_STRIP * 15 + e) * 2];
          d = sample_code(cs, code.x);
          if (row > 0) {
            const float d2 = sample_code(cs, code.y);
            d = (isnan(d) || isnan(d2)) ? CUDART_NAN_F : (0.5f * d + 0.5f * d2);
          }
        } else {
          const int scol = e - row * 15 - 7;
          d = strip_sample(cs, 4, pd.bx, pd.by, row, scol, -1);
          if (row > 0) {
            const float d2 = strip_sample(cs, 4, pd.bx, pd.by, row, scol, 1);
            d = (isnan(d) || isnan(d2)) ? CUDART_NAN_F : (0.5f * d + 0.5f * d2);
          }
        }
        if (sc.strips && !corr_out) sc.strips[(tile * P + pi) * RE + e] = d;  // kept for the adjoint
        float v = d + cfg.corr_offset;
        if (v < 0.0f) v = 0.0f;
        if (log_mode) cmb[t] += logf(v);
        else cmb[t] *= cfg.twice_diagonal ? v * v : v;
      }
    }
  }
  __syncwarp();
}

// phase C, lane-parallel half: the combined strip (geometric mean of the pairs' strips) into
// combo (shared) and sc.combo, and this lane's getMaxXSOrtho profile value (lanes 0-14 the
// horizontal pairs' column j, lanes 16-30 the vertical pairs' row j; -inf elsewhere)
template <int NT, bool OACC = false>
__device__ __forceinline__ float fwd_extract_values(const SceneDev &sc, const CorrConst &cfg, int quad, int P, int RE,
                                                    bool log_mode, int ncomb, size_t tile, float *combo, int lane,
                                                    const float cmb[8], const float *oprod) {
#pragma unroll
  for (int t = 0; t < NT; t++) {
    const int e = lane + 32 * t;
    if (e < RE) {
      float v = cmb[t];
      if (log_mode) v = isnan(v) ? CUDART_NAN_F : (isinf(v) ? 0.0f : expf(v / cfg.num_combo) - cfg.corr_offset);
      else if (v > 0.0f) v = powf(v, 1.0f / ncomb) - cfg.corr_offset;
      combo[e] = v;
      if (sc.combo) sc.combo[tile * RE + e] = v;  // kept for the adjoint (and the split extraction)
    }
  }
  float sum = -CUDART_INF_F;
  if (quad && (cfg.num_hor > 0 || cfg.num_vert > 0)) {
    // the surfaces of this tile were just written by this warp (L1/L2 resident)
    const int half = lane >> 4, j = lane & 15;
    const int np = half ? cfg.num_vert : cfg.num_hor;
    if (j < 15 && np > 0) {
      // the symmetrised profile is even in i (d[i] == d[14 - i]), so rows 0..7 carry it; all
      // loads of one pair are issued before their use
      float prod[8];
#pragma unroll
      for (int i = 0; i < 8; i++) prod[i] = OACC ? oprod[i] : 1.f;
      for (int k = 0; k < (OACC ? 0 : np); k++) {
        const float *cc = sc.corr + (tile * P + (half ? cfg.vert_pairs[k] : cfg.hor_pairs[k])) * TP_CORR;
        const int stride = half ? 1 : 15, base = half ? j * 15 : j;
        float a[8], b[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          a[i] = cc[base + i * stride];
          b[i] = cc[base + (14 - i) * stride];
        }
#pragma unroll
        for (int i = 0; i < 8; i++) prod[i] *= 0.5f * (a[i] + b[i]) + cfg.corr_offset;
      }
      sum = 0.f;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float p = prod[i];
        const float v = (p > 0.0f) ? ((np == 2) ? sqrtf(p) : ((np == 1) ? p : powf(p, 1.0f / np))) - cfg.corr_offset
                                   : -cfg.corr_offset;
        sum += v * ((i < 7) ? cfg.notch[i] + cfg.notch[14 - i] : cfg.notch[7]);
      }
    }
  }
  __syncwarp();
  return sum;
}

// phase C, serial half: integer argmax and windowed centroid of the combined strip (getMaxXYInt,
// getMaxXCm), the maxima of the ortho profiles (getMaxXSOrtho), the disparity record
__device__ __forceinline__ void fwd_extract_finish(const SceneDev &sc, const CorrConst &cfg, int quad, size_t tile,
                                                   const float *combo, float sum, int lane) {
  float res[TP_NDISP];
#pragma unroll
  for (int k = 0; k < TP_NDISP; k++) res[k] = (k == 2 || k == 4 || k == 6) ? 0.f : CUDART_NAN_F;
  {
    // integer argmax on row 0 (getMaxXYInt): first maximum over the non-NaN entries
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
    if (vmax >= cfg.min_corr) {
      const int ix = imx - 7;
      res[0] = (float)(-ix);
      res[2] = vmax;
      res[8] = (float)ix;
      int dh = cfg.strip_rows;
      float wys = 1.0f;
      if (dh > cfg.wndy_size) dh = cfg.wndy_size;
      else if (dh < cfg.wndy_size) {
        float swy = cfg.wndy[0];
        for (int i = 1; i < dh; i++) swy += cfg.wndy[i];
        wys = 1.0f / swy;
      }
      float s0 = 0.f, sx = 0.f;
      const int x0 = 7 + ix, nk = dh * 2 * cfg.wndx_size;
      for (int k = lane; k < nk; k += 32) {  // windowed centroid (getMaxXCm), one sample per lane
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
      }
      s0 = warp_sum(s0);
      sx = warp_sum(sx);
      if (s0 != 0.0f) {
        res[1] = -(ix + sx / s0 / 2);
        res[7] = s0;
      }
    }
  }
  if (quad && (cfg.num_hor > 0 || cfg.num_vert > 0)) {
    // getMaxXSOrtho: lanes 0-14 horizontal pairs, lanes 16-30 vertical pairs
    const int half = lane >> 4, j = lane & 15;
    float best = sum;
    int bi = (j < 15) ? j : 99;
#pragma unroll
    for (int o2 = 8; o2 > 0; o2 >>= 1) {  // within each 16-lane half
      const float ob = __shfl_xor_sync(0xffffffffu, best, o2);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o2);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    const int ic = bi, base = half << 4;
    const float f0 = __shfl_sync(0xffffffffu, sum, base + (ic > 0 ? ic - 1 : 0));
    const float f1 = __shfl_sync(0xffffffffu, sum, base + ic);
    const float f2 = __shfl_sync(0xffffffffu, sum, base + (ic < 14 ? ic + 1 : 14));
    float xc = (float)ic;
    if (ic > 0 && ic < 14) {
      const float den = f0 - 2.0f * f1 + f2;
      if (den != 0.0f) xc = ic + 0.5f * (f0 - f2) / den;
    }
    int ir = (int)floorf(xc + 0.5f);
    ir = ir < 0 ? 0 : (ir > 14 ? 14 : ir);
    const float fr = __shfl_sync(0xffffffffu, sum, base + ir);
    const float hx = __shfl_sync(0xffffffffu, xc, 0), hs = __shfl_sync(0xffffffffu, fr, 0);
    const float vx = __shfl_sync(0xffffffffu, xc, 16), vs = __shfl_sync(0xffffffffu, fr, 16);
    if (cfg.num_hor > 0) { res[3] = -(hx - 7.0f); res[4] = hs / 8.0f; }
    if (cfg.num_vert > 0) { res[5] = -(vx - 7.0f); res[6] = vs / 8.0f; }
  }
  float *dm = sc.disp + tile * TP_NDISP;
  if (lane < TP_NDISP) {
    float v = res[0];
#pragma unroll
    for (int k = 1; k < TP_NDISP; k++) if (lane == k) v = res[k];
    dm[lane] = v;
  }
  __syncwarp();
}

// phase C: combined strip, integer argmax, centroid, ortho maxima, disparity record
template <int NT, bool OACC = false>
__device__ __forceinline__ void fwd_extract(const SceneDev &sc, const CorrConst &cfg, int quad, int P, int RE,
                                            bool log_mode, int ncomb, size_t tile, float *scr, int lane,
                                            const float cmb[8], const float *oprod = nullptr) {
  const float sum = fwd_extract_values<NT, OACC>(sc, cfg, quad, P, RE, log_mode, ncomb, tile, scr, lane, cmb, oprod);
  fwd_extract_finish(sc, cfg, quad, tile, scr, sum, lane);
}

// ---------------------------------------------------------------------------
// Staged windows: a warp copies the 16x16 windows of four sensors into shared memory with 16-byte
// cp.async chunks (lanes 8q..8q+7 sensor q), from the 16-byte boundary at or below the window's
// corner.  The fold then reads shared memory; read from global memory, each of its loads touches 32
// image rows, one L1 access each.  Image rows start on 16-byte boundaries because the pitch is a
// multiple of 8 pixels.  Windows that cross the image border are copied pair by pair with the edge mirroring.
// Rows of u16 windows are 24 pixels (three chunks); rows of float windows 20 (five chunks).  The sensors' windows
// lie 8 banks apart, so that a dense fold's reads (eight rows of four sensors) meet in a bank 3.4 times on average
// over the corners' positions (u16 without the 8 floats 4.2; even and odd rows apart 2.2, but that costs more
// instructions than it saves accesses: 693 -> 705 us at 4 x 2592x1936).
// ---------------------------------------------------------------------------
template <bool U16>
struct Stage {
  using T = float;
  static constexpr int CH = 4, NCH = 5, ROW = 20, WIN = 328;  // pixels per chunk, chunks per row, row, window (floats)
};
template <>
struct Stage<true> {
  using T = uint16_t;
  static constexpr int CH = 8, NCH = 3, ROW = 24, WIN = 200;
};

__device__ __forceinline__ void cp_async16(void *dst_smem, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
// a pair of pixels: 4 bytes of u16, 8 of float
__device__ __forceinline__ void cp_async_pair(uint16_t *dst_smem, const uint16_t *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_pair(float *dst_smem, const float *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// pixel source of subtile_clt: a staged window, column sx of the 16-byte aligned copy
template <bool U16>
struct SWin {
  const typename Stage<U16>::T *base;
  int sx;
  float scale;
  __device__ __forceinline__ float at(int row, int col) const {
    return (float)base[row * Stage<U16>::ROW + sx + col] * scale;
  }
};

// lane r (0..7) of a sensor's 8 lanes copies its share of the window at corner (tlx, tly) into dst; a
// row's last chunk is left out where it would pass the row's end (the corner is then 16-byte aligned
// and the window lies in the chunks before it)
template <bool U16>
__device__ __forceinline__ void stage_window(const SceneDev &sc, const void *image, int tlx, int tly, float *dst_f, int r) {
  using S = Stage<U16>;
  using T = typename S::T;
  const T *img = (const T *)image;
  T *dst = (T *)dst_f;
  const int x0 = tlx & ~(S::CH - 1), W = sc.width, H = sc.height;
  const int64_t pitch = sc.img_pitch;
  if (tlx >= 0 && tly >= 0 && tlx <= W - 16 && tly <= H - 16) {
    const bool last = x0 + S::ROW <= W;
#pragma unroll
    for (int j = 0; j < 2 * S::NCH; j++) {
      const int k = r + 8 * j, row = k / S::NCH, part = k - row * S::NCH;
      if (part < S::NCH - 1 || last)
        cp_async16(dst + row * S::ROW + part * S::CH, img + (size_t)(tly + row) * pitch + x0 + part * S::CH);
    }
  } else {
    // The edge mirroring (mirror()) keeps a column's parity and W is even, so a pair of columns
    // (even, odd) comes from a pair: (0, 1) or (W - 2, W - 1) outside.  A cp.async per pair.
    constexpr int PR = S::ROW / 2;
#pragma unroll 2
    for (int j = 0; j < 2 * PR; j++) {
      const int k = r + 8 * j, row = k / PR, x = x0 + 2 * (k - row * PR);
      const int xs = x < 0 ? 0 : (x >= W ? W - 2 : x);
      cp_async_pair(dst + row * S::ROW + (x - x0), img + (size_t)mirror(tly + row, H) * pitch + xs);
    }
  }
}

}  // namespace
