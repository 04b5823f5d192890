// tp_adjoint.cu -- hand-written adjoint of the forward chain (mono and Bayer colour sensors).
//
// For every tile the centroid disparity d (getMaxXCm over the combined strip,
// Correlation2d.java:936-1032) is a function of the residual shifts (rx, ry)
// of each sensor's window (ImageDtt.java:4940-4943), which follow the port
// coordinates, which follow the per-sensor extrinsics and the tile's target
// disparity (GeometryCorrection.getPortsCoordinatesAndDerivatives,
// GeometryCorrection.java:2159-2314).  The adjoint kernel computes, per tile,
// d and dd/d(port x, port y) of every sensor by reverse mode through
//   centroid -> strip combination (geometric mean) -> strip sampling ->
//   15x15 unfold -> 2D DCT-IIe/DST-IIe -> LPF -> fat-zero normalised product
// (Correlation2d.java:197-231, 556-790; DttRad2.java:443-489, 595-614) down to
// dd/dCLT of each sensor, then by forward mode through the CLT's dependence
// on the residual shift: the phase rotation (fract_shift, ImageDtt.java:
// 5490-5584) differentiated analytically, and the shifted fold window
// (DttRad2.get_shifted_fold_2d, 263-314) differentiated through its cos/sin
// mix.  The integer window corners and the integer argmax are piecewise
// constant and are held fixed.
//
// A second kernel contracts those port sensitivities with the FP64 port
// derivatives of the plan (azimuth, tilt, roll, zoom, disparity) into the
// per-tile Jacobian rows and the gradient of a per-tile loss.
//
// GB300 layout: one CTA of four warps per tile.  The tile's CLT [S][256]
// (read back from HBM or recomputed from the image) and its gradient [S][256]
// live in shared memory; warp 0 takes the centroid of the combined strip the
// forward kernel kept; then the warps split the pairs, each running a pair's
// reverse chain in registers and per-warp buffers (the transposed DCT-IIe is
// the transposed butterfly of the forward one) and adding into the gradient;
// the pairs go in rounds of four on distinct sensors (scheduled on the host),
// a barrier between rounds, so the gradient sums over the pairs are taken in a
// fixed order without atomics (a pair's strip taps go into its own 15x15
// gradient with one warp's shared-memory atomics); finally the warps split the
// sensors for the forward-mode shift derivatives.
#include "tp_adjoint.cuh"
#include "tp_pairs.cuh"
#include "tp_launch.h"

__global__ void __launch_bounds__(32 * AD_NW, 4) adjoint_kernel(const __grid_constant__ SceneDev sc,
                                                             const __grid_constant__ AdjShape as,
                                                             const __grid_constant__ CorrConst cfg, float *sens,
                                                             float *dval) {
  extern __shared__ float sm[];
  __shared__ float s_d;
  __shared__ float s_sens[2 * TP_MAXS * 3];  // dd/d(port x, y) of every (sensor, colour)
  __shared__ float s_lpf[64];                // the correlation LPF, read per lane
  for (int i = threadIdx.x; i < 64; i += blockDim.x) s_lpf[i] = cfg.lpf[i];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 3, r = lane & 7;
  const int S = as.S, C = as.C, P = as.P, RE = as.RE;
  float *s_clt = sm;                      // [S][C][256]
  float *s_g = s_clt + S * C * TP_CLT;    // [S][C][256] dd/dCLT
  float *gcmb = s_g + S * C * TP_CLT;     // [240] dd/dcombo
  float *gG = gcmb + 240;             // [240] combo + offset
  float *gs = gG + 240 + warp * 816;  // per warp: [240] dd/dsurface of the current pair
  float *qb = gs + 240;               // [4][72] quadrant buffer
  float *tb = qb + 288;               // [4][72] transpose buffer
  const short *strip_code = &sc.corr_cfg->strip_code[0][0][0];
  const float inv_n = 1.0f / cfg.num_combo;

  for (int task = blockIdx.x; task < sc.num_tasks; task += gridDim.x) {
    const int txy = sc.task_txy[task];
    const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
    // ---------------- the tile's CLT ----------------
    if (as.recompute) {
      // every (sensor, colour) item, four per 8-lane group: a Bayer colour as the sparse plane of
      // its pixels (the dense fold of the masked window is the forward's CLT of that plane)
      const int items = S * C;
      for (int g = warp; g < (items + 3) / 4; g += AD_NW) {
        const int it = g * 4 + q;
        const int itc = it < items ? it : items - 1;
        const int s = itc / C, c = itc - s * C;
        const SubtilePlan p = sc.plan[(size_t)task * items + itc];
        float ahs, ahc, avs, avc;
        __sincosf(CUDART_PI_F * 0.0625f * p.rx, &ahs, &ahc);
        __sincosf(CUDART_PI_F * 0.0625f * p.ry, &avs, &avc);
        const FoldIdx fv = fold_idx(r);
        float vw0, vw1, hw0[8], hw1[8], o[4][8];
        fold_weights(ahc, ahs, avc, avs, fv, vw0, vw1, hw0, hw1);
        if (C == 1) {
          fold_dtt_dense(make_win(sc, p, s), fv, vw0, vw1, hw0, hw1, r, tb + q * 72, o);
        } else {
          BayerWin bw;
          bw.w = make_win(sc, p, s, c);
          bw.c = c;
          bw.rr = sc.bayer_red_row;
          bw.rc = sc.bayer_red_col;
          fold_dtt_dense(bw, fv, vw0, vw1, hw0, hw1, r, tb + q * 72, o);
        }
        convolve(o, (p.kidx >= 0) ? sc.kernels[s] + (size_t)p.kidx * TP_CLT : nullptr, r);
        rotate(o, p.rx, p.ry, r);
        if (it < items) {
#pragma unroll
          for (int m = 0; m < 4; m++)
#pragma unroll
            for (int v = 0; v < 8; v++) s_clt[it * TP_CLT + m * 64 + r * 8 + v] = o[m][v];
        }
      }
    } else {
      const float4 *src = (const float4 *)(sc.clt + tile * S * C * TP_CLT);
      for (int i = tid; i < S * C * 64; i += 32 * AD_NW) ((float4 *)s_clt)[i] = __ldg(src + i);
    }
    for (int i = tid; i < S * C * TP_CLT; i += 32 * AD_NW) s_g[i] = 0.f;

    // ---------------- centroid of the forward's combined strip, and dd/dcombo ----------------
    if (warp == 0) {
      for (int e = lane; e < 240; e += 32) {
        gG[e] = (e < RE) ? sc.combo[tile * RE + e] : 0.f;
        gcmb[e] = 0.f;
      }
      __syncwarp();
      const float dres = strip_centroid(cfg, gG, gcmb, lane);
      // G = combo + offset, the geometric mean the strip entries enter
      for (int e = lane; e < RE; e += 32) gG[e] = gG[e] + cfg.corr_offset;
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

    // ---------------- reverse pass over the pairs, one round of AD_NW pairs at a time ----------------
    // A round's pairs are on distinct sensors (the host's schedule), so the warps add their CLT
    // gradients into disjoint parts of s_g; the barrier after each round orders the rounds, so
    // every gradient entry is summed in the same order in every run.  With the forward's strip
    // samples recorded and one entry per lane, the next round's sample is loaded one round ahead
    // so its latency overlaps this pair.
    const bool pre = as.use_strips && RE <= 32;
    const short *sched = &sc.corr_cfg->adj_round[0][0];
    int pnext = cfg.adj_rounds > 0 ? sched[warp] : -1;
    float vnext = 0.f;
    if (pre && pnext >= 0 && lane < RE) vnext = sc.strips[(tile * P + pnext) * RE + lane];
    for (int rd = 0; rd < cfg.adj_rounds; rd++) {
      const int pi = pnext;
      const float vcur = vnext;
      pnext = rd + 1 < cfg.adj_rounds ? sched[(rd + 1) * AD_NW + warp] : -1;
      if (pre && pnext >= 0 && lane < RE) vnext = sc.strips[(tile * P + pnext) * RE + lane];
      do {  // this warp's pair of the round (break: nothing to add)
        if (pi < 0) break;
        const PairDev pd = cfg.pairs[pi];
        if (!pd.in_combo) break;
        const float *c = sc.corr + (tile * P + pi) * TP_CORR;
        for (int i = lane; i < 240; i += 32) gs[i] = 0.f;
        for (int i = lane; i < 288; i += 32) qb[i] = 0.f;
        __syncwarp();
        // strip entries: d combo / d v_p = G / (n v_p) for the geometric mean of n pairs
        bool any = false;
        for (int e = lane; e < RE; e += 32) {
          if (gcmb[e] == 0.f) continue;
          const float d = pre ? vcur
                              : (as.use_strips ? sc.strips[(tile * P + pi) * RE + e]
                                               : strip_entry(c, strip_code, pd, e));
          const float v = d + cfg.corr_offset;
          if (!(v > 0.0f)) continue;
          const float f = __fdividef(gcmb[e] * gG[e] * inv_n, v);
          const int row = e / 15;
          const float half = row > 0 ? 0.5f : 1.0f;
          for (int side = 0; side < (row > 0 ? 2 : 1); side++) {
            int idx[4];
            float wt[4];
            int n;
            if (pd.kind <= 3) {
              const short2 code = *(const short2 *)&strip_code[(pd.kind * TP_MAX_STRIP * 15 + e) * 2];
              n = code_taps(side ? code.y : code.x, idx, wt);
            } else {
              n = general_taps(pd.bx, pd.by, row, e - row * 15 - 7, side ? 1 : -1, idx, wt);
            }
            for (int k = 0; k < n; k++) atomicAdd(&gs[idx[k]], f * half * wt[k]);
          }
          any = true;
        }
        if (!__any_sync(0xffffffffu, any)) break;
        __syncwarp();
        // 15x15 unfold (DttRad2.corr_unfold_tile) transposed into the four quadrants
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const int a = (lane >> 3) + 4 * k, b = lane & 7;
          const float g1 = gs[(7 + a) * 15 + 7 + b];
          const float g2 = b ? gs[(7 + a) * 15 + 7 - b] : 0.f;
          const float g3 = a ? gs[(7 - a) * 15 + 7 + b] : 0.f;
          const float g4 = (a && b) ? gs[(7 - a) * 15 + 7 - b] : 0.f;
          qb[a * 9 + b] = 0.25f * (((g1 + g2) + g3) + g4);
          if (b) qb[72 + a * 9 + b - 1] = 0.25f * (((g1 - g2) + g3) - g4);
          if (a) qb[144 + (a - 1) * 9 + b] = 0.25f * (((g1 + g2) - g3) - g4);
          if (a && b) qb[216 + (a - 1) * 9 + b - 1] = 0.25f * (((g1 - g2) - g3) + g4);
        }
        __syncwarp();
        // 2D DCT-IIe/DST-IIe transposed: forward Z = Ta X^T Tb^T, so Xbar = Tb^T Zbar^T Ta
        {
          float z[8], v[8];
#pragma unroll
          for (int k = 0; k < 8; k++) z[k] = qb[q * 72 + k * 9 + r];  // column r of Zbar
          dtt2e_transposed(z, v, (q >> 1) & 1);                        // row r of V = Zbar^T Ta
#pragma unroll
          for (int n = 0; n < 8; n++) tb[q * 72 + r * 9 + n] = v[n];
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; k++) z[k] = tb[q * 72 + k * 9 + r];  // column r of V
          dtt2e_transposed(z, v, q & 1);                               // column r of Xbar
#pragma unroll
          for (int k = 0; k < 8; k++) qb[q * 72 + k * 9 + r] = v[k];
          __syncwarp();
        }
        // LPF, colour mix and the fat-zero normalised product of each colour
        // (correlateSingleColorFD / correlateCompositeFD): acc = sum_c w_c t_c / (a2_c + fz2_c)
        float gq[4][2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int idx = lane + 32 * h;
          const float l = s_lpf[idx];
          const int off = (idx >> 3) * 9 + (idx & 7);
#pragma unroll
          for (int qq = 0; qq < 4; qq++) gq[qq][h] = qb[qq * 72 + off] * l;
        }
        const float fzz = cfg.fat_zero * cfg.fat_zero;
        for (int c = 0; c < C; c++) {
          const float wgt = (C == 1) ? 1.0f : cfg.col_weights[c];
          const float *c1 = s_clt + ((size_t)pd.cam1 * C + c) * TP_CLT;
          const float *c2 = s_clt + ((size_t)pd.cam2 * C + c) * TP_CLT;
          float d1[4][2], d2[4][2], a2[2], ia2[2], s1v[2], s2v[2];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float s1 = 0.f, s2 = 0.f;
#pragma unroll
            for (int m = 0; m < 4; m++) {
              d1[m][h] = c1[m * 64 + lane + 32 * h];
              d2[m][h] = c2[m * 64 + lane + 32 * h];
              s1 = fmaf(d1[m][h], d1[m][h], s1);
              s2 = fmaf(d2[m][h], d2[m][h], s2);
            }
            // |d1| |d2| with the forward's approximate square root; ia2 = 1 / a2 (0 where a2 = 0)
            const float pr = s1 * s2;
            ia2[h] = (pr > 0.0f) ? rsqrtf(pr) : 0.0f;
            a2[h] = pr * ia2[h];
            s1v[h] = s1;
            s2v[h] = s2;
          }
          const float fz2 = warp_sum(a2[0] + a2[1]) * (1.0f / 64) * fzz;
          float tg[4][2], dbar[2];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const float u = __fdividef(1.0f, a2[h] + fz2);
            const float t0 = d1[0][h] * d2[0][h] + d1[1][h] * d2[1][h] + d1[2][h] * d2[2][h] + d1[3][h] * d2[3][h];
            const float t1 = -d1[1][h] * d2[0][h] + d1[0][h] * d2[1][h] - d1[3][h] * d2[2][h] + d1[2][h] * d2[3][h];
            const float t2 = -d1[2][h] * d2[0][h] - d1[3][h] * d2[1][h] + d1[0][h] * d2[2][h] + d1[1][h] * d2[3][h];
            const float t3 = d1[3][h] * d2[0][h] - d1[2][h] * d2[1][h] - d1[1][h] * d2[2][h] + d1[0][h] * d2[3][h];
            const float swbar = gq[0][h] * t0 + gq[1][h] * t1 + gq[2][h] * t2 + gq[3][h] * t3;
            dbar[h] = -wgt * swbar * u * u;
            const float sw = wgt * u;
#pragma unroll
            for (int qq = 0; qq < 4; qq++) tg[qq][h] = gq[qq][h] * sw;
          }
          const float dsum = warp_sum(dbar[0] + dbar[1]) * (1.0f / 64) * fzz;
          float *g1p = s_g + ((size_t)pd.cam1 * C + c) * TP_CLT, *g2p = s_g + ((size_t)pd.cam2 * C + c) * TP_CLT;
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int idx = lane + 32 * h;
            const float a2bar = dbar[h] + dsum;
            const float T0 = tg[0][h], T1 = tg[1][h], T2 = tg[2][h], T3 = tg[3][h];
            float g1[4], g2[4];
            g1[0] = T0 * d2[0][h] + T1 * d2[1][h] + T2 * d2[2][h] + T3 * d2[3][h];
            g1[1] = T0 * d2[1][h] - T1 * d2[0][h] + T2 * d2[3][h] - T3 * d2[2][h];
            g1[2] = T0 * d2[2][h] + T1 * d2[3][h] - T2 * d2[0][h] - T3 * d2[1][h];
            g1[3] = T0 * d2[3][h] - T1 * d2[2][h] - T2 * d2[1][h] + T3 * d2[0][h];
            g2[0] = T0 * d1[0][h] - T1 * d1[1][h] - T2 * d1[2][h] + T3 * d1[3][h];
            g2[1] = T0 * d1[1][h] + T1 * d1[0][h] - T2 * d1[3][h] - T3 * d1[2][h];
            g2[2] = T0 * d1[2][h] - T1 * d1[3][h] + T2 * d1[0][h] - T3 * d1[1][h];
            g2[3] = T0 * d1[3][h] + T1 * d1[2][h] + T2 * d1[1][h] + T3 * d1[0][h];
            // a2 = sqrt(s1 s2): d a2 / d d1[m] = d1[m] s2 / a2
            const float k1 = a2bar * s2v[h] * ia2[h];
            const float k2 = a2bar * s1v[h] * ia2[h];
#pragma unroll
            for (int m = 0; m < 4; m++) {  // no other warp adds to these sensors in this round
              g1p[m * 64 + idx] += fmaf(k1, d1[m][h], g1[m]);
              g2p[m * 64 + idx] += fmaf(k2, d2[m][h], g2[m]);
            }
          }
        }
        __syncwarp();
      } while (0);
      __syncthreads();
    }

    // ---------------- dd/drx, dd/dry per sensor and colour (forward mode on the CLT) ----------------
    const int items = S * C;
    for (int g = warp; g < (items + 3) / 4; g += AD_NW) {
      const int it = g * 4 + q;
      const int itc = it < items ? it : items - 1;
      const int s = itc / C, c = itc - s * C;
      const SubtilePlan p = sc.plan[(size_t)task * S * C + itc];
      float gxy[2];
      if (C == 1) {
        shift_sens(sc, make_win(sc, p, s), p, s, s_clt + (size_t)itc * TP_CLT, s_g + (size_t)itc * TP_CLT,
                   tb + q * 72, r, it < items, gxy);
      } else {
        BayerWin bw;
        bw.w = make_win(sc, p, s, c);
        bw.c = c;
        bw.rr = sc.bayer_red_row;
        bw.rc = sc.bayer_red_col;
        shift_sens(sc, bw, p, s, s_clt + (size_t)itc * TP_CLT, s_g + (size_t)itc * TP_CLT, tb + q * 72, r,
                   it < items, gxy);
      }
      if (r == 0 && it < items) {
        s_sens[it * 2] = gxy[0];
        s_sens[it * 2 + 1] = gxy[1];
      }
    }
    __syncthreads();
    // a sensor's colours share its port: their sensitivities add, in colour order
    for (int i = tid; i < 2 * S; i += 32 * AD_NW) {
      const int s = i >> 1, k = i & 1;
      float v = 0.f;
      for (int c = 0; c < C; c++) v += s_sens[(s * C + c) * 2 + k];
      sens[(tile * S + s) * 2 + k] = v;
    }
    if (tid == 0) dval[tile] = dres;
    __syncthreads();
  }
}

// Per tile: Jacobian rows of d w.r.t. the sensors' (azimuth, tilt, roll, zoom)
// and the tile disparity, and the loss gradient with dL/dd = dl_dd (or 2 d).
// One thread per (task, sensor); a block holds 256 / S tasks.  The per-task sum
// over sensors and the block's partial sums of the extrinsic gradient (to
// `partial`) are taken in a fixed order, so the result is deterministic.
__global__ void __launch_bounds__(256) adjoint_contract_kernel(const __grid_constant__ SceneDev sc,
                                                              const float *sens, const float *dval,
                                                              const float *dl_dd, float *jac_e, float *jac_d,
                                                              float *grad_d, float *partial) {
  __shared__ float s_jd[256];
  __shared__ float s_ge[256][4];
  const int S = sc.num_sensors, tpb = 256 / S;
  const int lt = threadIdx.x / S, s = threadIdx.x - lt * S;
  const int task = blockIdx.x * tpb + lt;
  const bool act = lt < tpb && task < sc.num_tasks;
  float jd = 0.f, ge[4] = {0.f, 0.f, 0.f, 0.f};
  size_t tile = 0;
  float gbar = 0.f;
  if (act) {
    const int txy = sc.task_txy[task];
    tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
    const float d = dval[tile];
    gbar = isnan(d) ? 0.f : (dl_dd ? dl_dd[tile] : 2.0f * d);
    const double *pd = sc.port_deriv + ((size_t)task * S + s) * 10;
    const float jx = sens[(tile * S + s) * 2], jy = sens[(tile * S + s) * 2 + 1];
    float j4[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      j4[k] = jx * (float)pd[k] + jy * (float)pd[5 + k];
      ge[k] = gbar * j4[k];
    }
    *(float4 *)(jac_e + (tile * S + s) * 4) = make_float4(j4[0], j4[1], j4[2], j4[3]);
    jd = jx * (float)pd[4] + jy * (float)pd[9];
  }
  s_jd[threadIdx.x] = jd;
#pragma unroll
  for (int k = 0; k < 4; k++) s_ge[threadIdx.x][k] = ge[k];
  __syncthreads();
  if (act && s == 0) {  // sensors in order
    float t = 0.f;
    for (int q = 0; q < S; q++) t += s_jd[lt * S + q];
    jac_d[tile] = t;
    grad_d[tile] = gbar * t;
  }
  if (threadIdx.x < S * 4) {  // the block's tasks in order
    const int ss = threadIdx.x >> 2, k = threadIdx.x & 3;
    float v = 0.f;
    for (int q = 0; q < tpb; q++) v += s_ge[q * S + ss][k];
    partial[(size_t)blockIdx.x * S * 4 + threadIdx.x] = v;
  }
}

// One block per extrinsic coordinate i: thread t sums the partials of blocks t, t + 256, ... in
// order, then a fixed tree over the 256 threads (deterministic; a single thread walking all
// partials waited on one dependent load per block)
__global__ void __launch_bounds__(256) adjoint_final_kernel(const float *partial, int nblocks, int n,
                                                            float *grad_e) {
  __shared__ float s[256];
  const int i = blockIdx.x, t = threadIdx.x;
  float v = 0.f;
  for (int b = t; b < nblocks; b += 256) v += partial[(size_t)b * n + i];
  s[t] = v;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (t < h) s[t] += s[t + h];
    __syncthreads();
  }
  if (t == 0) grad_e[i] = s[0];
}

// The strip samples of a forward that did not record them, from its stored surfaces (the recorded values' bits: the
// forward's own functions on the same surfaces): a warp per (task, pair), strips of at most 32 entries.  With them
// the per-tile kernel of a scene does not depend on what the handle ran before.
__global__ void __launch_bounds__(128) sample_strips_kernel(const __grid_constant__ SceneDev sc, int RE) {
  const int lane = threadIdx.x & 31, P = sc.num_pairs;
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), task = i / P, pi = i - task * P;
  if (task >= sc.num_tasks || lane >= RE) return;
  const CorrDev &cd = *sc.corr_cfg;
  const int kind = cd.pairs[pi].kind;
  if (!cd.pairs[pi].in_combo) return;
  const int txy = sc.task_txy[task];
  const size_t at = ((size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff)) * P + pi;
  const float *c = sc.corr + at * TP_CORR;
  sc.strips[at * RE + lane] = kind == 4 ? tap_strip(c, *((const float4 *)cd.gen_tap[pi] + lane), cd.gen_cell[pi][lane], lane >= 15)
                                        : strip_of(c, quad_code(&cd.strip_code[0][0][0], kind, lane), lane);
}

cudaError_t upload_adjoint_constants() {
  cudaError_t e = upload_dtt_constants();
  if (e != cudaSuccess) return e;
  return cudaSuccess;
}

int adjoint_smem_bytes(int S, int C) { return (S * C * 2 * TP_CLT + 240 + 240 + AD_NW * 816) * 4; }

cudaError_t launch_adjoint(const SceneDev &sc, const CorrConst &cc, int recompute, int use_strips, float *sens,
                           float *dval,
                           const float *dl_dd, float *jac_e, float *jac_d, float *grad_d, float *partial,
                           float *grad_e, cudaStream_t st) {
  if (sc.num_tasks <= 0) return cudaSuccess;
  if ((sc.num_colors != 1 && sc.num_colors != 3) || !sc.port_deriv || !sc.combo) return cudaErrorInvalidValue;
  AdjShape as;
  as.S = sc.num_sensors;
  as.C = sc.num_colors;
  as.P = sc.num_pairs;
  as.RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  as.per_warp = adjoint_smem_bytes(as.S, as.C) / 4;
  as.recompute = recompute;
  as.use_strips = (use_strips && sc.strips) ? 1 : 0;
  const int bytes = adjoint_smem_bytes(as.S, as.C);
  cudaError_t e;
  const bool many = sc.strips && adjoint_many_ok(sc, recompute), quad = sc.strips && adjoint_quad_ok(sc, recompute);
  if (many || quad) {
    if (!as.use_strips) {
      sample_strips_kernel<<<(sc.num_tasks * sc.num_pairs + 3) / 4, 128, 0, st>>>(sc, as.RE);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    e = many ? launch_adjoint_many(sc, cc, sens, dval, st) : launch_adjoint_quad(sc, cc, sens, dval, st);
  } else {
    int res = 0;
    e = kernel_residency((const void *)adjoint_kernel, 32 * AD_NW, bytes, &res);
    if (e != cudaSuccess) return e;
    if (res < 1) return cudaErrorInvalidConfiguration;
    adjoint_kernel<<<sc.num_tasks < res ? sc.num_tasks : res, 32 * AD_NW, bytes, st>>>(sc, as, cc, sens, dval);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return e;
  const int nb = (sc.num_tasks + 256 / sc.num_sensors - 1) / (256 / sc.num_sensors);
  adjoint_contract_kernel<<<nb, 256, 0, st>>>(sc, sens, dval, dl_dd, jac_e, jac_d, grad_d, partial);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  adjoint_final_kernel<<<sc.num_sensors * 4, 256, 0, st>>>(partial, nb, sc.num_sensors * 4, grad_e);
  return cudaGetLastError();
}
