// tp_adjoint_quad.cu -- the adjoint's per-tile kernel for Bayer scenes of a standard quad.
//
// adjoint_kernel (tp_adjoint.cu) splits a quad's six pairs over its warps in rounds of two pairs, with
// all three colours of a pair in one warp and a barrier a round: two of four warps wait most of the time.
// Here a tile has three warps.  Each takes a couple of pairs (two per instruction, tp_adjoint_pairs.cuh)
// from the strip to the filtered spectra; after one barrier each takes a colour through all six pairs,
// keeping the four sensors' gradients in registers, and on to the shift derivatives of the colour's four
// sub-tiles, whose windows were staged at the start and whose Bayer planes are folded without their
// zeros.
// Measured on 4x648x488 with kernel tables (4,941 tiles): 280 -> 116 us.  What bounds it now: latency at
// 15 warps an SM (128 registers a thread) and, at this size, the last of 6.5 rounds of tiles.
#include "tp_adjoint_pairs.cuh"
#include "tp_launch.h"

namespace {

constexpr int AQ_NW = 3;
// floats: CLT and its gradient [3 colours][4][256], spectra of the three couples, strip, windows
template <bool U16>
__host__ __device__ constexpr int aq_floats() {
  return 2 * 3 * 1024 + 3 * QP_BUF + AQ_NW * 64 + AQ_NW * 4 * Stage<U16>::WIN;
}

// The strip gradients of a couple (lanes 0-14 the first pair's, lanes 16-30 the second's) spread into the
// surface gradients g[2][228].  A quad's strip entries lie a cell apart, so no two lanes share a cell.
__device__ __forceinline__ void scatter_quad(float *g, float f0, float f1, const short *strip_code, int kind, int lane) {
  const int j = min(lane & 15, 14);
  float *gp = g + (lane >> 4) * AM_SURF;
  const short2 c0 = *(const short2 *)&strip_code[(kind * TP_MAX_STRIP * 15 + j) * 2];
  const short2 c1 = *(const short2 *)&strip_code[(kind * TP_MAX_STRIP * 15 + 15 + j) * 2];
  auto add = [&](int code, float f) {  // cell in bits 0-7, half steps right and down in bits 8 and 9
    add_entry(gp + (code & 255), f, f != 0.f && code >= 0, (code & 0x100) ? 0.5f : 0.f, (code & 0x200) ? 0.5f : 0.f, 0, 0);
  };
  add(c0.x, f0);
  add(c1.x, 0.5f * f1);
  add(c1.y, 0.5f * f1);
}

// the part of shift_sens after the folded gradient gf (row r of the lane's sub-tile): the fold of a Bayer
// plane's pixels under the window's derivative by each direction, dotted with gf, added to gdir.  A red
// or blue plane has one pixel per folded value, a green one two; the arithmetic is the dense fold's without
// the terms that are zero.
template <bool GREEN, typename PIX>
__device__ __forceinline__ void fold_deriv_bayer(const PIX &w, const SubtilePlan &p, int pc, int pr, const float gf[4][8],
                                                 int r, float gdir[2]) {
  float ahs, ahc, avs, avc;
  __sincosf(CUDART_PI_F * 0.0625f * p.rx, &ahs, &ahc);
  __sincosf(CUDART_PI_F * 0.0625f * p.ry, &avs, &avc);
  const FoldIdx fv = fold_idx(r);
  // the pixel of column src0 (src1) of folded column j lies in source row 0 or 1 of the lane; red, blue:
  // only the column of parity pc, in the row of parity pr; green: pc is the parity of row + column
  float px[8][GREEN ? 2 : 1];
  bool in1[8];  // red, blue: column src1 holds the pixel; green: column src0's pixel lies in row src1
  const bool row1 = (fv.src0 & 1) != pr;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const FoldIdx fh = fold_idx(j);
    if (GREEN) {
      in1[j] = ((fv.src0 + fh.src0) & 1) != pc;
      px[j][0] = w.at(in1[j] ? fv.src1 : fv.src0, fh.src0);
      px[j][GREEN ? 1 : 0] = w.at(in1[j] ? fv.src0 : fv.src1, fh.src1);
    } else {
      in1[j] = (fh.src0 & 1) != pc;
      px[j][0] = w.at(row1 ? fv.src1 : fv.src0, in1[j] ? fh.src1 : fh.src0);
    }
  }
#pragma unroll
  for (int dir = 0; dir < 2; dir++) {
    float vw0, vw1, hw0[8], hw1[8];
    if (dir == 0) fold_weights(-K16 * ahs, K16 * ahc, avc, avs, fv, vw0, vw1, hw0, hw1);
    else fold_weights(ahc, ahs, -K16 * avs, K16 * avc, fv, vw0, vw1, hw0, hw1);
    float acc = 0.f;
#pragma unroll
    for (int vb = 0; vb < 2; vb++) {
      const float k0 = (vb ? fv.ss0 : fv.sc0) * vw0, k1 = (vb ? fv.ss1 : fv.sc1) * vw1;
#pragma unroll
      for (int hb = 0; hb < 2; hb++)
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const FoldIdx fh = fold_idx(j);
          const float h0 = (hb ? fh.ss0 : fh.sc0) * hw0[j], h1 = (hb ? fh.ss1 : fh.sc1) * hw1[j];
          float f;
          if (GREEN) {
            const float v0 = (in1[j] ? k1 : k0) * px[j][0], v1 = (in1[j] ? k0 : k1) * px[j][GREEN ? 1 : 0];
            f = fmaf(h1, v1, h0 * v0);
          } else {
            f = (in1[j] ? h1 : h0) * ((row1 ? k1 : k0) * px[j][0]);
          }
          acc = fmaf(f, gf[vb * 2 + hb][j], acc);
        }
    }
    gdir[dir] += acc;
  }
}

}  // namespace

template <bool U16>
__global__ void __launch_bounds__(32 * AQ_NW, 5) adjoint_quad_kernel(const __grid_constant__ SceneDev sc,
                                                                     const __grid_constant__ CorrConst cfg, int RE,
                                                                     float *sens, float *dval) {
  extern __shared__ float sm[];
  __shared__ unsigned s_any[3];    // lanes with a strip gradient, per couple (lower half: its first pair)
  __shared__ float s_sens[12 * 2]; // dd/d(port x, port y) of every (sensor, colour)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3, r = lane & 7;
  const int c = warp;  // this warp's colour (and its couple)
  float *s_clt = sm + c * 1024;                 // the colour's CLT [4][256]
  float *s_g = sm + 3072 + c * 1024;            // and its gradient
  float2 *spec = (float2 *)(sm + 6144);         // [3][288] spectra of the couples
  float2 *mine = spec + c * (QP_BUF / 2);
  float *gcmb = sm + 6144 + 3 * QP_BUF + c * 64, *gG = gcmb + 32;
  float *win = sm + 6144 + 3 * QP_BUF + AQ_NW * 64 + c * 4 * Stage<U16>::WIN;
  const short *strip_code = &sc.corr_cfg->strip_code[0][0][0];
  const float inv_n = 1.0f / cfg.num_combo;
  const float l0 = cfg.lpf[lane], l1 = cfg.lpf[lane + 32];
  const int rr = sc.bayer_red_row, rc = sc.bayer_red_col, j = lane & 15;
  const int pair = 2 * c + (lane >> 4);         // this half-warp's pair
  const int kind = c < 2 ? c : 2 + (lane >> 4);

  for (int task = blockIdx.x; task < sc.num_tasks; task += gridDim.x) {
    const int txy = sc.task_txy[task];
    const size_t tile = (size_t)(txy >> 16) * sc.tilesX + (txy & 0xffff);
    const SubtilePlan p = sc.plan[((size_t)task * 4 + q) * 3 + c];
    stage_window<U16>(sc, sc.images[q], p.tlx, p.tly, win + q * Stage<U16>::WIN, r);
    {
      const float *src = sc.clt + tile * 12 * TP_CLT + c * TP_CLT;
#pragma unroll
      for (int i = 0; i < 8; i++) {  // 4 sensors x 64 chunks of 16 bytes
        const int k = lane + 32 * i;
        cp_async16(s_clt + k * 4, src + (k >> 6) * 3 * TP_CLT + (k & 63) * 4);
      }
      cp_async_commit();
    }
    gG[lane] = lane < RE ? sc.combo[tile * RE + lane] : 0.f;
    gcmb[lane] = 0.f;
    // this half-warp's strip samples: entries j of the two strip rows
    const float n0 = (j < 15 && j < RE) ? sc.strips[(tile * 6 + pair) * RE + j] : 0.f;
    const float n1 = (j < 15 && 15 + j < RE) ? sc.strips[(tile * 6 + pair) * RE + 15 + j] : 0.f;
    __syncwarp();
    const float dres = strip_centroid(cfg, gG, gcmb, lane);  // the same in every warp
    if (isnan(dres)) {
      if (threadIdx.x == 0) dval[tile] = CUDART_NAN_F;
      if (threadIdx.x < 8) sens[tile * 8 + threadIdx.x] = 0.f;
      cp_async_wait_all();
      __syncwarp();
      continue;
    }
    // ---------------- the warp's couple: strip to filtered spectra ----------------
    {
      // dd/d(strip entry) of a pair: d combo / d v_p = G / (n v_p), G = combo + offset
      auto grad = [&](int e, float n) {
        if (j >= 15 || e >= RE || gcmb[e] == 0.f || !cfg.pairs[pair].in_combo) return 0.f;
        const float v = n + cfg.corr_offset;
        return v > 0.0f ? __fdividef(gcmb[e] * (gG[e] + cfg.corr_offset) * inv_n, v) : 0.f;
      };
      const float f0 = grad(j, n0), f1 = grad(15 + j, n1);
      const unsigned any = __ballot_sync(0xffffffffu, f0 != 0.f || f1 != 0.f);
      if (lane == 0) s_any[c] = any;
      if (any) {
        for (int i = lane; i < AM_SURF / 2; i += 32) ((float4 *)mine)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        scatter_quad((float *)mine, f0, f1, strip_code, kind, lane);
        couple_unsurface((const float *)mine, mine, lane);
      }
    }
    cp_async_wait_all();  // this colour's CLT and windows
    __syncthreads();
    // ---------------- the warp's colour: gradients of its CLT through the six pairs ----------------
    float g[4][4][2];
#pragma unroll
    for (int s = 0; s < 4; s++)
#pragma unroll
      for (int m = 0; m < 4; m++) g[s][m][0] = g[s][m][1] = 0.f;
    const float wgt = cfg.col_weights[c];
    // couples of the standard quad: 0-1 and 2-3, 0-2 and 1-3, 0-3 and 2-1
    auto couple = [&](int k, auto a1, auto a2, auto b1, auto b2) {
      constexpr int A1 = decltype(a1)::value, A2 = decltype(a2)::value, B1 = decltype(b1)::value, B2 = decltype(b2)::value;
      const unsigned any = s_any[k];
      if (!any) return;
      const bool one = any & 0xffffu, two = any >> 16;
      const float *d = s_clt + lane;
      couple_products_grad(cfg, wgt, d + A1 * TP_CLT, d + A2 * TP_CLT, d + B1 * TP_CLT, d + B2 * TP_CLT, l0, l1,
                           spec + k * (QP_BUF / 2), lane, [&](int h, int m, float2 x, float2 y) {
                             if (one) {
                               g[A1][m][h] += x.x;
                               g[A2][m][h] += y.x;
                             }
                             if (two) {
                               g[B1][m][h] += x.y;
                               g[B2][m][h] += y.y;
                             }
                           });
    };
    couple(0, Int<0>(), Int<1>(), Int<2>(), Int<3>());
    couple(1, Int<0>(), Int<2>(), Int<1>(), Int<3>());
    couple(2, Int<0>(), Int<3>(), Int<2>(), Int<1>());
#pragma unroll
    for (int s = 0; s < 4; s++)
#pragma unroll
      for (int m = 0; m < 4; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) s_g[s * TP_CLT + m * 64 + 32 * h + lane] = g[s][m][h];
    __syncwarp();
    // ---------------- dd/drx, dd/dry of the colour's four sub-tiles ----------------
    {
      float gdir[2], gf[4][8];
      const float *kp = (p.kidx >= 0) ? sc.kernels[q] + (size_t)p.kidx * TP_CLT : nullptr;
      // the transposes go through the sub-tile's CLT once it is read
      shift_grad(p, kp, s_clt + q * TP_CLT, s_g + q * TP_CLT, s_clt + q * TP_CLT, r, gdir, gf);
      SWin<U16> w;
      w.base = (const typename Stage<U16>::T *)(win + q * Stage<U16>::WIN);
      w.sx = p.tlx & (Stage<U16>::CH - 1);
      w.scale = sc.color_scale[c];
      if (c < 2) fold_deriv_bayer<false>(w, p, ((c == 0 ? rc : 1 - rc) - p.tlx) & 1, ((c == 0 ? rr : 1 - rr) - p.tly) & 1, gf, r, gdir);
      else fold_deriv_bayer<true>(w, p, (p.tlx + p.tly + rc + rr + 1) & 1, 0, gf, r, gdir);
      float out[2];
      shift_out(sc, p, q, gdir, out);
      if (r == 0) {
        s_sens[(q * 3 + c) * 2] = out[0];
        s_sens[(q * 3 + c) * 2 + 1] = out[1];
      }
    }
    __syncthreads();
    // a sensor's colours share its port: their sensitivities add, in colour order
    if (threadIdx.x < 8) {
      const int s = threadIdx.x >> 1, k = threadIdx.x & 1;
      float v = 0.f;
      for (int i = 0; i < 3; i++) v += s_sens[(s * 3 + i) * 2 + k];
      sens[tile * 8 + threadIdx.x] = v;
    }
    if (threadIdx.x == 0) dval[tile] = dres;
  }
}

cudaError_t upload_adjoint_quad_constants() { return upload_dtt_constants(); }

// a Bayer standard quad, images of one type, a strip of at most 32 entries, the stored CLT
bool adjoint_quad_ok(const SceneDev &sc, int recompute) {
  const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  return !recompute && sc.num_colors == 3 && quad_forward_ok(sc) && RE <= 32;
}

cudaError_t launch_adjoint_quad(const SceneDev &sc, const CorrConst &cc, float *sens, float *dval, cudaStream_t st) {
  const int RE = (sc.strip_rows < sc.wndy_size ? sc.strip_rows : sc.wndy_size) * 15;
  auto go = [&](auto kernel, int bytes) -> cudaError_t {
    int res = 0;
    const cudaError_t e = kernel_residency((const void *)kernel, 32 * AQ_NW, bytes, &res);
    if (e != cudaSuccess) return e;
    if (res < 1) return cudaErrorInvalidConfiguration;
    kernel<<<sc.num_tasks < res ? sc.num_tasks : res, 32 * AQ_NW, bytes, st>>>(sc, cc, RE, sens, dval);
    return cudaGetLastError();
  };
  return sc.img_dtype[0] == 1 ? go(adjoint_quad_kernel<true>, aq_floats<true>() * 4) : go(adjoint_quad_kernel<false>, aq_floats<false>() * 4);
}
