// tp_adjoint_pairs.cuh -- the adjoint's pair chain with two pairs per instruction (tp_pairs.cuh): strip taps,
// unfold and transforms transposed, the gradients of the normalised products.
#pragma once
#include "tp_adjoint.cuh"
#include "tp_pairs.cuh"

namespace {

constexpr int AM_SURF = 228;  // a pair's surface gradient (rounded to 16 bytes)

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
      if (now && v[k] != 0.f) g[o[k]] = g[o[k]] + v[k];
      __syncwarp();
    }
  }
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

// The gradients of two pairs' normalised products of one colour (weight wgt), from the gradients b of their
// filtered spectra; a1, a2, b1, b2: the first and second pair's two sensors' coefficients (at the lane's
// index).  add(h, m, x, y) gets the gradients of the first (x) and second (y) sensors' coefficient
// m * 64 + 32 * h + lane of the two pairs.
template <typename ADD>
__device__ __forceinline__ void couple_products_grad(const CorrConst &cfg, float wgt, const float *a1, const float *a2c,
                                                     const float *b1, const float *b2, float l0, float l1,
                                                     const float2 *b, int lane, ADD add) {
  const int off = (lane >> 3) * 9 + (lane & 7);
  const float fzz = cfg.fat_zero * cfg.fat_zero;
  float2 d1[2][4], d2[2][4], a2[2], ia2[2], s1v[2], s2v[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int o = m * 64 + 32 * h;
      d1[h][m] = make_float2(a1[o], b1[o]);
      d2[h][m] = make_float2(a2c[o], b2[o]);
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
    dbar[h] = mul2(mul2(mul2(dup2(-wgt), sw), u), u);
    const float2 wu = mul2(dup2(wgt), u);
#pragma unroll
    for (int m = 0; m < 4; m++) tg[h][m] = mul2(gq[m], wu);
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
    for (int m = 0; m < 4; m++) add(h, m, fma2(k1, d[m], g1[m]), fma2(k2, e[m], g2[m]));
  }
}

}  // namespace
