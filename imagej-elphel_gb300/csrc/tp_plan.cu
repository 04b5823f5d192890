// tp_plan.cu -- stage 1 (port coordinates) and per-sub-tile window planning, FP64.
//
// Tile selection (integer window corner, kernel tile) must match the FP64
// reference bit for bit, so this translation unit evaluates the geometry in
// double precision with explicitly rounded operations (__dadd_rn etc. are never
// contracted into FMAs) in the operation order of
// GeometryCorrection.getPortsCoordinatesAndDerivatives and
// ImageDtt.extract_correct_tile.  Two FP64 lanes per SM bound it at full size (an FP64 instruction
// takes 64 issue slots), the chain of dependent FP64 instructions at small ones.  So what is exact in
// integers (conversions, rounding to a corner, kernel centres) is done there, products that are the
// same for every tile come with the geometry, zero radial coefficients are not evaluated, and small
// task lists take a thread per (task, sensor).  Measured, before -> now: 4x2592x1936 Bayer with kernel
// tables (78,408 tasks) 155 -> 65 us, 4x640x480 (4,800) 39 -> 11 us, 16x640x512 with derivatives 71 -> 43 us,
// 16 batched 4x512x384 mono scenes 51 -> 23 us.
#include "tp.h"
#include "tp_internal.h"
#include <math_constants.h>

#define DADD(a, b) __dadd_rn((a), (b))
#define DSUB(a, b) __dsub_rn((a), (b))
#define DMUL(a, b) __dmul_rn((a), (b))
#define DDIV(a, b) __ddiv_rn((a), (b))
#define DSQRT(a) __dsqrt_rn(a)

// java.lang.Math.round(double), exact round-half-up
__device__ __forceinline__ double java_round(double x) {
  double f = floor(x);
  return (DSUB(x, f) >= 0.5) ? DADD(f, 1.0) : f;
}

// Window corner (an integral double) -> int.  A corner further than TP_PORT_MARGIN outside the
// image is moved to the margin keeping its parity: every pixel of such a window is outside the
// image, and the mirrored edge pixels it reads (Win::at, mirror) depend only on the corner's
// parity, so the window content is unchanged and the int arithmetic of the kernels that read it
// cannot overflow.  NaN (a port beyond the reverse distortion table) goes to the lower bound.
__device__ __forceinline__ int clamp_corner(double t, int n) {
  const double lo = -(double)(TP_PORT_MARGIN + 16), hi = (double)(n + TP_PORT_MARGIN);
  if (t >= lo && t <= hi) return (int)t;
  const int par = (t == t) ? (int)fabs(fmod(t, 2.0)) : 0;
  return (t > hi) ? (int)hi - (((int)hi & 1) ^ par) : (int)lo + (((int)lo & 1) ^ par);
}

// GeometryCorrection.getRByRDist (GeometryCorrection.java:2802-2827)
__device__ double r_by_rdist(const double *tbl, int len, double rDist) {
  if (rDist < 0) return CUDART_NAN;
  double q = DDIV(rDist, 0.001);
  int index = (int)floor(q);
  if (index >= len - 1) return CUDART_NAN;
  return DADD(tbl[index], DMUL(DSUB(tbl[index + 1], tbl[index]), DSUB(q, (double)index)));
}

// Exact conversions by bit assembly.  FP64 instructions (conversions among them) issue at 1/64 of
// the integer rate here and bound this file's kernels, so everything that is exact in integers stays
// there.
__device__ __forceinline__ double f2d(float f) {
  const unsigned u = __float_as_uint(f), e = (u >> 23) & 255u;
  if (e - 1u < 254u)  // normal
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))), (int)(u << 29));
  if ((u << 1) == 0u) return __hiloint2double((int)u, 0);
  return (double)f;
}
__device__ __forceinline__ double i2d(int n) { return (n < (1 << 24) && n > -(1 << 24)) ? f2d((float)n) : (double)n; }
// n / 2 (n = 0: 0)
__device__ __forceinline__ double half_i2d(int n) {
  const double d = i2d(n);
  return n ? __hiloint2double(__double2hiint(d) - (1 << 20), __double2loint(d)) : 0.0;
}
// java_round(x / 2^k) as an integer for |x| < 2^30: floor(2 x / 2^k) is an arithmetic shift of the
// signed mantissa, and java_round(y) = (floor(2 y) + 1) >> 1.  Returns false (n unset) beyond, and for NaN.
__device__ __forceinline__ bool jround(double x, int k, int &n) {
  const int hi = __double2hiint(x), e = ((hi >> 20) & 0x7ff) - 1023;
  if (e >= 30) return false;
  const long long m = ((long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(x);
  const int sh = min(51 - e + k, 63);
  n = (int)((((hi < 0 ? -m : m) >> sh) + 1) >> 1);
  return true;
}

// undistorted tile centre, the sensor-independent head of getPortsCoordinatesAndDerivatives, with
// the centre model (gc_main, 2179-2185); px, py: the centre (2 px - width is exact in integers)
__device__ __forceinline__ void center_undistort(const GeomDev &g, const double *tbl, int px, int py, double &pXc,
                                                 double &pYc) {
  const double pXcd = half_i2d(2 * px - g.c_pixel_width);
  const double pYcd = half_i2d(2 * py - g.c_pixel_height);
  const double rD = DMUL(DMUL(DSQRT(DADD(DMUL(pXcd, pXcd), DMUL(pYcd, pYcd))), 0.001), g.c_pixel_size);
  const double rND2R = r_by_rdist(tbl, g.tbl_len, DDIV(rD, g.c_distortion_radius));
  pXc = DMUL(pXcd, rND2R);
  pYc = DMUL(pYcd, rND2R);
}

// A rotation times (v0, v1, fl_pix): the third product is the same for every tile and comes with the
// geometry (m2f[i] = m[i][2] * fl_pix), summed last as in the reference's matrix product.
__device__ __forceinline__ double row_vec(const double m[3], double m2f, double v0, double v1) {
  return DADD(DADD(DMUL(m[0], v0), DMUL(m[1], v1)), m2f);
}

// sensor part of getPortsCoordinatesAndDerivatives (GeometryCorrection.java:2159-2314) for one sensor;
// (pXc, pYc): the task's undistorted centre, the same for every sensor.  The radial polynomial runs to
// the last nonzero coefficient only (g.n_rad): a zero one adds 0 x (a finite number).  Where that
// number would not be finite (pXci or pYci out of range or NaN), or the radius is 0 (its derivatives are
// then NaN), all seven are taken.
template <bool DERIV>
__device__ __forceinline__ void sensor_port(const GeomDev &g, double pXc, double pYc, double disparity, int i,
                                            double &ox, double &oy, double *deriv /* [2][5] */) {
  const double fl_pix = g.fl_pix;
  const double v0 = DSUB(pXc, DMUL(disparity, g.rXY[i][0])), v1 = DSUB(pYc, DMUL(disparity, g.rXY[i][1]));
  const double r0 = row_vec(g.rots[i][0], g.rots_f[i][0], v0, v1);
  const double r1 = row_vec(g.rots[i][1], g.rots_f[i][1], v0, v1);
  const double r2 = row_vec(g.rots[i][2], g.rots_f[i][2], v0, v1);
  const double norm_z = DDIV(fl_pix, r2);
  const double pXci = DMUL(r0, norm_z), pYci = DMUL(r1, norm_z);
  const int lim = (1023 + 100) << 20;  // 2^100
  const int hx = __double2hiint(pXci) & 0x7fffffff, hy = __double2hiint(pYci) & 0x7fffffff;
  const int n_rad = (hx < lim && hy < lim && (hx | hy)) ? g.n_rad : 7;
  double rD2rND = 1.0, ri = 0.0, rNDi = 0.0;
  if (n_rad) {
    rNDi = DSQRT(DADD(DMUL(pXci, pXci), DMUL(pYci, pYci)));
    ri = DMUL(rNDi, g.ri_scale);
    double rri = 1.0;
    for (int j = 0; j < n_rad; j++) {
      rri = DMUL(rri, ri);
      rD2rND = DADD(rD2rND, DMUL(g.rad_coeff[j], DSUB(rri, 1.0)));
    }
    ox = DADD(DMUL(pXci, rD2rND), g.pXY0[i][0]);
    oy = DADD(DMUL(pYci, rD2rND), g.pXY0[i][1]);
  } else {
    ox = DADD(pXci, g.pXY0[i][0]);
    oy = DADD(pYci, g.pXY0[i][1]);
  }
  if constexpr (DERIV) {
    // quotients shared by the five parameters (a product with a reciprocal where the reference
    // divides: the derivatives differ from its by an ulp, the ports are not touched)
    const double inv_rz = DDIV(1.0, r2);
    const double pXr = DMUL(pXci, inv_rz), pYr = DMUL(pYci, inv_rz);
    double ri_rnd = 0.0, drD2rND_dri = 0.0;
    if (n_rad) {
      ri_rnd = DDIV(g.ri_scale, rNDi);
      double rri = 1.0;
      for (int j = 0; j < n_rad; j++) {
        drD2rND_dri = DADD(drD2rND_dri, DMUL(g.rad_dcoeff[j], rri));
        rri = DMUL(rri, ri);
      }
    }
#pragma unroll
    for (int k = 0; k < 5; k++) {  // azimuth, tilt, roll, zoom; then the tile disparity
      double d0, d1, d2;
      if (k < 4) {
        d0 = row_vec(g.drots[i][k][0], g.drots_f[i][k][0], v0, v1);
        d1 = row_vec(g.drots[i][k][1], g.drots_f[i][k][1], v0, v1);
        d2 = row_vec(g.drots[i][k][2], g.drots_f[i][k][2], v0, v1);
      } else {  // d (v0, v1, fl_pix) / d disparity = (-rX, -rY, 0), rotated
        d0 = g.drot_disp[i][0];
        d1 = g.drot_disp[i][1];
        d2 = g.drot_disp[i][2];
      }
      const double dpX = DSUB(DMUL(d0, norm_z), DMUL(pXr, d2));
      const double dpY = DSUB(DMUL(d1, norm_z), DMUL(pYr, d2));
      if (!n_rad) {
        deriv[k] = dpX;
        deriv[5 + k] = dpY;
      } else if (k == 2) {  // roll: the reference keeps only the rotation term
        deriv[k] = DMUL(dpX, rD2rND);
        deriv[5 + k] = DMUL(dpY, rD2rND);
      } else {
        const double dri = DMUL(ri_rnd, DADD(DMUL(pXci, dpX), DMUL(pYci, dpY)));
        const double drD = DMUL(drD2rND_dri, dri);
        deriv[k] = DADD(DMUL(dpX, rD2rND), DMUL(pXci, drD));
        deriv[5 + k] = DADD(DMUL(dpY, rD2rND), DMUL(pYci, drD));
      }
    }
  }
}

// window corner and residual shift along one axis (ImageDtt.java:4940-4943) from px = the window's
// exact corner: TL = -java_round(-px), residual = -(px - TL)
__device__ __forceinline__ void corner(double px, int n, int &tl, float &res) {
  int m;
  if (jround(-px, 0, m)) {
    const int lo = -(TP_PORT_MARGIN + 16), hi = n + TP_PORT_MARGIN;
    tl = -m;
    res = (float)(-DSUB(px, i2d(tl)));
    if (tl < lo || tl > hi) {  // clamp_corner
      const int par = tl & 1;
      tl = (tl > hi) ? hi - ((hi & 1) ^ par) : lo + ((lo & 1) ^ par);
    }
  } else {  // beyond +-2^30 pixels, or NaN
    const double t = -java_round(-px);
    tl = clamp_corner(t, n);
    res = (float)(-DSUB(px, t));
  }
}

// kernel tile along one axis: round(c / ks) + 1 within the table, and the distance from its centre
__device__ __forceinline__ int kernel_tile(double c, int ks, int ks_log2, int nk, double &d) {
  int m;
  if (ks_log2 < 0 || !jround(c, ks_log2, m)) m = (int)java_round(DDIV(c, (double)ks));
  int kt = m + 1;
  kt = kt < 0 ? 0 : (kt >= nk ? nk - 1 : kt);
  // ((kt - 1) + 0.5) * ks
  const long long c2 = (2ll * kt - 1) * ks;
  d = DSUB(c, (c2 < (1 << 30) && c2 > -(1 << 30)) ? half_i2d((int)c2) : DMUL(DADD((double)(kt - 1), 0.5), (double)ks));
  return kt;
}

// Thread per (task, run of sensors): the centre is undistorted once per thread, the kernel tile
// found once per sensor (it depends on the port only), then each colour's window corner and residual
// shift (ImageDtt.java:4904-4943).
// sensors [s0, s1) of one task
template <bool DERIV>
__device__ __forceinline__ void plan_task(const SceneDev &sc, int task, int s0, int s1) {
  const int S = sc.num_sensors, C = sc.num_colors;
  const int txy = sc.task_txy[task];
  const int tx = txy & 0xffff, ty = txy >> 16;
  double pXc = 0.0, pYc = 0.0, disparity = 0.0;
  if (sc.ports_from_geometry) {
    center_undistort(*sc.geom, sc.rdist_tbl, tx * TP_DTT + TP_DTT / 2, ty * TP_DTT + TP_DTT / 2, pXc, pYc);
    disparity = f2d(sc.task_disp[task]);
    // a rig's auxiliary camera: disparity_main * aux radius / main radius (ImageDtt.java:8973)
    if (sc.geom->rig) disparity = DDIV(DMUL(disparity, sc.geom->disp_num), sc.geom->disp_den);
  }
  const int ks = sc.kernel_step;
  const int ks_log2 = (ks > 0 && (ks & (ks - 1)) == 0) ? 31 - __clz(ks) : -1;
  for (int s = s0; s < s1; s++) {
    double cx, cy;
    if (sc.ports_from_geometry) {
      double dv[10];
      sensor_port<DERIV>(*sc.geom, pXc, pYc, disparity, s, cx, cy, dv);
      if constexpr (DERIV) {
        double *o = sc.port_deriv + ((size_t)task * S + s) * 10;
#pragma unroll
        for (int k = 0; k < 10; k++) o[k] = dv[k];
      }
    } else {
      cx = f2d(sc.task_xy[((size_t)task * S + s) * 2]);
      cy = f2d(sc.task_xy[((size_t)task * S + s) * 2 + 1]);
    }
    sc.ports[((size_t)task * S + s) * 2] = cx;
    sc.ports[((size_t)task * S + s) * 2 + 1] = cy;
    int ktx = 0, kty = 0;
    double kdx = 0.0, kdy = 0.0;
    if (sc.kh > 0) {
      ktx = kernel_tile(cx, ks, ks_log2, sc.kh, kdx);
      kty = kernel_tile(cy, ks, ks_log2, sc.kv, kdy);
    }
    const double cx8 = DSUB(cx, (double)TP_DTT), cy8 = DSUB(cy, (double)TP_DTT);
    for (int c = 0; c < C; c++) {
      double px = cx8, py = cy8;
      SubtilePlan p;
      p.kidx = -1;
      if (sc.kh > 0) {
        p.kidx = (kty * sc.kh + ktx) * C + c;
        const float4 *ce4 = (const float4 *)(sc.kext[s] + (size_t)p.kidx * 8);
        const float4 e0 = __ldg(ce4), e1 = __ldg(ce4 + 1);  // data_x, data_y, -, -, dxc_dx, dxc_dy, dyc_dx, dyc_dy
        px = DSUB(px, DADD(DADD(f2d(e0.x), DMUL(f2d(e1.x), kdx)), DMUL(f2d(e1.y), kdy)));
        py = DSUB(py, DADD(DADD(f2d(e0.y), DMUL(f2d(e1.z), kdx)), DMUL(f2d(e1.w), kdy)));
      }
      corner(px, sc.width, p.tlx, p.rx);
      corner(py, sc.height, p.tly, p.ry);
      sc.plan[((size_t)task * S + s) * C + c] = p;
    }
  }
}

// gs sensors per thread
template <bool DERIV>
__global__ void plan_kernel(SceneDev sc, int gs) {
  const int groups = (sc.num_sensors + gs - 1) / gs;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= sc.num_tasks * groups) return;
  const int task = i / groups, s0 = (i - task * groups) * gs;
  plan_task<DERIV>(sc, task, s0, min(s0 + gs, sc.num_sensors));
}

// the plans of a batch of scenes in one launch: thread per task of the
// concatenated task lists, scene found by binary search over the task offsets
__global__ void plan_batch_kernel(const SceneDev *__restrict__ scenes, const int *__restrict__ task_off, int n) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= task_off[n]) return;
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (task_off[mid] <= g) lo = mid;
    else hi = mid - 1;
  }
  const SceneDev &sc = scenes[lo];
  const int task = g - task_off[lo];
  plan_task<false>(sc, task, 0, sc.num_sensors);
  const int txy = sc.task_txy[task];
  sc.tile_task[(txy >> 16) * sc.tilesX + (txy & 0xffff)] = task;
}

__global__ void tile_task_map_kernel(SceneDev sc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < sc.num_tasks) {
    int txy = sc.task_txy[i];
    int tile = (txy >> 16) * sc.tilesX + (txy & 0xffff);
    if (tile >= 0 && tile < sc.tilesX * sc.tilesY) sc.tile_task[tile] = i;
  }
}

// Sensors per thread: with few threads the kernel is a chain of dependent FP64 instructions, so each
// takes one sensor; with many the FP64 pipes are full, and four sensors share the centre's part.
// The line: about one warp per scheduler of the chip's 152 SMs (32 x 4 x 152 threads).  One and four sensors a thread:
// 4 sensors, 4,800 tasks 8.2 and 12.4 us, 9,882 11.0 and 14.4, 19,602 16.5 and 14.8, 78,408 52.3 and 34.9;
// 16 sensors, 1,280 8.3 and 12.4, 5,120 16.5 and 15.4.
cudaError_t launch_plan(const SceneDev &sc, cudaStream_t st) {
  if (sc.num_tasks <= 0) return cudaSuccess;
  int gs = 1;
  while (gs < 4 && sc.num_tasks * ((sc.num_sensors + gs - 1) / gs) > 32 * 4 * 152) gs *= 2;
  const int n = sc.num_tasks * ((sc.num_sensors + gs - 1) / gs);
  if (sc.port_deriv && sc.ports_from_geometry) plan_kernel<true><<<(n + 63) / 64, 64, 0, st>>>(sc, gs);
  else plan_kernel<false><<<(n + 63) / 64, 64, 0, st>>>(sc, gs);
  return cudaGetLastError();
}

// tile maps are cleared by the caller (cudaMemsetAsync per scene) before this launch
cudaError_t launch_plan_batch(const SceneDev *scenes_dev, const int *task_off_dev, int n, int total_tasks,
                              cudaStream_t st) {
  if (total_tasks <= 0) return cudaSuccess;
  plan_batch_kernel<<<(total_tasks + 63) / 64, 64, 0, st>>>(scenes_dev, task_off_dev, n);
  return cudaGetLastError();
}

cudaError_t launch_tile_task_map(const SceneDev &sc, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(sc.tile_task, 0xff, sizeof(int) * sc.tilesX * sc.tilesY, st);
  if (e != cudaSuccess) return e;
  if (sc.num_tasks <= 0) return cudaSuccess;
  tile_task_map_kernel<<<(sc.num_tasks + 255) / 256, 256, 0, st>>>(sc);
  return cudaGetLastError();
}

// Row-major compaction of tiles with tile_op != 0 into the task list
// (GPUTileProcessor.setFullFrameImages order), a block per 1024 tiles, deterministic: each block needs
// the count of the tiles before its own.  Up to CB_SELF blocks it counts them itself (they are in L2, a
// load per thread and block before it), so one launch does; beyond, a first launch counts per block.  One and two
// launches: 4,800 tiles 4.2 and 7.2 us, 40,000 6.2 and 8.2, 78,408 7.9 and 8.2, 131,072 (128 blocks) 8.3 and 8.2.
// tile_task (or null): the tile's task or -1.
constexpr int CB = 1024, CB_SELF = 128;

__global__ void compact_count_kernel(const int *tile_op, int num_tiles, int *block_counts) {
  const int i = blockIdx.x * CB + threadIdx.x;
  const int n = __syncthreads_count(i < num_tiles && tile_op[i] != 0);
  if (threadIdx.x == 0) block_counts[blockIdx.x] = n;
}

__global__ void __launch_bounds__(CB) compact_scatter_kernel(const int *tile_op, const float *disparity, int tilesX,
                                                             int num_tiles, const int *block_counts, int *task_txy,
                                                             int *task_op, float *task_disp, int *num_tasks,
                                                             int *tile_task) {
  __shared__ int warp_sums[32], before_sums[32];
  __shared__ int base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int b = 0;  // tiles before this block's (this thread's share)
  if (block_counts) {
    for (int k = threadIdx.x; k < blockIdx.x; k += CB) b += block_counts[k];
  } else {
    for (int k = 0; k < blockIdx.x; k++) b += tile_op[k * CB + threadIdx.x] != 0;
  }
  const int i = blockIdx.x * CB + threadIdx.x;
  const int op = (i < num_tiles) ? tile_op[i] : 0;
  const int flag = op != 0;
  const unsigned m = __ballot_sync(0xffffffffu, flag);
  const int pre = __popc(m & ((1u << lane) - 1u));
  b = __reduce_add_sync(0xffffffffu, b);
  if (lane == 31) warp_sums[warp] = pre + flag;
  if (lane == 0) before_sums[warp] = b;
  __syncthreads();
  if (warp == 0) {
    const int v = warp_sums[lane];
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const int before = __reduce_add_sync(0xffffffffu, before_sums[lane]);
    if (lane == 31) {
      base = before;
      if (blockIdx.x == gridDim.x - 1) *num_tasks = before + incl;
    }
    warp_sums[lane] = incl - v;
  }
  __syncthreads();
  const int pos = base + warp_sums[warp] + pre;
  if (flag) {
    const int ty = i / tilesX, tx = i - ty * tilesX;
    task_txy[pos] = tx | (ty << 16);
    task_op[pos] = op;
    task_disp[pos] = disparity ? disparity[i] : 0.0f;
  }
  if (tile_task && i < num_tiles) tile_task[i] = flag ? pos : -1;
}

static cudaError_t compact(const int *tile_op, const float *disparity, int tilesX, int num_tiles, int *task_txy,
                           int *task_op, float *task_disp, int *num_tasks_dev, int *tile_task, int *counts,
                           cudaStream_t st) {
  const int nb = num_tiles > 0 ? (num_tiles + CB - 1) / CB : 1;
  if (nb <= CB_SELF) counts = nullptr;
  else compact_count_kernel<<<nb, CB, 0, st>>>(tile_op, num_tiles, counts);
  compact_scatter_kernel<<<nb, CB, 0, st>>>(tile_op, disparity, tilesX, num_tiles, counts, task_txy, task_op,
                                            task_disp, num_tasks_dev, tile_task);
  return cudaGetLastError();
}

// the caller sizes num_tasks_dev for 1 + number of 1024-tile blocks
cudaError_t launch_compact_tasks(const int *tile_op, const float *disparity, int tilesX, int num_tiles,
                                 int *task_txy, int *task_op, float *task_disp, int *num_tasks_dev, int *tile_task,
                                 cudaStream_t st) {
  return compact(tile_op, disparity, tilesX, num_tiles, task_txy, task_op, task_disp, num_tasks_dev, tile_task,
                 num_tasks_dev + 1, st);
}

// ---------------------------------------------------------------------------
// Task compaction that allocates nothing: the per-block counts go to a fixed
// file-scope device array instead of a handle's buffer.  Every count slot the
// scatter reads is written earlier in the same call by compact_count_kernel,
// so nothing has to start at zero; concurrent calls on one device share the
// array and race.
// ---------------------------------------------------------------------------
constexpr int COMPACT_SCRATCH_BLOCKS = 1024;  // x CB tiles per block = 1,048,576 tiles
static __device__ __align__(256) int g_compact_scratch[COMPACT_SCRATCH_BLOCKS];

int compact_scratch_max_tiles() { return COMPACT_SCRATCH_BLOCKS * CB; }

cudaError_t compact_scratch_address(int **ptr) {
  return cudaGetSymbolAddress((void **)ptr, g_compact_scratch);
}

cudaError_t launch_compact_tasks_scratch(const int *tile_op, const float *disparity, int tilesX, int num_tiles,
                                         int *task_txy, int *task_op, float *task_disp, int *num_tasks_dev,
                                         int *scratch, cudaStream_t st) {
  if ((num_tiles + CB - 1) / CB > COMPACT_SCRATCH_BLOCKS) return cudaErrorInvalidValue;
  return compact(tile_op, disparity, tilesX, num_tiles, task_txy, task_op, task_disp, num_tasks_dev, nullptr, scratch,
                 st);
}
