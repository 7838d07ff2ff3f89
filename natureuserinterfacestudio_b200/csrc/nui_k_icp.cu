// Point-to-plane ICP: every iteration of every level in one launch, no host round trip; up to four
// sessions over the whole device (k_icp_wide), more by a thread-block cluster each (k_icp_cluster).
//
// Per pixel (icp_block_kernel, icp.cl:222-292): rebuild the level's vertex from its depth,
// transform it by the running estimate, project into the previous camera with
// full-resolution intrinsics, bilinearly sample the world reference normal and vertex
// (icp.cl:192-220; a tap NaN -> no match), and if |q - p| < distThres form the row
// [n x p, n | n.(q - p)].  A warp adds the outer products of its pixels' rows in FP64 on the
// tensor path (exact products of the FP32 row values), and the warps' sums are joined in an
// order that the image size fixes, by every block of k_icp_wide or the first of a cluster, which
// run the host step of
// NuiKinfuOpenCLDepthTracker::IterativeClosestPoint (NuiKinfuOpenCLDepthTracker.cpp:324-496):
// Levenberg-Marquardt accept/reject, FP64 determinant check and Cholesky solve, ZYX Euler
// increment composed in FP64.  The next iteration reads the updated estimate.
#include <cooperative_groups.h>

#include "nui_device.cuh"

namespace nui {

// Bilinear sample with holes; taps whose linear index falls past the map read as holes (the
// last tap has the largest index).  A hole is NaN in a component and makes that component of
// the sample NaN whatever its weight, so the caller tests the sample instead of the taps.
__device__ __forceinline__ float3 bilinear_holes(const float4* __restrict__ src, float px, float py, int W,
                                                 int N) {
  const int ix = (int)floorf(px), iy = (int)floorf(py);
  const float dx = px - (float)ix, dy = py - (float)iy;
  const int ia = ix + iy * W;
  if (ia + W + 1 >= N) return f3(qnan(), qnan(), qnan());
  const float3 a = xyz(__ldg(src + ia)), b = xyz(__ldg(src + ia + 1)), c = xyz(__ldg(src + ia + W)),
               d = xyz(__ldg(src + ia + W + 1));
  const float ex = 1.0f - dx, ey = 1.0f - dy;
  float3 r;
  r.x = a.x * ex * ey + b.x * dx * ey + c.x * ex * dy + d.x * dx * dy;
  r.y = a.y * ex * ey + b.y * dx * ey + c.y * ex * dy + d.y * dx * dy;
  r.z = a.z * ex * ey + b.z * dx * ey + c.z * ex * dy + d.z * dx * dy;
  return r;
}

// a / b rounded to nearest, given r = 1 / b rounded to nearest (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): a
// quotient within one ulp plus its exactly computed remainder times r rounds correctly.  The
// first remainder step brings a r within one ulp, the second rounds.  Exact while nothing
// under- or overflows: b in 2^-40 .. 2^40, a zero or in 2^-80 .. 2^80 in magnitude; a smaller a
// gives a quotient within two ulps.
__device__ __forceinline__ float div_shared(float a, float b, float r) {
  float q = a * r;
  q = __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
  return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}
// The quotients of a test.
__global__ void k_div_shared(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ q, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) q[i] = div_shared(a[i], b[i], 1.0f / b[i]);
}

// ---------------------------------------------------------------- photometric rows
// One model point of the colour tracker's term (color_icp_block_kernel, colorIcp.cl:
// 119-178, in the tracker's convention), at the finest level: the world point m of the
// previous raycast, whose colour is the previous frame's at the same pixel (the raycast
// is rendered from the previous pose), is taken to the current camera by the running
// estimate, p = R^T (m - t), projected and rounded to a pixel of the current colour
// image; the residual is the colour difference (units of 1/255) and its derivative in
// each ICP parameter x_k is  grad(I) . d(proj)/dp . dp/dx_k  with dp/dx_k = R^T (e_k x m)
// for the rotations and -R^T e_k for the translations (the depth ICP's update
// R <- Rinc^-1 R, t <- Rinc^-1 t + tinc).  Colours count with alpha 255.  The point's terms
// are the upper triangle of [D | -diff]^T [D | -diff] by rows (21 + 6) and |diff|^2.
struct ColorRow {
  float3 D[6], nd;  // derivatives per parameter and -diff, a value per colour channel
  // adds the 28 terms -- the upper triangle of [D | nd] by rows (21 + 6), then |diff|^2 --
  // and a count to the sums
  __device__ __forceinline__ void add_to(double (&acc)[29]) const {
    int q = 0;
#pragma unroll
    for (int a = 0; a < 6; ++a) {
#pragma unroll
      for (int b = a; b < 6; ++b) acc[q++] += (double)dot3(D[a], D[b]);
      acc[q++] += (double)dot3(D[a], nd);
    }
    acc[27] += (double)dot3(nd, nd);
    acc[28] += 1.0;
  }
};
__device__ __forceinline__ bool color_row(const SessionDesc& s, int i, const float* R, const float3 t, ColorRow& row) {
  const float3 m = xyz(__ldg(s.vref + i));
  if (isnan3(m)) return false;
  const uchar4 mc = __ldg(s.cprev + i);
  if (mc.w != 255) return false;
  const float3 d = sub3(m, t);
  const float3 c0 = f3(R[0], R[3], R[6]), c1 = f3(R[1], R[4], R[7]), c2 = f3(R[2], R[5], R[8]);
  const float3 p = f3(dot3(c0, d), dot3(c1, d), dot3(c2, d));
  const float fx = s.cam.fx, fy = s.cam.fy, cx = s.cam.cx, cy = s.cam.cy;
  const int lw = s.W, lh = s.H;
  const int u = (int)roundf(p.x * fx / p.z + cx), v = (int)roundf(p.y * fy / p.z + cy);
  if (!(u >= 0 && u < lw && v >= 0 && v < lh)) return false;
  const int li = v * lw + u;
  const uchar4 co = __ldg(reinterpret_cast<const uchar4*>(s.bgra) + li);
  const uchar4 gx = __ldg(s.cgx[0] + li), gy = __ldg(s.cgy[0] + li);
  if (co.w != 255 || gx.w != 255 || gy.w != 255) return false;
  const float k255 = 1.0f / 255.0f;
  const float3 diff = mul3(f3((float)co.x - (float)mc.x, (float)co.y - (float)mc.y, (float)co.z - (float)mc.z), k255);
  const float3 g1 = mul3(f3((float)(signed char)gx.x, (float)(signed char)gx.y, (float)(signed char)gx.z), k255);
  const float3 g2 = mul3(f3((float)(signed char)gy.x, (float)(signed char)gy.y, (float)(signed char)gy.z), k255);
  const float zz = p.z * p.z;
  // D[k] = jx g1 + jy g2 with (jx, jy) = f (p.z dp - dp.z p) / zz for
  // dp = (dot3(c0, w), dot3(c1, w), dot3(c2, w)), w = e_k x m (k < 3) or -e_k, without the
  // terms of w's zeros
  auto derive = [&](auto quotient) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const float3 dp = k == 0 ? f3(c0.y * -m.z + c0.z * m.y, c1.y * -m.z + c1.z * m.y, c2.y * -m.z + c2.z * m.y)
                      : k == 1 ? f3(c0.x * m.z + c0.z * -m.x, c1.x * m.z + c1.z * -m.x, c2.x * m.z + c2.z * -m.x)
                      : k == 2 ? f3(c0.x * -m.y + c0.y * m.x, c1.x * -m.y + c1.y * m.x, c2.x * -m.y + c2.y * m.x)
                      : k == 3 ? f3(-c0.x, -c1.x, -c2.x)
                      : k == 4 ? f3(-c0.y, -c1.y, -c2.y)
                               : f3(-c0.z, -c1.z, -c2.z);
      const float jx = fx * quotient(p.z * dp.x - dp.z * p.x), jy = fy * quotient(p.z * dp.y - dp.z * p.y);
      row.D[k] = f3(jx * g1.x + jy * g2.x, jx * g1.y + jy * g2.y, jx * g1.z + jy * g2.z);
    }
  };
  // the twelve quotients by zz share its reciprocal for points between a micrometre and 10^6 m
  // away along every axis that counts: the numerators are then below the end of div_shared's range.
  // One that cancels to less than 2^-80 may end two ulps off (a derivative below 2^-28).
  const float far = fmaxf(fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fmaxf(fabsf(m.x), fabsf(m.y))), fmaxf(fabsf(m.z), p.z));
  if (zz > 1e-12f && far < 1e6f) {
    const float rzz = 1.0f / zz;
    derive([&](float a) { return div_shared(a, zz, rzz); });
  } else {
    derive([&](float a) { return a / zz; });
  }
  row.nd = f3(-diff.x, -diff.y, -diff.z);
  return true;
}

// ---------------------------------------------------------------- FP64 host step
// The 6x6 algebra of the host step runs at the end of every iteration, while all other blocks
// wait, so its latency counts: the rows are spread over the lanes of a warp, so that the
// quotients of a column form at once, and every value still comes from the same operations in
// the same order as in a serial elimination.

// Determinant by Gaussian elimination with partial pivoting (the first row holding the
// largest |entry| of the column): lane r < 6 holds row r. Called by a whole warp; every lane
// gets the result.
__device__ __forceinline__ double det6(double (&a)[6]) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  double det = 1.0;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    int piv = c;
    double best = fabs(__shfl_sync(full, a[c], c));
#pragma unroll
    for (int r = c + 1; r < 6; ++r) {
      const double v = fabs(__shfl_sync(full, a[c], r));
      if (v > best) {
        best = v;
        piv = r;
      }
    }
    if (best == 0.0) return 0.0;
    if (piv != c) {
      const int src = lane == c ? piv : lane == piv ? c : lane;
#pragma unroll
      for (int k = c; k < 6; ++k) a[k] = __shfl_sync(full, a[k], src);
      det = -det;
    }
    const double p = __shfl_sync(full, a[c], c);
    det *= p;
    const double f = a[c] / p;
#pragma unroll
    for (int k = c + 1; k < 6; ++k) {
      const double q = __shfl_sync(full, a[k], c);
      if (lane > c) a[k] -= f * q;
    }
  }
  return det;
}

// Cholesky factorisation A = L L^T and the two triangular solves; false if a pivot is not
// positive.  Lane i < 6 holds row i of A, lane 6 the right-hand side, which goes through the
// factorisation as a seventh row (the forward substitution). Called by a whole warp; every lane
// gets x.
__device__ __forceinline__ bool llt_solve6(double (&a)[6], double (&x)[6]) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  double diag[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const double d = __shfl_sync(full, a[j], j);
    if (!(d > 0.0)) return false;
    diag[j] = sqrt(d);
    a[j] = a[j] / diag[j];  // L[i][j] below the diagonal
#pragma unroll
    for (int k = j + 1; k < 6; ++k) a[k] -= a[j] * __shfl_sync(full, a[j], k);
  }
#pragma unroll
  for (int i = 5; i >= 0; --i) {
    double t = __shfl_sync(full, a[i], 6);
#pragma unroll
    for (int k = i + 1; k < 6; ++k) t -= __shfl_sync(full, a[i], k) * x[k];
    x[i] = t / diag[i];
  }
  return true;
}

// Rz(g) Ry(b) Rx(a) (AngleAxis composition at NuiKinfuOpenCLDepthTracker.cpp:486), from
// the angles' sines and cosines
__device__ __forceinline__ void euler_zyx(double sa, double ca, double sb, double cb, double sg, double cg,
                                          double (&R)[9]) {
  const double Rz[9] = {cg, -sg, 0, sg, cg, 0, 0, 0, 1};
  const double Ry[9] = {cb, 0, sb, 0, 1, 0, -sb, 0, cb};
  const double Rx[9] = {1, 0, 0, 0, ca, -sa, 0, sa, ca};
  double T[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double s = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) s += Rz[i * 3 + k] * Ry[k * 3 + j];
      T[i * 3 + j] = s;
    }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double s = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) s += T[i * 3 + k] * Rx[k * 3 + j];
      R[i * 3 + j] = s;
    }
}

// Copies the fields (d <- s), a field element a thread (called by the block's threads, the
// first 27 of which copy); T, U: TrackState or IcpLm.
template <class T, class U>
__device__ __forceinline__ void lm_copy(T* d, const U* s) {
  const int k = threadIdx.x;
  if (k < 9) d->R[k] = s->R[k], d->Rg[k] = s->Rg[k];
  if (k < 3) d->t[k] = s->t[k], d->tg[k] = s->tg[k];
  if (k < 27) d->good[k] = s->good[k];
  if (k < kMaxLevels) d->icp_iters[k] = s->icp_iters[k];
  if (k == 0) {
    d->lambda = s->lambda;
    d->err_old = s->err_old;
    d->error = s->error;
    d->count = s->count;
    d->level_done = s->level_done;
    d->status = s->status;
    d->iterations_run = s->iterations_run;
  }
}

// The LM step on the reduced sums (NuiKinfuOpenCLDepthTracker.cpp:324-496) by a block's first
// two warps, in phases separated by barriers of theirs alone: accept or reject and the 27
// normalised sums a thread each, the Cholesky solve and the determinant on a warp each, the
// increments' sines and cosines on three threads, the composition on one.  Every value comes
// from the same FP64 operations in the same order as a one-thread step, which took 8 us (4.5
// with the solve and the determinant on a thread each; 3.9 now).
struct IcpStepScratch {
  double A[6][6], b[6], x[6], det, sc[6];
  int go, solved;
};
__device__ __forceinline__ void icp_step_sync() { asm volatile("bar.sync 1, 64;" ::: "memory"); }
// Term t of the 29 among a warp's 64 sums: (i, j) of the upper triangle of [row, 1] by rows,
// at 8 i + j; then r^2 (6, 6) and the count (7, 7).
__device__ __forceinline__ int icp_term_at(int t) {
  if (t >= 27) return t == 27 ? 54 : 63;
  int i = 0, j = t;
  while (j >= 7 - i) j -= 7 - i, ++i;
  return 8 * i + i + j;
}
__device__ __noinline__ void icp_host_step(IcpLm* ts, IcpStepScratch& w, const double* sums, int iter,
                                              unsigned min_count) {
  const int tid = threadIdx.x;
  // accept or reject (every thread, alike)
  float err = (float)sums[27];
  const float cnt = (float)sums[28];
  err = (cnt > 0.f) ? sqrtf(err) / cnt : 3.402823466e+38f;
  // level start: lambda = 1, Rgood = Rcurr, errorOld = 1e20
  const float err_old = iter == 0 ? 1e20f : ts->err_old, l0 = iter == 0 ? 1.0f : ts->lambda;
  const bool reject = cnt < (float)min_count || err > err_old;
  const float lambda = reject ? l0 * 10.0f : l0 / 10.0f;
  double v = 0.0;
  if (tid < 27) v = reject ? ts->good[tid] : sums[tid];
  icp_step_sync();  // (the state has been read)
  if (tid == 0) {
    ts->error = err;
    ts->count = cnt;
    ts->iterations_run += 1;
    ts->lambda = lambda;
    ts->err_old = reject ? err_old : err;
    if (iter == 0) ts->level_done = reject ? 1 : 0;
    w.go = 1;
  }
  if (tid >= 32 && tid < 44) {  // back to the last good pose, or this one is good
    const int k = tid - 32;
    float *c = k < 9 ? ts->R + k : ts->t + k - 9, *g = k < 9 ? ts->Rg + k : ts->tg + k - 9;
    if (reject && iter > 0) *c = *g;
    else *g = *c;
  }
  if (reject && iter == 0) return;
  if (tid < 27) {  // sum sh = (i, j) of the upper triangle of [J|r] by rows, over the count
    if (!reject) ts->good[tid] = v;
    const int at = icp_term_at(tid), i = at >> 3, j = at & 7;
    v = v / (double)cnt;
    if (j == 6) {
      w.b[i] = v;
    } else {
      if (i == j) v *= (double)(1.0f + lambda);
      w.A[i][j] = v;
      w.A[j][i] = v;
    }
  }
  icp_step_sync();
  // a singular system (|det| < 1e-15 or NaN) or a failed factorisation loses tracking
  double a[6];
  const int row = min(tid & 31, 6);
#pragma unroll
  for (int k = 0; k < 6; ++k) a[k] = row < 6 ? w.A[row][k] : w.b[k];
  if (tid < 32) {
    double x[6];
    const bool solved = llt_solve6(a, x);
    if (tid == 0) {
      w.solved = solved ? 1 : 0;
#pragma unroll
      for (int r = 0; r < 6; ++r) w.x[r] = x[r];
    }
  } else {
    const double det = det6(a);
    if (tid == 32) w.det = det;
  }
  icp_step_sync();
  if (tid == 0) {
    if (!w.solved || !(fabs(w.det) >= 1e-15)) {
      ts->status = 3;
      w.go = 0;
    } else {
      const float al = (float)w.x[0], be = (float)w.x[1], ga = (float)w.x[2];
      if (al * al + be * be + ga * ga < 1e-6f) {
        ts->level_done = 1;
        w.go = 0;
      }
    }
  }
  icp_step_sync();
  if (!w.go) return;
  if (tid < 3) {  // sin and cos of the increment's angles (alpha, beta, gamma)
    double sn, cs;
    sincos((double)(float)w.x[tid], &sn, &cs);
    w.sc[2 * tid] = sn;
    w.sc[2 * tid + 1] = cs;
  }
  icp_step_sync();
  if (tid == 0) {
    double Ri[9];
    euler_zyx(w.sc[0], w.sc[1], w.sc[2], w.sc[3], w.sc[4], w.sc[5], Ri);
    float t0[3], R0[9];
#pragma unroll
    for (int i = 0; i < 3; ++i) t0[i] = ts->t[i];
#pragma unroll
    for (int i = 0; i < 9; ++i) R0[i] = ts->R[i];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double s = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) s += Ri[k * 3 + i] * (double)t0[k];
      ts->t[i] = (float)(s + (double)(float)w.x[3 + i]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double s = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) s += Ri[k * 3 + i] * (double)R0[k * 3 + j];
        ts->R[i * 3 + j] = (float)s;
      }
  }
}

// One product of the FP64 tensor path: D (8 x 8) += A (8 x 4) B (4 x 8).  Lane l holds
// A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}], so a lane's value of
// component l / 4 of row l % 4 serves as both operands of a sum of outer products.
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// What a depth pass reads for every pixel, in shared memory (the pass's registers are all taken:
// held there, the intrinsics had other values spilled in its loop): the running estimate and the
// previous camera pose (the reference maps' frame), a row and its translation a float4, R | t and
// R_inv | t; fx, fy, cx, cy; and a level's 1 / fx, 1 / fy, cx, cy as level_vertex forms them.
struct IcpPoses {
  float4 cur[3], prev[3], cam, lvl[kMaxLevels];
};
__device__ __forceinline__ void icp_cameras(IcpPoses& P, const SessionDesc& s) {  // a level a thread
  const int l = threadIdx.x;
  if (l == 0) P.cam = make_float4(s.cam.fx, s.cam.fy, s.cam.cx, s.cam.cy);
  if (l < kMaxLevels) {
    const float div = (float)(1 << l);
    P.lvl[l] = make_float4(div * s.cam.fx_inv, div * s.cam.fy_inv, s.cam.cx / div, s.cam.cy / div);
  }
}
// Fills three rows from a matrix and a translation (a row's column a thread, 12 threads).
__device__ __forceinline__ void icp_pose_rows(float4* rows, const float* R, const float* t) {
  const int k = threadIdx.x >> 2, c = threadIdx.x & 3;
  if (threadIdx.x < 12) reinterpret_cast<float*>(rows)[threadIdx.x] = c < 3 ? R[3 * k + c] : t[k];
}
__device__ __forceinline__ float dot_row(float4 r, float3 v) { return dot3(f3(r.x, r.y, r.z), v); }

// The row of one pixel (level pixel (x, y) at depth dep): false without a match, else
// [n x p, n | n.(q - p), 1].
__device__ __forceinline__ bool icp_depth_row(const SessionDesc& s, int level, int x, int y, float dep,
                                              const IcpPoses& P, float4& ra, float4& rb) {
  if (isnan(dep)) return false;
  const float4 k = P.lvl[level];
  const float3 v = f3(dep * (((float)x - k.z) * k.x), dep * (((float)y - k.w) * k.y), dep);  // level_vertex
  const float4 r0 = P.cur[0], r1 = P.cur[1], r2 = P.cur[2];
  const float3 pv = f3(dot_row(r0, v) + r0.w, dot_row(r1, v) + r1.w, dot_row(r2, v) + r2.w);
  const float4 q0 = P.prev[0], q1 = P.prev[1], q2 = P.prev[2];
  const float3 pd = f3(pv.x - q0.w, pv.y - q1.w, pv.z - q2.w);
  const float3 pp = f3(dot_row(q0, pd), dot_row(q1, pd), dot_row(q2, pd));
  const float4 c = P.cam;
  const float u = pp.x * c.x / pp.z + c.z;
  const float vv = pp.y * c.y / pp.z + c.w;
  const int W = s.W, H = s.H;
  if (!(u >= 0.0f && u < (float)W && vv >= 0.0f && vv < (float)H)) return false;
  // both maps sampled at once (their eight loads in flight together), then tested: a hole
  // of either makes the distance or the residual NaN
  const float3 rn = bilinear_holes(s.nref, u, vv, W, W * H);
  const float3 rv = bilinear_holes(s.vref, u, vv, W, W * H);
  const float3 diff = sub3(rv, pv);
  const float dist = sqrtf(dot3(diff, diff)), res = dot3(rn, diff);
  if (!(dist < s.dist_thr) || isnan(res)) return false;
  const float3 r = cross3(rn, pv);
  ra = make_float4(r.x, r.y, r.z, rn.x);
  rb = make_float4(rn.y, rn.z, res, 1.0f);
  return true;
}

// ---------------------------------------------------------------- the order of the sums
// The FP64 sums of an image's pixels are formed in an order that its size alone fixes, so a
// session's poses do not depend on how many blocks track it, on how wide they are or on the other
// sessions of the launch.  The pixels are cut into runs of 32 (one a lane) and leaves of a few
// consecutive runs.  Leaves u, u + 143, u + 286, ... are unit u, at most 32 of them (photometric
// rows: 12, as a leaf ends with 31 exchanges between the lanes, and their blocks have half the
// warps).  A leaf's rows are summed by one warp, run by run; a unit's leaves by the binary tree
// that joins those whose place differs in its highest bit first; and the units in fixed groups of
// nine, these by such a tree.  Blocks take whole units, and whichever stages fall to a thread, a
// warp or a block, the sums are the same (a leaf that does not exist adds zero, which changes no
// bit).
//
// 143 units are a block on each of 143 of the 148 SMs for one session, on 72 for each of two, on 36
// for each of four, and twelve each for a cluster of twelve; consecutive leaves in consecutive
// units keep a block on neighbouring pixels (such a cluster's on 1152 of every 13728 at 640 x 480)
// and spread every part of the image over all units.  143 is odd: with 144 a unit's photometric
// leaves lay in the same columns of a 640 x 480 image (sixteen such sessions: 1558 us against 1497).
// What it costs: with sums that followed the launch's shape a 640 x 480 depth session took 77 us
// alone and sixteen 234, now 82 and 255; colour-tracked 150 and 1312, now 167 and 1428.
struct IcpCut {
  int g, leaves, units;  // runs a leaf; leaves of the image; units that have any
  __device__ __forceinline__ IcpCut() {}
  // n pixels in at most `most` leaves of at least `least` runs
  __device__ __forceinline__ IcpCut(int n, int most, int least) {
    const int runs = (n + 31) >> 5;
    g = max(least, (runs + most - 1) / most);
    leaves = (runs + g - 1) / g;
    units = min(kIcpUnits, leaves);
  }
  __device__ __forceinline__ int of(int u) const { return (leaves - u + kIcpUnits - 1) / kIcpUnits; }  // unit u's leaves
};

// The leaves of n consecutive units from u on as tasks, dealt to the block's warps in turn, row by
// row of the units (leaf j of each, then leaf j + 1), so that a later task has a later leaf.  A
// task's number is its slot, so there are at most kIcpRoom and, past the end, a block's warps more.
struct IcpDeal {
  int n;
  unsigned recip;  // 2^20 / n and less than one more: exact quotients by n of such numbers
  __device__ __forceinline__ void form(int n_) { n = n_, recip = (1u << 20) / (unsigned)n_ + 1u; }
  __device__ __forceinline__ int leaf(int u, int task) const {
    return (int)((unsigned)task * recip >> 20) * (kIcpUnits - n) + u + task;
  }
};
// What a block does in the passes over one image: its units, as many at a time as have room for
// their leaves' sums in the slots, and the deals of those and of the rest.  Formed once for all
// iterations, each of which its divisions would cost a microsecond.
struct IcpPlan {
  IcpCut cut;
  int u0, mine;
  IcpDeal deal[2];
  __device__ __forceinline__ static int first(const IcpCut& c, int rank, int parts) { return rank * c.units / parts; }
  __device__ __forceinline__ void form(const IcpCut& c, int rank, int parts, int room) {
    const int f = first(c, rank, parts), n = first(c, rank + 1, parts) - f, at_once = max(1, min(n, room / c.of(0)));
    deal[0].form(at_once);
    deal[1].form(max(1, n % at_once));
    cut = c, u0 = f, mine = n;
  }
};
// The plans of a session's levels, and of its photometric rows, a thread each, and whose each unit
// is (its block, and its place there).
__device__ __forceinline__ IcpCut icp_cut(const SessionDesc& s, int q) {
  return q < kMaxLevels ? IcpCut((s.W >> q) * (s.H >> q), 32 * kIcpUnits, 1) : IcpCut(s.W * s.H, 12 * kIcpUnits, 2);
}
__device__ __forceinline__ void icp_plans(const SessionDesc& s, IcpPlan* plans, bool color, int rank, int parts, int room) {
  const int q = (int)threadIdx.x;
  if (q < s.levels || (q == kMaxLevels && color)) plans[q].form(icp_cut(s, q), rank, parts, room);
}
__device__ __forceinline__ void icp_owners(const SessionDesc& s, unsigned short (*owner)[kIcpUnits], bool color, int parts) {
  for (int i = threadIdx.x; i < (kMaxLevels + 1) * kIcpUnits; i += blockDim.x) {
    const int q = i / kIcpUnits, u = i % kIcpUnits;
    if (q >= s.levels && !(q == kMaxLevels && color)) continue;
    const IcpCut c = icp_cut(s, q);
    const int r = ((u + 1) * parts - 1) / c.units;
    if (u < c.units) owner[q][u] = (unsigned short)(r << 8 | (u - IcpPlan::first(c, r, parts)));
  }
}

// The terms of the 29 that a lane's two sums of a warp's 8 x 8 are, -1: none.
__device__ __forceinline__ int icp_lane_term(int i, int j) {
  if (i < 6) return j >= i && j < 7 ? 7 * i - i * (i - 1) / 2 + j - i : -1;
  return i == j ? 21 + i : -1;
}

// The depth rows of the units of a deal, from u0 on, their outer products added to a warp's 8 x 8
// FP64 sums (d0, d1: this lane's two of them) leaf by leaf.  The 29 sums of a pixel
// are the upper triangle of the outer product of [row, 1]: JtJ, Jtr, r^2 and the count.  The rows'
// FP32 values are widened, so every product is exact and only the sums round.
//
// The pass waits on its eight map gathers.  The sums of a warp take two doubles a lane instead
// of 29 a thread (58 registers), which lets 1024 threads of 64 registers share an SM instead of
// 512 of 128, so twice the warps wait at once (track at 640 x 480: 337 -> 281 us; 39 sessions:
// 164 -> 147 M warp instructions a launch).
__device__ __forceinline__ void icp_depth_pass(const SessionDesc& s, int level, const IcpCut& cut, const IcpDeal& deal,
                                               int u0, const IcpPoses& P, float* stage, double* slots) {
  const int w = s.W >> level, n = w * (s.H >> level);
  const float* __restrict__ Dl = s.dlev[level];
  const int lane = threadIdx.x & 31;
  const int c = lane >> 2, src = (lane & 3) * 4 + (c < 4 ? c : kIcpHalf + c - 4);
  float4* const sa = reinterpret_cast<float4*>(stage) + lane;
  float4* const sb = reinterpret_cast<float4*>(stage + kIcpHalf) + lane;
  const int terms = (icp_lane_term(c, 2 * (lane & 3)) & 0xff) | icp_lane_term(c, 2 * (lane & 3) + 1) << 8;
  // a pixel's row: its index over the width, rounded down by a reciprocal of 32 bits that is one
  // too large at most
  const unsigned recip = 0xffffffffu / (unsigned)w + 1u;
  int task = (int)(threadIdx.x >> 5), leaf = deal.leaf(u0, task);
  int left = cut.g, i = leaf * left * 32 + lane;  // (runs past the image's end have no pixel)
  float dn = i < n ? __ldg(Dl + i) : qnan();
  double d0 = 0.0, d1 = 0.0;
  while (leaf < cut.leaves) {
    const float dep = dn;
    int y = (int)__umulhi((unsigned)i, recip), x = i - y * w;
    if (x < 0) x += w, --y;
    // the next pixel's depth is in flight while the current one's row forms
    double* const slot = slots + task * kIcpTerms;
    const bool ends = --left == 0;
    i += 32;
    if (ends) {
      task += (int)(blockDim.x >> 5);
      leaf = deal.leaf(u0, task);
      left = cut.g;
      i = leaf * left * 32 + lane;
    }
    dn = i < n ? __ldg(Dl + i) : qnan();
    float4 ra = make_float4(0.f, 0.f, 0.f, 0.f), rb = ra;
    const bool ok = icp_depth_row(s, level, x, y, dep, P, ra, rb);
    if (__any_sync(0xffffffffu, ok)) {
      *sa = ra;
      *sb = rb;
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const double v = (double)stage[16 * q + src];
        dmma(d0, d1, v, v);
      }
      __syncwarp();
    }
    if (ends) {
      if ((terms & 0xff) != 0xff) slot[terms & 0xff] = d0;
      if (terms >= 0) slot[terms >> 8] = d1;
      d0 = d1 = 0.0;
    }
  }
}

// The photometric rows of the model points of the units of a deal, their 28 FP32 terms and the
// count added to a lane's FP64 sums; a leaf's by a reduce-scatter over the warp's lanes,
// terms padded to 32: at each of five steps a lane keeps half of its values, sends the other half
// to its partner and adds what it receives, so lane k ends with the leaf's sum of term k after 31
// exchanges.
__device__ __forceinline__ void icp_color_pass(const SessionDesc& s, const IcpCut& cut, const IcpDeal& deal, int u0,
                                               const IcpPoses& P, double* slots) {
  const int NM = s.W * s.H, lane = threadIdx.x & 31;
  const float4 r0 = P.cur[0], r1 = P.cur[1], r2 = P.cur[2];
  const float R[9] = {r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r2.x, r2.y, r2.z};
  const float3 tc = f3(r0.w, r1.w, r2.w);
#pragma unroll 1
  for (int task = (int)(threadIdx.x >> 5), leaf; (leaf = deal.leaf(u0, task)) < cut.leaves; task += (int)(blockDim.x >> 5)) {
    double acc[kIcpTerms];
#pragma unroll
    for (int q = 0; q < kIcpTerms; ++q) acc[q] = 0.0;
    const int i0 = leaf * cut.g * 32 + lane, i1 = min(NM, i0 + 32 * cut.g);
#pragma unroll 1
    for (int i = i0; i < i1; i += 32) {
      ColorRow row;
      if (!color_row(s, i, R, tc, row)) continue;
      row.add_to(acc);
    }
    double v[32];
#pragma unroll
    for (int q = 0; q < 32; ++q) v[q] = q < kIcpTerms ? acc[q] : 0.0;
#pragma unroll
    for (int half = 16; half > 0; half >>= 1) {
      const bool upper = lane & half;
#pragma unroll
      for (int j = 0; j < half; ++j) {
        const double send = upper ? v[j] : v[j + half];
        const double keep = upper ? v[j + half] : v[j];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, send, half);
      }
    }
    if (lane < kIcpTerms) slots[task * kIcpTerms + lane] = v[0];
  }
}

// The last stages of a tree by a group of lanes, as many as the block has warps (8, 16 or 32), of
// which there are 32: a group a term (icp_my_term), a lane an entry; every lane gets the sum.
__device__ __forceinline__ int icp_my_term() { return (int)(threadIdx.x / (blockDim.x >> 5)); }
__device__ __forceinline__ int icp_my_entry() { return (int)(threadIdx.x & ((blockDim.x >> 5) - 1)); }
__device__ __forceinline__ double icp_group_sum(double v) {
  for (int off = (int)(blockDim.x >> 6); off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// Unit sums from the leaves' in the slots, handed to put(unit, term, sum): a term of a unit by a
// group of as many lanes as the block has warps, or by four, two or one, as they suffice.
template <class Put>
__device__ __forceinline__ void icp_unit_sums(const IcpCut& cut, int u0, int kc, const double* slots, Put put) {
  __syncthreads();
  if (kc < 3) {
    const int t = icp_my_term(), e = icp_my_entry(), warps = (int)(blockDim.x >> 5);
    for (int k = 0; k < kc; ++k) {
      const int have = t < kIcpTerms ? cut.of(u0 + k) : 0;
      auto at = [&](int j) { return j < have ? slots[(j * kc + k) * kIcpTerms + t] : 0.0; };
      double v = at(e);
      if (warps < 32) v += at(e + 16);
      if (warps < 16) v += at(e + 8) + at(e + 24);
      v = icp_group_sum(v);
      if (e == 0 && t < kIcpTerms) put(u0 + k, t, v);
    }
  } else {
    const bool few = cut.of(0) <= 8;
    const int log = kc * 128 <= (int)blockDim.x ? 2 : kc * 64 <= (int)blockDim.x ? 1 : 0;
    for (int i = threadIdx.x; i < kc * 32 << log; i += blockDim.x) {
      const int o = i & ((1 << log) - 1), t = i >> log & 31, k = i >> log >> 5, have = t < kIcpTerms ? cut.of(u0 + k) : 0;
      const double* const p = slots + k * kIcpTerms + t;
      auto eight = [&](int j) {  // leaves j, j + 4, ..., j + 28
        if (few) return (j < have ? p[j * kc * kIcpTerms] : 0.0) + (j + 4 < have ? p[(j + 4) * kc * kIcpTerms] : 0.0);
        double v[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = j + 4 * m < have ? p[(j + 4 * m) * kc * kIcpTerms] : 0.0;
        return ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
      };
      double a = eight(o);
      if (log == 2) {
        a += __shfl_xor_sync(0xffffffffu, a, 2);
      } else {
        a += eight(o + 2);
      }
      if (log > 0) {
        a += __shfl_xor_sync(0xffffffffu, a, 1);
      } else {
        const double b = eight(1);
        a += b + eight(3);
      }
      if (o == 0 && t < kIcpTerms) put(u0 + k, t, a);
    }
  }
  __syncthreads();  // the slots are used again
}

// The sums of the block's units of one pass.  All threads must call it; the block has 8, 16 or 32
// warps (photometric rows: 8 or 16).
template <class Put>
__device__ __forceinline__ void icp_depth_sums(const SessionDesc& s, int level, const IcpPlan& plan, const IcpPoses& P,
                                               float* stage0, double* slots, Put put) {
  for (int done = 0; done < plan.mine; done += plan.deal[0].n) {
    const IcpDeal& deal = plan.deal[done + plan.deal[0].n > plan.mine];
    const int u = plan.u0 + done;
    icp_depth_pass(s, level, plan.cut, deal, u, P, stage0 + (threadIdx.x >> 5) * (kIcpStageBytes / 4), slots);
    icp_unit_sums(plan.cut, u, deal.n, slots, put);
  }
}
template <class Put>
__device__ __forceinline__ void icp_color_sums(const SessionDesc& s, const IcpPlan& plan, const IcpPoses& P, double* slots,
                                               Put put) {
  for (int done = 0; done < plan.mine; done += plan.deal[0].n) {
    const IcpDeal& deal = plan.deal[done + plan.deal[0].n > plan.mine];
    const int u = plan.u0 + done;
    icp_color_pass(s, plan.cut, deal, u, P, slots);
    icp_unit_sums(plan.cut, u, deal.n, slots, put);
  }
}

// The image's sums from its units': get(u, t) reads term t of unit u (the photometric terms from 32
// on).  A warp joins half a group of nine units, a group, or two groups 8 apart (of 32, 16 or 8
// warps), a lane a term; then as above.  The photometric normal equations and residual enter weighted, the count stays the
// depth count.  All threads must call it.
template <bool COLOR, class Get>
__device__ __forceinline__ void icp_image_sums(const SessionDesc& s, const IcpCut& cut, const IcpCut& ccut, bool photo,
                                               float* stage0, double* sums, Get get) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (int)(blockDim.x >> 5);
  double* const w = reinterpret_cast<double*>(stage0);
  auto joined = [&](int units, int t) {
    auto at = [&](int u) { return u < units && lane < kIcpTerms ? get(u, t) : 0.0; };
    static_assert(kIcpUnits <= 9 * 16, "the order of the units' sums");
    auto half0 = [&](int u) {  // units u, u + 16, u + 32, u + 48 and u + 128
      const double v0 = at(u), v1 = at(u + 16), v2 = at(u + 32), v3 = at(u + 48), v8 = at(u + 128);
      return ((v0 + v1) + (v2 + v3)) + v8;
    };
    auto half1 = [&](int u) {  // the other four of its sixteenth
      const double v4 = at(u + 64), v5 = at(u + 80), v6 = at(u + 96), v7 = at(u + 112);
      return (v4 + v5) + (v6 + v7);
    };
    if (!COLOR && warps == 32) return warp < 16 ? half0(warp) : half1(warp - 16);
    double a = half0(warp) + half1(warp);
    if (warps == 8) a += half0(warp + 8) + half1(warp + 8);
    return a;
  };
  w[33 * warp + lane] = joined(cut.units, lane);
  if (COLOR && photo) w[33 * (warps + warp) + lane] = joined(ccut.units, 32 + lane);
  __syncthreads();
  const int term = icp_my_term(), e = icp_my_entry();
  double a = icp_group_sum(w[33 * e + term]);
  if (COLOR && photo) {
    const double c = icp_group_sum(w[33 * (warps + e) + term]);
    if (term < kIcpTerms - 1) a += (double)s.photo_w * c;
  }
  if (e == 0) sums[term] = a;
  __syncthreads();  // (the staging memory is used again)
}

// NuiKinfuOpenCLShiftScene::integrateVolume -> shiftVolume (NuiKinfuOpenCLShiftScene.cpp:
// 288-362): before a shifting volume integrates, every axis on which the camera lies
// voxel_shift or more voxels from the basis moves the volume by voxel_shift voxels; the
// camera's local translation moves back by the same distance and the offset forward.  The
// frame's shift is left in ts->shift for the fetch / roll kernels that follow.
__device__ void shift_decide(const SessionDesc& s, TrackState* ts) {
  ts->shift[0] = ts->shift[1] = ts->shift[2] = 0;
  const int vs = s.voxel_shift;
  if (vs <= 0 || s.fmt < 0) return;
  float st[3];
  int tr[3];
  for (int a = 0; a < 3; ++a) {
    st[a] = ts->xf.t[a] - s.shift_basis[a];
    const int f = (int)floorf(st[a] / s.cell[a]);
    tr[a] = st[a] < 0.f ? max(-vs, f) : min(vs, f);
  }
  for (int a = 0; a < 3; ++a)
    if (abs(tr[a]) >= vs) {
      ts->shift[a] = tr[a];
      ts->voff[a] += tr[a];
      st[a] -= (float)tr[a] * s.cell[a];
    }
  for (int a = 0; a < 3; ++a) {
    ts->xf.t[a] = st[a] + s.shift_basis[a];
    ts->t[a] = ts->xf.t[a];
  }
}

// After the last ICP iteration (or on frame 0): the pose, the integration gate
// (NuiKinfuTrackingEngine.cpp:115-127), and the estimate for the next frame.
// shift_now: the tick's finalize makes the shifting volume's shift of an integrating
// frame here; the step-wise track leaves it to the integration call (k_open_gate).
__device__ __forceinline__ void track_finalize(const SessionDesc& s, TrackState* ts, int shift_now) {
  if (s.kind == kFirstFrame) {
    ts->integrate = ts->status == 0 ? 1 : 0;
    ts->shift[0] = ts->shift[1] = ts->shift[2] = 0;
    if (ts->integrate && shift_now) shift_decide(s, ts);
    return;
  }
  ts->shift[0] = ts->shift[1] = ts->shift[2] = 0;
  if (ts->status != 0) {  // tracking lost: keep the previous pose, skip the rest
    for (int i = 0; i < 9; ++i) ts->R[i] = ts->xf.R[i];
    for (int i = 0; i < 3; ++i) ts->t[i] = ts->xf.t[i];
    ts->integrate = 0;
    return;
  }
  double a[9];
  for (int i = 0; i < 9; ++i) a[i] = ts->R[i];
  const double c00 = a[4] * a[8] - a[5] * a[7], c01 = a[5] * a[6] - a[3] * a[8], c02 = a[3] * a[7] - a[4] * a[6];
  const double det = a[0] * c00 + a[1] * c01 + a[2] * c02;
  const double inv[9] = {c00, a[2] * a[7] - a[1] * a[8], a[1] * a[5] - a[2] * a[4],
                         c01, a[0] * a[8] - a[2] * a[6], a[2] * a[3] - a[0] * a[5],
                         c02, a[1] * a[6] - a[0] * a[7], a[0] * a[4] - a[1] * a[3]};
  for (int i = 0; i < 9; ++i) {
    ts->xf.R[i] = ts->R[i];
    ts->xf.R_inv[i] = (float)(inv[i] / det);
  }
  for (int i = 0; i < 3; ++i) ts->xf.t[i] = ts->t[i];
  // rotation angle of R^-1 * R_last and translation distance
  double tr = 0;
  for (int i = 0; i < 3; ++i)
    for (int k = 0; k < 3; ++k) tr += (double)ts->R[k * 3 + i] * (double)ts->lastR[k * 3 + i];
  const double cv = fmin(1.0, fmax(-1.0, (tr - 1.0) / 2.0));
  const double rn = acos(cv);
  // translations compared globally: local + the volume's offset (0 for a fixed volume)
  double tn = 0;
  for (int i = 0; i < 3; ++i) {
    const float g = ts->voff[i] ? ts->t[i] + (float)ts->voff[i] * s.cell[i] : ts->t[i];
    tn += ((double)(g - ts->lastT[i])) * ((double)(g - ts->lastT[i]));
  }
  tn = sqrt(tn);
  ts->integrate = ((float)((rn + tn) / 2) >= s.integ_thr) ? 1 : 0;
  if (ts->integrate) {
    if (shift_now) shift_decide(s, ts);
    for (int i = 0; i < 9; ++i) ts->lastR[i] = ts->R[i];
    for (int i = 0; i < 3; ++i) ts->lastT[i] = ts->voff[i] ? ts->t[i] + (float)ts->voff[i] * s.cell[i] : ts->t[i];
  }
}

// The end of a session's tracking, by one thread: the above for an active session, then status,
// gate and pose of this tick into the packed arrays that the host reads back with one copy.
__device__ __noinline__ void track_end(const SessionDesc& s, const TrackOut& out) {
  TrackState* ts = s.ts;
  if (ts == nullptr) return;
  if (s.kind >= 0) track_finalize(s, ts, out.shift_now);
  if (!out.pose || !out.status) return;
  float* const pose = out.pose + 14 * s.slot;
  out.status[2 * s.slot] = s.kind < 0 ? 0 : ts->status;
  out.status[2 * s.slot + 1] = ts->integrate;
  for (int k = 0; k < 9; ++k) pose[k] = ts->xf.R[k];
  for (int k = 0; k < 3; ++k) pose[9 + k] = ts->xf.t[k];
  pose[12] = ts->error;
  pose[13] = ts->count;
}

// The same as a launch of its own, behind the clusters (inside them it cost a batch of 64 more
// than the launch: 40.0 ms for six ticks against 39.4).
__global__ void k_track_end(const SessionDesc* __restrict__ descs, int fam, const TrackOut out) {
  const SessionDesc& s = descs[blockIdx.x];
  if (threadIdx.x == 0 && in_family(s, fam)) track_end(s, out);
}

// All ICP iterations of every level of one frame, one thread-block cluster per session
// (NuiKinfuOpenCLDepthTracker::IterativeClosestPoint, NuiKinfuOpenCLDepthTracker.cpp:240-504).
// The C blocks of a cluster (C = 2..16, a launch attribute: the ICP tuning's blocks per
// session) share the level's units; every iteration each block leaves its units' sums in its own
// shared memory, a cluster barrier makes them visible, block 0 adds them up through distributed
// shared memory and runs the host step (LM accept/reject, FP64 Cholesky, pose update), and a
// second barrier publishes the new estimate, which every block reads from block 0's shared
// memory.  The hardware schedules a cluster's blocks together and its barriers need no polling;
// every block takes the same exits at the same points, since each decision comes from block 0's
// published state.  One launch per tick replaces one launch per iteration, and sessions whose
// levels stop early leave their SMs to the others.
//
// The block size is the launch's (256, 512 or 1024 threads, see launch_icp_cluster): the same
// code with kIcpStageBytes of dynamic shared memory a warp, slots for `room` leaves and the sums
// of the block's units behind them.  Launches without a colour-tracked session take the
// variant without the photometric rows (64 registers, up to 1024 threads); the rows' 29 FP64
// sums a thread need 128 (up to 512).
template <bool COLOR>
__global__ void __launch_bounds__(COLOR ? 512 : 1024, 1)
    k_icp_cluster(const SessionDesc* __restrict__ descs, int fam, int room) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const SessionDesc& s = descs[blockIdx.y];
  if (s.kind != kTrackFrame || !in_family(s, fam)) return;  // the same for every block of the cluster
  TrackState* ts = s.ts;
  const int rank = (int)cluster.block_rank(), C = (int)cluster.num_blocks();
  extern __shared__ __align__(16) float icp_stage[];
  __shared__ IcpPoses P;
  __shared__ double sums[32];
  __shared__ IcpLm lm;  // block 0: the tracker state during the kernel
  __shared__ IcpStepScratch hw;  // block 0: the LM step's intermediate values
  __shared__ IcpPlan plans[kMaxLevels + 1];  // of the levels, and of the photometric rows
  __shared__ unsigned short owner[kMaxLevels + 1][kIcpUnits];  // whose each unit is, and its place there
  double* const slots = reinterpret_cast<double*>(icp_stage + (blockDim.x >> 5) * (kIcpStageBytes / 4));
  icp_plans(s, plans, COLOR, rank, C, room);
  if (rank == 0) icp_owners(s, owner, COLOR, C);
  // this block's units' sums: depth, then photometric
  constexpr int kCols = COLOR ? 64 : 32;
  double* const mine = slots + room * kIcpTerms;
  icp_pose_rows(P.cur, ts->R, ts->t);
  icp_pose_rows(P.prev, ts->xf.R_inv, ts->xf.t);
  icp_cameras(P, s);
  const int status0 = ts->status;
  if (rank == 0) lm_copy(&lm, ts);
  // every block has read the initial state before block 0 writes any of it
  cluster.sync();
  if (status0 != 0) return;
  for (int level = s.levels - 1; level >= 0; --level) {
    const bool photo = COLOR && s.photo_w > 0.f && level == 0;
    const IcpPlan &plan = plans[level], &cplan = plans[kMaxLevels];
    for (int iter = 0; iter < s.iters[level]; ++iter) {
      icp_depth_sums(s, level, plan, P, icp_stage, slots, [&](int u, int t, double v) { mine[(u - plan.u0) * kCols + t] = v; });
      if (photo) icp_color_sums(s, cplan, P, slots, [&](int u, int t, double v) { mine[(u - cplan.u0) * kCols + 32 + t] = v; });
      cluster.sync();  // every block's sums are visible to block 0
      if (rank == 0) {
        if (threadIdx.x == 0) lm.icp_iters[level] += 1u;
        icp_image_sums<COLOR>(s, plan.cut, cplan.cut, photo, icp_stage, sums, [&](int u, int t) {
          const unsigned o = owner[t < 32 ? level : kMaxLevels][u];
          return cluster.map_shared_rank(mine, o >> 8)[(o & 255) * kCols + t];
        });
        if (threadIdx.x < 64) icp_host_step(&lm, hw, sums, iter, s.icp_min_count[level]);
      }
      cluster.sync();  // block 0's new estimate is visible to every block
      // (block 0 writes its state again only behind the next iteration's first barrier)
      const IcpLm* lm0 = cluster.map_shared_rank(&lm, 0);
      icp_pose_rows(P.cur, lm0->R, lm0->t);
      const int flags[2] = {lm0->status, lm0->level_done};
      __syncthreads();
      if (flags[0] != 0) {  // tracking lost: every block leaves together
        if (rank == 0) lm_copy(ts, &lm);
        cluster.sync();     // (block 0's shared memory stays alive until all have read it)
        return;
      }
      if (flags[1]) break;
    }
  }
  if (rank == 0) lm_copy(ts, &lm);
  cluster.sync();  // no block leaves while another may still read block 0's shared memory
}

// All ICP iterations of a small batch's sessions, each over its share of the whole device (a
// block an SM, launched cooperatively: all blocks are resident, so they may wait for one
// another).  Every iteration a block leaves its units' sums in the session's part of `work` and
// counts itself in; when all have, every block adds all the sums, in the same order, and runs the
// LM step on its own copy of the state, so nothing has to be sent back.  A wait that runs out (it
// cannot with all blocks resident) marks the workspace and ends the frame as stalled, and so does
// every later launch on it at once, until the host has cleared it (icp_recover).
//
// What bounds it is latency: an iteration is a pass of a few us, a trip through L2 and the LM
// step.  A cluster is at most 16 SMs, on which a pass of a colour-tracked 640 x 480 level takes
// 120 us; a launch an iteration costs 2 us even after the level has ended (a level that starts
// close to its end runs one iteration of the ten).  A 640 x 480 depth session's iterations, over
// its levels and on 72 SMs, take 12.4 us (pass and unit sums 5.1, arriving and waiting 2.0, the
// image's sums 1.0, LM step 4.3; on 143 the pass is 3.9), with photometric rows 16.1 (pass 3.7,
// those and the wait 6.9).
template <bool COLOR>
__global__ void __launch_bounds__(COLOR ? 512 : 1024, 1)
    k_icp_wide(const SessionDesc* __restrict__ descs, int fam, int room, IcpWide* __restrict__ work, const TrackOut out) {
  const SessionDesc& s = descs[blockIdx.y];
  if (!in_family(s, fam)) return;  // (this and the next: the same for every block of the session)
  if (s.kind != kTrackFrame) {
    if (blockIdx.x == 0 && threadIdx.x == 0) track_end(s, out);
    return;
  }
  TrackState* ts = s.ts;
  IcpWide& f = work[blockIdx.y];
  extern __shared__ __align__(16) float icp_stage[];
  __shared__ IcpPoses P;
  __shared__ double sums[32];
  __shared__ IcpLm lm;
  __shared__ IcpStepScratch hw;
  __shared__ int state, limit;  // -1: the wait ran out; its polls
  const int B = (int)gridDim.x;
  lm_copy(&lm, ts);  // (written again only when every block has counted itself in for the last time)
  icp_pose_rows(P.prev, ts->xf.R_inv, ts->xf.t);
  icp_cameras(P, s);
  icp_pose_rows(P.cur, ts->R, ts->t);
  if (threadIdx.x == 0) {
    state = *(volatile unsigned*)&f.stalled ? -1 : 0;
    limit = f.polls > 0 ? f.polls : kIcpPolls;
  }
  __shared__ IcpPlan plans[kMaxLevels + 1];  // of the levels, and of the photometric rows
  icp_plans(s, plans, COLOR, (int)blockIdx.x, B, room);
  __syncthreads();
  if (lm.status != 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) track_end(s, out);
    return;
  }
  double* const slots = reinterpret_cast<double*>(icp_stage + (blockDim.x >> 5) * (kIcpStageBytes / 4));
  unsigned turn = 0;  // iterations of this launch
  bool go = state == 0;
  for (int level = s.levels - 1; level >= 0 && go; --level) {
    const bool photo = COLOR && s.photo_w > 0.f && level == 0;
    const IcpPlan &plan = plans[level], &cplan = plans[kMaxLevels];
    for (int iter = 0; iter < s.iters[level]; ++iter) {
      // (two sets of sums in turn: a block may be one iteration ahead of one that still reads)
      double(*const part)[64] = f.part[turn & 1];
      icp_depth_sums(s, level, plan, P, icp_stage, slots, [&](int u, int t, double v) { part[u][t] = v; });
      if (photo) icp_color_sums(s, cplan, P, slots, [&](int u, int t, double v) { part[u][32 + t] = v; });
      __syncthreads();
      ++turn;
      if (threadIdx.x == 0) {
        unsigned e;
        int polls = 0;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&f.arrived) : "memory");
        do {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(e) : "l"(&f.arrived) : "memory");
        } while (e < turn * (unsigned)B && ++polls < limit);
        if (e < turn * (unsigned)B) {
          f.stalled = 1u;
          state = -1;
        }
      }
      __syncthreads();
      if (state != 0) {
        go = false;
        break;
      }
      if (threadIdx.x == 0) lm.icp_iters[level] += 1u;
      icp_image_sums<COLOR>(s, plan.cut, cplan.cut, photo, icp_stage, sums, [&](int u, int t) { return __ldcg(&part[u][t]); });
      if (threadIdx.x < 64) icp_host_step(&lm, hw, sums, iter, s.icp_min_count[level]);
      __syncthreads();
      icp_pose_rows(P.cur, lm.R, lm.t);
      const int lost = lm.status, done = lm.level_done;
      __syncthreads();
      if (lost != 0) go = false;
      if (lost != 0 || done) break;
    }
  }
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0 && state != 0) lm.status = kIcpStalled;
    __syncthreads();
    lm_copy(ts, &lm);
    __syncthreads();
    if (threadIdx.x == 0) track_end(s, out);
  }
  if (threadIdx.x == 0 && state == 0 && atomicAdd(&f.left, 1u) == (unsigned)B - 1u) {  // every block has made its last read
    f.left = 0u;
    f.arrived = 0u;
  }
}

template __global__ void k_icp_cluster<false>(const SessionDesc*, int, int);
template __global__ void k_icp_cluster<true>(const SessionDesc*, int, int);
template __global__ void k_icp_wide<false>(const SessionDesc*, int, int, IcpWide*, const TrackOut);
template __global__ void k_icp_wide<true>(const SessionDesc*, int, int, IcpWide*, const TrackOut);

// Start of an integration the host requests directly (step-wise calls): the gate opens, the
// counters it reports start over (for a voxel hash, the failures before it are noted) and the
// shift is made.
__global__ void k_open_gate(const SessionDesc* __restrict__ descs) {
  const SessionDesc& s = descs[blockIdx.x];
  if (threadIdx.x != 0 || s.kind < 0) return;
  s.ts->integrate = 1;
  s.ts->touched = 0ull;
  if (s.hcount) {
    s.hcount[kHashFailedBefore] = s.hcount[kHashFailed];
    s.hcount[kHashFaultsBefore] = s.hcount[kHashChainFaults];
  }
  shift_decide(s, s.ts);
}

// nui_set_pose: the camera pose and the tracker's estimate.
__global__ void k_set_pose(TrackState* ts, const __grid_constant__ DevXform m) {
  const int k = threadIdx.x;
  if (k < 9) {
    ts->xf.R[k] = ts->R[k] = m.R[k];
    ts->xf.R_inv[k] = m.R_inv[k];
  }
  if (k < 3) ts->xf.t[k] = ts->t[k] = m.t[k];
}

}  // namespace nui
