// Point-to-plane ICP: every iteration of every level in one launch, one thread-block
// cluster per session, no host round trip.
//
// Per pixel (icp_block_kernel, icp.cl:222-292): rebuild the level's vertex from its depth,
// transform it by the running estimate, project into the previous camera with
// full-resolution intrinsics, bilinearly sample the world reference normal and vertex
// (icp.cl:192-220; a tap NaN -> no match), and if |q - p| < distThres form the row
// [n x p, n | n.(q - p)].  A warp adds the outer products of its pixels' rows in FP64 on the
// tensor path (exact products of the FP32 row values); blocks add their warps' sums, the
// cluster's first block the blocks' (distributed shared memory, fixed order), and it runs the
// host step of
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
// under- or overflows: b in 2^-40 .. 2^40, a zero or in 2^-80 .. 2^80 in magnitude.
__device__ __forceinline__ float div_shared(float a, float b, float r) {
  float q = a * r;
  q = __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
  return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
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
  // away along every axis that counts: the numerators are then far inside div_shared's range
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

// What a depth pass reads for every pixel: held in registers through the pass (the barriers
// of the staging would have it loaded again for each pixel).
struct IcpView {
  const float4 *nref, *vref;
  float fx, fy, cx, cy;      // full-resolution intrinsics
  float fxi, fyi, cxl, cyl;  // the level's, as level_vertex forms them
  float fW, fH, thr;
  int W, N;
  __device__ __forceinline__ IcpView(const SessionDesc& s, int level)
      : nref(s.nref), vref(s.vref), fx(s.cam.fx), fy(s.cam.fy), cx(s.cam.cx), cy(s.cam.cy),
        fxi((float)(1 << level) * s.cam.fx_inv), fyi((float)(1 << level) * s.cam.fy_inv),
        cxl(s.cam.cx / (float)(1 << level)), cyl(s.cam.cy / (float)(1 << level)), fW((float)s.W), fH((float)s.H),
        thr(s.dist_thr), W(s.W), N(s.W * s.H) {}
};
// The running estimate and the previous camera pose (the reference maps' frame), a row and
// its translation a float4: R | t, and R_inv | t.
struct IcpPoses {
  float4 cur[3], prev[3];
};
// Fills three rows from a matrix and a translation (a row's column a thread, 12 threads).
__device__ __forceinline__ void icp_pose_rows(float4* rows, const float* R, const float* t) {
  const int k = threadIdx.x >> 2, c = threadIdx.x & 3;
  if (threadIdx.x < 12) reinterpret_cast<float*>(rows)[threadIdx.x] = c < 3 ? R[3 * k + c] : t[k];
}
__device__ __forceinline__ float dot_row(float4 r, float3 v) { return dot3(f3(r.x, r.y, r.z), v); }

// The row of one pixel (level pixel (x, y) at depth dep): false without a match, else
// [n x p, n | n.(q - p), 1].
__device__ __forceinline__ bool icp_depth_row(const IcpView& c, int x, int y, float dep, const IcpPoses& P,
                                              float4& ra, float4& rb) {
  if (isnan(dep)) return false;
  const float3 v = f3(dep * (((float)x - c.cxl) * c.fxi), dep * (((float)y - c.cyl) * c.fyi), dep);  // level_vertex
  const float4 r0 = P.cur[0], r1 = P.cur[1], r2 = P.cur[2];
  const float3 pv = f3(dot_row(r0, v) + r0.w, dot_row(r1, v) + r1.w, dot_row(r2, v) + r2.w);
  const float4 q0 = P.prev[0], q1 = P.prev[1], q2 = P.prev[2];
  const float3 pd = f3(pv.x - q0.w, pv.y - q1.w, pv.z - q2.w);
  const float3 pp = f3(dot_row(q0, pd), dot_row(q1, pd), dot_row(q2, pd));
  const float u = pp.x * c.fx / pp.z + c.cx;
  const float vv = pp.y * c.fy / pp.z + c.cy;
  if (!(u >= 0.0f && u < c.fW && vv >= 0.0f && vv < c.fH)) return false;
  // both maps sampled at once (their eight loads in flight together), then tested: a hole
  // of either makes the distance or the residual NaN
  const float3 rn = bilinear_holes(c.nref, u, vv, c.W, c.N);
  const float3 rv = bilinear_holes(c.vref, u, vv, c.W, c.N);
  const float3 diff = sub3(rv, pv);
  const float dist = sqrtf(dot3(diff, diff)), res = dot3(rn, diff);
  if (!(dist < c.thr) || isnan(res)) return false;
  const float3 r = cross3(rn, pv);
  ra = make_float4(r.x, r.y, r.z, rn.x);
  rb = make_float4(rn.y, rn.z, res, 1.0f);
  return true;
}

// How a level's pixels are dealt: runs of T x per pixels, of which this thread's part (a block
// or a warp of T threads, thread `tid` of it) takes run `rank`, rank + C, ...
struct IcpDeal {
  int T, tid, per, rank, C;
};

// The depth rows of the level's pixels that fall to this thread's part, their outer products added to the warp's 8 x 8 FP64
// sums (d0, d1: this lane's two of them).  The 29 sums of a pixel are the upper triangle of
// the outer product of [row, 1]: JtJ, Jtr, r^2 and the count.  The rows' FP32 values are
// widened, so every product is exact and only the sums round.
//
// The pass waits on its eight map gathers.  The sums of a warp take two doubles a lane instead
// of 29 a thread (58 registers), which lets 1024 threads of 64 registers share an SM instead of
// 512 of 128, so twice the warps wait at once (track at 640 x 480: 337 -> 281 us; 39 sessions:
// 164 -> 147 M warp instructions a launch).
__device__ __forceinline__ void icp_depth_pass(const SessionDesc& s, int level, const IcpDeal& deal,
                                               const IcpPoses& P, float* stage, double& d0, double& d1) {
  const IcpView view(s, level);
  const int w = s.W >> level, n = w * (s.H >> level);
  const float* __restrict__ Dl = s.dlev[level];
  const int T = deal.T, per = deal.per, C = deal.C, lane = threadIdx.x & 31;
  const int c = lane >> 2, src = (lane & 3) * 4 + (c < 4 ? c : kIcpHalf + c - 4);
  float4* const sa = reinterpret_cast<float4*>(stage) + lane;
  float4* const sb = reinterpret_cast<float4*>(stage + kIcpHalf) + lane;
  // the next pixel's depth is in flight while the current one's row forms; a pixel's column
  // and row advance with its index, by T within a run and by the rest of the other blocks'
  // runs after it
  const int jump = T * ((C - 1) * per + 1), ty = T / w, tx = T - ty * w, jy = jump / w, jx = jump - jy * w;
  int base = deal.rank * T * per, k = 0;
  int i = base + deal.tid, y = i / w, x = i - y * w;
  float dn = i < n ? __ldg(Dl + i) : qnan();
  while (base < n) {
    const int cx = x, cy = y;
    const float dep = dn;
    const bool step = ++k < per;
    if (!step) {
      k = 0;
      base += C * T * per;
    }
    i += step ? T : jump;
    x += step ? tx : jx;
    y += step ? ty : jy;
    if (x >= w) x -= w, ++y;
    dn = i < n ? __ldg(Dl + i) : qnan();
    float4 ra = make_float4(0.f, 0.f, 0.f, 0.f), rb = ra;
    const bool ok = icp_depth_row(view, cx, cy, dep, P, ra, rb);
    if (!__any_sync(0xffffffffu, ok)) continue;
    *sa = ra;
    *sb = rb;
    __syncwarp();
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const double x = (double)stage[16 * g + src];
      dmma(d0, d1, x, x);
    }
    __syncwarp();
  }
}

// The photometric rows of the model points that fall to this thread's part, their 28 FP32 terms and
// the count added to this thread's FP64 sums.
__device__ __forceinline__ void icp_color_pass(const SessionDesc& s, const IcpDeal& deal, const IcpPoses& P,
                                               double (&acc)[kIcpTerms]) {
  const int NM = s.W * s.H, T = deal.T, per = deal.per;
  const float4 r0 = P.cur[0], r1 = P.cur[1], r2 = P.cur[2];
  const float R[9] = {r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r2.x, r2.y, r2.z};
  const float3 tc = f3(r0.w, r1.w, r2.w);
#pragma unroll 1
  for (int base = deal.rank * T * per; base < NM; base += deal.C * T * per)
#pragma unroll 1
    for (int k = 0; k < per; ++k) {
      const int i = base + k * T + deal.tid;
      ColorRow row;
      if (i >= NM || !color_row(s, i, R, tc, row)) continue;
      row.add_to(acc);
    }
}

// Block sums from the warps' sums, each warp's left in its part of the staging memory: the
// lanes of a warp are dealt over 32 / warps terms (icp_my_term), a lane takes a warp's term (at
// index `at` of its 64 doubles) and the lanes add up pairwise; every lane of a term's group
// gets its sum.  (A thread a term, adding the warps one after another, took 0.9 us of 32 warps.)
// All threads must call it; the block has 8, 16 or 32 warps.
__device__ __forceinline__ int icp_my_term() { return (int)(threadIdx.x / (blockDim.x >> 5)); }
__device__ __forceinline__ double icp_group_sum(double v) {
  for (int off = (int)(blockDim.x >> 6); off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ double icp_warps_sum(const float* stage0, int at) {
  const int src = (int)(threadIdx.x & ((blockDim.x >> 5) - 1));
  __syncthreads();
  const double v = reinterpret_cast<const double*>(stage0 + src * (kIcpStageBytes / 4))[at];
  __syncthreads();  // the staging memory is used again
  return icp_group_sum(v);
}

// The block's sums of one pass, this thread's term (icp_my_term, at `at` of a warp's 64 for the
// depth rows): of the depth rows, and of the photometric ones.  All threads must call it.
__device__ __forceinline__ double icp_depth_sums(const SessionDesc& s, int level, const IcpDeal& deal,
                                                 const IcpPoses& P, float* stage0, int at) {
  float* const stage = stage0 + (threadIdx.x >> 5) * (kIcpStageBytes / 4);  // this warp's
  double* const wsum = reinterpret_cast<double*>(stage);
  const int lane = threadIdx.x & 31;
  double d0 = 0.0, d1 = 0.0;
  icp_depth_pass(s, level, deal, P, stage, d0, d1);
  wsum[2 * lane] = d0;
  wsum[2 * lane + 1] = d1;
  return icp_warps_sum(stage0, at);
}
// (a warp's sums by a reduce-scatter over its lanes, terms padded to 32: at each of five
// steps a lane keeps half of its values, sends the other half to its partner and adds what it
// receives, so lane k ends with the warp's sum of term k after 31 exchanges)
__device__ __forceinline__ double icp_color_sums(const SessionDesc& s, const IcpDeal& deal, const IcpPoses& P,
                                                 float* stage0) {
  double acc[kIcpTerms];
#pragma unroll
  for (int k = 0; k < kIcpTerms; ++k) acc[k] = 0.0;
  icp_color_pass(s, deal, P, acc);
  const int lane = threadIdx.x & 31;
  double v[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = k < kIcpTerms ? acc[k] : 0.0;
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
  reinterpret_cast<double*>(stage0 + (threadIdx.x >> 5) * (kIcpStageBytes / 4))[lane] = v[0];
  return icp_warps_sum(stage0, icp_my_term());
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
// session) share the level's pixels (runs of blockDim.x x per pixels); every iteration each
// block reduces its FP64 sums into its own shared memory, a cluster barrier makes them
// visible, block 0 adds the blocks' sums in rank order through distributed shared memory and
// runs the host step (LM accept/reject, FP64 Cholesky, pose update), and a second barrier
// publishes the new estimate, which every block reads from block 0's shared memory.  The
// hardware schedules a cluster's blocks together and its barriers need no polling; every
// block takes the same exits at the same points, since each decision comes from block 0's
// published state.  One launch per tick replaces one launch per iteration, and sessions
// whose levels stop early leave their SMs to the others.
//
// The block size is the launch's (256, 512 or 1024 threads, see launch_track): the same code
// with kIcpStageBytes of dynamic shared memory a warp.  Launches without a colour-tracked
// session take the variant without the photometric rows (64 registers, up to 1024 threads);
// the rows' 29 FP64 sums a thread need 128 (up to 512).
template <bool COLOR>
__global__ void __launch_bounds__(COLOR ? 512 : 1024, 1)
    k_icp_cluster(const SessionDesc* __restrict__ descs, int fam, int ppt) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const SessionDesc& s = descs[blockIdx.y];
  if (s.kind != kTrackFrame || !in_family(s, fam)) return;  // the same for every block of the cluster
  TrackState* ts = s.ts;
  const int rank = (int)cluster.block_rank(), C = (int)cluster.num_blocks();
  extern __shared__ __align__(16) float icp_stage[];
  __shared__ IcpPoses P;
  __shared__ double part[2][32];  // this block's depth / photometric sums
  __shared__ double sums[kIcpTerms];
  __shared__ IcpLm lm;  // block 0: the tracker state during the kernel
  __shared__ IcpStepScratch hw;  // block 0: the LM step's intermediate values
  icp_pose_rows(P.cur, ts->R, ts->t);
  icp_pose_rows(P.prev, ts->xf.R_inv, ts->xf.t);
  const int status0 = ts->status;
  if (rank == 0) lm_copy(&lm, ts);
  // every block has read the initial state before block 0 writes any of it
  cluster.sync();
  if (status0 != 0) return;
  const int term = icp_my_term(), at = icp_term_at(term);
  const bool writes = term < kIcpTerms && (threadIdx.x & ((blockDim.x >> 5) - 1)) == 0;  // a thread a term
  for (int level = s.levels - 1; level >= 0; --level) {
    // runs no longer than leave every block one: a level's few runs would otherwise fall
    // unevenly on the cluster's blocks (19 runs of 1024 pixels for 16 at 160 x 120), and a
    // pass waits for its slowest block
    const int per = max(1, min(ppt, (s.W >> level) * (s.H >> level) / (C * (int)blockDim.x)));
    const IcpDeal deal{(int)blockDim.x, (int)threadIdx.x, per, rank, C};
    const bool photo = COLOR && s.photo_w > 0.f && level == 0;
    for (int iter = 0; iter < s.iters[level]; ++iter) {
      double D = icp_depth_sums(s, level, deal, P, icp_stage, at);
      if (writes) part[0][term] = D;
      if (photo) {
        D = icp_color_sums(s, deal, P, icp_stage);
        if (writes) part[1][term] = D;
      }
      cluster.sync();  // every block's sums are visible to block 0
      if (rank == 0 && threadIdx.x < 64) {
        if (threadIdx.x < kIcpTerms) {
          // the blocks' sums in rank order; the photometric normal equations and residual
          // enter weighted, the count stays the depth count
          double a = 0.0, c = 0.0;
          for (int r = 0; r < C; ++r) {
            const double* pr = cluster.map_shared_rank(&part[0][0], r);
            a += pr[threadIdx.x];
            if (photo) c += pr[32 + threadIdx.x];
          }
          if (photo && threadIdx.x < kIcpTerms - 1) a += (double)s.photo_w * c;
          sums[threadIdx.x] = a;
        }
        icp_step_sync();
        if (threadIdx.x == 0) lm.icp_iters[level] += 1u;
        icp_host_step(&lm, hw, sums, iter, s.icp_min_count[level]);
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
// another).  Every iteration a block leaves its sums in the session's part of `work` and counts
// itself in; when all have, every block adds all the sums, in the same order, and runs the LM
// step on its own copy of the state, so nothing has to be sent back.  A wait that runs out (it
// cannot with all blocks resident) marks the workspace and loses the frame, as every later launch
// on the workspace does at once.
//
// What bounds it is latency: an iteration is a pass of a few us, a trip through L2 and the LM
// step.  A cluster is at most 16 SMs, on which a pass of a colour-tracked 640 x 480 level takes
// 120 us; a launch an iteration costs 2 us even after the level has ended (a level that starts
// close to its end runs one iteration of the ten).  At 640 x 480 a depth iteration takes 12 us
// (pass 3.3, waiting 1.0, sums 1.5, LM step 3.9; 7 us at the coarser levels) and a photometric
// one 20.
template <bool COLOR>
__global__ void __launch_bounds__(COLOR ? 512 : 1024, 1)
    k_icp_wide(const SessionDesc* __restrict__ descs, int fam, IcpWide* __restrict__ work, const TrackOut out) {
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
  __shared__ int state;  // -1: the wait ran out
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (int)(blockDim.x >> 5), B = (int)gridDim.x;
  lm_copy(&lm, ts);  // (written again only when every block has counted itself in for the last time)
  icp_pose_rows(P.prev, ts->xf.R_inv, ts->xf.t);
  icp_pose_rows(P.cur, ts->R, ts->t);
  if (threadIdx.x == 0) state = *(volatile unsigned*)&f.stalled ? -1 : 0;
  __syncthreads();
  if (lm.status != 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) track_end(s, out);
    return;
  }
  // runs of a warp, dealt over the blocks first
  const IcpDeal deal{32, lane, 1, warp * B + (int)blockIdx.x, warps * B};
  const int term = icp_my_term(), at = icp_term_at(term), src = (int)(threadIdx.x & (warps - 1));
  unsigned turn = 0;  // iterations of this launch
  bool go = state == 0;
  for (int level = s.levels - 1; level >= 0 && go; --level) {
    const bool photo = COLOR && s.photo_w > 0.f && level == 0;
    for (int iter = 0; iter < s.iters[level]; ++iter) {
      // (two sets of sums in turn: a block may be one iteration ahead of one that still reads)
      double(*const part)[64] = f.part[turn & 1];
      const double D = icp_depth_sums(s, level, deal, P, icp_stage, at);
      if (term < kIcpTerms && src == 0) part[blockIdx.x][term] = D;
      if (photo) {
        const double E = icp_color_sums(s, deal, P, icp_stage);
        if (term < kIcpTerms && src == 0) part[blockIdx.x][32 + term] = E;
      }
      __syncthreads();
      ++turn;
      if (threadIdx.x == 0) {
        unsigned e;
        int polls = 0;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&f.arrived) : "memory");
        do {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(e) : "l"(&f.arrived) : "memory");
        } while (e < turn * (unsigned)B && ++polls < kIcpPolls);
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
      // the blocks' sums: warp w adds the terms (a lane each) of blocks w, w + warps, ..., then
      // the warps' sums are added pairwise
      double a = 0.0, c = 0.0;
      for (int b0 = warp; b0 < B; b0 += 5 * warps) {
        double u[5], v[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const int b = b0 + k * warps;
          u[k] = b < B ? __ldcg(&part[b][lane]) : 0.0;
          v[k] = COLOR && photo && b < B ? __ldcg(&part[b][32 + lane]) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < 5; ++k) a += u[k], c += v[k];
      }
      double* const w = reinterpret_cast<double*>(icp_stage);
      w[33 * warp + lane] = a;
      if (COLOR) w[33 * (warps + warp) + lane] = c;
      __syncthreads();
      a = icp_group_sum(w[33 * src + term]);
      if (COLOR) c = icp_group_sum(w[33 * (warps + src) + term]);
      // the photometric normal equations and residual enter weighted, the count stays the depth
      // count
      if (src == 0) sums[term] = photo && term < kIcpTerms - 1 ? a + (double)s.photo_w * c : a;
      if (threadIdx.x == 0) lm.icp_iters[level] += 1u;
      __syncthreads();
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
    if (threadIdx.x == 0 && state != 0) lm.status = 3;
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
template __global__ void k_icp_wide<false>(const SessionDesc*, int, IcpWide*, const TrackOut);
template __global__ void k_icp_wide<true>(const SessionDesc*, int, IcpWide*, const TrackOut);

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
