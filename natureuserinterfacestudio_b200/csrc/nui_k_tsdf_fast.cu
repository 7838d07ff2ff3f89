// Dense TSDF integration in tolerance mode: the FP16 serving formats (NUI_TSDF_F16_U8,
// NUI_TSDF_F16_F16).  Same update as integrateTsdfVolumeKernel (tsdfVolume.cl:31-190) --
// project the voxel centre with R_inv, round to a pixel, sdf = ray depth - |voxel - camera|,
// update when sdf >= -trunc with tsdf = min(1, sdf / trunc), running average capped at
// weight 128, colour averaged inside the band -- evaluated with each voxel's position
// computed directly (fused multiply-adds, approximate reciprocal and square root) instead of
// the reference's incremental z sums.  Results agree with the reference within the TSDF
// tolerance (1e-3 truncation units, well above the half-precision quantum), not bit for bit;
// the int16 and FP32 formats keep the exact kernel (nui_k_tsdf.cu).  This file is compiled
// with contraction on.
//
// Work decomposition: the volume is cut into tiles of 32 (x) x 8 (y) x 8 (z) voxels.
// k_integrate_cull tests every tile on one thread: tiles entirely behind the camera,
// projecting outside the image, or farther from the camera than the largest ray depth of
// the pixel tiles they project to plus the truncation are dropped without a memory access;
// the kept ones are appended to the session's tile list.  k_integrate_fast deals the listed
// tiles round robin to its blocks (the kept tiles cluster in the frustum, so a fixed
// tile-to-block map would leave most blocks idle), lane = x: a tile's voxel rows are brought
// into shared memory by asynchronous copies, its depth pixels into registers, then updated
// from there (only updated voxels are written back), and the 8^3 bricks of the tile that had
// an update are re-classified from the same shared copy -- the brick summary the exact path
// leaves to k_brick_summary.
#include <type_traits>

#include "nui_device.cuh"

namespace nui {

// Tile culling, one thread per tile: a tile can hold an updated voxel only if part of it
// is in front of the camera, projects into the image, and is no farther from the camera
// than the largest ray depth of the pixel tiles it projects to plus the truncation.  The
// corners' camera coordinates follow from one corner and the tile's three edge vectors.
template <int FMT>
__global__ void __launch_bounds__(256) k_integrate_cull(const SessionDesc* __restrict__ descs) {
  const SessionDesc& s = descs[blockIdx.y];
  if (s.kind < 0 || s.fmt != FMT || !s.ts->integrate) return;
  const int rx = s.res[0], ry = s.res[1], rz = s.res[2];
  const int ntx = (rx + 31) >> 5, nty = (ry + 7) >> 3, ntz = (rz + 7) >> 3;
  const int tile = blockIdx.x * blockDim.x + threadIdx.x;
  if (tile >= ntx * nty * ntz) return;
  const DevXform& m = s.ts->xf;
  const float* Ri = m.R_inv;
  const float c0 = s.cell[0], c1 = s.cell[1], c2 = s.cell[2];
  const int x0 = (tile % ntx) << 5, y0 = ((tile / ntx) % nty) << 3, z0 = (tile / (ntx * nty)) << 3;
  const int xn = min(32, rx - x0), yn = min(8, ry - y0), zn = min(8, rz - z0);
  const float gx = ((float)(x0 - rx / 2) + 0.5f) * c0 - m.t[0];
  const float gy = ((float)(y0 - ry / 2) + 0.5f) * c1 - m.t[1];
  const float gz = ((float)z0 + 0.5f) * c2 - m.t[2];
  const float ex = (float)(xn - 1) * c0, ey = (float)(yn - 1) * c1, ez = (float)(zn - 1) * c2;
  const float3 v0 = f3(Ri[0] * gx + Ri[1] * gy + Ri[2] * gz, Ri[3] * gx + Ri[4] * gy + Ri[5] * gz,
                       Ri[6] * gx + Ri[7] * gy + Ri[8] * gz);
  const float3 dx = f3(Ri[0] * ex, Ri[3] * ex, Ri[6] * ex), dy = f3(Ri[1] * ey, Ri[4] * ey, Ri[7] * ey),
               dz = f3(Ri[2] * ez, Ri[5] * ez, Ri[8] * ez);
  const float fx = s.cam.fx, fy = s.cam.fy, ccx = s.cam.cx, ccy = s.cam.cy;
  const float fW = (float)s.W, fH = (float)s.H;
  float u0 = 3.4e38f, u1 = -3.4e38f, w0 = 3.4e38f, w1 = -3.4e38f;
  int front = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float3 v = v0;
    if (k & 1) v = add3(v, dx);
    if (k & 2) v = add3(v, dy);
    if (k & 4) v = add3(v, dz);
    if (v.z > 1e-6f) {
      ++front;
      const float iz = __fdividef(1.f, v.z);
      const float u = fx * v.x * iz + ccx, w = fy * v.y * iz + ccy;
      u0 = fminf(u0, u);
      u1 = fmaxf(u1, u);
      w0 = fminf(w0, w);
      w1 = fmaxf(w1, w);
    }
  }
  bool keep = front > 0;
  if (keep) {
    if (front < 8) {  // straddles the camera plane: the footprint is unbounded
      u0 = 0.f, u1 = fW - 1.f, w0 = 0.f, w1 = fH - 1.f;
    } else {
      u0 = fmaxf(u0 - 1.f, 0.f), u1 = fminf(u1 + 1.f, fW - 1.f);
      w0 = fmaxf(w0 - 1.f, 0.f), w1 = fminf(w1 + 1.f, fH - 1.f);
    }
    keep = u0 <= u1 && w0 <= w1;
  }
  if (keep) {
    // largest ray depth over the pixel tiles of the footprint (the frame's largest when the
    // footprint spans more than 64 of them); 0 = no valid depth there
    const int ptx = (s.W + kTile - 1) / kTile;
    const int a0 = (int)u0 / kTile, a1 = (int)u1 / kTile, b0 = (int)w0 / kTile, b1 = (int)w1 / kTile;
    float mx = 0.f;
    if ((a1 - a0 + 1) * (b1 - b0 + 1) <= 64) {
      for (int b = b0; b <= b1; ++b)
        for (int a = a0; a <= a1; ++a) mx = fmaxf(mx, __ldg(s.tile_max + b * ptx + a));
    } else {
      mx = __int_as_float(s.ts->dmax_bits);
    }
    // nearest distance from the camera to the tile's box of voxel centres
    const float bx = fmaxf(fmaxf(gx, -(gx + ex)), 0.f), by = fmaxf(fmaxf(gy, -(gy + ey)), 0.f),
                bz = fmaxf(fmaxf(gz, -(gz + ez)), 0.f);
    const float dmin = sqrtf(bx * bx + by * by + bz * bz);
    keep = mx > 0.f && !(dmin > mx + s.trunc + 1e-3f * (1.f + dmin));
  }
  // append the kept tile to the session's list (one atomic per warp)
  const unsigned act = __activemask(), kept = __ballot_sync(act, keep);
  const int lane = threadIdx.x & 31;
  unsigned base = 0;
  if (kept && lane == __ffs(act) - 1) base = atomicAdd(&s.ts->fast_count, (unsigned)__popc(kept));
  base = __shfl_sync(act, base, __ffs(act) - 1);
  if (keep) s.fast_tiles[base + __popc(kept & ((1u << lane) - 1u))] = (unsigned)tile;
}

// Asynchronous copies global -> shared (cp.async): the data lands in shared memory without
// passing through registers, so a lane can have a whole tile's requests in flight.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The roundings of the update are written out (a fused multiply-add or separate operations), so
// that they do not hang on how the compiler contracts around the loops: a voxel's result is the
// same wherever it is computed, here and in fast_color.
__device__ __forceinline__ float3 fast_camera(const float (&R)[9], float gx, float gy, float gz) {
  auto row = [&](float a, float b, float c) { return __fmaf_rn(c, gz, __fmaf_rn(a, gx, __fmul_rn(b, gy))); };
  return f3(row(R[0], R[1], R[2]), row(R[3], R[4], R[5]), row(R[6], R[7], R[8]));
}
// camera step of one y row
__device__ __forceinline__ float3 fast_step(const float (&R)[9], float c1) {
  return f3(__fmul_rn(R[1], c1), __fmul_rn(R[4], c1), __fmul_rn(R[7], c1));
}
__device__ __forceinline__ float3 fast_next(float3 v, float3 e) {
  return f3(__fadd_rn(v.x, e.x), __fadd_rn(v.y, e.y), __fadd_rn(v.z, e.z));
}
// the pixel coordinate; exact ties round up, as OpenCL's round(): they are frequent (pixel
// centres and voxel centres sit on rational grids), and half-to-even would split them
__device__ __forceinline__ int fast_pixel(float f, float v, float iz, float c) {
  return round_half_up(__fmaf_rn(__fmul_rn(f, v), iz, c));
}
// centre of voxel i on an axis, relative to the camera
__device__ __forceinline__ float fast_centre(int i, float c, float t) { return __fmaf_rn((float)i + 0.5f, c, -t); }

// Running colour average of the voxel of row yy of the slice at gz, whose pixel is found again
// by the same operations as in the request phase: the reference's arithmetic exactly (no product
// to contract, IEEE division), so that colours agree bit for bit wherever the same voxels are
// updated.
__device__ __noinline__ void fast_color(const SessionDesc& s, unsigned vi, float gx, float gy0, float gz, int yy) {
  const float(&Ri)[9] = s.ts->xf.R_inv;
  const float3 ey = fast_step(Ri, s.cell[1]);
  float3 v = fast_camera(Ri, gx, gy0, gz);
  for (int k = 0; k < yy; ++k) v = fast_next(v, ey);
  const float iz = __fdividef(1.f, v.z);
  const int px = fast_pixel(s.cam.fx, v.x, iz, s.cam.cx), py = fast_pixel(s.cam.fy, v.y, iz, s.cam.cy);
  if ((unsigned)px >= (unsigned)s.W || (unsigned)py >= (unsigned)s.H) return;
  const uchar4 nc = reinterpret_cast<const uchar4*>(s.bgra)[py * s.W + px];
  if (nc.w == 0) return;
  const uchar4 vc = s.cvol[vi];
  const float den = (float)vc.w + 1.f;
  uchar4 o;
  o.x = (unsigned char)fminf(fmaxf(((float)(vc.x * vc.w) + (float)nc.x) / den, 0.f), 255.f);
  o.y = (unsigned char)fminf(fmaxf(((float)(vc.y * vc.w) + (float)nc.y) / den, 0.f), 255.f);
  o.z = (unsigned char)fminf(fmaxf(((float)(vc.z * vc.w) + (float)nc.z) / den, 0.f), 255.f);
  o.w = min((unsigned char)s.max_cw, (unsigned char)(vc.w + 1));
  s.cvol[vi] = o;
}

// A warp's share of a tile in shared memory: kFastRows rows of 32 voxels.
constexpr int kFastSlices = 8 / kFastWarps;    // z slices of a tile a warp takes
constexpr int kFastRows = 8 * kFastSlices;
template <int FMT>
struct FastRows {
  __align__(16) __half fh[FMT == 2 ? kFastRows : 1][32];   // F16_U8: tsdf
  __align__(16) uint8_t wb[FMT == 2 ? kFastRows : 1][32];  // F16_U8: weight
  __align__(16) __half2 f2[FMT == 2 ? 1 : kFastRows][32];  // F16_F16: (tsdf, weight)
  __device__ __forceinline__ void get(int r, int lane, float& F, int& W) const {
    if (FMT == 2) {
      F = __half2float(fh[r][lane]);
      W = wb[r][lane];
    } else {
      const __half2 v = f2[r][lane];
      F = __low2float(v);
      W = (int)__high2float(v);
    }
  }
};

// The tiles the cull listed, dealt round robin to the blocks, two z slices of a tile a warp,
// lane = x.  Per tile:
//  1. the warp's rows of voxels are requested as 16-byte pieces into shared memory (4 + 2
//     pieces a row for FP16 + u8, 8 for FP16 + FP16), and each lane projects its sixteen
//     voxels and loads the depths they land on (NaN when on none) -- all in flight at once;
//  2. the update: sd = depth - |voxel - camera|, the running average, stores of the updated
//     voxels (and their new values into the shared copy);
//  3. the 8^3 bricks of the tile that had an update are re-classified from the shared copies,
//     the warps' findings joined.
// Rows that are not whole (a tile past the volume's x end) or not 16-byte aligned (x sizes
// not a multiple of 16) are loaded lane by lane instead.
//
// A tile is a chain of a projection, a load and an update a row.  One warp that took all 64
// rows of a tile through shared memory (16 KB, 121 registers, 12 warps an SM) spent most issue
// slots waiting (44 % used), and a single session's launch was one tile's latency: 39 sessions
// 852 -> 518 us, one 384^3 session 116 -> 44 us.
template <int FMT>
__global__ void __launch_bounds__(32 * kFastWarps, 5) k_integrate_fast(const SessionDesc* __restrict__ descs) {
  const SessionDesc& s = descs[blockIdx.y];
  if (s.kind < 0 || s.fmt != FMT || !s.ts->integrate) return;
  __shared__ FastRows<FMT> rows[kFastWarps];
  __shared__ unsigned found[4][kFastWarps];  // per warp: updated, weighted, unweighted, nonpositive columns
  const int rx = s.res[0], ry = s.res[1], rz = s.res[2];
  const int ntx = (rx + 31) >> 5, nty = (ry + 7) >> 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FastRows<FMT>& sm = rows[warp];
  const DevXform& m = s.ts->xf;
  float Ri[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) Ri[k] = m.R_inv[k];
  const float t0 = m.t[0], t1 = m.t[1], t2 = m.t[2];
  const float c0 = s.cell[0], c1 = s.cell[1], c2 = s.cell[2];
  const float fx = s.cam.fx, fy = s.cam.fy, ccx = s.cam.cx, ccy = s.cam.cy;
  const int W = s.W, H = s.H;
  const float trunc = s.trunc, tinv = 1.f / trunc;
  const float* __restrict__ depth = s.dscaled;
  const unsigned slice = (unsigned)rx * (unsigned)ry;
  const int hx = rx / 2, hy = ry / 2;
  const bool color = s.cvol && s.bgra;
  // whole rows start 16-byte aligned in every plane when the x size is a multiple of 16
  const bool aligned = (rx & 15) == 0 && ((reinterpret_cast<uintptr_t>(s.vol) | reinterpret_cast<uintptr_t>(s.wvol)) & 15) == 0;
  unsigned int touched_total = 0, bricks = 0;

  const unsigned count = *(volatile const unsigned*)&s.ts->fast_count;
  for (unsigned li = blockIdx.x; li < count; li += gridDim.x) {
    const int tile = (int)__ldg(s.fast_tiles + li);
    const int x0 = (tile % ntx) << 5, y0 = ((tile / ntx) % nty) << 3;
    const int z0 = ((tile / (ntx * nty)) << 3) + warp * kFastSlices;  // the warp's first slice
    const int xn = min(32, rx - x0), yn = min(8, ry - y0), zn = max(0, min(kFastSlices, rz - z0));
    const int x = x0 + lane;
    const bool xin = lane < xn;
    const bool whole = aligned && xn == 32;
    const float gx = fast_centre(x - hx, c0, t0), gy0 = fast_centre(y0 - hy, c1, t1);
    const float3 ey = fast_step(Ri, c1);

    // FULL: the warp's rows are all inside the volume and aligned
    unsigned int touched = 0;  // voxels this lane updated in the tile
    auto update = [&](auto full) {
      constexpr bool FULL = decltype(full)::value;
      // ---- 1. requests: the rows' voxels and depth pixels
      const unsigned v0 = (unsigned)x + (unsigned)rx * (unsigned)y0 + slice * (unsigned)z0;
      if (FULL || whole) {
        // the rows' 16-byte pieces dealt over the lanes, no lane idle and no branch per row
        constexpr int kPieces = FMT == 2 ? 6 : 8;
#pragma unroll
        for (int i = 0; i < kFastRows * kPieces / 32; ++i) {
          const int j = 32 * i + lane, r = j / kPieces, piece = j - r * kPieces, yy = r & 7, zz = r >> 3;
          if (!FULL && (yy >= yn || zz >= zn)) continue;
          const unsigned rb = (unsigned)x0 + (unsigned)rx * (unsigned)(y0 + yy) + slice * (unsigned)(z0 + zz);
          if (FMT == 2) {
            if (piece < 4) cp_async16(&sm.fh[r][piece * 8], reinterpret_cast<const __half*>(s.vol) + rb + piece * 8);
            else cp_async16(&sm.wb[r][(piece - 4) * 16], s.wvol + rb + (piece - 4) * 16);
          } else {
            cp_async16(&sm.f2[r][piece * 4], reinterpret_cast<const __half2*>(s.vol) + rb + piece * 4);
          }
        }
      }
      float dep[kFastRows];
#pragma unroll
      for (int zz = 0; zz < kFastSlices; ++zz) {
        float3 v = fast_camera(Ri, gx, gy0, fast_centre(z0 + zz, c2, t2));
#pragma unroll
        for (int yy = 0; yy < 8; ++yy) {
          const int r = zz * 8 + yy;
          dep[r] = __int_as_float(0x7fffffff);
          if (FULL || (xin && yy < yn && zz < zn)) {
            if (v.z > 0.f) {
              const float iz = __fdividef(1.f, v.z);
              const int px = fast_pixel(fx, v.x, iz, ccx), py = fast_pixel(fy, v.y, iz, ccy);
              if ((unsigned)px < (unsigned)W && (unsigned)py < (unsigned)H) dep[r] = __ldg(depth + py * W + px);
            }
            if (!FULL && !whole) {
              const unsigned vi = v0 + (unsigned)rx * yy + slice * zz;
              if (FMT == 2) {
                sm.fh[r][lane] = reinterpret_cast<const __half*>(s.vol)[vi];
                sm.wb[r][lane] = s.wvol[vi];
              } else {
                sm.f2[r][lane] = reinterpret_cast<const __half2*>(s.vol)[vi];
              }
            }
          }
          v = fast_next(v, ey);
        }
      }
      cp_async_wait_all();
      __syncwarp();

      // ---- 2. the update, from shared memory
      const float gx2 = __fmul_rn(gx, gx);
#pragma unroll
      for (int zz = 0; zz < kFastSlices; ++zz) {
        const float gz = fast_centre(z0 + zz, c2, t2), gz2 = __fmul_rn(gz, gz);
#pragma unroll
        for (int yy = 0; yy < 8; ++yy) {
          const int r = zz * 8 + yy;
          const float gy = __fmaf_rn((float)yy, c1, gy0);
          const float r2 = __fadd_rn(__fmaf_rn(gy, gy, gx2), gz2);
          const float sd = __fmaf_rn(-r2, rsqrtf(r2), dep[r]);
          if (!(sd >= -trunc)) continue;  // also a voxel without a depth (NaN), or outside the volume
          float F;
          int Wt;
          sm.get(r, lane, F, Wt);
          const unsigned vi = v0 + (unsigned)rx * yy + slice * zz;
          const float tsdf = fminf(1.0f, sd * tinv);
          const float tn = __fdividef(__fmaf_rn(F, (float)Wt, tsdf), (float)(Wt + 1));
          const int wn = min(Wt + 1, 128);
          if (FMT == 2) {
            const __half h = __float2half_rn(tn);
            reinterpret_cast<__half*>(s.vol)[vi] = h;
            s.wvol[vi] = (uint8_t)wn;
            sm.fh[r][lane] = h;
            sm.wb[r][lane] = (uint8_t)wn;
          } else {
            const __half2 h = __floats2half2_rn(tn, (float)wn);
            reinterpret_cast<__half2*>(s.vol)[vi] = h;
            sm.f2[r][lane] = h;
          }
          touched += 1u;
          if (color && fabsf(sd) < trunc) fast_color(s, vi, gx, gy0, gz, yy);
        }
      }
    };
    if (whole && yn == 8 && zn == kFastSlices) update(std::true_type());
    else update(std::false_type());
    touched_total += touched;
    // ---- 3. classification of the bricks (lanes 8b .. 8b+7) that had an update, from the
    // shared copies (which hold the values just written)
    const unsigned upd = __ballot_sync(0xffffffffu, touched != 0u);
    if (lane == 0) found[0][warp] = upd;
    __syncthreads();
    unsigned any = 0u;
#pragma unroll
    for (int w = 0; w < kFastWarps; ++w) any |= found[0][w];
    if (any != 0u && s.occ) {
      const bool mine = (any >> (lane & ~7)) & 0xffu;
      bool weighted = false, unweighted = false, nonpos = false;
      if (mine && xin) {
#pragma unroll
        for (int zz = 0; zz < kFastSlices; ++zz)
#pragma unroll
          for (int yy = 0; yy < 8; ++yy) {
            if (zz >= zn || yy >= yn) continue;
            float F;
            int Wt;
            sm.get(zz * 8 + yy, lane, F, Wt);
            weighted |= Wt > 0;
            unweighted |= Wt <= 0;
            nonpos |= Wt > 0 && !(F > 0.f);
          }
      }
      const unsigned bw = __ballot_sync(0xffffffffu, weighted), bu = __ballot_sync(0xffffffffu, unweighted),
                     bn = __ballot_sync(0xffffffffu, nonpos);
      if (lane == 0) found[1][warp] = bw, found[2][warp] = bu, found[3][warp] = bn;
      __syncthreads();
      if (warp == 0 && (lane & 7) == 0 && mine && xin) {
        unsigned b[3] = {0u, 0u, 0u};
#pragma unroll
        for (int w = 0; w < kFastWarps; ++w)
#pragma unroll
          for (int k = 0; k < 3; ++k) b[k] |= found[1 + k][w];
        const unsigned g = 0xffu << lane;
        const uint8_t st = (b[2] & g) ? kBrickMixed : !(b[0] & g) ? kBrickEmpty : (b[1] & g) ? kBrickNoNeg : kBrickPositive;
        s.occ[occ_index(s, x, y0, z0)] = st;
        ++bricks;
      }
    }
    __syncthreads();  // found is written again by the next tile
  }
  const unsigned int t = __reduce_add_sync(0xffffffffu, touched_total);
  const unsigned int b = __reduce_add_sync(0xffffffffu, bricks);
  if (lane == 0 && t) atomicAdd(&s.ts->touched, (unsigned long long)t);
  if (lane == 0 && b) atomicAdd(&s.ts->bricks, (unsigned long long)b);
  // the session's last block to finish empties the list for the next integration (every
  // block has read the count by then)
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&s.ts->fast_done, 1u) == gridDim.x - 1) {
    s.ts->tiles += count;
    s.ts->fast_count = 0u;
    s.ts->fast_done = 0u;
  }
}

template __global__ void k_integrate_cull<2>(const SessionDesc*);
template __global__ void k_integrate_cull<3>(const SessionDesc*);
template __global__ void k_integrate_fast<2>(const SessionDesc*);
template __global__ void k_integrate_fast<3>(const SessionDesc*);

}  // namespace nui
