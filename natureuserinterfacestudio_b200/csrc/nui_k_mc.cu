// Marching cubes over the dense volume (marchingCubeKernel, marchingCube.cl:100-256) with
// deterministic prefix-sum compaction (the role of NuiOpenCLPrefixSum, prefixSum.cl:10-232).
//
// Order: cubes are emitted in the order of the reference's own CPU extraction
// (NuiKinfuOpenCLScene::Volume2Mesh, NuiKinfuOpenCLScene.cpp:823-836): y outermost, then x,
// then z.  A block owns 128 consecutive x of one y row, so its cubes form one contiguous run
// of that order (64 or 32 where that leaves few blocks).
//   k_mc_count  which 32-cube chunks of every column hold triangles (a bit each), and the
//               vertices of every block
//   k_mc_scan   exclusive scan of the block totals (one block, warp-shuffle scan)
//   k_mc_emit   the triangles' cubes of the block listed in order, a thread a cube
// Per cube: skip if any corner has weight <= 0; case bit i = tsdf_i < 0; vertices on the
// table's edges by clamped linear interpolation (vertex_interp, marchingCube.cl:86-91);
// positions ((x + 0.5 - rx/2) c, (-y - 0.5 + ry/2) c, (z + 0.5) c) (getNodeCoo :81-84).
//
// What bounds it is the reading of the volume near the surfaces and the vertices written.  A
// thread that walked its column's cubes one after another, eight corners and eight brick
// states each, waited 255 times for its loads, twice; here a warp takes 32 columns x 8
// slices: the brick states in one round, then nine slices of two rows, all loads in flight, the neighbour columns' corners by shuffle -- two voxels a cube instead
// of eight -- and nothing where no brick holds a voxel behind a surface.  The emission walks
// only the chunks the count marked.
// The whole call into device buffers: 256^3 FP32 (1.2 M vertices) 1.55 ms -> 168 us; 512^3
// FP16 + u8 with colours (4.9 M vertices) 8.2 ms -> 760 us.
#include "nui_device.cuh"
#include "nui_mc_tables.h"

namespace nui {

constexpr int kMcThreads = 256;
__constant__ uint64_t c_tri[256];

cudaError_t mc_upload_tables(cudaStream_t st) {
  return cudaMemcpyToSymbolAsync(c_tri, NUI_MC_TRI_PACKED, sizeof(NUI_MC_TRI_PACKED), 0, cudaMemcpyHostToDevice, st);
}

// Bit 0: the voxel has a weight; bit 1: its tsdf is negative.
template <int FMT>
__device__ __forceinline__ unsigned voxel_class(const SessionDesc& s, size_t i) {
  if (FMT == 0) {
    const short2 v = reinterpret_cast<const short2*>(s.vol)[i];
    return (v.y > 0 ? 1u : 0u) | (v.x < 0 ? 2u : 0u);
  }
  float f;
  int w;
  Voxel<FMT>::load(s, i, f, w);
  return (w > 0 ? 1u : 0u) | (f < 0.f ? 2u : 0u);
}

// The cubes of 32 columns (x0 + lane, y) over slices z .. z + 7 (x0 a multiple of 32, z of 8):
// calls visit(slice, c) on every lane for every slice whose cubes can hold triangles, c the
// case of the lane's cube or -1 (a corner without weight, or no cube there).  A cube with
// triangles has a corner with tsdf < 0, whose brick is mixed (or awaits classification), so
// the slices are passed over without such a brick at or next to them.  All lanes must call it.
template <int FMT, class Visit>
__device__ __forceinline__ void mc_slices(const SessionDesc& s, int x0, int y, int z, Visit visit) {
  const unsigned rx = (unsigned)s.res[0], ry = (unsigned)s.res[1];
  const int rz = s.res[2];
  const int lane = threadIdx.x & 31;
  if (s.occ) {
    const int bx = (s.res[0] + 7) >> 3, by = (s.res[1] + 7) >> 3, bz = (rz + 7) >> 3;
    // 5 x 2 x 2 bricks
    const int r = lane % 10, X = (x0 >> 3) + r % 5, Y = (y + r / 5) >> 3, Z = (z >> 3) + lane / 10;
    uint8_t st = kBrickEmpty;
    if (lane < 20 && X < bx && Y < by && Z < bz) st = __ldg(s.occ + X + bx * (Y + by * Z));
    if (!__any_sync(0xffffffffu, st == kBrickMixed || st == kBrickDirty)) return;
  }
  const unsigned x = (unsigned)(x0 + lane), slice = rx * ry;
  const bool in = x < rx, cube = x + 1 < rx;
  // nine slices of the two rows; lanes 0..17 also read the column after the warp's last one
  const unsigned i0 = x + rx * (unsigned)y + slice * (unsigned)z;
  unsigned p[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    p[k] = 0u;
    if (in && z + k < rz) p[k] = voxel_class<FMT>(s, i0 + slice * k) | voxel_class<FMT>(s, i0 + slice * k + rx) << 2;
  }
  unsigned e = 0u;
  if (lane < 18 && (unsigned)x0 + 32 < rx && z + (lane >> 1) < rz)
    e = voxel_class<FMT>(s, (unsigned)x0 + 32 + rx * (unsigned)(y + (lane & 1)) + slice * (unsigned)(z + (lane >> 1)));
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    unsigned t = __shfl_down_sync(0xffffffffu, p[k], 1);
    const unsigned e0 = __shfl_sync(0xffffffffu, e, 2 * k), e1 = __shfl_sync(0xffffffffu, e, 2 * k + 1);
    if (lane == 31) t = e0 | e1 << 2;
    p[k] |= t << 4;
  }
  // a slice's corners: bits 0, 2, 4, 6 weights and 1, 3, 5, 7 signs of (x, y), (x, y + 1),
  // (x + 1, y), (x + 1, y + 1)
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (z + k >= rz - 1) break;
    auto bits = [](unsigned q) { return (q >> 1 & 1u) | (q >> 4 & 2u) | (q >> 5 & 4u) | (q & 8u); };
    const bool ok = cube && (p[k] & p[k + 1] & 0x55u) == 0x55u;
    visit(z + k, ok ? (int)(bits(p[k]) | bits(p[k + 1]) << 4) : -1);
  }
}

// cols: columns of one y row a block takes (32, 64 or 128)
template <int FMT>
__global__ void __launch_bounds__(kMcThreads) k_mc_count(const SessionDesc* __restrict__ descs, int cols,
                                                         unsigned int* colchunks, unsigned long long* blocktot,
                                                         uint8_t* cases) {
  const SessionDesc& s = descs[0];
  const int rx = s.res[0], rz = s.res[2];
  const int tilesX = (rx - 1 + cols - 1) / cols;
  const int y = blockIdx.x / tilesX, xb = (blockIdx.x % tilesX) * cols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, steps = (rz - 1 + 7) / 8;
  __shared__ uint8_t nverts[256];
  __shared__ unsigned chunks[128];
  __shared__ unsigned wsum[kMcThreads / 32];
  nverts[threadIdx.x] = (uint8_t)(3 * (int)(c_tri[threadIdx.x] >> 60));
  if (threadIdx.x < 128) chunks[threadIdx.x] = 0u;
  __syncthreads();
  unsigned n = 0;
  for (int task = warp, tiles = cols >> 5; task < tiles * steps; task += kMcThreads / 32) {
    const int step = task / tiles, q = task - step * tiles, x0 = xb + 32 * q;
    if (x0 >= rx - 1) continue;
    uint8_t* const out = cases ? cases + ((size_t)y * (rx - 1) + x0 + lane) * (size_t)(rz - 1) : nullptr;
    if (out && x0 + lane < rx - 1)
      for (int z = 8 * step; z < min(8 * step + 8, rz - 1); ++z) out[z] = 0;
    unsigned m = 0;
    mc_slices<FMT>(s, x0, y, 8 * step, [&](int z, int c) {
      if (c > 0) {
        m += nverts[c];
        if (out) out[z] = (uint8_t)c;
      }
    });
    n += m;
    if (m) atomicOr(&chunks[32 * q + lane], 1u << (step >> 2));
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) wsum[warp] = n;
  __syncthreads();
  if ((int)threadIdx.x < cols && xb + (int)threadIdx.x < rx - 1)
    colchunks[(size_t)y * (rx - 1) + xb + threadIdx.x] = chunks[threadIdx.x];
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int i = 0; i < kMcThreads / 32; ++i) t += wsum[i];
    blocktot[blockIdx.x] = t;
  }
}

// Exclusive scan of n block totals in place, total in out[n]; one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_mc_scan(unsigned long long* tot, int n) {
  __shared__ unsigned long long warp_tot[32];
  __shared__ unsigned long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int base = 0; base < n; base += 1024) {
    const int i = base + threadIdx.x;
    unsigned long long v = i < n ? tot[i] : 0ull;
    unsigned long long inc = v;
    for (int off = 1; off < 32; off <<= 1) {
      unsigned long long o = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += o;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      unsigned long long w = warp_tot[lane], wi = w;
      for (int off = 1; off < 32; off <<= 1) {
        unsigned long long o = __shfl_up_sync(0xffffffffu, wi, off);
        if (lane >= off) wi += o;
      }
      warp_tot[lane] = wi - w;  // exclusive prefix of the warp totals
    }
    __syncthreads();
    const unsigned long long excl = carry + warp_tot[warp] + inc - v;
    __syncthreads();
    if (i < n) tot[i] = excl;
    if (threadIdx.x == 1023) carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) tot[n] = carry;
}

// Exclusive scan of v over the block's threads in order; *total (shared) receives the sum.
__device__ __forceinline__ unsigned mc_block_scan(unsigned v, unsigned* wsum, unsigned& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned inc = v;
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned o = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += o;
  }
  __syncthreads();  // the previous call's sums are no longer read
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  unsigned before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kMcThreads / 32; ++w) {
    before += w < warp ? wsum[w] : 0u;
    total += wsum[w];
  }
  return before + inc - v;
}

// Three passes over the block's columns: the triangles' cubes of the marked chunks as bit
// masks; their counts scanned in column-major order (the output's); then 256 cubes at a time,
// a thread a cube for its corners, then a thread a vertex, so that the vertices are written in
// whole lines and cubes with many triangles do not hold up the others.
template <int FMT>
__global__ void __launch_bounds__(kMcThreads) k_mc_emit(const SessionDesc* __restrict__ descs, int cols,
                                                        const unsigned int* colchunks,
                                                        const unsigned long long* blockoff, float* pos,
                                                        float* col, unsigned long long cap) {
  const SessionDesc& s = descs[0];
  const int rx = s.res[0], ry = s.res[1], rz = s.res[2];
  const int tilesX = (rx - 1 + cols - 1) / cols;
  const int y = blockIdx.x / tilesX, xb = (blockIdx.x % tilesX) * cols;
  unsigned long long base = blockoff[blockIdx.x];
  if (base == blockoff[blockIdx.x + 1] || base >= cap) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nch = (rz - 1 + 31) / 32, steps = (rz - 1 + 7) / 8;
  const int entries = cols * nch;  // a column's chunks, column after column
  extern __shared__ unsigned mc_smem[];
  unsigned* const mask = mc_smem;              // an entry's cubes with triangles
  unsigned* const before = mc_smem + entries;  // cubes of the entries before it
  __shared__ unsigned wsum[kMcThreads / 32];
  __shared__ float f8[8][kMcThreads];  // the batch's cubes: corner values,
  __shared__ uint64_t words[kMcThreads];  // case words,
  __shared__ unsigned at[kMcThreads];     // column and slice,
  __shared__ unsigned off[kMcThreads];    // first vertex in the batch
  for (int k = threadIdx.x; k < entries; k += kMcThreads) mask[k] = 0u;
  __syncthreads();
  for (int task = warp, tiles = cols >> 5; task < tiles * steps; task += kMcThreads / 32) {
    const int step = task / tiles, q = task - step * tiles, x0 = xb + 32 * q, x = x0 + lane, ch = step >> 2;
    const bool mine = x < rx - 1 && (colchunks[(size_t)y * (rx - 1) + x] >> ch & 1u);
    if (!__any_sync(0xffffffffu, mine)) continue;
    unsigned m = 0;
    mc_slices<FMT>(s, x0, y, 8 * step, [&](int z, int c) {
      if (c > 0 && c < 255) m |= 1u << (z & 31);
    });
    if (m) atomicOr(&mask[(32 * q + lane) * nch + ch], m);
  }
  __syncthreads();
  const int per = (entries + kMcThreads - 1) / kMcThreads;
  unsigned cnt = 0, cubes;
  for (int k = 0; k < per; ++k) {
    const int e = threadIdx.x * per + k;
    if (e < entries) cnt += __popc(mask[e]);
  }
  unsigned run = mc_block_scan(cnt, wsum, cubes);
  for (int k = 0; k < per; ++k) {
    const int e = threadIdx.x * per + k;
    if (e >= entries) break;
    before[e] = run;
    run += __popc(mask[e]);
  }
  __syncthreads();
  const float c0 = s.cell[0], c1 = s.cell[1], c2 = s.cell[2];
  const float hx = (float)(rx >> 1), hy = (float)(ry >> 1);
  const unsigned slice = (unsigned)rx * (unsigned)ry;
  const uchar4* const cvol = s.cvol;
  // corner k of a cube at offset (kCX >> k & 1, kCY >> k & 1, kCZ >> k & 1); edge e from corner
  // e & 7 to the nibble of kE1
  constexpr unsigned kCX = 0x66u, kCY = 0xCCu, kCZ = 0xF0u;
  constexpr uint64_t kE1 = 0x765447650321ull;
  for (unsigned i0 = 0; i0 < cubes && base < cap; i0 += kMcThreads) {
    const unsigned i = i0 + threadIdx.x, live = min(cubes - i0, (unsigned)kMcThreads);
    unsigned nv = 0;
    if (i < cubes) {
      int lo = 0, hi = entries;  // the last entry with before <= i holds cube i
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (before[mid] <= i) lo = mid;
        else hi = mid;
      }
      unsigned m = mask[lo];
      for (unsigned r = i - before[lo]; r > 0; --r) m &= m - 1u;
      const int cl = lo / nch, z = 32 * (lo - cl * nch) + __ffs(m) - 1;
      const unsigned v0 = (unsigned)(xb + cl) + (unsigned)rx * (unsigned)y + slice * (unsigned)z;
      int c = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float f;
        int w;
        Voxel<FMT>::load(s, v0 + (kCX >> k & 1u) + (unsigned)rx * (kCY >> k & 1u) + slice * (kCZ >> k & 1u), f, w);
        f8[k][threadIdx.x] = f;
        c += (f < 0) ? (1 << k) : 0;
      }
      words[threadIdx.x] = c_tri[c];
      at[threadIdx.x] = (unsigned)cl << 16 | (unsigned)z;
      nv = 3u * (unsigned)(c_tri[c] >> 60);
    }
    unsigned batch;
    off[threadIdx.x] = mc_block_scan(nv, wsum, batch);
    __syncthreads();
    for (unsigned j = threadIdx.x; j < batch && base + j < cap; j += kMcThreads) {
      unsigned q = 0;  // the last cube with off <= j
#pragma unroll
      for (unsigned h = kMcThreads / 2; h > 0; h >>= 1)
        if (q + h < live && off[q + h] <= j) q += h;
      const unsigned e = (unsigned)(words[q] >> (4 * (j - off[q]))) & 0xFu;
      const unsigned a = e & 7u, b = (unsigned)(kE1 >> (4 * e)) & 0xFu;
      const int x = xb + (int)(at[q] >> 16), z = (int)(at[q] & 0xffffu);
      const int ax = x + (int)(kCX >> a & 1u), ay = y + (int)(kCY >> a & 1u), az = z + (int)(kCZ >> a & 1u);
      const int bx = x + (int)(kCX >> b & 1u), by = y + (int)(kCY >> b & 1u), bz = z + (int)(kCZ >> b & 1u);
      const float3 pa = f3(((float)ax + 0.5f - hx) * c0, (-(float)ay - 0.5f + hy) * c1, ((float)az + 0.5f) * c2);
      const float3 pb = f3(((float)bx + 0.5f - hx) * c0, (-(float)by - 0.5f + hy) * c1, ((float)bz + 0.5f) * c2);
      const float fa = f8[a][q], fb = f8[b][q];
      float t = (0.f - fa) / (fb - fa + 1e-15f);
      t = fminf(fmaxf(t, 0.0f), 1.0f);
      const unsigned long long out = base + j;
      if (pos) {
        pos[3 * out] = pa.x + (pb.x - pa.x) * t;
        pos[3 * out + 1] = pa.y + (pb.y - pa.y) * t;
        pos[3 * out + 2] = pa.z + (pb.z - pa.z) * t;
      }
      if (col) {
        float4 cc = make_float4(0.f, 0.f, 0.f, 1.f);
        if (cvol) {
          const bool near_a = fabsf(fa) < fabsf(fb);
          const unsigned vi = near_a ? (unsigned)ax + (unsigned)rx * ay + slice * az : (unsigned)bx + (unsigned)rx * by + slice * bz;
          const uchar4 v = cvol[vi];
          cc = make_float4((float)v.z / 255.f, (float)v.y / 255.f, (float)v.x / 255.f, 1.f);
        }
        reinterpret_cast<float4*>(col)[out] = cc;
      }
    }
    base += batch;
    __syncthreads();  // the batch's cubes are no longer read
  }
}

#define NUI_MC_INST(F)                                                                                       \
  template __global__ void k_mc_count<F>(const SessionDesc*, int, unsigned int*, unsigned long long*,     \
                                         uint8_t*);                                                           \
  template __global__ void k_mc_emit<F>(const SessionDesc*, int, const unsigned int*, const unsigned long long*, \
                                        float*, float*, unsigned long long);
NUI_MC_INST(0)
NUI_MC_INST(1)
NUI_MC_INST(2)
NUI_MC_INST(3)

}  // namespace nui
