// Element functions of the medium packing (grids -> 64-byte lookup cells,
// albedo state pairs, majorants), of the per-pixel sample reduction and of
// the gradient fold (cell gradients -> voxel gradients), shared by the
// single-job and the batched kernels.
#pragma once
#include "rcv_volume.cuh"

namespace rcv {

// Cells of a (dx+1)(dy+1)(dz+1) lattice: the 8 clamped corner voxels of the
// old and the new density, x pairs as value and difference (trilerp_diff).
// Called by whole warps with consecutive i, one cell per lane (none from nc
// on); mo and mn receive maxima of voxels of the old and of the new density,
// which over all cells cover every voxel.
// Bound by the stores, 64 bytes per cell.  Two lanes write a cell, one per
// state, so that a warp's store is 1024 consecutive bytes (256^3: 200 us, 6.1
// TB/s); a lane that wrote its own cell in two such stores took 243 us, in
// four of 16 bytes, half sectors of 32 lines each, 309.
// 32-bit index arithmetic: 4 (dx+1)(dy+1)(dz+1) < 2^32 is enforced on the host.
__device__ __forceinline__ void pack_cells(int64_t i, int64_t nc, int dx, int dy, int dz,
                                           const float* __restrict__ old_d, const float* __restrict__ new_d,
                                           float4* __restrict__ cells, float& mo, float& mn) {
  const uint32_t ex = (uint32_t)(dx + 1), ey = (uint32_t)(dy + 1);
  const int lane = threadIdx.x & 31, state = lane & 1;
  const float* __restrict__ d = state ? new_d : old_d;
  float m = 0.0f;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int64_t c = i - lane + 16 * half + (lane >> 1);
    if (c >= nc) break;
    const uint32_t row = (uint32_t)c / ex;
    const int cx = int((uint32_t)c - row * ex);
    const uint32_t cz_u = row / ey;
    const int cy = int(row - cz_u * ey), cz = int(cz_u);
    const uint32_t x0 = (uint32_t)clampi(cx - 1, dx - 1), x1 = (uint32_t)clampi(cx, dx - 1);
    const uint32_t y0 = (uint32_t)clampi(cy - 1, dy - 1), y1 = (uint32_t)clampi(cy, dy - 1);
    const uint32_t z0 = (uint32_t)clampi(cz - 1, dz - 1) * (uint32_t)dy,
                   z1 = (uint32_t)clampi(cz, dz - 1) * (uint32_t)dy;
    const auto pairs = [&](uint32_t r0, uint32_t r1) {  // rows of the corners
      const float a0 = d[r0 + x0], a1 = d[r0 + x1], b0 = d[r1 + x0], b1 = d[r1 + x1];
      m = fmaxf(m, fmaxf(fmaxf(a0, a1), fmaxf(b0, b1)));
      return make_float4(a0, a1 - a0, b0, b1 - b0);
    };
    const float4 lo = pairs((z0 + y0) * (uint32_t)dx, (z0 + y1) * (uint32_t)dx);
    const float4 hi = pairs((z1 + y0) * (uint32_t)dx, (z1 + y1) * (uint32_t)dx);
    store_pair(cells + c * 4 + 2 * state, lo, hi);
  }
  mo = state ? 0.0f : m;
  mn = state ? m : 0.0f;
}

// Voxels whose trilinear weight can be non-zero inside supergrid cell c of
// S cells along an axis of D voxels: x in [c/S, (c+1)/S) reads voxels
// floor(xD - 1/2) and floor(xD - 1/2) + 1, clamped to [0, D-1].
__device__ __forceinline__ void supergrid_span(int c, int S, int D, int& lo, int& hi) {
  const int64_t a = 2 * int64_t(c) * D - S, b = 2 * int64_t(c + 1) * D - S, den = 2 * int64_t(S);
  const int64_t fa = a >= 0 ? a / den : -((-a + den - 1) / den);  // floor division
  const int64_t fb = b >= 0 ? b / den : -((-b + den - 1) / den);
  lo = clampi((int)fa, D - 1);
  hi = clampi((int)fb + 1, D - 1);
}

// Majorants of supergrid cell i (x fastest): scale * the largest old / new
// density (non-negative part) over its voxel span; two = max of both states.
// Called by a whole warp, 8 lanes along x and 4 rows at a time: a cell of
// factor 8 spans up to 1000 voxels of each state, which one thread took one
// after the other (128^3: 82 us, too few threads to hide the loads; a warp
// per cell 24 us).
__device__ __forceinline__ void supergrid_cell(int64_t i, const int sg[3], int dx, int dy, int dz, float scale,
                                               const float* __restrict__ old_d, const float* __restrict__ new_d,
                                               float* __restrict__ sg_two, float* __restrict__ sg_new) {
  const int cx = int(i % sg[0]), cy = int((i / sg[0]) % sg[1]), cz = int(i / (int64_t(sg[0]) * sg[1]));
  int x0, x1, y0, y1, z0, z1;
  supergrid_span(cx, sg[0], dx, x0, x1);
  supergrid_span(cy, sg[1], dy, y0, y1);
  supergrid_span(cz, sg[2], dz, z0, z1);
  const int lane = threadIdx.x & 31;
  float mo = 0.0f, mn = 0.0f;
  for (int z = z0; z <= z1; ++z)
    for (int y = y0 + (lane >> 3); y <= y1; y += 4)
      for (int x = x0 + (lane & 7); x <= x1; x += 8) {
        const int64_t v = (int64_t(z) * dy + y) * dx + x;
        mo = fmaxf(mo, old_d[v]);
        mn = fmaxf(mn, new_d[v]);
      }
  // non-negative floats order like their bits
  mo = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mo)));
  mn = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mn)));
  if (lane == 0) {
    sg_two[i] = scale * fmaxf(mo, mn);
    sg_new[i] = scale * mn;
  }
}

// Voxel i of the old and the new RGB albedo as one 32-byte pair.
__device__ __forceinline__ void pack_albedo(int64_t i, const float* __restrict__ old_a,
                                            const float* __restrict__ new_a, float4* __restrict__ albedo) {
  store_pair(albedo + i * 2, make_float4(old_a[i * 3 + 0], old_a[i * 3 + 1], old_a[i * 3 + 2], 0.0f),
             make_float4(new_a[i * 3 + 0], new_a[i * 3 + 1], new_a[i * 3 + 2], 0.0f));
}

// Sum of a pixel's per-path radiance slots in sample order, divided by spp
// (the box-filter film develop of plugins/twostatevolpath.py:80-89).  Slots
// are [path][new, old] for two-state launches and [path] otherwise.  Called by
// whole blocks of kReduceBlock threads, one pixel per thread (`pix` of
// consecutive threads consecutive, none from npix on).  The slots of a warp's
// 32 pixels are one stretch of memory; a thread that reads its own pixel's
// slots touches another 128-byte line than its neighbours with every load
// (3.4 TB/s).  So the warp loads 8 slots of each of its pixels at a time, 128
// consecutive bytes per 8 lanes, into shared memory, where each thread adds up
// its row (stride 9: no bank conflicts): 512^2 x
// 16 spp of both states 41 -> 26 us (5.2 TB/s), 512^2 x 256 spp of one 305 -> 192
// us (5.6 TB/s of 6.8).
constexpr int kReduceBlock = 256;
constexpr int kReduceChunk = 8;
constexpr int kReduceTile = kReduceBlock * (kReduceChunk + 1);

template <bool kTwo>
__device__ __forceinline__ void reduce_pixel(const float4* __restrict__ path_out, int64_t path_begin, int64_t pix,
                                             int64_t npix, int spp, float4* tile, V3& out_new, V3& out_old) {
  constexpr int K = kTwo ? 2 : 1;
  float nx = 0.0f, ny = 0.0f, nz = 0.0f, ox = 0.0f, oy = 0.0f, oz = 0.0f;
  const int64_t row = int64_t(spp) * K;  // slots of a pixel
  const int lane = threadIdx.x & 31;
  const int64_t pix0 = pix - lane;
  const float4* src = path_out + path_begin * K + pix0 * row;
  float4* rows = tile + (threadIdx.x & ~31u) * (kReduceChunk + 1);
  const float4* mine = rows + lane * (kReduceChunk + 1);
  const int here = npix - pix0 < 32 ? int(npix - pix0 < 0 ? 0 : npix - pix0) : 32;  // pixels of this warp
  const int col = lane & (kReduceChunk - 1), first = lane / kReduceChunk;
  for (int64_t s = 0; s < row; s += kReduceChunk) {
    const int n = row - s < kReduceChunk ? int(row - s) : kReduceChunk;
    float4 v[kReduceChunk];
#pragma unroll
    for (int r = 0; r < kReduceChunk; ++r) {
      const int p = first + r * (32 / kReduceChunk);
      v[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (col < n && p < here) v[r] = __ldcs(src + p * row + s + col);
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kReduceChunk; ++r) rows[(first + r * (32 / kReduceChunk)) * (kReduceChunk + 1) + col] = v[r];
    __syncwarp();
    for (int k = 0; k < n; k += K) {
      const float4 a = mine[k];
      nx += a.x;
      ny += a.y;
      nz += a.z;
      if (kTwo) {
        const float4 b = mine[k + 1];
        ox += b.x;
        oy += b.y;
        oz += b.z;
      }
    }
  }
  const float fs = (float)spp;
  out_new = V3{nx / fs, ny / fs, nz / fs};
  out_old = V3{ox / fs, oy / fs, oz / fs};
}

// Block-wide max of the voxel densities into maxbits[0] (old), [1] (new);
// every thread of the block must call it (blockDim a multiple of 32).
// Non-negative floats order like their bits.  One atomicMax per block and
// state, skipped when the word already holds at least the block's value:
// every value it ever holds is the maximum of some voxels, so a smaller one
// cannot change the result, and a stale read only costs an unneeded atomic.
// (Per-warp atomics on the same two words serialised in one L2 slice and
// took most of a 128^3 grid's packing time.)
__device__ __forceinline__ void reduce_majorants(float mo, float mn, uint32_t* maxbits) {
  __shared__ uint32_t s_max[2][32];
  uint32_t bo = __float_as_uint(fmaxf(mo, 0.0f)), bn = __float_as_uint(fmaxf(mn, 0.0f));
  bo = __reduce_max_sync(0xffffffffu, bo);
  bn = __reduce_max_sync(0xffffffffu, bn);
  const unsigned w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_max[0][w] = bo;
    s_max[1][w] = bn;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const unsigned nw = (blockDim.x + 31) >> 5;
    bo = threadIdx.x < nw ? s_max[0][threadIdx.x] : 0u;
    bn = threadIdx.x < nw ? s_max[1][threadIdx.x] : 0u;
    bo = __reduce_max_sync(0xffffffffu, bo);
    bn = __reduce_max_sync(0xffffffffu, bn);
    if (threadIdx.x == 0) {
      if (bo != 0u && bo > __ldcg(maxbits + 0)) atomicMax(maxbits + 0, bo);
      if (bn != 0u && bn > __ldcg(maxbits + 1)) atomicMax(maxbits + 1, bn);
    }
  }
}

// Whether cell c of an axis of D voxels uses voxel v as its corner `bit`
// (corner 0 is voxel clamp(c - 1), corner 1 voxel clamp(c)).  Only cells v
// and v + 1 can, so a voxel has at most 4 (cell, bit) pairs per axis.
__device__ __forceinline__ bool fold_uses(int c, int bit, int v, int D) {
  return c <= D && clampi(c - 1 + bit, D - 1) == v;
}

// Calls f(entry) with the address of each corner entry (C floats; 8 per cell)
// of voxel (x, y, z), in the order z, y, x candidate, each by cell and then
// corner bit.  Along an axis those are the cell's corner 1 and the next one's
// corner 0, and at the grid's faces, where cells clamp, the other corners.
// The x faces are two predicated entries (one lane of a warp has one); trying
// all 64 candidate slots for every voxel was bound by their tests, a branch
// for inner voxels by its divergence (256^3, with the tiles of
// fold_density_kernel: 194 -> 148 us; 96-byte records of 64^3: 13.7 -> 13.4).
template <int C, class F>
__device__ __forceinline__ void fold_entries(int x, int y, int z, int dx, int dy, int dz,
                                             const float* __restrict__ gcells, F f) {
  const int64_t row = int64_t(dx + 1) * (8 * C), plane = row * (dy + 1);
  const float* own = gcells + z * plane + y * row + int64_t(x) * (8 * C);
  const auto along_x = [&](const float* r) {
    if (x == 0) f(r);
    f(r + C);
    f(r + 8 * C);
    if (x == dx - 1) f(r + 9 * C);
  };
  if (y > 0 && y < dy - 1 && z > 0 && z < dz - 1) {
    along_x(own + 6 * C);
    along_x(own + row + 4 * C);
    along_x(own + plane + 2 * C);
    along_x(own + plane + row);
    return;
  }
  for (int kz = 0; kz < 4; ++kz) {
    if (!fold_uses(z + (kz >> 1), kz & 1, z, dz)) continue;
    for (int ky = 0; ky < 4; ++ky)
      if (fold_uses(y + (ky >> 1), ky & 1, y, dy))
        along_x(own + (kz >> 1) * plane + (ky >> 1) * row + (2 * (ky & 1) + 4 * (kz & 1)) * C);
  }
}

// Voxel i of a grid (32-bit index arithmetic: fewer than 2^30 voxels).
__device__ __forceinline__ void voxel_of(int64_t i, int dx, int dy, int& x, int& y, int& z) {
  const uint32_t row = (uint32_t)i / (uint32_t)dx;
  x = int((uint32_t)i - row * (uint32_t)dx);
  const uint32_t z_u = row / (uint32_t)dy;
  y = int(row - z_u * (uint32_t)dy);
  z = int(z_u);
}

// Gradient of a voxel: the sum of its corner entries (8 floats per cell).
__device__ __forceinline__ float fold_voxel(int x, int y, int z, int dx, int dy, int dz,
                                            const float* __restrict__ gcells) {
  float g = 0.0f;
  fold_entries<1>(x, y, z, dx, dy, dz, gcells, [&](const float* r) { g += *r; });
  return g;
}

// RGB gradient of an albedo voxel from the albedo cell records (24 floats per
// cell: corner k = bx + 2 by + 4 bz, then R, G, B), summed in the order of
// fold_voxel.
__device__ __forceinline__ V3 fold_voxel_rgb(int x, int y, int z, int dx, int dy, int dz,
                                             const float* __restrict__ gcells) {
  V3 g{0.0f, 0.0f, 0.0f};
  fold_entries<3>(x, y, z, dx, dy, dz, gcells, [&](const float* r) {
    g = V3{g.x + r[0], g.y + r[1], g.z + r[2]};
  });
  return g;
}

}  // namespace rcv
