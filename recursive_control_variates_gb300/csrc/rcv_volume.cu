// Volumetric kernels of librcv and their C-ABI entry points:
// medium packing + majorants, persistent two-state primal, single-state
// primal and seed-replay adjoint, the per-pixel sample reduction and the
// gradient fold back to voxel layout.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "rcv_common.h"
#include "rcv_pack.cuh"
#include "rcv_trace_kernels.cuh"

namespace rcv {

// ------------------------------------------------------------------ packing
// One thread per cell / albedo voxel (na: albedo grid voxels).
__global__ void pack_medium_kernel(int dx, int dy, int dz, const float* __restrict__ old_d,
                                   const float* __restrict__ new_d, float4* __restrict__ cells,
                                   const float* __restrict__ old_a, const float* __restrict__ new_a,
                                   float4* __restrict__ albedo, int64_t na, uint32_t* __restrict__ maxbits) {
  const int64_t nc = int64_t(dx + 1) * (dy + 1) * (dz + 1);
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  float mo, mn;
  pack_cells(i, nc, dx, dy, dz, old_d, new_d, cells, mo, mn);
  if (albedo != nullptr && i < na) pack_albedo(i, old_a, new_a, albedo);
  // majorant: maximum density of each state (non-negative part)
  reduce_majorants(mo, mn, maxbits);
}

// ----------------------------------------------------------------- tracing
// Tracer variants by index mode + kTraceModes * (supergrid + 2 * counting +
// 4 * environment map), then those of job tables (rcv_trace_table.cu).
template <bool kSG, bool kCount, bool kEnv>
struct TraceVariants {
  static constexpr TraceKernel k[kTraceModes] = {
      trace_kernel<kTwoState, kSG, kCount, kEnv, false>, trace_kernel<kSingle, kSG, kCount, kEnv, false>,
      trace_kernel<kAdjoint, kSG, kCount, kEnv, false>,  trace_kernel<kReplay, kSG, kCount, kEnv, false>,
      trace_kernel<kForward, kSG, kCount, kEnv, false>,  trace_kernel<kTape, kSG, kCount, kEnv, false>};
};
static const TraceKernel* const kTraceTables[12] = {
    TraceVariants<false, false, false>::k, TraceVariants<true, false, false>::k,
    TraceVariants<false, true, false>::k,  TraceVariants<true, true, false>::k,
    TraceVariants<false, false, true>::k,  TraceVariants<true, false, true>::k,
    TraceVariants<false, true, true>::k,   TraceVariants<true, true, true>::k,
    kJobTableTracers[0], kJobTableTracers[1], kJobTableTracers[2], kJobTableTracers[3]};
constexpr int kTraceVariants = 12 * kTraceModes;

static int trace_variant(int mode, bool sg, bool count, bool env, bool table) {
  return mode + kTraceModes * ((sg ? 1 : 0) + (count ? 2 : 0) + (table ? 8 : (env ? 4 : 0)));
}
static TraceKernel trace_kernel_of(int variant) { return kTraceTables[variant / kTraceModes][variant % kTraceModes]; }

// Majorant supergrid of a medium (both states' cells and the new state's).
__global__ void supergrid_kernel(int sx, int sy, int sz, int dx, int dy, int dz, float scale,
                                 const float* __restrict__ old_d, const float* __restrict__ new_d,
                                 float* __restrict__ sg_two, float* __restrict__ sg_new) {
  const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;  // one warp per cell
  if (i >= int64_t(sx) * sy * sz) return;
  const int sg[3] = {sx, sy, sz};
  supergrid_cell(i, sg, dx, dy, dz, scale, old_d, new_d, sg_two, sg_new);
}

// ------------------------------------------------------ hand-out ordering
// Pixels are handed to the persistent tracer most-expensive first, so that
// the queue ends on cheap paths instead of on a few long ones: by the
// measured path lengths of the previous call (cost_bucket), or by the length
// of the pixel-centre ray's chord through the medium cube, in 256 buckets
// (bucket 0 = longest; misses last by chord).  By measured lengths a path that
// misses counts the rest of its round of kWalkSteps: its pixel comes among the
// cheap ones, and the stores of missed paths go on beside walks.  Charged
// nothing, missed pixels went last, as one stretch of stores: 512^2 x 256-spp
// target 9.85 -> 10.01 ms, step of 512^2 x 16 spp 2.002 -> 2.016, others alike.
constexpr int kOrderBuckets = 256;

// Pixels without a cost (a workspace's first call, the samples of supergrid
// media that left at once, the volpathsimple adjoint, which keeps none): the chord through the cube,
// times one plus the optical depth along it (8 points of the pixel's central
// ray).  A first call in the order of the film's rows ended on whatever its
// last rows held: first step of 512^2 x 16 spp 2060 -> 1892 us (by the chord
// alone 1946), of five 107 x 83 views 1486 -> 1362 (1400), first target of
// 512^2 x 256 spp 9.3 -> 8.8 ms.
__device__ __forceinline__ int estimated_key(const VolJob& J, int pix) {
  V3 o, d;
  camera_ray(J, pix % J.width, pix / J.width, 0.5f, 0.5f, o, d);
  float tn, tf;
  slab(o, recip(d), tn, tf);
  tn = fmaxf(tn, 0.0f);
  if (!(tn < tf)) return cost_bucket(0u);
  const float step = (tf - tn) * 0.125f;
  float sum = 0.0f;
  for (int k = 0; k < 8; ++k) sum += density_new(J, locate(J, advance(o, tn + ((float)k + 0.5f) * step, d)));
  const float est = (tf - tn) * 16.0f * (1.0f + J.scale * sum * step);
  return cost_bucket((uint32_t)fminf(fmaxf(est, 0.0f), 1e9f) + 1u);
}

__device__ __forceinline__ int order_key(const OrderJob& O, int pix) {
  const uint32_t c = O.cost != nullptr ? O.cost[pix] : 0u;
  if (c != 0u) return cost_bucket(c);
  return O.chord ? chord_key(O.J, pix) : estimated_key(O.J, pix);
}

__global__ void order_count_kernel(const __grid_constant__ OrderJob A, const __grid_constant__ OrderJob B) {
  const OrderJob& O = blockIdx.y == 0 ? A : B;
  __shared__ uint32_t hist[kOrderBuckets];
  for (int k = threadIdx.x; k < kOrderBuckets; k += blockDim.x) hist[k] = 0;
  __syncthreads();
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix < O.npix) atomicAdd(&hist[order_key(O, pix)], 1u);
  __syncthreads();
  for (int k = threadIdx.x; k < kOrderBuckets; k += blockDim.x)
    if (hist[k]) atomicAdd(O.buckets + k, hist[k]);
}

// Films of up to kOrderSmall pixels: one block per job clears the workspace's
// head, counts, scans and places, in one launch instead of a clear per job and
// two more (64^2: one of 5.6 us for 4 of 1 to 2.3 us, which cost the host 4.5
// us each; at 128^2 it takes 16 us, so the line lies between).
constexpr int kOrderSmall = 8192;
constexpr int kOrderSmallBlock = 1024;

__global__ void __launch_bounds__(kOrderSmallBlock) order_small_kernel(const __grid_constant__ OrderJob A,
                                                                       const __grid_constant__ OrderJob B) {
  const OrderJob& O = blockIdx.x == 0 ? A : B;
  __shared__ uint32_t next[kOrderBuckets];
  const int t = threadIdx.x;
  if (O.head != nullptr)
    for (int i = t; i < int(kRenderHeadBytes / sizeof(uint32_t)); i += kOrderSmallBlock)
      reinterpret_cast<uint32_t*>(O.head)[i] = 0u;
  if (t < kOrderBuckets) next[t] = 0u;
  __syncthreads();
  for (int pix = t; pix < O.npix; pix += kOrderSmallBlock) atomicAdd(&next[order_key(O, pix)], 1u);
  __syncthreads();
  if (t < 32) {  // exclusive prefix sum, 8 buckets per lane
    uint32_t n[kOrderBuckets / 32], own = 0u;
    for (int k = 0; k < kOrderBuckets / 32; ++k) own += n[k] = next[t * (kOrderBuckets / 32) + k];
    uint32_t sum = own;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, sum, off);
      if (t >= off) sum += v;
    }
    sum -= own;
    for (int k = 0; k < kOrderBuckets / 32; ++k) {
      next[t * (kOrderBuckets / 32) + k] = sum;
      sum += n[k];
    }
  }
  __syncthreads();
  for (int pix = t; pix < O.npix; pix += kOrderSmallBlock) {
    O.order[atomicAdd(&next[order_key(O, pix)], 1u)] = (uint32_t)pix;
    if (O.cost != nullptr) O.cost[pix] = 0u;  // the next tracer call accumulates afresh
  }
}

// Every block derives the buckets' first slots from the counts itself (256
// values; a launch of its own for the scan cost more than that).
__global__ void __launch_bounds__(kOrderBuckets) order_place_kernel(const __grid_constant__ OrderJob A,
                                                                    const __grid_constant__ OrderJob B) {
  const OrderJob& O = blockIdx.y == 0 ? A : B;
  if (int(blockIdx.x * blockDim.x) >= O.npix) return;  // the other job's film is larger
  __shared__ uint32_t first[kOrderBuckets], warp_sum[kOrderBuckets / 32];
  const int t = threadIdx.x;
  const uint32_t n = __ldcg(O.buckets + t);
  uint32_t sum = n;  // inclusive in the warp
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, sum, off);
    if ((t & 31) >= off) sum += v;
  }
  if ((t & 31) == 31) warp_sum[t >> 5] = sum;
  __syncthreads();
  for (int w = 0; w < (t >> 5); ++w) sum += warp_sum[w];
  first[t] = sum - n;
  __syncthreads();
  const int pix = blockIdx.x * blockDim.x + t;
  const bool valid = pix < O.npix;
  place_block(valid ? order_key(O, pix) : 0, valid, (uint32_t)pix, O.buckets + kOrderBuckets, O.order, first);
  if (valid && O.cost != nullptr) O.cost[pix] = 0u;  // the next tracer call accumulates afresh
}

// Sum of a pixel's samples in sample order, divided by spp (the box-filter
// film develop of plugins/twostatevolpath.py:80-89).
template <bool kTwo>
__global__ void __launch_bounds__(kReduceBlock) reduce_paths_kernel(const float4* __restrict__ path_out,
                                                                    int64_t path_begin, int64_t npix, int spp,
                                                                    float* __restrict__ out_new,
                                                                    float* __restrict__ out_old) {
  __shared__ float4 tile[kReduceTile];
  const int64_t pix = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  V3 n, o;
  reduce_pixel<kTwo>(path_out, path_begin, pix, npix, spp, tile, n, o);
  if (pix >= npix) return;
  out_new[pix * 3 + 0] = n.x;
  out_new[pix * 3 + 1] = n.y;
  out_new[pix * 3 + 2] = n.z;
  if (kTwo) {
    out_old[pix * 3 + 0] = o.x;
    out_old[pix * 3 + 1] = o.y;
    out_old[pix * 3 + 2] = o.z;
  }
}

// ------------------------------------------------------------ gradient fold
// Blocks take tiles of kFoldX x kFoldY x kFoldZ voxels, so that the cells that
// neighbouring rows share come from the L1 (256^3: 148 us, 4.1 TB/s of records
// read once; in runs of 256 voxels of one row 215, in tiles of 32 x 4 x 4 171;
// 32 x 4 x 2 and 32 x 2 x 1 as good).  A lane that took its neighbour's corner
// by a shuffle in place of a load was slower (214 to 243).
constexpr int kFoldX = 32, kFoldY = 2, kFoldZ = 2, kFoldBlock = kFoldX * kFoldY * kFoldZ;

static unsigned fold_grid(const int32_t d[3]) {
  // ceil per axis in 64 bits; fewer than 2^30 voxels, so the product fits
  return unsigned(((int64_t(d[0]) + kFoldX - 1) / kFoldX) * ((int64_t(d[1]) + kFoldY - 1) / kFoldY) *
                  ((int64_t(d[2]) + kFoldZ - 1) / kFoldZ));
}

// The block's voxel of this thread; false outside the grid.
__device__ __forceinline__ bool fold_tile(int dx, int dy, int dz, int& x, int& y, int& z) {
  const uint32_t nx = (uint32_t(dx) + kFoldX - 1) / kFoldX, ny = (uint32_t(dy) + kFoldY - 1) / kFoldY;
  const uint32_t row = blockIdx.x / nx, plane = row / ny;
  x = int(blockIdx.x - row * nx) * kFoldX + int(threadIdx.x % kFoldX);
  y = int(row - plane * ny) * kFoldY + int(threadIdx.x / kFoldX % kFoldY);
  z = int(plane) * kFoldZ + int(threadIdx.x / (kFoldX * kFoldY));
  return x < dx && y < dy && z < dz;
}

__global__ void __launch_bounds__(kFoldBlock) fold_density_kernel(int dx, int dy, int dz,
                                                                  const float* __restrict__ gcells,
                                                                  float* __restrict__ grad) {
  int x, y, z;
  if (!fold_tile(dx, dy, dz, x, y, z)) return;
  grad[(int64_t(z) * dy + y) * dx + x] += fold_voxel(x, y, z, dx, dy, dz, gcells);
}

__global__ void __launch_bounds__(kFoldBlock) fold_albedo_kernel(int adx, int ady, int adz,
                                                                 const float* __restrict__ gcells,
                                                                 float* __restrict__ grad) {
  int x, y, z;
  if (!fold_tile(adx, ady, adz, x, y, z)) return;
  const V3 g = fold_voxel_rgb(x, y, z, adx, ady, adz, gcells);
  float* r = grad + ((int64_t(z) * ady + y) * adx + x) * 3;
  r[0] += g.x;
  r[1] += g.y;
  r[2] += g.z;
}

// Forward mode: the tangent of the density packed like a cell gradient
// record (8 corners, the layout tangent_density reads), and the albedo
// tangent as one float4 per albedo voxel.
__global__ void pack_tangent_kernel(int dx, int dy, int dz, const float* __restrict__ t,
                                    float4* __restrict__ cells) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= int64_t(dx + 1) * (dy + 1) * (dz + 1)) return;
  const uint32_t ex = (uint32_t)(dx + 1), ey = (uint32_t)(dy + 1);
  const uint32_t row = (uint32_t)i / ex;
  const int cx = int((uint32_t)i - row * ex);
  const uint32_t cz_u = row / ey;
  const int cy = int(row - cz_u * ey), cz = int(cz_u);
  const int x0 = clampi(cx - 1, dx - 1), x1 = clampi(cx, dx - 1);
  const int y0 = clampi(cy - 1, dy - 1), y1 = clampi(cy, dy - 1);
  const int z0 = clampi(cz - 1, dz - 1), z1 = clampi(cz, dz - 1);
  auto v = [&](int x, int y, int z) { return t[(int64_t(z) * dy + y) * dx + x]; };
  cells[i * 2 + 0] = make_float4(v(x0, y0, z0), v(x1, y0, z0), v(x0, y1, z0), v(x1, y1, z0));
  cells[i * 2 + 1] = make_float4(v(x0, y0, z1), v(x1, y0, z1), v(x0, y1, z1), v(x1, y1, z1));
}

__global__ void pack_tangent_albedo_kernel(int64_t na, const float* __restrict__ t, float4* __restrict__ out) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= na) return;
  out[i] = make_float4(t[i * 3 + 0], t[i * 3 + 1], t[i * 3 + 2], 0.0f);
}

// ------------------------------------------------------------- host helpers
static int validate_medium(const rcv_medium* m) {
  RCV_REQUIRE(m != nullptr, "medium is NULL");
  RCV_REQUIRE(m->dims[0] > 0 && m->dims[1] > 0 && m->dims[2] > 0, "grid dims must be positive");
  RCV_REQUIRE(uint64_t(m->dims[0] + 1) * uint64_t(m->dims[1] + 1) * uint64_t(m->dims[2] + 1) * 4u <
                  (uint64_t(1) << 32),
              "grid too large: (Dx+1)(Dy+1)(Dz+1) must be below 2^30");
  RCV_REQUIRE(m->density_old != nullptr && m->density_new != nullptr, "density grids are NULL");
  RCV_REQUIRE((m->albedo_old == nullptr) == (m->albedo_new == nullptr),
              "albedo_old and albedo_new must both be set or both be NULL");
  RCV_REQUIRE(m->workspace != nullptr, "medium workspace is NULL");
  RCV_REQUIRE((reinterpret_cast<uintptr_t>(m->workspace) & 255u) == 0,
              "medium workspace must be 256-byte aligned");
  RCV_REQUIRE(m->scale >= 0.0f, "medium scale must be non-negative");
  RCV_REQUIRE(m->majorant_factor >= 0, "majorant_factor must be >= 0");
  const bool own = m->albedo_dims[0] != 0 || m->albedo_dims[1] != 0 || m->albedo_dims[2] != 0;
  RCV_REQUIRE(!own || (m->albedo_dims[0] > 0 && m->albedo_dims[1] > 0 && m->albedo_dims[2] > 0),
              "albedo_dims must be all positive or all 0");
  return RCV_OK;
}

int make_volume_job(const rcv_medium* m, const rcv_sensor* s, const rcv_volpath_options* o,
                    uint32_t seed, int spp, VolJob* J) {
  int rc = validate_medium(m);
  if (rc) return rc;
  RCV_REQUIRE(s != nullptr && o != nullptr, "sensor / options are NULL");
  RCV_REQUIRE(s->width > 0 && s->height > 0, "film size must be positive");
  RCV_REQUIRE(spp > 0, "spp must be positive");
  RCV_REQUIRE(o->max_depth >= -1, "max_depth must be >= -1");
  RCV_REQUIRE(int64_t(s->width) * s->height * spp < (int64_t(1) << 32),
              "width * height * spp must be below 2^32 (one random stream per path)");
  const int n_cams = s->count > 1 ? s->count : 1;
  RCV_REQUIRE(n_cams <= RCV_MAX_SENSORS, "a batch sensor has at most %d sub-sensors", RCV_MAX_SENSORS);
  RCV_REQUIRE(s->width % n_cams == 0, "batch film width %d is not a multiple of its %d sensors", s->width,
              n_cams);
  float inv_box[3];
  for (int a = 0; a < 3; ++a) {
    RCV_REQUIRE(m->box_size[a] >= 0.0f && std::isfinite(m->box_size[a]) && std::isfinite(m->box_min[a]),
                "medium box must have a finite, non-negative size");
    inv_box[a] = m->box_size[a] > 0.0f ? 1.0f / m->box_size[a] : 1.0f;
  }
  std::memset(J, 0, sizeof(VolJob));
  J->width = s->width;
  J->height = s->height;
  J->spp = spp;
  J->n_cams = n_cams;
  J->inv_box = V3{inv_box[0], inv_box[1], inv_box[2]};
  J->box = V3{m->box_size[0] > 0.0f ? m->box_size[0] : 1.0f, m->box_size[1] > 0.0f ? m->box_size[1] : 1.0f,
              m->box_size[2] > 0.0f ? m->box_size[2] : 1.0f};
  if (o->envmap != nullptr) {
    const rcv_envmap* e = o->envmap;
    RCV_REQUIRE(e->width > 0 && e->height > 0 && e->workspace != nullptr &&
                    (reinterpret_cast<uintptr_t>(e->workspace) & 255u) == 0,
                "environment map: positive size and a 256-byte aligned workspace are required");
    RCV_REQUIRE(std::isfinite(e->scale) && e->scale >= 0.0f, "environment map scale must be finite and >= 0");
    const EnvLayout EL = env_layout(e->width, e->height);
    const char* ew = static_cast<const char*>(e->workspace);
    J->env.valid = 1;
    J->env.w = e->width;
    J->env.h = e->height;
    J->env.inv_w = 1.0f / (float)e->width;
    J->env.inv_h = 1.0f / (float)e->height;
    J->env.scale = e->scale;
    J->env.tex = reinterpret_cast<const float4*>(ew + EL.tex);
    J->env.cond = reinterpret_cast<const float*>(ew + EL.cond);
    J->env.marg = reinterpret_cast<const float*>(ew + EL.marg);
    J->env.hdr = reinterpret_cast<const float*>(ew + EL.hdr);
  }
  for (int k = 0; k < n_cams; ++k) {
    const float* o = k == 0 ? s->origin : s->more[k - 1].origin;
    const float* f = k == 0 ? s->forward : s->more[k - 1].forward;
    const float* r = k == 0 ? s->right : s->more[k - 1].right;
    const float* u = k == 0 ? s->up : s->more[k - 1].up;
    // camera origin in box coordinates; the directions stay in world space
    J->cam[k].o = V3{(o[0] - m->box_min[0]) * inv_box[0], (o[1] - m->box_min[1]) * inv_box[1],
                     (o[2] - m->box_min[2]) * inv_box[2]};
    J->cam[k].f = V3{f[0], f[1], f[2]};
    J->cam[k].r = V3{r[0], r[1], r[2]};
    J->cam[k].u = V3{u[0], u[1], u[2]};
  }
  J->inv_w = 1.0f / (float)s->width;
  J->inv_h = 1.0f / (float)s->height;
  J->max_depth = o->max_depth < 0 ? 0x7fffffff : o->max_depth;
  J->rr_depth = o->rr_depth;
  J->hide_emitters = o->hide_emitters;
  J->seed = seed;
  J->dx = m->dims[0];
  J->dy = m->dims[1];
  J->dz = m->dims[2];
  J->scale = m->scale;
  J->fdx = (float)m->dims[0];
  J->fdy = (float)m->dims[1];
  J->fdz = (float)m->dims[2];
  J->long_axis = (m->dims[0] | m->dims[1] | m->dims[2]) >= (1 << 21) ? 1 : 0;
  const MediumLayout L = medium_layout(m);
  char* ws = static_cast<char*>(m->workspace);
  J->cells = reinterpret_cast<const float4*>(ws + L.cells);
  J->albedo = m->albedo_old ? reinterpret_cast<const float4*>(ws + L.albedo) : nullptr;
  int32_t ad[3];
  albedo_dims_of(m, ad);
  J->adx = ad[0];
  J->ady = ad[1];
  J->adz = ad[2];
  J->albedo_own_res = (ad[0] != m->dims[0] || ad[1] != m->dims[1] || ad[2] != m->dims[2]) ? 1 : 0;
  J->albedo_const[0] = m->albedo_value[0];
  J->albedo_const[1] = m->albedo_value[1];
  J->albedo_const[2] = m->albedo_value[2];
  J->maxbits = reinterpret_cast<const uint32_t*>(ws + L.maxbits);
  J->sg[0] = supergrid_cells(m->dims[0], m->majorant_factor);
  J->sg[1] = supergrid_cells(m->dims[1], m->majorant_factor);
  J->sg[2] = supergrid_cells(m->dims[2], m->majorant_factor);
  for (int a = 0; a < 3; ++a) J->sg_inv[a] = J->sg[a] > 0 ? 1.0f / (float)J->sg[a] : 0.0f;
  J->sg_two = J->sg[0] > 0 ? reinterpret_cast<const float*>(ws + L.sg_two) : nullptr;
  J->sg_new = J->sg[0] > 0 ? reinterpret_cast<const float*>(ws + L.sg_new) : nullptr;
  J->grad_cells = reinterpret_cast<float4*>(ws + L.grad_cells);
  J->grad_albedo = m->albedo_old ? reinterpret_cast<float4*>(ws + L.grad_albedo) : nullptr;
  J->path_begin = 0;
  J->path_count = int64_t(s->width) * s->height * spp;
  return RCV_OK;
}

// Resident blocks per SM of each tracer variant (queried once per process).
static int resident_blocks(int variant) {
  static std::once_flag once;
  static int blocks[kTraceVariants];
  std::call_once(once, [] {
    for (int v = 0; v < kTraceVariants; ++v) {
      blocks[v] = 1;
      if (trace_kernel_of(v) == nullptr) continue;  // a mode that job tables do not run
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks[v], trace_kernel_of(v), kTraceBlock, 0);
      if (blocks[v] < 1) blocks[v] = 1;
    }
  });
  return blocks[variant];
}

static int sm_count() {
  static std::once_flag once;
  static int n = 1;
  std::call_once(once, [] {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n < 1) n = 1;
  });
  return n;
}

int tracer_sm_count() { return sm_count(); }

int paths_per_fetch(int64_t total, int most) {
  const int64_t share = total / (int64_t(sm_count()) * 24 * 8);
  return share < most ? (int)(share < 2 ? (most < 2 ? most : 2) : share) : most;
}

void warm_launch_config() {
  (void)resident_blocks(0);
  (void)sm_count();
  warm_pair_config();
}

static_assert(kOrderBuckets == kRenderOrderBuckets, "order bucket count mismatch");
static_assert(int64_t(kTapeChunk) == kTapeChunkSlots, "tape chunk mismatch");

int order_pixels(const OrderJob* jobs, int n, cudaStream_t st) {
  const OrderJob& A = jobs[0];
  const OrderJob& B = jobs[n - 1];
  if (A.npix <= kOrderSmall && B.npix <= kOrderSmall) {
    order_small_kernel<<<(unsigned)n, kOrderSmallBlock, 0, st>>>(A, B);
    return launched("order launch");
  }
  for (int k = 0; k < n; ++k)
    if (jobs[k].head != nullptr) RCV_TRY_CUDA(cudaMemsetAsync(jobs[k].head, 0, kRenderHeadBytes, st), "counters reset");
  const dim3 grid(grid_for(A.npix > B.npix ? A.npix : B.npix, kOrderBuckets), (unsigned)n);
  order_count_kernel<<<grid, kOrderBuckets, 0, st>>>(A, B);
  int rc = launched("order_count launch");
  if (rc) return rc;
  order_place_kernel<<<grid, kOrderBuckets, 0, st>>>(A, B);
  return launched("order_place launch");
}

// Work queue of a persistent launch over `total` paths of one job (jobs ==
// null) or of a device job table; zeroes its hand-out counter on `st`.
int make_queue(int mode, const VolJob* jobs, int njobs, int64_t total, const rcv_volpath_options* o,
               unsigned long long* queue_counter, float4* path_out, const AdjBuffers* adj, uint64_t* counters,
               cudaStream_t st, Queue* out, bool zeroed) {
  Queue& Q = *out;
  std::memset(&Q, 0, sizeof(Q));
  Q.counter = queue_counter;
  Q.path_out = (mode == kTwoState || mode == kSingle) ? path_out : nullptr;
  if (mode == kAdjoint || mode == kReplay || mode == kForward || mode == kTape) {
    RCV_REQUIRE(adj != nullptr && adj->ckpt && adj->ckpt_count && adj->path_ltot, "adjoint buffers missing");
    RCV_REQUIRE(total < (int64_t(1) << 32), "an adjoint launch must have fewer than 2^32 paths");
    Q.ckpt = adj->ckpt;
    Q.ckpt_count = adj->ckpt_count;
    Q.ckpt_cap = adj->ckpt_cap;
    Q.path_ltot = adj->path_ltot;
    if (adj->tape != nullptr) {
      // tape pass, or the replay of the paths it lost
      RCV_REQUIRE(mode == kTape || mode == kReplay, "the tape serves the gradient only");
      RCV_REQUIRE(total < (int64_t(1) << 30) && adj->ckpt_cap < (int64_t(1) << 30) &&
                      adj->tape_cap <= (int64_t(1) << 32) - int64_t(kTapeChunk),
                  "too many paths for the tape adjoint");
      RCV_REQUIRE(adj->tape_f != nullptr && adj->entered != nullptr && adj->entered_count != nullptr &&
                      adj->cam_w != nullptr,
                  "the tape needs its extinction terms and the list of entered paths");
      Q.tape = adj->tape;
      Q.tape_f = adj->tape_f;
      Q.entered = adj->entered;
      Q.entered_count = adj->entered_count;
      Q.tape_count = adj->tape_count;
      Q.tape_cap = adj->tape_cap;
      Q.lost_list = adj->lost_list;
      Q.lost_count = adj->lost_count;
    }
  }
  RCV_REQUIRE(mode != kTape || Q.tape != nullptr, "the tape pass needs a tape");
  Q.counters = reinterpret_cast<unsigned long long*>(counters);
  Q.jobs = jobs;
  Q.njobs = njobs;
  Q.total = total;
  // a large launch of one job takes up to 256 at a time: a fetch costs its warp
  // an atomic's latency and all warps share the counter (67 M paths of 512^2 x
  // 256 spp: 32 / 64 / 128 / 256 per fetch 10.98 / 10.48 / 10.06 / 9.77 ms), and
  // there a fetch of 1/64 of a warp's share leaves no tail (16.8 M paths of
  // 1024^2 alike at 64 to 256; a table of 24 uneven jobs, 34.8 M paths, 17.75 ms
  // at 64, 18.45 at 256)
  int most = 64;
  if (o != nullptr && o->batch > 0)
    most = o->batch;
  else if (jobs == nullptr)
    most = (int)std::min<int64_t>(256, std::max<int64_t>(64, total / (int64_t(sm_count()) * 24 * 64)));
  RCV_REQUIRE(most <= (1 << 20), "batch must be <= 2^20");
  Q.batch = paths_per_fetch(total, most);
  Q.defer = (o != nullptr && o->defer > 0) ? o->defer : 8;
  RCV_REQUIRE(Q.defer <= 32, "defer must be in [1, 32]");
  if (!zeroed) RCV_TRY_CUDA(cudaMemsetAsync(Q.counter, 0, sizeof(unsigned long long), st), "queue reset");
  return RCV_OK;
}

// Persistent launch over `total` paths of one job (jobs == null) or of a
// device job table.
int launch_persistent(int mode, const VolJob& J, const VolJob* jobs, int njobs, int64_t total,
                      const rcv_volpath_options* o, unsigned long long* queue_counter,
                      float4* path_out, const AdjBuffers* adj, uint64_t* counters, cudaStream_t st,
                      bool supergrid, bool zeroed) {
  Queue Q;
  int rc = make_queue(mode, jobs, njobs, total, o, queue_counter, path_out, adj, counters, st, &Q, zeroed);
  if (rc) return rc;
  const bool sg = supergrid || (jobs == nullptr && J.sg[0] > 0);
  // an environment map belongs to a single job (batched tables take the constant environment)
  const int variant = trace_variant(mode, sg, counters != nullptr, jobs == nullptr && J.env.valid != 0, jobs != nullptr);
  RCV_REQUIRE(trace_kernel_of(variant) != nullptr, "tracer mode %d does not take a job table", mode);
  int per_sm = resident_blocks(variant);
  if (o != nullptr && o->blocks_per_sm > 0 && o->blocks_per_sm < per_sm) per_sm = o->blocks_per_sm;
  // replay: the checkpoint tasks come on top of one camera task per path
  const int64_t tasks = (mode == kReplay || mode == kForward) ? 2 * total : total;
  const int64_t warps_needed = (tasks + Q.batch - 1) / Q.batch;
  int64_t blocks = (warps_needed + (kTraceBlock / 32) - 1) / (kTraceBlock / 32);
  const int64_t cap = int64_t(sm_count()) * per_sm;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  const unsigned g = (unsigned)blocks;
  trace_kernel_of(variant)<<<g, kTraceBlock, 0, st>>>(J, Q);
  return launched("trace kernel launch");
}

int launch_reduce(bool two, const float4* po, int64_t path_begin, int64_t npix, int spp,
                  float* out_new, float* out_old, cudaStream_t st) {
  const int block = kReduceBlock;
  if (two)
    reduce_paths_kernel<true><<<grid_for(npix, block), block, 0, st>>>(po, path_begin, npix, spp,
                                                                     out_new, out_old);
  else
    reduce_paths_kernel<false><<<grid_for(npix, block), block, 0, st>>>(po, path_begin, npix, spp,
                                                                      out_new, nullptr);
  return launched("reduce_paths launch");
}

int launch_fold(const rcv_medium* m, float* grad_density, float* grad_albedo, cudaStream_t st) {
  const MediumLayout L = medium_layout(m);
  const char* ws = static_cast<const char*>(m->workspace);
  fold_density_kernel<<<fold_grid(m->dims), kFoldBlock, 0, st>>>(
      m->dims[0], m->dims[1], m->dims[2], reinterpret_cast<const float*>(ws + L.grad_cells), grad_density);
  int rc = launched("fold_density launch");
  if (rc) return rc;
  if (grad_albedo != nullptr && m->albedo_old != nullptr) {
    int32_t ad[3];
    albedo_dims_of(m, ad);
    fold_albedo_kernel<<<fold_grid(ad), kFoldBlock, 0, st>>>(
        ad[0], ad[1], ad[2], reinterpret_cast<const float*>(ws + L.grad_albedo), grad_albedo);
    rc = launched("fold_albedo launch");
  }
  return rc;
}

int reset_gradients(const rcv_medium* m, bool albedo, cudaStream_t st) {
  const MediumLayout L = medium_layout(m);
  char* ws = static_cast<char*>(m->workspace);
  const int64_t nc = int64_t(m->dims[0] + 1) * (m->dims[1] + 1) * (m->dims[2] + 1);
  RCV_TRY_CUDA(cudaMemsetAsync(ws + L.grad_cells, 0, nc * 32, st), "gradient reset");
  if (albedo && m->albedo_old != nullptr) {
    int32_t ad[3];
    albedo_dims_of(m, ad);
    RCV_TRY_CUDA(cudaMemsetAsync(ws + L.grad_albedo, 0, albedo_grad_bytes(ad), st), "gradient reset");
  }
  return RCV_OK;
}

}  // namespace rcv

using namespace rcv;

extern "C" uint64_t rcv_medium_workspace_bytes(const int32_t dims[3], int32_t has_albedo_grid,
                                               int32_t majorant_factor) {
  if (dims == nullptr || dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0 || majorant_factor < 0) return 0;
  return medium_layout(dims, has_albedo_grid ? dims : nullptr, majorant_factor).total;
}

extern "C" uint64_t rcv_medium_workspace_bytes_for(const rcv_medium* m) {
  if (m == nullptr || m->dims[0] <= 0 || m->dims[1] <= 0 || m->dims[2] <= 0 || m->majorant_factor < 0) return 0;
  for (int a = 0; a < 3; ++a)
    if (m->albedo_dims[a] < 0) return 0;
  return medium_layout(m).total;
}

// Environment-map tables: one thread per row packs its texels with their
// sampling weight f = luminance * sin(theta of the row centre) and writes the
// row's conditional CDF from double prefix sums taken in order; then one
// thread writes the marginal CDF over the rows and the normalisation.
__global__ void env_rows_kernel(int w, int h, float inv_h, const float* __restrict__ texels, float4* __restrict__ tex,
                                float* __restrict__ cond, double* __restrict__ rows) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= h) return;
  const float sin_i = env_row_sin(i, inv_h);
  double sum = 0.0;
  for (int j = 0; j < w; ++j) {
    const float* t = texels + (int64_t(i) * w + j) * 3;
    const float f = env_luminance(t[0], t[1], t[2]) * sin_i;
    tex[int64_t(i) * w + j] = make_float4(t[0], t[1], t[2], f);
    sum += (double)f;
  }
  rows[i] = sum;
  float* c = cond + int64_t(i) * (w + 1);
  double acc = 0.0;
  for (int j = 0; j < w; ++j) {
    c[j] = sum > 0.0 ? (float)(acc / sum) : (float)((double)j / (double)w);
    acc += (double)tex[int64_t(i) * w + j].w;
  }
  c[w] = 1.0f;
}

__global__ void env_marginal_kernel(int w, int h, const double* __restrict__ rows, float* __restrict__ marg,
                                    float* __restrict__ hdr) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  double total = 0.0;
  for (int i = 0; i < h; ++i) total += rows[i];
  double acc = 0.0;
  for (int i = 0; i < h; ++i) {
    marg[i] = total > 0.0 ? (float)(acc / total) : (float)((double)i / (double)h);
    acc += rows[i];
  }
  marg[h] = 1.0f;
  hdr[0] = total > 0.0 ? (float)((double)w * (double)h / total) : 0.0f;
  hdr[1] = total > 0.0 ? 1.0f : 0.0f;
}

extern "C" uint64_t rcv_envmap_workspace_bytes(int32_t width, int32_t height) {
  if (width <= 0 || height <= 0) return 0;
  return env_layout(width, height).total;
}

extern "C" int rcv_envmap_prepare(const rcv_envmap* e, void* stream) {
  RCV_REQUIRE(e != nullptr && e->texels != nullptr, "environment map or its texels are NULL");
  RCV_REQUIRE(e->width > 0 && e->height > 0 && int64_t(e->width) * e->height < (int64_t(1) << 30),
              "environment map size must be positive and below 2^30 texels");
  RCV_REQUIRE(e->workspace != nullptr && (reinterpret_cast<uintptr_t>(e->workspace) & 255u) == 0,
              "environment map workspace must be non-NULL and 256-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const EnvLayout L = env_layout(e->width, e->height);
  char* ws = static_cast<char*>(e->workspace);
  env_rows_kernel<<<grid_for(e->height, 128), 128, 0, st>>>(
      e->width, e->height, 1.0f / (float)e->height, e->texels, reinterpret_cast<float4*>(ws + L.tex),
      reinterpret_cast<float*>(ws + L.cond), reinterpret_cast<double*>(ws + L.rows));
  int rc = launched("envmap rows launch");
  if (rc) return rc;
  env_marginal_kernel<<<1, 1, 0, st>>>(e->width, e->height, reinterpret_cast<const double*>(ws + L.rows),
                                       reinterpret_cast<float*>(ws + L.marg), reinterpret_cast<float*>(ws + L.hdr));
  return launched("envmap marginal launch");
}

extern "C" uint64_t rcv_render_workspace_bytes(int32_t width, int32_t height, int32_t spp,
                                               int32_t mode) {
  if (width <= 0 || height <= 0 || spp <= 0 || mode < 0 || mode > 2) return 0;
  const int64_t npix = int64_t(width) * height;
  return render_layout(npix, npix * spp, mode).total;
}

extern "C" uint64_t rcv_render_adjoint_workspace_bytes(int32_t width, int32_t height, int32_t spp,
                                                       const rcv_volpath_options* o) {
  if (width <= 0 || height <= 0 || spp <= 0) return 0;
  const int64_t npix = int64_t(width) * height, paths = npix * spp;
  const uint64_t forward = render_layout(npix, paths, kAdjoint, adjoint_room(paths, o, true)).total;
  const uint64_t backward = render_layout(npix, paths, kAdjoint, adjoint_room(paths, o, false)).total;
  return backward > forward ? backward : forward;
}

extern "C" int rcv_medium_prepare(const rcv_medium* m, void* stream) {
  int rc = validate_medium(m);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const MediumLayout L = medium_layout(m);
  char* ws = static_cast<char*>(m->workspace);
  RCV_TRY_CUDA(cudaMemsetAsync(ws + L.maxbits, 0, 16, st), "majorant reset");
  const int64_t nc = int64_t(m->dims[0] + 1) * (m->dims[1] + 1) * (m->dims[2] + 1);
  const int64_t na = (int64_t)albedo_voxels_of(m);
  const int block = 256;
  pack_medium_kernel<<<grid_for(nc > na ? nc : na, block), block, 0, st>>>(
      m->dims[0], m->dims[1], m->dims[2], m->density_old, m->density_new,
      reinterpret_cast<float4*>(ws + L.cells), m->albedo_old, m->albedo_new,
      m->albedo_old ? reinterpret_cast<float4*>(ws + L.albedo) : nullptr, na,
      reinterpret_cast<uint32_t*>(ws + L.maxbits));
  rc = launched("pack_medium launch");
  if (rc || m->majorant_factor == 0) return rc;
  const int sx = supergrid_cells(m->dims[0], m->majorant_factor);
  const int sy = supergrid_cells(m->dims[1], m->majorant_factor);
  const int sz = supergrid_cells(m->dims[2], m->majorant_factor);
  supergrid_kernel<<<grid_for(int64_t(sx) * sy * sz * 32, 128), 128, 0, st>>>(
      sx, sy, sz, m->dims[0], m->dims[1], m->dims[2], m->scale, m->density_old, m->density_new,
      reinterpret_cast<float*>(ws + L.sg_two), reinterpret_cast<float*>(ws + L.sg_new));
  return launched("supergrid launch");
}

// Adjoint stages: both launches, the radiance pass alone, or the replay alone
// (which reuses the pixel order, checkpoints and total radiance the radiance
// pass left in the same workspace).
enum AdjStage { kAdjBoth = 0, kAdjRadiance = 1, kAdjReplay = 2, kAdjForward = 3 };

static int check_workspace(const void* workspace) {
  RCV_REQUIRE(workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0,
              "render workspace must be non-NULL and 256-byte aligned");
  return RCV_OK;
}

// A job's pixel hand-out order (RCV_ORDER_*); jobs that sort their pixels are
// added to `sort` for order_pixels, which clears the head of their workspace
// (queue counters, order buckets); the others' is cleared here.  `keep`: the
// order and the counters are those that an earlier stage left there.
static int order_job(VolJob& J, const rcv_volpath_options* o, char* ws, const RenderLayout& L, bool keep,
                     OrderJob* sort, int* nsort, cudaStream_t st) {
  J.pixel_order = nullptr;
  J.pixel_cost = nullptr;
  const int order = o == nullptr ? RCV_ORDER_COST : o->order;
  RCV_REQUIRE(order == RCV_ORDER_COST || order == RCV_ORDER_ROW_MAJOR || order == RCV_ORDER_LONGEST_FIRST,
              "unknown pixel order %d", order);
  if (order == RCV_ORDER_ROW_MAJOR) {
    if (!keep) RCV_TRY_CUDA(cudaMemsetAsync(ws, 0, kRenderHeadBytes, st), "counters reset");
    return RCV_OK;
  }
  uint32_t* cost = order == RCV_ORDER_COST ? reinterpret_cast<uint32_t*>(ws + L.cost) : nullptr;
  if (!keep) {
    OrderJob& O = sort[(*nsort)++];
    O.J = J;
    O.head = ws;
    O.npix = J.width * J.height;
    O.buckets = reinterpret_cast<uint32_t*>(ws + L.buckets);
    O.order = reinterpret_cast<uint32_t*>(ws + L.order);
    O.cost = cost;
    O.chord = order == RCV_ORDER_LONGEST_FIRST;
  }
  J.pixel_order = reinterpret_cast<const uint32_t*>(ws + L.order);
  J.pixel_cost = cost;
  return RCV_OK;
}

// The gradient comes from the event tape (RCV_ADJOINT_TAPE), except in forward
// mode and for jobs of too many paths.
static bool uses_tape(const VolJob& J, const rcv_volpath_options* o, int stage) {
  return (o == nullptr || o->adjoint == RCV_ADJOINT_TAPE) && stage != kAdjForward && tape_fits(J.path_count);
}

// float4s of a job's density (or albedo) gradient records.
static int64_t gradient_float4s(const VolJob& J, bool albedo) {
  if (albedo) return J.grad_albedo != nullptr ? int64_t(J.adx + 1) * (J.ady + 1) * (J.adz + 1) * 6 : 0;
  return int64_t(J.dx + 1) * (J.dy + 1) * (J.dz + 1) * 2;
}

// Whether the tape's weights pass clears the gradient records: up to 64 MB,
// where the launches saved count; beyond, cudaMemsetAsync (256^3: the clear is
// bound by memory either way, 104 + 85 us apart and 184 together).
static bool clears_in_weights(const VolJob& J) {
  return gradient_float4s(J, false) + gradient_float4s(J, true) <= (int64_t(1) << 22);
}

// Adjoint buffers of a job in its workspace (queue counters at qc: hand-out,
// records, tape slots, lost paths).  *tape: the gradient comes from the tape.
static int adjoint_buffers(const VolJob& J, const rcv_volpath_options* o, char* ws, const RenderLayout& L,
                           const AdjRoom& room, unsigned long long* qc, int stage, AdjBuffers* out,
                           bool* tape_out) {
  AdjBuffers& A = *out;
  std::memset(&A, 0, sizeof(A));
  A.ckpt = reinterpret_cast<float4*>(ws + L.ckpt);
  A.ckpt_count = qc + 1;
  A.ckpt_cap = room.ckpts;
  A.path_ltot = reinterpret_cast<float4*>(ws + L.ltot);
  const int adjoint = o == nullptr ? RCV_ADJOINT_TAPE : o->adjoint;
  const int per_path = o == nullptr ? 0 : o->tape_events_per_path;
  RCV_REQUIRE(adjoint == RCV_ADJOINT_TAPE || adjoint == RCV_ADJOINT_REPLAY, "unknown adjoint %d", adjoint);
  RCV_REQUIRE(per_path >= 0 && per_path <= kTapeSlotsPerPath,
              "tape_events_per_path must be in [0, %d]", int(kTapeSlotsPerPath));
  const bool tape = uses_tape(J, o, stage);
  if (tape) {
    A.tape = reinterpret_cast<float4*>(ws + L.tape);
    A.tape_count = qc + 2;
    A.tape_cap = per_path > 0 ? tape_capacity(J.path_count, per_path) : room.slots;
    A.lost_list = reinterpret_cast<uint32_t*>(ws + L.lost);
    A.lost_count = qc + 3;
    A.tape_f = tape_terms(ws + L.tape, room.slots);
    A.cam_w = reinterpret_cast<float2*>(ws + L.cam_w);
    A.entered = reinterpret_cast<uint32_t*>(ws + L.entered);
    A.entered_count = qc + 5;
  }
  *tape_out = tape;
  if (tape && clears_in_weights(J)) {
    A.clear_cells = gradient_float4s(J, false);
    A.clear_albedo = gradient_float4s(J, true);
  }
  return RCV_OK;
}

// Orders the pixels, runs the persistent tracer of one job and, for the
// primal tracers, reduces the per-path radiance into the output image(s).
static int run_single_job(int mode, VolJob& J, const rcv_volpath_options* o, void* workspace,
                          uint64_t* counters, float* img_new, float* img_old, cudaStream_t st,
                          int stage = kAdjBoth) {
  int rc = check_workspace(workspace);
  if (rc) return rc;
  const int64_t npix = int64_t(J.width) * J.height;
  const AdjRoom room = adjoint_room(J.path_count, o, stage == kAdjForward);
  const RenderLayout L = render_layout(npix, J.path_count, mode, room);
  char* ws = static_cast<char*>(workspace);
  OrderJob sort[1];
  int nsort = 0;
  rc = order_job(J, o, ws, L, stage == kAdjReplay, sort, &nsort, st);
  if (rc == RCV_OK && nsort > 0) rc = order_pixels(sort, nsort, st);
  if (rc) return rc;
  float4* po = reinterpret_cast<float4*>(ws + L.path_out);
  unsigned long long* qc = reinterpret_cast<unsigned long long*>(ws + L.counter);
  if (mode == kAdjoint) {
    AdjBuffers A;
    bool tape = false;
    rc = adjoint_buffers(J, o, ws, L, room, qc, stage, &A, &tape);
    if (rc) return rc;
    if (stage != kAdjReplay) {
      rc = launch_persistent(tape ? kTape : kAdjoint, J, nullptr, 0, J.path_count, o, qc, nullptr, &A, counters,
                             st, false, true);
      if (rc || stage == kAdjRadiance) return rc;
    }
    if (tape) {
      // weights of the event records: the second half of the checkpoint buffer
      float4* weights = reinterpret_cast<float4*>(ws + L.ckpt + uint64_t(A.ckpt_cap) * 32u);
      rc = launch_tape_gradient(J, nullptr, 0, A, weights, qc + 4, counters, sm_count(), st);
      if (rc) return rc;
      // the paths whose events did not fit, replayed whole
    }
    return launch_persistent(stage == kAdjForward ? kForward : kReplay, J, nullptr, 0, J.path_count, o, qc + 4,
                             nullptr, &A, counters, st, false, tape);
  }
  rc = launch_persistent(mode, J, nullptr, 0, J.path_count, o, qc, po, nullptr, counters, st, false, true);
  if (rc) return rc;
  return launch_reduce(mode == kTwoState, po, 0, npix, J.spp, img_new, img_old, st);
}

extern "C" int rcv_render_twostates_volume(const rcv_medium* m, const rcv_sensor* s,
                                           const rcv_volpath_options* o, uint32_t seed,
                                           int32_t spp, float* img_old, float* img_new,
                                           void* workspace, uint64_t* counters, void* stream) {
  VolJob J;
  int rc = make_volume_job(m, s, o, seed, spp, &J);
  if (rc) return rc;
  RCV_REQUIRE(img_old != nullptr && img_new != nullptr, "output images are NULL");
  return run_single_job(kTwoState, J, o, workspace, counters, img_new, img_old,
                        static_cast<cudaStream_t>(stream));
}

extern "C" int rcv_render_volume(const rcv_medium* m, const rcv_sensor* s,
                                 const rcv_volpath_options* o, uint32_t seed, int32_t spp,
                                 float* img, void* workspace, uint64_t* counters, void* stream) {
  VolJob J;
  int rc = make_volume_job(m, s, o, seed, spp, &J);
  if (rc) return rc;
  RCV_REQUIRE(img != nullptr, "output image is NULL");
  return run_single_job(kSingle, J, o, workspace, counters, img, nullptr, static_cast<cudaStream_t>(stream));
}

// The two-state primal of (seed, spp) and the adjoint's radiance pass of
// (seed_grad, spp_grad) on the same medium: one persistent launch that runs
// both (rcv_pair.cu), where the two launches in a row would each end on
// their longest paths.  With event counting, the replay adjoint or
// separate_tracers the two run as separate launches.
extern "C" int rcv_render_twostates_volume_and_adjoint_radiance(
    const rcv_medium* m, const rcv_sensor* s, const rcv_volpath_options* o, uint32_t seed, int32_t spp,
    float* img_old, float* img_new, void* workspace, uint32_t seed_grad, int32_t spp_grad, void* adjoint_workspace,
    uint64_t* counters, void* stream) {
  VolJob JA, JB;
  int rc = make_volume_job(m, s, o, seed, spp, &JA);
  if (rc) return rc;
  rc = make_volume_job(m, s, o, seed_grad, spp_grad, &JB);
  if (rc) return rc;
  RCV_REQUIRE(img_old != nullptr && img_new != nullptr, "output images are NULL");
  RCV_REQUIRE(workspace != adjoint_workspace, "the render and the adjoint need separate workspaces");
  RCV_REQUIRE(o == nullptr || o->separate_tracers == 0 || o->separate_tracers == 1,
              "separate_tracers must be 0 or 1");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = check_workspace(workspace);
  if (rc == RCV_OK) rc = check_workspace(adjoint_workspace);
  if (rc) return rc;
  const int64_t npix = int64_t(JA.width) * JA.height;
  const RenderLayout LA = render_layout(npix, JA.path_count, kTwoState);
  const AdjRoom room = adjoint_room(JB.path_count, o, false);
  const RenderLayout LB = render_layout(npix, JB.path_count, kAdjoint, room);
  char* wa = static_cast<char*>(workspace);
  char* wb = static_cast<char*>(adjoint_workspace);
  unsigned long long* qa = reinterpret_cast<unsigned long long*>(wa + LA.counter);
  unsigned long long* qb = reinterpret_cast<unsigned long long*>(wb + LB.counter);
  AdjBuffers A;
  bool tape = false;
  rc = adjoint_buffers(JB, o, wb, LB, room, qb, kAdjRadiance, &A, &tape);
  if (rc) return rc;
  if (counters != nullptr || !tape || (o != nullptr && o->separate_tracers)) {
    rc = run_single_job(kTwoState, JA, o, workspace, counters, img_new, img_old, st);
    if (rc) return rc;
    return run_single_job(kAdjoint, JB, o, adjoint_workspace, counters, nullptr, nullptr, st, kAdjRadiance);
  }
  OrderJob sort[2];
  int nsort = 0;
  rc = order_job(JA, o, wa, LA, false, sort, &nsort, st);
  if (rc == RCV_OK) rc = order_job(JB, o, wb, LB, false, sort, &nsort, st);
  if (rc == RCV_OK && nsort > 0) rc = order_pixels(sort, nsort, st);
  if (rc) return rc;
  float4* po = reinterpret_cast<float4*>(wa + LA.path_out);
  Queue QA, QB;
  rc = make_queue(kTwoState, nullptr, 0, JA.path_count, o, qa, po, nullptr, nullptr, st, &QA, true);
  if (rc == RCV_OK) rc = make_queue(kTape, nullptr, 0, JB.path_count, o, qb, nullptr, &A, nullptr, st, &QB, true);
  if (rc == RCV_OK) rc = launch_pair(JA, QA, JB, QB, o, st, false);
  if (rc) return rc;
  return launch_reduce(true, po, 0, npix, JA.spp, img_new, img_old, st);
}

static int backward_volume(const rcv_medium* m, const rcv_sensor* s, const rcv_volpath_options* o, uint32_t seed,
                           int32_t spp, const float* grad_img, float* grad_density, float* grad_albedo,
                           void* workspace, uint64_t* counters, void* stream, int stage) {
  VolJob J;
  int rc = make_volume_job(m, s, o, seed, spp, &J);
  if (rc) return rc;
  RCV_REQUIRE(grad_img != nullptr && grad_density != nullptr, "gradient buffers are NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool want_albedo = grad_albedo != nullptr && m->albedo_old != nullptr;
  if (!want_albedo) J.grad_albedo = nullptr;
  if (!uses_tape(J, o, stage) || !clears_in_weights(J)) {  // else the tape's weights pass clears them
    rc = reset_gradients(m, want_albedo, st);
    if (rc) return rc;
  }
  J.grad_img = grad_img;
  rc = run_single_job(kAdjoint, J, o, workspace, counters, nullptr, nullptr, st, stage);
  if (rc) return rc;
  return launch_fold(m, grad_density, want_albedo ? grad_albedo : nullptr, st);
}

extern "C" int rcv_render_backward_volume(const rcv_medium* m, const rcv_sensor* s,
                                          const rcv_volpath_options* o, uint32_t seed,
                                          int32_t spp, const float* grad_img,
                                          float* grad_density, float* grad_albedo,
                                          void* workspace, uint64_t* counters, void* stream) {
  return backward_volume(m, s, o, seed, spp, grad_img, grad_density, grad_albedo, workspace, counters, stream,
                         kAdjBoth);
}

extern "C" int rcv_render_forward_volume(const rcv_medium* m, const rcv_sensor* s,
                                         const rcv_volpath_options* o, uint32_t seed, int32_t spp,
                                         const float* tangent_density, const float* tangent_albedo,
                                         float* dimg, void* workspace, uint64_t* counters, void* stream) {
  VolJob J;
  int rc = make_volume_job(m, s, o, seed, spp, &J);
  if (rc) return rc;
  RCV_REQUIRE(dimg != nullptr, "output derivative image is NULL");
  RCV_REQUIRE(tangent_density != nullptr || tangent_albedo != nullptr, "no tangent given");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // the medium's gradient records hold the packed tangent during the call
  const MediumLayout L = medium_layout(m);
  char* ws = static_cast<char*>(m->workspace);
  const int64_t nc = int64_t(m->dims[0] + 1) * (m->dims[1] + 1) * (m->dims[2] + 1);
  const int block = 256;
  if (tangent_density != nullptr) {
    pack_tangent_kernel<<<grid_for(nc, block), block, 0, st>>>(m->dims[0], m->dims[1], m->dims[2],
                                                               tangent_density,
                                                               reinterpret_cast<float4*>(ws + L.grad_cells));
    rc = launched("pack_tangent launch");
    if (rc) return rc;
  } else {
    RCV_TRY_CUDA(cudaMemsetAsync(ws + L.grad_cells, 0, nc * 32, st), "tangent reset");
  }
  const bool albedo = tangent_albedo != nullptr && m->albedo_old != nullptr;
  if (albedo) {
    const int64_t na = (int64_t)albedo_voxels_of(m);
    pack_tangent_albedo_kernel<<<grid_for(na, block), block, 0, st>>>(
        na, tangent_albedo, reinterpret_cast<float4*>(ws + L.grad_albedo));
    rc = launched("pack_tangent_albedo launch");
    if (rc) return rc;
  } else {
    J.grad_albedo = nullptr;
  }
  RCV_TRY_CUDA(cudaMemsetAsync(dimg, 0, size_t(J.width) * J.height * 3 * sizeof(float), st), "derivative reset");
  J.out_img = dimg;
  return run_single_job(kAdjoint, J, o, workspace, counters, nullptr, nullptr, st, kAdjForward);
}

extern "C" int rcv_render_adjoint_radiance(const rcv_medium* m, const rcv_sensor* s,
                                           const rcv_volpath_options* o, uint32_t seed, int32_t spp,
                                           void* workspace, uint64_t* counters, void* stream) {
  VolJob J;
  int rc = make_volume_job(m, s, o, seed, spp, &J);
  if (rc) return rc;
  return run_single_job(kAdjoint, J, o, workspace, counters, nullptr, nullptr, static_cast<cudaStream_t>(stream),
                        kAdjRadiance);
}

extern "C" int rcv_render_backward_replay(const rcv_medium* m, const rcv_sensor* s,
                                          const rcv_volpath_options* o, uint32_t seed, int32_t spp,
                                          const float* grad_img, float* grad_density, float* grad_albedo,
                                          void* workspace, uint64_t* counters, void* stream) {
  return backward_volume(m, s, o, seed, spp, grad_img, grad_density, grad_albedo, workspace, counters, stream,
                         kAdjReplay);
}

// ------------------------------------------------- allocation-free render
// Single-state render for callers that cannot allocate device memory: code
// running where cudaMalloc is unavailable or forbidden, such as a host that
// owns a fixed memory pool and hands this library only its inputs and
// outputs, or a real-time loop that may not allocate between frames.  Its
// scratch (work-queue counter, pixel order, per-path radiance) lives in this
// file-scope array instead of a caller buffer.  Every GPU that loads librcv
// holds the array until the process exits.
namespace rcv {

constexpr uint64_t kNoAllocScratchBytes = uint64_t(16) << 20;  // 16 MiB
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Device address of g_noalloc_scratch on the current device.  In host code the
// symbol is only a host-side stand-in, so the address is looked up once per
// device (with that device current) and cached.  The cached address belongs to
// the device's primary context; a cudaDeviceReset ends its validity, which is
// why callers may not use the entry point on that device afterwards.
static int noalloc_scratch(void** out) {
  static std::mutex mu;
  static void* addr[kNoAllocMaxDevices] = {};
  int dev = 0;
  RCV_TRY_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
  RCV_REQUIRE(dev >= 0 && dev < kNoAllocMaxDevices, "device ordinal %d is not supported", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (addr[dev] == nullptr) {
    void* p = nullptr;
    RCV_TRY_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch), "cudaGetSymbolAddress(scratch)");
    addr[dev] = p;
  }
  *out = addr[dev];
  return RCV_OK;
}

}  // namespace rcv

extern "C" int rcv_render_volume_noalloc(const rcv_medium* m, const rcv_sensor* s,
                                         const rcv_volpath_options* o, uint32_t seed, int32_t spp,
                                         float* img, uint64_t* counters, void* stream) {
  VolJob J;
  int rc = make_volume_job(m, s, o, seed, spp, &J);
  if (rc) return rc;
  RCV_REQUIRE(img != nullptr, "output image is NULL");
  const uint64_t need = render_layout(int64_t(J.width) * J.height, J.path_count, kSingle).total;
  RCV_REQUIRE(need <= kNoAllocScratchBytes,
              "rcv_render_volume_noalloc: width*height*spp = %lld needs %llu bytes of scratch, "
              "more than its static %llu bytes (16 MiB); use rcv_render_volume with caller scratch",
              (long long)J.path_count, (unsigned long long)need,
              (unsigned long long)kNoAllocScratchBytes);
  void* ws = nullptr;
  rc = noalloc_scratch(&ws);
  if (rc) return rc;
  return run_single_job(kSingle, J, o, ws, counters, img, nullptr, static_cast<cudaStream_t>(stream));
}
