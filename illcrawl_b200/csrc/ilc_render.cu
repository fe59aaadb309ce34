// ilc_render.cu -- line-of-sight projection over the camera plane: the whole
// parallel_runge_kutta_fehlberg host loop (integration.cpp:84-307,
// volumetric_integration.cpp:32-88) as one kernel launch.
//
// Four lanes own one pixel's integrator and run its RKF4(5) steps to the end of
// the ray, one lane per integrand point (ilc_raylist.cuh); steps that are long
// against a cell are walked one ray per thread (ilc_walk4.cuh): fixed ones by a
// rule on the launch, adaptive ones as far as each ray's steps stay long. A ray's
// state depends only on its own evaluations, so this is the same computation as
// the reference's lock-step loop with stream compaction, without its
// per-iteration host synchronisations.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "ilc_device.cuh"
#include "ilc_internal.h"
#include "ilc_raylist.cuh"
#include "ilc_walk4.cuh"

namespace ilc {

GridView make_grid_view(const Context& c) {
  GridView g;
  std::memset(&g, 0, sizeof(g));  // padding too: the bytes key the batched launch graph
  g.min0 = c.gp.min[0]; g.min1 = c.gp.min[1]; g.min2 = c.gp.min[2];
  g.cs0 = c.gp.cs[0]; g.cs1 = c.gp.cs[1]; g.cs2 = c.gp.cs[2];
  g.half0 = 0.5f * c.gp.cs[0]; g.half1 = 0.5f * c.gp.cs[1]; g.half2 = 0.5f * c.gp.cs[2];
  g.cell_radius = 0.5f * sqrtf((c.gp.cs[0] * c.gp.cs[0] + c.gp.cs[1] * c.gp.cs[1]) +
                               c.gp.cs[2] * c.gp.cs[2]);
  g.n0 = c.gp.n[0]; g.n1 = c.gp.n[1]; g.n2 = c.gp.n[2];
  g.cells = c.cells.as<int2>();
  g.parts = c.parts.as<float4>();
  g.codes = c.codes.as<uint16_t>();
  g.inv_w0 = 16.0f / c.gp.cs[0];
  g.inv_w1 = 16.0f / c.gp.cs[1];
  g.inv_w2 = 16.0f / c.gp.cs[2];
  // slack for the float rounding of cell keys and cell boxes: a 1024th of a
  // cell, and at least 8 ulp of the largest coordinate of the grid
  float ext = 0.0f;
  for (int k = 0; k < 3; ++k)
    ext = std::fmax(ext, std::fmax(std::fabs(c.gp.min[k]),
                                   std::fabs(c.gp.min[k] + (float)c.gp.n[k] * c.gp.cs[k])));
  g.margin = std::fmax(std::fmax(std::fmax(c.gp.cs[0], c.gp.cs[1]), c.gp.cs[2]) / 1024.0f,
                       ext * 9.5367431640625e-07f);
  return g;
}

namespace {

struct RenderK {
  CamView cam;
  float z0, z_end;
  double atol, rtol;
  int controller;
  int64_t fixed_steps;
  float fixed_h;
  const float* replay_h;    // frozen per-ray sequences (ray-major, rec_cap each)
  const int32_t* replay_n;  // steps per ray
  int64_t max_steps;
  int row_stride;   // render every row_stride-th row of tiles (1 = all)
  int row0;         // first pixel row (a multiple of the tile height)
  int row_end;      // one past the last pixel row
  float* rec_h;     // optional: accepted step sizes per ray (ray-major, rec_cap each)
  int32_t* rec_n;   // optional: number of accepted steps per ray
  int64_t rec_cap;
  float scale;
  int apply_scale;
  float* out;
  double* out_d;        // optional (frozen replay): the line integrals summed in double
  uint64_t* ray_stats;  // optional: per ray (steps, accepted, cells visited, candidates)
  unsigned long long* queue;  // ray counter
  unsigned long long n_rays;  // 128 per 16 x 8 tile
  unsigned tiles_x;
  float4* over;               // list overflow, kOver per resident ray
  LeaveRule leave;            // rays walked first, and those left to the lists
};

constexpr int kRenderBlocks = 4;  // per SM, by registers and shared memory
constexpr int kTileX = 16, kTileY = 8;

struct RenderMem {
  char4 spiral[1000];
  WarpLists lists[kListWarps];
};

// Pixel of ray q: 16 x 8 pixel tiles row by row, 4 x 2 pixels of a tile in a
// row of 8 rays, so a warp's rays start as neighbours.
__device__ __forceinline__ void ray_pixel(const RenderK& a, unsigned long long q, int& ix,
                                          int& iy) {
  const unsigned tile = (unsigned)(q >> 7), t = (unsigned)(q & 127u);
  const int bx = (int)(tile % a.tiles_x), by = (int)(tile / a.tiles_x);
  const int sub = (int)(t >> 3);  // 4 x 4 blocks of 4 x 2 pixels
  ix = bx * kTileX + (sub & 3) * 4 + (int)(t & 3u);
  iy = a.row0 + by * a.row_stride * kTileY + (sub >> 2) * 2 + (int)((t >> 2) & 1u);
}

// Every group of 4 lanes (one per integrand point) takes the next ray of the
// queue when its ray has ended. Modes: frozen per-ray sequences, uniform
// frozen steps, adaptive with either controller.
__global__ void __launch_bounds__(kListThreads, kRenderBlocks)
render_kernel(const __grid_constant__ RenderK a, const __grid_constant__ GridView g,
              const char4* __restrict__ spiral_g, uint32_t* __restrict__ flags,
              unsigned long long* __restrict__ stats) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RenderMem& M = *reinterpret_cast<RenderMem*>(smem_raw);
  load_spiral(M.spiral, spiral_g);
  const int lane = threadIdx.x & 31;
  const int r = lane >> 2, pj = lane & 3;
  WarpLists& W = M.lists[threadIdx.x >> 5];
  const unsigned wg = blockIdx.x * kListWarps + (threadIdx.x >> 5);
  if (lane == 0) W.over = a.over + (size_t)wg * kRays * kOver;
  const float ext0 = 0.06f * g.cs0;
  const float lx = a.cam.look0, ly = a.cam.look1, lz = a.cam.look2;
  const float fa = (float)a.atol, fr = (float)a.rtol;
  bool have = false, drained = false, fresh = true;
  int ix = 0, iy = 0;
  float px = 0.0f, py = 0.0f, pz = 0.0f;
  float I = 0.0f, z = 0.0f, h = 1.0f, k1 = 0.0f;
  double Id = 0.0;  // out_d: the same increments summed in double
  int64_t lray = 0, limit = 0;
  const float* hs = nullptr;
  unsigned long long steps = 0, acc = 0;
  WalkStats ws;
  for (;;) {
    for (;;) {
      const unsigned want = __ballot_sync(kAll, !have && !drained && pj == 0);
      if (!want) break;
      const unsigned long long q = take_rays(a.queue, want, fresh, lane, wg);
      fresh = false;
      if (!have && !drained) {
        drained = q >= list_rays(a.leave, a.n_rays);
        if (!drained) {
          ray_pixel(a, list_ray(a.leave, q), ix, iy);
          have = ix < a.cam.nx && iy < a.row_end;
        }
        if (have) {
          // per-ray arrays are indexed from the launch's first row
          lray = (int64_t)(iy - a.row0) * a.cam.nx + ix;
          pixel_corner(a.cam, ix, iy, px, py, pz);
          I = 0.0f;
          Id = 0.0;
          k1 = 0.0f;
          z = a.z0;
          h = a.fixed_steps > 0 ? a.fixed_h : 1.0f;
          steps = acc = 0;
          limit = a.max_steps;
          if (a.replay_h) {
            const int64_t nr = a.replay_n[lray];
            limit = nr < 0 ? 0 : (nr > a.rec_cap ? a.rec_cap : nr);
            hs = a.replay_h + lray * a.rec_cap;
          } else if (a.fixed_steps > 0) {
            limit = a.fixed_steps;
          }
          if (pj == 0) ray_reset(W.meta[r], ext0);
        }
      }
      __syncwarp();
    }
    if (!__any_sync(kAll, have)) break;
    const bool frozen = a.replay_h || a.fixed_steps > 0;
    const bool go = have && (int64_t)steps < limit && (frozen || z < a.z_end);
    if (go && a.replay_h) h = hs[steps];
    const float zq = step_point(z, h, pj);
    PointSlots s;
    eval_points<false>(g, M.spiral, W, lane, go, px, py, pz, lx, ly, lz, zq, h, s, ws);
    float e[4];
    share4(go ? slots_value(s) : 0.0f, lane, e);
    if (go) {
      if (frozen) {
        // every step accepted, I += delta4
        float d4 = 25.f / 216.f * k1 + 1408.f / 2565.f * e[0] + 2197.f / 4101.f * e[1] -
                   1.f / 5.f * e[2];
        d4 *= h;
        I = I + d4;
        if (a.out_d) Id += (double)d4;
        z += h;
        k1 = e[2];
        ++steps;
        ++acc;
      } else {
        const float zb = z, hb = h;
        float next[4];
        if (a.controller == ILC_CONTROLLER_REF32)
          rkf_advance_ref32(I, z, h, k1, fa, fr, a.z_end, e, kEps, kHmin, kHmax, next);
        else
          rkf_advance_fp64(I, z, h, k1, a.atol, a.rtol, a.z_end, e, kEps, kHmin, kHmax, next);
        ++steps;
        if (z != zb) {
          if (pj == 0 && a.rec_h && (int64_t)acc < a.rec_cap)
            a.rec_h[lray * a.rec_cap + (int64_t)acc] = hb;
          ++acc;
        }
      }
    }
    const bool more = (int64_t)steps < limit;
    const bool fin = have && (!go || (frozen ? !more : !(z < a.z_end)));
    if (__any_sync(kAll, fin)) {
      // the ray's search counters over its 4 lanes
      unsigned long long cells = ws.cells, cands = ws.cands;
#pragma unroll
      for (int off = 1; off < 4; off <<= 1) {
        cells += __shfl_xor_sync(kAll, cells, off);
        cands += __shfl_xor_sync(kAll, cands, off);
      }
      if (fin) {
        if (pj == 0) {
          const size_t pix = (size_t)iy * a.cam.nx + ix;
          if (a.out) a.out[pix] = a.apply_scale ? I * a.scale : I;
          if (a.out_d) a.out_d[pix] = a.apply_scale ? Id * (double)a.scale : Id;
          if (!frozen && a.rec_n) {
            a.rec_n[lray] = (int32_t)min((int64_t)acc, a.rec_cap);
            if ((int64_t)acc > a.rec_cap) atomicOr(flags, FLAG_REC_OVERFLOW);
          }
          if (a.ray_stats) {
            uint64_t* q = a.ray_stats + 4 * lray;
            q[0] = steps;
            q[1] = acc;
            q[2] = cells;
            q[3] = cands;
          }
          const bool at_limit = !frozen && z < a.z_end;
          if (at_limit) atomicOr(flags, FLAG_STEP_LIMIT);
          atomicAdd(&stats[0], steps);
          atomicAdd(&stats[1], acc);
          atomicAdd(&stats[2], 4ull * steps);
          atomicAdd(&stats[3], cells);
          atomicAdd(&stats[4], cands);
          atomicMax(&stats[5], steps);
          atomicAdd(&stats[6], at_limit ? 1ull : 0ull);
        }
        ws.cells = 0;
        ws.cands = 0;
        have = false;
      }
    }
    __syncwarp();
  }
}

// The rays of one tile, a ray per thread, every step walked from scratch for its 4
// points together (ilc_walk4.cuh). kFixed: uniform frozen steps; otherwise frozen
// per-ray sequences or adaptive steps, as in render_kernel, and rays whose steps
// suit the lists are left.
template <bool kFixed>
__device__ __forceinline__ void walk_tile(const RenderK& a, const GridView& g,
                                          const char4* __restrict__ spiral, SlotMem& slot_mem,
                                          uint32_t* __restrict__ flags,
                                          unsigned long long* __restrict__ stats,
                                          unsigned long long tile) {
  const unsigned long long q = 128 * tile + walk_ray();
  int ix, iy;
  ray_pixel(a, q, ix, iy);
  const bool active = ix < a.cam.nx && iy < a.row_end;
  Walk4Stats ws;
  unsigned long long steps = 0, acc = 0, at_limit = 0;
  bool leave = false;
  if (active) {
    float px, py, pz, pts[4];
    pixel_corner(a.cam, ix, iy, px, py, pz);
    const int64_t lray = (int64_t)(iy - a.row0) * a.cam.nx + ix;  // in the launch's rows
    float I = 0.0f, z = a.z0, h = kFixed ? a.fixed_h : 1.0f, k1 = 0.0f;
    const float fa = (float)a.atol, fr = (float)a.rtol;
    double Id = 0.0;  // out_d: the same increments summed in double
    const bool frozen = kFixed || a.replay_h;
    int64_t limit = kFixed ? a.fixed_steps : a.max_steps;
    const float* hs = nullptr;
    if (!kFixed && a.replay_h) {
      const int64_t nr = a.replay_n[lray];
      limit = nr < 0 ? 0 : (nr > a.rec_cap ? a.rec_cap : nr);
      hs = a.replay_h + lray * a.rec_cap;
    }
    Pace pace = pace_start(z);
    while ((int64_t)steps < limit && (frozen || z < a.z_end)) {
      if (!kFixed && hs) h = hs[steps];
      ws.scans = 0;
      rkf_points(z, h, pts);
      float e[4];
      nn8_step4<false>(g, spiral, slot_mem, px, py, pz, a.cam.look0, a.cam.look1, a.cam.look2,
                       pts, e, ws);
      ++steps;
      if (frozen) {
        // every step accepted, I += delta4
        float d4 = 25.f / 216.f * k1 + 1408.f / 2565.f * e[0] + 2197.f / 4101.f * e[1] -
                   1.f / 5.f * e[2];
        d4 *= h;
        I = I + d4;
        if (a.out_d) Id += (double)d4;
        z += h;
        k1 = e[2];
        ++acc;
      } else {
        const float zb = z, hb = h;
        if (a.controller == ILC_CONTROLLER_REF32)
          rkf_advance_ref32(I, z, h, k1, fa, fr, a.z_end, e, kEps, kHmin, kHmax, pts);
        else
          rkf_advance_fp64(I, z, h, k1, a.atol, a.rtol, a.z_end, e, kEps, kHmin, kHmax, pts);
        if (z != zb) {
          if (a.rec_h && (int64_t)acc < a.rec_cap)
            a.rec_h[lray * a.rec_cap + (int64_t)acc] = hb;
          ++acc;
        }
      }
      if (!kFixed && a.leave.left &&
          pace_slow(pace, a.leave, z, a.z_end, h, steps, ws.scans) &&
          (int64_t)steps < limit && (frozen || z < a.z_end)) {
        leave = true;
        break;
      }
    }
    if (leave) {
      steps = acc = 0;
      ws = Walk4Stats();
    } else {
      const size_t pix = (size_t)iy * a.cam.nx + ix;
      if (a.out) a.out[pix] = a.apply_scale ? I * a.scale : I;
      if (a.out_d) a.out_d[pix] = a.apply_scale ? Id * (double)a.scale : Id;
      if (!frozen && a.rec_n) {
        a.rec_n[lray] = (int32_t)min((int64_t)acc, a.rec_cap);
        if ((int64_t)acc > a.rec_cap) atomicOr(flags, FLAG_REC_OVERFLOW);
      }
      if (a.ray_stats) {
        uint64_t* rs = a.ray_stats + 4 * lray;
        rs[0] = steps;
        rs[1] = acc;
        rs[2] = ws.cells;
        rs[3] = ws.cands;
      }
      if (!frozen && z < a.z_end) {
        at_limit = 1;
        atomicOr(flags, FLAG_STEP_LIMIT);
      }
    }
  }
  const int lane = threadIdx.x & 31;
  if (!kFixed && a.leave.left) mark_left(a.leave, active, leave, q, lane);
  unsigned long long cells = ws.cells, cands = ws.cands, sum = steps, most = steps;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    cells += __shfl_xor_sync(kAll, cells, off);
    cands += __shfl_xor_sync(kAll, cands, off);
    sum += __shfl_xor_sync(kAll, sum, off);
    acc += __shfl_xor_sync(kAll, acc, off);
    at_limit += __shfl_xor_sync(kAll, at_limit, off);
    most = max(most, __shfl_xor_sync(kAll, most, off));
  }
  if (lane == 0) {
    atomicAdd(&stats[0], sum);
    atomicAdd(&stats[1], acc);
    atomicAdd(&stats[2], 4ull * sum);
    atomicAdd(&stats[3], cells);
    atomicAdd(&stats[4], cands);
    atomicMax(&stats[5], most);
    if (at_limit) atomicAdd(&stats[6], at_limit);
  }
}

// The resident blocks take tiles row by row from the queue until none is left.
template <bool kFixed>
__global__ void __launch_bounds__(kSlotThreads, kRenderBlocks)
walk_kernel(const __grid_constant__ RenderK a, const __grid_constant__ GridView g,
            const char4* __restrict__ spiral_g, uint32_t* __restrict__ flags,
            unsigned long long* __restrict__ stats) {
  __shared__ char4 spiral[1000];
  __shared__ SlotMem slot_mem;
  __shared__ unsigned long long next_tile;
  load_spiral(spiral, spiral_g);
  for (;;) {
    if (threadIdx.x == 0) next_tile = atomicAdd(a.queue + 1, 1ull);
    __syncthreads();
    const unsigned long long t = next_tile;
    __syncthreads();
    if (128 * t >= a.n_rays) break;
    walk_tile<kFixed>(a, g, spiral, slot_mem, flags, stats, t);
  }
}

}  // namespace

// Fixed steps of a length h that is not small against a cell leave few steps per
// candidate list, and many neighbouring rays fill the warps of a plain walk: then
// the walk of every step, one ray per thread, is the faster one. Its time hardly
// grows up to some 16,000 rays (its slowest warp sets it), the lists' time grows
// with the rays and falls with the steps per list. Lists / walk in ms (1,048,576
// cells of 118 kpc, 6 Mpc, NFW core): 50^2 rays with 16 / 256 / 2048 steps 1.4 /
// 8.5 / 23 against 5.0 / 39 / 261; 200^2 11.6 / 57 / 125 against 6.1 / 51 / 329;
// 400^2 33 / 157 / 391 against 7.8 / 65 / 420; 1024^2 200 / 948 / 2371 against
// 22 / 185 / 1304. With 20,000 cells the slowest warp is shorter and the walk is
// ahead from half as many rays (150^2, 32 steps: 9.3 against 4.7 ms).
//
// Adaptive rays leave the walk below that length, with the rays that are still
// under way for the rays (LeaveRule).
LeaveRule walk_rule(Context& c, double rays, unsigned long long n_rays,
                    unsigned long long* queue) {
  const double cell = ((double)c.gp.cs[0] + c.gp.cs[1] + c.gp.cs[2]) / 3.0;
  const double line = 16384.0 * std::fmin(1.0, std::pow((double)c.n_particles / 1048576.0, 0.19));
  LeaveRule r;
  std::memset(&r, 0, sizeof(r));  // padding too: the bytes key the batched launch graph
  r.even = (float)(0.28 * cell * line);
  r.line = (float)line;
  r.least = (float)(0.01 * cell);
  if (!(rays > kWalkRays * line) || n_rays > 0xffffffffull) return r;
  const size_t marks = ((size_t)n_rays / 8 + 15) / 16 * 16;
  if (c.rays_left.ensure(marks + 4 * (size_t)n_rays) != cudaSuccess) {
    cudaGetLastError();  // (all rays take lists then)
    return r;
  }
  r.rays = (float)rays;
  r.n_marks = n_rays;
  r.done = queue + 2;
  r.n_left = reinterpret_cast<uint32_t*>(queue + 3);
  r.left = c.rays_left.as<uint8_t>();
  r.list = c.rays_left.as<uint32_t>() + marks / 4;
  return r;
}

namespace {

// The numbers of the marked rays in their order, by one block: 4 us for 65,536 rays,
// 11 us for 1,048,576.
constexpr int kCompact = 1024;
__global__ void __launch_bounds__(kCompact)
left_list_kernel(const uint32_t* __restrict__ marks, uint32_t words, uint32_t* __restrict__ list,
                 uint32_t* __restrict__ n_left) {
  __shared__ uint32_t part[32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t base = 0;
  for (uint32_t w0 = 0; w0 < words; w0 += 4 * kCompact) {
    uint32_t m[4], n = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const uint32_t w = w0 + 4 * threadIdx.x + k;
      m[k] = w < words ? marks[w] : 0u;
      n += __popc(m[k]);
    }
    if (!__syncthreads_or((int)n)) continue;
    const uint32_t incl = (uint32_t)warp_inclusive((int)n, (int)lane);
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    const uint32_t below = (uint32_t)warp_inclusive((int)part[lane], (int)lane);
    uint32_t at = base + incl - n + (warp ? __shfl_sync(kAll, below, warp - 1) : 0u);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      for (uint32_t b = m[k]; b; b &= b - 1)
        list[at++] = 32 * (w0 + 4 * threadIdx.x + k) + __ffs(b) - 1;
    }
    base += __shfl_sync(kAll, below, 31);
    __syncthreads();
  }
  if (threadIdx.x == 0) *n_left = base;
}

}  // namespace

cudaError_t left_list_launch(Context& c, const LeaveRule& r) {
  left_list_kernel<<<1, kCompact, 0, c.stream>>>(reinterpret_cast<const uint32_t*>(r.left),
                                                 (uint32_t)(r.n_marks / 32), r.list, r.n_left);
  return cudaGetLastError();
}

cudaError_t render_residency(int occ, int* id) {
  cudaError_t e;
  int lists = 0, walk = 0;
  if ((e = cudaFuncSetAttribute(render_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(RenderMem))) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&lists, render_kernel, kListThreads,
                                                         sizeof(RenderMem))) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&walk, walk_kernel<false>,
                                                         kSlotThreads, 0)))
    return e;
  *id = occ > 0 ? 64 * std::min(lists, occ) + std::min(walk, occ) : 64 * lists + walk;
  return cudaSuccess;
}

cudaError_t render_launch(Context& c, const RenderArgs& a, float* kernel_ms) {
  cudaError_t e;
  if ((e = c.flags.ensure(kFlagsBytes))) return e;
  if ((e = cudaMemsetAsync(c.flags.p, 0, kFlagsBytes, c.stream))) return e;
  RenderK k;
  k.cam.look0 = a.cam[0]; k.cam.look1 = a.cam[1]; k.cam.look2 = a.cam[2];
  k.cam.b00 = a.cam[3]; k.cam.b01 = a.cam[4]; k.cam.b02 = a.cam[5];
  k.cam.b10 = a.cam[6]; k.cam.b11 = a.cam[7]; k.cam.b12 = a.cam[8];
  k.cam.min0 = a.cam[9]; k.cam.min1 = a.cam[10]; k.cam.min2 = a.cam[11];
  k.cam.ps = a.cam[12];
  k.cam.nx = a.nx; k.cam.ny = a.ny;
  k.z0 = a.z0; k.z_end = a.z_end;
  k.atol = a.atol; k.rtol = a.rtol;
  k.controller = a.controller;
  k.fixed_steps = a.fixed_steps;
  k.fixed_h = a.fixed_h;
  k.replay_h = a.replay_h;
  k.replay_n = a.replay_n;
  k.max_steps = c.max_steps;
  k.row_stride = a.row_stride > 1 ? a.row_stride : 1;
  k.row0 = a.row0;
  k.row_end = a.rows > 0 ? std::min(a.ny, a.row0 + a.rows) : a.ny;
  k.rec_h = a.rec_h;
  k.rec_n = a.rec_n;
  k.rec_cap = a.rec_cap;
  k.scale = a.scale;
  k.apply_scale = a.apply_scale ? 1 : 0;
  k.out = a.out;
  k.out_d = a.out_d;
  k.ray_stats = a.ray_stats;
  const GridView g = make_grid_view(c);
  const int tile_rows = (k.row_end - k.row0 + kTileY - 1) / kTileY;
  k.tiles_x = (unsigned)((a.nx + kTileX - 1) / kTileX);
  const unsigned long long tiles =
      (unsigned long long)k.tiles_x * (unsigned)((tile_rows + k.row_stride - 1) / k.row_stride);
  k.n_rays = 128ull * tiles;
  if ((e = c.tile_queue.ensure(256))) return e;
  if ((e = cudaMemsetAsync(c.tile_queue.p, 0, kQueueBytes, c.stream))) return e;
  k.queue = c.tile_queue.as<unsigned long long>();
  // fixed steps: walk or lists; otherwise a walk of many rays and lists for those it leaves
  const bool fixed = a.fixed_steps > 0 && !a.replay_h;
  const double rays = (double)a.nx * (double)(k.row_end - k.row0) / (double)k.row_stride;
  k.leave = walk_rule(c, fixed ? 0.0 : rays, k.n_rays, k.queue);
  c.leave = k.leave;
  const bool walks =
      fixed ? (rays - k.leave.line) * a.fixed_h > k.leave.even : k.leave.left != nullptr;
  const bool lists = !fixed || !walks;
  // as many blocks as are resident, or `occ` per SM
  const int occ = a.occupancy_override >= 0 ? a.occupancy_override : c.render_occupancy;
  const auto walker = fixed ? walk_kernel<true> : walk_kernel<false>;
  int sms = 0, per_sm = 0, per_sm_w = 0;
  if ((e = cudaFuncSetAttribute(render_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(RenderMem))) ||
      (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device)) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_w, walker, kSlotThreads, 0)) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, render_kernel, kListThreads,
                                                         sizeof(RenderMem))))
    return e;
  if (occ > 0) {
    per_sm = std::min(per_sm, occ);
    per_sm_w = std::min(per_sm_w, occ);
  }
  // (lists: down to one ray per warp: the rays of a small image build and replay
  // their lists next to each other instead of in turn)
  const unsigned blocks = (unsigned)std::min<unsigned long long>(
      (unsigned long long)sms * std::max(per_sm, 1), 128 / kListWarps * tiles);
  const unsigned blocks_w = (unsigned)std::min<unsigned long long>(
      (unsigned long long)sms * std::max(per_sm_w, 1), tiles);
  if (lists && (e = c.list_over.ensure((size_t)blocks * kListWarps * kRays * kOver * 16))) return e;
  k.over = c.list_over.as<float4>();
  if (!c.ev0) {
    if ((e = cudaEventCreate(&c.ev0)) || (e = cudaEventCreate(&c.ev1))) return e;
  }
  cudaEventRecord(c.ev0, c.stream);
  unsigned long long* stats = reinterpret_cast<unsigned long long*>(c.flags.as<char>() + 64);
  if (walks) {
    ++c.launches;
    walker<<<blocks_w, kSlotThreads, 0, c.stream>>>(k, g, c.spiral.as<char4>(),
                                                    c.flags.as<uint32_t>(), stats);
    if ((e = cudaGetLastError())) return e;
    if (lists) {
      ++c.launches;
      if ((e = left_list_launch(c, k.leave))) return e;
    }
  }
  if (lists) {
    ++c.launches;
    render_kernel<<<blocks, kListThreads, sizeof(RenderMem), c.stream>>>(
        k, g, c.spiral.as<char4>(), c.flags.as<uint32_t>(), stats);
    if ((e = cudaGetLastError())) return e;
  }
  cudaEventRecord(c.ev1, c.stream);
  if (kernel_ms) {
    if ((e = cudaEventSynchronize(c.ev1))) return e;
    cudaEventElapsedTime(kernel_ms, c.ev0, c.ev1);
  }
  return cudaSuccess;
}

}  // namespace ilc
