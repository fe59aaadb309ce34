// ilc_batched.cu -- batched render: many cameras (jobs), aperture masks,
// per-ray chords and V value channels per cell (e.g. 128 X-ray energy bins)
// in one persistent launch fed by a work queue of 32-ray tiles.
//
// The reference renders each (camera, energy bin) as a separate projection
// with its own host loop (animation.cpp:29-100,264-283; spectrum.cpp:89-109).
// Here every warp takes the next tile from a global queue until the queue is
// empty, so rays of very different length (masked apertures, chords of a
// sphere) keep all SMs busy, and the V channels of a ray share one nn8 walk
// per integrand point: the walk yields the 8 neighbours' sorted indices and
// weights once, and the channel values are gathered from a cell-major table
// (one 4*V-byte row per neighbour, read coalesced by the warp).
//
// Step control: one step sequence per ray for all channels, from the joint
// FP64 controller (per channel the single-channel error ratio, minimum over
// channels, accept only if every channel accepts). With V = 1 this is the
// single-ray FP64 controller operation for operation, so a one-channel job
// without mask or chord reproduces the plain render bit for bit.
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <string>
#include <vector>

#include "ilc_device.cuh"
#include "ilc_internal.h"
#include "ilc_raylist.cuh"
#include "ilc_walk4.cuh"

namespace ilc {

GridView make_grid_view(const Context& c);  // ilc_render.cu

namespace {

struct BatchK {
  const JobDev* jobs;
  int n_jobs;
  uint64_t n_items;
  int V;
  const float* chan;
  float* out;
  float* state;   // multi-channel: per ray slot I[V], k1[V], candidate I[V], k5[V]
  double atol, rtol;
  int64_t max_steps;
  int tile_w;
  const uint32_t* order;
  unsigned long long* queue;
  float4* over;   // list overflow, kOver per resident ray
  LeaveRule leave;  // rays walked first, and those left to the lists
  float* walk_state;  // state of the walk kernel's rays, 4 V floats per thread
};

__device__ __forceinline__ int tile_rows(int tw) { return tw > 0 ? 32 / tw : 1; }

// Ray ti of the job's work item t: its pixel; false outside the image. Compact tiles
// are tw x th pixels, th = 32 / tw.
__device__ __forceinline__ bool item_pixel(const JobDev& J, int tw, int th, uint64_t t, int ti,
                                           int& ix, int& iy) {
  bool inside;
  if (tw > 0) {
    const int tx = (int)(t % (uint64_t)J.tiles_x), ty = (int)(t / (uint64_t)J.tiles_x);
    ix = tx * tw + ti % tw;
    iy = ty * th + ti / tw;
    inside = ix < J.nx && iy < J.ny;
  } else {  // strided: pixels t, t + T, t + 2T, ... (T = items of the job)
    const uint64_t pix = t + (uint64_t)ti * (uint64_t)J.tiles_x;
    inside = pix < (uint64_t)J.nx * (uint64_t)J.ny;
    ix = inside ? (int)(pix % (uint64_t)J.nx) : J.nx;
    iy = inside ? (int)(pix / (uint64_t)J.nx) : J.ny;
  }
  return inside;
}
// Largest k with jobs[k].item_begin <= item.
__device__ __forceinline__ int find_job(const JobDev* __restrict__ jobs, int n, uint64_t item) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].item_begin <= item) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Aperture mask, chord of the job's sphere and the ray's float origin.
// Every operation is a single IEEE double or float operation (no
// contraction), in the order the host-side definition uses.
__device__ __forceinline__ void ray_span(const JobDev& j, int ix, int iy, bool& masked,
                                         float o[3], float& len) {
  masked = false;
  if (j.aperture > 0.0) {
    const double dx = ((double)ix + 0.5 - 0.5 * (double)j.nx) * j.ps_d;
    const double dy = ((double)iy + 0.5 - 0.5 * (double)j.ny) * j.ps_d;
    if (dx * dx + dy * dy > j.aperture * j.aperture) masked = true;
  }
  const float tx = (float)ix * j.ps, ty = (float)iy * j.ps;
  float pix[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) pix[i] = (j.minp[i] + tx * j.b0[i]) + ty * j.b1[i];
  if (!(j.radius > 0.0)) {
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = pix[i];
    len = (float)j.z_range;
    return;
  }
  const double txd = (double)ix * j.ps_d, tyd = (double)iy * j.ps_d;
  double w[3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
    w[i] = j.centre[i] - ((j.minp_d[i] + txd * j.b0_d[i]) + tyd * j.b1_d[i]);
  const double t = (w[0] * j.look_d[0] + w[1] * j.look_d[1]) + w[2] * j.look_d[2];
  const double ww = (w[0] * w[0] + w[1] * w[1]) + w[2] * w[2];
  const double b2 = ww - t * t;
  const double r2 = j.radius * j.radius;
  double half = b2 < r2 ? sqrt(r2 - b2) : 0.0;
  const double mh = 0.5 * j.min_chord;
  if (half < mh) half = mh;
  double z0 = t - half;
  const double z1 = t + half;
  if (z0 < 0.0) z0 = 0.0;
  len = z1 > z0 ? (float)(z1 - z0) : 0.0f;
  const float z0f = (float)z0;
#pragma unroll
  for (int i = 0; i < 3; ++i) o[i] = pix[i] + z0f * j.look[i];
}

// One channel's FP64 step candidate: returns I + delta4 (as the accepted
// value) and sets x to the channel's error ratio
// max(atol, |I/z' rtol|) h / (2 |delta5 - delta4|), or 16 if delta4 == delta5.
// rz = 1 / z', correctly rounded: I / z' is q + (I - q z') rz with q = I rz, each
// one rounding, which is the correctly rounded quotient (Markstein's theorem;
// I is a float, so nothing leaves the double range).
__device__ __forceinline__ float channel_step(float Ic, float k1c, float e0, float e1, float e2,
                                              float e3, double hd, double zd, double rz,
                                              double atol, double rtol, double& x) {
  double d4 = 25.0 / 216.0 * (double)k1c + 1408.0 / 2565.0 * (double)e0 +
              2197.0 / 4101.0 * (double)e1 - 1.0 / 5.0 * (double)e2;
  double d5 = 16.0 / 135.0 * (double)k1c + 6656.0 / 12825.0 * (double)e0 +
              28561.0 / 56430.0 * (double)e1 - 9.0 / 50.0 * (double)e2 + 2.0 / 55.0 * (double)e3;
  d4 *= hd;
  d5 *= hd;
  x = 16.0;
  if (d4 != d5) {
    const double err = fabs(d5 - d4);
    const double q = (double)Ic * rz;
    const double quo = fabs(q) <= DBL_MAX ? fma(fma(-q, zd, (double)Ic), rz, q) : q;
    const double srt = fabs(quo * rtol);
    const double ot = fmax(atol, srt);
    x = ot * hd / (2.0 * err);
  }
  return (float)((double)Ic + d4);
}

// V > 1: the hand-over of a step's slots from the points' lanes to the warp.
struct ChanHand {
  float w[32][kRays];   // row 8 j + t: weight of slot t of point j
  int id[32][kRays];    // its sorted particle index (-1: empty)
  float ws[4][kRays];   // sum of point j's weights
};

// The step (zr, hr) of one ray for all channels, by a whole warp: the channels'
// values at the 4 points, the joint step control, and the ray's state (I[V], k1[V] and
// room for their candidates) if the step is accepted. w, ids, sums: the ray's column
// of slot weights, indices (32 rows 8 j + t) and sums of weights (4 rows), kStride
// words apart. nh: the next step size.
template <int kStride>
__device__ __forceinline__ bool channels_step(const BatchK& a, const float* w, const int* ids,
                                              const float* sums, float* Is, float zr, float hr,
                                              int lane, double& nh) {
  float* Ks = Is + a.V;
  const double hd = (double)hr;
  const double zd = (double)(zr + hr), rz = 1.0 / zd;
  double xl = __longlong_as_double(0x7ff0000000000000ll);  // +inf
  bool x0nan = false;
  // candidate values (I + delta4, k5): a lane's last group stays in
  // registers, earlier ones (V > 128) go to the ray's scratch half; they
  // are committed once the warp knows the step is accepted
  float* Es = Ks + a.V;
  float* E2s = Es + a.V;
  int held = -1;
  float4 hi4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hk4 = hi4;
  if ((a.V & 3) == 0) {
    // rows of V = 4G floats: lane handles float4 groups lane, lane+32, ...
    // (channels 4g..4g+3), one 16-byte load per neighbour and group
    const int G = a.V >> 2;
    const float4* __restrict__ chan4 = reinterpret_cast<const float4*>(a.chan);
#pragma unroll 1
    for (int gi = lane; gi < G; gi += 32) {
      if (held >= 0) {
        reinterpret_cast<float4*>(Es)[held] = hi4;
        reinterpret_cast<float4*>(E2s)[held] = hk4;
      }
      held = gi;
      const float4 i4 = reinterpret_cast<const float4*>(Is)[gi];
      const float4 k4 = reinterpret_cast<const float4*>(Ks)[gi];
      float ev[4][4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        float dot[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int id = ids[(p * 8 + q) * kStride];
          const float4 v = id >= 0 ? __ldg(&chan4[(size_t)id * G + gi])
                                   : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          const float wq = w[(p * 8 + q) * kStride];
          dot[0] = __fmaf_rn(wq, v.x, dot[0]);
          dot[1] = __fmaf_rn(wq, v.y, dot[1]);
          dot[2] = __fmaf_rn(wq, v.z, dot[2]);
          dot[3] = __fmaf_rn(wq, v.w, dot[3]);
        }
        const float wsum = sums[p * kStride];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ev[p][k] = (wsum != 0.0f && dot[k] != 0.0f) ? dot[k] / wsum : 0.0f;
      }
      const float ic[4] = {i4.x, i4.y, i4.z, i4.w}, kc[4] = {k4.x, k4.y, k4.z, k4.w};
      float en[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        double x;
        en[k] = channel_step(ic[k], kc[k], ev[0][k], ev[1][k], ev[2][k], ev[3][k], hd, zd,
                             rz, a.atol, a.rtol, x);
        if (gi == 0 && k == 0 && isnan(x)) x0nan = true;
        xl = fmin(xl, x);
      }
      hi4 = make_float4(en[0], en[1], en[2], en[3]);
      hk4 = make_float4(ev[2][0], ev[2][1], ev[2][2], ev[2][3]);
    }
  } else {
#pragma unroll 1
    for (int c = lane; c < a.V; c += 32) {
      float ev[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        float dot = 0.0f;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int id = ids[(p * 8 + q) * kStride];
          const float v = id >= 0 ? __ldg(&a.chan[(size_t)id * a.V + c]) : 0.0f;
          dot = __fmaf_rn(w[(p * 8 + q) * kStride], v, dot);
        }
        const float wsum = sums[p * kStride];
        ev[p] = (wsum != 0.0f && dot != 0.0f) ? dot / wsum : 0.0f;
      }
      double x;
      Es[c] = channel_step(Is[c], Ks[c], ev[0], ev[1], ev[2], ev[3], hd, zd, rz, a.atol,
                           a.rtol, x);
      E2s[c] = ev[2];
      if (c == 0 && isnan(x)) x0nan = true;
      xl = fmin(xl, x);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) xl = fmin(xl, __shfl_xor_sync(kAll, xl, off));
  // The host-side definition takes x_0 and then every smaller x_c:
  // a NaN x_0 gives NaN, any other NaN is passed over.
  const bool n0 = __shfl_sync(kAll, x0nan, 0);
  const double xmin = n0 ? __longlong_as_double(0x7ff8000000000000ll) : xl;
  double sc = sqrt(sqrt(xmin));
  nh = sc * hd;
  if (nh < (double)kHmin) nh = (double)kHmin;
  else if (nh > (double)kHmax) nh = (double)kHmax;
  sc = nh / hd;
  const bool accept = !(sc < 0.95);
  if (accept) {
    if (held >= 0) {
      reinterpret_cast<float4*>(Is)[held] = hi4;
      reinterpret_cast<float4*>(Ks)[held] = hk4;
#pragma unroll 1
      for (int gi = lane; gi < held; gi += 32) {
        reinterpret_cast<float4*>(Is)[gi] = reinterpret_cast<const float4*>(Es)[gi];
        reinterpret_cast<float4*>(Ks)[gi] = reinterpret_cast<const float4*>(E2s)[gi];
      }
    } else if ((a.V & 3) != 0) {
#pragma unroll 1
      for (int c = lane; c < a.V; c += 32) {
        Is[c] = Es[c];
        Ks[c] = E2s[c];
      }
    }
  }
  return accept;
}

template <bool kMulti> struct BlockMem {
  char4 spiral[1000];
  WarpLists lists[kListWarps];
  ChanHand hand[kMulti ? kListWarps : 1];
  // the block's work counters (steps, accepted, -, cells, candidates, max
  // steps of a ray, rays at the step limit)
  unsigned long long stats[7];
};

constexpr int kWalkBlocks = 4;  // per SM

// kMulti: V > 1 channels from the table; the slots carry sorted indices.
// Otherwise they carry the values (V = 1: the table's, or the particles' own
// q). Every group of 4 lanes takes the next
// ray of the queue when its ray has ended, so a warp's 8 rays need not be of
// one length. Bound by instruction issue of the list replays (DRAM idle, the
// grid sits in L2).
template <bool kMulti, int kMinBlocks>
__global__ void __launch_bounds__(kListThreads, kMinBlocks)
batched_kernel(const __grid_constant__ BatchK a, const __grid_constant__ GridView g,
               const char4* __restrict__ spiral_g, uint32_t* __restrict__ flags,
               unsigned long long* __restrict__ stats) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BlockMem<kMulti>& M = *reinterpret_cast<BlockMem<kMulti>*>(smem_raw);
  if (threadIdx.x < 7) M.stats[threadIdx.x] = 0ull;
  load_spiral(M.spiral, spiral_g);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane >> 2, pj = lane & 3;
  WarpLists& W = M.lists[warp];
  const unsigned wg = blockIdx.x * kListWarps + warp;
  if (lane == 0) W.over = a.over + (size_t)wg * kRays * kOver;
  ChanHand& H = M.hand[kMulti ? warp : 0];
  // (kept with V > 1: spectra of 16^2 pixels lose 4 % to the division at each ray; with
  // V = 1 the register is worth more)
  const int tw = a.tile_w, th = tile_rows(tw);
  float* wstate = kMulti ? a.state + ((size_t)blockIdx.x * kListThreads / 4 +
                                      (size_t)warp * kRays) * 4 * (size_t)a.V
                         : nullptr;
  const float ext0 = 0.06f * g.cs0;
  // this group's ray
  bool have = false, drained = false, fresh = true;
  float ox = 0.0f, oy = 0.0f, oz = 0.0f, lx = 0.0f, ly = 0.0f, lz = 0.0f, len = 0.0f;
  float z = 0.0f, h = 1.0f, I = 0.0f, k1 = 0.0f, scale = 0.0f;
  size_t out = 0, plane = 0;
  uint32_t rs = 0, ra = 0;
  WalkStats ws;
  for (;;) {
    // groups without a ray take the next ones
    for (;;) {
      const unsigned want = __ballot_sync(kAll, !have && !drained && pj == 0);
      if (!want) break;
      const unsigned long long q = take_rays(a.queue, want, fresh, lane, wg);
      fresh = false;
      if (!have && !drained) {
        if (q >= list_rays(a.leave, 32ull * a.n_items)) {
          drained = true;
        } else {
          const unsigned long long ray = list_ray(a.leave, q);
          const unsigned long long qi = ray >> 5;
          const uint64_t item = a.order ? (uint64_t)a.order[qi] : qi;
          const JobDev& J = a.jobs[find_job(a.jobs, a.n_jobs, item)];
          int ix, iy;
          const bool inside = item_pixel(J, tw, kMulti ? th : tile_rows(tw),
                                         item - J.item_begin, (int)(ray & 31), ix, iy);
          if (inside) {
            bool masked;
            float o[3];
            ray_span(J, ix, iy, masked, o, len);
            plane = (size_t)J.nx * (size_t)J.ny;
            out = J.out_offset + (size_t)iy * J.nx + ix;
            if (masked || !(0.0f < len)) {  // no step: the pixel is 0
              const float v = masked ? 0.0f : 0.0f * J.scale;
              for (int c = pj; c < a.V; c += 4) a.out[out + (size_t)c * plane] = v;
            } else {
              have = true;
              ox = o[0];
              oy = o[1];
              oz = o[2];
              lx = J.look[0];
              ly = J.look[1];
              lz = J.look[2];
              scale = J.scale;
              z = 0.0f;
              h = 1.0f;
              I = 0.0f;
              k1 = 0.0f;
              rs = 0;
              ra = 0;
              if (pj == 0) ray_reset(W.meta[r], ext0);
              if (kMulti) {
                float* st = wstate + (size_t)r * 4 * a.V;
                for (int c = pj; c < 4 * a.V; c += 4) st[c] = 0.0f;
              }
            }
          }
        }
      }
      __syncwarp();
    }
    if (!__any_sync(kAll, have)) break;
    const float zq = step_point(z, h, pj);
    PointSlots s;
    bool go = have;
    if (go && (int64_t)rs >= a.max_steps) {
      if (pj == 0) atomicAdd(&M.stats[6], 1ull);
      go = false;
    }
    eval_points<kMulti>(g, M.spiral, W, lane, go, ox, oy, oz, lx, ly, lz, zq, h, s, ws);
    if (!kMulti) {
      float e[4];
      share4(go ? slots_value(s) : 0.0f, lane, e);
      if (go) {
        const float zb = z;
        float next[4];
        rkf_advance_fp64(I, z, h, k1, a.atol, a.rtol, len, e, kEps, kHmin, kHmax, next);
        ++rs;
        if (z != zb) ++ra;
      }
    } else {
      if (go) {
        float w[8], sum;
        slot_weights(s, w, sum);
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          H.w[8 * pj + t][r] = w[t];
          H.id[8 * pj + t][r] = __float_as_int(s.v[t]);
        }
        H.ws[pj][r] = sum;
      }
      __syncwarp();
      unsigned gom = __ballot_sync(kAll, go && pj == 0);
      bool my_acc = false;
      double my_nh = 0.0;
      while (gom) {
        const int gl = __ffs(gom) - 1, tr = gl >> 2;
        gom &= gom - 1;
        const float zr = __shfl_sync(kAll, z, gl), hr = __shfl_sync(kAll, h, gl);
        double nh;
        const bool accept =
            channels_step<kRays>(a, &H.w[0][tr], &H.id[0][tr], &H.ws[0][tr],
                                 wstate + (size_t)tr * 4 * a.V, zr, hr, lane, nh);
        if (r == tr) {
          my_acc = accept;
          my_nh = nh;
        }
      }
      __syncwarp();
      if (go) {
        const float znew = z + h;
        if (my_acc) z = znew;
        h = (float)my_nh;
        if (z + h >= len) h = len - z + kEps;
        ++rs;
        if (my_acc) ++ra;
      }
    }
    // rays that ended (or reached the step limit)
    const bool fin = have && (!go || !(z < len));
    if (fin) {
      if (kMulti) {
        const float* Is = wstate + (size_t)r * 4 * a.V;
        for (int c = pj; c < a.V; c += 4) a.out[out + (size_t)c * plane] = Is[c] * scale;
      } else if (pj == 0) {
        a.out[out] = I * scale;
      }
      if (pj == 0) {
        atomicAdd(&M.stats[0], (unsigned long long)rs);
        atomicAdd(&M.stats[1], (unsigned long long)ra);
        atomicMax(&M.stats[5], (unsigned long long)rs);
      }
      atomicAdd(&M.stats[3], (unsigned long long)ws.cells);
      atomicAdd(&M.stats[4], (unsigned long long)ws.cands);
      ws.cells = 0;
      ws.cands = 0;
      have = false;
    }
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (M.stats[6]) atomicOr(flags, FLAG_STEP_LIMIT);
    atomicAdd(&stats[0], M.stats[0]);
    atomicAdd(&stats[1], M.stats[1]);
    atomicAdd(&stats[2], 4ull * M.stats[0]);
    atomicAdd(&stats[3], M.stats[3]);
    atomicAdd(&stats[4], M.stats[4]);
    atomicMax(&stats[5], M.stats[5]);
    atomicAdd(&stats[6], M.stats[6]);
  }
}

// Point J's slots to weights in place (the indices stay), and their sum.
template <int J> __device__ __forceinline__ void slots_to_weights(const Step4& s, float& sum) {
  float w[8], ws;
  s4_weights<J>(s, w, ws);
#pragma unroll
  for (int t = 0; t < 8; ++t) s4_d(s, J, t) = w[t];
  sum = ws;
}

// The rays of every work item walked, a ray per thread, a warp to an item, every
// step from scratch for its 4 points together (ilc_walk4.cuh), until they end or
// their steps suit the lists, to which they are then left. kIdx: the slots hold
// indices (V > 1, or a value table); otherwise the particles' own values.
template <bool kMulti, bool kIdx>
__global__ void __launch_bounds__(kSlotThreads, kWalkBlocks)
batched_walk_kernel(const __grid_constant__ BatchK a, const __grid_constant__ GridView g,
                    const char4* __restrict__ spiral_g, uint32_t* __restrict__ flags,
                    unsigned long long* __restrict__ stats) {
  __shared__ char4 spiral[1000];
  __shared__ SlotMem slot_mem;
  __shared__ float slot_ws[kMulti ? 4 : 1][kSlotThreads];
  __shared__ unsigned long long blk[7];  // as BlockMem::stats
  if (threadIdx.x < 7) blk[threadIdx.x] = 0ull;
  load_spiral(spiral, spiral_g);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tw = a.tile_w, th = tile_rows(tw);
  float* wstate = kMulti ? a.walk_state + ((size_t)blockIdx.x * kSlotThreads +
                                           (size_t)warp * 32) * 4 * (size_t)a.V
                         : nullptr;
  for (;;) {
    unsigned long long turn = 0;
    if (lane == 0) turn = atomicAdd(a.queue + 1, 1ull);
    turn = __shfl_sync(kAll, turn, 0);
    if (turn >= a.n_items) break;
    const uint64_t item = a.order ? (uint64_t)a.order[turn] : turn;
    const JobDev& J = a.jobs[find_job(a.jobs, a.n_jobs, item)];
    int ix, iy;
    const bool inside = item_pixel(J, tw, th, item - J.item_begin, lane, ix, iy);
    bool masked = true;
    float o[3] = {0.0f, 0.0f, 0.0f}, len = 0.0f;
    if (inside) ray_span(J, ix, iy, masked, o, len);
    const float lx = J.look[0], ly = J.look[1], lz = J.look[2];
    bool run = inside && !masked, leave = false;
    float z = 0.0f, h = 1.0f, I = 0.0f, k1 = 0.0f;
    uint32_t rs = 0, ra = 0;
    Walk4Stats ws;
    Pace pace = pace_start(0.0f);
    if (kMulti) {
      for (int i = lane; i < 32 * 4 * a.V; i += 32) wstate[i] = 0.0f;
      __syncwarp();
    }
    while (__any_sync(kAll, run && z < len)) {
      if (run && z < len && (int64_t)rs >= a.max_steps) {
        atomicAdd(&blk[6], 1ull);
        run = false;
      }
      const bool go = run && z < len;
      ws.scans = 0;
      if (go) {
        float pts[4];
        rkf_points(z, h, pts);
        if (!kMulti) {
          float e[4];
          nn8_step4<kIdx>(g, spiral, slot_mem, o[0], o[1], o[2], lx, ly, lz, pts, e, ws);
          const float zb = z;
          rkf_advance_fp64(I, z, h, k1, a.atol, a.rtol, len, e, kEps, kHmin, kHmax, pts);
          ++rs;
          if (z != zb) ++ra;
        } else {
          Step4 s;
          s4_bind(s, slot_mem);
          nn8_walk_step4<true>(g, spiral, o[0], o[1], o[2], lx, ly, lz, pts, s, ws);
          slots_to_weights<0>(s, slot_ws[0][threadIdx.x]);
          slots_to_weights<1>(s, slot_ws[kMulti ? 1 : 0][threadIdx.x]);
          slots_to_weights<2>(s, slot_ws[kMulti ? 2 : 0][threadIdx.x]);
          slots_to_weights<3>(s, slot_ws[kMulti ? 3 : 0][threadIdx.x]);
        }
      }
      if (kMulti) {
        __syncwarp();
        unsigned gom = __ballot_sync(kAll, go);
        bool my_acc = false;
        double my_nh = 0.0;
        while (gom) {
          const int r = __ffs(gom) - 1;
          gom &= gom - 1;
          const float zr = __shfl_sync(kAll, z, r), hr = __shfl_sync(kAll, h, r);
          const int t = warp * 32 + r;  // ray r's slot columns: weights, indices
          double nh;
          const bool accept =
              channels_step<kSlotThreads>(a, &slot_mem.d[0][t],
                                          reinterpret_cast<const int*>(&slot_mem.v[0][t]),
                                          &slot_ws[0][t], wstate + (size_t)r * 4 * a.V, zr, hr,
                                          lane, nh);
          if (lane == r) {
            my_acc = accept;
            my_nh = nh;
          }
        }
        __syncwarp();
        if (go) {
          const float znew = z + h;
          if (my_acc) z = znew;
          h = (float)my_nh;
          if (z + h >= len) h = len - z + kEps;
          ++rs;
          if (my_acc) ++ra;
        }
      }
      if (go && pace_slow(pace, a.leave, z, len, h, rs, ws.scans) && z < len) {
        leave = true;
        run = false;
      }
    }
    const bool counted = inside && !masked && !(J.radius > 0.0);  // as in BatchArgs::rays
    mark_left(a.leave, counted, leave, 32 * turn + lane, lane);
    if (!kMulti) {
      if (inside && !leave)
        a.out[J.out_offset + (size_t)iy * J.nx + ix] = masked ? 0.0f : I * J.scale;
    } else {
      const size_t plane = (size_t)J.nx * (size_t)J.ny;
      for (int r = 0; r < 32; ++r) {
        const int ixr = __shfl_sync(kAll, ix, r), iyr = __shfl_sync(kAll, iy, r);
        const bool out_r = __shfl_sync(kAll, inside && !leave, r),
                   m_r = __shfl_sync(kAll, masked, r);
        if (!out_r) continue;
        const float* Is = wstate + (size_t)r * 4 * a.V;
        for (int c = lane; c < a.V; c += 32)
          a.out[J.out_offset + (size_t)c * plane + (size_t)iyr * J.nx + ixr] =
              m_r ? 0.0f : Is[c] * J.scale;
      }
      __syncwarp();
    }
    if (!leave) {
      atomicAdd(&blk[0], (unsigned long long)rs);
      atomicAdd(&blk[1], (unsigned long long)ra);
      atomicAdd(&blk[3], (unsigned long long)ws.cells);
      atomicAdd(&blk[4], (unsigned long long)ws.cands);
      atomicMax(&blk[5], (unsigned long long)rs);
    }
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (blk[6]) atomicOr(flags, FLAG_STEP_LIMIT);
    atomicAdd(&stats[0], blk[0]);
    atomicAdd(&stats[1], blk[1]);
    atomicAdd(&stats[2], 4ull * blk[0]);
    atomicAdd(&stats[3], blk[3]);
    atomicAdd(&stats[4], blk[4]);
    atomicMax(&stats[5], blk[5]);
    atomicAdd(&stats[6], blk[6]);
  }
}

__global__ void channels_sort_kernel(const float* __restrict__ in,
                                     const uint32_t* __restrict__ s2u, uint64_t n, int V,
                                     float* __restrict__ out) {
  const uint64_t total = n * (uint64_t)V;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t p = i / (uint64_t)V, c = i - p * (uint64_t)V;
    out[i] = in[(uint64_t)s2u[p] * V + c];
  }
}

// Per-tile cost estimate of one job: every particle in front of the camera
// (and within its depth when the job has no chord) adds its cell's
// occupancy to the tile its pixel column falls in, so tiles whose rays cross
// many particles in dense cells -- the long, expensive rays -- score high.
__global__ void tile_cost_kernel(const float4* __restrict__ parts,
                                 const uint32_t* __restrict__ keys,
                                 const int2* __restrict__ cells, uint64_t n, JobDev J, int tw,
                                 int th, float* __restrict__ cost) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const float4 p = parts[i];
    const float dx = p.x - J.minp[0], dy = p.y - J.minp[1], dz = p.z - J.minp[2];
    const float u = (dx * J.b0[0] + dy * J.b0[1] + dz * J.b0[2]) / J.ps;
    const float v = (dx * J.b1[0] + dy * J.b1[1] + dz * J.b1[2]) / J.ps;
    const float t = dx * J.look[0] + dy * J.look[1] + dz * J.look[2];
    if (!(u >= 0.0f) || !(v >= 0.0f) || !(u < (float)J.nx) || !(v < (float)J.ny)) continue;
    if (!(t >= 0.0f) || (!(J.radius > 0.0) && !(t <= (float)J.z_range))) continue;
    const int ix = (int)u, iy = (int)v;
    const int2 be = cells[keys[i]];
    const uint64_t item = tw > 0 ? (uint64_t)(iy / th) * J.tiles_x + (uint64_t)(ix / tw)
                                 : ((uint64_t)iy * J.nx + ix) % (uint64_t)J.tiles_x;
    atomicAdd(&cost[J.item_begin + item], (float)(be.y - be.x));
  }
}

// One channel: 4 blocks of 128 threads per SM, by registers (128) and shared memory
// (227 KB); V > 1 adds the hand-over and runs 3.
static_assert(sizeof(BlockMem<false>) <= 50 * 1024 && sizeof(BlockMem<true>) <= 57 * 1024,
              "4 and 3 blocks per SM, with shared memory left for L1");
template <bool kMulti> struct Variant {
  static constexpr int kBlocks = kMulti ? 3 : 4;
  static constexpr size_t kSmem = sizeof(BlockMem<kMulti>);
  static auto kernel() { return batched_kernel<kMulti, kBlocks>; }
};

// Resident blocks: what registers and shared memory allow, or `occ` per SM.
template <bool kMulti> cudaError_t persistent_blocks(const Context& c, int occ, int* blocks) {
  using Vt = Variant<kMulti>;
  int sms = 0, per_sm = 0;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(Vt::kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)Vt::kSmem)))
    return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device))) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, Vt::kernel(), kListThreads,
                                                         Vt::kSmem)))
    return e;
  if (occ > 0) per_sm = std::min(per_sm, occ);
  *blocks = sms * std::max(per_sm, 1);
  return cudaSuccess;
}

template <bool kMulti>
cudaError_t launch_variant(Context& c, const BatchK& k, const GridView& g, int blocks) {
  using Vt = Variant<kMulti>;
  unsigned long long* stats = reinterpret_cast<unsigned long long*>(c.flags.as<char>() + 64);
  Vt::kernel()<<<blocks, kListThreads, Vt::kSmem, c.stream>>>(k, g, c.spiral.as<char4>(),
                                                              c.flags.as<uint32_t>(), stats);
  return cudaGetLastError();
}

// The walk kernel for these channels, and its resident blocks.
using WalkKernel = void (*)(BatchK, GridView, const char4*, uint32_t*, unsigned long long*);
WalkKernel walk_kernel(const BatchK& k, const GridView& g) {
  return k.V > 1  ? batched_walk_kernel<true, true>
         : g.vals ? batched_walk_kernel<false, true>
                  : batched_walk_kernel<false, false>;
}
cudaError_t walk_blocks(const Context& c, WalkKernel kernel, int occ, int* blocks) {
  int sms = 0, per_sm = 0;
  cudaError_t e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device)) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSlotThreads, 0)))
    return e;
  if (occ > 0) per_sm = std::min(per_sm, occ);
  *blocks = sms * std::max(per_sm, 1);
  return cudaSuccess;
}

// blocks_w: of the walk in front (0: none).
cudaError_t enqueue(Context& c, const BatchK& k, const GridView& g, int blocks, int blocks_w) {
  cudaError_t e;
  if ((e = cudaMemsetAsync(c.flags.p, 0, kFlagsBytes, c.stream))) return e;
  if ((e = cudaMemsetAsync(c.queue.p, 0, kQueueBytes, c.stream))) return e;
  if (blocks_w > 0) {
    walk_kernel(k, g)<<<blocks_w, kSlotThreads, 0, c.stream>>>(
        k, g, c.spiral.as<char4>(), c.flags.as<uint32_t>(),
        reinterpret_cast<unsigned long long*>(c.flags.as<char>() + 64));
    if ((e = cudaGetLastError()) || (e = left_list_launch(c, k.leave))) return e;
  }
  return k.V == 1 ? launch_variant<false>(c, k, g, blocks)
                  : launch_variant<true>(c, k, g, blocks);
}

}  // namespace

cudaError_t batched_residency(int n_channels, int occ, int* id) {
  Context c;  // (only its device is read)
  cudaError_t e;
  BatchK k{};
  k.V = n_channels;
  GridView g{};
  int lists = 0, walk = 0;
  if ((e = cudaGetDevice(&c.device)) ||
      (e = n_channels > 1 ? persistent_blocks<true>(c, occ, &lists)
                          : persistent_blocks<false>(c, occ, &lists)) ||
      (e = walk_blocks(c, walk_kernel(k, g), occ, &walk)))
    return e;
  *id = 4096 * lists + walk;
  return cudaSuccess;
}

cudaError_t channels_sort_launch(Context& c, const float* in, uint64_t n, int V, float* out) {
  const uint64_t total = n * (uint64_t)V;
  const unsigned blocks = (unsigned)std::min<uint64_t>((total + 255) / 256, 148ull * 16);
  ++c.launches;
  channels_sort_kernel<<<blocks > 0 ? blocks : 1, 256, 0, c.stream>>>(in, c.s2u.as<uint32_t>(),
                                                                       n, V, out);
  return cudaGetLastError();
}

cudaError_t batched_order(Context& c, BatchArgs& a, const std::vector<JobDev>& jobs) {
  cudaError_t e;
  const uint64_t m = a.n_items;
  if ((e = c.item_cost.ensure(m * 4)) || (e = c.item_order.ensure(m * 4))) return e;
  if ((e = cudaMemsetAsync(c.item_cost.p, 0, m * 4, c.stream))) return e;
  const int tw = a.tile_w, th = a.tile_w > 0 ? 32 / a.tile_w : 1;
  const uint64_t n = c.n_particles;
  const unsigned blocks = (unsigned)std::min<uint64_t>((n + 255) / 256, 148ull * 8);
  for (const JobDev& j : jobs) {
    tile_cost_kernel<<<blocks > 0 ? blocks : 1, 256, 0, c.stream>>>(
        c.parts.as<float4>(), c.sorted_keys, c.cells.as<int2>(), n, j, tw, th,
        c.item_cost.as<float>());
    ++c.launches;
  }
  if ((e = cudaGetLastError())) return e;
  std::vector<float> cost(m);
  if ((e = cudaMemcpyAsync(cost.data(), c.item_cost.p, m * 4, cudaMemcpyDeviceToHost,
                           c.stream)) ||
      (e = cudaStreamSynchronize(c.stream)))
    return e;
  std::vector<uint32_t> order(m);
  for (uint64_t i = 0; i < m; ++i) order[i] = (uint32_t)i;
  std::stable_sort(order.begin(), order.end(),
                   [&](uint32_t x, uint32_t y) { return cost[x] > cost[y]; });
  if ((e = cudaMemcpyAsync(c.item_order.p, order.data(), m * 4, cudaMemcpyHostToDevice,
                           c.stream)) ||
      (e = cudaStreamSynchronize(c.stream)))
    return e;
  a.order = c.item_order.as<uint32_t>();
  return cudaSuccess;
}

// The launch sequence (reset of the flags and the queue, persistent kernel)
// runs as a CUDA graph, instantiated once per set of launch parameters and
// replayed while they stay the same (repeated frames of one job set).
cudaError_t batched_launch(Context& c, const BatchArgs& a, float* kernel_ms) {
  cudaError_t e;
  if ((e = c.flags.ensure(kFlagsBytes))) return e;
  if ((e = c.queue.ensure(256))) return e;
  BatchK k;
  std::memset(&k, 0, sizeof(k));  // the bytes are the graph's key
  k.jobs = a.jobs;
  k.n_jobs = a.n_jobs;
  k.n_items = a.n_items;
  k.V = a.V;
  k.chan = a.chan;
  k.out = a.out;
  k.atol = a.atol;
  k.rtol = a.rtol;
  k.max_steps = c.max_steps;
  k.tile_w = a.tile_w;
  k.order = a.order;
  k.queue = c.queue.as<unsigned long long>();
  int blocks = 0;
  if ((e = a.V > 1 ? persistent_blocks<true>(c, a.occupancy, &blocks)
                   : persistent_blocks<false>(c, a.occupancy, &blocks)))
    return e;
  if (a.V > 1) {
    if ((e = c.chan_state.ensure((size_t)blocks * (kListThreads / 4) * 4 * (size_t)k.V * 4)))
      return e;
    k.state = c.chan_state.as<float>();
  }
  if ((e = c.list_over.ensure((size_t)blocks * kListWarps * kRays * kOver * 16))) return e;
  k.over = c.list_over.as<float4>();
  GridView g = make_grid_view(c);
  if (a.V == 1) g.vals = a.chan;
  // many rays: walked first, the lists get those that the walk leaves
  int blocks_w = 0;
  k.leave = walk_rule(c, a.rays, 32 * a.n_items, k.queue);
  if (k.leave.left) {
    if ((e = walk_blocks(c, walk_kernel(k, g), a.occupancy, &blocks_w))) return e;
    if (a.V > 1 && c.walk_state.ensure((size_t)blocks_w * kSlotThreads * 4 * (size_t)k.V * 4)) {
      cudaGetLastError();  // (no memory for the channels' states: lists for all rays)
      k.leave.left = nullptr;
      blocks_w = 0;
    }
    k.walk_state = c.walk_state.as<float>();
  }
  if (!c.ev0) {
    if ((e = cudaEventCreate(&c.ev0)) || (e = cudaEventCreate(&c.ev1))) return e;
  }
  std::string key(reinterpret_cast<const char*>(&k), sizeof(k));
  key.append(reinterpret_cast<const char*>(&g), sizeof(g));
  key.append(reinterpret_cast<const char*>(&blocks), sizeof(blocks));
  key.append(reinterpret_cast<const char*>(&blocks_w), sizeof(blocks_w));
  if (!c.batch_exec || key != c.batch_key) {
    if (c.batch_exec) {
      cudaGraphExecDestroy(c.batch_exec);
      c.batch_exec = nullptr;
    }
    c.batch_key.clear();
    cudaGraph_t graph = nullptr;
    if ((e = cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal))) return e;
    const cudaError_t el = enqueue(c, k, g, blocks, blocks_w);
    e = cudaStreamEndCapture(c.stream, &graph);
    if (el) {
      if (graph) cudaGraphDestroy(graph);
      return el;
    }
    if (e) return e;
    e = cudaGraphInstantiate(&c.batch_exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e) {
      c.batch_exec = nullptr;
      return e;
    }
    c.batch_key = key;
  }
  cudaEventRecord(c.ev0, c.stream);
  c.launches += blocks_w > 0 ? 3 : 1;
  if ((e = cudaGraphLaunch(c.batch_exec, c.stream))) return e;
  cudaEventRecord(c.ev1, c.stream);
  if (kernel_ms) {
    if ((e = cudaEventSynchronize(c.ev1))) return e;
    cudaEventElapsedTime(kernel_ms, c.ev0, c.ev1);
  }
  return cudaSuccess;
}

}  // namespace ilc
