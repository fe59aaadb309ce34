// ilc_adjoint.cu -- gradient of an image loss with respect to per-cell log
// density and log temperature, through the nn8 reconstruction and the RKF
// line-of-sight integral, with the neighbour choice fixed and the step
// sequence frozen from the forward pass (checkpointed per ray, or recomputed).
//
// With fixed neighbours and frozen steps a pixel is linear in the per-cell
// values q: every accepted step adds h (25/216 k1 + 1408/2565 e0 +
// 2197/4101 e1 - 1/5 e2) (integration.cl:63-67,118), k1 being the previous
// accepted step's e2 (0 before the first), and every e is the nn8 finalize
// sum(w v)/sum(w) (volumetric_nn8_reconstruction.cl:212-270), so
// d e / d v_p = w_p / sum(w). The adjoint replays each ray's steps, evaluates
// e0, e1, e2 (e3 only enters the error estimate) and scatters
// dL/dI * coefficient * w_p / sum(w) into dL/dq_p. The per-cell chain rule
// then multiplies by dq/dln rho and dq/dln T of the adaptive band flux
// (ilc_adjoint_cell.cuh).
#include "ilc_adjoint_cell.cuh"
#include "ilc_device.cuh"
#include "ilc_internal.h"
#include "ilc_quantity.cuh"
#include "ilc_raylist.cuh"
#include "ilc_walk4.cuh"

namespace ilc {

namespace {

// q (bit-identical to xray_flux_kernel), dq/dlnT, dq/dlnrho for one cell.
template <int kWhich>
__device__ void band_flux_tangent(const float* t, const GauntView& G, float Emin, float Emax,
                                  float reltol, float T, float xe, float rho, float dL, float* q,
                                  double* dq) {
  const GauntViewD GD{G.w, G.h, G.x0, G.y0, G.dx, G.dy};
  const float atol = reltol, rtol = 1.0f, eps = 0.0f, hmin = 1.e-3f, hmax = 100.f;
  float I = 0.0f, z = Emin, h = (Emax - Emin) * reltol;
  double dI = 0, dz = 0, dh = 0, dk1, dkE;
  const float end = Emax;
  float k1 = brems(t, G, z, 1.0f, T, xe, rho, dL, G.w);
  brems_tangent(t, GD, z, T, xe, rho, dL, kWhich, &dk1, &dkE, (double)k1);
  float p[4];
  double dp[4] = {0, 0, 0, 0};
  rkf_points(z, h, p);
  const double c[4] = {3. / 8., 12. / 13., 1.0, 0.5};
  int guard = 0;
  while (z < end && guard < 100000) {
    float e[4];
    double de[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      e[j] = brems(t, G, p[j], 1.0f, T, xe, rho, dL, G.w);
      double pl, pe;
      brems_tangent(t, GD, p[j], T, xe, rho, dL, kWhich, &pl, &pe, (double)e[j]);
      de[j] = pl + pe * dp[j];
    }
    const float b4 = 25.f / 216.f * k1 + 1408.f / 2565.f * e[0] + 2197.f / 4101.f * e[1] -
                     1.f / 5.f * e[2];
    const float b5 = 16.f / 135.f * k1 + 6656.f / 12825.f * e[0] + 28561.f / 56430.f * e[1] -
                     9.f / 50.f * e[2] + 2.f / 55.f * e[3];
    const double db4 = 25. / 216. * dk1 + 1408. / 2565. * de[0] + 2197. / 4101. * de[1] -
                       1. / 5. * de[2];
    const double db5 = 16. / 135. * dk1 + 6656. / 12825. * de[0] + 28561. / 56430. * de[1] -
                       9. / 50. * de[2] + 2. / 55. * de[3];
    const double dd4 = db4 * (double)h + (double)b4 * dh;
    const double dd5 = db5 * (double)h + (double)b5 * dh;
    const float d4 = b4 * h, d5 = b5 * h;
    const float est4 = I + d4;
    const double dest4 = dI + dd4;
    const float old = z;
    const double dold = dz;
    z += h;
    dz += dh;
    float s = 2.0f;
    double ds = 0;
    if (d4 != d5) {
      const float err = fabsf(d5 - d4);
      const double derr = sgnd((double)d5 - (double)d4) * (dd5 - dd4);
      const float ratio = I / z * rtol;
      const float srt = fabsf(ratio);
      const double dsrt = sgnd((double)ratio) * (double)rtol *
                          (dI / (double)z - (double)I * dz / ((double)z * (double)z));
      const float ot = fmaxf(atol, srt);
      const double dot_ = srt > atol ? dsrt : 0.0;
      s = sqrtf(sqrtf(ot * h / (2.0f * err)));
      ds = (double)s * 0.25 * (dot_ / (double)ot + dh / (double)h - derr / (double)err);
    }
    float nh = s * h;
    double dnh = ds * (double)h + (double)s * dh;
    if (nh < hmin) { nh = hmin; dnh = 0; }
    else if (nh > hmax) { nh = hmax; dnh = 0; }
    s = nh / h;
    if (s < 0.95f) {
      z = old;
      dz = dold;
    } else {
      I = est4;
      dI = dest4;
      k1 = e[2];
      dk1 = de[2];
    }
    h = nh;
    dh = dnh;
    if (z + h >= end) { h = end - z + eps; dh = -dz; }
    rkf_points(z, h, p);
#pragma unroll
    for (int j = 0; j < 4; ++j) dp[j] = dz + c[j] * dh;
    ++guard;
  }
  *q = I;
  *dq = dI;
}

__global__ void __launch_bounds__(256)
xray_flux_grad_kernel(const float* __restrict__ table, GauntView G, const float* __restrict__ rho,
                      const float* __restrict__ u, const float* __restrict__ xe, uint64_t n,
                      float z, float dL, float emin, float emax, int num_samples,
                      float* __restrict__ q_out, int q_stride, float* __restrict__ dq_lnT,
                      float* __restrict__ dq_lnrho) {
  __shared__ float t[81 * 146];
  for (int i = threadIdx.x; i < G.w * G.h; i += blockDim.x) t[i] = table[i];
  __syncthreads();
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const float T = temperature(u[i], xe[i]);
    const float e0 = (1.f + z) * emin, e1 = (1.f + z) * emax, rt = 1.f / (float)num_samples;
    float q;
    double dT, dR;
    band_flux_tangent<0>(t, G, e0, e1, rt, T, xe[i], rho[i], dL, &q, &dT);
    band_flux_tangent<1>(t, G, e0, e1, rt, T, xe[i], rho[i], dL, &q, &dR);
    q_out[i * q_stride] = q;
    dq_lnT[i] = (float)dT;
    dq_lnrho[i] = (float)dR;
  }
}

// L = sum over pixels of (log I - log I_target)^2 on the scaled image; the
// seed per ray is dL/dI_raw = 2 (log I - log I_target) / I_raw. Pixels with a
// non-positive value or target are left out of the loss (log undefined).
__global__ void loss_seed_kernel(const float* __restrict__ img, const float* __restrict__ target,
                                 int64_t npix, float scale, float* __restrict__ seed,
                                 double* __restrict__ loss) {
  double part = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npix;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float I = img[i], tg = target[i];
    float s = 0.0f;
    if (I > 0.0f && tg > 0.0f && isfinite(I) && isfinite(tg)) {
      const double r = log((double)I) - log((double)tg);
      part += r * r;
      const double raw = (double)I / (double)scale;
      s = (float)(2.0 * r / raw);
    }
    seed[i] = s;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, part);
}

// A point's slots as the scatter needs them: d e / d v_p = w_p / sum(w).
struct ScatterSlots {
  float w[8], ws;
  int id[8];
};

__device__ __forceinline__ void scatter_slots(const PointSlots& s, ScatterSlots& o) {
  slot_weights(s, o.w, o.ws);
#pragma unroll
  for (int t = 0; t < 8; ++t) o.id[t] = __float_as_int(s.v[t]);
}

// Adds c * w_p / sum(w) to grad at the slots' sorted particle indices (nothing
// where the finalize has no weight). The accumulator is double: a cell's
// gradient sums contributions of both signs from many rays, and fp32
// accumulation loses digits to cancellation.
__device__ __forceinline__ void scatter(const ScatterSlots& s, double c,
                                        double* __restrict__ grad) {
  if (c == 0.0 || !(s.ws > 0.0f) || !isfinite(s.ws)) return;
  const double f = c / (double)s.ws;
#pragma unroll
  for (int t = 0; t < 8; ++t)
    if (s.id[t] >= 0 && s.w[t] != 0.0f) atomicAdd(&grad[s.id[t]], f * (double)s.w[t]);
}

// nn8 value of a point (finalize order) with the values read by index.
__device__ __forceinline__ float value_by_id(const ScatterSlots& s,
                                             const float4* __restrict__ parts) {
  float dot = 0.0f;
#pragma unroll
  for (int t = 0; t < 8; ++t)
    dot = __fmaf_rn(s.w[t], s.id[t] >= 0 ? __ldg(&parts[s.id[t]].w) : 0.0f, dot);
  return (s.ws != 0.0f && dot != 0.0f) ? dot / s.ws : 0.0f;
}

struct AdjK {
  CamView cam;
  float z0, z_end;
  double atol, rtol;
  int controller;
  int64_t max_steps;
  int mode;                        // ILC_ADJOINT_CHECKPOINT / _RECOMPUTE
  const float* __restrict__ rec_h;  // checkpoint: accepted step sizes, ray-major
  const int32_t* __restrict__ rec_n;
  int64_t rec_cap;
  const float* __restrict__ seed;  // dL/dI_raw per pixel (whole image)
  double* __restrict__ grad;       // dL/dq per sorted particle
  int row0, row_end;               // pixel rows of this launch; rec_* indexed from row0
  unsigned long long* queue;       // ray counter
  unsigned long long n_rays;       // 128 per 16 x 8 tile
  unsigned tiles_x;
  float4* over;                    // list overflow, kOver per resident ray
  LeaveRule leave;                 // a forward pass that walked first: the rays it left
};

// Pixel of ray q, numbered as in the render kernel.
__device__ __forceinline__ void adjoint_pixel(const AdjK& a, unsigned long long q, int& ix,
                                              int& iy) {
  const unsigned tile = (unsigned)(q >> 7), t = (unsigned)(q & 127u);
  const int sub = (int)(t >> 3);
  ix = (int)(tile % a.tiles_x) * 16 + (sub & 3) * 4 + (int)(t & 3u);
  iy = a.row0 + (int)(tile / a.tiles_x) * 8 + (sub >> 2) * 2 + (int)((t >> 2) & 1u);
}

constexpr int kAdjBlocks = 4;

struct AdjMem {
  char4 spiral[1000];
  WarpLists lists[kListWarps];
};

// Four lanes per ray, as in the render kernel: lane j scatters point j (point
// 3 only enters the error estimate, and a checkpointed replay does not need
// it). Point 2 of an accepted step is the next one's k1: its lane holds its
// slots back until the next step's size is known and scatters both terms at
// once.
__global__ void __launch_bounds__(kListThreads, kAdjBlocks)
adjoint_kernel(const __grid_constant__ AdjK a, const __grid_constant__ GridView g,
               const char4* __restrict__ spiral_g, uint32_t* __restrict__ flags,
               unsigned long long* __restrict__ stats) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  AdjMem& M = *reinterpret_cast<AdjMem*>(smem_raw);
  load_spiral(M.spiral, spiral_g);
  const int lane = threadIdx.x & 31;
  const int r = lane >> 2, pj = lane & 3;
  WarpLists& W = M.lists[threadIdx.x >> 5];
  const unsigned wg = blockIdx.x * kListWarps + (threadIdx.x >> 5);
  if (lane == 0) W.over = a.over + (size_t)wg * kRays * kOver;
  const float ext0 = 0.06f * g.cs0;
  const float lx = a.cam.look0, ly = a.cam.look1, lz = a.cam.look2;
  const float fa = (float)a.atol, fr = (float)a.rtol;
  const bool replay = a.mode == ILC_ADJOINT_CHECKPOINT;
  bool have = false, drained = false, fresh = true;
  float px = 0.0f, py = 0.0f, pz = 0.0f, gi = 0.0f;
  float I = 0.0f, z = 0.0f, h = 1.0f, k1 = 0.0f;
  int64_t limit = 0;
  const float* hs = nullptr;
  unsigned long long steps = 0;
  bool have_prev = false;
  ScatterSlots prev;
  double prev_c = 0.0;
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
          int ix, iy;
          adjoint_pixel(a, list_ray(a.leave, q), ix, iy);
          if (ix < a.cam.nx && iy < a.row_end) {
            gi = a.seed[(int64_t)iy * a.cam.nx + ix];
            have = gi != 0.0f;
            const int64_t ray = (int64_t)(iy - a.row0) * a.cam.nx + ix;  // in the launch's rows
            pixel_corner(a.cam, ix, iy, px, py, pz);
            limit = replay ? a.rec_n[ray] : a.max_steps;
            hs = replay ? a.rec_h + ray * a.rec_cap : nullptr;
          }
        }
        if (have) {
          I = 0.0f;
          k1 = 0.0f;
          z = a.z0;
          h = 1.0f;
          steps = 0;
          have_prev = false;
          if (pj == 0) ray_reset(W.meta[r], ext0);
        }
      }
      __syncwarp();
    }
    if (!__any_sync(kAll, have)) break;
    const bool go = have && (int64_t)steps < limit && (replay || z < a.z_end);
    if (go && replay) h = hs[steps];
    const float zq = step_point(z, h, pj);
    PointSlots s;
    eval_points<true>(g, M.spiral, W, lane, go && !(replay && pj == 3), px, py, pz, lx,
                               ly, lz, zq, h, s, ws);
    ScatterSlots cur;
    if (go && !(replay && pj == 3)) scatter_slots(s, cur);
    bool accepted = go;
    const float hb = h;
    if (replay) {
      if (go) z += h;
    } else {
      float e[4];
      share4(go ? value_by_id(cur, g.parts) : 0.0f, lane, e);
      if (go) {
        const float zb = z;
        float next[4];
        if (a.controller == ILC_CONTROLLER_REF32)
          rkf_advance_ref32(I, z, h, k1, fa, fr, a.z_end, e, kEps, kHmin, kHmax, next);
        else
          rkf_advance_fp64(I, z, h, k1, a.atol, a.rtol, a.z_end, e, kEps, kHmin, kHmax, next);
        accepted = z != zb;
      }
    }
    if (go) ++steps;
    if (accepted) {
      if (pj < 2) {
        scatter(cur, (double)(gi * (pj == 0 ? hb * 1408.f / 2565.f : hb * 2197.f / 4101.f)),
                a.grad);
      } else if (pj == 2) {
        if (have_prev) scatter(prev, prev_c + (double)(gi * (hb * 25.f / 216.f)), a.grad);
        prev = cur;
        prev_c = (double)(gi * (-hb / 5.f));
        have_prev = true;
      }
    }
    const bool fin = have && (!go || (replay ? (int64_t)steps >= limit : !(z < a.z_end)));
    if (fin) {
      if (pj == 2 && have_prev) scatter(prev, prev_c, a.grad);
      if (pj == 0) {
        if (!replay && z < a.z_end) atomicOr(flags, FLAG_STEP_LIMIT);
        atomicAdd(&stats[0], steps);
      }
      have = false;
    }
    __syncwarp();
  }
  atomicAdd(&stats[3], (unsigned long long)ws.cells);
  atomicAdd(&stats[4], (unsigned long long)ws.cands);
}

// Point J's slots of a walked step as the scatter needs them.
template <int J> __device__ __forceinline__ void scatter_slots(const Step4& s, ScatterSlots& o) {
  s4_weights<J>(s, o.w, o.ws);
#pragma unroll
  for (int t = 0; t < 8; ++t) o.id[t] = __float_as_int(s4_v(s, J, t));
}
template <int J>
__device__ __forceinline__ void scatter_point(const Step4& s, float c, double* __restrict__ grad) {
  ScatterSlots o;
  scatter_slots<J>(s, o);
  scatter(o, (double)c, grad);
}

// The rays that a forward pass walked to their end, a ray per thread, as it walked
// them (walk_kernel in ilc_render.cu): their steps are long against a cell.
__global__ void __launch_bounds__(kSlotThreads, kAdjBlocks)
adjoint_walk_kernel(const __grid_constant__ AdjK a, const __grid_constant__ GridView g,
                    const char4* __restrict__ spiral_g, uint32_t* __restrict__ flags,
                    unsigned long long* __restrict__ stats) {
  __shared__ char4 spiral[1000];
  __shared__ SlotMem slot_mem;
  __shared__ unsigned long long next_tile;
  load_spiral(spiral, spiral_g);
  const float lx = a.cam.look0, ly = a.cam.look1, lz = a.cam.look2;
  const float fa = (float)a.atol, fr = (float)a.rtol;
  const bool replay = a.mode == ILC_ADJOINT_CHECKPOINT;
  for (;;) {
    if (threadIdx.x == 0) next_tile = atomicAdd(a.queue + 1, 1ull);
    __syncthreads();
    const unsigned long long q = 128 * next_tile + walk_ray();
    __syncthreads();
    if (q >= a.n_rays) break;  // (all of the block)
    if ((a.leave.left[q >> 3] >> (q & 7u)) & 1u) continue;
    int ix, iy;
    adjoint_pixel(a, q, ix, iy);
    if (ix >= a.cam.nx || iy >= a.row_end) continue;
    const float gi = a.seed[(int64_t)iy * a.cam.nx + ix];
    if (gi == 0.0f) continue;
    const int64_t ray = (int64_t)(iy - a.row0) * a.cam.nx + ix;  // in the launch's rows
    float px, py, pz;
    pixel_corner(a.cam, ix, iy, px, py, pz);
    const int64_t limit = replay ? a.rec_n[ray] : a.max_steps;
    const float* hs = replay ? a.rec_h + ray * a.rec_cap : nullptr;
    float I = 0.0f, z = a.z0, h = 1.0f, k1 = 0.0f;
    unsigned long long steps = 0;
    ScatterSlots prev;  // point 2 of the last accepted step: the next one's k1
    double prev_c = 0.0;
    bool have_prev = false;
    Walk4Stats ws;
    while ((int64_t)steps < limit && (replay || z < a.z_end)) {
      if (replay) h = hs[steps];
      float pts[4];
      rkf_points(z, h, pts);
      Step4 s;
      s4_bind(s, slot_mem);
      nn8_walk_step4<true>(g, spiral, px, py, pz, lx, ly, lz, pts, s, ws);
      const float zb = z, hb = h;
      if (replay) {
        z += h;
      } else {
        const float e[4] = {s4_value<0, true>(g, s), s4_value<1, true>(g, s),
                            s4_value<2, true>(g, s), s4_value<3, true>(g, s)};
        if (a.controller == ILC_CONTROLLER_REF32)
          rkf_advance_ref32(I, z, h, k1, fa, fr, a.z_end, e, kEps, kHmin, kHmax, pts);
        else
          rkf_advance_fp64(I, z, h, k1, a.atol, a.rtol, a.z_end, e, kEps, kHmin, kHmax, pts);
      }
      ++steps;
      if (!replay && z == zb) continue;
      scatter_point<0>(s, gi * (hb * 1408.f / 2565.f), a.grad);
      scatter_point<1>(s, gi * (hb * 2197.f / 4101.f), a.grad);
      if (have_prev) scatter(prev, prev_c + (double)(gi * (hb * 25.f / 216.f)), a.grad);
      scatter_slots<2>(s, prev);
      prev_c = (double)(gi * (-hb / 5.f));
      have_prev = true;
    }
    if (have_prev) scatter(prev, prev_c, a.grad);
    if (!replay && z < a.z_end) atomicOr(flags, FLAG_STEP_LIMIT);
    atomicAdd(&stats[0], steps);
    atomicAdd(&stats[3], (unsigned long long)ws.cells);
    atomicAdd(&stats[4], (unsigned long long)ws.cands);
  }
}

// dL/dln rho and dL/dln T in the original particle order.
__global__ void cell_grad_kernel(const double* __restrict__ grad_sorted,
                                 const uint32_t* __restrict__ s2u, uint64_t n,
                                 const float* __restrict__ dq_lnrho,
                                 const float* __restrict__ dq_lnT, float* __restrict__ g_lnrho,
                                 float* __restrict__ g_lnT) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t o = s2u[i];
  const double gq = grad_sorted[i];
  g_lnrho[o] = (float)(gq * (double)dq_lnrho[o]);
  g_lnT[o] = (float)(gq * (double)dq_lnT[o]);
}

}  // namespace

GridView make_grid_view(const Context& c);

cudaError_t adjoint_cell_launch(Context& c, const float* rho, const float* u, const float* xe,
                                uint64_t n, float z, float dL, float emin, float emax,
                                int num_samples, float* q_out, int q_stride, float* dq_lnT,
                                float* dq_lnrho) {
  GauntView G{c.gw, c.gh, c.gx0, c.gy0, c.gdx, c.gdy};
  const uint64_t want = (n + 255) / 256;
  const unsigned blocks = (unsigned)(want < 148 * 16 ? want : 148 * 16);
  ++c.launches;
  xray_flux_grad_kernel<<<blocks, 256, 0, c.stream>>>(c.gaunt.as<float>(), G, rho, u, xe, n, z,
                                                       dL, emin, emax, num_samples, q_out,
                                                       q_stride, dq_lnT, dq_lnrho);
  return cudaGetLastError();
}

cudaError_t adjoint_seed_launch(Context& c, const float* img, const float* target, int64_t npix,
                                float scale, float* seed, double* loss, bool reset_loss) {
  if (reset_loss) {
    cudaError_t e = cudaMemsetAsync(loss, 0, sizeof(double), c.stream);
    if (e) return e;
  }
  ++c.launches;
  loss_seed_kernel<<<148 * 4, 256, 0, c.stream>>>(img, target, npix, scale, seed, loss);
  return cudaGetLastError();
}

cudaError_t adjoint_ray_launch(Context& c, const RenderArgs& r, int mode, const float* seed,
                               double* grad, float* kernel_ms) {
  cudaError_t e;
  if ((e = c.flags.ensure(kFlagsBytes))) return e;
  if ((e = cudaMemsetAsync(c.flags.p, 0, kFlagsBytes, c.stream))) return e;
  AdjK k;
  k.cam.look0 = r.cam[0]; k.cam.look1 = r.cam[1]; k.cam.look2 = r.cam[2];
  k.cam.b00 = r.cam[3]; k.cam.b01 = r.cam[4]; k.cam.b02 = r.cam[5];
  k.cam.b10 = r.cam[6]; k.cam.b11 = r.cam[7]; k.cam.b12 = r.cam[8];
  k.cam.min0 = r.cam[9]; k.cam.min1 = r.cam[10]; k.cam.min2 = r.cam[11];
  k.cam.ps = r.cam[12];
  k.cam.nx = r.nx; k.cam.ny = r.ny;
  k.z0 = r.z0; k.z_end = r.z_end;
  k.atol = r.atol; k.rtol = r.rtol;
  k.controller = r.controller;
  k.max_steps = c.max_steps;
  k.mode = mode;
  k.rec_h = r.rec_h;
  k.rec_n = r.rec_n;
  k.rec_cap = r.rec_cap;
  k.seed = seed;
  k.grad = grad;
  k.row0 = r.row0;
  k.row_end = r.rows > 0 ? (r.row0 + r.rows < r.ny ? r.row0 + r.rows : r.ny) : r.ny;
  const GridView g = make_grid_view(c);
  k.tiles_x = (unsigned)((r.nx + 15) / 16);
  const unsigned long long tiles =
      (unsigned long long)k.tiles_x * (unsigned)((k.row_end - k.row0 + 7) / 8);
  k.n_rays = 128ull * tiles;
  if ((e = c.tile_queue.ensure(256))) return e;
  if ((e = cudaMemsetAsync(c.tile_queue.p, 0, 16, c.stream))) return e;
  k.queue = c.tile_queue.as<unsigned long long>();
  // (the rays of the forward pass over the same rows)
  k.leave = c.leave;
  int sms = 0, per_sm = 0, per_sm_w = 0;
  if ((e = cudaFuncSetAttribute(adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(AdjMem))) ||
      (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device)) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, adjoint_kernel, kListThreads,
                                                         sizeof(AdjMem))) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_w, adjoint_walk_kernel,
                                                         kSlotThreads, 0)))
    return e;
  const unsigned long long resident = (unsigned long long)sms * (per_sm > 0 ? per_sm : 1);
  // (down to one ray per warp)
  const unsigned long long most = 128 / kListWarps * tiles;
  const unsigned blocks = (unsigned)(resident < most ? resident : most);
  if ((e = c.list_over.ensure((size_t)blocks * kListWarps * kRays * kOver * 16))) return e;
  k.over = c.list_over.as<float4>();
  if (!c.ev0) {
    if ((e = cudaEventCreate(&c.ev0)) || (e = cudaEventCreate(&c.ev1))) return e;
  }
  cudaEventRecord(c.ev0, c.stream);
  if (k.leave.left) {
    const unsigned long long fit = (unsigned long long)sms * (per_sm_w > 0 ? per_sm_w : 1);
    ++c.launches;
    adjoint_walk_kernel<<<(unsigned)(fit < tiles ? fit : tiles), kSlotThreads, 0, c.stream>>>(
        k, g, c.spiral.as<char4>(), c.flags.as<uint32_t>(),
        reinterpret_cast<unsigned long long*>(c.flags.as<char>() + 64));
    if ((e = cudaGetLastError())) return e;
  }
  ++c.launches;
  adjoint_kernel<<<blocks, kListThreads, sizeof(AdjMem), c.stream>>>(
      k, g, c.spiral.as<char4>(), c.flags.as<uint32_t>(),
      reinterpret_cast<unsigned long long*>(c.flags.as<char>() + 64));
  if ((e = cudaGetLastError())) return e;
  cudaEventRecord(c.ev1, c.stream);
  if (kernel_ms) {
    if ((e = cudaEventSynchronize(c.ev1))) return e;
    cudaEventElapsedTime(kernel_ms, c.ev0, c.ev1);
  }
  return cudaSuccess;
}

cudaError_t adjoint_chain_launch(Context& c, const double* grad, uint64_t n, const float* dq_lnrho,
                                 const float* dq_lnT, float* g_lnrho, float* g_lnT) {
  ++c.launches;
  cell_grad_kernel<<<(unsigned)((n + 255) / 256), 256, 0, c.stream>>>(
      grad, c.s2u.as<uint32_t>(), n, dq_lnrho, dq_lnT, g_lnrho, g_lnT);
  return cudaGetLastError();
}

}  // namespace ilc
