// ilc_quantity.cuh -- per-cell X-ray quantities of the reference
// (quantities.cl:38-136, 156-239) as device functions, shared by the quantity
// kernels and the adjoint.
//
// The OpenCL image lookup (read_imagef, CLK_FILTER_LINEAR, CLK_ADDRESS_CLAMP,
// unnormalised coordinates; tabulated_function.cl:26-59) is done in software
// with exact fp32 weights: the sample at u blends texels floor(u-0.5) and
// floor(u-0.5)+1 with weight frac(u-0.5); texels outside the table read 0.
#pragma once

#include "ilc_device.cuh"

namespace ilc {

// The table with two rows and columns of zeros around it: a lookup next to or
// outside the table then reads its zeros like any other texel. Very long or
// wide tables, which would not fit shared memory that way, stay unpadded.
constexpr int kPad = 2;
constexpr int kTableFloats = (81 + 2 * kPad) * (146 + 2 * kPad) + 2;  // a multiple of 4
inline int table_pad(int w, int h) {
  return (int64_t)(w + 2 * kPad) * (h + 2 * kPad) <= kTableFloats ? kPad : 0;
}

struct GauntView {
  int w, h;
  float x0, y0, dx, dy;
  int pad = 0;  // kPad, or 0: the table is not padded
};

__device__ __forceinline__ float texel(const float* __restrict__ t, const GauntView& G, int i,
                                       int j, int stride) {
  if (i < 0 || j < 0 || i >= G.w || j >= G.h) return 0.0f;
  return t[j * stride + i];
}

__device__ __forceinline__ float gaunt_sample(const float* __restrict__ t, const GauntView& G,
                                              float u, float v, int stride) {
  if (!(u == u) || !(v == v)) return 0.0f;
  u = fminf(fmaxf(u, -4.0f), (float)(G.w + 4));
  v = fminf(fmaxf(v, -4.0f), (float)(G.h + 4));
  const float us = u - 0.5f, vs = v - 0.5f;
  const float fu = floorf(us), fv = floorf(vs);
  const int i0 = (int)fu, j0 = (int)fv;
  const float a = us - fu, b = vs - fv;
  const float ia = 1.0f - a, ib = 1.0f - b;
  return ((ia * ib * texel(t, G, i0, j0, stride) + a * ib * texel(t, G, i0 + 1, j0, stride)) +
          ia * b * texel(t, G, i0, j0 + 1, stride)) +
         a * b * texel(t, G, i0 + 1, j0 + 1, stride);
}

// Constants of quantities.cl:29-36.
constexpr float kXH = 0.76f;
constexpr float kB = 8.61733e-5f;
constexpr float kRyd = 13.605f;

__device__ __forceinline__ float temperature(float u, float xe) {
  const float mu = 4.0f / (1.0f + 3.0f * kXH + 4.0f * kXH * xe);
  return (5.f / 3.f - 1.0f) * u * mu * 121.1475502f;
}

__device__ __forceinline__ float g_ff(const float* t, const GauntView& G, float E, float T,
                                      float Z, int stride) {
  const float gam2 = Z * Z * kRyd / (kB * T);
  const float u = 1.e3f * E / (kB * T);
  const float rx = (ilc_logf(gam2) - G.x0) / G.dx;
  const float ry = (ilc_logf(u) - G.y0) / G.dy;
  return gaunt_sample(t, G, rx, ry, stride);
}

// t: the table's first texel, rows of `stride`.
__device__ __forceinline__ float brems(const float* t, const GauntView& G, float E, float dE,
                                       float T, float xe, float rho, float r, int stride) {
  const float ion = 4.046263f * rho * xe;
  const float Z = 1.0f;
  const float Tinv = 1000.f / (kB * T);
  const float r2 = r * r;
  const float rs = 1.0f / sqrtf(T);
  return 0.002535f * dE * Z * Z * ion * ion * g_ff(t, G, E, T, Z, stride) * rs * ilc_expf(-E * Tinv) /
         r2;
}

// ---------------------------------------------------------------------------
// brems() with what depends on one cell, one energy or one call alone kept out
// of the inner loops. Every operation that remains is brems' own, in its order;
// its divisions by values that do not change from one evaluation to the next
// (kB T, the table spacing, r^2) go through their reciprocal. A cell or an
// energy outside the plain range (below) takes brems itself.
// ---------------------------------------------------------------------------

// a / b, correctly rounded, for y = 1 / b correctly rounded: q = a y is within
// two ulp, the first correction makes it faithful, the second correctly rounded
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990; no difference from IEEE division in 7e9 pairs, all-ones and
// near-one divisors among them). Needs a, b, a / b and a 2^-24 in the normal range.
__device__ __forceinline__ float div_by(float a, float b, float y) {
  float q = a * y;
  q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// Per call: 1 / table spacing along log u, r^2 and its reciprocal, the range of
// dividends of r^2 and then of a plain energy.
struct EmitCall {
  float dy, ydy, y0, r, r2, yr2, vmin, vmax;
  bool ok;
};

__device__ __forceinline__ bool plain_energy(float E) { return E >= 1e-8f && E <= 1e8f; }

__device__ __forceinline__ EmitCall emit_call(const GauntView& G, float r) {
  EmitCall k;
  k.dy = G.dy;
  k.ydy = 1.0f / G.dy;
  k.y0 = G.y0;
  k.r = r;
  k.r2 = r * r;
  k.yr2 = 1.0f / k.r2;
  // (r from 1e-10 to 1e10 in any unit: a luminosity distance is 3e7 kpc at redshift
  // 3.5 and 1e8 at 10; with brems for every cell, 1,000,000 cells take 210 us instead
  // of 91)
  k.ok = G.pad == kPad && G.dy >= 1e-6f && G.dy <= 1e6f && fabsf(G.y0) <= 1e6f && k.r2 >= 1e-20f &&
         k.r2 <= 1e20f;
  k.vmin = fmaxf(1e-20f, 1e-26f * k.r2);
  k.vmax = fminf(1e28f, 1e26f * k.r2);
  return k;
}

// Per cell. col: column of its left texel in the padded table; < 0: the cell
// takes brems.
struct EmitCell {
  float kbt, ykbt, tinv, rs, ion, a;
  int col;
};

__device__ __forceinline__ EmitCell emit_cell(const GauntView& G, const EmitCall& k, float T,
                                              float xe, float rho) {
  EmitCell c;
  c.kbt = kB * T;
  c.ykbt = 1.0f / c.kbt;
  c.tinv = 1000.f / c.kbt;
  c.rs = 1.0f / sqrtf(T);
  c.ion = 4.046263f * rho * xe;
  const float rx = (ilc_logf(kRyd / c.kbt) - G.x0) / G.dx;
  const float us = fminf(fmaxf(rx, -4.0f), (float)(G.w + 4)) - 0.5f;
  const float fu = floorf(us);
  const int i0 = (int)fu;
  c.a = us - fu;
  // (texels further out than the padding are zero as well)
  c.col = k.ok && rx == rx && c.kbt >= 1e-15f && c.kbt <= 1e15f
              ? min(max(i0, -kPad), G.w + kPad - 2) + kPad
              : -1;
  return c;
}

// (m - 1) / (m + 1) for m in [1/sqrt(2), sqrt(2)], correctly rounded: one Newton
// step on the hardware's reciprocal, then div_by (Markstein, as above; all
// of the 8,388,617 floats of the range compared with IEEE division: no difference).
__device__ __forceinline__ float log_ratio(float m) {
  const float b = m + 1.0f;
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  y = __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
  return div_by(m - 1.0f, b, y);
}

// ilc_logf of a positive normal number.
__device__ __forceinline__ float log_normal(float x) {
  const unsigned b = __float_as_uint(x);
  int e = (int)(b >> 23) - 127;
  float m = __uint_as_float((b & 0x007fffffu) | 0x3f800000u);
  const bool up = m > 1.41421356f;
  m = up ? m * 0.5f : m;
  e = up ? e + 1 : e;
  const float s = log_ratio(m);
  const float s2 = s * s;
  float p = 0.0909090909f;
  p = p * s2 + 0.111111111f;
  p = p * s2 + 0.142857143f;
  p = p * s2 + 0.2f;
  p = p * s2 + 0.333333333f;
  p = p * s2 + 1.0f;
  const float lm = (2.0f * s) * p;
  const float fe = (float)e;
  return fe * 0.693145751953125f + (lm + fe * 1.42860682e-06f);
}

// ilc_expf of a finite number that is not positive.
__device__ __forceinline__ float exp_negative(float x) {
  const float n = rintf(x * 1.44269504f);
  const float r = (x - n * 0.693145751953125f) - n * 1.42860682e-06f;
  float p = 1.98412698e-04f;
  p = p * r + 1.38888889e-03f;
  p = p * r + 8.33333333e-03f;
  p = p * r + 4.16666667e-02f;
  p = p * r + 1.66666667e-01f;
  p = p * r + 0.5f;
  p = p * r + 1.0f;
  p = p * r + 1.0f;
  const int ni = (int)n;
  const bool low = ni < -126;
  p = low ? p * __uint_as_float(0x00800000u) : p;
  const float v = p * __uint_as_float((unsigned)(ni + (low ? 126 + 127 : 127)) << 23);
  return x < -103.972084f ? 0.0f : v;
}

// brems with the table as it lies in shared memory.
static __device__ __noinline__ float brems_any(const float* t, const GauntView& G, float E,
                                               float dE, float T, float xe, float rho, float r) {
  const int stride = G.w + 2 * G.pad;
  return brems(t + G.pad * stride + G.pad, G, E, dE, T, xe, rho, r, stride);
}

// brems(E, dE) of a cell with its column in range, from the padded table t, for
// a plain energy; pre = 0.002535f * dE. kOverE: divided by E, whose reciprocal
// is yE. Without branches, so that several evaluations overlap; `ok` is cleared
// where a dividend leaves the range of div_by.
template <bool kOverE = false>
__device__ __forceinline__ float emit(const float* __restrict__ t, const GauntView& G,
                                      const EmitCall& k, const EmitCell& c, float E, float pre,
                                      bool& ok, float yE = 0.0f) {
  const float u = div_by(1.e3f * E, c.kbt, c.ykbt);
  const float ry = div_by(log_normal(u) - k.y0, k.dy, k.ydy);
  // (limits within the zeros around the table)
  const float vs = fminf(fmaxf(ry, -1.5f), (float)G.h + 0.5f) - 0.5f;
  const float fv = floorf(vs);
  const int row = (int)fv + kPad, stride = G.w + 2 * kPad;
  const float a = c.a, b = vs - fv;
  const float ia = 1.0f - a, ib = 1.0f - b;
  const float* __restrict__ q = t + row * stride + c.col;
  const float t00 = q[0], t10 = q[1], t01 = q[stride], t11 = q[stride + 1];
  const float g = ((ia * ib * t00 + a * ib * t10) + ia * b * t01) + a * b * t11;
  const float v = pre * c.ion * c.ion * g * c.rs * exp_negative(-E * c.tinv);
  // (zero, outside the table or beyond the exponential's range, stays zero)
  ok = ok && (v == 0.0f || (fabsf(v) >= k.vmin && fabsf(v) <= k.vmax));
  const float f = div_by(v, k.r2, k.yr2);
  return v == 0.0f ? v : (kOverE ? div_by(f, E, yE) : f);
}

// integrate_spectral_flux (quantities.cl:156-239): (rel_tol, 1) passed as
// (absolute, relative) tolerance, epsilon 0, step bounds [1e-3, 100].
// kPhoton = PHOTON_FLUX: every emission sample is divided by its energy.
template <bool kPhoton = false>
__device__ __forceinline__ float band_flux(const float* t, const GauntView& G, const EmitCall& k,
                                           float Emin, float Emax, float reltol, float T,
                                           float xe, float rho) {
  const EmitCell c = emit_cell(G, k, T, xe, rho);
  // (every sample lies between the limits)
  const bool plain = c.col >= 0 && plain_energy(Emin) && plain_energy(Emax);
  constexpr float pre = 0.002535f * 1.0f;
  float em = 0.0f, E = Emin;
  const float end = Emax;
  float dE = (end - E) * reltol;
  bool ok = plain;
  float k1 = plain ? emit(t, G, k, c, E, pre, ok) : 0.0f;
  if (!ok) k1 = brems_any(t, G, E, 1.0f, T, xe, rho, k.r);
  if (kPhoton) k1 = k1 / E;
  float p[4];
  rkf_points(E, dE, p);
  int guard = 0;
  while (E < end && guard < 100000) {
    float v[4];
    ok = plain;
    if (plain) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = emit(t, G, k, c, p[j], pre, ok);
    }
    if (!ok) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = brems_any(t, G, p[j], 1.0f, T, xe, rho, k.r);
    }
    if (kPhoton) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = v[j] / p[j];
    }
    rkf_advance_ref32(em, E, dE, k1, reltol, 1.0f, end, v, 0.0f, 1.e-3f, 100.f, p);
    ++guard;
  }
  return em;
}

// A 1D tabulated function (util::tabulated_function, tabulated_function.hpp:
// 35-103): n samples from x0 in steps of dx. Used for the Chandra ARF.
struct ArfView {
  int n;
  float x0, dx;
};

// evaluate_tabulated_function (tabulated_function.cl:31-44): the 1D form of
// the software image lookup above; samples outside the table read 0.
__device__ __forceinline__ float tab1d(const float* __restrict__ t, const ArfView& A, float x) {
  float u = (x - A.x0) / A.dx;
  if (!(u == u)) return 0.0f;
  u = fminf(fmaxf(u, -4.0f), (float)(A.n + 4));
  const float us = u - 0.5f;
  const float fu = floorf(us);
  const int i0 = (int)fu;
  const float a = us - fu;
  const float t0 = (i0 >= 0 && i0 < A.n) ? __ldg(t + i0) : 0.0f;
  const float t1 = (i0 + 1 >= 0 && i0 + 1 < A.n) ? __ldg(t + i0 + 1) : 0.0f;
  return (1.0f - a) * t0 + a * t1;
}

// A channel of get_chandra_xray_count_rate_with_temp (quantities.cl:432-460):
// the photon count rate of the channel (E, dE) at redshift z times the ARF at E
// (cm^2 -> m^2), get_spectral_brems_count_rate (quantities.cl:251-260) being
// the emission divided by the redshifted energy.
struct Channel {
  float Ez, yEz;  // redshifted energy and its reciprocal (0: not a plain energy)
  float dEz, pre; // redshifted width, 0.002535f * width
  float av;       // effective area
};

template <bool kRate>
__device__ __forceinline__ Channel make_channel(const float* __restrict__ arf, const ArfView& A,
                                                float E, float dE, float z) {
  Channel h;
  h.av = kRate ? tab1d(arf, A, E) * 1.e-4f : 0.0f;
  h.Ez = (1.f + z) * E;
  h.yEz = plain_energy(h.Ez) ? 1.0f / h.Ez : 0.0f;
  h.dEz = (1.f + z) * dE;
  h.pre = 0.002535f * h.dEz;
  return h;
}

// The channel's rate, or (kRate = false) its emission alone, of one cell.
template <bool kRate>
__device__ __forceinline__ float channel_value(const float* t, const GauntView& G,
                                               const EmitCall& k, const EmitCell& c,
                                               const Channel& h, float T, float xe, float rho) {
  bool ok = c.col >= 0 && h.yEz != 0.0f;
  float v = 0.0f;
  if (ok) v = emit<kRate>(t, G, k, c, h.Ez, h.pre, ok, h.yEz);
  if (!ok) {
    v = brems_any(t, G, h.Ez, h.dEz, T, xe, rho, k.r);
    if (kRate) v = v / h.Ez;
  }
  return kRate ? v * h.av : v;
}

}  // namespace ilc
