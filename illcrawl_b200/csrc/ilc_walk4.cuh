// ilc_walk4.cuh -- the nn8 walk for the 4 integrand points of one RKF step,
// done as one pass over the grid.
//
// The 4 points of a step lie within one step length (typically < 1 kpc) of
// each other, so almost always in the same grid cell and subcell: they then
// share the reference's spiral cell order, and one walk serves all four. Each
// point keeps its own 8 slots, its own search radius and its own early break
// (volumetric_nn8_reconstruction.cl:157-171): a point stops taking part at the
// cell where its own break condition holds, exactly as its single-point walk
// would. Every point therefore sees the same cells and candidates in the same
// order as alone, and its slots evolve identically -- the result is the
// reference's, bit for bit. What is shared is the spiral/cell bookkeeping and
// the candidate loads (one 16-byte load serves four distance tests). Points in
// a different cell or subcell are walked in a further pass.
//
// Used for steps that are long against a cell over many rays, where a candidate
// list (ilc_raylist.cuh) would serve too few steps: one walk costs about the same
// whatever the step, and 32 neighbouring rays share its cells in L1 (1024^2 rays x
// 64 fixed steps through 1,048,576 cells: 62 ms, with lists 558 ms).
// Bound by instruction issue and, below some 20,000 rays, by the warp that
// crosses the densest cells.
#pragma once

#include "ilc_internal.h"
#include "ilc_raylist.cuh"

namespace ilc {

// Threads per block of every kernel that walks with Step4: the slot arrays of
// thread i live in shared memory at index i of each of the 64 rows.
constexpr int kSlotThreads = 128;
constexpr int kSlotRows = 4 * 8;  // (point, slot) pairs

// Shared-memory storage of one block's slot arrays: distance rows, then value
// (or index) rows; row (j, t) holds entry t of point j for all threads.
struct SlotMem {
  float d[kSlotRows][kSlotThreads];
  float v[kSlotRows][kSlotThreads];
};

// Counters of a walked ray.
struct Walk4Stats : WalkStats {
  uint32_t scans = 0;  // candidates scanned, a quarter of those behind codes
};

struct Step4 {
  float qx[4], qy[4], qz[4];
  float* sd;      // this thread's distance column: sd[(j * 8 + t) * kSlotThreads]
  float* sv;      // this thread's value column
  float R[4];
  float rr[4];    // (R + cell_radius)^2: the early-break threshold
  float crad;     // cell radius
  unsigned mi;    // per point j, bits 4j..4j+3: its first maximal slot; while
                  // R == FLT_MAX: its next empty slot
};

__device__ __forceinline__ float& s4_d(const Step4& s, int j, int t) {
  return s.sd[(j * 8 + t) * kSlotThreads];
}
__device__ __forceinline__ float& s4_v(const Step4& s, int j, int t) {
  return s.sv[(j * 8 + t) * kSlotThreads];
}

__device__ __forceinline__ void s4_bind(Step4& s, SlotMem& m) {
  s.sd = &m.d[0][threadIdx.x];
  s.sv = &m.v[0][threadIdx.x];
}

template <int J> __device__ __forceinline__ void s4_set_mi(Step4& s, unsigned k) {
  s.mi = (s.mi & ~(15u << (4 * J))) | (k << (4 * J));
}

// The larger of two (distance, slot) pairs, the left one on ties.
__device__ __forceinline__ void max_left(float& d, int& i, float d2, int i2) {
  const bool right = d2 > d;
  d = right ? d2 : d;
  i = right ? i2 : i;
}

// Search radius and first maximal slot (volumetric_nn8_reconstruction.cl:
// 135-143), as a pairwise tournament: three levels instead of a chain of
// eight; keeping the left pair on ties gives the first slot holding the
// maximum, as the sequential scan does (distances are non-negative, so the
// scan's start at 0 changes nothing).
template <int J> __device__ __forceinline__ void s4_rescan(Step4& s) {
  float d[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) d[t] = s4_d(s, J, t);
  int i0 = 0, i2 = 2, i4 = 4, i6 = 6;
  float a0 = d[0], a2 = d[2], a4 = d[4], a6 = d[6];
  max_left(a0, i0, d[1], 1);
  max_left(a2, i2, d[3], 3);
  max_left(a4, i4, d[5], 5);
  max_left(a6, i6, d[7], 7);
  max_left(a0, i0, a2, i2);
  max_left(a4, i4, a6, i6);
  max_left(a0, i0, a4, i4);
  const float r = a0;
  const int m = i0;
  s.R[J] = r;
  s4_set_mi<J>(s, (unsigned)m);
  const float b = r + s.crad;
  s.rr[J] = b * b;
}

template <int J> __device__ __forceinline__ void s4_init(Step4& s, float empty_value) {
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    s4_d(s, J, t) = FLT_MAX;
    s4_v(s, J, t) = empty_value;
  }
  s.R[J] = FLT_MAX;
  const float b = FLT_MAX + s.crad;
  s.rr[J] = b * b;
  s4_set_mi<J>(s, 0u);
}

// Insertion into point J's slots. While fewer than 8 slots are filled the
// search radius is FLT_MAX (a full set of 8 finite distances makes it
// smaller) and the first-max slot is the next empty one, so the k-th
// accepted candidate goes to slot k without a rescan; the 8th insertion
// rescans. Afterwards: replace the first-max slot and rescan.
template <int J> __device__ __forceinline__ void s4_insert(Step4& s, float dist, float val) {
  const int k = (int)((s.mi >> (4 * J)) & 15u);
  s4_d(s, J, k) = dist;
  s4_v(s, J, k) = val;
  if (s.R[J] == FLT_MAX) {
    s4_set_mi<J>(s, (unsigned)(k + 1));
    if (k == 7) s4_rescan<J>(s);
  } else {
    s4_rescan<J>(s);
  }
}

// Squared-distance threshold of point J: R*R rounded up (a squared distance
// above it cannot give dist < R); +inf while R is FLT_MAX.
template <int J> __device__ __forceinline__ float s4_r2up(const Step4& s) {
  return __fmul_ru(s.R[J], s.R[J]);
}

// Candidate test of point J against its threshold thr: s4_r2up while J takes
// part in the walk, -1 once it has left it (no squared distance passes). thr
// follows R through insertions.
template <int J>
__device__ __forceinline__ void s4_test(Step4& s, float& thr, float d2, float val) {
  if (d2 <= thr) {
    const float dist = sqrtf(d2);
    if (dist < s.R[J]) {
      s4_insert<J>(s, dist, val);
      thr = s4_r2up<J>(s);
    }
  }
}

// Weights of point J's slots (get_weight3d) and their sum, in slot order.
template <int J> __device__ __forceinline__ void s4_weights(const Step4& s, float w[8], float& ws) {
#pragma unroll
  for (int t = 0; t < 8; ++t) w[t] = weight3d(s4_d(s, J, t));
  ws = 0.0f;
#pragma unroll
  for (int t = 0; t < 8; ++t) ws = ws + w[t];
}

// Value of point J (finalize order). kIdx: the slots hold sorted indices, the
// values are read from vals, or from the particles where that is null.
template <int J, bool kIdx>
__device__ __forceinline__ float s4_value(const GridView& g, const Step4& s) {
  float w[8], ws;
  s4_weights<J>(s, w, ws);
  float dot = 0.0f;
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    float v = s4_v(s, J, t);
    if (kIdx) {
      const int id = __float_as_int(v);
      v = id < 0 ? 0.0f : (g.vals ? __ldg(&g.vals[id]) : __ldg(&g.parts[id].w));
    }
    dot = __fmaf_rn(w[t], v, dot);
  }
  return (ws != 0.0f && dot != 0.0f) ? dot / ws : 0.0f;
}

__device__ __forceinline__ void cand_insert(Step4& s, float thr[4], const float d2[4],
                                            float pay) {
  s4_test<0>(s, thr[0], d2[0], pay);
  s4_test<1>(s, thr[1], d2[1], pay);
  s4_test<2>(s, thr[2], d2[2], pay);
  s4_test<3>(s, thr[3], d2[3], pay);
}

// Candidate p against the active points; the slots take its value, or (kIdx) its
// sorted index.
// With a shared x/y part, every point's squared distance is fl(fxy + fz^2)
// >= fxy (rounding is monotone and fz^2 >= 0), so a candidate whose fxy
// exceeds the largest threshold thrmax cannot be inserted for any point.
// thrmax may be stale (larger than the current thresholds): the test only
// skips work that could not insert.
template <bool kSharedXY, bool kIdx>
__device__ __forceinline__ void test_candidate(Step4& s, float thr[4], float thrmax,
                                               const float4& P, int p) {
  float d2[4];
  if (kSharedXY) {
    const float fx = P.x - s.qx[0], fy = P.y - s.qy[0];
    const float fxy = fx * fx + fy * fy;
    if (fxy > thrmax) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float fz = P.z - s.qz[j];
      d2[j] = fxy + fz * fz;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float fx = P.x - s.qx[j], fy = P.y - s.qy[j], fz = P.z - s.qz[j];
      d2[j] = (fx * fx + fy * fy) + fz * fz;
    }
  }
  cand_insert(s, thr, d2, kIdx ? __int_as_float(p) : P.w);
}

// Cells with more candidates than this are scanned through their sub-box codes.
constexpr int kPruneMin = 16;

// Field range of the sub-boxes of a cell that meet the box [qlo - ext, qhi + ext]
// (code_hits): the union of the cubes of half-width ext = max R + margin around
// the active points. A candidate in any other sub-box is farther than its
// point's R from every active point (the margin exceeds every rounding error of
// the codes and of the distance), so it would not be inserted. False: none.
__device__ __forceinline__ bool prune_range(const GridView& g, int ix, int iy, int iz,
                                            const float qlo[3], const float qhi[3], float ext,
                                            uint32_t& lo, uint32_t& hi) {
  const float mx = g.min0 + (float)ix * g.cs0;
  const float my = g.min1 + (float)iy * g.cs1;
  const float mz = g.min2 + (float)iz * g.cs2;
  uint32_t l0, l1, l2, h0, h1, h2;
  const bool x = code_range(qlo[0] - ext - mx, qhi[0] + ext - mx, g.inv_w0, l0, h0);
  const bool y = code_range(qlo[1] - ext - my, qhi[1] + ext - my, g.inv_w1, l1, h1);
  const bool z = code_range(qlo[2] - ext - mz, qhi[2] + ext - mz, g.inv_w2, l2, h2);
  lo = (l0 | (l1 << 5) | (l2 << 10)) * 0x10001u;
  hi = ((h0 | (h1 << 5) | (h2 << 10)) * 0x10001u) | kGuard;
  return x && y && z;
}

// One walk over the spiral of (cx, cy, cz, sub) for the points in `mask`.
// kSharedXY: all 4 points have bit-identical x and y (a view along the z
// axis), so the x/y part of every squared distance, (dx*dx + dy*dy), is one
// value for the 4 points and is evaluated once -- the same operations in the
// same order, hence the same bits, as evaluating it per point.
template <bool kSharedXY, bool kIdx>
__device__ __forceinline__ void walk4(const GridView& g, const char4* __restrict__ spiral,
                                      Step4& s, unsigned mask, int cx, int cy, int cz, int sub,
                                      Walk4Stats& st) {
  const char4* order = spiral + sub * 125;
  unsigned act = mask;
  float thr[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) thr[j] = ((mask >> j) & 1u) ? __fmul_ru(s.R[j], s.R[j]) : -1.0f;
  // bounding box of the group's points (for the sub-box pruning)
  float qlo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, qhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if ((mask >> j) & 1u) {
      qlo[0] = fminf(qlo[0], s.qx[j]); qhi[0] = fmaxf(qhi[0], s.qx[j]);
      qlo[1] = fminf(qlo[1], s.qy[j]); qhi[1] = fmaxf(qhi[1], s.qy[j]);
      qlo[2] = fminf(qlo[2], s.qz[j]); qhi[2] = fmaxf(qhi[2], s.qz[j]);
    }
  for (int it = 0; it < 125; ++it) {
    const char4 o = order[it];
    const int ix = cx + o.x, iy = cy + o.y, iz = cz + o.z;
    const float ccx = (g.min0 + (float)ix * g.cs0) + g.half0;
    const float ccy = (g.min1 + (float)iy * g.cs1) + g.half1;
    const float ccz = (g.min2 + (float)iz * g.cs2) + g.half2;
    {
      // early break per point: |c - q|^2 > (R + cell_radius)^2
      unsigned brk = 0;
      if (kSharedXY) {
        const float ex = ccx - s.qx[0], ey = ccy - s.qy[0];
        const float exy = ex * ex + ey * ey;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float ez = ccz - s.qz[j];
          if (exy + ez * ez > s.rr[j]) brk |= 1u << j;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float ex = ccx - s.qx[j], ey = ccy - s.qy[j], ez = ccz - s.qz[j];
          if ((ex * ex + ey * ey) + ez * ez > s.rr[j]) brk |= 1u << j;
        }
      }
      act &= ~brk;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((brk >> j) & 1u) thr[j] = -1.0f;
    }
    if (!act) break;
    if ((unsigned)ix >= (unsigned)g.n0 || (unsigned)iy >= (unsigned)g.n1 ||
        (unsigned)iz >= (unsigned)g.n2)
      continue;
    // largest insertion threshold of the points still walking, fixed for
    // this cell (thresholds only shrink, so it stays an upper bound)
    const float thrmax = fmaxf(fmaxf(thr[0], thr[1]), fmaxf(thr[2], thr[3]));
    // ix + iy nx + iz nx ny, in 32 bits (the grid build rejects 2^32 cells or more)
    const uint32_t key = (uint32_t)ix + (uint32_t)g.n0 * ((uint32_t)iy + (uint32_t)g.n1 * (uint32_t)iz);
    const int2 be = __ldg(&g.cells[key]);
    const unsigned na = __popc(act);
    st.cells += na;
    st.cands += na * (uint32_t)max(be.y - be.x, 0);
    if (be.x >= be.y) continue;
    {
      // Every particle of the cell lies in its box (to within the rounding of
      // the cell keys, which g.margin covers). If the box is farther from the
      // points' bounding box than the largest threshold allows, no candidate
      // of the cell can be inserted for any point: the cell is counted as
      // visited, and its scan is skipped.
      const float gx = fmaxf(fmaxf(qlo[0] - (ccx + g.half0), (ccx - g.half0) - qhi[0]) - g.margin,
                             0.0f);
      const float gy = fmaxf(fmaxf(qlo[1] - (ccy + g.half1), (ccy - g.half1) - qhi[1]) - g.margin,
                             0.0f);
      const float gz = fmaxf(fmaxf(qlo[2] - (ccz + g.half2), (ccz - g.half2) - qhi[2]) - g.margin,
                             0.0f);
      if ((gx * gx + gy * gy) + gz * gz > thrmax) continue;
    }
    st.scans += be.y - be.x > kPruneMin ? (uint32_t)(be.y - be.x) >> 2 : (uint32_t)(be.y - be.x);
    if (be.y - be.x > kPruneMin) {
      // Dense cell: candidates in ascending index order, 8 codes per load. The
      // range follows the search radius as it shrinks while the cell is scanned
      // (one from a larger radius stays conservative), and once no sub-box is
      // within reach no later candidate of the cell can be inserted.
      float rused = -1.0f;
      uint32_t lo = 0, hi = 0;
      for (int pw = be.x & ~7; pw < be.y; pw += 8) {
        float rmax = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if ((act >> j) & 1u) rmax = fmaxf(rmax, s.R[j]);
        if (rmax != rused) {
          rused = rmax;
          if (!prune_range(g, ix, iy, iz, qlo, qhi, rmax + g.margin, lo, hi)) break;
        }
        unsigned hits = code_hits(load_codes(g, pw, 0), lo, hi, pw, be.x, be.y);
        while (hits) {
          const int p = pw + __ffs(hits) - 1;
          hits &= hits - 1;
          test_candidate<kSharedXY, kIdx>(s, thr, thrmax, __ldg(&g.parts[p]), p);
        }
      }
      continue;
    }
    float4 P = __ldg(&g.parts[be.x]);
    for (int p = be.x; p < be.y; ++p) {
      const float4 N = (p + 1 < be.y) ? __ldg(&g.parts[p + 1]) : P;  // prefetch
      test_candidate<kSharedXY, kIdx>(s, thr, thrmax, P, p);
      P = N;
    }
  }
}

// nn8 walk of the 4 points of one step; the slots are left in s.
template <bool kIdx>
__device__ __forceinline__ void nn8_walk_step4(const GridView& g,
                                               const char4* __restrict__ spiral, float px,
                                               float py, float pz, float lx, float ly, float lz,
                                               const float zq[4], Step4& s, Walk4Stats& st) {
  int cx[4], cy[4], cz[4], sb[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    s.qx[j] = px + zq[j] * lx;
    s.qy[j] = py + zq[j] * ly;
    s.qz[j] = pz + zq[j] * lz;
  }
  const bool shared_xy = (s.qx[0] == s.qx[1] && s.qx[0] == s.qx[2] &&
                                   s.qx[0] == s.qx[3] && s.qy[0] == s.qy[1] &&
                                   s.qy[0] == s.qy[2] && s.qy[0] == s.qy[3]);
  // points with bit-identical x and y (a view along z) share their x/y cell
  // and subcell: located once
  int cx0, sx0, cy0, sy0;
  locate_axis(s.qx[0], g.min0, g.cs0, g.half0, cx0, sx0);
  locate_axis(s.qy[0], g.min1, g.cs1, g.half1, cy0, sy0);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    int sx = sx0, sy = sy0, sz;
    cx[j] = cx0;
    cy[j] = cy0;
    if (j > 0 && !shared_xy) {
      locate_axis(s.qx[j], g.min0, g.cs0, g.half0, cx[j], sx);
      locate_axis(s.qy[j], g.min1, g.cs1, g.half1, cy[j], sy);
    }
    locate_axis(s.qz[j], g.min2, g.cs2, g.half2, cz[j], sz);
    sb[j] = sx + 2 * sy + 4 * sz;
  }
  s.crad = g.cell_radius;
  const float empty = kIdx ? __int_as_float(-1) : 0.0f;
  s4_init<0>(s, empty);
  s4_init<1>(s, empty);
  s4_init<2>(s, empty);
  s4_init<3>(s, empty);
  unsigned todo = 0xFu;
  while (todo) {
    const int j0 = __ffs(todo) - 1;
    int c0x = cx[0], c0y = cy[0], c0z = cz[0], s0 = sb[0];
#pragma unroll
    for (int j = 1; j < 4; ++j)
      if (j == j0) { c0x = cx[j]; c0y = cy[j]; c0z = cz[j]; s0 = sb[j]; }
    unsigned mask = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (((todo >> j) & 1u) && cx[j] == c0x && cy[j] == c0y && cz[j] == c0z && sb[j] == s0)
        mask |= 1u << j;
    if (shared_xy)
      walk4<true, kIdx>(g, spiral, s, mask, c0x, c0y, c0z, s0, st);
    else
      walk4<false, kIdx>(g, spiral, s, mask, c0x, c0y, c0z, s0, st);
    todo &= ~mask;
  }
}

// nn8 values of the 4 points of one step (e[j] for point j).
template <bool kIdx>
__device__ __forceinline__ void nn8_step4(const GridView& g, const char4* __restrict__ spiral,
                                          SlotMem& sm, float px, float py, float pz, float lx,
                                          float ly, float lz, const float zq[4], float e[4],
                                          Walk4Stats& st) {
  Step4 s;
  s4_bind(s, sm);
  nn8_walk_step4<kIdx>(g, spiral, px, py, pz, lx, ly, lz, zq, s, st);
  e[0] = s4_value<0, kIdx>(g, s);
  e[1] = s4_value<1, kIdx>(g, s);
  e[2] = s4_value<2, kIdx>(g, s);
  e[3] = s4_value<3, kIdx>(g, s);
}

// ---------------------------------------------------------------------------
// Adaptive steps. Whether a list serves a ray's steps well is known only on the
// way: steps long against a cell, of a loose tolerance away from the cores, use a
// list once and are walked; short ones, and steps through dense cells, which one
// thread would scan while the others wait, are left to the lists. A launch of many
// rays therefore walks first and marks the rays it leaves; the list kernel takes
// these from their start, in its own order (the costliest first; a few steps each
// are done twice). Projections of 262,144 cells, lists alone -> walk and lists, in ms
// (the walk alone, as it was before there were lists): outer 500 kpc at rtol 1e-2
// 256^2 5.6 -> 3.1 (3.2), 512^2 20.7 -> 5.9 (6.4), 1024^2 79.6 -> 16.9 (18.7), at 2e-3
// 10 -> 10 (17), 36 -> 13 (20), 137 -> 39 (41), at 1e-3 42 -> 42 (92), 129 -> 127 (154);
// 2 Mpc through the core at 1e-2: 43 -> 45 (531), 113 -> 70 (507), 422 -> 183 (418).
// Band map of 4,194,304 cells, 500 kpc, 1e-2, 1024^2: 111 -> 38 (45). 32 channels of
// the outer slab, 512^2, 1e-2: 80 -> 29 (31); adjoint of a 256^2 map, 100 kpc, 1e-2:
// 11.5 -> 6.4 (6.1). The walk's kernels take 4 blocks of 128 threads per SM (128
// registers).
// ---------------------------------------------------------------------------
// What the list kernels take from their queue: all rays, or those left.
__device__ __forceinline__ unsigned long long list_rays(const LeaveRule& r,
                                                        unsigned long long all) {
  return r.left ? *r.n_left : all;
}
__device__ __forceinline__ unsigned long long list_ray(const LeaveRule& r, unsigned long long q) {
  return r.left ? r.list[q] : q;
}

// A ray begins with short steps whatever its tolerance (h = 1, then the least one,
// 0.2), which grow by the step. Looks at the pace come every kNextLook steps, the
// first three by rules of their own.
constexpr uint32_t kNextLook = 8, kFirstLook = 8, kSecondLook = 16, kThirdLook = 24;
constexpr uint32_t kDenseStep = 512;  // scans of a step's 4 points

struct Pace {
  float z;
  uint32_t next;
};

__device__ __forceinline__ Pace pace_start(float z) { return Pace{z, kFirstLook}; }

// After a step of a ray to z_end that ended at z, with the next one h, and made
// `scans` scans: is the ray to be left?
__device__ __forceinline__ bool pace_slow(Pace& p, const LeaveRule& r, float z, float z_end,
                                          float h, unsigned long long steps, uint32_t scans) {
  if (z + h >= z_end) return false;  // the last step
  if (scans > kDenseStep) return true;
  if (steps < p.next) return false;
  float rays = r.rays, pace = (z - p.z) / (float)kNextLook;
  // What the steps grow to: h after 8 and 16 steps is 0.21 and 0.28 at rtol 1e-3, 0.34
  // and 0.9 at 1.5e-3, 0.5 and 2 at 2e-3, 1 and 7 at 3e-3, 6 and 100 (the largest step)
  // at 1e-2, and the later mean steps are some 1, 7, 11, 15 and 25.
  if (p.next == kFirstLook) {
    pace = (h * h) * (h * h) / (kHmin * kHmin * kHmin);
  } else if (p.next == kSecondLook) {
    pace = 2.0f * h;
  } else if (p.next != kThirdLook) {
    // The rays still under way are those the lists would get. They make their steps
    // again: the more there are of these against those still to come, the dearer.
    rays -= (float)*(volatile unsigned long long*)r.done;
    rays *= 1.0f + (float)steps * pace / (z_end - z);
  }
  p.z = z;
  p.next += kNextLook;
  return pace < fmaxf(r.even / fmaxf(rays - r.line, 1.0f), r.least);
}

// The ray of a 16 x 8 tile that this thread walks, in the list kernels' numbering (4 x
// 2 pixels in a row of 8 rays): each warp an 8 x 4 block of pixels, so its 32 rays are
// neighbours.
__device__ __forceinline__ unsigned walk_ray() {
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, b = lane >> 3;
  const unsigned sub = (2 * (warp >> 1) + (b >> 1)) * 4 + 2 * (warp & 1u) + (b & 1u);
  return 8 * sub + (lane & 7u);
}

// The marks of a warp's rays, 8 of which in a row have numbers in a row.
__device__ __forceinline__ void mark_left(const LeaveRule& r, bool active, bool leave,
                                          unsigned long long ray, int lane) {
  const unsigned m = __ballot_sync(kAll, leave), n = __popc(__ballot_sync(kAll, active));
  if ((lane & 7) == 0) r.left[ray >> 3] = (uint8_t)(m >> lane);
  if (lane == 0) atomicAdd(r.done, (unsigned long long)n);
}

}  // namespace ilc
