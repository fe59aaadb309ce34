// ilc_nn8.cu -- nn8 reconstruction at arbitrary query points: the fused
// volumetric_nn8_reconstruction + finalize kernels
// (volumetric_nn8_reconstruction.cl:87-270), one warp per query, or for many
// queries one lane per query, taken in the order of their cells and subcells.
//
// merge = false starts from empty lists (is_first_run); merge = true continues
// from the lists the previous call left, which is how the reference combines
// particle blocks (volumetric_nn8_reconstruction.cl:112-126).
#include <algorithm>

#include "ilc_device.cuh"
#include "ilc_internal.h"
#include "ilc_raylist.cuh"

namespace ilc {

namespace {

// Bin of a query point for the order in which the queries are taken: its cell
// (clamped to the grid) and subcell, shifted right to at most 2^kBinBits bins.
// Points of one bin share the spiral order, hence cells and candidates.
// Random queries left the lanes of a warp in cells far apart: 2^20 uniform
// queries of 262,144 particles took 3,284 us (a third of it one lane scanning
// the halo's core), now 654 us with 45 us for the sort and 92 us for the queries
// left to the warp kernel; 74 % of the issue slots, 13 of 32 lanes.
constexpr int kBinBits = 20;
struct QueryBins {
  int n0, n1, n2, shift;
};

__device__ __forceinline__ uint32_t query_bin(const GridView& g, const QueryBins& b,
                                              const float4& q) {
  // (order only: nothing depends on the rounding here; NaN goes to 0. The upper
  // limit is an integer one: 2 n - 1 as a float is 2 n, a cell too far, on axes
  // of more than 2^23 cells.)
  const float h0 = (q.x - g.min0) * (2.0f / g.cs0), h1 = (q.y - g.min1) * (2.0f / g.cs1),
              h2 = (q.z - g.min2) * (2.0f / g.cs2);
  const uint32_t i0 = min(__float2uint_rz(fmaxf(h0, 0.0f)), 2u * (uint32_t)b.n0 - 1u);
  const uint32_t i1 = min(__float2uint_rz(fmaxf(h1, 0.0f)), 2u * (uint32_t)b.n1 - 1u);
  const uint32_t i2 = min(__float2uint_rz(fmaxf(h2, 0.0f)), 2u * (uint32_t)b.n2 - 1u);
  const uint64_t cell = (i0 >> 1) + (uint64_t)b.n0 * ((i1 >> 1) + (uint64_t)b.n1 * (i2 >> 1));
  return (uint32_t)((8 * cell + ((i0 & 1u) | ((i1 & 1u) << 1) | ((i2 & 1u) << 2))) >> b.shift);
}

__global__ void query_count_kernel(GridView g, QueryBins b, const float4* __restrict__ pts,
                                   uint64_t n, uint32_t* __restrict__ count,
                                   uint2* __restrict__ place) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t k = query_bin(g, b, pts[i]);
  place[i] = make_uint2(k, atomicAdd(&count[k], 1u));
}

__global__ void query_order_kernel(const uint32_t* __restrict__ first,
                                   const uint2* __restrict__ place, uint64_t n,
                                   uint32_t* __restrict__ order) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint2 p = place[i];
  order[first[p.x] + p.y] = (uint32_t)i;
}

// Slots of one query: squared distances (kExact: distances, as the lists of a
// previous block hold them) and candidate indices.
struct QuerySlots {
  float d[8];
  int id[8];
};

// The walk of nn8_walk() (ilc_device.cuh) for one query; cells whose box lies
// beyond the search radius are counted and not scanned. Without lists to
// continue, squared distances can stand for distances, as in a list replay
// (ilc_raylist.cuh; kExact: distances themselves). Returns false, with the slots in
// no defined state, where two of them are too close for that, and at a cell with
// more than kHard candidates within reach, which one lane would scan while the
// others wait.
constexpr int kHard = 96;
template <bool kExact>
__device__ __forceinline__ bool query_walk(const GridView& g, const char4* __restrict__ spiral,
                                           float qx, float qy, float qz, QuerySlots& s,
                                           WalkStats& st) {
  int cx, cy, cz, sx, sy, sz;
  locate_axis(qx, g.min0, g.cs0, g.half0, cx, sx);
  locate_axis(qy, g.min1, g.cs1, g.half1, cy, sy);
  locate_axis(qz, g.min2, g.cs2, g.half2, cz, sz);
  const char4* order = spiral + (sx + 2 * sy + 4 * sz) * 125;
  const float inf = __int_as_float(0x7f800000);
  float M = max8(s.d);                            // the slot maximum
  float T = kExact ? __fmul_ru(M, M) : M;         // squared distances above it cannot enter
  float rb = (kExact ? M : fminf(sqrtf(M), FLT_MAX)) + g.cell_radius;
  float rr = rb * rb;
  bool close = false;
#pragma unroll 1
  for (int it = 0; it < 125; ++it) {
    const char4 o = order[it];
    const int ix = cx + o.x, iy = cy + o.y, iz = cz + o.z;
    const float ex = ((g.min0 + (float)ix * g.cs0) + g.half0) - qx;
    const float ey = ((g.min1 + (float)iy * g.cs1) + g.half1) - qy;
    const float ez = ((g.min2 + (float)iz * g.cs2) + g.half2) - qz;
    if ((ex * ex + ey * ey) + ez * ez > rr) break;
    if ((unsigned)ix >= (unsigned)g.n0 || (unsigned)iy >= (unsigned)g.n1 ||
        (unsigned)iz >= (unsigned)g.n2)
      continue;
    // in 32 bits (the grid build rejects 2^32 cells or more)
    const uint32_t key =
        (uint32_t)ix + (uint32_t)g.n0 * ((uint32_t)iy + (uint32_t)g.n1 * (uint32_t)iz);
    const int2 be = __ldg(&g.cells[key]);
    const int nc = max(be.y - be.x, 0);
    st.cells += 1;
    st.cands += (uint32_t)nc;
    if (nc == 0) continue;
    const float gx = fmaxf(fabsf(ex) - g.half0 - g.margin, 0.0f);
    const float gy = fmaxf(fabsf(ey) - g.half1 - g.margin, 0.0f);
    const float gz = fmaxf(fabsf(ez) - g.half2 - g.margin, 0.0f);
    if (((gx * gx + gy * gy) + gz * gz) * 0.99999f > T) continue;
    if (nc > kHard) return false;
    const float before = M;
    float4 P = __ldg(&g.parts[be.x]);
#pragma unroll 1
    for (int p = be.x; p < be.y; ++p) {
      const float4 C = P;
      P = __ldg(&g.parts[p + 1 < be.y ? p + 1 : p]);
      const float fx = C.x - qx, fy = C.y - qy, fz = C.z - qz;
      float d = (fx * fx + fy * fy) + fz * fz;
      if (d <= T) {
        if (kExact) d = sqrtf(d);
        if (d < M) {
          bool open = true;  // the first maximal slot
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const bool eq = s.d[q] == M;
            const bool hit = open && eq;
            open = open && !eq;
            s.d[q] = hit ? d : s.d[q];
            s.id[q] = hit ? p : s.id[q];
          }
          const float top = max8(s.d);
          if (!kExact) close = close || (M < inf && top >= M * 0.99999952f);
          M = top;
          T = kExact ? __fmul_ru(M, M) : M;
        }
      }
    }
    if (M != before) {
      rb = (kExact ? M : fminf(sqrtf(M), FLT_MAX)) + g.cell_radius;
      rr = rb * rb;
    }
  }
  return !close;
}

// One query per lane, in the given order or that of their bins; those that
// query_walk() gives up are listed in hard[0..]. kMerge implies kExact.
template <bool kMerge, bool kExact>
__global__ void __launch_bounds__(256)
nn8_query_kernel(const __grid_constant__ GridView g, const char4* __restrict__ spiral_g,
                 const float4* __restrict__ pts, const uint32_t* __restrict__ order, uint64_t n,
                 uint32_t* __restrict__ hard, uint32_t* __restrict__ n_hard, float* __restrict__ list_d, float* __restrict__ list_v,
                 int32_t* __restrict__ list_id, float* __restrict__ out,
                 int32_t* __restrict__ idx8, float* __restrict__ d8,
                 const uint32_t* __restrict__ s2u, unsigned long long* __restrict__ stats) {
  __shared__ char4 spiral[1000];
  load_spiral(spiral, spiral_g);
  const uint64_t turn = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  WalkStats st;
  if (turn < n) {
    const uint64_t i = order ? order[turn] : turn;
    const float4 q = pts[i];
    QuerySlots s;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      // Lists carry original indices; entries kept from the previous call are
      // tagged with the top bit so they are not mapped through this grid's s2u.
      s.d[j] = kMerge ? list_d[8 * i + j] : kExact ? FLT_MAX : __int_as_float(0x7f800000);
      const int32_t o = kMerge ? list_id[8 * i + j] : -1;
      s.id[j] = o >= 0 ? (int32_t)(0x80000000u | (uint32_t)o) : -1;
    }
    if (!query_walk<kExact>(g, spiral, q.x, q.y, q.z, s, st)) {
      st.cells = st.cands = 0;
      hard[atomicAdd(n_hard, 1u)] = (uint32_t)i;
    } else {
      // finalize in slot order (volumetric_nn8_reconstruction.cl:212-270); a
      // slot not replaced keeps its list entry
      float w[8], v[8], ws = 0.0f, dot = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int32_t id = s.id[j];
        if (!kExact) s.d[j] = id < 0 ? FLT_MAX : sqrtf(s.d[j]);
        v[j] = id >= 0 ? __ldg(&g.parts[id].w) : (kMerge ? list_v[8 * i + j] : 0.0f);
        w[j] = weight3d(s.d[j]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ws = ws + w[j];
#pragma unroll
      for (int j = 0; j < 8; ++j) dot = __fmaf_rn(w[j], v[j], dot);
      out[i] = (ws != 0.0f && dot != 0.0f) ? dot / ws : 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int32_t id = s.id[j];
        s.id[j] =
            id == -1 ? -1 : (id < 0 ? (int32_t)((uint32_t)id & 0x7fffffffu) : (int32_t)s2u[id]);
      }
      // rows of 8: two 16-byte stores each
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 dd = make_float4(s.d[4 * h], s.d[4 * h + 1], s.d[4 * h + 2], s.d[4 * h + 3]);
        const int4 ii = make_int4(s.id[4 * h], s.id[4 * h + 1], s.id[4 * h + 2], s.id[4 * h + 3]);
        reinterpret_cast<float4*>(list_d)[2 * i + h] = dd;
        reinterpret_cast<float4*>(list_v)[2 * i + h] =
            make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
        reinterpret_cast<int4*>(list_id)[2 * i + h] = ii;
        // (the caller's arrays need not be aligned)
        if (idx8) {
          idx8[8 * i + 4 * h] = ii.x;
          idx8[8 * i + 4 * h + 1] = ii.y;
          idx8[8 * i + 4 * h + 2] = ii.z;
          idx8[8 * i + 4 * h + 3] = ii.w;
        }
        if (d8) {
          d8[8 * i + 4 * h] = dd.x;
          d8[8 * i + 4 * h + 1] = dd.y;
          d8[8 * i + 4 * h + 2] = dd.z;
          d8[8 * i + 4 * h + 3] = dd.w;
        }
      }
    }
  }
  // warp-aggregated traffic counters
  unsigned long long c = st.cells, k = st.cands;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    c += __shfl_xor_sync(0xffffffffu, c, off);
    k += __shfl_xor_sync(0xffffffffu, k, off);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&stats[3], c);
    atomicAdd(&stats[4], k);
  }
}

// ---------------------------------------------------------------------------
// Warp-cooperative form of the same walk: one warp per query.
//
// Lanes 0-7 hold the 8 (distance, value, index) slots. The spiral is taken 32
// cells at a time (lane L: cell it0 + L); the candidates of the cells that the
// search radius reaches come in walk order, up to 32 to a batch (lane k:
// candidate k): whole small cells together, large cells 32 at a time or, past
// their first 64 candidates, through their sub-box codes (ilc_raylist.cuh). A
// ballot finds the first candidate that passes the test at the current radius;
// it replaces the first maximal slot (the reference's rule, with its strict <
// on rounded distances), the radius shrinks, and the next ballot follows. The
// early break is applied at every cell in order with the radius of that
// moment: a ballot of the cells whose centre is beyond R + cell radius gives
// the first cell the walk stops at. The slots go through the same insertions
// as in the one-thread walk, and the result is the same bit for bit. The
// maximum slot is found with __reduce_max_sync over the distances' bit
// patterns (non-negative floats order as unsigned integers) and the first slot
// holding it with a ballot. 1,000 queries of 20,000 particles: 322 -> 37 us;
// 65,537 of 1,000,003: 1,833 -> 168 us (one lane per query before; 184 us with
// a square root and a copy of the value per insertion).
// ---------------------------------------------------------------------------
// This lane's slot (lanes 0-7): squared distance, or (exact) distance, and
// candidate. M: the slot maximum, mi its first slot, T: squared distances above
// it cannot enter, rr: the early-break threshold.
struct WarpSlots {
  float d;
  int32_t id;
  float M, T, rr;
  int mi;
};

__device__ __forceinline__ void warp_rescan(WarpSlots& s, int lane, bool exact) {
  const unsigned bits = __reduce_max_sync(kAll, lane < 8 ? __float_as_uint(s.d) : 0u);
  s.M = __uint_as_float(bits);
  s.mi = __ffs(__ballot_sync(kAll, lane < 8 && __float_as_uint(s.d) == bits)) - 1;
  s.T = exact ? __fmul_ru(s.M, s.M) : s.M;
}

__device__ __forceinline__ void warp_break_radius(WarpSlots& s, float crad, bool exact) {
  const float b = (exact ? s.M : fminf(sqrtf(s.M), FLT_MAX)) + crad;
  s.rr = b * b;
}

struct QueryWarpMem {
  int owner[32];
  int hits[kHits];
};

// exact: on rounded distances, as the reference; otherwise on squared ones (as
// in a list replay), returning false where two are too close for that.
__device__ __forceinline__ bool nn8_walk_warp(const GridView& g, const char4* __restrict__ spiral,
                                              QueryWarpMem& W, float qx, float qy, float qz,
                                              WarpSlots& s, int lane, bool exact,
                                              WalkStats& st) {
  int cx, cy, cz, sx, sy, sz;
  locate_axis(qx, g.min0, g.cs0, g.half0, cx, sx);
  locate_axis(qy, g.min1, g.cs1, g.half1, cy, sy);
  locate_axis(qz, g.min2, g.cs2, g.half2, cz, sz);
  const char4* order = spiral + (sx + 2 * sy + 4 * sz) * 125;
  const float crad = g.cell_radius, inf = __int_as_float(0x7f800000);
  bool close = false;
  warp_break_radius(s, crad, exact);
#pragma unroll 1
  for (int it0 = 0; it0 < 125; it0 += 32) {
    // this lane's cell of the chunk
    const bool valid_cell = it0 + lane < 125;
    const char4 o = order[valid_cell ? it0 + lane : 124];
    const int ix = cx + o.x, iy = cy + o.y, iz = cz + o.z;
    const float ccx = (g.min0 + (float)ix * g.cs0) + g.half0;
    const float ccy = (g.min1 + (float)iy * g.cs1) + g.half1;
    const float ccz = (g.min2 + (float)iz * g.cs2) + g.half2;
    const float ex = ccx - qx, ey = ccy - qy, ez = ccz - qz;
    const float cd = (ex * ex + ey * ey) + ez * ez;
    const bool ing = valid_cell && (unsigned)ix < (unsigned)g.n0 &&
                     (unsigned)iy < (unsigned)g.n1 && (unsigned)iz < (unsigned)g.n2;
    int b0 = 0, nc = 0;
    if (ing) {
      const uint32_t key =
          (uint32_t)ix + (uint32_t)g.n0 * ((uint32_t)iy + (uint32_t)g.n1 * (uint32_t)iz);
      const int2 be = __ldg(&g.cells[key]);
      b0 = be.x;
      nc = max(be.y - be.x, 0);
    }
    // squared distance to the cell's box; its candidates are all beyond it
    const float gx = fmaxf(fabsf(ex) - g.half0 - g.margin, 0.0f);
    const float gy = fmaxf(fabsf(ey) - g.half1 - g.margin, 0.0f);
    const float gz = fmaxf(fabsf(ez) - g.half2 - g.margin, 0.0f);
    const float box2 = ((gx * gx + gy * gy) + gz * gz) * 0.99999f;
    int cur = 0;          // first cell whose break test is still due
    int brk = -1;         // cell the walk stops at (-1: none in this chunk)
    int q = 0, qe = 0;    // candidates to load next, then
    int cp = 0, ce = 0;   // candidates to read through their codes, of
    int cell = 0;         // this lane's cell
    int hb = 0, he = 0;   // buffered hits
    uint4 nx;
#pragma unroll 1
    for (;;) {
      bool valid;
      int p, k;
      if (q < qe) {
        p = q + lane;
        valid = p < qe;
        if (!valid) p = q;
        k = cell;
        q += 32;
      } else if (cp < ce || hb < he) {
        const float e = (exact ? s.M : sqrtf(s.M)) * 1.00001f + g.margin;
        uint32_t l0, h0, l1, h1, l2, h2;
        const float mx = __shfl_sync(kAll, ccx, cell) - g.half0,
                    my = __shfl_sync(kAll, ccy, cell) - g.half1,
                    mz = __shfl_sync(kAll, ccz, cell) - g.half2;
        if (!(code_range(qx - e - mx, qx + e - mx, g.inv_w0, l0, h0) &
              code_range(qy - e - my, qy + e - my, g.inv_w1, l1, h1) &
              code_range(qz - e - mz, qz + e - mz, g.inv_w2, l2, h2))) {
          cp = ce;
          hb = he = 0;
          continue;
        }
        const uint32_t lo = (l0 | (l1 << 5) | (l2 << 10)) * 0x10001u;
        const uint32_t hi = (h0 | (h1 << 5) | (h2 << 10)) * 0x10001u | kGuard;
#pragma unroll 1
        while (cp < ce && he - hb < 32) {
          const int pw = cp & ~7, q0 = pw + 8 * lane;
          unsigned hit = code_hits(nx, lo, hi, q0, cp, ce);
          const int incl = warp_inclusive(__popc(hit), lane);
          const int tot = __shfl_sync(kAll, incl, 31);
          if (tot > kHits - 32) {  // most of them: loaded without the codes
            if (hb < he) break;    // (after the buffered ones)
            q = cp;
            qe = min(pw + 256, ce);
          } else if (tot) {
            if (he + tot > kHits) {  // the pending hits (fewer than 32) to the front
              const int h = W.hits[min(hb + lane, kHits - 1)];
              __syncwarp();
              W.hits[lane] = h;
              he -= hb;
              hb = 0;
              __syncwarp();
            }
            int pos = he + incl - __popc(hit);
            while (hit) {
              W.hits[pos++] = q0 + __ffs(hit) - 1;
              hit &= hit - 1;
            }
            he += tot;
          }
          cp = min(pw + 256, ce);
          if (cp < ce) nx = load_codes(g, cp, lane);
          if (q < qe) break;
        }
        if (hb == he) continue;
        __syncwarp();
        k = cell;
        valid = hb + lane < he;
        p = W.hits[valid ? hb + lane : hb];
        hb = min(hb + 32, he);
        if (hb == he) hb = he = 0;
        __syncwarp();
      } else {
        // the cells up to the first due break with candidates within reach
        const unsigned bm = __ballot_sync(kAll, valid_cell && lane >= cur && cd > s.rr);
        const int kb = bm ? __ffs(bm) - 1 : 32;
        const bool el = nc > 0 && lane >= cur && lane < kb && box2 <= s.T;
        const unsigned em = __ballot_sync(kAll, el);
        if (!em) {
          if (bm) brk = kb;
          break;
        }
        const int incl = warp_inclusive(el ? min(nc, 33) : 0, lane);
        const bool in = el && incl <= 32;
        const unsigned inm = __ballot_sync(kAll, in);
        cell = __ffs(em) - 1;
        if (!((inm >> cell) & 1u)) {  // a cell with more than 32 candidates
          q = __shfl_sync(kAll, b0, cell);
          ce = q + __shfl_sync(kAll, nc, cell);
          qe = cp = ce - q > kCodedMin ? q + kDirect : ce;
          if (cp < ce) nx = load_codes(g, cp, lane);
          cur = cell + 1;
          continue;
        }
        // the next whole cells that together have at most 32 candidates
        const int tot = __shfl_sync(kAll, incl, 31 - __clz(inm));
        const int excl = incl - nc;
        if (in) W.owner[__popc(inm & ((1u << lane) - 1u))] = lane;
        const unsigned starts = __reduce_or_sync(kAll, in ? 1u << excl : 0u);
        __syncwarp();
        const int src = W.owner[__popc(starts & (0xffffffffu >> (31 - lane))) - 1];
        p = __shfl_sync(kAll, b0 - excl, src) + lane;
        valid = lane < tot;
        if (!valid) p = 0;
        k = src;
        __syncwarp();
      }
      const float4 P = __ldg(&g.parts[p]);
      const float fx = P.x - qx, fy = P.y - qy, fz = P.z - qz;
      const float d2 = (fx * fx + fy * fy) + fz * fz;
      int last = -1;
      if (s.M == inf) {
        // (not exact) empty slots: the first 8 candidates fill them, no break
        // being possible before
        const unsigned fm = __ballot_sync(kAll, valid && d2 < inf);
        if ((fm & 0xffu) == 0xffu && __ballot_sync(kAll, lane < 8 && s.id != -1) == 0u) {
          if (lane < 8) {
            s.d = d2;
            s.id = p;
          }
          warp_rescan(s, lane, exact);
          cur = max(cur, __shfl_sync(kAll, k, 7) + 1);
          last = 7;
          warp_break_radius(s, crad, exact);
        }
      }
      bool stale = false;  // rr is behind M
      for (;;) {
        const unsigned hm = __ballot_sync(kAll, valid && lane > last && d2 <= s.T);
        if (!hm) break;
        const int i = __ffs(hm) - 1;
        last = i;
        const int ck = __shfl_sync(kAll, k, i);
        if (ck >= cur) {  // break tests of the cells up to this candidate's cell
          if (stale) warp_break_radius(s, crad, exact);
          stale = false;
          const unsigned due = __ballot_sync(kAll, valid_cell && lane >= cur && lane <= ck &&
                                                       cd > s.rr);
          if (due) {
            brk = __ffs(due) - 1;
            break;
          }
          cur = ck + 1;
        }
        float d = __shfl_sync(kAll, d2, i);
        if (exact) d = sqrtf(d);
        if (d < s.M) {
          const int pk = __shfl_sync(kAll, p, i);
          if (lane == s.mi) {
            s.d = d;
            s.id = pk;
          }
          const float before = s.M;
          warp_rescan(s, lane, exact);
          close = close || (before < inf && s.M >= before * 0.99999952f);
          stale = true;
        }
      }
      if (stale) warp_break_radius(s, crad, exact);
      if (brk >= 0) break;
      if (q >= qe && cp >= ce && hb >= he) {
        // the batch's cells are done: the break tests due at them
        const int lastk = __shfl_sync(kAll, k, 31);
        const unsigned due =
            __ballot_sync(kAll, valid_cell && lane >= cur && lane <= lastk && cd > s.rr);
        if (due) {
          brk = __ffs(due) - 1;
          break;
        }
        cur = max(cur, lastk + 1);
      }
    }
    // statistics: the in-grid cells before the break and their candidates
    const int seen = brk < 0 ? 32 : brk;
    st.cells += __popc(__ballot_sync(kAll, ing && lane < seen));
    const int incl = warp_inclusive(lane < seen ? nc : 0, lane);
    st.cands += (uint32_t)__shfl_sync(kAll, incl, 31);
    if (brk >= 0) break;
  }
  return exact || !close;
}

// todo: the queries to take (nullptr: all n), n_todo of them (device counter).
__global__ void __launch_bounds__(256)
nn8_query_warp_kernel(const __grid_constant__ GridView g, const char4* __restrict__ spiral_g,
                      const float4* __restrict__ pts, const uint32_t* __restrict__ todo,
                      const uint32_t* __restrict__ n_todo, uint64_t n, int merge,
                      float* __restrict__ list_d, float* __restrict__ list_v,
                      int32_t* __restrict__ list_id, float* __restrict__ out,
                      int32_t* __restrict__ idx8, float* __restrict__ d8,
                      const uint32_t* __restrict__ s2u, unsigned long long* __restrict__ stats) {
  __shared__ char4 spiral[1000];
  __shared__ QueryWarpMem mem[8];
  if (todo) n = *n_todo;
  if (blockIdx.x * (uint64_t)(blockDim.x >> 5) >= n) return;
  load_spiral(spiral, spiral_g);
  const int lane = threadIdx.x & 31;
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  WalkStats st;
  unsigned long long cells = 0, cands = 0;
  for (uint64_t turn = blockIdx.x * (uint64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); turn < n;
       turn += warps) {
    const uint64_t i = todo ? todo[turn] : turn;
    const float4 q = pts[i];
    WarpSlots s;
    bool exact = merge != 0;
    for (;;) {
      s.d = exact ? FLT_MAX : __int_as_float(0x7f800000);
      s.id = -1;
      if (merge && lane < 8) {
        s.d = list_d[8 * i + lane];
        const int32_t o = list_id[8 * i + lane];
        s.id = o >= 0 ? (int32_t)(0x80000000u | (uint32_t)o) : -1;
      }
      warp_rescan(s, lane, exact);
      st.cells = st.cands = 0;
      if (nn8_walk_warp(g, spiral, mem[threadIdx.x >> 5], q.x, q.y, q.z, s, lane, exact, st))
        break;
      exact = true;
    }
    cells += st.cells;
    cands += st.cands;
    if (!exact) s.d = s.id < 0 ? FLT_MAX : sqrtf(s.d);
    // a slot not replaced keeps its list entry
    float v = 0.0f;
    if (lane < 8 && s.id >= 0) v = __ldg(&g.parts[s.id].w);
    else if (lane < 8 && merge) v = list_v[8 * i + lane];
    // finalize in slot order (volumetric_nn8_reconstruction.cl:212-270)
    const float w = weight3d(s.d);
    float ws = 0.0f, dot = 0.0f;
#pragma unroll
    for (int t = 0; t < 8; ++t) ws = ws + __shfl_sync(kAll, w, t);
#pragma unroll
    for (int t = 0; t < 8; ++t)
      dot = __fmaf_rn(__shfl_sync(kAll, w, t), __shfl_sync(kAll, v, t), dot);
    if (lane == 0) out[i] = (ws != 0.0f && dot != 0.0f) ? dot / ws : 0.0f;
    if (lane < 8) {
      const int32_t id = s.id;
      const int32_t orig =
          id == -1 ? -1 : (id < 0 ? (int32_t)((uint32_t)id & 0x7fffffffu) : (int32_t)s2u[id]);
      list_d[8 * i + lane] = s.d;
      list_v[8 * i + lane] = v;
      list_id[8 * i + lane] = orig;
      if (idx8) idx8[8 * i + lane] = orig;
      if (d8) d8[8 * i + lane] = s.d;
    }
  }
  if (lane == 0) {
    atomicAdd(&stats[3], cells);
    atomicAdd(&stats[4], cands);
  }
}

}  // namespace

GridView make_grid_view(const Context& c);

// The queries ordered by bin (a counting sort; the order within a bin is the
// atomics', which no result depends on). `at`: words of query_sort in front.
cudaError_t query_order(Context& c, const GridView& g, const float4* pts, uint64_t n, size_t at,
                        const uint32_t** order) {
  cudaError_t e;
  QueryBins b{g.n0, g.n1, g.n2, 0};
  while (((8 * c.gp.total - 1) >> b.shift) >= (1ull << kBinBits)) ++b.shift;
  const uint64_t bins = ((8 * c.gp.total - 1) >> b.shift) + 1;
  // counts (then first positions), scan scratch, places, order
  const size_t words = (bins + 3) / 4 * 4,
               off_place = words + (scan_scratch_words(bins) + 3) / 4 * 4;
  if ((e = c.query_sort.ensure((at + off_place + 3 * n) * 4))) return e;
  uint32_t* count = c.query_sort.as<uint32_t>() + at;
  uint2* place = reinterpret_cast<uint2*>(count + off_place);
  uint32_t* ord = reinterpret_cast<uint32_t*>(place + n);
  if ((e = cudaMemsetAsync(count, 0, off_place * 4, c.stream))) return e;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  query_count_kernel<<<blocks, 256, 0, c.stream>>>(g, b, pts, n, count, place);
  c.launches += 2;
  if ((e = exclusive_scan_long(c, count, bins, count + words))) return e;
  query_order_kernel<<<blocks, 256, 0, c.stream>>>(count, place, n, ord);
  *order = ord;
  return cudaGetLastError();
}

// Queries from which on ILC_QUERY_THREAD walks one query per lane, and from
// which on it orders them first. Fewer leave SMs idle that way, and the slowest
// lane's chain of loads (150-250 us among clustered particles) is the time: warp
// and ordered lane walks take 34 / 175 us for 1,000 queries, 184 / 165-247 us for
// 65,537, 331 / 180-280 us for 131,072 and 2,360 / 510-860 us for 1,048,576
// (20,000 to 4,194,304 particles of a halo, whose grids have 3-30 % of their cells
// occupied).
constexpr uint64_t kThreadMin = 81920;
// In an even grid (Context::even: particles in four of five cells or more, at most
// a thousandth of them beyond the 48th of their cell) no lane's walk is long and
// order gains little: from 24,576 queries on the lanes are ahead of the warps, and
// up to 393,216 the sort costs more than it saves. A few queries whose distances are
// too close for squared ones would cost the warp kernel's latency (65,537 random
// queries in 116 us, 81,000 in 135), so such grids are walked on rounded distances.
// Whole calls in us, 100,000 uniform particles, random queries (in the order of their
// cells): 16,384 by warps 68 (67), lanes 94 (80); 24,576: 84 (85), 88 (75); 36,000: 102
// (99), 88 (78); 65,537: 165 (158), ordered lanes 135 (131), lanes 101 (86); 81,000:
// 198 (192), 147 (142), 109 (92); 200,000: 439 (418), 189 (183), 168 (130); 394,000
// ordered 235 (228), 393,000 unordered 246 (196).
constexpr uint64_t kEvenMin = 24576, kEvenOrder = 393216;

cudaError_t nn8_query_launch(Context& c, const float4* pts, uint64_t n, bool merge, float* out,
                             int32_t* idx8, float* d8) {
  cudaError_t e;
  if ((e = c.list_d.ensure(n * 32)) || (e = c.list_v.ensure(n * 32)) ||
      (e = c.list_id.ensure(n * 32)) || (e = c.flags.ensure(kFlagsBytes)))
    return e;
  if ((e = cudaMemsetAsync(c.flags.p, 0, kFlagsBytes, c.stream))) return e;
  c.list_n = n;
  const GridView g = make_grid_view(c);
  unsigned long long* stats =
      reinterpret_cast<unsigned long long*>(c.flags.as<char>() + 64);
  const uint32_t *hard = nullptr, *n_hard = nullptr;
  const bool even = c.even;
  if (c.query_engine == ILC_QUERY_THREAD && n >= (even ? kEvenMin : kThreadMin) &&
      n <= 0xffffffffull) {
    // the list of the queries left to the warp kernel, then the sort's arrays
    const uint32_t* order = nullptr;
    const size_t list = (n + 3) / 4 * 4;
    if ((e = even && n < kEvenOrder ? c.query_sort.ensure(list * 4)
                                    : query_order(c, g, pts, n, list, &order)))
      return e;
    uint32_t* left = c.query_sort.as<uint32_t>();
    uint32_t* n_left = c.flags.as<uint32_t>() + kLeftWord;
    ++c.launches;
    const auto kernel = merge ? nn8_query_kernel<true, true> : even ? nn8_query_kernel<false, true> : nn8_query_kernel<false, false>;
    kernel<<<(unsigned)((n + 255) / 256), 256, 0, c.stream>>>(
        g, c.spiral.as<char4>(), pts, order, n, left, n_left, c.list_d.as<float>(),
        c.list_v.as<float>(), c.list_id.as<int32_t>(), out, idx8, d8, c.s2u.as<uint32_t>(),
        stats);
    if ((e = cudaGetLastError())) return e;
    n_hard = n_left;
    hard = left;
  }
  // one warp per query; persistent blocks of 8 warps, as many as are resident
  int sms = 0, per_sm = 0;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device)) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, nn8_query_warp_kernel, 256, 0)))
    return e;
  const uint64_t cap = (uint64_t)sms * (uint64_t)(per_sm > 0 ? per_sm : 1);
  const unsigned wb = (unsigned)std::min<uint64_t>((n + 7) / 8, cap);
  ++c.launches;
  nn8_query_warp_kernel<<<wb, 256, 0, c.stream>>>(
      g, c.spiral.as<char4>(), pts, hard, n_hard, n, merge ? 1 : 0, c.list_d.as<float>(),
      c.list_v.as<float>(), c.list_id.as<int32_t>(), out, idx8, d8, c.s2u.as<uint32_t>(), stats);
  return cudaGetLastError();
}

}  // namespace ilc
