// ilc_raylist.cuh -- nn8 reconstruction along rays from candidate lists that a
// warp builds once per ray segment and that its steps replay.
//
// A warp carries 8 rays, 4 lanes each, one lane per integrand point of an RKF
// step. A step moves a fraction of a kpc among particles tens of kpc apart, so
// consecutive steps search the same cells and insert nearly the same
// candidates. What a search needs is only the candidates that can enter the 8
// slots at all; for all points of a segment of the ray (within one cell and
// subcell, hence one spiral order) those are found once:
//
//   Let c be the segment's midpoint, b its half length, R_i(x) the search
//   radius (8th smallest distance) after the first i candidates of the walk
//   at x. Distances and R_i move by at most |x - c| <= b, so a candidate with
//   d(c) >= R_i(c) + 2 b cannot be inserted for any point of the segment.
//
// The build runs the walk at c with that threshold, the 32 lanes taking the
// cells of the spiral and the candidates 32 at a time, and appends the
// survivors in walk order. A lane then replays its point's walk over the list
// alone, with the exact distances, comparisons, replacement rule and finalize
// of the one-thread walk: the candidates left out would not have been
// inserted, so the slots, and every result, are that walk's bit for bit.
//
// The early break (volumetric_nn8_reconstruction.cl:157-171) is kept exactly:
// cells that no point of the segment can break at are settled in the build; of
// the others, up to the first at which every point breaks, the list keeps the
// centre, the visited-cell and candidate counts in front of it and where the
// candidates up to the next one end in the list, and each lane tests its own
// break at each of them, in turn with their candidates.
// A list that overflows is built again for the step's points alone, then for
// one point alone, and at last that point is walked by one thread. All bounds
// carry slack for the rounding of positions (`del`) and of distances (1e-5
// relative, against rounding errors below 1e-6).
//
// Why this split. Walking every step from scratch, one ray per thread, issued
// 770 warp instructions per step with 10 of 32 lanes active (band map of
// 4,194,304 cells, 1 Mpc from the core), and a warp whose rays cross a dense
// cell spent 100-600 us per step scanning it 16 candidates at a time in one
// lane. Here 32 lanes make a search for several steps, and a cell of 20,000
// candidates is scanned 256 at a time. Counted on a B200 over six renders,
// before list lengths followed their cost: one search per 6-19 steps, 14-28
// candidates and 6-10 break cells per list, 22-25 of 32 lanes replaying in
// sparse cells but 4-8 where core rays have a warp to themselves. Times there,
// before -> after: band map of the outer 1.5 Mpc slab of 4,194,304 cells,
// 256^2: 600 -> 197 ms; projection of 262,144 cells, 256^2, 3 Mpc: 1,450 ->
// 292 ms; 101 x 75 tilted band map through the core of 1 M cells: 1,570 ->
// 34 ms; 2048 fixed steps, 200^2: 327 -> 128 ms; 128-bin spectra of three
// cameras: 942 -> 33 ms; adjoint of a 64^2 band map: 1,413 -> 85 ms. Bound by
// instruction issue (44 % of the slots; small outer-slab band map), dependent
// arithmetic with 4 warps per scheduler (stalls of 2.3 cycles per issue) and
// instruction fetch (2.0); the grid stays in L2 (DRAM 2 MB read per launch).
// Images of very many rays gain less, since there the walks from scratch filled
// the chip too: 1024^2 band map of 4,194,304 cells, 6 Mpc: 12.16 -> 10.55 s. Steps
// that are long against a cell use a list once or twice, and lose: launches of many
// rays walk those (ilc_walk4.cuh).
#pragma once

#include "ilc_device.cuh"

namespace ilc {

constexpr int kRays = 8;             // rays of a warp
constexpr int kUnc = 20;             // cells a list's points may break at
constexpr int kCap = 48;             // candidates of a list in shared memory
constexpr int kOver = 207;           // and further ones in global memory (dense cores)
constexpr int kCapAll = kCap + kOver;  // 255: positions fit a byte
constexpr int kHits = 96;            // build: buffered hits of the sub-box codes
constexpr int kListThreads = 128;    // threads of a block: 4 warps, 32 rays
constexpr int kListWarps = kListThreads / 32;
constexpr unsigned kAll = 0xffffffffu;

// Per ray: the z range the list holds for, its candidates and break cells, and
// how far the next list reaches.
struct RayMeta {
  float za, zb, ext;
  int n, nu, all;   // candidates before the first break cell; break cells; candidates
};

struct WarpLists {
  // odd row lengths: the 8 rays' rows start at different banks
  float4 ent[kRays][kCap + 1];   // x, y, z, value (or sorted index bits)
  float4 unc[kRays][kUnc + 1];   // cell centre; bits 0-7: in-grid cells before, 8-15: end of
                                 // its candidates in ent
  uint32_t unp[kRays][kUnc + 1]; // candidates of the cells before
  RayMeta meta[kRays];
  int owner[32];                 // build: cell (lane) of each batch cell
  int hits[kHits];               // build: candidates whose sub-box is within reach
  unsigned char ek[kCapAll + 1]; // build: spiral position of each candidate's cell
  float4* over;                  // the 8 rays' kOver further candidates
};

__device__ __forceinline__ float4 list_entry(const WarpLists& W, int r, int t) {
  return t < kCap ? W.ent[r][t] : W.over[r * kOver + (t - kCap)];
}

__device__ __forceinline__ void ray_reset(RayMeta& m, float ext) {
  m.za = 1.0f;
  m.zb = 0.0f;
  m.ext = ext;
}

// One point walked by one thread (the path of last resort): distances and
// values (or indices) of its slots to out[0..7].
template <bool kIdx>
__device__ __noinline__ void point_walk(const GridView& g, const char4* spiral, float x, float y,
                                        float z, float4* out, WalkStats& st) {
  Slots<true> s;
  s.init();
  nn8_walk<true>(g, spiral, x, y, z, s, st);
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int id = s.id[t];
    const float v = id < 0 ? 0.0f : (g.vals ? __ldg(&g.vals[id]) : s.v[t]);
    out[t] = make_float4(s.d[t], kIdx ? __int_as_float(id) : v, 0.0f, 0.0f);
  }
}

// Cell index and subcell half (0/1) of a point along one axis
// (volumetric_nn8_reconstruction.cl:129-155, one component).
__device__ __forceinline__ void locate_axis(float q, float mn, float cs, float half, int& c,
                                            int& sh) {
  c = clamp_cell(to_int_sat(floorf((q - mn) / cs)));
  const float m = mn + (float)c * cs;
  const int si = to_int_sat(floorf((q - m) / half));
  sh = min(max(si, 0), 1);
}

// Rounding of the positions o + z l of a ray up to |z| = zm, and of the cell and
// subcell found from them: at most a dozen roundings of 2^-24 of the largest term
// (16 here), in every sum of |o_i| and |zm l_i|.
__device__ __forceinline__ float ray_rounding(float ox, float oy, float oz, float zm,
                                              float len_l) {
  return ((fabsf(ox) + fabsf(oy)) + (fabsf(oz) + zm * len_l)) * 9.5367432e-7f;
}

// Largest z at which the ray is surely still in [lo, lo + half] along one axis.
__device__ __forceinline__ float axis_exit(float o, float l, float lo, float half, float margin) {
  if (l > 0.0f) return (lo + half - margin - o) / l;
  if (l < 0.0f) return (lo + margin - o) / l;
  return FLT_MAX;
}

// Build state at the segment's midpoint: lanes 0-7 hold the 8 smallest squared
// distances so far, R2 the largest of them, T2 the squared threshold.
struct BuildState {
  float s8, R2, R, T, T2, tb;
  int n;
  bool seeded;
};

__device__ __forceinline__ void build_radius(BuildState& b, int lane) {
  b.R2 = __uint_as_float(__reduce_max_sync(kAll, lane < 8 ? __float_as_uint(b.s8) : 0u));
  asm("sqrt.approx.f32 %0, %1;" : "=f"(b.R) : "f"(b.R2));  // (within the slack of T)
  b.T = (b.R + b.tb) * 1.00001f;
  b.T2 = b.T * b.T;
}

// Takes up to 32 candidates in walk order (lane = candidate, valid lanes
// first): updates the radius at every candidate that enters the 8 smallest
// and appends the candidates below the threshold of their turn.
template <bool kIdx>
__device__ __forceinline__ void build_take(const GridView& g, BuildState& b, WarpLists& W, int r, int lane,
                                           bool valid, const float4& P, float d2, int p, int k) {
  const unsigned lt = (1u << lane) - 1u;
  bool keep = false;
  int last = -1;
  if (!b.seeded) {
    if ((__ballot_sync(kAll, valid && d2 < b.R2) & 0xffu) == 0xffu) {
      if (lane < 8) {
        b.s8 = d2;
        keep = true;
      }
      last = 7;
      build_radius(b, lane);
    }
    b.seeded = true;
  }
  for (;;) {
    const unsigned rm = __ballot_sync(kAll, valid && lane > last && d2 < b.R2);
    const int i = rm ? __ffs(rm) - 1 : 31;
    if (valid && lane > last && lane <= i && d2 < b.T2) keep = true;
    if (!rm) break;
    const float dn = __shfl_sync(kAll, d2, i);
    const int ml = __ffs(__ballot_sync(kAll, lane < 8 && b.s8 == b.R2)) - 1;
    if (lane == ml) b.s8 = dn;
    build_radius(b, lane);
    last = i;
  }
  const unsigned km = __ballot_sync(kAll, keep);
  if (keep) {
    const int pos = b.n + __popc(km & lt);
    if (pos < kCapAll) {
      const float v = kIdx ? __int_as_float(p) : (g.vals ? __ldg(&g.vals[p]) : P.w);
      const float4 e = make_float4(P.x, P.y, P.z, v);
      if (pos < kCap) W.ent[r][pos] = e;
      else W.over[r * kOver + (pos - kCap)] = e;
      W.ek[pos] = (unsigned char)k;
    }
  }
  b.n += __popc(km);
}

__device__ __forceinline__ int warp_inclusive(int v, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int t = __shfl_up_sync(kAll, v, off);
    if (lane >= off) v += t;
  }
  return v;
}

// Cells with more than kCodedMin candidates: the first kDirect are loaded (they
// bring the radius down), the rest are read through their 2-byte sub-box
// codes, 256 at a time, and only those whose sub-box meets the cube of the
// threshold around the midpoint are loaded: a candidate outside it is farther
// away than the threshold (which only shrinks).
constexpr int kDirect = 64, kCodedMin = 160;
constexpr uint32_t kGuard = 0x42104210u;  // guard bits 4, 9, 14 of both codes

// 4-bit field range [lo, hi] of [a, b] along one axis; false: none.
__device__ __forceinline__ bool code_range(float a, float b, float inv_w, uint32_t& lo,
                                           uint32_t& hi) {
  const float tl = a * inv_w, th = b * inv_w;
  lo = tl > 0.0f ? (uint32_t)fminf(tl, 15.0f) : 0u;
  hi = th < 15.0f ? (uint32_t)fmaxf(th, 0.0f) : 15u;
  return th >= 0.0f && tl < 16.0f;
}

__device__ __forceinline__ uint4 load_codes(const GridView& g, int p, int lane) {
  return __ldg(reinterpret_cast<const uint4*>(g.codes) + (p >> 3) + lane);
}

// Hits among the 256 codes at pw (lane: 8 of them in w), of those in [p0, p1).
__device__ __forceinline__ unsigned code_hits(const uint4& w, uint32_t lo, uint32_t hi, int q0,
                                              int p0, int p1) {
  const uint32_t words[4] = {w.x, w.y, w.z, w.w};
  unsigned hit = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    // a guard bit survives both subtractions where lo <= field <= hi
    const uint32_t m = (((words[j] | kGuard) - lo) & (hi - words[j]) & kGuard) ^ kGuard;
    hit |= ((m & 0xffffu) == 0u ? 1u : 0u) << (2 * j);
    hit |= ((m >> 16) == 0u ? 1u : 0u) << (2 * j + 1);
  }
  if (q0 < p0) hit &= p0 - q0 < 8 ? 0xffu << (p0 - q0) : 0u;
  if (q0 + 8 > p1) hit &= p1 > q0 ? 0xffu >> (8 - (p1 - q0)) : 0u;
  return hit;
}

// Cell `it` of the spiral around (cx, cy, cz).
struct SpiralCell {
  float ccx, ccy, ccz, D;  // centre, distance from the segment's midpoint
  int b0, nc;              // first candidate, candidates (0 outside the grid)
  bool valid, ing;
};

__device__ __forceinline__ SpiralCell spiral_cell(const GridView& g,
                                                  const char4* __restrict__ order, int it, int cx,
                                                  int cy, int cz, float qx, float qy, float qz) {
  SpiralCell s;
  s.valid = it < 125;
  const char4 o = order[s.valid ? it : 124];
  const int ix = cx + o.x, iy = cy + o.y, iz = cz + o.z;
  s.ccx = (g.min0 + (float)ix * g.cs0) + g.half0;
  s.ccy = (g.min1 + (float)iy * g.cs1) + g.half1;
  s.ccz = (g.min2 + (float)iz * g.cs2) + g.half2;
  const float ex = s.ccx - qx, ey = s.ccy - qy, ez = s.ccz - qz;
  s.D = sqrtf((ex * ex + ey * ey) + ez * ez);
  s.ing = s.valid && (unsigned)ix < (unsigned)g.n0 && (unsigned)iy < (unsigned)g.n1 &&
          (unsigned)iz < (unsigned)g.n2;
  s.b0 = 0;
  s.nc = 0;
  if (s.ing) {
    // in 32 bits (the grid build rejects 2^32 cells or more)
    const uint32_t key =
        (uint32_t)ix + (uint32_t)g.n0 * ((uint32_t)iy + (uint32_t)g.n1 * (uint32_t)iz);
    const int2 be = __ldg(&g.cells[key]);
    s.b0 = be.x;
    s.nc = max(be.y - be.x, 0);
  }
  return s;
}

// Builds ray r's list for the points at z in [za, zb] of the ray o + z l, all
// located in cell (cx, cy, cz), subcell `sub`. All arguments are warp-uniform.
// Returns the candidates looked at, or -1 when the range has to be narrowed.
template <bool kIdx>
__device__ __forceinline__ int build_list(const GridView& g, const char4* __restrict__ spiral,
                                           WarpLists& W, int r, int lane, float ox, float oy,
                                           float oz, float lx, float ly, float lz, float len_l,
                                           int cx, int cy, int cz, int sub, float za, float zb) {
  const char4* order = spiral + sub * 125;
  const float zc = za + 0.5f * (zb - za);
  const float qx = ox + zc * lx, qy = oy + zc * ly, qz = oz + zc * lz;
  const float del = ray_rounding(ox, oy, oz, fabsf(zb), len_l);
  const float bb = 0.5f * (zb - za) * len_l * 1.00001f + del;
  const float crad = g.cell_radius;
  if (!(bb < 1e15f) || !(crad < 1e15f)) return -1;
  BuildState b;
  b.s8 = __int_as_float(0x7f800000);
  b.R2 = b.R = b.T2 = b.s8;
  b.tb = 2.0f * bb;
  b.n = 0;
  b.seeded = false;
  int tested = 0;
  SpiralCell first;
  int kend = 125;  // cells from here on are not visited
  __syncwarp();
#pragma unroll 1
  for (int it0 = 0; it0 < 125; it0 += 32) {
    const SpiralCell s = spiral_cell(g, order, it0 + lane, cx, cy, cz, qx, qy, qz);
    if (it0 == 0) first = s;
    // squared distance from the midpoint to the cell's box
    const float gx = fmaxf(fabsf(s.ccx - qx) - g.half0 - g.margin, 0.0f);
    const float gy = fmaxf(fabsf(s.ccy - qy) - g.half1 - g.margin, 0.0f);
    const float gz = fmaxf(fabsf(s.ccz - qz) - g.half2 - g.margin, 0.0f);
    const float box2 = ((gx * gx + gy * gy) + gz * gz) * 0.99999f;
    int cur = 0;          // first cell not taken yet
    int q = 0, qe = 0;    // candidates to load next
    int cp = 0, ce = 0;   // candidates to read through their codes next
    int cell = 0;         // their cell's lane
    int hb = 0, he = 0;   // buffered hits
    uint4 nx;             // the codes at cp & ~7
    unsigned brk = 0;
    // one batch of up to 32 candidates in walk order per turn
#pragma unroll 1
    for (;;) {
      bool valid;
      int p, k;
      if (q < qe) {
        p = q + lane;
        valid = p < qe;
        if (!valid) p = q;
        k = it0 + cell;
        q += 32;
      } else if (cp < ce || hb < he) {
        const float e = b.T + g.margin;
        uint32_t l0, h0, l1, h1, l2, h2;
        const float mx = __shfl_sync(kAll, s.ccx, cell) - g.half0,
                    my = __shfl_sync(kAll, s.ccy, cell) - g.half1,
                    mz = __shfl_sync(kAll, s.ccz, cell) - g.half2;
        // (none: no later candidate of the cell is within reach)
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
        k = it0 + cell;
        valid = hb + lane < he;
        p = W.hits[valid ? hb + lane : hb];
        hb = min(hb + 32, he);
        if (hb == he) hb = he = 0;
        __syncwarp();
      } else {
        // cells from the first at which every point surely breaks are not visited
        brk = __ballot_sync(
            kAll, s.valid && lane >= cur && s.D - bb > (b.R + bb + crad) * 1.00001f);
        const int kb = brk ? __ffs(brk) - 1 : 32;
        const bool el = s.nc > 0 && lane >= cur && lane < kb && box2 <= b.T2;
        const unsigned em = __ballot_sync(kAll, el);
        if (!em) break;
        const int incl = warp_inclusive(el ? min(s.nc, 33) : 0, lane);
        const bool in = el && incl <= 32;
        const unsigned bm = __ballot_sync(kAll, in);
        cell = __ffs(em) - 1;
        if (!((bm >> cell) & 1u)) {  // a cell with more than 32 candidates
          q = __shfl_sync(kAll, s.b0, cell);
          ce = q + __shfl_sync(kAll, s.nc, cell);
          tested += ce - q;
          qe = cp = ce - q > kCodedMin ? q + kDirect : ce;
          if (cp < ce) nx = load_codes(g, cp, lane);
          cur = cell + 1;
          continue;
        }
        // the next whole cells that together have at most 32 candidates
        const int lastl = 31 - __clz(bm);
        const int tot = __shfl_sync(kAll, incl, lastl);
        const int excl = incl - s.nc;
        if (in) W.owner[__popc(bm & ((1u << lane) - 1u))] = lane;
        const unsigned starts = __reduce_or_sync(kAll, in ? 1u << excl : 0u);
        __syncwarp();
        const int src = W.owner[__popc(starts & (0xffffffffu >> (31 - lane))) - 1];
        p = __shfl_sync(kAll, s.b0 - excl, src) + lane;
        valid = lane < tot;
        if (!valid) p = 0;
        k = it0 + src;
        tested += tot;
        cur = lastl + 1;
        __syncwarp();
      }
      const float4 P = __ldg(&g.parts[p]);
      const float fx = P.x - qx, fy = P.y - qy, fz = P.z - qz;
      const float d2 = (fx * fx + fy * fy) + fz * fz;
      if (!__any_sync(kAll, valid && d2 < b.T2)) continue;
      build_take<kIdx>(g, b, W, r, lane, valid, P, d2, p, k);
      if (b.n > kCapAll) return -1;
    }
    if (brk) {
      kend = it0 + __ffs(brk) - 1;
      break;
    }
  }
  // the cells points may break at: those before kend (125: the spiral's end)
  // that are not surely visited, and kend, at which every point breaks
  int nu = 0;
  uint32_t cells_run = 0, cands_run = 0;
  const float vis_r = (b.R - bb + crad) * 0.99999f;
#pragma unroll 1
  for (int it0 = 0; it0 <= kend; it0 += 32) {
    const SpiralCell s =
        it0 == 0 ? first : spiral_cell(g, order, it0 + lane, cx, cy, cz, qx, qy, qz);
    const int it = it0 + lane;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned ingm = __ballot_sync(kAll, s.ing);
    const int incl = warp_inclusive(s.nc, lane);
    const bool may = it <= kend && (it == kend || !(s.D + bb <= vis_r));
    const unsigned mm = __ballot_sync(kAll, may);
    const int u = nu + __popc(mm & lt);
    if (may && u < kUnc) {
      const uint32_t before = cells_run + __popc(ingm & lt);
      W.unc[r][u] = make_float4(s.ccx, s.ccy, s.ccz, __uint_as_float(before));
      W.unp[r][u] = cands_run + (uint32_t)(incl - s.nc);
      W.owner[u] = it;
    }
    nu += __popc(mm);
    cells_run += __popc(ingm);
    cands_run += (uint32_t)__shfl_sync(kAll, incl, 31);
  }
  if (nu > kUnc) return -1;
  __syncwarp();
  // candidates before the first of them, and up to each next one
  const int ku = W.owner[0];
  int n = b.n;
  for (int e0 = 0; e0 < b.n; e0 += 32) {
    const bool late = e0 + lane < b.n && (int)W.ek[e0 + lane] >= ku;
    const unsigned lm = __ballot_sync(kAll, late);
    if (lm) {
      n = e0 + __ffs(lm) - 1;
      break;
    }
  }
  if (lane < nu) {
    int end = n;
    if (lane + 1 < nu) {
      const int kn = W.owner[lane + 1];
      while (end < b.n && (int)W.ek[end] < kn) ++end;
    }
    W.unc[r][lane].w = __uint_as_float(__float_as_uint(W.unc[r][lane].w) | ((unsigned)end << 8));
  }
  if (lane == 0) {
    RayMeta& m = W.meta[r];
    m.za = za;
    m.zb = zb;
    m.n = n;
    m.nu = nu;
    m.all = b.n;
  }
  __syncwarp();
  return tested;
}

// A lane's slots after its point's walk: distances and values (indices);
// plain: every squared distance is plain_d2.
struct PointSlots {
  float d[8], v[8];
  bool plain;
};

__device__ __forceinline__ float max8(const float d[8]) {
  return fmaxf(fmaxf(fmaxf(d[0], d[1]), fmaxf(d[2], d[3])),
               fmaxf(fmaxf(d[4], d[5]), fmaxf(d[6], d[7])));
}

// Replays the walk of the point (x, y, z) over ray r's list.
//
// The walk compares rounded distances and replaces the first maximal slot.
// Squared distances order the same way unless two of them lie within a few
// ulp of each other (their roots may then be equal) or are equal, which
// matters only for the slot maximum and the candidate that replaces it: the
// new maximum is then within 2^-21 of the old one. The replay runs on squared
// distances, with 8 square roots at the end; where that happened (or slots may
// stay empty) it runs again on the distances themselves.
template <bool kIdx>
__device__ __forceinline__ void replay_point(const GridView& g, const WarpLists& W, int r,
                                             float x, float y, float z, PointSlots& o,
                                             WalkStats& st) {
  const RayMeta& m = W.meta[r];
  const int n = m.n, nu = m.nu;
  bool exact = n < 8;
  int ix[8], u;
  for (;;) {
    // the first 8 candidates fill the slots
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const float4 P = W.ent[r][t];
      const float fx = P.x - x, fy = P.y - y, fz = P.z - z;
      o.d[t] = (fx * fx + fy * fy) + fz * fz;
      ix[t] = t;
    }
    if (exact) {
#pragma unroll
      for (int t = 0; t < 8; ++t) o.d[t] = t < n ? sqrtf(o.d[t]) : FLT_MAX;
    }
    float M = max8(o.d);                       // the slot maximum
    float T = exact ? __fmul_ru(M, M) : M;     // squared distances above it cannot enter
    bool close = false;
    int t = min(8, n), end = n;
    u = 0;
    for (;;) {
#pragma unroll 1
      for (; t < end; ++t) {
        const float4 P = list_entry(W, r, t);
        const float fx = P.x - x, fy = P.y - y, fz = P.z - z;
        float d = (fx * fx + fy * fy) + fz * fz;
        if (d <= T) {
          if (exact) d = sqrtf(d);
          if (d < M) {
            bool open = true;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const bool eq = o.d[q] == M;
              const bool hit = open && eq;
              open = open && !eq;
              o.d[q] = hit ? d : o.d[q];
              ix[q] = hit ? t : ix[q];
            }
            const float top = max8(o.d);
            close = close || top >= M * 0.99999952f;
            M = top;
            T = exact ? __fmul_ru(M, M) : M;
          }
        }
      }
      // the break, cell by cell (the last one breaks every point)
      const float rb = (exact ? M : sqrtf(M)) + g.cell_radius;
      const float rr = rb * rb;
      bool more = false;
#pragma unroll 1
      for (; u < nu - 1; ++u) {
        const float4 c = W.unc[r][u];
        const float ex = c.x - x, ey = c.y - y, ez = c.z - z;
        if ((ex * ex + ey * ey) + ez * ez > rr) break;
        end = (int)((__float_as_uint(c.w) >> 8) & 0xffu);
        if (t < end) {
          more = true;
          ++u;
          break;
        }
      }
      if (!more) break;
    }
    if (exact || !close) break;
    exact = true;
  }
  st.cells += __float_as_uint(W.unc[r][u].w) & 0xffu;
  st.cands += W.unp[r][u];
  if (m.all <= kCap && n >= 8) {
#pragma unroll
    for (int q = 0; q < 8; ++q) o.v[q] = W.ent[r][ix[q]].w;
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q)
      o.v[q] = o.d[q] < FLT_MAX ? list_entry(W, r, ix[q]).w : (kIdx ? __int_as_float(-1) : 0.0f);
  }
  o.plain = false;
  if (!exact) {
    float lo = fminf(o.d[0], o.d[1]);
#pragma unroll
    for (int q = 2; q < 8; ++q) lo = fminf(lo, o.d[q]);
    o.plain = plain_d2(lo) && plain_d2(max8(o.d));
    if (o.plain) {
#pragma unroll
      for (int q = 0; q < 8; ++q) o.d[q] = sqrt_normal(o.d[q]);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) o.d[q] = sqrtf(o.d[q]);
    }
  }
}

// nn8 slots of the lanes' points: lane 4r + j holds point j of ray r at
// position (x, y, z) = o + zq l, h the ray's step. `active` lanes get their
// slots. The whole warp calls this together.
template <bool kIdx>
__device__ __forceinline__ void eval_points(const GridView& g, const char4* __restrict__ spiral,
                                            WarpLists& W, int lane, bool active, float ox,
                                            float oy, float oz, float lx, float ly, float lz,
                                            float zq, float h, PointSlots& o, WalkStats& st) {
  const float x = ox + zq * lx, y = oy + zq * ly, z = oz + zq * lz;
  const int r = lane >> 2;
  const unsigned mine = 0xfu << (lane & 28);
  bool todo = active;
  for (;;) {
    bool listed = false;
    if (todo) {
      const RayMeta& m = W.meta[r];
      listed = zq >= m.za && zq <= m.zb;
    }
    const unsigned lm = __ballot_sync(kAll, listed) & mine;
    const unsigned todom = __ballot_sync(kAll, todo), rm = todom & mine;
    // rays with a point that their list does not hold for: all of their
    // points get a new list if they share their cell and subcell, otherwise
    // the listed points go first
    const bool part = todo && lm != rm;
    if (__any_sync(kAll, part)) {
      int cx = 0, cy = 0, cz = 0, sub = 0;
      if (part) {
        int sx, sy, sz;
        locate_axis(x, g.min0, g.cs0, g.half0, cx, sx);
        locate_axis(y, g.min1, g.cs1, g.half1, cy, sy);
        locate_axis(z, g.min2, g.cs2, g.half2, cz, sz);
        sub = sx + 2 * sy + 4 * sz;
      }
      const int rl = rm ? __ffs(rm) - 1 : lane;
      const int fx = __shfl_sync(kAll, cx, rl), fy = __shfl_sync(kAll, cy, rl),
                fz = __shfl_sync(kAll, cz, rl), fs = __shfl_sync(kAll, sub, rl);
      const bool same = part && cx == fx && cy == fy && cz == fz && sub == fs;
      const unsigned sm = __ballot_sync(kAll, same) & mine;
      unsigned need = __ballot_sync(kAll, part && (lm == 0u || sm == rm));
#pragma unroll 1
      while (need) {
        const int lead = __ffs(need) - 1, lr = lead >> 2;
        need &= ~(0xfu << (lead & 28));
        const int bx = __shfl_sync(kAll, cx, lead), by = __shfl_sync(kAll, cy, lead),
                  bz = __shfl_sync(kAll, cz, lead), bs = __shfl_sync(kAll, sub, lead);
        const float rox = __shfl_sync(kAll, ox, lead), roy = __shfl_sync(kAll, oy, lead),
                    roz = __shfl_sync(kAll, oz, lead);
        const float rlx = __shfl_sync(kAll, lx, lead), rly = __shfl_sync(kAll, ly, lead),
                    rlz = __shfl_sync(kAll, lz, lead);
        const float zl = __shfl_sync(kAll, zq, lead), hl = __shfl_sync(kAll, h, lead);
        // finite positions only: anything else is walked by one thread
        const bool fin = fabsf(x) < 1e15f && fabsf(y) < 1e15f && fabsf(z) < 1e15f &&
                         fabsf(zq) < 1e15f;
        const bool lead_ok = (__ballot_sync(kAll, fin) >> lead) & 1u;
        // the ray's other pending points in the same cell and subcell
        const bool mate = r == lr && ((todom >> lane) & 1u) && fin && cx == bx && cy == by &&
                          cz == bz && sub == bs;
        float zlo = mate ? zq : zl, zhi = mate ? zq : zl;
#pragma unroll
        for (int off = 1; off < 4; off <<= 1) {
          zlo = fminf(zlo, __shfl_xor_sync(kAll, zlo, off));
          zhi = fmaxf(zhi, __shfl_xor_sync(kAll, zhi, off));
        }
        zlo = __shfl_sync(kAll, zlo, lead);
        zhi = __shfl_sync(kAll, zhi, lead);
        bool ok = false;
        if (lead_ok && fabsf(rox) < 1e15f && fabsf(roy) < 1e15f && fabsf(roz) < 1e15f) {
          const float len_l = sqrtf((rlx * rlx + rly * rly) + rlz * rlz);
          float ext = W.meta[lr].ext;
          // as far as the ray surely stays in the subcell: half the grid's margin
          // covers the rounding at the grid's own coordinates (8 roundings of 16),
          // the rest, or twice the ray's own rounding where that is more (a camera
          // thousands of box lengths away), that of its points. (Not their sum: a
          // ray close along a face gets a list per step within that distance; 128-bin
          // spectra and a tilted map lost up to 7 % to a margin 8 % wider.)
          const float zm = fmaxf(fmaxf(fabsf(zlo), fabsf(zhi)), fabsf(zlo + ext));
          const float keep =
              fmaxf(g.margin, 2.0f * ray_rounding(rox, roy, roz, zm, len_l));
          const float ex =
              axis_exit(rox, rlx, (g.min0 + (float)bx * g.cs0) + (float)(bs & 1) * g.half0,
                        g.half0, keep);
          const float ey =
              axis_exit(roy, rly, (g.min1 + (float)by * g.cs1) + (float)((bs >> 1) & 1) * g.half1,
                        g.half1, keep);
          const float ez =
              axis_exit(roz, rlz, (g.min2 + (float)bz * g.cs2) + (float)(bs >> 2) * g.half2,
                        g.half2, keep);
          const float reach = fminf(zlo + ext, fminf(ex, fminf(ey, ez)));
          float a = zlo, b = reach > zhi ? reach : zhi;
          int tested = -1;
#pragma unroll 1
          for (int attempt = 0; attempt < 3; ++attempt) {
            if (attempt == 1) {
              if (!(b > zhi)) continue;
              b = zhi;
            }
            if (attempt == 2) {
              if (!(zhi > zlo)) break;
              a = b = zl;
            }
            tested = build_list<kIdx>(g, spiral, W, lr, lane, rox, roy, roz, rlx, rly, rlz, len_l,
                                      bx, by, bz, bs, a, b);
            if (tested >= 0) break;
            ext *= 0.6f;
          }
          ok = tested >= 0;
          if (ok) {
            const int n = W.meta[lr].n, nu = W.meta[lr].nu;
            // The cost per step is least where a build's share of it equals
            // what its length adds to each replay. In warp instructions: a
            // build takes about 500, 0.4 per candidate looked at and 30 per
            // candidate kept; a candidate or break cell beyond the 16 of a
            // point's own list 14 of a replay. (6 / 12 / 24 for the 14:
            // projection 348 / 335 / 347 ms, 2048 fixed steps 151 / 128 / 133
            // ms, tilted band map through a core 37 / 35 / 33 ms; a fixed aim
            // of 34 candidates, 62 behind long searches: 418 / 151 / 45 ms.)
            const float build = (500.0f + 0.4f * (float)tested + 30.0f * (float)n) * hl;
            const float replay = 14.0f * (float)(n + nu - 16) * (b - a);
            // (Break cells near the limit, where a build is lost, shorten it at
            // once: projection 337 -> 292 ms, adjoint of a 64^2 map 108 -> 85
            // ms, with 48 instead of 64 candidates in shared memory, which
            // leaves 70 KB of L1 for the grid.)
            if (nu > kUnc - 6) ext *= 0.6f;
            else if (build < 0.8f * replay || n > 200) ext *= 0.85f;
            else if (build > 1.25f * replay) ext *= 1.2f;
          }
          ext = fminf(fmaxf(ext, g.half0 * 1e-4f), g.cs0);
          __syncwarp();
          if (lane == 0) W.meta[lr].ext = ext;
          __syncwarp();
        }
        if (!ok) {
          if (lane == lead) {
            WalkStats ps;
            point_walk<kIdx>(g, spiral, x, y, z, W.ent[lr], ps);
            st.cells += ps.cells;
            st.cands += ps.cands;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
              o.d[t] = W.ent[lr][t].x;
              o.v[t] = W.ent[lr][t].y;
            }
            W.meta[lr].za = 1.0f;
            W.meta[lr].zb = 0.0f;
            o.plain = false;
            todo = false;
          }
          __syncwarp();
        }
      }
      if (todo) {
        const RayMeta& m = W.meta[r];
        listed = zq >= m.za && zq <= m.zb;
      }
    }
    if (todo && listed) {
      replay_point<kIdx>(g, W, r, x, y, z, o, st);
      todo = false;
    }
    __syncwarp();
    if (!__any_sync(kAll, todo)) break;
  }
}

// get_weight3d and finalize in slot order
// (volumetric_nn8_reconstruction.cl:44-50,212-270).
__device__ __forceinline__ void slot_weights(const PointSlots& s, float w[8], float& ws) {
  if (s.plain) {
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const float i2 = rcp_normal(s.d[t] * s.d[t]);
      const float i4 = i2 * i2;
      w[t] = (i4 * i4) * i2;
    }
  } else {
#pragma unroll
    for (int t = 0; t < 8; ++t) w[t] = weight3d(s.d[t]);
  }
  ws = 0.0f;
#pragma unroll
  for (int t = 0; t < 8; ++t) ws = ws + w[t];
}

__device__ __forceinline__ float slots_value(const PointSlots& s) {
  float w[8], ws;
  slot_weights(s, w, ws);
  float dot = 0.0f;
#pragma unroll
  for (int t = 0; t < 8; ++t) dot = __fmaf_rn(w[t], s.v[t], dot);
  return (ws != 0.0f && dot != 0.0f) ? dot / ws : 0.0f;
}

// The queue positions of the rays that the groups in `want` (bits of their
// first lanes) take next. The first rays are dealt out one per warp, then a
// second one per warp and so on: the queue's head holds the costliest rays,
// and two of them in one warp would build their lists one after the other.
__device__ __forceinline__ unsigned long long take_rays(unsigned long long* queue, unsigned want,
                                                        bool first, int lane, unsigned wg) {
  const unsigned long long warps = (unsigned long long)gridDim.x * kListWarps;
  if (first) return (unsigned long long)(lane >> 2) * warps + wg;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(queue, (unsigned long long)__popc(want));
  return warps * kRays + __shfl_sync(kAll, base, 0) +
         __popc(want & ((1u << (lane & 28)) - 1u));
}

// Position of point j of the step (z, h) (rkf_points).
__device__ __forceinline__ float step_point(float z, float h, int j) {
  const float c = j == 0 ? 3.f / 8.f : j == 1 ? 12.f / 13.f : j == 2 ? 1.0f : 0.5f;
  return z + c * h;
}

// The 4 points' values of a ray, on all of its lanes.
__device__ __forceinline__ void share4(float v, int lane, float e[4]) {
  const int b = lane & 28;
#pragma unroll
  for (int j = 0; j < 4; ++j) e[j] = __shfl_sync(kAll, v, b + j);
}

}  // namespace ilc
