// ilc_quantity.cu -- per-cell quantity transforms of the X-ray path
// (quantities.cl:38-136, 156-260, 354-675) with the thermally averaged Gaunt
// factor table (gaunt_factor.cpp:30-41) resident in shared memory and the
// Chandra ARF (chandra.cpp, class chandra::arf) read through the read-only
// cache.
//
// The OpenCL image lookup (read_imagef, CLK_FILTER_LINEAR, CLK_ADDRESS_CLAMP,
// unnormalised coordinates; tabulated_function.cl:26-59) is done in software
// with exact fp32 weights: the sample at u blends texels floor(u-0.5) and
// floor(u-0.5)+1 with weight frac(u-0.5); texels outside the table read 0.
#include "ilc_device.cuh"
#include "ilc_internal.h"
#include "ilc_quantity.cuh"

namespace ilc {

namespace {

constexpr int kThreads = 256;
constexpr int kBlocksPerSm = 4;    // by the table in shared memory (51 KB) and 64 registers

// The (padded) Gaunt table into shared memory, 16 bytes at a time (the buffer is
// a multiple of 16 bytes long).
__device__ __forceinline__ void load_table(float* dst, const float* __restrict__ src, int n) {
  const float4* __restrict__ s4 = reinterpret_cast<const float4*>(src);
  for (int i = threadIdx.x; i < (n + 3) / 4; i += blockDim.x)
    reinterpret_cast<float4*>(dst)[i] = __ldg(s4 + i);
  __syncthreads();
}

// The 32-cell group this warp takes first: the groups are dealt over all blocks,
// then over a block's warps.
__device__ __forceinline__ uint64_t first_group() {
  return (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
}
__device__ __forceinline__ uint64_t first_cell() {
  return first_group() * 32 + (threadIdx.x & 31);
}

// xray_flux (quantities.cl:354-385); kPhoton: xray_photon_flux
// (quantities.cl:640-675), the band integral of emission / photon energy,
// converted from per m^2 to per cm^2. One cell per thread. Bound by
// instruction issue (84 % of the slots; 9 to 13 emission evaluations per cell
// for 12 B in and 4 B out). The four evaluations of a step overlap because
// emit() has no branches; with brems() and its IEEE divisions in their place
// 4,194,304 cells took 494 us, now 321.
template <bool kPhoton>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
xray_flux_kernel(const float* __restrict__ table, const __grid_constant__ GauntView G,
                 const float* __restrict__ rho, const float* __restrict__ u,
                 const float* __restrict__ xe, uint64_t n, float z, float dL, float emin,
                 float emax, int num_samples, float* __restrict__ out, int stride) {
  extern __shared__ __align__(16) float t[];
  load_table(t, table, (G.w + 2 * G.pad) * (G.h + 2 * G.pad));
  const EmitCall k = emit_call(G, dL);
  for (uint64_t i = first_cell(); i < n; i += (uint64_t)gridDim.x * kThreads) {
    const float T = temperature(u[i], xe[i]);
    const float f = band_flux<kPhoton>(t, G, k, (1.f + z) * emin, (1.f + z) * emax,
                                       1.f / (float)num_samples, T, xe[i], rho[i]);
    out[i * stride] = kPhoton ? f * 1.e-4f : f;
  }
}

// chandra_xray_total_count_rate (quantities.cl:510-557): the count rate summed
// in channel order over every ARF channel k, at energy x0 + k * dx with
// width dx. One cell per thread; a block computes each channel once, in chunks
// in shared memory, for all of its cells, instead of every thread for itself.
// 1024 channels of 131,072 cells: 1,718 -> 696 us (144 warp instructions per
// evaluation, 77 % of the issue slots).
constexpr int kChunk = 128;
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
chandra_total_kernel(const float* __restrict__ table, const __grid_constant__ GauntView G,
                     const float* __restrict__ arf, ArfView A, const float* __restrict__ rho,
                     const float* __restrict__ u, const float* __restrict__ xe, uint64_t n,
                     float z, float dL, float* __restrict__ out) {
  extern __shared__ __align__(16) float t[];
  Channel* ch = reinterpret_cast<Channel*>(t + kTableFloats);
  load_table(t, table, (G.w + 2 * G.pad) * (G.h + 2 * G.pad));
  const EmitCall k = emit_call(G, dL);
  // whole rounds of the block, so that all of its threads meet at the chunks;
  // a round's warps take 32 cells each, dealt over all blocks
  const uint64_t groups = (n + 31) / 32, warps = (uint64_t)gridDim.x * (kThreads / 32);
  const uint64_t w0 = first_group();
  for (uint64_t g0 = 0; g0 < groups; g0 += warps) {
    const uint64_t i = (g0 + w0) * 32 + (threadIdx.x & 31);
    const bool mine = i < n;
    const float x = mine ? xe[i] : 1.0f, r = mine ? rho[i] : 0.0f;
    const float T = temperature(mine ? u[i] : 1.0f, x);
    const EmitCell c = emit_cell(G, k, T, x, r);
    float em = 0.0f;
    for (int q0 = 0; q0 < A.n; q0 += kChunk) {
      __syncthreads();
      for (int q = threadIdx.x; q < kChunk && q0 + q < A.n; q += kThreads) {
        const float e = A.x0 + (float)(q0 + q) * A.dx;
        ch[q] = make_channel<true>(arf, A, e, A.dx, z);
      }
      __syncthreads();
      const int m = min(kChunk, A.n - q0);
      if (!mine) continue;
      int q = 0;
      if (c.col >= 0) {
        // two channels at a time: their evaluations overlap
        for (; q + 2 <= m; q += 2) {
          const Channel h0 = ch[q], h1 = ch[q + 1];
          bool ok = h0.yEz != 0.0f && h1.yEz != 0.0f;
          const float v0 = emit<true>(t, G, k, c, h0.Ez, h0.pre, ok, h0.yEz) * h0.av;
          const float v1 = emit<true>(t, G, k, c, h1.Ez, h1.pre, ok, h1.yEz) * h1.av;
          if (ok) {
            em += v0;
            em += v1;
          } else {
            em += channel_value<true>(t, G, k, c, h0, T, x, r);
            em += channel_value<true>(t, G, k, c, h1, T, x, r);
          }
        }
      }
      for (; q < m; ++q) em += channel_value<true>(t, G, k, c, ch[q], T, x, r);
    }
    if (mine) out[i] = em;
  }
}

// chandra_xray_spectral_count_rate (quantities.cl:584-622): one channel.
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
chandra_bin_kernel(const float* __restrict__ table, const __grid_constant__ GauntView G,
                   const float* __restrict__ arf, ArfView A, const float* __restrict__ rho,
                   const float* __restrict__ u, const float* __restrict__ xe, uint64_t n, float z,
                   float dL, float e, float de, float* __restrict__ out) {
  extern __shared__ __align__(16) float t[];
  load_table(t, table, (G.w + 2 * G.pad) * (G.h + 2 * G.pad));
  const EmitCall k = emit_call(G, dL);
  const Channel h = make_channel<true>(arf, A, e, de, z);
  for (uint64_t i = first_cell(); i < n; i += (uint64_t)gridDim.x * kThreads) {
    const float T = temperature(u[i], xe[i]);
    const EmitCell c = emit_cell(G, k, T, xe[i], rho[i]);
    out[i] = channel_value<true>(t, G, k, c, h, T, xe[i], rho[i]);
  }
}

// xray_spectral_flux (quantities.cl:400-430)
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
xray_bin_kernel(const float* __restrict__ table, const __grid_constant__ GauntView G,
                const float* __restrict__ rho, const float* __restrict__ u,
                const float* __restrict__ xe, uint64_t n, float z, float dL, float e, float de,
                float* __restrict__ out) {
  extern __shared__ __align__(16) float t[];
  load_table(t, table, (G.w + 2 * G.pad) * (G.h + 2 * G.pad));
  const EmitCall k = emit_call(G, dL);
  const Channel h = make_channel<false>(nullptr, ArfView{}, e, de, z);
  for (uint64_t i = first_cell(); i < n; i += (uint64_t)gridDim.x * kThreads) {
    const float T = temperature(u[i], xe[i]);
    const EmitCell c = emit_cell(G, k, T, xe[i], rho[i]);
    out[i] = channel_value<false>(t, G, k, c, h, T, xe[i], rho[i]);
  }
}

// xray_spectral_flux (kChandra: chandra_xray_spectral_count_rate) for n_bins
// bins at once, cell-major out[i * n_bins + b] as ilc_render_batched reads it
// (the quantity of each frame of spectrum_generator, spectrum.cpp:89-109, or
// of chandra_spectrum_quantity_generator, spectrum.cpp:45-65).
//
// A warp takes `group` cells (at most 32): each lane prepares one of them in
// shared memory, then the lanes run over the group x n_bins outputs, which are
// consecutive in memory.
// So what depends on the cell is computed once instead of once per bin, and
// what depends on the bin once per block and chunk of bins. 128 bins of 300,007
// cells: 592 -> 256 us; 3 blocks per SM (71 registers, 66 KB).
constexpr int kBinChunk = 128;
struct CellShare {
  EmitCell c;
  float T, xe, rho;
  float pad;  // 11 words: consecutive cells start at different banks
};
template <bool kChandra>
__global__ void __launch_bounds__(kThreads, 3)
bins_kernel(const float* __restrict__ table, const __grid_constant__ GauntView G,
            const float* __restrict__ arf, ArfView A, const float* __restrict__ rho,
            const float* __restrict__ u, const float* __restrict__ xe, uint64_t n, float z,
            float dL, const float* __restrict__ e, const float* __restrict__ de, int n_bins,
            int group, float* __restrict__ out) {
  extern __shared__ __align__(16) float t[];
  Channel* ch = reinterpret_cast<Channel*>(t + kTableFloats);
  CellShare* cells = reinterpret_cast<CellShare*>(ch + kBinChunk) + (threadIdx.x & ~31u);
  load_table(t, table, (G.w + 2 * G.pad) * (G.h + 2 * G.pad));
  const EmitCall k = emit_call(G, dL);
  const int lane = threadIdx.x & 31;
  const uint64_t groups = (n + group - 1) / group;
  const uint64_t warps = (uint64_t)gridDim.x * (kThreads / 32);
  const uint64_t w0 = first_group();
  for (int b0 = 0; b0 < n_bins; b0 += kBinChunk) {
    const int nb = min(kBinChunk, n_bins - b0);
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += kThreads)
      ch[b] = make_channel<kChandra>(arf, A, e[b0 + b], de[b0 + b], z);
    __syncthreads();
    for (uint64_t g = w0; g < groups; g += warps) {
      const uint64_t i0 = g * group;
      const int m = (int)min((uint64_t)group, n - i0);
      __syncwarp();
      if (lane < m) {
        CellShare s;
        s.xe = xe[i0 + lane];
        s.rho = rho[i0 + lane];
        s.T = temperature(u[i0 + lane], s.xe);
        s.c = emit_cell(G, k, s.T, s.xe, s.rho);
        cells[lane] = s;
      }
      __syncwarp();
      // outputs (cell, bin), bins fastest, 32 further on each turn; two turns
      // at a time, whose evaluations overlap
      const int dc = 32 / nb, db = 32 - dc * nb;
      int cell = lane / nb, bin = lane - cell * nb;
      while (cell < m) {
        int cell1 = cell + dc, bin1 = bin + db;
        if (bin1 >= nb) {
          bin1 -= nb;
          ++cell1;
        }
        const bool two = cell1 < m;
        const CellShare& s0 = cells[cell];
        const CellShare& s1 = cells[two ? cell1 : cell];
        const Channel &h0 = ch[bin], &h1 = ch[bin1];
        bool ok = s0.c.col >= 0 && s1.c.col >= 0 && h0.yEz != 0.0f && h1.yEz != 0.0f;
        float v0 = 0.0f, v1 = 0.0f;
        if (ok) {
          v0 = emit<kChandra>(t, G, k, s0.c, h0.Ez, h0.pre, ok, h0.yEz);
          v1 = emit<kChandra>(t, G, k, s1.c, h1.Ez, h1.pre, ok, h1.yEz);
          if (kChandra) {
            v0 = v0 * h0.av;
            v1 = v1 * h1.av;
          }
        }
        if (!ok) {
          v0 = channel_value<kChandra>(t, G, k, s0.c, h0, s0.T, s0.xe, s0.rho);
          v1 = channel_value<kChandra>(t, G, k, s1.c, h1, s1.T, s1.xe, s1.rho);
        }
        float* o = out + i0 * (uint64_t)n_bins + b0;
        o[(uint64_t)cell * n_bins + bin] = v0;
        if (two) o[(uint64_t)cell1 * n_bins + bin1] = v1;
        cell = cell1 + dc;
        bin = bin1 + db;
        if (bin >= nb) {
          bin -= nb;
          ++cell;
        }
      }
    }
  }
}
constexpr size_t kBinsSmem =
    kTableFloats * 4 + kBinChunk * sizeof(Channel) + kThreads * sizeof(CellShare);

// mean_temperature (quantities.cl:268-284)
__global__ void temperature_kernel(const float* __restrict__ u, const float* __restrict__ xe,
                                   uint64_t n, float* __restrict__ out) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = temperature(u[i], xe[i]);
}

// As many blocks as are resident (per_sm each), so that a block loads the
// table once; fewer for a few cells. A block's warps take 32 cells each, dealt
// over all blocks first, so that every SM gets its share of a few cells too.
unsigned resident_blocks(const Context& c, uint64_t groups, int per_sm) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
  const uint64_t want = groups, fit = (uint64_t)(sms > 0 ? sms : 148) * per_sm;
  return (unsigned)(want < fit ? want : fit);
}

GauntView gaunt_view(const Context& c) {
  return GauntView{c.gw, c.gh, c.gx0, c.gy0, c.gdx, c.gdy, table_pad(c.gw, c.gh)};
}
ArfView arf_view(const Context& c) { return ArfView{c.arf_n, c.arf_x0, c.arf_dx}; }

// Cells per warp of a bin table: enough for about 32 turns of its lanes, and
// fewer, down to one, while that leaves warps without a group. (300,007 cells of
// 128 bins: 268 us in groups of 32, 256 us in groups of 8; 300 cells of 128
// bins: 52 us and 28 us, 34 us when every output was a thread of its own.)
int bin_group(uint64_t n, int n_bins) {
  int group = 32;
  while (group > 1 && ((int64_t)group * n_bins > 1024 ||
                       ((int64_t)group * n_bins > 32 && n / group < 148 * 3 * (kThreads / 32))))
    group /= 2;
  return group;
}

// Launches one of the kernels above, a warp to each of `groups`, with its
// dynamic shared memory.
template <class... P, class... Q>
cudaError_t launch(Context& c, void (*kernel)(P...), uint64_t groups, int per_sm, size_t smem,
                   Q... args) {
  const cudaError_t e = cudaFuncSetAttribute(
      kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e) return e;
  ++c.launches;
  kernel<<<resident_blocks(c, groups, per_sm), kThreads, smem, c.stream>>>(
      c.gaunt_pad.as<float>(), gaunt_view(c), args...);
  return cudaGetLastError();
}
constexpr size_t kTableSmem = kTableFloats * 4;

}  // namespace

cudaError_t quantity_xray_flux_launch(Context& c, const float* rho, const float* u,
                                      const float* xe, uint64_t n, float z, float dL,
                                      float emin, float emax, int num_samples, float* out,
                                      int out_stride) {
  return launch(c, xray_flux_kernel<false>, (n + 31) / 32, kBlocksPerSm, kTableSmem, rho, u, xe, n, z, dL,
                emin, emax, num_samples, out, out_stride);
}

cudaError_t quantity_xray_photon_flux_launch(Context& c, const float* rho, const float* u,
                                             const float* xe, uint64_t n, float z, float dL,
                                             float emin, float emax, int num_samples,
                                             float* out) {
  return launch(c, xray_flux_kernel<true>, (n + 31) / 32, kBlocksPerSm, kTableSmem, rho, u, xe, n, z, dL,
                emin, emax, num_samples, out, 1);
}

cudaError_t quantity_chandra_total_launch(Context& c, const float* rho, const float* u,
                                          const float* xe, uint64_t n, float z, float dL,
                                          float* out) {
  return launch(c, chandra_total_kernel, (n + 31) / 32, kBlocksPerSm, kTableSmem + kChunk * sizeof(Channel),
                c.arf.as<float>(), arf_view(c), rho, u, xe, n, z, dL, out);
}

cudaError_t quantity_chandra_bin_launch(Context& c, const float* rho, const float* u,
                                        const float* xe, uint64_t n, float z, float dL, float e,
                                        float de, float* out) {
  return launch(c, chandra_bin_kernel, (n + 31) / 32, kBlocksPerSm, kTableSmem, c.arf.as<float>(),
                arf_view(c), rho, u, xe, n, z, dL, e, de, out);
}

cudaError_t quantity_chandra_bins_launch(Context& c, const float* rho, const float* u,
                                         const float* xe, uint64_t n, float z, float dL,
                                         const float* e, const float* de, int n_bins,
                                         float* out) {
  const int group = bin_group(n, n_bins);
  return launch(c, bins_kernel<true>, (n + group - 1) / group, 3, kBinsSmem, c.arf.as<float>(),
                arf_view(c), rho, u, xe, n, z, dL, e, de, n_bins, group, out);
}

cudaError_t quantity_xray_bin_launch(Context& c, const float* rho, const float* u,
                                     const float* xe, uint64_t n, float z, float dL, float e,
                                     float de, float* out) {
  return launch(c, xray_bin_kernel, (n + 31) / 32, kBlocksPerSm, kTableSmem, rho, u, xe, n, z, dL, e, de,
                out);
}

cudaError_t quantity_xray_bins_launch(Context& c, const float* rho, const float* u,
                                      const float* xe, uint64_t n, float z, float dL,
                                      const float* e, const float* de, int n_bins, float* out) {
  const int group = bin_group(n, n_bins);
  return launch(c, bins_kernel<false>, (n + group - 1) / group, 3, kBinsSmem, c.arf.as<float>(),
                arf_view(c), rho, u, xe, n, z, dL, e, de, n_bins, group, out);
}

cudaError_t quantity_temperature_launch(Context& c, const float* u, const float* xe,
                                        uint64_t n, float* out) {
  ++c.launches;
  temperature_kernel<<<(unsigned)((n + 255) / 256), 256, 0, c.stream>>>(u, xe, n, out);
  return cudaGetLastError();
}

}  // namespace ilc
