// k_dust.cu - grain opacity, grain re-emission CDF and grain radiative
// equilibrium of a dust-only grid.  Compiled with --fmad=false: every FP32
// operation rounds separately, in the order the reference writes it.
#include "k_dust.cuh"
#include "setup_internal.h"

#include <algorithm>
#include <vector>

namespace mcx {

namespace {

__device__ __forceinline__ float tdAt(const float* td, int n, int ai, int nSz, int c, int C1) {
  return td[((size_t)n * (nSz + 1) + ai) * C1 + c];
}

// getFlux of source/continuum_mod.f90:358-405 for a blackbody
__device__ float blackbody(float energy, float temperature) {
  const float hcRyd_k = 157893.94f, hPlanck = 6.6262e-27f;
  const float constant = 0.5250229f / hPlanck;
  if (hcRyd_k * energy / temperature > 86.f)
    return constant * energy * energy * energy * expf(-hcRyd_k * energy / temperature);
  const float denominator = expf(hcRyd_k * energy / temperature) - 1.f;
  if (denominator <= 0.f) return 3.32154e-6f * energy * energy * temperature / hPlanck;
  return constant * energy * energy * energy / denominator;
}

// A thread holds one cell and kOpBins bins: each grain temperature and each
// abundance product is read or formed once for its bins.  Bound by memory then
// (opacity read and written, scaOpac written); 61^3 shell, 215 bins: 0.70 -> 0.22 ms.
constexpr int kOpBins = 8;

__global__ void __launch_bounds__(256)
dustOpacityKernel(DustDev d, const float* __restrict__ ndust, const float* __restrict__ tdust,
                  float* __restrict__ opacity, float* __restrict__ scaOpac) {
  const int C1 = d.nCells + 1;
  const int c = blockIdx.x * blockDim.x + threadIdx.x + 1, f0 = blockIdx.y * kOpBins;
  if (c > d.nCells) return;
  const int nf = min(kOpBins, d.nbins - f0);
  const float nd = ndust[c];
  float sca[kOpBins], absO[kOpBins];
#pragma unroll
  for (int u = 0; u < kOpBins; ++u) sca[u] = absO[u] = 0.f;
  for (int n = 0; n < d.nSpecies; ++n)
    for (int ai = 0; ai < d.nSizes; ++ai) {
      if (!(tdAt(tdust, n + 1, ai + 1, d.nSizes, c, C1) < d.tsub[n])) continue;
      const size_t o = ((size_t)n * d.nSizes + ai) * d.nbins + f0;
      const float w = d.abun[n] * d.weight[ai] * nd;
#pragma unroll
      for (int u = 0; u < kOpBins; ++u) {
        if (u < nf) {
          sca[u] = sca[u] + w * d.Csca[o + u];
          absO[u] = absO[u] + w * d.Cabs[o + u];
        }
      }
    }
#pragma unroll
  for (int u = 0; u < kOpBins; ++u) {
    if (u < nf) {
      const size_t idx = (size_t)(f0 + u) * C1 + c;
      scaOpac[idx] = sca[u];
      opacity[idx] = opacity[idx] + (sca[u] + absO[u]);
    }
  }
}

// The cumulative re-emission of 32 cells a block, one per lane: kPdfWarps warps
// work out four bins each of a tile (kinds outside, so a grain's temperature is
// read once for them, the sum over the kinds in its own order), then the first
// warp continues the cumulative sum over the tile while the others go on with the
// next.  Bound by the exponentials and divisions.  A thread walking all bins of its
// cell took 1.6 ms on the 61^3 shell (215 bins), and three more passes to normalise and
// transpose 0.3; 0.98 and 0.09 now.
constexpr int kPdfWarps = 8, kPdfBins = 4, kPdfTile = kPdfWarps * kPdfBins;

__global__ void __launch_bounds__(32 * kPdfWarps)
dustPDFKernel(DustDev d, const float* __restrict__ tdust, float* __restrict__ pdf) {
  __shared__ float tile[2][kPdfTile][32];
  const int C1 = d.nCells + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int at = blockIdx.x * 32 + lane + 1;
  const bool valid = at <= d.nCells;
  const int c = valid ? at : d.nCells;
  const int nb = d.nbins;
  float acc = 0.f;
  for (int t0 = 0, buf = 0; t0 < nb; t0 += kPdfTile, buf ^= 1) {
    const int i0 = t0 + warp * kPdfBins;
    if (i0 < nb) {
      float nu[kPdfBins], wid[kPdfBins], v[kPdfBins];
#pragma unroll
      for (int u = 0; u < kPdfBins; ++u) {
        const int i = min(i0 + u, nb - 1);
        nu[u] = d.nu[i];
        wid[u] = d.widFlx[i];
        v[u] = 0.f;
      }
      for (int n = 0; n < d.nSpecies; ++n)
        for (int ai = 0; ai < d.nSizes; ++ai) {
          const float td = tdAt(tdust, n + 1, ai + 1, d.nSizes, c, C1);
          if (!(td > 0.f && td < d.tsub[n])) continue;
          const float* ca = d.Cabs + ((size_t)n * d.nSizes + ai) * nb;
#pragma unroll
          for (int u = 0; u < kPdfBins; ++u)
            v[u] = v[u] + ca[min(i0 + u, nb - 1)] * blackbody(nu[u], td) * wid[u] * d.weight[ai] * d.abun[n];
        }
#pragma unroll
      for (int u = 0; u < kPdfBins; ++u) tile[buf][warp * kPdfBins + u][lane] = v[u];
    }
    __syncthreads();   // one per tile: a buffer is written again two tiles on
    if (warp == 0) {
      const int m = min(kPdfTile, nb - t0);
      for (int r = 0; r < m; ++r) {
        acc = t0 + r == 0 ? tile[buf][r][lane] : acc + tile[buf][r][lane];
        if (valid) pdf[(size_t)(t0 + r) * C1 + c] = acc;
      }
    }
  }
}

// The distribution normalised, in both layouts: 32 x 32 tiles through shared
// memory.  Row 0 and column 0 of the transpose follow what pdf holds there.
__global__ void __launch_bounds__(256)
dustNormaliseKernel(int nCells, int nb, float* __restrict__ pdf, const float* __restrict__ tot, float* __restrict__ cdfT) {
  __shared__ float tile[32][33];
  const size_t C1 = (size_t)nCells + 1;
  const int c0 = blockIdx.x * 32, b0 = blockIdx.y * 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int c = c0 + x;
  if (c <= nCells) {
    const float t = tot[c];
#pragma unroll
    for (int r = y; r < 32; r += 8) {
      const int b = b0 + r;
      if (b >= nb) break;
      const size_t at = (size_t)b * C1 + c;
      float v = pdf[at];
      if (c >= 1) {
        v = b == nb - 1 ? 1.f : v / t;
        pdf[at] = v;
      }
      tile[r][x] = v;
    }
  }
  __syncthreads();
  if (b0 + x < nb) {
#pragma unroll
    for (int r = y; r < 32; r += 8)
      if (c0 + r <= nCells) cdfT[(size_t)(c0 + r) * nb + b0 + x] = tile[x][r];
  }
}

// locate (source/interpolation_mod.f90:49-106) on an ascending table
__device__ int locateAsc(const float* xa, int n, float x) {
  if (x > xa[n - 1]) return n;
  if (x < xa[0]) return 0;
  int jlow = 0, jup = n + 1;
  for (int it = 0; it < 10000; ++it) {
    if (jup - jlow < 1) break;
    const int jm = (jup + jlow) / 2;
    if (xa[jm - 1] == x) return jm;
    if (x > xa[jm - 1]) {
      if (jlow == jm) break;
      jlow = jm;
    } else {
      jup = jm;
    }
  }
  return jlow;
}

// 32 cells a block, one per lane; each warp sums the absorbed energy of kTKinds
// grain kinds over the bins (each sum in the order of the bins), so J is read,
// rounded and divided by pi once per kTKinds kinds instead of once per kind, from
// the table of cross sections staged in shared memory.  Bound by the loads of J (FP64);
// 61^3 shell: 2.7 -> 0.35 ms.
constexpr int kTKinds = 8, kTMaxWarps = 8, kTBins = 32;

__global__ void __launch_bounds__(32 * kTMaxWarps)
dustTKernel(DustDev d, const double* __restrict__ jste, float* __restrict__ tdust, int32_t* converged,
            int32_t* black) {
  __shared__ __align__(16) float ca[kTBins][kTMaxWarps * kTKinds];
  const int C1 = d.nCells + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int at = blockIdx.x * 32 + lane + 1;
  const bool valid = at <= d.nCells;
  const int c = valid ? at : d.nCells;
  const int nb = d.nbins, nSz = d.nSizes, kinds = d.nSpecies * nSz;
  const float pi = 3.141592654f;
  const float xOld = tdAt(tdust, 0, 0, nSz, c, C1);
  bool hit = false;
  for (int g0 = 0; g0 == 0 || g0 < kinds; g0 += warps * kTKinds) {
    const int k0 = g0 + warp * kTKinds;
    float integral[kTKinds];
#pragma unroll
    for (int k = 0; k < kTKinds; ++k) integral[k] = 0.f;
    for (int b0 = 0; b0 < nb; b0 += kTBins) {
      __syncthreads();
      for (int k = warp; k < warps * kTKinds; k += warps)
        ca[lane][k] = b0 + lane < nb && g0 + k < kinds ? d.Cabs[(size_t)(g0 + k) * nb + b0 + lane] : 0.f;
      __syncthreads();
      const int m = min(kTBins, nb - b0);
      const double* J = jste + (size_t)b0 * C1 + c;
#pragma unroll 8
      for (int i = 0; i < m; ++i) {
        const float j = (float)J[(size_t)i * C1];
        hit |= j > 0.f;
        const float jp = j / pi;
        const float4 a0 = *(const float4*)&ca[i][warp * kTKinds], a1 = *(const float4*)&ca[i][warp * kTKinds + 4];
        integral[0] = integral[0] + a0.x * jp;
        integral[1] = integral[1] + a0.y * jp;
        integral[2] = integral[2] + a0.z * jp;
        integral[3] = integral[3] + a0.w * jp;
        integral[4] = integral[4] + a1.x * jp;
        integral[5] = integral[5] + a1.y * jp;
        integral[6] = integral[6] + a1.z * jp;
        integral[7] = integral[7] + a1.w * jp;
      }
    }
    if (valid && hit) {
#pragma unroll
      for (int k = 0; k < kTKinds; ++k) {
        const int kind = k0 + k;
        if (kind < kinds) {
          const float* em = d.emInt + (size_t)kind * kNTemps;
          const int iT = locateAsc(em, kNTemps, integral[k]);
          float t;
          if (iT <= 0) t = 1.f;
          else if (iT >= kNTemps) t = (float)kNTemps;
          else t = (float)iT + (integral[k] - em[iT - 1]) * ((float)(iT + 1) - (float)iT) / (em[iT] - em[iT - 1]);
          tdust[((size_t)(kind / nSz + 1) * (nSz + 1) + (kind % nSz + 1)) * C1 + c] = t;
        }
      }
    }
  }
  __syncthreads();   // the block's grain temperatures are written
  if (warp != 0 || !valid) return;
  black[c] = hit ? 0 : 1;
  converged[c] = 0;
  if (!hit) {
    atomicAdd(&d.counters->noHit, 1ull);
    return;
  }
  for (int ai = 1; ai <= nSz; ++ai) tdust[(size_t)ai * C1 + c] = 0.f;
  float t00 = 0.f;
  for (int n = 0; n < d.nSpecies; ++n) {
    float tn0 = 0.f;
    for (int ai = 0; ai < nSz; ++ai) tn0 = tn0 + tdust[((size_t)(n + 1) * (nSz + 1) + (ai + 1)) * C1 + c] * d.weight[ai];
    tdust[((size_t)(n + 1) * (nSz + 1)) * C1 + c] = tn0;
    t00 = t00 + tn0 * d.abun[n];
  }
  tdust[c] = t00;
  const float delta = (t00 - xOld) / xOld;
  const int conv = fabsf(delta) <= d.xhiLimit ? 1 : 0;
  converged[c] = conv;
  atomicAdd(&d.counters->updated, 1ull);
  if (conv) atomicAdd(&d.counters->converged, 1ull);
}

}  // namespace

DustData::~DustData() {
  for (int i = 0; i < nBlocks; ++i)
    if (blocks[i]) cudaFree(blocks[i]);
}

std::string dustDataCreate(const Setup& s, std::unique_ptr<DustData>& out) {
  auto dd = std::make_unique<DustData>();
  DustDev& d = dd->dev;
  const DustTables& t = s.dust;
  d.nbins = s.nbins; d.nCells = s.nCells; d.nSpecies = t.nSpecies; d.nSizes = t.nSizes;
  d.xhiLimit = s.p.XHILimit;
  std::string err;
  auto up = [&](const void* src, size_t bytes) -> void* {
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes ? bytes : 1);
    if (e != cudaSuccess) { err = std::string("dust tables: ") + cudaGetErrorString(e); return nullptr; }
    dd->blocks[dd->nBlocks++] = p;
    if (bytes && src) {
      e = cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice);
      if (e != cudaSuccess) err = std::string("dust tables: ") + cudaGetErrorString(e);
    }
    return p;
  };
  d.nu = (const float*)up(s.nu.data(), s.nu.size() * 4);
  d.widFlx = (const float*)up(s.widFlx.data(), s.widFlx.size() * 4);
  d.Cabs = (const float*)up(t.Cabs.data(), t.Cabs.size() * 4);
  d.Csca = (const float*)up(t.Csca.data(), t.Csca.size() * 4);
  d.abun = (const float*)up(t.grainAbun.data(), t.grainAbun.size() * 4);
  d.tsub = (const float*)up(t.TdustSublime.data(), t.TdustSublime.size() * 4);
  d.weight = (const float*)up(t.grainWeight.data(), t.grainWeight.size() * 4);
  d.emInt = (const float*)up(t.emIntegral.data(), t.emIntegral.size() * 4);
  d.counters = (DustCounters*)up(nullptr, sizeof(DustCounters));
  d.total = (float*)up(nullptr, ((size_t)s.nCells + 1) * sizeof(float));
  if (!err.empty()) return err;
  out = std::move(dd);
  return "";
}

cudaError_t launchDustOpacity(const DustDev& d, const float* ndust, const float* tdust, float* opacity, float* scaOpac,
                              cudaStream_t s) {
  const int T = 256;
  dustOpacityKernel<<<dim3((d.nCells + T - 1) / T, (d.nbins + kOpBins - 1) / kOpBins), T, 0, s>>>(d, ndust, tdust, opacity,
                                                                                                  scaOpac);
  return cudaGetLastError();
}

cudaError_t launchDustPDF(const DustDev& d, const float* tdust, float* dustPDF, float* dustCDFT, cudaStream_t s) {
  const size_t C1 = (size_t)d.nCells + 1;
  dustPDFKernel<<<(d.nCells + 31) / 32, 32 * kPdfWarps, 0, s>>>(d, tdust, dustPDF);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)   // the last bin's row becomes 1: its sums are kept aside
    e = cudaMemcpyAsync(d.total, dustPDF + (size_t)(d.nbins - 1) * C1, C1 * sizeof(float), cudaMemcpyDeviceToDevice, s);
  if (e != cudaSuccess) return e;
  dustNormaliseKernel<<<dim3((unsigned)((C1 + 31) / 32), (d.nbins + 31) / 32), 256, 0, s>>>(d.nCells, d.nbins, dustPDF,
                                                                                           d.total, dustCDFT);
  return cudaGetLastError();
}

cudaError_t launchDustT(const DustDev& d, const double* jste, float* tdust, int32_t* converged, int32_t* black,
                        cudaStream_t s) {
  const int warps = std::max(1, std::min(kTMaxWarps, (d.nSpecies * d.nSizes + kTKinds - 1) / kTKinds));
  cudaError_t e = cudaMemsetAsync(d.counters, 0, sizeof(DustCounters), s);
  if (e != cudaSuccess) return e;
  dustTKernel<<<(d.nCells + 31) / 32, 32 * warps, 0, s>>>(d, jste, tdust, converged, black);
  return cudaGetLastError();
}

}  // namespace mcx
