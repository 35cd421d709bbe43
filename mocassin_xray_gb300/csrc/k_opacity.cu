// k_opacity.cu - per-cell opacity kappa(nu) for every active cell at once.
//
// Restates ionizationDriver / BoltGaunt / getGauntFF / eDenSum / addOpacity
// (source/ionization_mod.f90:26-477) as one kernel: a thread owns kOpCells cells
// and walks one chunk of the frequency mesh (blockIdx.y), kOpBins bins at a
// time, so that the store kappa[nu][cell] of a warp is one coalesced 128-byte
// row segment.  The bound-free terms are listed per group of kOpBins bins (built
// once on the host in the reference's summation order: H, HeI, HeII, then
// element / ion / shell) with the cross section at each bin, 0 where a shell is
// closed: a term costs a slot, two 16-byte cross-section loads (the same for
// every lane) and one shared-memory density per cell, and feeds
// kOpBins x kOpCells FMAs, each bin's in the reference's order (an FMA with a
// zero cross section leaves the sum as it is).  One bin at a time every term
// took three loads for one FMA.  Arithmetic is FP32 as in the reference.
// Measured, 41^3 cells x 600 bins, 7 elements: 0.85 ms with one bin and one cell
// a thread, 0.30 ms now; bound by issue (the FMAs and the Gaunt factor).
// Behaviours of the reference kept here: the free-free prefactor has no H+ or
// He++ term (density(1,2) and density(2,3) are never filled,
// source/ionization_mod.f90:71-84), and an empty shell adds one term at bin 2
// (inOpacity's loop bound, source/ionization_mod.f90:451-476).
#include <algorithm>

#include "k_opacity.cuh"
#include "mcx_device.cuh"
#include "k_gaunt.cuh"

namespace mcx {

constexpr int kOpThreads = 128, kOpCells = 2;

__global__ void __launch_bounds__(kOpThreads)
opacityKernel(OpacityDev t, const float* __restrict__ hden, const float* __restrict__ te,
              const float* __restrict__ ne, const float* __restrict__ ionDen, const float* __restrict__ gauntTe,
              const uint8_t* __restrict__ compute, float* __restrict__ opacity) {
  extern __shared__ float sDen[];   // [nSlots][kOpCells][blockDim.x]
  const int T = blockDim.x;
  const size_t C1 = (size_t)t.nCells + 1;
  const float Te1Ryd = 1.578866e5f;
  int cell[kOpCells];
  bool valid[kOpCells], any = false;
  float Te[kOpCells], Ne[kOpCells], fac1[kOpCells], fac2[kOpCells], c[kOpCells][9], con[kOpCells], gamma2[kOpCells];
#pragma unroll
  for (int w = 0; w < kOpCells; ++w) {
    cell[w] = (blockIdx.x * kOpCells + w) * T + threadIdx.x + 1;
    valid[w] = cell[w] <= t.nCells && compute[cell[w]];
    any = any || valid[w];
    Te[w] = 1.f; Ne[w] = 0.f; fac1[w] = 0.f; fac2[w] = 0.f; con[w] = 0.f; gamma2[w] = 0.f;
#pragma unroll
    for (int k = 0; k < 9; ++k) c[w][k] = 0.f;
    if (valid[w]) {
      Te[w] = te[cell[w]]; Ne[w] = ne[cell[w]];
      const float H = hden[cell[w]];
      float wsum = 0.f;
      for (int s = 0; s < t.nSlots; ++s) {
        float d = ionDen[(size_t)cell[w] + C1 * (size_t)t.slotPlane[s]] * t.slotAbun[s] * H;
        sDen[(s * kOpCells + w) * T + threadIdx.x] = d;
        wsum += t.slotFFWeight[s] * d;
      }
      // addOpacity free-free prefactor (source/ionization_mod.f90:366-368)
      fac1[w] = (Ne[w] / 1.e10f) * (wsum / 1.e10f) / sqrtf(Te[w]);
      fac2[w] = fac1[w] * Te1Ryd / Te[w];
      gauntCoeffs(0.f, log10f(gauntTe[cell[w]]), c[w], con[w], gamma2[w]);
    } else {
      for (int s = 0; s < t.nSlots; ++s) sDen[(s * kOpCells + w) * T + threadIdx.x] = 0.f;
    }
  }
  if (!any) return;
  const float* den = sDen + threadIdx.x;
  const int groups = (t.nbins + kOpBins - 1) / kOpBins;
  const int chunk = (groups + gridDim.y - 1) / gridDim.y;
  const int g0 = blockIdx.y * chunk, g1 = min(groups, g0 + chunk);
  for (int g = g0; g < g1; ++g) {
    const int b0 = g * kOpBins;
    float op[kOpCells][kOpBins];
#pragma unroll
    for (int q = 0; q < kOpBins; ++q) {
      const int i = min(b0 + q, t.nbins - 1);
      const float nui = t.nu[i], xb = t.xsec[i + t.bremsP0], l10 = t.log10nu[i];
#pragma unroll
      for (int w = 0; w < kOpCells; ++w) {
        const float ex = Te1Ryd / Te[w] + nui;
        const float boltz = ex > 84.f ? 0.f : expf(-ex);
        const float gf = gauntAt(c[w], con[w], gamma2[w], l10);
        op[w][q] = boltz < 0.995f ? xb * (1.f - boltz) * gf * fac1[w] : xb * nui * gf * fac2[w];
      }
    }
    const int e1 = t.termStart[g + 1];
#pragma unroll 4
    for (int e = t.termStart[g]; e < e1; ++e) {
      const float4 xa = __ldg(t.termXs + 2 * (size_t)e), xc = __ldg(t.termXs + 2 * (size_t)e + 1);
      const float* d = den + __ldg(t.termSlot + e) * (kOpCells * T);
#pragma unroll
      for (int w = 0; w < kOpCells; ++w) {
        const float dw = d[w * T];
        op[w][0] += xa.x * dw; op[w][1] += xa.y * dw; op[w][2] += xa.z * dw; op[w][3] += xa.w * dw;
        op[w][4] += xc.x * dw; op[w][5] += xc.y * dw; op[w][6] += xc.z * dw; op[w][7] += xc.w * dw;
      }
    }
#pragma unroll
    for (int q = 0; q < kOpBins; ++q) {
      const int i = b0 + q;
      if (i >= t.nbins) break;
      const float kn = t.lgCompton ? t.KNsigmaT[i] : 0.f;
#pragma unroll
      for (int w = 0; w < kOpCells; ++w) {
        float o = op[w][q];
        if (t.lgCompton) o += kn * Ne[w];
        if (valid[w]) opacity[(size_t)cell[w] + C1 * (size_t)i] = o;
      }
    }
  }
}

// Cells with an infinite density again, with the terms of the open shells alone: 0
// times infinity is no zero.  (A density that is no number makes the free-free sum, and
// with it every bin, NaN.)  Such a cell is told by its first bin, so that the kernel above
// need not look: a test of its own there, on no cell, cost it 25 of 380 us, this kernel costs 4.
__global__ void __launch_bounds__(kOpThreads)
opacityOpenShellsKernel(OpacityDev t, const float* __restrict__ hden, const float* __restrict__ te,
                        const float* __restrict__ ne, const float* __restrict__ ionDen, const float* __restrict__ gauntTe,
                        const uint8_t* __restrict__ compute, float* __restrict__ opacity) {
  const size_t C1 = (size_t)t.nCells + 1;
  const float* xs = reinterpret_cast<const float*>(t.termXs);
  const int cell = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (cell > t.nCells || !compute[cell] || isfinite(opacity[cell])) return;
  const float Te = te[cell], Ne = ne[cell], H = hden[cell];
  auto density = [&](int s) { return ionDen[(size_t)cell + C1 * (size_t)t.slotPlane[s]] * t.slotAbun[s] * H; };
  float wsum = 0.f;
  for (int s = 0; s < t.nSlots; ++s) wsum += t.slotFFWeight[s] * density(s);
  const float fac1 = (Ne / 1.e10f) * (wsum / 1.e10f) / sqrtf(Te);
  if (!isinf(fac1)) return;
  const float fac2 = fac1 * 1.578866e5f / Te;
  float c[9], con, gamma2;
  gauntCoeffs(0.f, log10f(gauntTe[cell]), c, con, gamma2);
  for (int i = 0; i < t.nbins; ++i) {
    const int g = i / kOpBins, q = i % kOpBins;
    const float ex = 1.578866e5f / Te + t.nu[i];
    const float boltz = ex > 84.f ? 0.f : expf(-ex);
    const float gf = gauntAt(c, con, gamma2, t.log10nu[i]), xb = t.xsec[i + t.bremsP0];
    float op = boltz < 0.995f ? xb * (1.f - boltz) * gf * fac1 : xb * t.nu[i] * gf * fac2;
    for (int e = t.termStart[g]; e < t.termStart[g + 1]; ++e)
      if (t.termOpen[e] >> q & 1) op += xs[(size_t)e * kOpBins + q] * density(t.termSlot[e]);
    if (t.lgCompton) op += t.KNsigmaT[i] * Ne;
    opacity[(size_t)cell + C1 * (size_t)i] = op;
  }
}

cudaError_t launchOpacity(const OpacityDev& t, const float* hden, const float* te, const float* ne,
                          const float* ionDen, const float* gauntTe, const uint8_t* compute, float* opacity,
                          cudaStream_t stream) {
  int threads = kOpThreads;
  auto bytes = [&](int n) { return (size_t)t.nSlots * kOpCells * n * sizeof(float); };
  while (threads > 32 && bytes(threads) > 100 * 1024) threads >>= 1;
  const size_t smem = bytes(threads);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  const int blocks = (t.nCells + threads * kOpCells - 1) / (threads * kOpCells);
  const int groups = (t.nbins + kOpBins - 1) / kOpBins;
  if (smem > 48 * 1024) {
    cudaError_t e = allowSmem(opacityKernel, smem);
    if (e != cudaSuccess) return e;
  }
  // some 24 blocks per SM of the 152: a chunk of high frequencies has several times
  // the open shells of a low one, and with few blocks per SM the last ones run
  // alone (41^3 cells: 0.39 ms with 8, 0.30 with 24)
  const int chunks = std::max(1, std::min((24 * 152 + blocks - 1) / blocks, groups));
  opacityKernel<<<dim3(blocks, chunks), threads, smem, stream>>>(t, hden, te, ne, ionDen, gauntTe, compute, opacity);
  opacityOpenShellsKernel<<<(t.nCells + kOpThreads - 1) / kOpThreads, kOpThreads, 0, stream>>>(
      t, hden, te, ne, ionDen, gauntTe, compute, opacity);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256)
skipMaskKernel(const float* __restrict__ te, const float* __restrict__ ne, const float* __restrict__ teOld,
               const float* __restrict__ neOld, int nCells, bool first, uint8_t* __restrict__ mask,
               unsigned long long* __restrict__ counts) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  bool compute = false;
  if (cell >= 1 && cell <= nCells)
    compute = first || !((fabsf(te[cell] - teOld[cell]) / teOld[cell]) < 0.005f &&
                         (fabsf(ne[cell] - neOld[cell]) / neOld[cell]) < 0.005f);
  if (cell <= nCells) mask[cell] = compute ? 1 : 0;
  const int n = __syncthreads_count(compute), all = __syncthreads_count(cell >= 1 && cell <= nCells);
  if (threadIdx.x == 0 && n) atomicAdd(counts, (unsigned long long)n);
  if (threadIdx.x == 0 && all > n) atomicAdd(counts + 1, (unsigned long long)(all - n));
}

cudaError_t launchSkipMask(const float* te, const float* ne, const float* teOld, const float* neOld, int nCells,
                           bool first, uint8_t* mask, unsigned long long* counts, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), stream);
  if (e != cudaSuccess) return e;
  skipMaskKernel<<<(nCells + 1 + 255) / 256, 256, 0, stream>>>(te, ne, teOld, neOld, nCells, first, mask, counts);
  return cudaGetLastError();
}

// The cache is one serial chain over the cells: the temperature changes only at a
// cell more than 10 % away from it, and two chains that differ soon meet a cell
// that sets both to the same.  So a lane runs kReplayChunk cells from the
// temperature that the kReplayLead chunks before them lead to, from an assumed
// one (gauntChunksKernel, a warp's cells staged through shared memory), and then
// one block per grid checks what each chunk started with (gauntReplayKernel): a
// chunk either passes its temperature on or ends with one of its own, so it
// really starts with the end of the nearest earlier chunk that has one.  Those that
// started with another run again up to where they meet what they stored, a few
// rounds side by side and then, in order, one after another.  41^3 cells: 0.4 ms as a
// serial chain on the host, 0.11 with a chunk of all cells per thread of one block
// (bound by what one SM loads), 0.023 now; a 19^3 sphere, whose smooth temperatures
// make the chains slow to meet, 0.041 and 0.038 (0.054 with one chunk of lead, 0.050 with seven).
constexpr int kReplayChunk = 32, kReplayLead = 3, kReplayThreads = 1024, kReplayWarps = 4, kReplayRounds = 6;
constexpr unsigned kReplayOff = 0xffffffffu;     // a cell without its mask: a NaN that no temperature is stored as

// chunk states: what it started with, what it ended with, whether that is its own
struct ReplayChunks { float* in; float* out; uint8_t* own; };
__device__ __forceinline__ ReplayChunks replayChunks(float* scratch, int nChunks, int first, int grid) {
  const int at = first / kReplayChunk + grid;
  return {scratch + at, scratch + nChunks + at, reinterpret_cast<uint8_t*>(scratch + 2 * (size_t)nChunks) + at};
}

__global__ void __launch_bounds__(32 * kReplayWarps)
gauntChunksKernel(const float* __restrict__ te, const uint8_t* __restrict__ mask, const int32_t* __restrict__ order,
                  const int32_t* __restrict__ gridOff, int nOrdered, int nChunks, const float* __restrict__ state,
                  float* __restrict__ scratch, float* __restrict__ gauntTe) {
  constexpr int kRows = 32 + kReplayLead;
  __shared__ float sT[kReplayWarps][kRows][33];   // the warp's chunks and those before them
  const int first = gridOff ? gridOff[blockIdx.y] : 0, last = gridOff ? gridOff[blockIdx.y + 1] : nOrdered;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int at = first + (blockIdx.x * kReplayWarps + warp) * 32 * kReplayChunk;   // the warp's first cell
  if (at >= last) return;
  float (*t)[33] = sT[warp];
#pragma unroll 12
  for (int r = 0; r < kRows; ++r) {              // every load in flight, in range or not
    const int i = at + (r - kReplayLead) * kReplayChunk + lane;
    const bool here = i >= first && i < last;
    const int k = here ? i : first, cell = order ? order[k] : k + 1;
    const bool on = mask[cell] != 0;
    unsigned x = __float_as_uint(te[cell]);
    if (x == kReplayOff) x = 0x7fffffffu;
    t[r][lane] = __uint_as_float(here && on ? x : kReplayOff);
  }
  __syncwarp();
  const float start = state[blockIdx.y];
  const int j = (at - first) / kReplayChunk + lane;   // this lane's chunk
  float cur = start;
  bool known = j <= kReplayLead;                       // the first ones follow from the state itself
  for (int k = 0; k < kReplayLead * kReplayChunk; ++k) {
    const float x = t[lane + k / kReplayChunk][k % kReplayChunk];
    if (__float_as_uint(x) == kReplayOff) continue;
    if (!known || fabsf(1.f - cur / x) > 0.10f) { cur = x; known = true; }
  }
  __syncwarp();
  const float in = cur;
  bool own = false;
  for (int k = 0; k < kReplayChunk; ++k) {
    const float x = t[lane + kReplayLead][k];
    const bool on = __float_as_uint(x) != kReplayOff;
    if (on && fabsf(1.f - cur / x) > 0.10f) { cur = x; own = true; }
    t[lane + kReplayLead][k] = on ? cur : 0.f;
  }
  if (first + j * kReplayChunk < last) {
    const ReplayChunks c = replayChunks(scratch, nChunks, first, blockIdx.y);
    c.in[j] = in;
    c.out[j] = cur;
    c.own[j] = own ? 1 : 0;
  }
  __syncwarp();
  for (int r = kReplayLead; r < kRows; ++r) {
    const int i = at + (r - kReplayLead) * kReplayChunk + lane;
    if (i < last) gauntTe[order ? order[i] : i + 1] = t[r][lane];
  }
}

__global__ void __launch_bounds__(kReplayThreads)
gauntReplayKernel(const float* __restrict__ te, const uint8_t* __restrict__ mask, const int32_t* __restrict__ order,
                  const int32_t* __restrict__ gridOff, int nOrdered, int nChunks, float* __restrict__ state,
                  float* scratch, float* gauntTe) {
  __shared__ int sLast[kReplayThreads / 32];
  const int first = gridOff ? gridOff[blockIdx.x] : 0, last = gridOff ? gridOff[blockIdx.x + 1] : nOrdered;
  const int n = (last - first + kReplayChunk - 1) / kReplayChunk;
  const int per = (n + kReplayThreads - 1) / kReplayThreads;
  const int lo = min((int)threadIdx.x * per, n), hi = min(lo + per, n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const ReplayChunks c = replayChunks(scratch, nChunks, first, blockIdx.x);
  const float start = state[blockIdx.x];
  // chunk j from `in`, up to where it meets what it stored
  auto run = [&](int j, float in) {
    float t = in;
    bool own = false;
    const int i1 = min(first + (j + 1) * kReplayChunk, last);
    for (int i0 = first + j * kReplayChunk; i0 < i1; i0 += 8) {
      int cell[8];
      float x[8], was[8];
      bool on[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {                   // eight cells' loads in flight
        const int i = min(i0 + u, i1 - 1);
        cell[u] = order ? order[i] : i + 1;
        x[u] = te[cell[u]];
        was[u] = gauntTe[cell[u]];
        on[u] = i0 + u < i1 && mask[cell[u]];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (!on[u]) continue;
        if (fabsf(1.f - t / x[u]) > 0.10f) { t = x[u]; own = true; }
        if (__float_as_uint(was[u]) == __float_as_uint(t)) {   // the rest is as it was, the end too
          c.in[j] = in;
          if (own) c.own[j] = 1;
          return;
        }
        gauntTe[cell[u]] = t;
      }
    }
    c.in[j] = in;
    c.out[j] = t;
    c.own[j] = own ? 1 : 0;
  };
  bool settled = false;
  for (int round = 0; round < kReplayRounds && !settled; ++round) {
    int j = -1;                                       // the last of this thread's chunks with a temperature of its own
    for (int k = lo; k < hi; ++k)
      if (c.own[k]) j = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, j, o);
      if (lane >= o) j = max(j, up);
    }
    if (lane == 31) sLast[warp] = j;
    __syncthreads();
    int before = __shfl_up_sync(0xffffffffu, j, 1);
    if (lane == 0) before = -1;
    for (int w = 0; w < warp; ++w) before = max(before, sLast[w]);
    float real = before < 0 ? start : c.out[before];
    __syncthreads();                                  // every end read before any changes
    bool wrong = false;
    for (int k = lo; k < hi; ++k) {
      if (__float_as_uint(real) != __float_as_uint(c.in[k])) {
        run(k, real);
        wrong = true;
      }
      if (c.own[k]) real = c.out[k];
    }
    settled = !__syncthreads_or(wrong);
  }
  if (threadIdx.x == 0) {
    float t = start;
    if (settled) {
      if (n > 0) t = c.out[n - 1];
    } else {
      for (int k = 0; k < n; ++k) {
        if (__float_as_uint(t) != __float_as_uint(c.in[k])) run(k, t);
        t = c.out[k];
      }
    }
    state[blockIdx.x] = t;
  }
}

int gauntReplayChunks(int nGrids, int nOrdered) { return nOrdered / kReplayChunk + nGrids + 1; }

cudaError_t launchGauntReplay(const float* te, const uint8_t* mask, const int32_t* order, const int32_t* gridOff,
                              int nGrids, int nOrdered, float* state, float* scratch, float* gauntTe,
                              cudaStream_t stream) {
  const int nChunks = gauntReplayChunks(nGrids, nOrdered), perBlock = kReplayWarps * 32 * kReplayChunk;
  gauntChunksKernel<<<dim3(std::max(1, (nOrdered + perBlock - 1) / perBlock), nGrids), 32 * kReplayWarps, 0, stream>>>(
      te, mask, order, gridOff, nOrdered, nChunks, state, scratch, gauntTe);
  gauntReplayKernel<<<nGrids, kReplayThreads, 0, stream>>>(te, mask, order, gridOff, nOrdered, nChunks, state, scratch,
                                                           gauntTe);
  return cudaGetLastError();
}

}  // namespace mcx
