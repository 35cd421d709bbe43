// k_emission.cu - the emission phase for every gas cell at once.
//
// Restates emissionDriver / fb_ff / twoPhoton / RecLinesEmission /
// setDiffusePDF (source/emission_mod.f90:36-252, :336-1151, :1528-1919) for gas
// without dust.  A lane has one cell, so the store recPDF[nu][cell] of a warp is one
// coalesced row segment, and the warps of a block share out the bins; the cumulative
// sum is taken in the reference's order and precision (REAL partial sums).
// Everything that depends only on the frequency mesh (Milne-relation
// prefactors, heavy-ion cross sections times g0/g1, two-photon spectral shapes,
// the gamma-edge pair covering each bin) is tabulated once on the host in FP64
// and stored in FP32, so the per-cell work is FP32 exponentials and FMAs.
#include "k_emission.cuh"
#include "mcx_device.cuh"

#include "k_gaunt.cuh"
#include "setup_internal.h"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

namespace mcx {

namespace {

constexpr double kPi = 3.141592654;
constexpr double kHcRyd_k = 157893.94, kHcRyd = 2.1799153e-11, kCRyd = 3.2898423e15, kHPlanck = 6.6262e-27;

template <typename T>
cudaError_t up(EmissionData& d, const std::vector<T>& v, const T** out) {
  void* p = nullptr;
  size_t n = v.empty() ? sizeof(T) : v.size() * sizeof(T);
  cudaError_t e = cudaMalloc(&p, n);
  if (e != cudaSuccess) return e;
  d.blocks[d.nBlocks++] = p;
  if (!v.empty()) e = cudaMemcpy(p, v.data(), n, cudaMemcpyHostToDevice);
  *out = static_cast<const T*>(p);
  return e;
}

}  // namespace

EmissionData::~EmissionData() {
  for (int i = 0; i < nBlocks; ++i) cudaFree(blocks[i]);
}

std::string emissionDataCreate(const Setup& s, std::unique_ptr<EmissionData>& out) {
  auto d = std::make_unique<EmissionData>();
  EmissionDev& e = d->dev;
  const EmissionTables& em = s.em;
  const int nb = s.nbins;
  const int E = std::max(s.nElemUsed, 1);
  e.nbins = nb; e.nCells = s.nCells; e.nstages = s.p.nstages; e.nElemUsed = E; e.nTk = em.nTk;
  for (int k = 0; k < 3; ++k) e.nlim[k] = em.nlim[k];
  e.nHydroFiles = em.nHydroFiles;
  e.HIPnuP = s.HlevNuP[0]; e.HeIPnuP = s.HeIlevNuP[0]; e.HeIIPnuP = s.HeIIlevNuP[0];
  const int HeIlast = em.edgeP[32 + em.nlim[1] - 1], HeIIlast = em.edgeP[64 + em.nlim[2] - 1];
  e.HeIlast = std::max(e.HIPnuP, HeIlast);                 // Milne HeI from here
  e.HeIIlast = std::max(e.HeIlast, HeIIlast);              // Milne HeII from here
  e.j2TsP = em.j2TsP;
  for (int k = 0; k < 4; ++k) e.HeIILymanP[k] = em.HeIILymanP[k];
  e.xrefH = s.elemXref[0]; e.xrefHe = s.elemXref[1];
  e.abunH = s.elemAbun[0]; e.abunHe = s.elemAbun[1];
  e.nuHIP = s.nu[e.HIPnuP - 1]; e.nuHeIP = s.nu[e.HeIPnuP - 1]; e.nuHeIIP = s.nu[e.HeIIPnuP - 1];

  std::vector<float> cw(nb), milne((size_t)3 * nb, 0.f), fbK(nb), t2H(nb, 0.f), t2HeII(nb, 0.f), t2HeI(nb, 0.f);
  std::vector<int16_t> pair((size_t)3 * nb, 0);
  for (int k = 0; k < 3; ++k)
    for (int p = 1; p <= em.nlim[k] / 2; ++p) {
      int iup = em.edgeP[k * 32 + 2 * p - 1], ilow = em.edgeP[k * 32 + 2 * p - 2];
      if (iup == ilow) return "fb_ff: frequency grid too coarse - divide by zero";
      for (int j = ilow; j <= iup - 1; ++j) pair[(size_t)k * nb + (j - 1)] = (int16_t)p;
    }
  const double constant = 4.9874105e-6;
  auto xsAt = [&](int xi) -> double { return (xi >= 1 && xi <= (int)s.xSec.size()) ? (double)s.xSec[xi - 1] : 0.; };
  for (int i = 1; i <= nb; ++i) {
    const double v = s.nu[i - 1], v3 = v * v * v;
    cw[i - 1] = (float)(kCRyd * (double)s.widFlx[i - 1] / 1.e15);
    fbK[i - 1] = (float)(4. * kPi * constant * kHcRyd * v3 * 1e20 * 1e20);
    if (i >= e.HIPnuP)
      milne[i - 1] = (float)(4. * kPi * xsAt(i - e.HIPnuP + 1 + s.HlevXSecP[0] - 1) * 2. * kHcRyd * constant * v3 * 1e20 * 1e20);
    if (i >= e.HeIlast)
      milne[nb + i - 1] = (float)(4. * kPi * xsAt(i - e.HeIPnuP + 1 + s.HeISingXSecP[0] - 1) * 0.5 * kHcRyd * constant * v3 * 1e20 * 1e20);
    if (i >= e.HeIIlast)
      milne[2 * nb + i - 1] = (float)(4. * kPi * xsAt(i - e.HeIIPnuP + 1 + s.HeIIXSecP[0] - 1) * 2. * kHcRyd * constant * v3 * 1e20 * 1e20);
    // hydro2phot spectral shapes (source/emission_mod.f90:660-726)
    if (v < 0.7496) {
      double y = v / 0.7496;
      double Ay = 202.0 * (y * (1 - y) * (1 - pow(4 * y * (1 - y), 0.8)) + 0.88 * pow(y * (1 - y), 1.53) * pow(4 * y * (1 - y), 0.8));
      t2H[i - 1] = (float)(kHPlanck * y * Ay / 8.2249 * 1e27);
    }
    if (v < 3.0) {
      double y = v / 3.0;
      double Ay = 64. * 0.9994667 * 202.0 * (y * (1 - y) * (1 - pow(4 * y * (1 - y), 0.8)) + 0.88 * pow(y * (1 - y), 1.53) * pow(4 * y * (1 - y), 0.8));
      t2HeII[i - 1] = (float)(kHPlanck * y * Ay / (8.226 * 64.) * 1e27);
    }
  }
  {  // HeI2photSub's table walk (source/emission_mod.f90:762-778), cell independent
    int j = 1;
    for (int i = 1; i <= nb; ++i) {
      double y = (double)s.nu[i - 1] / 1.514;
      if (y > (double)em.HeI2phot[0][j - 1]) j = j + 1;
      if (j >= 41) break;
      double fit1 = ((double)em.HeI2phot[1][j] - (double)em.HeI2phot[1][j - 1]) / ((double)em.HeI2phot[0][j] - (double)em.HeI2phot[0][j - 1]);
      double fit2 = (double)em.HeI2phot[1][j - 1] - (double)em.HeI2phot[0][j - 1] * fit1;
      double Ay = fit1 * y + fit2;
      if (Ay < 9.2163086E-03) Ay = 0.;
      t2HeI[i - 1] = (float)(Ay * 0.66262 * y / 51.3);
    }
  }
  // heavy free-bound CSR in the reference's summation order (element, ion)
  std::vector<int32_t> fbStart(nb + 1, 0);
  std::vector<FbTerm> fbTerm;
  std::vector<int32_t> fbPlane;
  const size_t nt = em.fbHeavy.size() / 7;
  for (int i = 1; i <= nb; ++i) {
    fbStart[i - 1] = (int32_t)fbTerm.size();
    for (size_t t = 0; t < nt; ++t) {
      const int32_t* T = &em.fbHeavy[7 * t];
      int elem = T[0], ion = T[1], IPnuP = T[2], highNuP = T[3], xSecP = T[4], g0 = T[5], g1 = T[6];
      if (i >= IPnuP && i < highNuP) {
        FbTerm f;
        f.xsg = (float)(xsAt(i + xSecP - IPnuP + 1 - 1) * ((double)g0 / (double)g1));
        f.dNu = s.nu[IPnuP - 1] - s.nu[i - 1];
        f.abun = s.elemAbun[elem - 1];
        const int32_t plane = (s.elemXref[elem - 1] - 1) + E * ion;   // stage ion+1
        f.slot = (int32_t)(std::find(fbPlane.begin(), fbPlane.end(), plane) - fbPlane.begin());
        if (f.slot == (int32_t)fbPlane.size()) fbPlane.push_back(plane);
        fbTerm.push_back(f);
      }
    }
  }
  fbStart[nb] = (int32_t)fbTerm.size();
  std::vector<float> fbMax(nb, 0.f);
  for (int i = 0; i < nb; ++i)
    for (int t = fbStart[i]; t < fbStart[i + 1]; ++t) fbMax[i] = t == fbStart[i] ? fbTerm[t].dNu : std::max(fbMax[i], fbTerm[t].dNu);
  e.nFbSlots = (int32_t)fbPlane.size();
  std::vector<int32_t> xrefAll(s.elemXref, s.elemXref + kNElements);
  std::vector<float> abunAll(s.elemAbun, s.elemAbun + kNElements);
  std::vector<int8_t> hOn(31, 0);
  for (int izp = 1; izp <= 30; ++izp) hOn[izp] = (s.elemOn[izp - 1] && s.p.nstages > izp) ? 1 : 0;
  std::vector<float> ffK((size_t)2 * nb, 0.f);
  std::vector<float> hb(72), rb(156), r2a(54), heiRec(408), ly(4), temps(12);
  for (int a = 0; a < 2; ++a) for (int i = 0; i < 9; ++i) for (int j = 0; j < 4; ++j) hb[(a * 9 + i) * 4 + j] = em.HbCoeff[a][i][j];
  for (int a = 0; a < 2; ++a) for (int j = 0; j < 3; ++j) for (int i = 0; i < 26; ++i) rb[(a * 3 + j) * 26 + i] = em.rbEdge[a][j][i];
  for (int j = 0; j < 3; ++j) for (int i = 0; i < 18; ++i) r2a[j * 18 + i] = em.r2aEdge[j][i];
  for (int l = 0; l < 34; ++l) for (int d2 = 0; d2 < 3; ++d2) for (int k = 0; k < 4; ++k) heiRec[(l * 3 + d2) * 4 + k] = em.HeIrec[l][d2][k];
  for (int k = 0; k < 4; ++k) ly[k] = em.HeIILyman[0][k];
  for (int k = 0; k < 12; ++k) temps[k] = em.hydroLinesTemps[k];

  cudaError_t err = cudaSuccess;
#define UP(vec, field) if (err == cudaSuccess) err = up(*d, vec, &e.field)
  UP(s.nu, nu); UP(cw, cRydWid); UP(pair, pairIdx); UP(em.edgeP, edgeP); UP(em.tk, tk); UP(em.logGamma, logGamma);
  UP(milne, milne); UP(fbStart, fbStart); UP(fbTerm, fbTerm); UP(fbPlane, fbPlane); UP(fbMax, fbDNuMax); UP(fbK, fbK); UP(t2H, twoPhH); UP(t2HeII, twoPhHeII);
  UP(t2HeI, twoPhHeI); UP(ly, heiiLyman); UP(em.hydroFileMap, hydroMap); UP(em.hydroDens, hydroDens);
  UP(em.hydroLines, hydroLines); UP(temps, hydroTemps); UP(hb, hbCoeff); UP(rb, rbEdge); UP(r2a, r2aEdge);
  UP(heiRec, heiRec); UP(hOn, hydroOn); UP(xrefAll, xrefAll); UP(abunAll, abunAll);
#undef UP
  if (err == cudaSuccess) {
    const float* fk = nullptr;
    err = up(*d, ffK, &fk);
    e.ffK = const_cast<float*>(fk);
  }
  if (err == cudaSuccess) {
    const float* pp = nullptr;
    err = up(*d, std::vector<float>((size_t)4 * kEmChunksMax * ((size_t)s.nCells + 1), 0.f), &pp);
    e.part = const_cast<float*>(pp);
  }
  if (err != cudaSuccess) return std::string("emission tables: ") + cudaGetErrorString(err);
  out = std::move(d);
  return "";
}

__global__ void emissionGauntKernel(EmissionDev e, float gauntTe) {
  float c0[9], con0, g20, c1[9], con1, g21;
  gauntCoeffs(0.f, log10f(gauntTe), c0, con0, g20);
  gauntCoeffs(0.30103f, log10f(gauntTe), c1, con1, g21);
  const float k = 4.f * 3.141592654f * 54.43f;
  for (int i = threadIdx.x + blockIdx.x * blockDim.x; i < e.nbins; i += blockDim.x * gridDim.x) {
    float l = log10f(e.nu[i]);
    e.ffK[i] = k * 1.f * gauntAt(c0, con0, g20, l);
    e.ffK[e.nbins + i] = k * 4.f * gauntAt(c1, con1, g21, l);
  }
}

cudaError_t launchEmissionGaunt(const EmissionDev& e, float gauntTe, cudaStream_t s) {
  emissionGauntKernel<<<(e.nbins + 255) / 256, 256, 0, s>>>(e, gauntTe);
  return cudaGetLastError();
}

// one table per nebula of a batch: table b (blockIdx.y) at temperature temps[b]
__global__ void emissionGauntBatchKernel(EmissionDev e, const float* __restrict__ temps) {
  const int b = blockIdx.y;
  float c0[9], con0, g20, c1[9], con1, g21;
  gauntCoeffs(0.f, log10f(temps[b]), c0, con0, g20);
  gauntCoeffs(0.30103f, log10f(temps[b]), c1, con1, g21);
  const float k = 4.f * 3.141592654f * 54.43f;
  float* ffK = e.ffK + (size_t)b * 2 * e.nbins;
  for (int i = threadIdx.x + blockIdx.x * blockDim.x; i < e.nbins; i += blockDim.x * gridDim.x) {
    float l = log10f(e.nu[i]);
    ffK[i] = k * 1.f * gauntAt(c0, con0, g20, l);
    ffK[e.nbins + i] = k * 4.f * gauntAt(c1, con1, g21, l);
  }
}

cudaError_t launchEmissionGauntBatched(const EmissionDev& e, const float* temps, int nTables, cudaStream_t s) {
  if (nTables <= 0) return cudaSuccess;
  emissionGauntBatchKernel<<<dim3((e.nbins + 255) / 256, nTables), 256, 0, s>>>(e, temps);
  return cudaGetLastError();
}

namespace {

__device__ __forceinline__ float ionFrac(const float* ionDen, size_t C1, size_t cell, int xref, int E, int stage,
                                         int nstages) {
  if (xref <= 0 || stage < 1 || stage > nstages) return 0.f;
  return ionDen[cell + C1 * (size_t)((xref - 1) + E * (stage - 1))];
}

// locate on an ascending float array (source/interpolation_mod.f90:49-106)
__device__ __forceinline__ int locateF(const float* xa, int n, float x) {
  if (x > xa[n - 1]) return n;
  if (x < xa[0]) return 0;
  int jlow = 0, jup = n + 1;
  for (int it = 0; it < 64; ++it) {
    if (jup - jlow < 1) break;
    int jm = (jup + jlow) >> 1;
    if (xa[jm - 1] == x) return jm;
    if (x > xa[jm - 1]) { if (jlow == jm) break; jlow = jm; } else jup = jm;
  }
  return jlow;
}

}  // namespace

// The emission phase in three kernels.  emissionCdfKernel: each chunk's
// cumulative sums from 0 into recPDF and its totals (the chunk's sum and its HI,
// HeI, HeII parts) into part[4][nChunks][C+1].  emissionLinesKernel: the
// chunks' offsets and norms, the recombination lines and totalLines.
// emissionNormaliseKernel: the offsets added, the distribution normalised and
// written in both layouts.
//
// The sums over a cell's bins are one serial FP32 chain per chunk, but the
// emissivities they add (some 450 instructions a bin, exponentials mostly) are
// independent: a block holds 32 cells, one per lane, and kWarps warps that work
// out two bins each of a tile of 2 kWarps; then four of the warps continue the
// four sums over the tile, in order.  A thread walking its cell's whole chunk
// left 18 warps per SM and took 0.95 ms at 41^3 cells x 600 bins; 0.65 ms now, eight blocks a SM.
// kWarps: 4 where the cells and chunks fill the GPU (the four sums then keep every
// warp busy), 16 on small grids or with a single chunk.
constexpr int kEmCells = 32, kEmBinsPerWarp = 2;
constexpr float kNoExp = -110.f;   // expf is 0 here and below; 0 times a density that is not finite is no zero

template <int kWarps>
__global__ void __launch_bounds__(32 * kWarps, kWarps == 4 ? 8 : 1)
emissionCdfKernel(EmissionDev e, const float* __restrict__ te, const float* __restrict__ ne,
                  const float* __restrict__ ionDen, const uint8_t* __restrict__ compute, float* __restrict__ recPDF,
                  float* __restrict__ part, int nChunks) {
  constexpr int kTile = kEmBinsPerWarp * kWarps;
  extern __shared__ float sm[];
  float* sIon = sm;                                        // [nFbSlots][32]
  float* sSum = sm + (size_t)e.nFbSlots * kEmCells;        // [2][4][kTile][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cellAt = blockIdx.x * kEmCells + lane + 1;
  const bool valid = cellAt <= e.nCells && compute[cellAt];
  if (!__any_sync(0xffffffffu, valid)) return;             // the same cells in every warp
  const size_t C1 = (size_t)e.nCells + 1;
  const int cell = valid ? cellAt : 0;
  bool odd = false;
  for (int t = warp; t < e.nFbSlots; t += kWarps) {
    const float x = ionDen[(size_t)cell + C1 * (size_t)e.fbPlane[t]];
    sIon[t * kEmCells + lane] = x;
    odd = odd || !(fabsf(x) <= FLT_MAX);
  }
  const float noExp = __syncthreads_or(odd) ? -INFINITY : kNoExp;
  const int nb = e.nbins, E = e.nElemUsed, S = e.nstages;
  const float* ffK = e.ffK + (e.ffIdx ? (size_t)e.ffIdx[cell] * 2 * (size_t)nb : (size_t)0);
  const float Te = te[cell], NeCell = ne[cell];
  float Ne = NeCell;
  const float sqrTe = sqrtf(Te), log10Te = log10f(Te);
  if (Ne < 1.e-5f) Ne = 1.e-5f;
  const float invTe15 = 1.f / (Te * sqrTe);
  const float hk = 157893.94f / Te;

  // gamma(T) interpolation in log-log (fb_ff, source/emission_mod.f90:388-424)
  int nT = 0;
  float tfac = 0.f, tden = 1.f;
  int tmode;   // 0 below, 1 above, 2 interpolate
  if (Te <= e.tk[0]) tmode = 0;
  else if (Te >= e.tk[e.nTk - 1]) tmode = 1;
  else { tmode = 2; nT = locateF(e.tk, e.nTk, Te); tfac = log10f(Te / e.tk[nT - 1]); tden = log10f(e.tk[nT] / e.tk[nT - 1]); }
  auto logG = [&](int k, int idx1) -> float {   // 1-based edge index
    const float* lg = e.logGamma + (size_t)k * e.nTk * 32;
    if (tmode == 0) return lg[idx1 - 1];
    if (tmode == 1) return lg[(size_t)(e.nTk - 1) * 32 + idx1 - 1];
    float a = lg[(size_t)(nT - 1) * 32 + idx1 - 1], b = lg[(size_t)nT * 32 + idx1 - 1];
    return a + (b - a) / tden * tfac;
  };

  // two-photon temperature/density factors (hydro2phot, HeI2photSub)
  float Q;
  if (Te <= 10000.f) Q = 5.31e-4f;
  else if (Te >= 20000.f) Q = 4.71e-4f;
  else Q = exp10f(log10f(5.31e-4f) + (log10f(4.71e-4f / 5.31e-4f) / log10f(2.f)) * log10f(Te / 10000.f));
  const float fH2 = 0.8368f * powf(Te * 1.e-4f, -0.723f) / (1.f + (Ne * Q) / 8.23f);
  float aHeII;
  if (Te <= 5000.f) aHeII = 6.161f;
  else if (Te >= 30000.f) aHeII = 2.035f;
  else if (Te <= 10000.f) aHeII = exp10f(log10f(6.161f) + log10f(4.091f / 6.161f) / log10f(2.f) * log10f(Te / 5000.f));
  else if (Te <= 15000.f) aHeII = exp10f(log10f(4.091f) + log10f(3.189f / 4.091f) / log10f(1.5f) * log10f(Te / 10000.f));
  else aHeII = exp10f(log10f(3.189f) + log10f(2.035f / 3.189f) / log10f(2.f) * log10f(Te / 15000.f));
  const float aHeI = 6.23f * powf(Te / 10000.f, -0.827f);

  const float xH2 = ionFrac(ionDen, C1, cell, e.xrefH, E, 2, S);
  const float xHe2 = ionFrac(ionDen, C1, cell, e.xrefHe, E, 2, S);
  const float xHe3 = ionFrac(ionDen, C1, cell, e.xrefHe, E, 3, S);
  const float wH = e.abunH * xH2 * Ne, wHe2 = e.abunHe * xHe2 * Ne, wHe3 = e.abunHe * xHe3 * Ne;

  // lines added to the partial sums of setDiffusePDF (source/emission_mod.f90:1617-1668)
  const float T4 = Te * 1.e-4f;
  const float corrHeI = 27.2f * powf(T4, -0.678f) * Ne * e.abunHe * xHe2 * 1.45673f * 2.1799153e-11f * 1e11f;
  const float lyA = exp10f(-0.792f * log10Te + 6.01f) * Ne * xHe3 * e.abunHe;

  const int chunkLen = (nb + nChunks - 1) / nChunks;
  const int q = blockIdx.y;
  const int i0 = 1 + q * chunkLen, i1 = min(nb, (q + 1) * chunkLen);
  int gP[3] = {0, 0, 0};
  float gL2[3] = {0.f, 0.f, 0.f}, gA[3] = {0.f, 0.f, 0.f}, gNu[3] = {0.f, 0.f, 0.f};
  float acc = 0.f;                                          // this warp's sum (warps 0 .. 3)
  for (int t0 = i0, buf = 0; t0 <= i1; t0 += kTile, buf ^= 1) {
  float* sT = sSum + (size_t)buf * 4 * kTile * kEmCells + lane;
#pragma unroll
  for (int u = 0; u < kEmBinsPerWarp; ++u) {
    const int b = warp * kEmBinsPerWarp + u, i = t0 + b;
    if (i > i1) break;
    const float v = e.nu[i - 1];
    float gHI = 0.f, gHeI = 0.f, gHeII = 0.f;
    float g[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      int p = e.pairIdx[(size_t)k * nb + (i - 1)];
      if (p > 0) {
        if (p != gP[k]) {   // a new edge pair: its fit, kept for the following bins of the pair
          int iup = e.edgeP[k * 32 + 2 * p - 1], ilow = e.edgeP[k * 32 + 2 * p - 2];
          float l2 = logG(k, 2 * p), l1 = logG(k, 2 * p - 1);
          gP[k] = p;
          gL2[k] = l2;
          gA[k] = (l2 - l1) / (e.nu[iup - 1] - e.nu[ilow - 1]);
          gNu[k] = e.nu[iup - 1];
        }
        g[k] = exp10f(gL2[k] + gA[k] * (v - gNu[k]));
      }
    }
    gHI = g[0]; gHeI = g[1]; gHeII = g[2];
    const float exff = expf(-v * hk) / sqrTe;
    if (i >= e.HIPnuP) {
      gHI = e.milne[i - 1] * invTe15 * expf((e.nuHIP - v) * hk) + ffK[i - 1] * exff;
      if (i >= e.HeIlast) {
        gHeI = e.milne[nb + i - 1] * invTe15 * expf((e.nuHeIP - v) * hk) + ffK[i - 1] * exff;
        if (i >= e.HeIIlast) gHeII = e.milne[2 * nb + i - 1] * invTe15 * expf((e.nuHeIIP - v) * hk) + ffK[nb + i - 1] * exff;
      }
    }
    float hv = 0.f;
    // far above an ion's threshold its exponential is 0 in FP32 (below e^-104):
    // the term adds nothing, and beyond all thresholds none does
    const int t1 = e.fbDNuMax[i - 1] * hk < noExp ? 0 : e.fbStart[i];
    for (int t = e.fbStart[i - 1]; t < t1; ++t) {
      const FbTerm f = e.fbTerm[t];
      if (f.dNu * hk < noExp) continue;
      hv += expf(f.dNu * hk) * f.xsg * sIon[f.slot * kEmCells + lane] * f.abun;
    }
    hv = hv * e.fbK[i - 1] * invTe15;
    float eHI = (gHI + e.twoPhH[i - 1] * fH2) * wH + hv * Ne;
    float eHeI = (gHeI + e.twoPhHeI[i - 1] * aHeI) * wHe2;
    float eHeII = (gHeII + e.twoPhHeII[i - 1] * aHeII) * wHe3;
    if (eHI < 1.e-15f) eHI = 0.f;
    if (eHeI < 1.e-15f) eHeI = 0.f;
    if (eHeII < 1.e-15f) eHeII = 0.f;
    const float cw = e.cRydWid[i - 1];
    float sHI = cw * eHI, sHeI = cw * eHeI, sHeII = cw * eHeII;
    sT[(0 * kTile + b) * kEmCells] = sHI;
    sT[(1 * kTile + b) * kEmCells] = sHeI;
    sT[(2 * kTile + b) * kEmCells] = sHeII;
    if (i == e.j2TsP) sHeI += corrHeI;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i == e.HeIILymanP[k]) sHeII += (k == 3) ? lyA : e.heiiLyman[k] * lyA;
    sT[(3 * kTile + b) * kEmCells] = sHI + sHeI + sHeII;
  }
  __syncthreads();
  // the tile's sums in the bins' order (a buffer is written again only after
  // the next tile's barrier, which follows these reads)
  if (warp < 4) {
    const float* s = sT + warp * kTile * kEmCells;
    const int n = min(kTile, i1 - t0 + 1);
    if (warp < 3) {
      for (int b = 0; b < n; ++b) acc += s[b * kEmCells];
    } else {
      for (int b = 0; b < n; ++b) {
        acc = acc + s[b * kEmCells];
        if (valid) recPDF[(size_t)cell + C1 * (size_t)(t0 + b - 1)] = acc;
      }
    }
  }
  }
  // part 0: the chunk's cumulative sum, 1 .. 3: HI, HeI, HeII
  if (warp < 4 && valid) part[((size_t)(warp == 3 ? 0 : warp + 1) * nChunks + q) * C1 + cell] = acc;
}

// One block per 32 cells, one per lane; the hydrogenic series of the elements and
// the HeI lines are shared out among the warps and added up by the first, in
// the reference's order.
constexpr int kEmLineWarps = 8, kHeILines = 34;
__global__ void __launch_bounds__(32 * kEmLineWarps)
emissionLinesKernel(EmissionDev e, const float* __restrict__ te, const float* __restrict__ ne,
                    const float* __restrict__ ionDen, const uint8_t* __restrict__ compute,
                    const float* __restrict__ forLines, const float* __restrict__ recPDF,
                    float* __restrict__ totalLines, float* __restrict__ part, int nChunks) {
  __shared__ float sL[31][kEmCells], sHb[31][kEmCells], sHe[kHeILines][kEmCells];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cellAt = blockIdx.x * kEmCells + lane + 1;
  const bool valid = cellAt <= e.nCells && compute[cellAt];
  if (!__any_sync(0xffffffffu, valid)) return;
  const size_t C1 = (size_t)e.nCells + 1;
  const int cell = valid ? cellAt : 0;
  const int nb = e.nbins, E = e.nElemUsed, S = e.nstages;
  const float Te = te[cell], NeCell = ne[cell];
  float Ne = NeCell;
  const float log10Te = log10f(Te), log10Ne = log10f(Ne);
  if (Ne < 1.e-5f) Ne = 1.e-5f;
  const float xHe2 = ionFrac(ionDen, C1, cell, e.xrefHe, E, 2, S);
  const float xHe3 = ionFrac(ionDen, C1, cell, e.xrefHe, E, 3, S);
  const float T4 = Te * 1.e-4f;

  // RecLinesEmission: hydrogenic recombination lines (source/emission_mod.f90:878-1085)
  const int elUp = (T4 > e.hydroTemps[11]) ? 2 : 8;
  for (int izp = 1, task = 0; izp <= 30; ++izp) {
    if (!e.hydroOn[izp]) continue;
    if (task++ % kEmLineWarps != warp) continue;
    const bool direct = izp <= elUp;
    const int row = direct ? izp : 2;
    const float scale = direct ? 1.f : 4.f / (float)(izp * izp);
    const float T4u = T4 * scale, Neu = Ne * scale;
    const float log10Neu = direct ? log10Ne : log10f(Ne * scale);
    int itemp = 1;
    for (int k = 1; k <= 12; ++k) if (T4u > e.hydroTemps[k - 1]) itemp = k;
    if (itemp < 12 && T4u > (e.hydroTemps[itemp] + e.hydroTemps[itemp - 1]) / 2.f) itemp = itemp + 1;
    const int f = e.hydroMap[(row - 1) * 12 + (itemp - 1)];
    const float* dens = e.hydroDens + (size_t)f * 13;
    const float* L = e.hydroLines + (size_t)f * 13 * 14 * 8;
    int idenp = 1;
    for (int k = 1; k <= 13; ++k) if (Neu > dens[k - 1] && dens[k - 1] > 0.f) idenp = k;
    const bool interp = (dens[12] > 0.f && idenp < 13) || (dens[12] == 0.f && idenp < 9);
    float sumL = 0.f;
    const float w = interp ? (Neu - dens[idenp - 1]) / (dens[idenp] - dens[idenp - 1]) : 0.f;
    for (int iup = 2; iup <= 15; ++iup)
      for (int ilow = 1; ilow <= (iup - 1 < 8 ? iup - 1 : 8); ++ilow) {
        float a = L[(((size_t)idenp - 1) * 14 + (iup - 2)) * 8 + (ilow - 1)];
        float vline = a;
        if (interp) vline = a + (L[(((size_t)idenp) * 14 + (iup - 2)) * 8 + (ilow - 1)] - a) * w;
        sumL += vline;
      }
    float Hbeta;
    const float* HbA = e.hbCoeff + (size_t)(row - 1) * 4;
    const float* HbB = e.hbCoeff + 36 + (size_t)(row - 1) * 4;
    if (direct) {
      if ((izp == 1 && T4 <= 3.f) || (izp > 1 && T4 <= e.hydroTemps[11])) {
        float zfit = (log10Ne - HbA[1]) / HbA[2];
        float Afit = HbA[0] * expf(-zfit * zfit / 2.f) + HbA[3];
        zfit = (log10Ne - HbB[1]) / HbB[2];
        float Bfit = HbB[0] * expf(-zfit * zfit / 2.f) + HbB[3];
        Hbeta = exp10f(Afit + Bfit * log10Te);
      } else {
        float yy1, yy2, x1, x2;
        const float wN = (idenp < 13) ? (Ne - dens[idenp - 1]) / (dens[idenp] - dens[idenp - 1]) : 0.f;
        if (izp == 1) {
          const float* e3 = e.rbEdge + 2 * 26;
          yy1 = e3[idenp - 1] + ((idenp < 13) ? (e3[idenp - 1] - e3[idenp]) * wN : 0.f);
          yy2 = e3[12 + idenp] + ((idenp < 13) ? (e3[12 + idenp] - e3[13 + idenp]) * wN : 0.f);
          x1 = e.rbEdge[0]; x2 = e.rbEdge[13];
        } else {
          const float* e3 = e.r2aEdge + 2 * 18;
          yy1 = e3[idenp - 1] + ((idenp < 13) ? (e3[idenp - 1] - e3[idenp]) * wN : 0.f);
          // r2aEdge(3, 9+idenp+1) lies past the table for idenp = 9: read as r2aEdge(3,18)
          yy2 = e3[8 + idenp] + ((idenp < 13) ? (e3[8 + idenp] - e3[9 + idenp < 18 ? 9 + idenp : 17]) * wN : 0.f);
          x1 = e.r2aEdge[0]; x2 = e.r2aEdge[9];
        }
        const float xx = log10f(T4 * 1.e4f);
        Hbeta = exp10f(yy1 - (yy1 - yy2) * (xx - x1) / (x2 - x1));
      }
    } else {
      const float log10TeZ = log10f(Te * scale);
      float zfit = (log10Neu - HbA[1]) / HbA[2];
      float Afit = HbA[0] * expf(-zfit * zfit / 2.f) + HbA[3];
      zfit = (log10Neu - HbB[1]) / HbB[2];
      float Bfit = HbB[0] * expf(-zfit * zfit / 2.f) + HbB[3];
      Hbeta = ((float)(izp * izp * izp) / 8.f) * exp10f(Afit + Bfit * log10TeZ);
    }
    const float xion = ionFrac(ionDen, C1, cell, e.xrefAll[izp - 1], E, izp + 1, S);
    Hbeta = Hbeta * Ne * xion * e.abunAll[izp - 1];
    sL[izp][lane] = sumL;
    sHb[izp][lane] = Hbeta;
  }
  // HeI recombination lines (source/emission_mod.f90:1100-1146)
  {
    float T4h = T4;
    if (T4h < 0.5f) T4h = 0.5f;
    if (T4h < 2.0f) T4h = 2.0f;
    int denint;
    if (NeCell <= 100.f) denint = 0;
    else if (NeCell <= 1.e4f) denint = 1;
    else if (NeCell <= 1.e6f) denint = 2;
    else denint = 3;
    for (int l = kEmLineWarps - 1 - warp; l < kHeILines; l += kEmLineWarps) {
      const float* C0 = e.heiRec + (size_t)l * 12;
      float r;
      if (denint > 0 && denint < 3) {
        const float* a = C0 + (denint - 1) * 4;
        const float* b = C0 + denint * 4;
        float x1 = a[0] * powf(T4h, a[1]) * expf(a[2] / T4h);
        float x2 = b[0] * powf(T4h, b[1]) * expf(b[2] / T4h);
        float p0 = exp10f(2.f * (float)denint), p1 = exp10f(2.f * (float)(denint + 1));
        r = x1 + ((x2 - x1) * (Ne - p0) / (p1 - p0));
      } else {
        const float* a = C0 + (denint == 0 ? 0 : 2) * 4;
        r = a[0] * powf(T4h, a[1]) * expf(a[2] / T4h);
      }
      sHe[l][lane] = r;
    }
  }
  __syncthreads();
  if (warp != 0 || !valid) return;
  float normRec = 0.f;
  for (int izp = 1; izp <= 30; ++izp)
    if (e.hydroOn[izp]) normRec += sL[izp][lane] * sHb[izp][lane];
  const float scaleHe = Ne * e.abunHe * xHe2;
  for (int l = 0; l < kHeILines; ++l) normRec += sHe[l][lane] * scaleHe;
  // the chunks' offsets and the norms in chunk order
  const int chunkLen = (nb + nChunks - 1) / nChunks;
  float normHI = 0.f, normHeI = 0.f, normHeII = 0.f, cum = 0.f, offLast = 0.f;
  for (int q = 0; q < nChunks; ++q) {
    float* p0 = part + ((size_t)0 * nChunks + q) * C1 + cell;
    const float sum = *p0;
    *p0 = cum;
    if (q == (nb - 1) / chunkLen) offLast = cum;
    cum = cum + sum;
    normHI += part[((size_t)1 * nChunks + q) * C1 + cell];
    normHeI += part[((size_t)2 * nChunks + q) * C1 + cell];
    normHeII += part[((size_t)3 * nChunks + q) * C1 + cell];
  }
  // the HeI and HeII lines of setDiffusePDF (source/emission_mod.f90:1617-1668)
  const float corrHeI = 27.2f * powf(T4, -0.678f) * Ne * e.abunHe * xHe2 * 1.45673f * 2.1799153e-11f * 1e11f;
  const float lyA = exp10f(-0.792f * log10Te + 6.01f) * Ne * xHe3 * e.abunHe;
  normHeI += corrHeI;
  normHeII += lyA * (1.f + e.heiiLyman[0] + e.heiiLyman[1] + e.heiiLyman[2]);
  const float tl = normRec + (forLines ? forLines[cell] : 0.f);
  part[((size_t)1 * nChunks) * C1 + cell] = offLast + recPDF[(size_t)cell + C1 * (size_t)(nb - 1)];
  totalLines[cell] = tl / (normHI + normHeI + normHeII + tl);
}

// The cumulative distribution normalised (source/emission_mod.f90:1880-1884),
// each chunk's entries shifted by the chunk's offset first, and written in the
// Fortran layout and, through a tile in shared memory, one row per cell.  Of the cells
// that the skip rule leaves out, the rows as they stand: a caller may have written
// them through mcx_device_ptr.
constexpr int kEmTile = 32;
__global__ void __launch_bounds__(256)
emissionNormaliseKernel(int nCells, int nb, const uint8_t* __restrict__ compute, const float* __restrict__ part, int nChunks,
                        float* __restrict__ recPDF, float* __restrict__ recCDFT) {
  __shared__ float tile[kEmTile][kEmTile + 1];
  const size_t C1 = (size_t)nCells + 1;
  const int chunkLen = (nb + nChunks - 1) / nChunks;
  const int b0 = blockIdx.y * kEmTile, c0 = blockIdx.x * kEmTile;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int cell = c0 + x;
  const int q0 = b0 / chunkLen, next = (q0 + 1) * chunkLen;   // a chunk is no shorter than a tile
  if (cell <= nCells) {
    const bool on = cell >= 1 && compute[cell];
    const float last = on ? part[((size_t)1 * nChunks) * C1 + cell] : 1.f;
#pragma unroll
    for (int r = y; r < kEmTile; r += 8) {
      const int b = b0 + r;
      if (b < nb) {
        const size_t at = (size_t)cell + C1 * (size_t)b;
        float v = recPDF[at];
        if (on) {
          v = b == nb - 1 ? 1.f : (part[(size_t)(b < next ? q0 : q0 + 1) * C1 + cell] + v) / last;
          recPDF[at] = v;
        }
        tile[r][x] = v;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = y; r < kEmTile; r += 8) {
    const int c = c0 + r, b = b0 + x;
    if (c <= nCells && b < nb) recCDFT[(size_t)c * nb + b] = tile[x][r];
  }
}

template <int kWarps>
static cudaError_t launchEmissionCdf(const EmissionDev& e, const float* te, const float* ne, const float* ionDen,
                                     const uint8_t* compute, float* recPDF, int nChunks, cudaStream_t s) {
  const size_t smem = ((size_t)e.nFbSlots + 2 * 4 * kEmBinsPerWarp * kWarps) * kEmCells * sizeof(float);
  cudaError_t err = allowSmem(emissionCdfKernel<kWarps>, smem);
  if (err != cudaSuccess) return err;
  emissionCdfKernel<kWarps><<<dim3((e.nCells + kEmCells - 1) / kEmCells, nChunks), 32 * kWarps, smem, s>>>(
      e, te, ne, ionDen, compute, recPDF, e.part, nChunks);
  return cudaGetLastError();
}

cudaError_t launchEmission(const EmissionDev& e, const float* te, const float* ne, const float* ionDen,
                           const uint8_t* compute, const float* forLines, float* recPDF, float* recCDFT,
                           float* totalLines, bool chunked, cudaStream_t s) {
  // the chunks set the order of the sums, so they go by the grid alone: about
  // eight groups of 128 cells per SM of the 152, each chunk at least 32 bins long
  const int groups = (e.nCells + 127) / 128;
  const int nChunks =
      chunked ? std::max(1, std::min({kEmChunksMax, (8 * 152 + groups - 1) / groups, e.nbins / 32})) : 1;
  const int blocks = (e.nCells + kEmCells - 1) / kEmCells;
  cudaError_t err = (long)blocks * nChunks >= 4 * 152
                        ? launchEmissionCdf<4>(e, te, ne, ionDen, compute, recPDF, nChunks, s)
                        : launchEmissionCdf<16>(e, te, ne, ionDen, compute, recPDF, nChunks, s);
  if (err != cudaSuccess) return err;
  emissionLinesKernel<<<blocks, 32 * kEmLineWarps, 0, s>>>(e, te, ne, ionDen, compute, forLines, recPDF, totalLines,
                                                           e.part, nChunks);
  emissionNormaliseKernel<<<dim3((e.nCells + 1 + kEmTile - 1) / kEmTile, (e.nbins + kEmTile - 1) / kEmTile), 256, 0, s>>>(
      e.nCells, e.nbins, compute, e.part, nChunks, recPDF, recCDFT);
  return cudaGetLastError();
}

}  // namespace mcx
