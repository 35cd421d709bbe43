// k_balance_impl.cuh - device code of the balance phase, compiled twice:
//   k_balance_f64.cu    real = double, --fmad=false: the plain FP64 path that is
//                       checked against the oracle operation by operation; its
//                       exp, log, log10 and pow are the portable routines of
//                       mcx_fmath.h, which the oracle uses too
//   k_balance_mixed.cu  real = float: rates, splines and exponentials in FP32
//                       (the reference's own REAL); the X-iteration loop in
//                       FP32 too (the ionisation ladder on the base-2
//                       logarithms of its products, its normalisation, H/He
//                       ratios and Ne); level populations by FP32 state
//                       reduction (the FP64 LU only for a level without an
//                       exit below it); line cooling read from per-ion cooling
//                       surfaces; only the Te bracketing of the secant step
//                       stays FP64
// The including file defines MCX_BAL_REAL, MCX_BAL_NS and MCX_BAL_EXACT.
//
// Reference routines: updateCell / iterateT (source/update_mod.f90:15-482),
// calcAlpha (:2298-2413), RRbadnell / DRbadnell (:2415-2450), radRecFit
// (:3094-3202), dielectronic (:3204-3305), collisionalIonisation
// (:3552-3582), photoionisation (:3584-3832), compton (:3834-3897),
// getPhotoRates (:3971-4040), ionBalance (:1575-1992), thermBalance
// (:887-1215), forLines (:1221-1262), equilibrium / luSlv
// (source/emission_mod.f90:2505-3106), splint (source/interpolation_mod.f90:286-335).
#include "k_balance.cuh"
#include "k_lines.cuh"
#include "setup_internal.h"
#include "mcx_exact.h"
#include "mcx_fmath.h"

#include <algorithm>
#include <functional>

namespace mcx {
namespace MCX_BAL_NS {

typedef MCX_BAL_REAL real;

#if MCX_BAL_EXACT
// Unqualified exp / log / log10 / pow calls of this namespace resolve here
// (before the global CUDA overloads): the portable routines shared with the
// oracle, so that both round alike and take the same branches.
__host__ __device__ __forceinline__ double exp(double x) { return mcx_fm_exp(x); }
__host__ __device__ __forceinline__ double log(double x) { return mcx_fm_log(x); }
__host__ __device__ __forceinline__ double log10(double x) { return mcx_fm_log10(x); }
__host__ __device__ __forceinline__ double pow(double x, double y) { return mcx_fm_pow(x, y); }
#endif

// a default-REAL constant of the reference, at its single-precision value, in
// the rate precision (RF) or in FP64 (RD)
#define RF(x) ((real)(x##f))
#define RD(x) ((double)(x##f))

__device__ __forceinline__ real kBoltz() { return RF(1.380658e-16); }    // constants_mod.f90:18
__device__ __forceinline__ real kRyd2erg() { return RF(2.1799e-11); }   // constants_mod.f90:20
__device__ __forceinline__ real kHcRyd() { return RF(2.1799153e-11); }  // update_mod.f90:64
__device__ __forceinline__ double kXMax() { return RD(0.99999); }       // constants_mod.f90:57

constexpr int kNE = 30;
// mixed precision: ions with elemAbun * ionDen below this skip the atom solve
// (their forbidden lines carry below 1e-7 of any cell's cooling)
constexpr double kNegligibleIon = 1e-12;

struct CellIdx {
  int cell, C1;
};

// Lanes a cell has in a round of the rates (see ratesOf).
constexpr int kGroup = MCX_BAL_EXACT ? 32 : 8, kCellsPerWarp = 32 / kGroup;

#if !MCX_BAL_EXACT
__device__ CoolAt coolStencil(double te, double ne);
__device__ __forceinline__ float2 surfaceAt(const float* tab, int atom, const CoolAt& a);
#endif
struct Lanes {
  int gl;           // lane within the cell's group
  unsigned mask;    // the group's lanes in the warp
};

__device__ __forceinline__ double& ionAt(const BalanceDev& b, const CellIdx& c, int z, int st) {
  return b.ion[((size_t)(st - 1) * b.nElemUsed + (b.xref[z] - 1)) * c.C1 + c.cell];
}

// ------------------------------------------------------------- rate functions

__device__ real rrBadnell(const BalanceDev& b, real te, int elem, int nel) {
  const float* t = b.RRb;
  auto RB = [&](int k) { return (real)t[((size_t)k * kNE + (elem - 1)) * (kNE + 1) + nel]; };
  real A = RB(0), B = RB(1), T0 = RB(2), T1 = RB(3), Cc = RB(4), T2 = RB(5);
  real bbad = B + Cc * exp(-T2 / te);
  const real h = (real)0.5, one = (real)1.;
  const real p0 = pow(te / T0, h);
  return A / (p0 * pow(one + p0, one - bbad) * pow(one + pow(te / T1, h), one + bbad));
}

// (rTe and teM15: 1 / te and te^-1.5, the same for every ion of a cell)
__device__ real drBadnell(const BalanceDev& b, real te, real rTe, real teM15, int elem, int nel) {
  real dr = 0;
  const float* E = b.DRbE + ((size_t)(elem - 1) * (kNE + 1) + nel) * 9;
  const float* Cc = b.DRbC + ((size_t)(elem - 1) * (kNE + 1) + nel) * 9;
  for (int idr = 0; idr < 9; ++idr) {
    if (Cc[idr] == 0.f && E[idr] >= 0.f) continue;   // most of the nine terms: they add 0
#if MCX_BAL_EXACT
    const real x = eqDivide((real)E[idr], te, rTe);
#else
    const real x = (real)E[idr] / te;
#endif
    if (x < (real)87.) dr = dr + (real)Cc[idr] * exp(-x);
  }
  (void)rTe;
  return dr * teM15;
}

__constant__ float kFeFit[3][10] = {
    {4.33e-10f, 3.91e-10f, 3.49e-10f, 3.16e-10f, 2.96e-10f, 2.59e-10f, 2.24e-10f, 1.91e-10f, 1.68e-10f, 1.46e-10f},
    {0.531f, 0.523f, 0.521f, 0.534f, 0.557f, 0.567f, 0.579f, 0.601f, 0.602f, 0.597f},
    {5.77e-02f, 6.15e-02f, 6.22e-02f, 6.02e-02f, 5.79e-02f, 5.65e-02f, 5.49e-02f, 5.10e-02f, 5.07e-02f, 5.22e-02f}};

__device__ real radRecFit(const BalanceDev& b, real te, int z, int n) {
  const real one = (real)1.;
  if ((n <= 3) || (n == 11) || ((z > 5) && (z < 9)) || (z == 10) || ((z == 26) && (n > 11))) {
    const float* r = b.rnew + ((size_t)(z - 1) * kNE + (n - 1)) * 4;
    real tt = sqrt(te / (real)r[2]);
    return (real)r[0] / (tt * pow(tt + one, one - (real)r[1]) * pow(one + sqrt(te / (real)r[3]), one + (real)r[1]));
  }
  real tt = te * RF(1.e-4);
  if ((z == 26) && (n <= 13))
    return (real)kFeFit[0][n - 4] / pow(tt, (real)kFeFit[1][n - 4] + (real)kFeFit[2][n - 4] * log10(tt));
  const float* r = b.rrec + ((size_t)(z - 1) * kNE + (n - 1)) * 2;
  return (real)r[0] / pow(tt, (real)r[1]);
}

// diRec(elem, ion) of dielectronic: the last row of dielectronic.dat for
// (elem, ion) whose temperature flag applies, or above 6e4 K the last row of
// aldrovandi.dat (the whole diRec array is replaced there).  The row indices
// are found at set-up (dielRow: last row with flag 0 or 1, with flag 0 or 2,
// and the aldrovandi row; -1 none).
__device__ real diRecOf(const BalanceDev& b, real te, int elem, int ion) {
  if (ion > b.nstages || elem < 1 || elem > 30 || ion < 1 || ion > 31) return 0;
  const real one = (real)1.;
  const int16_t* idx = b.dielRow + ((size_t)elem * 32 + ion) * 3;
  if (te > (real)60000.) {
    const int r = idx[2];
    if (r < 0) return 0;
    const float* d = b.aldro + (size_t)r * 6;
    real a = d[2], bb = d[3], t0 = d[4], t1 = d[5];
    return a * pow(te, (real)-1.5) * exp(-t0 / te) * (one + bb * exp(-t1 / te));
  }
  real t = te > (real)1000. ? te / (real)10000. : RF(0.1);
  const int r = te < (real)20000. ? idx[0] : idx[1];
  if (r < 0) return 0;
  const float* d = b.diel + (size_t)r * 8;
  real a = d[2], bb = d[3], cc = d[4], dd = d[5], f = d[6];
  return RF(1e-12) * (a / t + bb + cc * t + dd * (t * t)) * pow(t, (real)-1.5) * exp(-f / t);
}

// calcAlpha of one (element, ion) pair (source/update_mod.f90:2298-2413)
__device__ real alphaOf(const BalanceDev& b, real te, real rTe, real teM15, int elem, int ion) {
  real a;
  if (b.lgBadnell) {
    int nel = elem - ion;
    if (nel <= 11) {
      a = rrBadnell(b, te, elem, nel);
      a = a + drBadnell(b, te, rTe, teM15, elem, nel);
    } else {
      a = radRecFit(b, te, elem, elem - ion + 1);
      real di = diRecOf(b, te, elem, ion);
      if (di == (real)0. && ion < 7 && b.xref[8] > 0) di = diRecOf(b, te, 8, ion);
      a = a + (di > (real)0. ? di : (real)0.);
    }
  } else {
    a = radRecFit(b, te, elem, elem - ion + 1);
    if (elem >= 3) {
      real di = diRecOf(b, te, elem, ion);
      if (di == (real)0. && ion < 7) di = diRecOf(b, te, 8, ion);
      a = a + (di > (real)0. ? di : (real)0.);
    }
  }
  return a;
}

__device__ __forceinline__ real alphaOf(const BalanceDev& b, real te, int elem, int ion) {
  return alphaOf(b, te, (real)1. / te, pow(te, (real)-1.5), elem, ion);
}

#if !MCX_BAL_EXACT
__device__ __forceinline__ void lagrange4(float t, float* w);

// ln alphaTotal of pair k = (e - 1) * nstages + (ion - 1) at the nodes of its
// table, and the jump flags: an interval whose midpoint and quarter points the
// interpolant misses by more than 1e-5 holds a switch of the fits
__global__ void __launch_bounds__(128) alphaTableKernel(BalanceDev b, float* tab) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (i >= kAlphaN) return;
  const int e = k / b.nstages + 1, ion = k % b.nstages + 1;
  const int elem = b.zOf[e];
  const double h = (kAlphaLnT1 - kAlphaLnT0) / (kAlphaN - 1);
  const real a = ion <= min(b.nstages - 1, elem) ? alphaOf(b, (real)exp(kAlphaLnT0 + i * h), elem, ion) : (real)0.;
  tab[(size_t)k * kAlphaN + i] = a > 0.f ? logf(a) : -1.e30f;
}
__global__ void __launch_bounds__(128) alphaJumpKernel(BalanceDev b, const float* tab, uint8_t* jump) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (i >= kAlphaN) return;
  const int e = k / b.nstages + 1, ion = k % b.nstages + 1;
  const int elem = b.zOf[e];
  uint8_t bad = 1;
  if (i >= 1 && i + 2 < kAlphaN && ion <= min(b.nstages - 1, elem)) {
    const float* t = tab + (size_t)k * kAlphaN + (i - 1);
    bad = 0;
    if (t[0] < -1.e29f || t[1] < -1.e29f || t[2] < -1.e29f || t[3] < -1.e29f) bad = 1;
    const double h = (kAlphaLnT1 - kAlphaLnT0) / (kAlphaN - 1);
    for (int q = 1; q <= 3 && !bad; ++q) {
      const float f = 0.25f * q;
      float w[4];
      lagrange4(f, w);
      const float lnA = w[0] * t[0] + w[1] * t[1] + w[2] * t[2] + w[3] * t[3];
      const real ex = alphaOf(b, (real)exp(kAlphaLnT0 + (i + f) * h), elem, ion);
      if (!(ex > 0.f) || fabsf(expf(lnA - logf(ex)) - 1.f) > 1.e-5f) bad = 1;
    }
  }
  jump[(size_t)k * kAlphaN + i] = bad;
}

// alphaTotal of pair k at Te from the table (direct where the table cannot serve)
__device__ __forceinline__ real alphaLookup(const BalanceDev& b, int k, real teR, int elem, int ion) {
  const float s = (logf(teR) - (float)kAlphaLnT0) * (float)((kAlphaN - 1) / (kAlphaLnT1 - kAlphaLnT0));
  const int i = (int)s;
  if (s >= 1.f && i + 2 < kAlphaN && !b.alphaJump[(size_t)k * kAlphaN + i]) {
    const float* t = b.alphaTab + (size_t)k * kAlphaN + (i - 1);
    float w[4];
    lagrange4(s - (float)i, w);
    const float ref = __ldg(t + 1);
    return expf(ref) * expf(w[0] * (__ldg(t) - ref) + w[2] * (__ldg(t + 2) - ref) + w[3] * (__ldg(t + 3) - ref));
  }
  return alphaOf(b, teR, elem, ion);
}
#endif

// chex(z, ion, 1) * 1e-9 without the temperature fit (ionBalance's heavy elements)
__device__ __forceinline__ real chexRaw(const BalanceDev& b, int z, int ion) {
  return (real)b.chex[z * 32 + ion].x * RF(1.e-9);
}
// chex(z, ion, 1) at Te (source/update_mod.f90:1711-1720, :3788-3797)
__device__ real chexFit(const BalanceDev& b, int z, int ion, real te) {
  const float4 x = b.chex[z * 32 + ion];
  real a = (real)x.x * RF(1.e-9);
  real t4 = te / (real)10000.;
  real v = (te < (real)6000. || te > (real)5.e4) ? (real)0.
                                                 : a * pow(t4, (real)x.y) * ((real)1. + (real)x.z * exp((real)x.w * t4));
  return v < (real)0. ? (real)0. : v;
}

__device__ __forceinline__ const int32_t* outerOf(const BalanceDev& b, int z, int nElec) {
  return b.outer + ((size_t)(z - 1) * kNE + (nElec - 1)) * 3;
}

// ------------------------------------------------------ J-only integrals

// The parts of photoionisation / getPhotoRates / compton that depend on J
// alone: the cells that packets reached are marked and listed, the Compton sums
// formed, and J integrated over every shell's cross section.

// v > 0 on the bits (FP64 compares go through the FP64 pipe, two a cycle and SM)
__device__ __forceinline__ bool positive(double v) {
  return (unsigned long long)(__double_as_longlong(v) - 1) < 0x7ff0000000000000ull;
}

__device__ __forceinline__ bool positive(float v) { return v > 0.f; }

// f(i, J(i), table[i + shift - 1]) for i = lo .. hi in order, kAhead bins' loads in
// flight at a time: the sums are serial, the loads need not be.
template <int kAhead, typename FJ, typename F>
__device__ __forceinline__ void overBins(int lo, int hi, FJ J, const float* __restrict__ table, int shift, F f) {
  int i0 = lo;
  for (; i0 + kAhead - 1 <= hi; i0 += kAhead) {
    real v[kAhead];
    float x[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      v[u] = J(i0 + u);
      x[u] = __ldg(table + i0 + u + shift - 1);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) f(i0 + u, v[u], x[u]);
  }
#pragma unroll 4
  for (; i0 <= hi; ++i0) f(i0, J(i0), __ldg(table + i0 + shift - 1));
}

// One of compton's sums over the mesh of a cell whose J at bin i (1-based) is
// J(i): of J, of J / nu, and of the recoil heating of H and He.
template <typename F>
__device__ __forceinline__ real comptonSum(const BalanceDev& b, int which, F J) {
  const float* nu = b.nu;
  real s = 0;
  if (which == 0) {
    overBins<16>(1, b.nbins, J, nu, 0, [&](int, real rf, float) { s = s + rf; });
    return s * kRyd2erg();
  }
  if (which == 1) {
    overBins<16>(1, b.nbins, J, nu, 0, [&](int i, real rf, float nui) {
#if MCX_BAL_EXACT
      s = s + eqDivide(rf, (real)nui, b.rNu[i - 1]);
#else
      s = s + rf / (real)nui;
#endif
    });
    return s;
  }
  const int lo = max((which == 2 ? b.cRecoilHP : b.cRecoilHeP) + 1, 1);
  overBins<16>(lo, b.nbins, J, b.xsecRecoil, 0, [&](int i, real rf, float xs) {
    real energy = RF(2.66e-5) * (real)nu[i - 1] * (real)nu[i - 1] - (which == 2 ? (real)1. : RF(1.8));
    s = s + (real)xs * rf * energy;
  });
  return s;
}

// What J gives shell t: the rate, the heating without and in the
// secondary-ionisation tail.
template <typename F>
__device__ __forceinline__ void shellIntegral(const BalanceDev& b, int t, F J, real& rate, real& heat, real& heatTail) {
  const float* nu = b.nu;
  const float* xs = b.xsec;
  const real hcRyd = kHcRyd();
  const PhotoShell sh = b.shells[t];
  // quotients by hcRyd nu and by nu, in the FP64 build from their reciprocals
#if MCX_BAL_EXACT
  auto overHcNu = [&](real v, int i) { return eqDivide(v, hcRyd * (real)nu[i - 1], b.rHcNu[i - 1]); };
  auto overNu = [&](real v, int i) { return eqDivide(v, (real)nu[i - 1], b.rNu[i - 1]); };
#else
  auto overHcNu = [&](real v, int i) { return v / (hcRyd * (real)nu[i - 1]); };
  auto overNu = [&](real v, int i) { return v / (real)nu[i - 1]; };
#endif
  heatTail = 0;
  if (sh.ipNuP < 1 || sh.ipNuP > b.nbins) {   // threshold outside the mesh
    rate = sh.heavy ? (real)0. : RF(1.e-20);
    heat = 0;
    return;
  }
  if (!sh.heavy) {
    real n1 = RF(1.e-20), h1 = 0;
    const real nuIP = (real)nu[sh.ipNuP - 1];
    overBins<8>(sh.ipNuP, sh.highNuP, J, xs, sh.xsecP - sh.ipNuP, [&](int j, real jj, float xf) {
      const real ph = xf < 1.e-35f ? (real)0. : (real)xf;
      if (positive(jj)) {
        n1 = n1 + overHcNu(jj * ph, j);
        h1 = h1 + overNu(ph * jj * ((real)nu[j - 1] - nuIP), j);
      }
    });
    rate = n1;
    heat = h1;
    return;
  }
  const int nu1P = sh.ipNuP, IPnuP = sh.ipNuP;
  const int iup = min(sh.highNuP, b.nbins);
  const real augerE = hcRyd * (real)nu[nu1P - 1] * (real)sh.yield1;
  real g = 0, h = 0;
  const int top = min(iup, b.secIonP - 1);
  overBins<8>(nu1P + 1, top, J, xs, sh.xsecP - IPnuP, [&](int i, real jj, float xf) {
    if (positive(jj)) {
      const real ph = xf < 1.e-35f ? (real)0. : (real)xf;
      g = g + overHcNu(jj * ph, i);
      h = h + jj * ph;
    }
  });
  h = h - g * augerE;
  const real jIP = J(IPnuP);
  const real ph0 = xs[sh.xsecP - 1];
  g = g + jIP * ph0 / (hcRyd * (real)nu[IPnuP - 1]);
  h = h + jIP * ph0 * (hcRyd * (real)nu[IPnuP - 1] - augerE) / (hcRyd * (real)nu[IPnuP - 1]);
  real gh = 0, hh = 0;
#if MCX_BAL_EXACT
  const int ilow = max(IPnuP + 1, b.secIonP);
  for (int i = ilow; i <= iup; ++i) {
    const real v = jIP * (real)xs[i + sh.xsecP - IPnuP - 1];
    gh = gh + overHcNu(v, i);   // radField(IPnuP), as the reference
    hh = hh + v;
  }
#else
  // the same sums with radField(IPnuP) taken out of them (summed once at set-up)
  gh = jIP * (real)b.shellTail[2 * t];
  hh = jIP * (real)b.shellTail[2 * t + 1];
#endif
  g = g + gh;
  hh = hh - gh * augerE;
  rate = g;
  heat = h;
  heatTail = hh;
}

// The J the kernels below read: the estimators themselves, or in the mixed build
// their FP32 values (the precision they are used in), converted once.
#if MCX_BAL_EXACT
typedef double JReal;
#else
typedef float JReal;

// jste in FP32, and state[c] = 0 for the cells a packet reached (2 before): an
// FP64 conversion goes through the FP64 pipe, and the shells and sums read every
// bin some dozens of times.
constexpr int kJBins = 16;
__global__ void __launch_bounds__(256) jToFloatKernel(BalanceDev b, const double* __restrict__ jste, float* __restrict__ jF) {
  const size_t C1 = (size_t)b.nCells + 1;
  const size_t cell = blockIdx.x * (size_t)blockDim.x + threadIdx.x + 1;
  if (cell >= C1) return;
  const int i0 = blockIdx.y * kJBins;
  bool hit = false;
#pragma unroll
  for (int h = 0; h < kJBins; h += 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = i0 + h + u < b.nbins ? __ldg(jste + (size_t)(i0 + h + u) * C1 + cell) : 0.;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      hit = hit || positive(v[u]);
      if (i0 + h + u < b.nbins) jF[(size_t)(i0 + h + u) * C1 + cell] = (float)v[u];
    }
  }
  if (hit) b.state[cell] = 0;
}
#endif

// The cells reached, one thread per cell (blockIdx.y = 0), and compton's four
// sums, one thread per cell and sum (blockIdx.y = 0 .. 3): a serial chain over
// the mesh each.
__global__ void __launch_bounds__(128) hitComptonKernel(BalanceDev b, const JReal* __restrict__ jste) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x + 1, which = blockIdx.y;
  if (cell > b.nCells) return;
  const int C1 = b.nCells + 1;
  if (which == 0) {
#if MCX_BAL_EXACT
    // any J > 0, eight bins in flight at a time
    bool hit = false;
    for (int i0 = 1; i0 <= b.nbins && !hit; i0 += 8) {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = i0 + k <= b.nbins ? __ldg(jste + (size_t)(i0 + k - 1) * C1 + cell) : 0.;
#pragma unroll
      for (int k = 0; k < 8; ++k) hit = hit || positive(v[k]);
    }
#else
    bool hit = b.state[cell] == 0;
#endif
    if (b.evalMask && !b.evalMask[cell]) hit = false;
    b.state[cell] = hit ? 0 : 2;
    if (hit) b.list[atomicAdd(&b.listCount[0], 1u)] = cell;   // the cells of the first T-iteration
  }
  if (b.lgCompton)
    b.comp[(size_t)which * C1 + cell] =
        comptonSum(b, which, [&](int i) { return (real)__ldg(jste + (size_t)(i - 1) * C1 + cell); });
}

// One thread per (cell, photoionised shell), the shell fastest in the block
// index, so that a warp streams one shell's bins of 32 neighbouring cells' J
// rows and the shells of one block of cells, launched next to each other, read
// them from L2.
__global__ void __launch_bounds__(128) shellIntegralsKernel(BalanceDev b, const JReal* __restrict__ jste) {
  const int t = (int)(blockIdx.x % (unsigned)b.nShellsTot);
  const int cell = (int)(blockIdx.x / (unsigned)b.nShellsTot) * blockDim.x + threadIdx.x + 1;
  if (cell > b.nCells || b.state[cell] == 2) return;
  const int C1 = b.nCells + 1;
  real g, h, hh;
  shellIntegral(b, t, [&](int i) { return (real)__ldg(jste + (size_t)(i - 1) * C1 + cell); }, g, h, hh);
  const size_t o = (size_t)t * C1 + cell;
  b.gam[o] = g;
  b.heatA[o] = h;
  b.heatHi[o] = hh;
}

// Loads the grid state of the cells into the FP64 work arrays.
__global__ void loadStateKernel(BalanceDev b, const float* __restrict__ te, const float* __restrict__ ne,
                                const float* __restrict__ ionDen) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (cell > b.nCells) return;
  const int C1 = b.nCells + 1;
  b.te[cell] = te[cell];
  b.ne[cell] = ne[cell];
  const size_t nI = (size_t)b.nstages * b.nElemUsed;
  for (size_t k = 0; k < nI; ++k) b.ion[k * C1 + cell] = ionDen[k * C1 + cell];
  b.xOld[cell] = b.ion[(size_t)(b.xref[1] - 1) * C1 + cell];
  b.tHigh[cell] = 0.; b.tLow[cell] = 0.; b.resHigh[cell] = 0.; b.resLow[cell] = 0.;
  b.nIterT[cell] = 0;
  b.ibConv[cell] = 1;
  b.side[cell] = 0;
}

// ------------------------------------------------------------ a T-iteration

// The rates of one T-iteration of one cell (calcAlpha, photoionisation,
// collisionalIonisation, compton, ionBalance and the thermBalance terms without
// forLines) on a group of G lanes.  The cell's ionic fractions, recombination,
// collisional and photoionisation rates sit in the group's slice of shared
// memory, so the X-iterations of ionBalance read nothing from global memory.
// What is left is a serial chain per cell (up to 15 X-iterations of a few dozen
// dependent steps, 20 T-iterations), so its latency is what counts on small
// grids and in the last T-iterations, and the (element, ion) pairs are the unit
// of work: they are listed once per block (ElemMeta), and each X-iteration works
// out the ladder terms of every pair of every heavy element at once, one lane
// per pair, before one lane per element multiplies them up.  (One lane per
// element did that before: 26 stages of Fe, each with its Auger sums, in a row.)
// Every sum keeps the reference's order (one lane adds the terms in sequence),
// so the FP64 build matches the sequential code operation for operation.
// G: 32 in the FP64 build (4.2 -> 1.8 ms a T-iteration of 13^3 X-ray
// cells against 8 lanes a cell); in the mixed build by the numbers of pairs and
// cells (cellLanes).
//
// Per-element tables of the used elements, copied to shared memory once per
// block: the lanes of a warp index them by different elements at once, which
// the kernel-parameter (constant) bank would serialise.
struct ElemMeta {
  int32_t* zOf;     // [32] Z of used element e
  int32_t* xref;    // [32] e of Z (0 = off)
  float* abun;      // [32] elemAbun by Z
  int16_t* p0;      // [E][32] first photoionised shell of (e, ion)
  int16_t* nsh;     // [E][32] its number of shells
  int16_t* hFirst;  // [32] the first pair of the h-th heavy element (Z >= 3, in element order)
  int8_t* hE;       // [32] its e
  int8_t* pE;       // [nPairs] e and ion of the pairs ion = 1 .. min(Z, nstages - 1), e by e
  int8_t* pIon;
  int8_t* pH;       // [nPairs] the pair's heavy element
  real* chex;       // [nPairs] chexRaw
  float* augYield;  // the Auger electrons that feed each pair (BalanceDev)
  int16_t* augStart;
  int16_t* augShell;
  int8_t* augFrom;
  int8_t* augHead;
  int8_t* sH;       // [nPairs + 32] heavy element and stage of the ladders' terms, element by element
  int8_t* sSt;
  // mixed build: Ne's terms (stage - 1) abun X, those at (e - 1) nstages + stage - 1 = p mod 8 in the p-th of
  // eight lists; the j-th of list p at 8 j + p
  float* neW;
  int16_t* neAt;    // where X is
  int16_t* neCount; // [8]
  int nPairs, nHeavy;
};
__host__ __device__ inline int neTerms(const BalanceDev& b) { return MCX_BAL_EXACT ? 0 : (b.nElemUsed * b.nstages + 7) / 8 * 8; }

// Bytes of those tables.
__host__ __device__ inline size_t elemMetaBytes(const BalanceDev& b) {
  return (size_t)b.nPairs * 8 + 3 * 32 * 4 + (size_t)b.nAugers * 4 + 2 * (size_t)b.nElemUsed * 32 * 2 + 32 * 2 +
         ((size_t)b.nPairs + 1 + b.nAugers) * 2 + 32 + 3 * (size_t)b.nPairs + 2 * (size_t)b.nAugers +
         (size_t)neTerms(b) * 6 + 8 * 2 + 2 * ((size_t)b.nPairs + 32);
}

// The same in doubles: what precedes the cells' slices in shared memory.  (The two
// builds' tables differ, so each works it out for itself.)
__host__ __device__ inline int metaDoublesOf(const BalanceDev& b) { return (int)((elemMetaBytes(b) + 7) / 8); }

__device__ __forceinline__ ElemMeta loadElemMeta(const BalanceDev& b, void* sm) {
  const int E = b.nElemUsed, ns = b.nstages;
  ElemMeta m;
  m.nPairs = b.nPairs;
  m.chex = reinterpret_cast<real*>(sm);
  m.zOf = reinterpret_cast<int32_t*>(reinterpret_cast<char*>(sm) + (size_t)b.nPairs * 8);
  m.xref = m.zOf + 32;
  m.abun = reinterpret_cast<float*>(m.xref + 32);
  m.augYield = m.abun + 32;
  m.neW = m.augYield + b.nAugers;
  m.neAt = reinterpret_cast<int16_t*>(m.neW + neTerms(b));
  m.neCount = m.neAt + neTerms(b);
  m.p0 = m.neCount + 8;
  m.nsh = m.p0 + E * 32;
  m.hFirst = m.nsh + E * 32;
  m.augStart = m.hFirst + 32;
  m.augShell = m.augStart + b.nPairs + 1;
  m.hE = reinterpret_cast<int8_t*>(m.augShell + b.nAugers);
  m.pE = m.hE + 32;
  m.pIon = m.pE + b.nPairs;
  m.pH = m.pIon + b.nPairs;
  m.augFrom = m.pH + b.nPairs;
  m.augHead = m.augFrom + b.nAugers;
  m.sH = m.augHead + b.nAugers;
  m.sSt = m.sH + b.nPairs + 32;
  for (int i = threadIdx.x; i < 32; i += blockDim.x) {
    m.zOf[i] = i <= 30 ? b.zOf[i] : 0;
    m.xref[i] = i <= 30 ? b.xref[i] : 0;
    m.abun[i] = i <= 30 ? b.abun[i] : 0.f;
  }
  for (int i = threadIdx.x; i < E * 32; i += blockDim.x) {
    m.p0[i] = (int16_t)b.pairShell0[i];
    m.nsh[i] = (int16_t)b.pairNShell[i];
  }
  for (int i = threadIdx.x; i <= b.nPairs; i += blockDim.x) m.augStart[i] = b.augStart[i];
  for (int i = threadIdx.x; i < b.nAugers; i += blockDim.x) {
    m.augYield[i] = b.augYield[i];
    m.augShell[i] = b.augShell[i];
    m.augFrom[i] = b.augFrom[i];
    m.augHead[i] = b.augHead[i];
  }
#if !MCX_BAL_EXACT
  if (threadIdx.x < 8) {
    int j = 0;
    for (int k = threadIdx.x; k < E * ns; k += 8) {
      const int e = k / ns + 1, ion = k % ns + 1, elem = b.zOf[e];
      if (ion < 2 || ion > min(elem + 1, ns)) continue;
      m.neW[8 * j + threadIdx.x] = (float)(ion - 1) * b.abun[elem];
      m.neAt[8 * j + threadIdx.x] = (int16_t)((ion - 1) * E + (e - 1));
      ++j;
    }
    m.neCount[threadIdx.x] = (int16_t)j;
  }
#endif
  int n = 0, nSt = 0;
  m.nHeavy = 0;
  for (int e = 1; e <= E; ++e) {
    const int z = b.zOf[e], top = min(z, ns - 1);
    if (z >= 3) {
      if (threadIdx.x == 0) { m.hFirst[m.nHeavy] = (int16_t)n; m.hE[m.nHeavy] = (int8_t)e; }
      for (int i = threadIdx.x; i <= top; i += blockDim.x) {   // its topI + 1 stages
        m.sH[nSt + i] = (int8_t)m.nHeavy;
        m.sSt[nSt + i] = (int8_t)(i + 1);
      }
      nSt += top + 1;
      ++m.nHeavy;
    }
    for (int i = threadIdx.x; i < top; i += blockDim.x) {
      m.pE[n + i] = (int8_t)e;
      m.pIon[n + i] = (int8_t)(i + 1);
      m.pH[n + i] = (int8_t)(m.nHeavy - 1);
      m.chex[n + i] = chexRaw(b, z, i + 1);
    }
    n += top;
  }
  __syncthreads();
  return m;
}

// In the rate precision: FP64 in the plain build; FP32 in the mixed build,
// whose X-iterations then run without an FP64 instruction (GB300 issues FP64
// at 1/64 of the FP32 rate, and the loop is a long dependent chain).
struct WarpCell {
  real* X;       // [S][E] ionic fractions at (st-1)*E + (e-1), the global ionDen order
  real* AL;      // [pairs] alphaTotal
  real* CC;      // [pairs] collisional ionisation rate coefficient (coll1)
  real* PI;      // [nShellsTot] photoIon(1): rate per shell, with the reverse charge exchange; after
                 // ionBalance the heating per shell
  real* AUG;     // [nAugers] photoIon times the yield; mixed build: summed per stage, at its first entry
  real* S;       // mixed build: [nPairs] the shells' rates summed
  real* LAD;     // per heavy element rows of S+3 (kLadRows): the ladders; later the thermBalance terms
};
#if MCX_BAL_EXACT
constexpr int kLadRows = 4;   // out, inn, 1 / inn, mat
#else
constexpr int kLadRows = 2;   // log2(out / inn) and its running sums, exponentials
#endif

// A cell's slice of shared memory, in values of the rate precision.
__host__ __device__ inline int cellSlice(const BalanceDev& b) {
  const int lad = b.nHeavy * kLadRows * (b.nstages + 3), therm = 4 * b.nElemUsed + b.nPairs;
  return b.nElemUsed * b.nstages + (MCX_BAL_EXACT ? 2 : 3) * b.nPairs + b.nShellsTot + b.nAugers + (lad > therm ? lad : therm);
}

__device__ __forceinline__ WarpCell warpCell(const BalanceDev& b, real* at) {
  WarpCell w;
  w.X = at;
  w.AL = w.X + b.nElemUsed * b.nstages;
  w.CC = w.AL + b.nPairs;
  w.PI = w.CC + b.nPairs;
  w.AUG = w.PI + b.nShellsTot;
  w.S = w.AUG + b.nAugers;
  w.LAD = w.S + (MCX_BAL_EXACT ? 0 : b.nPairs);
  return w;
}

__device__ __forceinline__ real& xAt(const BalanceDev& b, const ElemMeta& m, const WarpCell& w, int z, int st) {
  return w.X[(st - 1) * b.nElemUsed + (m.xref[z] - 1)];
}

// ionBalance (source/update_mod.f90:1575-1992; the recursion as a loop) for
// the group's cell; returns lgConv (uniform across the group).  In the mixed
// build the ladder runs on the logarithms of its products (FP32 cannot hold
// the products themselves).
template <int G>
__device__ bool ionBalance(const BalanceDev& b, const ElemMeta& m, const WarpCell& w, const Lanes& L, double te,
                           double& ne, double hden) {
  const int ns = b.nstages, E = b.nElemUsed;
  const int zH = 1, zHe = 2;
  const bool heOn = m.xref[zHe] > 0;
  const real teR = (real)te;
  // the Te-only terms are the same on every X-iteration (the reference
  // recomputes them on each recursive call)
  real expFact = RF(157893.94) / teR;
  if (expFact > (real)75.) expFact = (real)75.;
  const real collIonH0 = RF(2.75E-16) * teR * sqrt(teR) * (RF(157893.94) / teR + (real)2.) * exp(-expFact);
  const real hdenR = (real)hden;
  real neR = (real)ne;
  // H on the group's first lane, He on its second
  real cxHHe[3] = {0, 0, 0}, piHHe[3] = {0, 0, 0}, alHHe[3] = {0, 0, 0};
  const int myZ = L.gl + 1;
  if (L.gl < 2 && m.xref[myZ]) {
    const int e = m.xref[myZ];
    int p = 0;
    while (m.pE[p] != e && p + 1 < m.nPairs) ++p;
    for (int ion = 1; ion <= min(myZ, ns - 1); ++ion) {
      cxHHe[ion] = chexFit(b, myZ, ion, teR);
      const int outShell = outerOf(b, myZ, myZ - ion + 1)[0];
      piHHe[ion] = w.PI[m.p0[(e - 1) * 32 + (ion - 1)] + outShell - 1];   // the outer shell's photoionisation rate
      alHHe[ion] = w.AL[p + ion - 1];
    }
  }
  const int hFirst = m.nHeavy ? m.hFirst[0] : m.nPairs;   // the heavy elements' pairs are the last ones
  const int ladRow = ns + 3;
  // what stays put over the X-iterations in the ladders' out terms
#if MCX_BAL_EXACT
  for (int c = L.gl; c < b.nAugers; c += G) w.AUG[c] = w.PI[m.augShell[c]] * (real)m.augYield[c];
#else
  // the photoionisation rates summed per ion, the Auger terms per (stage, ion fed), each multiplied by
  // X(stage) / X(ion) in the X-iteration
  for (int k = hFirst + L.gl; k < m.nPairs; k += G) {
    const int e = m.pE[k], ion = m.pIon[k];
    const int p0 = m.p0[(e - 1) * 32 + (ion - 1)], nsh = m.nsh[(e - 1) * 32 + (ion - 1)];
    real s = 0;
    for (int q = 0; q < nsh; ++q) s = s + w.PI[p0 + q];
    w.S[k] = s;
    for (int c = m.augStart[k], end = m.augStart[k + 1]; c < end;) {
      const int head = c;
      real A = 0;
      do A += w.PI[m.augShell[c]] * (real)m.augYield[c]; while (++c < end && !m.augHead[c]);
      w.AUG[head] = A;
    }
  }
#endif
  for (int nIterateX = 1;; ++nIterateX) {
    bool lgConv = true;
    const real HIOld = xAt(b, m, w, zH, 1);
    const real HeIOld = heOn ? xAt(b, m, w, zHe, 1) : (real)0.;
    const real HeIIOld = heOn ? xAt(b, m, w, zHe, 2) : (real)0.;
    __syncwarp(L.mask);
    // H and He (independent of each other within an X-iteration)
    if (L.gl < 2 && m.xref[myZ]) {
      const int elem = myZ;
      real ionRatio[3] = {0, 0, 0};
      real ionProd[3] = {1, 1, 1};
      real den = 1;
      real collIonH = collIonH0;
      for (int ion = 1; ion <= min(elem, ns - 1); ++ion) {
        real cx = cxHHe[ion];
        if (elem > 1 || ion > 1) collIonH = 0;
        real pi = piHHe[ion];
        const real num = pi + collIonH * neR + (real)0.;
        const real dnm = neR * alHHe[ion] + cx * hdenR * HIOld;
        ionRatio[ion] = num / dnm;
      }
      for (int ion = 1; ion <= min(elem, ns - 1); ++ion)
        for (int i = 1; i <= ion; ++i) ionProd[ion] = ionProd[ion] * ionRatio[i];
      for (int ion = 1; ion <= min(elem, ns - 1); ++ion) den = den + ionProd[ion];
      for (int ion = 1; ion <= min(elem + 1, ns); ++ion) {
        real v = ion == 1 ? (real)1. / den : ionProd[ion - 1] / den;
        if (v > (real)kXMax()) v = (real)kXMax();
        if (v < (real)RD(1.e-20)) v = (real)RD(1.e-20);
        xAt(b, m, w, elem, ion) = v;
      }
    }
    __syncwarp(L.mask);
    // X(H0) as just updated above (grid%ionDen in the reference)
    const real xH0now = xAt(b, m, w, zH, 1);
    // the ladders' terms, a lane per (element, stage)
    for (int k = hFirst + L.gl; k < m.nPairs; k += G) {
      const int e = m.pE[k], ion = m.pIon[k];
      const int h = m.pH[k];
      const real* XE = w.X + (e - 1);   // X of this element's stage ion at XE[(ion - 1) * E]
      const real xi = XE[(ion - 1) * E];
      real* row = w.LAD + (size_t)h * kLadRows * ladRow;
#if MCX_BAL_EXACT
      // out: the Auger electrons of the lower stages, then collisional and
      // photoionisation (and, at the last stage, its own Auger electrons), in
      // the order the reference's loop over stages, shells and electrons adds them
      const real rXi = 1. / xi;
      real o = 0, ratio = 1;
      int c = m.augStart[k];
      const int end = m.augStart[k + 1];
      for (; c < end && m.augFrom[c] > 0; ++c) {
        if (m.augHead[c]) ratio = xi > (real)1e-30 ? eqDivide(XE[(ion - m.augFrom[c] - 1) * E], xi, rXi) : (real)1.;
        o = o + w.AUG[c] * ratio;
      }
      o = o + w.CC[k] * neR;
      const int p0 = m.p0[(e - 1) * 32 + (ion - 1)], nsh = m.nsh[(e - 1) * 32 + (ion - 1)];
      for (int q = 0; q < nsh; ++q) {
        o = o + w.PI[p0 + q];
        // its own electrons (clamped at the last stage): X(ion) / X(ion) = 1
        for (; c < end && m.augShell[c] == p0 + q; ++c) o = o + w.AUG[c];
      }
      const real in_ = neR * w.AL[k] + m.chex[k] * hdenR * xH0now;
      row[ion] = o;
      row[ladRow + ion] = in_;
      row[2 * ladRow + ion] = 1. / in_;
#else
      // out (collisional and photoionisation, the Auger electrons of the stages
      // below and, clamped at the last stage, its own, times X(stage) / X(ion)) and
      // inn, and the base-2 logarithm of their quotient
      real o = w.CC[k] * neR + w.S[k];
      // (a stage whose shells no photon reaches adds nothing, whatever its fraction)
      for (int c = m.augStart[k + 1] - 1; c >= m.augStart[k]; --c)
        if (m.augHead[c] && w.AUG[c] != (real)0.)
          o = o + w.AUG[c] * (xi > (real)1e-30 ? __fdividef(XE[(ion - m.augFrom[c] - 1) * E], xi) : (real)1.);
      const real in_ = neR * w.AL[k] + m.chex[k] * hdenR * xH0now;
      row[ion + 1] = log2f(__fdividef(o, in_));
#endif
    }
    __syncwarp(L.mask);
    // the ladders' products, a lane per element
    for (int h = L.gl; h < m.nHeavy; h += G) {
      const int topI = min(m.zOf[m.hE[h]], ns - 1);
      real* row = w.LAD + (size_t)h * kLadRows * ladRow;
#if MCX_BAL_EXACT
      real* mat = row + 3 * ladRow;
      mat[1] = 1.;
      double last = 1., sumMat = 1.;
      for (int ion = 2; ion <= topI + 1; ++ion) {
        last = eqDivide(last * row[ion - 1], row[ladRow + ion - 1], row[2 * ladRow + ion - 1]);
        mat[ion] = last;
        sumMat = sumMat + last;
      }
      mat[0] = 1. / sumMat;
#else
      // running sums of the logarithms: the products span far more than FP32's
      // range, their logarithms do not; row[0] keeps the largest
      float lmax = 0.f, lcur = 0.f;
      row[1] = 0.f;
      for (int ion = 1; ion <= topI; ++ion) {
        lcur = lcur + row[ion + 1];
        row[ion + 1] = lcur;
        lmax = fmaxf(lmax, lcur);
      }
      row[0] = lmax;
#endif
    }
    __syncwarp(L.mask);
#if !MCX_BAL_EXACT
    // normalised against the largest term
    for (int k = L.gl; k < m.nPairs - hFirst + m.nHeavy; k += G) {
      const int h = m.sH[k], st = m.sSt[k];
      real* row = w.LAD + (size_t)h * kLadRows * ladRow;
      row[ladRow + st] = exp2f(row[st] - row[0]);
    }
    __syncwarp(L.mask);
    for (int h = L.gl; h < m.nHeavy; h += G) {
      const int top = min(m.zOf[m.hE[h]], ns - 1) + 1;
      real* row = w.LAD + (size_t)h * kLadRows * ladRow;
      float sum = 0.f;
      for (int st = 1; st <= top; ++st) sum += row[ladRow + st];
      row[ladRow] = row[0] + log2f(sum);
    }
    __syncwarp(L.mask);
#endif
    // the new fractions; the first X-iteration takes the geometric mean with the old ones
    for (int k = hFirst + L.gl; k < m.nPairs; k += G) {
      const int e = m.pE[k], ion = m.pIon[k];
      const int h = m.pH[k];
      const real* row = w.LAD + (size_t)h * kLadRows * ladRow;
      real* XE = w.X + (e - 1);
      const bool topMost = ion == min(m.zOf[e], ns - 1);
#if MCX_BAL_EXACT
      const real* mat = row + 3 * ladRow;
      const double sumMat = mat[0];
      if (topMost) XE[ion * E] = mat[ion + 1] * sumMat;
      double v;
      if (nIterateX < 2 && mat[ion] * sumMat > 0.) {
        double old = XE[(ion - 1) * E];
        if (old <= 0.) old = RD(1.e-5);
        v = pow(10., 0.5 * (log10(old) + log10(mat[ion] * sumMat)));
      } else {
        v = mat[ion] * sumMat;
      }
      if (v > kXMax()) v = kXMax();
      if (v < RD(1.e-20)) v = RD(1.e-20);
      XE[(ion - 1) * E] = v;
#else
      const float lsum = row[ladRow];
      if (topMost) XE[ion * E] = exp2f(row[ion + 1] - lsum);
      const float lx = row[ion] - lsum;
      float v;
      if (nIterateX < 2 && lx > -1.e30f) {
        float old = XE[(ion - 1) * E];
        if (old <= 0.f) old = 1.e-5f;
        v = exp2f(0.5f * (log2f(old) + lx));
      } else {
        v = exp2f(lx);
      }
      if (v > 0.99999f) v = 0.99999f;
      if (v < 1.e-20f) v = 1.e-20f;
      XE[(ion - 1) * E] = v;
#endif
    }
    __syncwarp(L.mask);
#if MCX_BAL_EXACT
    // Ne: the terms by lane, added in the reference's order by the group's first lane
    for (int k = L.gl; k < m.nPairs; k += G) {
      const int e = m.pE[k], st = m.pIon[k] + 1;
      const real x = w.X[(st - 1) * E + (e - 1)];
      w.LAD[k] = x >= (real)RD(1.e-10) ? (real)(st - 1) * (real)m.abun[m.zOf[e]] * x : (real)0.;
    }
    __syncwarp(L.mask);
    real nE = 0;
    if (L.gl == 0) {
#pragma unroll 8
      for (int k = 0; k < m.nPairs; ++k) nE = nE + w.LAD[k];
      nE = nE * hdenR;
      if (nE == (real)0.) nE = 1;
    }
    neR = __shfl_sync(L.mask, nE, 0, G);
#else
    // Ne: the (element, stage) terms in eight partial sums, added up in a
    // butterfly (four lanes keep two each; the lanes of a larger group beyond the
    // eighth repeat them), so that the result does not depend on G
    real nE = 0, half[2] = {0, 0};
#pragma unroll
    for (int part = 0; part < (G == 4 ? 2 : 1); ++part) {
      real s = 0;
      const int p = (L.gl & 7) + 4 * part, n = m.neCount[p];
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
        const real x = w.X[m.neAt[8 * j + p]];
        if (x >= (real)RD(1.e-10)) s = s + m.neW[8 * j + p] * x;
      }
      half[part] = s;
    }
    nE = half[0];
    if (G == 4) nE = nE + half[1];
#pragma unroll
    for (int o = G == 4 ? 2 : 4; o > 0; o >>= 1) nE += __shfl_xor_sync(L.mask, nE, o, G < 8 ? G : 8);
    nE = nE * hdenR;
    if (nE == (real)0.) nE = 1;
    neR = nE;
#endif
    ne = (double)neR;
    real dHI = (xAt(b, m, w, zH, 1) - HIOld) / HIOld;
    real dHeI = heOn ? (xAt(b, m, w, zHe, 1) - HeIOld) / HeIOld : (real)0.;
    real dHeII = heOn ? (xAt(b, m, w, zHe, 2) - HeIIOld) / HeIIOld : (real)0.;
    const real lim = (real)b.xTol;
    bool big = fabs(dHI) > lim || fabs(dHeI) > lim || fabs(dHeII) > lim;
    if (big && nIterateX < 15) continue;
    if (big && nIterateX == 15) lgConv = false;
    return lgConv;
  }
}

// What a T-iteration's rates leave for the secant step (the group's first lane).
struct CellTerms {
  double heat, coolA, coolHex, coolCollH, compHeat, compRecoil, compCool;
  bool conv;
};

// One T-iteration's rates of cell `cell`, whose X is in w.X and whose shell
// rates (before the reverse charge exchange) are in w.PI; shellHeat(t, heatef)
// gives photoIon(2) of shell t.  ne is updated.
template <int G, typename ShellHeat>
__device__ __forceinline__ CellTerms ratesOf(const BalanceDev& b, const ElemMeta& m, const WarpCell& w, const Lanes& L,
                                             int cell, double te, double& ne, double hden, ShellHeat shellHeat) {
  const int C1 = b.nCells + 1, ns = b.nstages, E = b.nElemUsed, nSh = b.nShellsTot;
  CellTerms out{};
  const real teR = (real)te;
  const real hdenR = (real)hden;
  // calcAlpha, one pair per lane
#if MCX_BAL_EXACT
  const real rTe = (real)1. / teR, teM15 = pow(teR, (real)-1.5);
#endif
  for (int k = L.gl; k < m.nPairs; k += G) {
    const int e = m.pE[k], ion = m.pIon[k], elem = m.zOf[e];
#if MCX_BAL_EXACT
    w.AL[k] = alphaOf(b, teR, rTe, teM15, elem, ion);
#else
    w.AL[k] = b.alphaTab ? alphaLookup(b, (e - 1) * ns + (ion - 1), teR, elem, ion) : alphaOf(b, teR, elem, ion);
#endif
  }
  __syncwarp(L.mask);
  real xe = 0;
  for (int e = 1; e <= E; ++e) {
    const int elem = m.zOf[e];
    xe = xe + (real)xAt(b, m, w, elem, 1) * (real)m.abun[elem] * hdenR;
  }
  xe = (real)ne / xe;
  real heatef;
  if (xe > RF(0.95)) heatef = 1;
  else {
    if (xe < RF(1.e-4)) xe = RF(1.e-4);
    heatef = RF(0.9971) * ((real)1. - pow((real)1. - pow(xe, RF(0.2663)), RF(1.3163)));
  }
  // reverse charge exchange: deltaE_k > 1 only for N0 and O0
  if (L.gl < 2) {
    const int elem = L.gl == 0 ? 7 : 8;
    const real dE = L.gl == 0 ? RF(10863.) : RF(2205.);
    if (m.xref[elem] && ns - 1 >= 1) {
      const int32_t* o = outerOf(b, elem, elem);
      const int nsh = m.nsh[(m.xref[elem] - 1) * 32];
      if (o[0] <= nsh) {
        real cx = chexFit(b, elem, 1, teR);
        real rev = cx * ((real)1. - (real)xAt(b, m, w, 1, 1)) * hdenR * (real)2. * exp(-dE / teR) / ((real)o[1] / (real)o[2]);
        const int off = m.p0[(m.xref[elem] - 1) * 32] + o[0] - 1;
        w.PI[off] = w.PI[off] + rev;
      }
    }
  }
  // collisionalIonisation: the reference returns from the whole routine at the
  // first pair (element outer, ion inner) with u > 80, so that pair and every
  // later one keep 0
  {
    const real tev = teR * RF(8.617385e-05);
    int firstStop = m.nPairs;
    for (int k = L.gl; k < m.nPairs; k += G) {
      const int e = m.pE[k], ion = m.pIon[k], elem = m.zOf[e];
      w.CC[k] = 0;
      if (ion > min(ns - 1, elem - 1)) continue;
      const int elec = elem - ion + 1;
      const float* cf = b.CF + ((size_t)(elem - 1) * kNE + (elec - 1)) * 5;
      real u = (real)cf[0] / tev;
      if (u > (real)80.) { firstStop = min(firstStop, k); continue; }
      w.CC[k] = (real)cf[2] * ((real)1. + (real)cf[1] * sqrt(u)) / ((real)cf[3] + u) * pow(u, (real)cf[4]) * exp(-u);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) firstStop = min(firstStop, __shfl_xor_sync(L.mask, firstStop, o, G));
    for (int k = L.gl; k < m.nPairs; k += G)
      if (k >= firstStop) w.CC[k] = 0;
  }
  __syncwarp(L.mask);
  // compton, with the state before ionBalance
  if (b.lgCompton && L.gl == 0) {
    const real s1 = (real)b.comp[0 * (size_t)C1 + cell], s2 = (real)b.comp[1 * (size_t)C1 + cell];
    const real rhH = (real)b.comp[2 * (size_t)C1 + cell], rhHe = (real)b.comp[3 * (size_t)C1 + cell];
    real cool = (RF(6.65e-25) * RF(6.75e-10) * teR * s2) / hdenR;
    real heat = (RF(6.65e-25) * s1 / RF(8.184e-7)) / hdenR;
    real he = m.xref[2] ? rhHe * ((real)xAt(b, m, w, 2, 1) * (real)m.abun[2]) * (real)2. : (real)0.;
    real recoil = (rhH * (real)xAt(b, m, w, 1, 1) * (real)m.abun[1] + he) * kRyd2erg();
    out.compCool = cool;
    out.compHeat = heat;
    out.compRecoil = recoil;
  }
  out.conv = ionBalance<G>(b, m, w, L, te, ne, hden);
  __syncwarp(L.mask);
  // thermBalance without forLines: the terms by lane, their sums in the
  // reference's order by one lane each
  const real neR = (real)ne;
  real* sFF = w.LAD;                 // [2 E] free-free of the H-like, then of the He-like ions
  real* sRec = sFF + 2 * E;          // [2 E] the same for recombination
  real* sColl = sRec + 2 * E;        // [pairs] collisional ionisation
  for (int l = L.gl; l < E; l += G) {
    const int e = l + 1;
    const int i = m.zOf[e];
    real ff = 0, rec = 0, ff2 = 0, rec2 = 0;
    if (ns > i) {
      real L = log10(teR / (real)(i * i));
      real Np = (real)xAt(b, m, w, i, i + 1) * (real)m.abun[i];
      real betaFF = (real)i * (RF(1.0108464E-11) + RF(9.7930778E-13) * L - RF(6.6433144E-13) * L * L +
                               RF(2.4793747E-13) * L * L * L - RF(2.3938215E-14) * L * L * L * L);
      ff = Np * neR * betaFF * kBoltz() * teR / sqrt(teR);
      real betaRec = (real)i * (RF(9.4255985E-11) - RF(4.04794384E-12) * L - RF(1.0055237E-11) * L * L +
                                RF(1.99266862E-12) * L * L * L - RF(1.06681387E-13) * L * L * L * L);
      rec = Np * neR * betaRec * kBoltz() * teR / sqrt(teR);
      if (i >= 2) {
        L = log10((real)4. * teR / (real)(i * i));
        Np = (real)xAt(b, m, w, i, i) * (real)m.abun[i];
        betaFF = ((real)i / (real)2.) * (RF(1.070073e-11) - RF(2.5730207e-13) * L + RF(2.109134e-13) * L * L);
        ff2 = Np * neR * betaFF * kBoltz() * teR / sqrt(teR);
        betaRec = ((real)i / (real)2.) * (RF(1.06926e-10) - RF(2.41756e-11) * L + RF(1.14542e-12) * L * L -
                                          RF(5.06535e-13) * L * L * L + RF(9.16745e-14) * L * L * L * L);
        rec2 = Np * neR * betaRec * kBoltz() * teR / sqrt(teR);
      }
    }
    // the reference skips terms that are not numbers
    sFF[l] = isnan(ff) ? (real)0. : ff;
    sRec[l] = isnan(rec) ? (real)0. : rec;
    sFF[E + l] = isnan(ff2) ? (real)0. : ff2;
    sRec[E + l] = isnan(rec2) ? (real)0. : rec2;
  }
  for (int k = L.gl; k < m.nPairs; k += G) {
    const int e = m.pE[k], ion = m.pIon[k], elem = m.zOf[e];
    const real c2 = (real)b.cionTherm[(elem - 1) * kNE + (ion - 1)] * w.CC[k] * kBoltz();
    sColl[k] = (real)m.abun[elem] * xAt(b, m, w, elem, ion) * c2 * neR;
  }
  // photoheating per shell (the secondary-ionisation tail times heatef)
  for (int t = L.gl; t < nSh; t += G) {
    const PhotoShell sh = b.shells[t];
    w.PI[t] = shellHeat(t, sh.heavy, heatef) * xAt(b, m, w, sh.elem, sh.ion) * (real)m.abun[sh.elem];
  }
  __syncwarp(L.mask);
  real acc = 0;
  {
    const real* p = L.gl == 0 ? sFF : (L.gl == 1 ? sRec : (L.gl == 2 ? sColl : w.PI));
    const int n = L.gl < 2 ? 2 * E : (L.gl == 2 ? m.nPairs : (L.gl == 3 ? nSh : 0));
#pragma unroll 8
    for (int k = 0; k < n; ++k) acc = acc + p[k];
  }
  const real coolFF = acc;
  const real coolRec = __shfl_sync(L.mask, acc, 1, G);
  const real coolCollH = __shfl_sync(L.mask, acc, 2, G);
  const real heatSte = __shfl_sync(L.mask, acc, 3, G);
  if (L.gl != 0) return out;
  // Te4 as the He-like loop leaves it: 4 Te / (i^2 1e4) of the last element with nstages > i
  real Te4 = teR / RF(1.e4);
  for (int e = 1; e <= E; ++e) {
    const int i = m.zOf[e];
    if (i < 2 || !(ns > i)) continue;
    Te4 = (real)4. * teR / ((real)(i * i) * RF(1.e4));
  }
  real coolColl;
  if (teR > (real)5000.)
    coolColl = (RF(2.47e-8) * exp(-RF(118338.) / teR) * pow(Te4, RF(-0.228)) +
                RF(1.32e-8) * exp(-RF(140252.) / teR) * pow(Te4, RF(-0.460))) * kHcRyd() * (real)xAt(b, m, w, 1, 1) * neR;
  else
    coolColl = 0;
  out.coolA = coolFF + coolRec;
  out.coolHex = coolColl;
  out.coolCollH = coolCollH;
  out.heat = heatSte;
  return out;
}

#if !MCX_BAL_EXACT
// The same with what balanceCellsKernel keeps beside it; even, for the FP64 sums.
__host__ __device__ inline size_t cellsSlice(const BalanceDev& b) {
  return ((size_t)cellSlice(b) + 3 * b.nShellsTot + 1) / 2 * 2 + 2 * (size_t)b.nAtoms;
}
#endif

template <int G>
__device__ __forceinline__ Lanes lanesOf() {
  const int lane = threadIdx.x & 31;
  return Lanes{lane % G, G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (lane / G * G)};
}

// A round of the rates: one T-iteration of every listed cell.  The FP64 build,
// and the mixed one where every ion's levels are solved per cell.
__global__ void __launch_bounds__(128) ratesKernel(BalanceDev b, const float* __restrict__ hdenG, int round) {
  extern __shared__ double wsm[];
  constexpr int G = kGroup;
  const Lanes L = lanesOf<G>();
  const int slot = threadIdx.x / G, cellsPerBlock = blockDim.x / G;
  const unsigned cnt = b.listCount[round];
  if ((unsigned)(blockIdx.x * cellsPerBlock) >= cnt) return;   // the whole block
  const ElemMeta m = loadElemMeta(b, wsm);
  const int C1 = b.nCells + 1, NP = b.nElemUsed * b.nstages, nSh = b.nShellsTot;
  const WarpCell w = warpCell(b, reinterpret_cast<real*>(wsm + metaDoublesOf(b)) + (size_t)slot * cellSlice(b));
  // the listed cells in strides of the grid (the grid is sized for the resident blocks)
  for (unsigned base = blockIdx.x * cellsPerBlock; base < cnt; base += gridDim.x * cellsPerBlock) {
    const unsigned li = base + slot;
    if (li >= cnt) continue;
    const int cell = b.list[(size_t)(round & 1) * C1 + li];
    __syncwarp(L.mask);
    for (int k = L.gl; k < NP; k += G) w.X[k] = (real)b.ion[(size_t)k * C1 + cell];
    for (int t = L.gl; t < nSh; t += G) w.PI[t] = (real)b.gam[(size_t)t * C1 + cell];
    const double te = b.te[cell];
    double ne = b.ne[cell];
    const CellTerms r = ratesOf<G>(b, m, w, L, cell, te, ne, (double)hdenG[cell], [&](int t, int heavy, real heatef) {
      const size_t o = (size_t)t * C1 + cell;
      return heavy ? (real)b.heatA[o] + (real)b.heatHi[o] * heatef : (real)b.heatA[o];
    });
    for (int k = L.gl; k < NP; k += G) b.ion[(size_t)k * C1 + cell] = (double)w.X[k];
    if (L.gl != 0) continue;
    b.nIterT[cell] = b.nIterT[cell] + 1;
    b.ibConv[cell] = r.conv ? 1 : 0;
    b.ne[cell] = ne;
#if !MCX_BAL_EXACT
    if (b.coolTab) b.coolAt[cell] = coolStencil(te, ne);
#endif
    b.coolA[cell] = r.coolA;
    b.coolHex[cell] = r.coolHex;
    b.coolCollH[cell] = r.coolCollH;
    b.heat[cell] = r.heat;
    if (b.lgCompton) {
      b.compCool[cell] = r.compCool;
      b.compHeat[cell] = r.compHeat;
      b.compRecoil[cell] = r.compRecoil;
    }
  }
}

// ------------------------------------------------------------- equilibrium

#if MCX_BAL_EXACT
__device__ __forceinline__ const real* atomTable(const BalanceDev& b) { return b.atomData; }
#else
__device__ __forceinline__ const real* atomTable(const BalanceDev& b) { return b.atomDataF; }
#endif

// splint with the interval search done once per atom: klo/khi and the
// weights depend only on x and the temperature points
struct SplineAt {
  int klo, khi;    // 1-based, 0 = below the table, -1 = above
  real a, bb, a3, b3, hh;
};

__device__ SplineAt splineAt(const real* xa, int n, real x) {
  SplineAt s{};
  if (x <= xa[0]) { s.klo = 0; return s; }
  if (x >= xa[n - 1]) { s.klo = -1; return s; }
  int klo = 1, khi = n;
  for (int i = 0; i < 1000; ++i) {
    if (khi - klo <= 1) break;
    int k = (khi + klo) / 2;
    if (xa[k - 1] > x) khi = k; else klo = k;
  }
  real h = xa[khi - 1] - xa[klo - 1];
  s.klo = klo;
  s.khi = khi;
  s.a = (xa[khi - 1] - x) / h;
  s.bb = (x - xa[klo - 1]) / h;
  s.a3 = s.a * s.a * s.a - s.a;
  s.b3 = s.bb * s.bb * s.bb - s.bb;
  s.hh = h * h;
  return s;
}

__device__ __forceinline__ real splineEval(const SplineAt& s, const real* ya, const real* y2a, int n) {
  if (s.klo == 0) return ya[0];
  if (s.klo < 0) return ya[n - 1];
  return s.a * ya[s.klo - 1] + s.bb * ya[s.khi - 1] + (s.a3 * y2a[s.klo - 1] + s.b3 * y2a[s.khi - 1]) * s.hh / (real)6.;
}

// The collision rate coefficients qeff of every level pair (source/emission_mod.f90:2884-2936):
// f(lo, up, qeff(lo,up), qeff(up,lo)) for lo < up, in the rate precision.
template <typename F>
__device__ __forceinline__ void collisionPairs(const BalanceDev& b, const int32_t* h, real TeR, real sqrTe,
                                               real log10Te, F f, int first = 0, int step = 1) {
  const real* D = atomTable(b);
  const double* eD = b.atomData + h[kAtOffE];
  const int nLev = h[kAtNLev], nT = h[kAtNTemp];
  const real* logT = D + h[kAtOffLogT];
  const real* qom = D + h[kAtOffQom];
  const real* y2 = D + h[kAtOffY2];
  const real* g = D + h[kAtOffG];
  const real* e = D + h[kAtOffE];
  const SplineAt sp = nT > 2 ? splineAt(logT, nT, log10Te) : SplineAt{};
  const real constant = (real)1.4388463, c863 = (real)8.63e-6;
  int p = 0;
  for (int i = 2; i <= nLev; ++i) {
    for (int j = i; j <= nLev; ++j, ++p) {
      if (step > 1 && p % step != first) continue;
      const real* qq = qom + (size_t)p * nT;
      real cs;
      if (nT == 1) cs = qq[0];
      else if (nT == 2) cs = qq[0] + (qq[1] - qq[0]) / (logT[1] - logT[0]) * (log10Te - logT[0]);
      else cs = splineEval(sp, qq, y2 + (size_t)p * nT, nT);
      if (eD[i - 2] <= eD[j - 1]) {
        real expFac = exp((e[i - 2] - e[j - 1]) * constant / TeR);
        f(i - 1, j, c863 * cs * expFac / (g[i - 2] * sqrTe), c863 * cs / (g[j - 1] * sqrTe));
      } else {
        real expFac = exp((e[j - 1] - e[i - 2]) * constant / TeR);
        f(i - 1, j, c863 * cs / (g[j - 1] * sqrTe), c863 * cs * expFac / (g[i - 2] * sqrTe));
      }
    }
  }
}

#if !MCX_BAL_EXACT
// The same populations by state reduction in FP32 (Grassmann, Taksar & Heyman,
// Oper. Res. 33 (1985) 1107).  Rows 2..n of equilibrium's matrix are the
// balance of level i between the rates r(j->i) = Ne qeff(j,i) + a(j,i) into it,
// the rates out of it and, with rec, a recombination source
// s_i = Ne ionDenUp alpha_i; row 1 is the normalisation.  Eliminating levels
// n..2 redirects the flows through each removed level k in proportion to its
// exits r(k->j) / D_k, D_k = sum_{j<k} r(k->j), and back-substitution gives
// n_k = n_1 u_k + v_k with u_k the share fed from level 1 and v_k the share
// fed by the sources; the normalisation fixes n_1.  Every step adds or
// multiplies non-negative numbers, so each population keeps a relative error
// of a few FP32 ulps whatever the spread of the rates; the unpivoted LU of the
// reference cancels and needs FP64.  Returns false (the caller falls back to
// the FP64 LU) when a level has no exit to the levels below it.
__device__ __forceinline__ bool gthParts(const BalanceDev& b, const int32_t* h, double Ne, double srcMul, bool rec,
                                         const double* alphaTotal, real TeR, real sqrTe, real log10Te, float* u,
                                         float* v) {
  const int n = h[kAtNLev];
  const float* A = b.atomDataF + h[kAtOffA];
  const float NeF = (float)Ne;
  float R[kMaxLevels + 1][kMaxLevels + 1];   // R[a][c]: rate from level a to level c
  for (int i = 1; i <= n; ++i)
    for (int j = 1; j <= n; ++j) R[i][j] = 0.f;
  collisionPairs(b, h, TeR, sqrTe, log10Te, [&](int lo, int up, real qLoUp, real qUpLo) {
    R[lo][up] = NeF * qLoUp;
    R[up][lo] = NeF * qUpLo + A[(size_t)(up - 1) * n + (lo - 1)];
  });
  float src[kMaxLevels + 1], Dk[kMaxLevels + 1];
  for (int i = 1; i <= n; ++i) src[i] = (rec && i >= 2) ? (float)(srcMul * alphaTotal[i]) : 0.f;
  for (int k = n; k >= 2; --k) {
    float d = 0.f;
    for (int j = 1; j < k; ++j) d += R[k][j];
    if (!(d > 0.f) || !(d < 3.0e38f)) return false;
    Dk[k] = d;
    const float rd = 1.f / d;
    for (int i = 1; i < k; ++i) {
      const float fi = R[i][k] * rd;
      if (fi != 0.f)
        for (int j = 1; j < k; ++j) R[i][j] += fi * R[k][j];   // R[i][i] collects unused self-loops
    }
    if (rec) {
      const float fs = src[k] * rd;
      if (fs != 0.f)
        for (int j = 2; j < k; ++j) src[j] += fs * R[k][j];
    }
  }
  u[1] = 1.f;
  v[1] = 0.f;
  for (int k = 2; k <= n; ++k) {
    float a = 0.f, c = rec ? src[k] : 0.f;
    for (int i = 1; i < k; ++i) {
      a += u[i] * R[i][k];
      if (rec) c += v[i] * R[i][k];
    }
    u[k] = a / Dk[k];
    v[k] = c / Dk[k];
  }
  return true;
}

__device__ __forceinline__ bool gthPops(const BalanceDev& b, const int32_t* h, double Ne, double ionDenUp, bool rec,
                                        const double* alphaTotal, real TeR, real sqrTe, real log10Te, double* y) {
  float u[kMaxLevels + 1], v[kMaxLevels + 1];
  if (!gthParts(b, h, Ne, Ne * ionDenUp, rec, alphaTotal, TeR, sqrTe, log10Te, u, v)) return false;
  const int n = h[kAtNLev];
  float su = 0.f, sv = 0.f;
  for (int k = 2; k <= n; ++k) {
    su += u[k];
    sv += v[k];
  }
  const float n1 = (1.f - sv) / (1.f + su);
  y[1] = n1;
  for (int k = 2; k <= n; ++k) y[k] = (double)(n1 * u[k] + v[k]);
  return true;
}
#endif

// equilibrium of one atom: the normalised level populations y[1..nLev]
// (source/emission_mod.f90:2884-2984).  Collision rates in the rate
// precision; the FP64 path solves the rate matrix by the reference's
// unpivoted LU, the mixed path by FP32 state reduction (gthPops).
// the recombination coefficients of equilibrium's source term, alphaTotal[1..nLev]
// (source/emission_mod.f90:2836-2880)
__device__ __forceinline__ void recAlphas(const BalanceDev& b, const int32_t* h, real TeR, double* alphaTotal) {
  const double* DD = b.atomData;
  const int nLev = h[kAtNLev];
  for (int i = 0; i <= nLev; ++i) alphaTotal[i] = 0.;
  {
    const double* rr = DD + h[kAtOffRec];
    const real one = (real)1.;
    if (h[kAtRecType] == kRecPowerLaw) {
      for (int r = 0; r < h[kAtNRec]; ++r) {
        const double* v = rr + r * 11;
        const int j = r + 2;
        real br = (float)v[0], z = (float)v[1];
        real ar0 = (float)v[2], ar1 = (float)v[3], ar2 = (float)v[4], ar3 = (float)v[5];
        real ad0 = (float)v[6], ad1 = (float)v[7], ad2 = (float)v[8], ad3 = (float)v[9], ad4 = (float)v[10];
        if (z > (real)0.) {
          real tz = TeR * RF(1.e-4) / (z * z);
          real t4 = TeR * RF(1.e-4);
          alphaTotal[j] = RF(1.e-13) * br * z * ar0 * pow(tz, ar1) / (one + ar2 * pow(tz, ar3)) +
                          RF(1.0e-12) * br * (ad0 / t4 + ad1 + ad2 * TeR * RF(1.e-4) + ad3 * (t4 * t4)) *
                              pow(t4, (real)-1.5) * exp(-ad4 * RF(1.e4) / TeR);
        }
      }
    } else if (h[kAtRecType] == kRecChianti) {
      for (int r = 0; r < h[kAtNRec]; ++r) {
        const double* v = rr + r * 5;
        int jj = (int)v[0];
        real a = (float)v[1], bb = (float)v[2], cc = (float)v[3], d = (float)v[4];
        real L = log10(TeR);
        alphaTotal[jj] = pow((real)10., a + bb * L + cc * (L * L) + d * (L * L * L));
      }
    }
  }
}

__device__ __forceinline__ void equilibriumPops(const BalanceDev& b, int atom, double Te, double Ne, double ionDenUp,
                                                bool rec, double* y) {
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const double* DD = b.atomData;
  const int nLev = h[kAtNLev];
  const double* A = DD + h[kAtOffA];
  const real TeR = (real)Te;
  const real sqrTe = sqrt(TeR), log10Te = log10(TeR);
  double alphaTotal[kMaxLevels + 1];
  if (rec) recAlphas(b, h, TeR, alphaTotal);
  else
    for (int i = 0; i <= nLev; ++i) alphaTotal[i] = 0.;
#if !MCX_BAL_EXACT
  if (gthPops(b, h, Ne, ionDenUp, rec, alphaTotal, TeR, sqrTe, log10Te, y)) return;
#endif
  real qeff[kMaxLevels + 1][kMaxLevels + 1];
  double x[kMaxLevels + 1][kMaxLevels + 1];
  for (int i = 1; i <= nLev; ++i) {
    y[i] = 0.;
    for (int j = 1; j <= nLev; ++j) { qeff[i][j] = 0; x[i][j] = 0.; }
  }
  collisionPairs(b, h, TeR, sqrTe, log10Te, [&](int lo, int up, real qLoUp, real qUpLo) {
    qeff[lo][up] = qLoUp;
    qeff[up][lo] = qUpLo;
  });
  for (int j = 1; j <= nLev; ++j) x[1][j] = 1.;
  y[1] = 1.;
  for (int i = 2; i <= nLev; ++i) {
    for (int j = 1; j <= nLev; ++j) {
      if (j != i) {
        x[i][j] = x[i][j] + Ne * (double)qeff[j][i];
        x[i][i] = x[i][i] - Ne * (double)qeff[i][j];
        if (j > i) x[i][j] = x[i][j] + A[(size_t)(j - 1) * nLev + (i - 1)];
        else x[i][i] = x[i][i] - A[(size_t)(i - 1) * nLev + (j - 1)];
      }
    }
    y[i] = -Ne * ionDenUp * alphaTotal[i];
  }
  const int n = nLev;
#if MCX_BAL_EXACT
  // lured + reslv as the reference writes them (no pivoting, multipliers recomputed)
  if (n > 1) {
    for (int i = 1; i <= n - 1; ++i)
      for (int k = i + 1; k <= n; ++k) {
        double factor = x[k][i] / x[i][i];
        for (int j = i + 1; j <= n; ++j) x[k][j] = x[k][j] - x[i][j] * factor;
      }
    for (int i = 1; i <= n - 1; ++i)
      for (int j = i + 1; j <= n; ++j) y[j] = y[j] - y[i] * x[j][i] / x[i][i];
    y[n] = y[n] / x[n][n];
    for (int i = 1; i <= n - 1; ++i) {
      int k = n - i;
      for (int j = k + 1; j <= n; ++j) y[k] = y[k] - y[j] * x[k][j];
      y[k] = y[k] / x[k][k];
    }
  } else {
    y[1] = y[1] / x[1][1];
  }
#else
  // the same unpivoted elimination with one reciprocal per pivot and the
  // multipliers kept for the forward substitution (FP64)
  double rdiag[kMaxLevels + 1];
  for (int i = 1; i <= n - 1; ++i) {
    const double r = 1. / x[i][i];
    rdiag[i] = r;
    for (int k = i + 1; k <= n; ++k) {
      const double factor = x[k][i] * r;
      x[k][i] = factor;
      for (int j = i + 1; j <= n; ++j) x[k][j] = x[k][j] - x[i][j] * factor;
    }
  }
  rdiag[n] = 1. / x[n][n];
  for (int i = 1; i <= n - 1; ++i)
    for (int j = i + 1; j <= n; ++j) y[j] = y[j] - y[i] * x[j][i];
  y[n] = y[n] * rdiag[n];
  for (int k = n - 1; k >= 1; --k) {
    double acc = y[k];
    for (int j = k + 1; j <= n; ++j) acc = acc - y[j] * x[k][j];
    y[k] = acc * rdiag[k];
  }
#endif
  double sumN = 0.;
  for (int i = 1; i <= nLev; ++i) sumN = sumN + y[i];
  for (int i = 1; i <= nLev; ++i) y[i] = y[i] / sumN;
}

#if !MCX_BAL_EXACT
// equilibrium of one atom: the sum over its lines of a(j,i)*E_ji*n_j*m1*m2*m3,
// sum_j n_j sum_i a(j,i) E_ji with the line factors summed at set-up: the per-line
// 1e-35 cut of the reference (eqLines has it) drops terms that are below 1e-12 of
// any cooling rate the balance resolves.
__device__ double equilibriumLines(const BalanceDev& b, int atom, double Te, double Ne, double ionDenUp, bool rec,
                                   double m1, double m2, double m3) {
  double y[kMaxLevels + 1];
  equilibriumPops(b, atom, Te, Ne, ionDenUp, rec, y);
  const double* P = b.linePow + (size_t)atom * (kMaxLevels + 1);
  const int n = b.atomHdr[(size_t)atom * kAtHdrSize + kAtNLev];
  double acc = 0.;
  for (int j = 2; j <= n; ++j) acc = acc + y[j] * P[j];
  return acc * m1 * m2 * m3;
}
#endif

// Tight mode: a cell whose ladder has not converged in this round goes on at the same Te and its
// residual is not used (the secant step skips it), so its line cooling is not solved; the last round
// a cell can have still gets it (with Te held, the residual of that round is the result).
__device__ __forceinline__ bool coolingUnused(const BalanceDev& b, int round, int lastRound, int cell) {
  return b.converge && !b.ibConv[cell] && b.nIterT[cell] < b.maxIterT && round + 1 < kMaxRounds && !lastRound;
}

#if MCX_BAL_EXACT
#include "k_equilibrium.cuh"
#else
// forLines of update_mod: one thread per (cell, ion with data)
__global__ void __launch_bounds__(128) atomsKernel(BalanceDev b, int round, int lastRound) {
  const int li = blockIdx.x * blockDim.x + threadIdx.x;
  const int atom = blockIdx.y;
  if ((unsigned)li >= b.listCount[round]) return;
  const int cell = b.list[(size_t)(round & 1) * (b.nCells + 1) + li];
  if (coolingUnused(b, round, lastRound, cell)) return;
  const CellIdx c{cell, b.nCells + 1};
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const int elem = h[kAtElem], ion = h[kAtIon];
  const int top = min(elem + 1, b.nstages);
  const double x = ionAt(b, c, elem, ion);
  // an ion below 1e-16 per H contributes < 1e-9 of the cooling: no solve
  if ((double)b.abun[elem] * x < kNegligibleIon) {
    b.forSum[(size_t)atom * c.C1 + cell] = 0.;
    return;
  }
  // forbiddenLines = fLineEm * elemAbun * ionDen * 1.9865e-16, summed where > 1e-35;
  // without the recombination term the ratio ionDen(ion+1)/ionDen(ion) is not used
  (void)top;
  b.forSum[(size_t)atom * c.C1 + cell] =
      equilibriumLines(b, atom, b.te[cell], b.ne[cell], 0., false, (double)b.abun[elem], x, RD(1.9865e-16));
}

// The emission phase's forLines (rec = .true., 1e-25 erg units): one thread
// per (cell, ion with data), each ion's line total into forSum[atom][cell].
__global__ void __launch_bounds__(128) forLinesAtomsKernel(BalanceDev b, const float* __restrict__ te,
                                                           const float* __restrict__ ne,
                                                           const float* __restrict__ ionDen,
                                                           const uint8_t* __restrict__ compute) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  const int atom = blockIdx.y;
  const int C1 = b.nCells + 1;
  if (cell >= C1 || !compute[cell]) return;
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const int elem = h[kAtElem], ion = h[kAtIon];
  const int top = min(elem + 1, b.nstages);
  const int e = b.xref[elem];
  const double x = ionDen[((size_t)(ion - 1) * b.nElemUsed + (e - 1)) * C1 + cell];
  double v = 0.;
  if ((double)b.abun[elem] * x >= kNegligibleIon)
  {
    double up = 0.;
    if (ion < top && x > 0.) up = (double)ionDen[((size_t)ion * b.nElemUsed + (e - 1)) * C1 + cell] / x;
    v = equilibriumLines(b, atom, te[cell], ne[cell], up, true, (double)b.abun[elem], x, RD(1.9865e9));
  }
  b.forSum[(size_t)atom * C1 + cell] = v;
}

#endif

#if !MCX_BAL_EXACT
// The emission phase's forLines from the surfaces: each cell placed on the
// grid once, then one thread per (cell, ion with data) forms
// (G + ionDenUp B) elemAbun ionDen 1.9865e9; cells outside the grid solve
// the ion directly.
__global__ void __launch_bounds__(128) surfaceStencilKernel(BalanceDev b, const float* __restrict__ te,
                                                            const float* __restrict__ ne,
                                                            const uint8_t* __restrict__ compute) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell > b.nCells || !compute[cell]) return;
  b.coolAt[cell] = coolStencil((double)te[cell], (double)ne[cell]);
}

__global__ void __launch_bounds__(128) forLinesSurfaceKernel(BalanceDev b, const float* __restrict__ te,
                                                             const float* __restrict__ ne,
                                                             const float* __restrict__ ionDen,
                                                             const uint8_t* __restrict__ compute) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  const int atom = blockIdx.y;
  const int C1 = b.nCells + 1;
  if (cell >= C1 || !compute[cell]) return;
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const int elem = h[kAtElem], ion = h[kAtIon];
  const int top = min(elem + 1, b.nstages);
  const int e = b.xref[elem];
  const double x = ionDen[((size_t)(ion - 1) * b.nElemUsed + (e - 1)) * C1 + cell];
  double v = 0.;
  if ((double)b.abun[elem] * x >= kNegligibleIon) {
    double up = 0.;
    if (ion < top && x > 0.) up = (double)ionDen[((size_t)ion * b.nElemUsed + (e - 1)) * C1 + cell] / x;
    const CoolAt a = b.coolAt[cell];
    double L;
    if (a.iT >= 0) {
      const float2 g = surfaceAt(b.coolTab, atom, a);
      const float2 r = surfaceAt(b.recTab, atom, a);
      L = (double)expf(g.x) * (double)expf(g.y) + up * (double)(r.x + r.y);
    } else {
      L = equilibriumLines(b, atom, te[cell], ne[cell], up, true, 1., 1., 1.);
    }
    v = L * (double)b.abun[elem] * x * RD(1.9865e9);
  }
  b.forSum[(size_t)atom * C1 + cell] = v;
}
#endif

// normFor of emissionDriver: the ions' line totals summed in the reference's ion order
__global__ void forLinesSumKernel(BalanceDev b, const uint8_t* __restrict__ compute, float* forLines) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  const int C1 = b.nCells + 1;
  if (cell >= C1 || !compute[cell]) return;
  double normFor = 0.;
  for (int atom = 0; atom < b.nAtoms; ++atom) normFor = normFor + b.forSum[(size_t)atom * C1 + cell];
  forLines[cell] = (float)normFor;
}

#if MCX_BAL_EXACT
// outputGas forbidden-line volume sums (source/output_mod.f90:410-432 with
// forLines at :1943-1984): per (cell, ion with data) the level populations of
// equilibrium(rec = .true.), weighted by elemAbun * ionDen * 1.9865e9 * Hden
// * dV over the cells with lgBlack < 1.  Each warp (32 consecutive cells)
// reduces level j into partial[group][forbBase[atom] + j - 1]; the line
// factors a(j,i) E_ji multiply the sums afterwards.
// For the ions of more than 17 levels, the first of eqOrder: their blocks of
// eqPopulations hold 16 cells, half a warp's group (eqLevelSumsKernel has the others).
__global__ void __launch_bounds__(128) forbLevelSumsKernel(BalanceDev b, LineSumArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int group = t >> 5;
  if (group >= a.nGroups) return;   // whole warps only
  const int cell = a.cellBase + t + 1;
  const int atom = b.eqOrder[blockIdx.y];
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const int elem = h[kAtElem], ion = h[kAtIon], nLev = h[kAtNLev];
  const int top = min(elem + 1, b.nstages);
  const size_t C1 = (size_t)b.nCells + 1;
  const int e = b.xref[elem];
  const bool valid = t + 1 <= a.nRange && a.black[cell] < 1;
  double y[kMaxLevels + 1];
  double w = 0.;
  if (valid) {
    const double x = a.ionDen[((size_t)(ion - 1) * b.nElemUsed + (e - 1)) * C1 + cell];
    double up = 0.;
    if (ion < top && x > 0.) up = (double)a.ionDen[((size_t)ion * b.nElemUsed + (e - 1)) * C1 + cell] / x;
    equilibriumPops(b, atom, a.te[cell], a.ne[cell], up, true, y);
    w = (double)b.abun[elem] * x * RD(1.9865e9) * (double)a.hden[cell] * a.vol[cell];
  } else {
    for (int j = 1; j <= nLev; ++j) y[j] = 0.;
  }
  double* row = a.partial + (size_t)group * a.nEntries + a.forbBase[atom];
  for (int j = 1; j <= nLev; ++j) {
    const double v = warpSumD(valid ? y[j] * w : 0.);
    if ((threadIdx.x & 31) == 0) row[j - 1] = v;
  }
}

cudaError_t launchLineCells(BalanceData& bd, const LineCellArgs& a, cudaStream_t s) {
  if (a.nReq <= 0 || bd.dev.nCells <= 0) return cudaSuccess;
  eqLineCellKernel<<<dim3(eqBlocks(bd.dev, bd.dev.nCells), a.nReq), kEqThreads, bd.dev.eqSmem, s>>>(bd.dev, a);
  return cudaGetLastError();
}

cudaError_t launchForbSums(BalanceData& bd, const LineSumArgs& a, cudaStream_t s) {
  BalanceDev& b = bd.dev;
  if (b.nAtoms <= 0 || a.nGroups <= 0) return cudaSuccess;
  const int T = 128, nb = (a.nGroups * 32 + T - 1) / T, many = b.levelAtoms[3];
  if (many > 0) forbLevelSumsKernel<<<dim3(nb, many), T, 0, s>>>(b, a);
  if (b.nAtoms > many)
    eqLevelSumsKernel<<<dim3(a.nGroups, b.nAtoms - many), kEqThreads, b.eqSmem, s>>>(b, a, many);
  return cudaGetLastError();
}
#endif

#if !MCX_BAL_EXACT
// ------------------------------------------------------------- cooling surfaces

// G and B of one atom at (Te, Ne): forLines' line sum per ion without the
// recombination term (G) and its slope in ionDenUp with it (B), so that the
// sum with the term is G + ionDenUp B.  The state reduction gives both from
// one solve: with sources Ne alpha_i, n_k = n_1 u_k + ionDenUp w_k and
// n_1 = (1 - ionDenUp W) / (1 + U), U = sum u_k, W = sum w_k; a level without
// an exit below it falls back to two LU solves.
__device__ __noinline__ void surfaceValues(const BalanceDev& b, int atom, double Te, double Ne, double& G, double& B) {
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const int n = h[kAtNLev];
  const real TeR = (real)Te;
  const real sqrTe = sqrt(TeR), log10Te = log10(TeR);
  double alphaTotal[kMaxLevels + 1];
  recAlphas(b, h, TeR, alphaTotal);
  float u[kMaxLevels + 1], v[kMaxLevels + 1];
  if (gthParts(b, h, Ne, Ne, true, alphaTotal, TeR, sqrTe, log10Te, u, v)) {
    const double* P = b.linePow + (size_t)atom * (kMaxLevels + 1);
    double U = 0., UP = 0., W = 0., WP = 0.;
    for (int k = 2; k <= n; ++k) {
      U += u[k];
      UP += (double)u[k] * P[k];
      W += v[k];
      WP += (double)v[k] * P[k];
    }
    G = UP / (1. + U);
    B = WP - W * G;
  } else {
    G = equilibriumLines(b, atom, Te, Ne, 0., false, 1., 1., 1.);
    B = equilibriumLines(b, atom, Te, Ne, 1., true, 1., 1., 1.) - G;
  }
}

// ln G and B of the atoms eqOrder[first ...] (of at most N levels) at the grid
// nodes (see k_balance.cuh); G below 1e-37 is stored as 1e-37 (an ion that cools by
// less is below any cooling rate the balance resolves).
//
// A node is the state reduction of surfaceValues, operation for operation.  Its
// collision rates depend on Te alone: a block takes P = 32 / L temperatures of one
// atom, works out their rates once into shared memory and solves kCoolNeTile
// densities with them, a warp P nodes at a time.  L lanes share a node, each with
// every L-th column of the matrix in registers; the sums over a row go by shuffles
// in the order of the levels, and of the FP64 sums at the end the first lane takes
// the shares fed from level 1, the second those fed by recombination.  A thread per
// node with its matrix in local memory worked out every rate (a spline, an
// exponential, four divisions) for each density again
// (the 30 ions of the 41^3 lognormal gas: 21 ms, 8.5 now; 89 of the X-ray gas: 67 ms).
// What bounds it is the FP64 pipe, an operation 64 cycles a warp and scheduler:
// widen() converts without it, levels that recombination does not feed are left
// out, two lanes share a quotient and a logarithm.
constexpr int kCoolWarps = 4, kCoolNeTile = 80;

// (double)f by integer operations where f is positive and normal, or 0
__device__ __forceinline__ double widen(float f) {
  const unsigned u = __float_as_uint(f);
  if (u - 0x00800000u < 0x7f000000u) return __hiloint2double((int)((u >> 3) + 0x38000000u), (int)(u << 29));
  return u == 0u ? 0. : (double)f;
}

template <int N, int L>
__global__ void __launch_bounds__(32 * kCoolWarps) coolNodesKernel(BalanceDev b, int first, float* __restrict__ tab,
                                                                   float* __restrict__ rtab) {
  constexpr int P = 32 / L, C = (N + L - 1) / L;
  static_assert(kCoolNTe % P == 0 && kCoolNNe % kCoolNeTile == 0, "whole tiles");
  __shared__ float sQ[N * N * P];   // [from][to][temperature]
  __shared__ float sA[N * N];       // [upper][lower]
  __shared__ double sAlpha[C * L * P], sPow[N], sNe[kCoolNeTile];   // 0 for the columns beyond the levels
  __shared__ unsigned sSources;     // the levels that recombination feeds
  static_assert(((C - 1) * L + L - 1) * P + P - 1 < (int)(sizeof(sAlpha) / sizeof(double)), "the last lane's last column");
  static_assert(N <= 31 && (kCoolNeTile / kCoolWarps) % 2 == 0, "a bit a level; an even number of densities a warp");
  if (threadIdx.x == 0) sSources = 0u;
  __syncthreads();
  const int atom = b.eqOrder[first + blockIdx.y];
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const int n = h[kAtNLev];
  const int iT0 = blockIdx.x * P, iN0 = blockIdx.z * kCoolNeTile;
  {
    const int p = threadIdx.x % P, worker = threadIdx.x / P;
    constexpr int workers = 32 * kCoolWarps / P;
    const double te = exp(kCoolLnTe0 + (iT0 + p) * ((kCoolLnTe1 - kCoolLnTe0) / (kCoolNTe - 1)));
    const real TeR = (real)te;
    const real sqrTe = sqrt(TeR), log10Te = log10(TeR);
    collisionPairs(b, h, TeR, sqrTe, log10Te, [&](int lo, int up, real qLoUp, real qUpLo) {
      sQ[((lo - 1) * N + up - 1) * P + p] = qLoUp;
      sQ[((up - 1) * N + lo - 1) * P + p] = qUpLo;
    }, worker, workers);
    if (worker == 0) {
      double alphaTotal[kMaxLevels + 1];
      recAlphas(b, h, TeR, alphaTotal);
      for (int i = 0; i < C * L; ++i) {
        sAlpha[i * P + p] = i >= 1 && i < n ? alphaTotal[i + 1] : 0.;
        if (i >= 1 && i < n && alphaTotal[i + 1] != 0.) atomicOr(&sSources, 1u << i);
      }
    }
    for (int k = threadIdx.x; k < n * n; k += 32 * kCoolWarps)
      sA[(k / n) * N + k % n] = k % n < k / n ? b.atomDataF[h[kAtOffA] + k] : 0.f;
    for (int k = threadIdx.x; k < n; k += 32 * kCoolWarps) sPow[k] = b.linePow[(size_t)atom * (kMaxLevels + 1) + k + 1];
    for (int k = threadIdx.x; k < kCoolNeTile; k += 32 * kCoolWarps)
      sNe[k] = exp(kCoolLnNe0 + (iN0 + k) * ((kCoolLnNe1 - kCoolLnNe0) / (kCoolNNe - 1)));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, l = lane % L, p = lane / L, lead = lane - l;
  const unsigned sources = sSources;
  double pS = 0., pSP = 0., pW = 0., pWP = 0.;
  bool pOk = true;
  int pR = 0;
  for (int r = threadIdx.x >> 5, turn = 0; r < kCoolNeTile; r += kCoolWarps, ++turn) {
    const double Ne = sNe[r];
    const float NeF = (float)Ne;
    float R[N][C], src[C], D[C];    // this lane's columns j = c L + l
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int j = c * L + l;
#pragma unroll
      for (int i = 0; i < N; ++i)
        R[i][c] = i < n && j < n && i != j ? fmaf(NeF, sQ[(i * N + j) * P + p], sA[i * N + j]) : 0.f;
      src[c] = (sources >> (c * L)) & ((1u << L) - 1u) ? (float)(Ne * sAlpha[j * P + p]) : 0.f;
      D[c] = 1.f;
    }
    bool ok = true;
#pragma unroll
    for (int k = N - 1; k >= 1; --k) {
      if (k < n) {
        float d = 0.f;
#pragma unroll
        for (int j = 0; j < k; ++j) d += L == 1 ? R[k][j / L] : __shfl_sync(0xffffffffu, R[k][j / L], lead + j % L);
        ok = ok && d > 0.f && d < 3.0e38f;
        if (l == k % L) D[k / L] = d;
        const float rd = 1.f / d;
#pragma unroll
        for (int i = 0; i < k; ++i) {
          const float fi = (L == 1 ? R[i][k / L] : __shfl_sync(0xffffffffu, R[i][k / L], lead + k % L)) * rd;
#pragma unroll
          for (int c = 0; c <= (k - 1) / L; ++c)
            if (L == 1 || c * L + l < k) R[i][c] += fi * R[k][c];   // the diagonal collects unused self-loops
        }
        const float fs = (L == 1 ? src[k / L] : __shfl_sync(0xffffffffu, src[k / L], lead + k % L)) * rd;
#pragma unroll
        for (int c = 0; c <= (k - 1) / L; ++c)
          if (L == 1 || c * L + l < k) src[c] += fs * R[k][c];
      }
    }
    // each level's shares once those below are known, added to the levels above
    float a[C], v[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      a[c] = R[0][c];
      v[c] = src[c];
    }
    double S = 0., SP = 0., S2 = 0., SP2 = 0.;
#pragma unroll
    for (int k = 1; k < N; ++k) {
      if (k < n) {
        float uk = a[k / L] / D[k / L], vk = v[k / L] / D[k / L];
        if (L > 1) {
          uk = __shfl_sync(0xffffffffu, uk, lead + k % L);
          vk = __shfl_sync(0xffffffffu, vk, lead + k % L);
        }
#pragma unroll
        for (int c = (k + 1) / L; c < C; ++c) {
          a[c] += uk * R[k][c];
          v[c] += vk * R[k][c];
        }
        const double x = widen(l == 0 ? uk : vk);
        S += x;
        SP += x * sPow[k];
        if (L == 1) {
          const double y = widen(vk);
          S2 += y;
          SP2 += y * sPow[k];
        }
      }
    }
    int rOut = r;
    if (L > 1) {
      // the quotient and the logarithm of two densities at once: the first lane
      // takes those of the density before, the second those of this one
      const bool second = (turn & 1) != 0;
      const double oS = __shfl_xor_sync(0xffffffffu, S, 1), oSP = __shfl_xor_sync(0xffffffffu, SP, 1);
      if (!second) {          // kept by the first lane
        pS = S; pSP = SP; pW = oS; pWP = oSP; pOk = ok; pR = r;
        continue;
      }
      if (l == 0) { S2 = pW; SP2 = pWP; S = pS; SP = pSP; ok = pOk; rOut = pR; }
      else { S2 = S; SP2 = SP; S = oS; SP = oSP; }
    }
    if (l < 2) {
      double g = SP / (1. + S);
      double bb = SP2 - S2 * g;
      const int iT = iT0 + p, iN = iN0 + rOut;
      if (!ok) surfaceValues(b, atom, exp(kCoolLnTe0 + iT * ((kCoolLnTe1 - kCoolLnTe0) / (kCoolNTe - 1))), sNe[rOut], g, bb);
      const size_t idx = ((size_t)atom * kCoolNNe + iN) * kCoolNTe + iT;
      tab[idx] = (float)log(fmax(g, 1e-37));
      rtab[idx] = (float)bb;
    }
  }
}

// weights of the 4-point Lagrange interpolant at nodes -1, 0, 1, 2 for t in [0, 1)
__device__ __forceinline__ void lagrange4(float t, float* w) {
  const float tm1 = t - 1.f, tm2 = t - 2.f, tp1 = t + 1.f;
  w[0] = -t * tm1 * tm2 * (1.f / 6.f);
  w[1] = tp1 * tm1 * tm2 * 0.5f;
  w[2] = -tp1 * t * tm2 * 0.5f;
  w[3] = tp1 * t * tm1 * (1.f / 6.f);
}

// Where a cell's (Te, Ne) sits on the cooling surfaces: the nodes iT, iN of
// the 4 x 4 stencil's second row and column and the fractions within the
// cell of the grid (iT = -1 outside it).
__device__ CoolAt coolStencil(double te, double ne) {
  const double sT = (log(te) - kCoolLnTe0) * ((kCoolNTe - 1) / (kCoolLnTe1 - kCoolLnTe0));
  const double sN = (log(ne) - kCoolLnNe0) * ((kCoolNNe - 1) / (kCoolLnNe1 - kCoolLnNe0));
  CoolAt a{-1, -1, 0.f, 0.f};
  if (sT >= 1. && sT < kCoolNTe - 2 && sN >= 1. && sN < kCoolNNe - 2) {
    a.iT = (int)sT;
    a.iN = (int)sN;
    a.tT = (float)(sT - a.iT);
    a.tN = (float)(sN - a.iN);
  }
  return a;
}

// A surface of atom `atom` ([nAtoms][kCoolNNe][kCoolNTe]) at the stencil a:
// 4-point Lagrange in both directions, summed as differences from the
// stencil's (iN, iT) node so that the FP32 sums keep the stored precision;
// returns the node value and the interpolated difference.
__device__ __forceinline__ float2 surfaceAt(const float* tab, int atom, const CoolAt& a) {
  float wT[4], wN[4];
  lagrange4(a.tT, wT);
  lagrange4(a.tN, wN);
  const float* t = tab + ((size_t)atom * kCoolNNe + (a.iN - 1)) * kCoolNTe + (a.iT - 1);
  const float ref = __ldg(t + kCoolNTe + 1);
  float acc = 0.f;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const float* row = t + (size_t)r * kCoolNTe;
    const float v = wT[0] * (__ldg(row) - ref) + wT[1] * (__ldg(row + 1) - ref) + wT[2] * (__ldg(row + 2) - ref) +
                    wT[3] * (__ldg(row + 3) - ref);
    acc += wN[r] * v;
  }
  return make_float2(ref, acc);
}

// An ion's solve where the cell lies outside the surfaces, out of line.
__device__ __noinline__ double solvedCooling(const BalanceDev& b, int atom, double te, double ne) {
  return equilibriumLines(b, atom, te, ne, 0., false, 1., 1., 1.);
}

// The line cooling of one ion, w = elemAbun ionDen
__device__ __forceinline__ double surfaceCooling(const BalanceDev& b, int atom, const CoolAt& a, double w, double te,
                                                 double ne) {
  if (w < kNegligibleIon) return 0.;
  double g;
  if (a.iT >= 0) {
    // exp of the node value and of the interpolated difference apart: each is exact to an FP32 ulp
    const float2 r = surfaceAt(b.coolTab, atom, a);
    g = (double)expf(r.x) * (double)expf(r.y);
  } else {
    g = solvedCooling(b, atom, te, ne);
  }
  return w * RD(1.9865e-16) * g;
}
#endif

// The bracket of a cell's Te iteration.
struct Bracket {
  double tHigh, tLow, resHigh, resLow;
  int8_t side;
};

// The secant step of iterateT (FP64 in both precisions) after T-iteration
// nIterateT of a cell, in round `round`: te and the bracket move on; true when
// the cell goes on iterating, false when it is done.
__device__ __forceinline__ bool secantStep(const BalanceDev& b, int cell, int round, int lastRound, int nIterateT,
                                           bool ibConv, double heat, double cool, double& te, Bracket& k) {
  const double res = heat - cool;
  bool done = true;
  const bool tight = b.converge != 0;
  // tight mode: a residual whose ionisation ladder has not converged is evaluated again at the same Te
  // (the X-iterations go on from where they stopped) rather than taken as a bracket end
  const bool xPending = tight && !ibConv;
  if (b.fixTe) {
    // Te held: the ladder goes on converging at this Te; the residual there is the result
    b.resid[cell] = res;
    done = !(xPending && nIterateT < b.maxIterT && round + 1 < kMaxRounds);
    if (done && !ibConv) atomicAdd(&b.counters->noIonBal, 1ull);
    return !done;
  }
  double Thigh = k.tHigh, Tlow = k.tLow, resHigh = k.resHigh, resLow = k.resLow;
  bool open = xPending || fabs(res) >= b.resTol * (fabs(cool) + fabs(heat)) / 2.;
  if (open && !xPending && tight && Thigh != 0. && Tlow != 0. && fabs(Thigh - Tlow) <= 1e-12 * (Thigh + Tlow)) {
    open = false;
    // closed on the rounding noise of the residual, or on a jump of heating - cooling (not a root)
    if (fabs(res) > 1e3 * b.resTol * (fabs(cool) + fabs(heat)) / 2.) k.side = 3;
  }
  if (open) {
    if (nIterateT < b.maxIterT) {
      if (xPending) {
      } else if (tight) {
        // Illinois: an end kept twice in a row has its residual halved
        const int8_t last = k.side;
        if (res < 0.) {
          if (last == 1 && Thigh != 0.) resHigh = resHigh * 0.5;
          resLow = res;
          Tlow = te;
          k.side = 1;
        } else {
          if (last == 2 && Tlow != 0.) resLow = resLow * 0.5;
          resHigh = res;
          Thigh = te;
          k.side = 2;
        }
        if (Thigh != 0. && Tlow != 0.) {
          te = Tlow - (Thigh - Tlow) * resLow / (resHigh - resLow);
        } else {
          const double f = 1. + fmin(0.2, b.stepMin * ldexp(1., min(nIterateT, 60)));
          te = res < 0. ? te / f : te * f;
        }
      } else {
        if (res < 0.) {
          resLow = res;
          Tlow = te;
          if (Thigh != 0.) te = Tlow - (Thigh - Tlow) * resLow / (resHigh - resLow);
          else te = te / RD(1.2);
        } else {
          resHigh = res;
          Thigh = te;
          if (Tlow != 0.) te = Tlow - (Thigh - Tlow) * resLow / (resHigh - resLow);
          else te = te * RD(1.2);
        }
        if (nIterateT >= 6 && fabs(Thigh - Tlow) <= (RD(0.002) * (Thigh + Tlow))) {
          if (res < 0.) { te = Thigh - 100.; Thigh = 0.; }
          else { te = Tlow + 100.; Tlow = 0.; }
        }
      }
      if (te <= 0.) te = 1.;
      done = lastRound != 0;   // a caller-imposed round limit ends the cell here
    } else {
      // (tight mode: a cell whose ladder never converged was never bracketed and keeps its Te)
      if (Thigh == 0. && Tlow == 0.) {
      } else if (Thigh == 0.) te = Tlow;
      else if (Tlow == 0.) te = Thigh;
      else te = (Thigh + Tlow) * 0.5;
      atomicAdd(&b.counters->noTeBal, 1ull);
    }
  }
  k.tHigh = Thigh; k.tLow = Tlow; k.resHigh = resHigh; k.resLow = resLow;
  if (done && !ibConv) atomicAdd(&b.counters->noIonBal, 1ull);
  return !done;
}

// heating - cooling and the secant step of one listed cell
__device__ __forceinline__ void secantCell(const BalanceDev& b, int round, int lastRound, int li) {
  const int C1 = b.nCells + 1;
  const int cell = b.list[(size_t)(round & 1) * C1 + li];
  double coolColl = b.coolHex[cell];
  for (int a = 0; a < b.nAtoms; ++a) coolColl = coolColl + b.forSum[(size_t)a * C1 + cell];
  const double ne = b.ne[cell];
  double heat = b.heat[cell];
  double cool = b.coolA[cell] + coolColl + b.coolCollH[cell];
  if (b.lgCompton) {
    heat = heat + b.compHeat[cell] * ne + b.compRecoil[cell];
    cool = cool + b.compCool[cell] * ne;
  }
  double te = b.te[cell];
  Bracket k{b.tHigh[cell], b.tLow[cell], b.resHigh[cell], b.resLow[cell], b.side[cell]};
  const bool on = secantStep(b, cell, round, lastRound, b.nIterT[cell], b.ibConv[cell] != 0, heat, cool, te, k);
  if (!b.fixTe) {
    b.te[cell] = te;
    b.tHigh[cell] = k.tHigh; b.tLow[cell] = k.tLow; b.resHigh[cell] = k.resHigh; b.resLow[cell] = k.resLow;
    b.side[cell] = k.side;
  }
  if (!on) b.state[cell] = 1;
  else if (round + 1 < kMaxRounds) b.list[(size_t)((round + 1) & 1) * C1 + atomicAdd(&b.listCount[round + 1], 1u)] = cell;
}

__global__ void __launch_bounds__(128) secantKernel(BalanceDev b, int round, int lastRound) {
  const unsigned cnt = b.listCount[round];
  for (unsigned li = blockIdx.x * blockDim.x + threadIdx.x; li < cnt; li += gridDim.x * blockDim.x)
    secantCell(b, round, lastRound, (int)li);
}

#if !MCX_BAL_EXACT
// The whole T-iteration of the mixed balance with cooling surfaces: a group of G
// lanes takes a cell from the list of cells that packets reached and runs its
// T-iterations one after another (rates, line cooling with the ions shared out
// among the lanes, secant step), then the next cell.  A cell depends on no other,
// so nothing waits for a round to end: as three launches a round, the last
// rounds of a 41^3 grid (a few slow cells) took 0.14 - 0.31 ms each whatever their
// number, and empty rounds their launches.  J's integrals and the fractions stay
// in shared memory between the T-iterations (41^3 lognormal
// gas: 9.5 -> 8.2 ms a balance; 5.8 with what the comments above tell).
// kIons: with the line cooling.  Its solve of a cell outside the surfaces has 16 KB of
// local memory a thread, 4.6 GB on the device once such a kernel is launched, which
// a gas without multi-level ions does not need.
template <int G, bool kIons>
__global__ void __launch_bounds__(128, 4) balanceCellsKernel(BalanceDev b, const float* __restrict__ hdenG, int rounds) {
  extern __shared__ double wsm[];
  const unsigned cnt = b.listCount[0];
  if (blockIdx.x * (blockDim.x / G) >= cnt) return;   // the whole block
  const Lanes L = lanesOf<G>();
  const ElemMeta m = loadElemMeta(b, wsm);
  const int C1 = b.nCells + 1, NP = b.nElemUsed * b.nstages, nSh = b.nShellsTot, nA = kIons ? b.nAtoms : 0;
  const int base = cellSlice(b);
  real* mine = reinterpret_cast<real*>(wsm + metaDoublesOf(b)) + (size_t)(threadIdx.x / G) * cellsSlice(b);
  const WarpCell w = warpCell(b, mine);
  real* pi0 = mine + base;            // [nSh] photoionisation rates without the reverse charge exchange
  real* heatA = pi0 + nSh;            // [nSh] heating without and
  real* heatHi = heatA + nSh;         // [nSh] in the secondary-ionisation tail
  double* forSum = reinterpret_cast<double*>(mine + (base + 3 * nSh + 1) / 2 * 2);   // [nAtoms]
  for (;;) {
    unsigned li = 0;
    if (L.gl == 0) li = atomicAdd(&b.listCount[1], 1u);
    li = __shfl_sync(L.mask, li, 0, G);
    if (li >= cnt) break;
    const int cell = b.list[li];
    for (int k = L.gl; k < NP; k += G) w.X[k] = (real)b.ion[(size_t)k * C1 + cell];
    for (int t = L.gl; t < nSh; t += G) {
      const size_t o = (size_t)t * C1 + cell;
      pi0[t] = (real)b.gam[o];
      heatA[t] = (real)b.heatA[o];
      heatHi[t] = (real)b.heatHi[o];
    }
    __syncwarp(L.mask);
    const double hden = (double)hdenG[cell];
    double te = b.te[cell], ne = b.ne[cell];
    Bracket k{b.tHigh[cell], b.tLow[cell], b.resHigh[cell], b.resLow[cell], b.side[cell]};
    int nIter = b.nIterT[cell], on = 1, conv = 1;
    for (int round = 0; round < rounds && on; ++round) {
      const int last = round == rounds - 1 && rounds < b.maxIterT ? 1 : 0;
      for (int t = L.gl; t < nSh; t += G) w.PI[t] = pi0[t];
      const CellTerms r = ratesOf<G>(b, m, w, L, cell, te, ne, hden, [&](int t, int heavy, real heatef) {
        return heavy ? heatA[t] + heatHi[t] * heatef : heatA[t];
      });
      ++nIter;
      conv = r.conv ? 1 : 0;
      // forLines of update_mod from the cooling surfaces, an ion per lane
      if constexpr (kIons) if (!(b.converge && !conv && nIter < b.maxIterT && round + 1 < kMaxRounds && !last)) {
        CoolAt a{};
        if (L.gl == 0) a = coolStencil(te, ne);
        a.iT = __shfl_sync(L.mask, a.iT, 0, G); a.iN = __shfl_sync(L.mask, a.iN, 0, G);
        a.tT = __shfl_sync(L.mask, a.tT, 0, G); a.tN = __shfl_sync(L.mask, a.tN, 0, G);
        for (int atom = L.gl; atom < nA; atom += G) {
          const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
          const int elem = h[kAtElem];
          forSum[atom] = surfaceCooling(b, atom, a, (double)b.abun[elem] * (double)xAt(b, m, w, elem, h[kAtIon]), te, ne);
        }
      }
      __syncwarp(L.mask);
      if (L.gl == 0) {
        double coolColl = r.coolHex;
#pragma unroll 4
        for (int a = 0; a < nA; ++a) coolColl = coolColl + forSum[a];
        double heat = r.heat;
        double cool = r.coolA + coolColl + r.coolCollH;
        if (b.lgCompton) {
          heat = heat + r.compHeat * ne + r.compRecoil;
          cool = cool + r.compCool * ne;
        }
        on = secantStep(b, cell, round, last, nIter, conv != 0, heat, cool, te, k) ? 1 : 0;
      }
      te = __shfl_sync(L.mask, te, 0, G);
      on = __shfl_sync(L.mask, on, 0, G);
    }
    for (int q = L.gl; q < NP; q += G) b.ion[(size_t)q * C1 + cell] = (double)w.X[q];
    if (L.gl == 0) {
      b.te[cell] = te;
      b.ne[cell] = ne;
      b.nIterT[cell] = nIter;
      b.ibConv[cell] = (int8_t)conv;
      b.side[cell] = k.side;
      if (!on) b.state[cell] = 1;
    }
    __syncwarp(L.mask);
  }
}
#endif

// Writes the results of the cells back to the grid (FP32) and the flags.
__global__ void storeKernel(BalanceDev b, BalanceGrid g) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (cell > b.nCells) return;
  const int C1 = b.nCells + 1;
  const int8_t st = b.state[cell];
  g.black[cell] = st == 2 ? 1 : 0;
  g.nIterT[cell] = st == 2 ? 0 : b.nIterT[cell];
  if (st == 2) {
    g.converged[cell] = 0;
    atomicAdd(&b.counters->noHit, 1ull);
    return;
  }
  g.te[cell] = (float)b.te[cell];
  g.ne[cell] = (float)b.ne[cell];
  const size_t nI = (size_t)b.nstages * b.nElemUsed;
  for (size_t k = 0; k < nI; ++k) g.ionDen[k * C1 + cell] = (float)b.ion[k * C1 + cell];
  const double xH0 = b.ion[(size_t)(b.xref[1] - 1) * C1 + cell];
  const double d = (xH0 - b.xOld[cell]) / b.xOld[cell];
  const int conv = fabs(d) <= (double)b.xhiLimit ? 1 : 0;
  g.converged[cell] = conv;
  atomicAdd(&b.counters->updated, 1ull);
  if (conv) atomicAdd(&b.counters->converged, 1ull);
  atomicMax(&b.counters->maxIterT, (unsigned long long)b.nIterT[cell]);
}

#undef RF
#undef RD

constexpr int kBuildL = MCX_BAL_EXACT ? 0 : 1;

size_t ratesSmem(const BalanceDev& b, int warps) {
  return (size_t)metaDoublesOf(b) * sizeof(double) +
         (size_t)warps * kCellsPerWarp * cellSlice(b) * sizeof(real);
}

// The block size (4, 2 or 1 warps) that keeps the most warps of kernel k resident with smem(warps) of shared memory.
struct BlockShape { int warps = 0, blocksPerSM = 0; };
template <typename K, typename F>
cudaError_t bestShape(K k, F smem, BlockShape& out) {
  for (int wps : {4, 2, 1}) {
    const size_t bytes = smem(wps);
    if (bytes > kMaxRatesSmem) continue;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxRatesSmem);
    if (e != cudaSuccess) return e;
    int blocks = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, 32 * wps, bytes);
    if (e != cudaSuccess) return e;
    if (blocks * wps > out.warps * out.blocksPerSM) out = BlockShape{wps, blocks};
  }
  return cudaSuccess;
}

#if !MCX_BAL_EXACT
template <int G>
size_t cellsSmem(const BalanceDev& b, int warps) {
  return (size_t)metaDoublesOf(b) * sizeof(double) +
         (size_t)warps * (32 / G) * cellsSlice(b) * sizeof(real);
}

// Lanes a cell has (no sum depends on it).  A cell's (element, ion) pairs are shared out
// among them, its serial parts and FP64 instructions among the cells of a warp: four
// where there are hardly any pairs; 32 on small grids, where a cell's own latency
// counts, and with many pairs; else eight.  ms a balance (first iteration) with 4, 8
// and 32 lanes:
//   pairs   cells 1e3 - 3e3       1e4                 2e4                  3.6e4 - 5e4          6.9e4
//    1      0.20  0.20  0.23   0.24  0.26  0.43   0.29  0.35  0.69   0.46  0.65  1.48
//    3      0.44  0.44  0.45   0.63  0.64  0.80   0.73  0.76  1.16   0.84  1.04  2.00
//   33      2.6   1.8   1.5    2.6   1.8   1.7    3.1   2.3   3.0    4.2   3.5   5.7
//   51      1.8   1.2   1.0    4.5   3.2   2.9    6.2   4.3   4.6    8.9   6.1   7.2   13.8   9.5  12.0
//   64                         5.8   3.8   3.1    7.4   5.0   4.5   10.8   7.1   7.1   18.6  11.6  12.5
//   78      4.2   2.7   1.7                       9.4   6.2   4.9   14.6   9.3   7.8   26.3  15.9  13.8
//  102      7.8   5.0   3.2   12.0   7.4   4.6   21.9  12.5   7.6   40.8  22.7  13.3   80.4  44.3  25.3
// (64 pairs in the second iteration at 6.9e4 cells: 9.3, 5.8, 4.7.)
inline int cellLanes(const BalanceDev& b) {
  const int g = b.nPairs <= 8 ? 4 : (b.nCells < 20000 || b.nPairs >= 64 ? 32 : 8);
  return b.cellsWarps[g == 4 ? 0 : (g == 8 ? 1 : 2)] > 0 ? g : 32;
}

template <int G>
cudaError_t launchCells(const BalanceDev& b, const BalanceGrid& g, int rounds, cudaStream_t s) {
  constexpr int k = G == 4 ? 0 : (G == 8 ? 1 : 2);
  const int perBlock = b.cellsWarps[k] * (32 / G);
  const int blocks = std::max(1, std::min((b.nCells + perBlock - 1) / perBlock, b.cellsBlocks[k] * b.smCount));
  const size_t smem = cellsSmem<G>(b, b.cellsWarps[k]);
  if (b.nAtoms > 0) balanceCellsKernel<G, true><<<blocks, 32 * b.cellsWarps[k], smem, s>>>(b, g.hden, rounds);
  else balanceCellsKernel<G, false><<<blocks, 32 * b.cellsWarps[k], smem, s>>>(b, g.hden, rounds);
  return cudaGetLastError();
}

#endif

cudaError_t launch(BalanceData& bd, const BalanceGrid& g, int maxRounds, cudaStream_t s, int atomSolves) {
  BalanceDev& b = bd.dev;
  const int C = b.nCells;
  if (C <= 0) return cudaSuccess;
  const int T = 128, nb = (C + T - 1) / T;
  cudaError_t e = cudaMemsetAsync(b.counters, 0, sizeof(BalanceCounters), s);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(b.listCount, 0, sizeof(unsigned) * (kMaxRounds + 1), s);
  if (e != cudaSuccess) return e;
#if MCX_BAL_EXACT
  const double* j = g.jste;
#else
  const float* j = g.jF;
  e = cudaMemsetAsync(b.state, 2, (size_t)C + 1, s);
  if (e != cudaSuccess) return e;
  jToFloatKernel<<<dim3((C + 255) / 256, (b.nbins + kJBins - 1) / kJBins), 256, 0, s>>>(b, g.jste, g.jF);
#endif
  hitComptonKernel<<<dim3(nb, b.lgCompton ? 4 : 1), T, 0, s>>>(b, j);
  if (b.nShellsTot > 0) shellIntegralsKernel<<<(unsigned)b.nShellsTot * (unsigned)nb, T, 0, s>>>(b, j);
  loadStateKernel<<<nb, T, 0, s>>>(b, g.te, g.ne, g.ionDen);
  const int rounds = std::min(std::max(maxRounds, 1), (int)b.maxIterT);
#if !MCX_BAL_EXACT
  if (!atomSolves && b.cellsWarps[2] > 0 && (b.coolTab || b.nAtoms == 0)) {
    const int lanes = cellLanes(b);
    e = lanes == 4 ? launchCells<4>(b, g, rounds, s)
                   : (lanes == 8 ? launchCells<8>(b, g, rounds, s) : launchCells<32>(b, g, rounds, s));
    if (e != cudaSuccess) return e;
    storeKernel<<<nb, T, 0, s>>>(b, g);
    return cudaGetLastError();
  }
#else
  (void)atomSolves;
#endif
  const BlockShape sh{b.ratesWarps[kBuildL], b.ratesBlocks[kBuildL]};
  const int cellsPerBlock = sh.warps * kCellsPerWarp;
  // the per-round kernels stride over their lists with grids of resident size, so
  // the late rounds (few listed cells) do not launch a block per cell of the grid
  const int rGrid = std::max(1, std::min((C + cellsPerBlock - 1) / cellsPerBlock, sh.blocksPerSM * b.smCount));
  const int sGrid = std::max(1, std::min(nb, 8 * b.smCount));
  // round r works on the cells listed for it (the first list holds every cell
  // a packet reached; each secant step lists the cells that go on)
  for (int r = 1; r <= rounds; ++r) {
    const int last = r == rounds && rounds < b.maxIterT ? 1 : 0;
    ratesKernel<<<rGrid, 32 * sh.warps, ratesSmem(b, sh.warps), s>>>(b, g.hden, r - 1);
#if MCX_BAL_EXACT
    if (b.nAtoms > 0) eqAtomsKernel<<<dim3(eqBlocks(b, C), b.nAtoms), kEqThreads, b.eqSmem, s>>>(b, r - 1, last);
#else
    if (b.nAtoms > 0) atomsKernel<<<dim3(nb, b.nAtoms), T, 0, s>>>(b, r - 1, last);
#endif
    secantKernel<<<sGrid, T, 0, s>>>(b, r - 1, last);
  }
  storeKernel<<<nb, T, 0, s>>>(b, g);
  return cudaGetLastError();
}

#if !MCX_BAL_EXACT
// the alphaTotal tables of every (element, ion) pair and their jump flags
cudaError_t buildAlphaTable(const BalanceData& bd, float* tab, uint8_t* jump, cudaStream_t s) {
  const int pairs = bd.dev.nElemUsed * bd.dev.nstages;
  if (pairs <= 0) return cudaSuccess;
  const dim3 grid((kAlphaN + 127) / 128, pairs);
  alphaTableKernel<<<grid, 128, 0, s>>>(bd.dev, tab);
  alphaJumpKernel<<<grid, 128, 0, s>>>(bd.dev, tab, jump);
  return cudaGetLastError();
}

// the surfaces of every atom into tab (ln G) and rtab (B), [nAtoms][kCoolNNe][kCoolNTe] floats each
cudaError_t buildCoolTable(const BalanceData& bd, float* tab, float* rtab, cudaStream_t s) {
  if (bd.dev.nAtoms <= 0) return cudaSuccess;
  int first = 0;   // eqOrder: most levels first
  auto launch = [&](auto kernel, int temps, int atoms) {
    if (atoms > 0)
      kernel<<<dim3(kCoolNTe / temps, atoms, kCoolNNe / kCoolNeTile), 32 * kCoolWarps, 0, s>>>(bd.dev, first, tab, rtab);
    first += atoms;
  };
  const int32_t* atoms = bd.dev.levelAtoms;
  launch(coolNodesKernel<kMaxLevels, 4>, 8, atoms[3]);
  launch(coolNodesKernel<17, 2>, 16, atoms[2]);
  launch(coolNodesKernel<10, 1>, 32, atoms[1]);
  launch(coolNodesKernel<5, 1>, 32, atoms[0]);
  return cudaGetLastError();
}
#endif

#if MCX_BAL_EXACT
// the equilibrium kernels' grids and shared memory for a model's ions
void equilibriumShape(int nAtoms, const std::function<int(int)>& levels, BalanceDev& d) {
  d.eqMinCells = 128;
  d.eqSmem = 0;
  for (int a = 0; a < nAtoms; ++a) {
    d.eqMinCells = std::min(d.eqMinCells, eqCells(levels(a)));
    d.eqSmem = std::max(d.eqSmem, (uint32_t)(eqDoubles(levels(a)) * sizeof(double)));
  }
}
#endif

cudaError_t prepare(BalanceData& bd) {
#if MCX_BAL_EXACT
  for (const void* k : {(const void*)eqAtomsKernel, (const void*)eqForLinesKernel, (const void*)eqLineCellKernel,
                        (const void*)eqLevelSumsKernel}) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)eqMaxSmem());
    if (e != cudaSuccess) return e;
  }
#endif
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&bd.dev.smCount, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  BlockShape sh;
  e = bestShape(ratesKernel, [&](int w) { return ratesSmem(bd.dev, w); }, sh);
  if (e != cudaSuccess) return e;
  if (!sh.warps) return cudaErrorInvalidValue;
  bd.dev.ratesWarps[kBuildL] = sh.warps;
  bd.dev.ratesBlocks[kBuildL] = sh.blocksPerSM;
#if !MCX_BAL_EXACT
  BlockShape shape[3];
  const bool ions = bd.dev.nAtoms > 0;
  e = bestShape(ions ? balanceCellsKernel<4, true> : balanceCellsKernel<4, false>,
                [&](int w) { return cellsSmem<4>(bd.dev, w); }, shape[0]);
  if (e == cudaSuccess)
    e = bestShape(ions ? balanceCellsKernel<8, true> : balanceCellsKernel<8, false>,
                  [&](int w) { return cellsSmem<8>(bd.dev, w); }, shape[1]);
  if (e == cudaSuccess)
    e = bestShape(ions ? balanceCellsKernel<32, true> : balanceCellsKernel<32, false>,
                  [&](int w) { return cellsSmem<32>(bd.dev, w); }, shape[2]);
  for (int k = 0; k < 3; ++k) {
    bd.dev.cellsWarps[k] = shape[k].warps;
    bd.dev.cellsBlocks[k] = shape[k].blocksPerSM;
  }
#endif
  return e;
}

cudaError_t launchForLines(BalanceData& bd, const float* te, const float* ne, const float* ionDen,
                           const uint8_t* compute, float* forLines, cudaStream_t s) {
  BalanceDev& b = bd.dev;
  const int C1 = b.nCells + 1, T = 128, nb = (C1 + T - 1) / T;
  if (b.nAtoms <= 0) return cudaSuccess;
#if !MCX_BAL_EXACT
  if (b.coolTab && b.recTab) {
    surfaceStencilKernel<<<nb, T, 0, s>>>(b, te, ne, compute);
    forLinesSurfaceKernel<<<dim3(nb, b.nAtoms), T, 0, s>>>(b, te, ne, ionDen, compute);
  } else
#endif
#if MCX_BAL_EXACT
    eqForLinesKernel<<<dim3(eqBlocks(b, C1), b.nAtoms), kEqThreads, b.eqSmem, s>>>(b, te, ne, ionDen, compute);
#else
    forLinesAtomsKernel<<<dim3(nb, b.nAtoms), T, 0, s>>>(b, te, ne, ionDen, compute);
#endif
  forLinesSumKernel<<<nb, T, 0, s>>>(b, compute, forLines);
  return cudaGetLastError();
}

}  // namespace MCX_BAL_NS
}  // namespace mcx
