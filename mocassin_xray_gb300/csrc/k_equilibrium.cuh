// k_equilibrium.cuh - equilibrium (source/emission_mod.f90:2505-3106) of many
// (cell, ion) pairs in FP64, a block at a time.  Included by k_balance_impl.cuh
// inside the namespace of its FP64 build.
//
// What bounds it: the FP64 pipe.  GB300 does two FP64 operations a cycle and SM,
// a division takes some twenty of them and one ion of n levels takes n^2 / 2
// collision rates (a spline, an exponential, two divisions), n^3 / 3 elimination
// steps and n^2 divisions.  A thread per (cell, ion) with its matrix in local
// memory spent more on the local memory than on the arithmetic, and the ions
// with most levels (27) ran for milliseconds on a few threads while the other
// SMs had finished.  Here a block takes one ion and eqCells(n) cells, one per
// lane, with the matrices in shared memory ([row][column][cell], so that a
// warp's accesses are contiguous) and kEqThreads / eqCells(n) workers that share
// the pairs and the rows of every cell; the ions with most levels go first.
// Every operation is the sequential code's, in its order, so the bits are too;
// the divisions that share a divisor take its correctly rounded reciprocal
// (eqDivide, mcx_exact.h).
#pragma once

constexpr int kEqThreads = 256;
// cells of a block by the ion's number of levels: the most that keep its
// matrices near 100 KB, two blocks an SM
__host__ __device__ constexpr int eqCells(int n) { return n > 18 ? 16 : (n > 12 ? 32 : (n > 6 ? 64 : 128)); }
constexpr int kEqParams = 9;   // Te, 1/Te, then the spline's klo, khi, a, b, a3, b3, h^2 (klo 0 / -1: below / above the table)
__host__ __device__ constexpr size_t eqDoubles(int n) {
  // the matrix, the populations, the pivots' reciprocals, g sqrt(Te) and its reciprocal, the parameters
  return ((size_t)n * n + 4 * (size_t)n + kEqParams) * eqCells(n);
}

// One block's view of its shared memory; i, j count from 0.
struct EqBlock {
  double* sm;
  int n, cells, cell, worker, workers;
  __device__ EqBlock(double* s, int levels) : sm(s), n(levels), cells(eqCells(levels)) {
    cell = threadIdx.x % cells;
    worker = threadIdx.x / cells;
    workers = kEqThreads / cells;
  }
  __device__ __forceinline__ double& x(int i, int j) const { return sm[(i * n + j) * cells + cell]; }
  __device__ __forceinline__ double& row(int k, int i) const { return sm[(n * n + k * n + i) * cells + cell]; }
  __device__ __forceinline__ double& y(int i) const { return row(0, i); }
  __device__ __forceinline__ double& rDiag(int i) const { return row(1, i); }
  __device__ __forceinline__ double& g(int i) const { return row(2, i); }
  __device__ __forceinline__ double& rG(int i) const { return row(3, i); }
  __device__ __forceinline__ double& par(int k) const { return sm[(n * n + 4 * n + k) * cells + cell]; }
};

// The normalised level populations of this lane's cell into q.y (every thread
// of the block calls it; synchronised on return).  rec: with the recombination term.
__device__ void eqPopulations(const BalanceDev& b, int atom, const EqBlock& q, double Te, double Ne, double ionDenUp,
                              bool rec) {
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const double* D = b.atomData;
  const int n = q.n, nT = h[kAtNTemp];
  const double* A = D + h[kAtOffA];
  const double* logT = D + h[kAtOffLogT];
  const double* qom = D + h[kAtOffQom];
  const double* y2 = D + h[kAtOffY2];
  const double* g = D + h[kAtOffG];
  const double* e = D + h[kAtOffE];
  __syncthreads();   // the block's shared memory is free
  if (q.worker == 0) {
    q.par(0) = Te;
    q.par(1) = 1. / Te;
    const double log10Te = log10(Te);
    if (nT > 2) {
      const SplineAt sp = splineAt(logT, nT, log10Te);
      q.par(2) = sp.klo; q.par(3) = sp.khi;
      q.par(4) = sp.a; q.par(5) = sp.bb; q.par(6) = sp.a3; q.par(7) = sp.b3; q.par(8) = sp.hh;
    } else {
      q.par(2) = log10Te;
    }
    if (rec) {
      double alphaTotal[kMaxLevels + 1];
      recAlphas(b, h, Te, alphaTotal);
      for (int i = 1; i < n; ++i) q.y(i) = -Ne * ionDenUp * alphaTotal[i + 1];
    } else {
      for (int i = 1; i < n; ++i) q.y(i) = -Ne * ionDenUp * 0.;
    }
    q.y(0) = 1.;
  }
  if (q.worker == q.workers - 1) {
    const double sqrTe = sqrt(Te);
    for (int i = 0; i < n; ++i) {
      const double gs = g[i] * sqrTe;
      q.g(i) = gs;
      q.rG(i) = 1. / gs;
    }
  }
  __syncthreads();
  // the collision rates of the level pairs times Ne: x(i, j) = Ne qeff(j, i)
  {
    const double rTe = q.par(1);
    SplineAt sp{};
    double lt = 0.;
    if (nT > 2) {
      sp.klo = (int)q.par(2); sp.khi = (int)q.par(3);
      sp.a = q.par(4); sp.bb = q.par(5); sp.a3 = q.par(6); sp.b3 = q.par(7); sp.hh = q.par(8);
    } else {
      lt = q.par(2);
    }
    const double constant = 1.4388463, c863 = 8.63e-6;
    int p = 0;
    for (int i = 2; i <= n; ++i)
      for (int j = i; j <= n; ++j, ++p) {
        if ((p & (q.workers - 1)) != q.worker) continue;
        const double* qq = qom + (size_t)p * nT;
        double cs;
        if (nT == 1) cs = qq[0];
        else if (nT == 2) cs = qq[0] + (qq[1] - qq[0]) / (logT[1] - logT[0]) * (lt - logT[0]);
        else if (sp.klo == 0) cs = qq[0];
        else if (sp.klo < 0) cs = qq[nT - 1];
        else {
          const double* yy = y2 + (size_t)p * nT;
          cs = sp.a * qq[sp.klo - 1] + sp.bb * qq[sp.khi - 1] +
               eqDivide((sp.a3 * yy[sp.klo - 1] + sp.b3 * yy[sp.khi - 1]) * sp.hh, 6., 1. / 6.);
        }
        const int lo = i - 2, up = j - 1;
        const bool rising = e[lo] <= e[up];
        const double expFac = exp(eqDivide((rising ? e[lo] - e[up] : e[up] - e[lo]) * constant, Te, rTe));
        const double cq = c863 * cs;
        const double qLo = eqDivide(rising ? cq * expFac : cq, q.g(rising ? lo : up), q.rG(rising ? lo : up));
        const double qUp = eqDivide(rising ? cq : cq * expFac, q.g(rising ? up : lo), q.rG(rising ? up : lo));
        q.x(up, lo) = 0. + Ne * qLo;
        q.x(lo, up) = 0. + Ne * qUp;
      }
  }
  __syncthreads();
  // the diagonal: what leaves each level, in the order of the levels
  for (int i = 1 + q.worker; i < n; i += q.workers) {
    double acc = 0.;
    for (int j = 0; j < n; ++j) {
      if (j == i) continue;
      acc = acc - q.x(j, i);
      if (j < i) acc = acc - A[(size_t)i * n + j];
    }
    q.x(i, i) = acc;
  }
  __syncthreads();
  // the radiative rates into each level; the first row is the normalisation
  for (int k = q.worker; k < n * n; k += q.workers) {
    const int i = k / n, j = k - i * n;
    if (i == 0) q.x(0, j) = 1.;
    else if (j > i) q.x(i, j) = q.x(i, j) + A[(size_t)j * n + i];
  }
  if (q.worker == 0) q.rDiag(0) = 1.;
  // lured + reslv as the reference writes them (no pivoting, multipliers
  // recomputed), the forward substitution of a row with its elimination
  for (int i = 0; i < n - 1; ++i) {
    __syncthreads();
    const double d = q.x(i, i), r = q.rDiag(i), yi = q.y(i);
    for (int k = i + 1 + q.worker; k < n; k += q.workers) {
      const double xki = q.x(k, i);
      const double factor = eqDivide(xki, d, r);
      for (int j = i + 1; j < n; ++j) q.x(k, j) = q.x(k, j) - q.x(i, j) * factor;
      q.y(k) = q.y(k) - eqDivide(yi * xki, d, r);
      if (k == i + 1) q.rDiag(k) = 1. / q.x(k, k);
    }
  }
  __syncthreads();
  if (q.worker == 0) {
    q.y(n - 1) = eqDivide(q.y(n - 1), q.x(n - 1, n - 1), q.rDiag(n - 1));
    for (int k = n - 2; k >= 0; --k) {
      double acc = q.y(k);
      for (int j = k + 1; j < n; ++j) acc = acc - q.y(j) * q.x(k, j);
      q.y(k) = eqDivide(acc, q.x(k, k), q.rDiag(k));
    }
    double sumN = 0.;
    for (int i = 0; i < n; ++i) sumN = sumN + q.y(i);
    const double r = 1. / sumN;
    for (int i = 0; i < n; ++i) q.y(i) = eqDivide(q.y(i), sumN, r);
  }
  __syncthreads();
}

// The sum over the ion's lines of a(j,i) E_ji n_j m1 m2 m3 that exceed 1e-35,
// lower level outer, upper level inner, from q.y; the result is the first worker's.
__device__ double eqLines(const BalanceDev& b, int atom, const EqBlock& q, double m1, double m2, double m3) {
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const double* DD = b.atomData;
  const int n = q.n;
  const double* A = DD + h[kAtOffA];
  const double* eD = DD + h[kAtOffE];
  const double atp = DD[h[kAtOffAtp]];
  const int iup2p = h[kAtIup2p];
  for (int k = q.worker; k < n * n; k += q.workers) {
    const int i = k / n, j = k - i * n;
    if (j <= i) continue;
    double aji = A[(size_t)j * n + i];
    if (aji == 0.) continue;
    const double Eji = eD[j] - eD[i];
    if (j + 1 == iup2p && i == 0 && atp > 0.) aji = aji - atp;
    q.x(i, j) = aji * Eji * q.y(j) * m1 * m2 * m3;
  }
  __syncthreads();
  double total = 0.;
  if (q.worker == 0)
    for (int i = 0; i < n - 1; ++i)
      for (int j = i + 1; j < n; ++j)
        if (A[(size_t)j * n + i] != 0.) {
          const double f = q.x(i, j);
          if (f > RD(1.e-35)) total = total + f;
        }
  return total;
}

// forLines of update_mod for the listed cells of a round: block (x, y) takes
// cells [x eqCells, ...) of the y-th ion in the order of b.eqOrder.
__global__ void __launch_bounds__(kEqThreads) eqAtomsKernel(BalanceDev b, int round, int lastRound) {
  extern __shared__ double eqSm[];
  const int atom = b.eqOrder[blockIdx.y];
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const EqBlock q(eqSm, h[kAtNLev]);
  const unsigned cnt = b.listCount[round];
  const unsigned first = blockIdx.x * (unsigned)q.cells;
  if (first >= cnt) return;
  const unsigned li = first + q.cell;
  const CellIdx c{b.list[(size_t)(round & 1) * (b.nCells + 1) + min(li, cnt - 1u)], b.nCells + 1};
  const bool on = li < cnt && !coolingUnused(b, round, lastRound, c.cell);
  if (!__syncthreads_or(on)) return;
  const int elem = h[kAtElem], ion = h[kAtIon];
  const double x = ionAt(b, c, elem, ion);
  // forbiddenLines = fLineEm * elemAbun * ionDen * 1.9865e-16, summed where > 1e-35;
  // without the recombination term the ratio ionDen(ion+1)/ionDen(ion) is not used
  eqPopulations(b, atom, q, b.te[c.cell], b.ne[c.cell], 0., false);
  const double v = eqLines(b, atom, q, (double)b.abun[elem], x, RD(1.9865e-16));
  if (on && q.worker == 0) b.forSum[(size_t)atom * c.C1 + c.cell] = v;
}

// The emission phase's forLines (rec = .true., 1e-25 erg units), each ion's line
// total into forSum[atom][cell].
__global__ void __launch_bounds__(kEqThreads) eqForLinesKernel(BalanceDev b, const float* __restrict__ te,
                                                             const float* __restrict__ ne,
                                                             const float* __restrict__ ionDen,
                                                             const uint8_t* __restrict__ compute) {
  extern __shared__ double eqSm[];
  const int atom = b.eqOrder[blockIdx.y];
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const EqBlock q(eqSm, h[kAtNLev]);
  const int C1 = b.nCells + 1;
  const int first = blockIdx.x * q.cells;
  if (first >= C1) return;
  const int at = first + q.cell;
  const bool on = at < C1 && compute[at];
  if (!__syncthreads_or(on)) return;
  const int cell = on ? at : b.nCells;
  const int elem = h[kAtElem], ion = h[kAtIon];
  const int top = min(elem + 1, b.nstages);
  const int e = b.xref[elem];
  const double x = ionDen[((size_t)(ion - 1) * b.nElemUsed + (e - 1)) * C1 + cell];
  double up = 0.;
  if (ion < top && x > 0.) up = (double)ionDen[((size_t)ion * b.nElemUsed + (e - 1)) * C1 + cell] / x;
  eqPopulations(b, atom, q, te[cell], ne[cell], up, true);
  const double v = eqLines(b, atom, q, (double)b.abun[elem], x, RD(1.9865e9));
  if (on && q.worker == 0) b.forSum[(size_t)atom * C1 + cell] = v;
}

// One requested line's luminosity per cell (source/output_mod.f90:1943-1984,
// :410-432): blockIdx.y is the request.
__global__ void __launch_bounds__(kEqThreads) eqLineCellKernel(BalanceDev b, LineCellArgs a) {
  extern __shared__ double eqSm[];
  const int k = blockIdx.y;
  const int atom = a.req[3 * k], lo = a.req[3 * k + 1], hi = a.req[3 * k + 2];
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const EqBlock q(eqSm, h[kAtNLev]);
  const int first = blockIdx.x * q.cells + 1;
  if (first > b.nCells) return;
  const int at = first + q.cell;
  const bool inside = at <= b.nCells;
  const int cell = inside ? at : b.nCells;
  const size_t C1 = (size_t)b.nCells + 1;
  const bool on = inside && a.black[cell] < 1;
  double v = 0.;
  if (__syncthreads_or(on)) {
    const int elem = h[kAtElem], ion = h[kAtIon], nLev = h[kAtNLev];
    const int top = min(elem + 1, b.nstages);
    const int e = b.xref[elem];
    const double x = a.ionDen[((size_t)(ion - 1) * b.nElemUsed + (e - 1)) * C1 + cell];
    double up = 0.;
    if (ion < top && x > 0.) up = (double)a.ionDen[((size_t)ion * b.nElemUsed + (e - 1)) * C1 + cell] / x;
    eqPopulations(b, atom, q, a.te[cell], a.ne[cell], up, true);
    const double* A = b.atomData + h[kAtOffA];
    const double* E = b.atomData + h[kAtOffE];
    const double atp = b.atomData[h[kAtOffAtp]];
    double aji = A[(size_t)(hi - 1) * nLev + (lo - 1)];
    if (on && aji != 0.) {
      const double Eji = E[hi - 1] - E[lo - 1];
      if (hi == h[kAtIup2p] && lo == 1 && atp > 0.) aji = aji - atp;
      v = aji * Eji * q.y(hi - 1) * (double)b.abun[elem] * x * RD(1.9865e9) * (double)a.hden[cell] * a.vol[cell];
    }
  }
  if (inside && q.worker == 0) a.out[(size_t)k * C1 + cell] = v;
}

// outputGas's level sums (forbLevelSumsKernel, operation for operation) for the
// ions eqOrder[firstAtom ...], of at most 17 levels: a block's cells are whole
// groups of 32, and a warp adds up a level over a group.
__global__ void __launch_bounds__(kEqThreads) eqLevelSumsKernel(BalanceDev b, LineSumArgs a, int firstAtom) {
  static_assert(eqCells(17) % 32 == 0, "whole groups");
  extern __shared__ double eqSm[];
  const int atom = b.eqOrder[firstAtom + blockIdx.y];
  const int32_t* h = b.atomHdr + (size_t)atom * kAtHdrSize;
  const EqBlock q(eqSm, h[kAtNLev]);
  const int first = blockIdx.x * q.cells;
  if (first >= a.nGroups * 32) return;
  const int at = first + q.cell, group = at >> 5;
  const size_t C1 = (size_t)b.nCells + 1;
  const bool valid = at < a.nRange && a.black[a.cellBase + at + 1] < 1;
  const int cell = valid ? a.cellBase + at + 1 : a.cellBase + 1;
  const int elem = h[kAtElem], ion = h[kAtIon];
  const int top = min(elem + 1, b.nstages);
  const int e = b.xref[elem];
  const bool any = __syncthreads_or(valid);
  double w = 0.;
  if (any) {
    const double x = a.ionDen[((size_t)(ion - 1) * b.nElemUsed + (e - 1)) * C1 + cell];
    double up = 0.;
    if (ion < top && x > 0.) up = (double)a.ionDen[((size_t)ion * b.nElemUsed + (e - 1)) * C1 + cell] / x;
    eqPopulations(b, atom, q, a.te[cell], a.ne[cell], up, true);
    w = (double)b.abun[elem] * x * RD(1.9865e9) * (double)a.hden[cell] * a.vol[cell];
  }
  double* row = a.partial + (size_t)group * a.nEntries + a.forbBase[atom];
  for (int j = q.worker; j < q.n; j += q.workers) {
    const double v = warpSumD(valid ? q.y(j) * w : 0.);
    if ((threadIdx.x & 31) == 0 && group < a.nGroups) row[j] = v;
  }
}

// Their shared memory for the ion that needs most, of any number of levels.
inline size_t eqMaxSmem() {
  size_t m = 0;
  for (int n = 1; n <= kMaxLevels; ++n) m = std::max(m, eqDoubles(n) * sizeof(double));
  return m;
}

// Grid width of the kernels above: enough blocks for the ion with the fewest cells a block.
inline unsigned eqBlocks(const BalanceDev& b, int cells) { return (unsigned)((cells + b.eqMinCells - 1) / b.eqMinCells); }
