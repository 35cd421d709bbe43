// k_transport.cuh - persistent Monte Carlo packet-transport kernel.
//
// GB300 design: a warp owns 32 or 60 packet histories, in slots of shared memory,
// refilled from a device work queue with one warp-aggregated atomic.  A lane
// steps one of them (a cell step of pathSegment a loop iteration) until it interacts
// or ends, queues it for the emission code and takes up another that is ready;
// the emissions run out of line, by the whole warp, once enough of them wait
// (slotLoop).  Packet geometry and optical depth run in
// the template precision R (float: the production path; double: the plain
// FP64 path); the mean-intensity estimator J_nu is accumulated with FP64
// atomics into the Fortran-layout array Jste[nu][cell], compensated: each
// atomic's exact rounding error (TwoSum of the value it returned and the
// deposit) goes to a second array Jlo, folded in after the launch, so the
// result is the correctly rounded sum of the deposits whatever their order.  The source spectrum
// CDF, the frequency mesh and the axes' walls are staged in shared memory.
//
// Physics follows the reference routine by routine (single mother grid):
//   energyPacketDriver/energyPacketRun   source/photon_mod.f90:28-741
//   initPhotonPacket / getNu2            source/photon_mod.f90:744-972
//   newPhotonPacket                      source/photon_mod.f90:976-1756
//   pathSegment                          source/photon_mod.f90:1758-4085
//   comptonScatter                       source/photon_mod.f90:6805-6848
// Packet k of a call (global id counter_base + k) draws its uniforms from its
// own Philox4x32-10 stream, so a history does not depend on scheduling.
// Jste(0,:), the dump row the reference fills for inactive cells and never
// reads, is not accumulated.
#pragma once
#include "k_transport_launch.h"
#include "mcx_device.cuh"
#include "mcx_exact.h"
#include "mcx_fmath.h"

#include <algorithm>

namespace mcx {

enum : int { PT_STELLAR = 0, PT_DIFFUSE = 1, PT_DUSTEMI = 2 };
// ST_INTERACT: an interaction whose outcome (absorbed or scattered) is still to be drawn
enum : int { ST_IDLE = 0, ST_EMIT = 1, ST_STEP = 2, ST_DONE = 3, ST_ESCAPE = 4, ST_INTERACT = 5 };

constexpr int kSafeLimit = 500000;        // pathSegment (source/photon_mod.f90:1873-1878)
constexpr int kSafeLimitPlane = 5000;     // the same, plane-parallel ionisation
constexpr int kRecursionLimit = 100000;   // recursionLimit (source/constants_mod.f90:70)

template <typename R> struct RMath;
template <> struct RMath<float> {
  static __device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
  static __device__ __forceinline__ float log_(float x) { return logf(x); }
  static __device__ __forceinline__ float cos_(float x) { return cosf(x); }
  static __device__ __forceinline__ float sin_(float x) { return sinf(x); }
  static __device__ __forceinline__ float abs_(float x) { return fabsf(x); }
  static __device__ __forceinline__ float min_(float a, float b) { return fminf(a, b); }
  // the step's quotients: reciprocal-approximation division (2 ulp; operands far below 2^126)
  static __device__ __forceinline__ float div_(float a, float b) { return __fdividef(a, b); }
};
// the plain FP64 path: log, cos and sin from the portable routines the oracle
// uses too (mcx_fmath.h), so that both draw the same packet histories
template <> struct RMath<double> {
  static __device__ __forceinline__ double sqrt_(double x) { return sqrt(x); }
  static __device__ __forceinline__ double log_(double x) { return mcx_fm_log(x); }
  static __device__ __forceinline__ double cos_(double x) { return mcx_fm_cos(x); }
  static __device__ __forceinline__ double sin_(double x) { return mcx_fm_sin(x); }
  static __device__ __forceinline__ double abs_(double x) { return fabs(x); }
  static __device__ __forceinline__ double min_(double a, double b) { return fmin(a, b); }
  static __device__ __forceinline__ double div_(double a, double b) { return a / b; }
};

// t cos(a) and t sin(a), out of line: the accurate sine and cosine are long,
// and inlined at each direction draw they would crowd the transport loop out
// of the instruction cache.
template <typename R>
struct CosSin { R c, s; };

template <typename R>
__device__ __noinline__ CosSin<R> scaledCosSin(R t, R a) {
  using M = RMath<R>;
  return CosSin<R>{t * M::cos_(a), t * M::sin_(a)};
}

// The isotropic direction initPhotonPacket draws from the uniforms r1, r2
// (source/photon_mod.f90:858-878): w = 2 r1 - 1, t = sqrt(1 - w^2),
// phi = pi (2 r2 - 1), (t cos phi, t sin phi, w).
template <typename R>
struct Dir3 { R x, y, z; };

template <typename R>
__device__ __forceinline__ Dir3<R> isoDirection(R r1, R r2) {
  using M = RMath<R>;
  const R w = R(2) * r1 - R(1);
  const R t = M::sqrt_(R(1) - w * w);
  const R ang = R(3.141592654) * (R(2) * r2 - R(1));
  const CosSin<R> cs = scaledCosSin<R>(t, ang);
  return Dir3<R>{cs.c, cs.s, w};
}

// One lane's share of a warp history's CDF search (see warpCdfIssue).
struct WarpCdf {
  float v;          // this lane's segment end
  int seg, segs;    // segment length (a multiple of 32) and segments probed
};

template <typename R>
struct Packet {
  using Real = R;
  static constexpr bool kWarp = false;   // one lane per history
  __device__ __forceinline__ void interacts(R prob) { probSca = prob; }
  __device__ __forceinline__ Dir3<R> startDir() const { return {ex, ey, ez}; }
  R x, y, z, vx, vy, vz;
  R ex, ey, ez;     // the direction the current path segment started with (the escape tally's)
  R nu, absTau, passProb;
  R probSca;        // of the interaction in hand (ST_INTERACT)
  int xP, yP, zP, nuP, origin;
  int type, lgStellar, nEmit, nStep;
  PacketRng rng;
};

// A packet of the persistent kernel, in shared memory: Packet without what can be
// worked out again (the key and the Philox block in use; of the direction the
// segment started with, which reflections turn into v, the signs), the
// scattering probability of an interaction in hand in place of the optical depth
// drawn for the flight.  I: the type of its indices, 16 bits beside tables in shared memory
// that end long before those do, int in a batch.  An odd number of words, so that a warp's accesses
// spread over the banks; the less of it, the more L1 is left (see transportKernel).
template <typename R, typename I = uint16_t>
struct Slot {
  using Real = R;
  static constexpr bool kWarp = false;
  R x, y, z, vx, vy, vz;
  R nu, absTau, passProb;
  I xP, yP, zP, nuP;
  int origin;
  int nEmit : 20;
  unsigned type : 3, lgStellar : 1, state : 4, signs : 3;
  int nStep;
  uint32_t p0, p1, k;   // the random stream's packet id and draws taken
  __device__ __forceinline__ void interacts(R prob) { passProb = prob; }
  __device__ __forceinline__ Dir3<R> startDir() const {
    using M = RMath<R>;
    const R ax = M::abs_(vx), ay = M::abs_(vy), az = M::abs_(vz);
    return {signs & 1u ? -ax : ax, signs & 2u ? -ay : ay, signs & 4u ? -az : az};
  }
  __device__ __forceinline__ Packet<R> unpack(uint64_t seed) const {
    Packet<R> a;
    a.x = x; a.y = y; a.z = z; a.vx = vx; a.vy = vy; a.vz = vz;
    const Dir3<R> e = startDir();
    a.ex = e.x; a.ey = e.y; a.ez = e.z;
    a.nu = nu; a.absTau = absTau; a.passProb = passProb; a.probSca = passProb;
    a.xP = xP; a.yP = yP; a.zP = zP; a.nuP = nuP; a.origin = origin;
    a.type = (int)type; a.lgStellar = (int)lgStellar; a.nEmit = nEmit; a.nStep = nStep;
    a.rng.init(seed, (uint64_t)p0 | (uint64_t)p1 << 32);
    a.rng.k = k;
    if (k & 3u) {
      const uint4 b = philoxBlock(p0, p1, k >> 2, a.rng.k0, a.rng.k1);
      a.rng.buf[0] = b.x; a.rng.buf[1] = b.y; a.rng.buf[2] = b.z; a.rng.buf[3] = b.w;
    }
    return a;
  }
  __device__ __forceinline__ void pack(const Packet<R>& a) {
    x = a.x; y = a.y; z = a.z; vx = a.vx; vy = a.vy; vz = a.vz;
    signs = (a.ex < R(0) ? 1u : 0u) | (a.ey < R(0) ? 2u : 0u) | (a.ez < R(0) ? 4u : 0u);
    nu = a.nu; absTau = a.absTau; passProb = a.passProb;
    xP = (I)a.xP; yP = (I)a.yP; zP = (I)a.zP; nuP = (I)a.nuP; origin = a.origin;
    type = (unsigned)a.type; lgStellar = (unsigned)a.lgStellar; nEmit = a.nEmit; nStep = a.nStep;
    k = a.rng.k;
  }
};
static_assert(sizeof(Slot<float>) == kSlotBytesF32 && sizeof(Slot<double>) == kSlotBytesF64 &&
                  sizeof(Slot<float, int>) == kSlotBytesF32 + 8 && sizeof(Slot<double, int>) == kSlotBytesF64 + 8,
              "k_transport_launch.h");
static_assert(kRecursionLimit < 1 << 19, "Slot::nEmit");

// A history run by a whole warp (the trapped-packet kernel): outside the
// speculated events every lane holds the same state and executes the same
// scalar arithmetic, so every lane computes the same values.  Its Philox
// stream is kept across the lanes: lane l holds block blk0 + l (draws
// 4 (blk0 + l) .. 4 (blk0 + l) + 3), so one refill covers the next 128 draws.
struct WarpRng {
  uint32_t k0, k1, p0, p1;
  uint32_t k;              // draws taken so far
  uint32_t blk0;           // first Philox block held by the warp
  uint4 b;                 // this lane's block, blk0 + lane
  __device__ __forceinline__ void fill(uint32_t first) {
    blk0 = first;
    b = philoxBlock(p0, p1, first + (threadIdx.x & 31u), k0, k1);
  }
  __device__ __forceinline__ void start(const PacketRng& r) {
    k0 = r.k0; k1 = r.k1; p0 = r.p0; p1 = r.p1; k = r.k;
    fill(k >> 2);
  }
  __device__ __forceinline__ uint32_t next() {
    if ((k >> 2) - blk0 >= 32u) fill(k >> 2);
    const int src = (int)((k >> 2) - blk0);
    const uint32_t c = k & 3u;
    ++k;
    return __shfl_sync(0xffffffffu, c == 0u ? b.x : (c == 1u ? b.y : (c == 2u ? b.z : b.w)), src);
  }
};

template <typename R>
struct WarpPacket {
  using Real = R;
  static constexpr bool kWarp = true;
  __device__ __forceinline__ void interacts(R prob) { probSca = prob; }
  __device__ __forceinline__ Dir3<R> startDir() const { return {ex, ey, ez}; }
  R x, y, z, vx, vy, vz;
  R ex, ey, ez;
  R nu, absTau, passProb;
  R probSca;        // of the interaction in hand (ST_INTERACT)
  int xP, yP, zP, nuP, origin;
  int type, lgStellar, nEmit, nStep;
  WarpRng rng;
  int2 cdfShape;     // warpCdfShape(nbins), computed once per launch; (0, 0): the search of one lane
  __device__ __forceinline__ void from(const Packet<R>& a) {
    x = a.x; y = a.y; z = a.z; vx = a.vx; vy = a.vy; vz = a.vz;
    ex = a.ex; ey = a.ey; ez = a.ez;
    nu = a.nu; absTau = a.absTau; passProb = a.passProb; probSca = a.probSca;
    xP = a.xP; yP = a.yP; zP = a.zP; nuP = a.nuP; origin = a.origin;
    type = a.type; lgStellar = a.lgStellar; nEmit = a.nEmit; nStep = a.nStep;
    rng.start(a.rng);
  }
};

// Whether this lane performs the history's side effects (atomics): every lane
// of a one-lane history, lane 0 of a warp history.
template <typename P>
__device__ __forceinline__ bool effectLane() { return !P::kWarp || (threadIdx.x & 31u) == 0u; }

struct LocalCounters {
  unsigned long long crossings = 0, interactions = 0, absorptions = 0, scatterings = 0;
  unsigned long long escaped = 0, lineEscapes = 0, trapped = 0, emissions = 0, errors = 0;
  double qPhot = 0.;
  __device__ __forceinline__ void add(const LocalCounters& o) {
    crossings += o.crossings; interactions += o.interactions; absorptions += o.absorptions; scatterings += o.scatterings;
    escaped += o.escaped; lineEscapes += o.lineEscapes; trapped += o.trapped; emissions += o.emissions;
    errors += o.errors; qPhot += o.qPhot;
  }
};

// The counts that steps make, in registers: LocalCounters goes by reference to
// the out-of-line emission code and so lives in local memory, too big beside the
// packets for the L1 that is left.
struct StepCounters {
  unsigned crossings = 0, interactions = 0, escaped = 0, trapped = 0, errors = 0;
  __device__ __forceinline__ void addTo(LocalCounters& lc) const {
    lc.crossings += crossings; lc.interactions += interactions; lc.escaped += escaped; lc.trapped += trapped;
    lc.errors += errors;
  }
};

template <typename R>
struct TransportShared {
  const float* nu;           // frequency mesh (shared memory)
};

// The walls of one axis of n cells in the geometry precision, W[0] .. W[n]: the
// axis's first and last values at the ends and between them W[w], halfway
// between the centres of cells w and w + 1 (1-based), the reference's
// (A(w) + A(w+1)) / 2.  A step needs two of them per axis, the wall ahead
// before and after the wall snap; taken from the axis they cost five clamped
// loads and the sums.
template <typename R>
__host__ __device__ __forceinline__ R axisWall(const float* A, int n, int w) {
  const int lo = w > 0 ? w - 1 : 0, hi = w < n ? w : n - 1;
  return ((R)A[lo] + (R)A[hi]) / R(2);
}

// The grid a packet travels in, read through accessors so that one emit /
// step code serves both kernels: OneGrid<R, plane> reads the context's single grid from
// the kernel parameters (walls and source CDF staged in shared memory);
// NebulaGeo holds, in registers, the nebula of a batch that the packet belongs
// to (axes, active map and CDF slices of the concatenated batch arrays; the
// active map holds batch-wide cell ids).  kWalls: the walls are in shared memory.
template <typename R, bool kPlane, bool kWalls>
struct OneGrid {
  const DevGrid& g;
  const R* wX; const R* wY; const R* wZ;     // walls, [nx+1] [ny+1] [nz+1]
  const float* sCdf;
  // wall w of an axis, from W or from the axis's values A
  __device__ __forceinline__ R wall(const R* W, const float* A, int n, int w) const {
    return kWalls ? W[w] : axisWall<R>(A, n, w);
  }
  __device__ __forceinline__ int nx() const { return g.nx; }
  __device__ __forceinline__ int ny() const { return g.ny; }
  __device__ __forceinline__ int nz() const { return g.nz; }
  __device__ __forceinline__ int symmetric() const { return g.symmetric; }
  __device__ __forceinline__ float rOut() const { return g.rOut; }
  __device__ __forceinline__ R wallX(int w) const { return wall(wX, g.xAxis, g.nx, w); }
  __device__ __forceinline__ R wallY(int w) const { return wall(wY, g.yAxis, g.ny, w); }
  __device__ __forceinline__ R wallZ(int w) const { return wall(wZ, g.zAxis, g.nz, w); }
  // the axes themselves: the plane-parallel source's birth cell only
  __device__ __forceinline__ const float* X() const { return g.xAxis; }
  __device__ __forceinline__ const float* Z() const { return g.zAxis; }
  __device__ __forceinline__ const int32_t* active() const { return g.active; }
  __device__ __forceinline__ bool activeFull() const { return g.activeFull != 0; }
  // fixed per instantiation: the kernels are built with and without the
  // plane-parallel source, so that other grids carry none of its code
  __device__ __forceinline__ constexpr bool plane() const { return kPlane; }
  __device__ __forceinline__ const float* cdf() const { return sCdf; }
  __device__ __forceinline__ int starIdx(int d) const { return g.starIdx[d]; }
  __device__ __forceinline__ float starPos(int d) const { return g.starPos[d]; }
};

template <typename R>
struct NebulaGeo {
  int nx_, ny_, nz_, symmetric_;
  float rOut_;
  const float* X_; const float* Y_; const float* Z_;
  const int32_t* active_;
  const float* cdf_;
  int starIdx_[3];
  float starPos_[3];
  __device__ __forceinline__ int nx() const { return nx_; }
  __device__ __forceinline__ int ny() const { return ny_; }
  __device__ __forceinline__ int nz() const { return nz_; }
  __device__ __forceinline__ int symmetric() const { return symmetric_; }
  __device__ __forceinline__ float rOut() const { return rOut_; }
  __device__ __forceinline__ R wallX(int w) const { return axisWall<R>(X_, nx_, w); }
  __device__ __forceinline__ R wallY(int w) const { return axisWall<R>(Y_, ny_, w); }
  __device__ __forceinline__ R wallZ(int w) const { return axisWall<R>(Z_, nz_, w); }
  __device__ __forceinline__ const float* X() const { return X_; }
  __device__ __forceinline__ const float* Z() const { return Z_; }
  __device__ __forceinline__ const int32_t* active() const { return active_; }
  __device__ __forceinline__ bool activeFull() const { return false; }
  __device__ __forceinline__ constexpr bool plane() const { return false; }
  __device__ __forceinline__ const float* cdf() const { return cdf_; }
  __device__ __forceinline__ int starIdx(int d) const { return starIdx_[d]; }
  __device__ __forceinline__ float starPos(int d) const { return starPos_[d]; }
};

template <typename Geo>
__device__ __forceinline__ int activeAt(const Geo& q, int i, int j, int k) {
  if (q.activeFull()) return ((i - 1) * q.ny() + (j - 1)) * q.nz() + k;
  return __ldg(q.active() + (size_t)(i - 1) + (size_t)q.nx() * ((size_t)(j - 1) + (size_t)q.ny() * (size_t)(k - 1)));
}

// The number of leading entries <= u of a row, by bisection of [lo, hi].
template <typename R>
__device__ __forceinline__ int countCDF(const float* row, int lo, int hi, R u) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (u >= (R)row[mid]) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// getNu2 on a monotone CDF: the reference's linear scan "last i with u >= cdf(i)"
// equals the count of leading entries <= u, found here by bisection.
template <typename R>
__device__ __forceinline__ int sampleCDF(const float* cdf, int len, int nbins, R u) {
  const int lo = countCDF<R>(cdf, 0, len < nbins ? len : nbins, u);
  int nuP = lo < 1 ? 1 : lo;
  if (nuP < nbins) ++nuP;
  return nuP;
}

// The guide to the re-emission CDFs (cellCdf's accelerator): entry b of a row
// is the count of entries <= b / kGuide, so a draw u in [b, b + 1] / kGuide
// finds its own count between entries b and b + 1: one load and a bisection of
// a few entries instead of one of the whole row (ten dependent loads for 600
// bins, each an L2 round trip in the bulk phase).  Built by one block per cell
// from the row itself at each transport: it reads the CDFs once.
static __global__ void __launch_bounds__(kGuide) guideKernel(const float* __restrict__ cdf, int nbins,
                                                             uint16_t* __restrict__ guide) {
  extern __shared__ float row[];
  const float* src = cdf + (size_t)blockIdx.x * nbins;
  for (int i = threadIdx.x; i < nbins; i += kGuide) row[i] = src[i];
  __syncthreads();
  uint16_t* out = guide + (size_t)blockIdx.x * (kGuide + 1);
  out[threadIdx.x] = (uint16_t)countCDF<float>(row, 0, nbins, (float)threadIdx.x * (1.f / kGuide));
  if (threadIdx.x == 0) out[kGuide] = (uint16_t)countCDF<float>(row, 0, nbins, 1.f);
}

// getNu2 on a cell's re-emission row, through the guide where there is one.
template <typename R>
__device__ __forceinline__ int cellCdf(const DevTransportIn& in, const float* cdf, int cell, int nbins, R u) {
  const float* row = cdf + (size_t)cell * nbins;
  int lo = 0, hi = nbins;
  if (in.guide) {
    const uint16_t* gr = in.guide + (size_t)cell * (kGuide + 1);
    const int b = min((int)(u * R(kGuide)), kGuide - 1);
    lo = __ldg(gr + b);
    hi = __ldg(gr + b + 1);
  }
  lo = countCDF<R>(row, lo, hi, u);
  const int nuP = lo < 1 ? 1 : lo;
  return nuP < nbins ? nuP + 1 : nuP;
}

// sampleCDF's count for a warp history, the 32 lanes comparing in parallel:
// first the last entry of each of up to 32 segments (issued by warpCdfIssue
// as soon as the row is known, before u is drawn), then the entries of the
// one segment that holds the answer.  On a monotone row the count of entries
// <= u does not depend on the order of the comparisons, so the result equals
// the bisection's.
// the segmentation of an m-entry row (fixed for a launch)
__device__ __forceinline__ int2 warpCdfShape(int m) {
  const int seg = 32 * ((m + 1023) / 1024);
  return make_int2(seg, m / seg);
}

__device__ __forceinline__ void warpCdfIssue(WarpCdf& c, const float* __restrict__ row, int2 shape) {
  const int lane = threadIdx.x & 31;
  c.seg = shape.x;
  c.segs = shape.y;
  c.v = lane < c.segs ? __ldg(row + (size_t)(lane + 1) * c.seg - 1) : 0.f;
}

template <typename R>
__device__ __forceinline__ int warpCdfFinish(const WarpCdf& c, const float* __restrict__ row, int m, int nbins, R u) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int s = __popc(__ballot_sync(FULL, lane < c.segs && u >= (R)c.v));
  const int base = s * c.seg;
  const int end = base + c.seg < m ? base + c.seg : m;
  int lo = base;
  for (int b = base; b < end; b += 32) {
    const bool in = b + lane < end;
    const float w = in ? __ldg(row + b + lane) : 0.f;
    lo += __popc(__ballot_sync(FULL, in && u >= (R)w));
  }
  int nuP = lo < 1 ? 1 : lo;
  if (nuP < nbins) ++nuP;
  return nuP;
}

template <typename P>
__device__ __forceinline__ typename P::Real draw(P& p) { return uniformFrom<typename P::Real>(p.rng.next()); }

// a path's optical depth to the next interaction, -ln(1 - u)
template <typename P>
__device__ __forceinline__ typename P::Real drawPassProb(P& p) {
  using R = typename P::Real;
  return -RMath<R>::log_(R(1) - draw(p));
}

// locate (source/interpolation_mod.f90:49-106) on the frequency mesh or an axis
template <typename R>
__device__ __forceinline__ int locateNu(const float* xa, int n, R x) {
  if (x > (R)xa[n - 1]) return n;
  if (x < (R)xa[0]) return 0;
  int jlow = 0, jup = n + 1;
  for (int it = 0; it < 64; ++it) {
    if (jup - jlow < 1) break;
    int jm = (jup + jlow) >> 1;
    R v = (R)xa[jm - 1];
    if (v == x) return jm;
    if (x > v) { if (jlow == jm) break; jlow = jm; } else jup = jm;
  }
  return jlow;
}

// initPhotonPacket (source/photon_mod.f90:744-896): position, frequency, an
// isotropic direction (re-drawn while a component is exactly zero) and the
// octant fold for stellar packets.
template <typename R, typename Geo, typename P>
__device__ __forceinline__ void initPacket(const Geo& q, const TransportShared<R>& sh, P& p, int nuP,
                                           bool line, bool stellar, int xP, int yP, int zP) {
  using M = RMath<R>;
  p.nuP = nuP;
  p.lgStellar = stellar;
  p.nu = line ? R(0) : (R)sh.nu[nuP - 1];
  if (stellar && q.plane()) {
    // the ionising plane (source/photon_mod.f90:795-856): born on y = 0 at a
    // uniform (x, z) within the axes' span, in the cell whose walls bracket it,
    // moving along +y
    const float* X = q.X(); const float* Z = q.Z();
    const int nx = q.nx(), nz = q.nz();
    R rnd = R(1) - draw(p);
    p.x = (R)X[0] + rnd * ((R)X[nx - 1] - (R)X[0]);
    xP = locateNu<R>(X, nx, p.x);
    if (xP < nx && xP > 0 && p.x >= ((R)X[xP - 1] + (R)X[xP]) / R(2)) xP = xP + 1;
    p.y = R(0);
    yP = 1;
    rnd = R(1) - draw(p);
    p.z = (R)Z[0] + rnd * ((R)Z[nz - 1] - (R)Z[0]);
    zP = locateNu<R>(Z, nz, p.z);
    if (zP < nz && zP > 0 && p.z >= ((R)Z[zP - 1] + (R)Z[zP]) / R(2)) zP = zP + 1;
    if (xP < 1) xP = 1;
    if (zP < 1) zP = 1;
    p.vx = R(0); p.vy = R(1); p.vz = R(0);
  } else {
    for (int rep = 0; rep < 1000000; ++rep) {
      const R r1 = draw(p);
      const R r2 = draw(p);
      const Dir3<R> d = isoDirection<R>(r1, r2);
      p.vx = d.x; p.vy = d.y; p.vz = d.z;
      if (p.vx != R(0) && p.vy != R(0) && p.vz != R(0)) break;
    }
    if (q.symmetric() && stellar) {
      if (p.vx < R(0)) p.vx = -p.vx;
      if (p.vy < R(0)) p.vy = -p.vy;
      if (p.vz < R(0)) p.vz = -p.vz;
    }
  }
  p.xP = xP; p.yP = yP; p.zP = zP;
  p.ex = p.vx; p.ey = p.vy; p.ez = p.vz;
  p.origin = (xP > 0 && yP > 0 && zP > 0) ? activeAt(q, xP, yP, zP) : 0;
}

// The escape tally (e.g. source/photon_mod.f90:2293-2378): plane 0 of
// escapedPackets always; with viewing angles also plane k when the direction's
// (theta, phi) bin belongs to view k, where theta bins cover [0, pi] in 20 and
// phi bins [0, 2 pi) in totAngleBinsPhi, phi = atan(vy / vx) truncated toward
// zero and taken as 0 for vx < 1e-35 (the reference's own binning: every
// packet leaving with vx <= 0 lands in phi bin 1, and since atan spans
// (-pi/2, pi/2) the bins between pi/2 and 3 pi/2 receive nothing).  Directions in no view's
// bins have viewPointPtheta = viewPointPphi = 0, which the reference's test
// counts as a match of view 0, adding deltaE to plane 0 a second time; both
// are reproduced.
// The (theta, phi) bins of a direction, out of line (acos and atan are long
// and run once per escaping packet).
template <typename R>
__device__ __noinline__ int2 viewBins(R vx, R vy, R vz, int totPhi) {
  const R dTheta = R(3.141592654) / R(20);
  const R dPhi = (R(2) * R(3.141592654)) / (R)totPhi;
  int idirT = (int)(acos(vz) / dTheta) + 1;
  if (idirT > 20) idirT = 20;
  if (idirT < 1) idirT = 1;
  int idirP = vx < R(1.e-35) ? 0 : (int)(atan(vy / vx) / dPhi);
  if (idirP < 0) idirP = totPhi + idirP;
  idirP = idirP + 1;
  if (idirP > totPhi) idirP = totPhi;
  return make_int2(idirT, idirP);
}

template <typename R, typename P, typename Counters>
__device__ __forceinline__ void escapeTally(const DevGrid& g, const DevTransportOut& out, const P& p,
                                            double deltaE, Counters& lc) {
  ++lc.escaped;
  if (!effectLane<P>()) return;
  const size_t plane = ((size_t)g.nCells + 1) * ((size_t)g.nbins + 1);
  const size_t at = (size_t)p.origin + ((size_t)g.nCells + 1) * (size_t)p.nuP;
  if (g.nAngle > 0) {
    // the direction the segment started with: pathSegment tallies
    // enPacket%direction, not the reflected vHat (source/photon_mod.f90:1837)
    const Dir3<R> e = p.startDir();
    const int2 bins = viewBins<R>(e.x, e.y, e.z, g.totPhi);
    const int idirT = bins.x, idirP = bins.y;
    const int k = g.viewPTheta[idirT];
    if ((g.totPhi > 1 && k == g.viewPPhi[idirP]) || (g.totPhi == 1 && k > 0))
      atomicAdd(out.escaped + plane * (size_t)k + at, deltaE);
  }
  atomicAdd(out.escaped + at, deltaE);
}

// A J deposit whose rounding error is still to be added to Jlo.  The FP64
// atomic returns the value it added to; that return is consumed one deposit
// later (or when the lane goes idle), so the wait for it hides behind the
// packet's next step instead of stalling this one.
struct PendingJ {
  double old, v;
  size_t idx;
  bool on;
};

// The exact rounding error of old + v by Fast2Sum (Dekker): with |a| >= |b|,
// b - ((a + b) - a) is exact, three dependent operations where TwoSum takes
// five; the error of a rounded sum is unique, so it is TwoSum's value.  A
// deposit of the FP32 geometry has 24 bits, so the FP64 sum of an entry is exact
// until it is some 2^29 times its smallest deposit and almost every error is 0;
// only the others go to Jlo.  The transport is bound by the L2's atomics (43 G/s
// whatever the deck, dust, gas or trapped histories alike), so an atomic not
// sent is time saved (61^3 dust shell, 1e7 packets: 23.5 -> 15.0 ms).
// (exactSum, mcx_exact.h: seen from the bits.)
template <typename R>
__device__ __forceinline__ void flushJ(const DevTransportOut& out, PendingJ& pj) {
  if (pj.on) {
    pj.on = false;
    if (sizeof(R) == 4 && exactSum(pj.old, pj.v)) return;
    const double s = pj.old + pj.v;
    const bool ord = fabs(pj.old) >= fabs(pj.v);
    const double big = ord ? pj.old : pj.v, small = ord ? pj.v : pj.old;
    const double err = small - (s - big);
    if (err != 0.) {
      atomicAdd(out.jlo + pj.idx, err);
      *out.jloUsed = 1ull;
    }
  }
}

template <typename R, bool kWarp>
__device__ __forceinline__ void deposit(const DevGrid& g, const DevTransportOut& out, int cell, int nuP, R dl,
                                        R dV, R deltaE, R costheta, PendingJ& pj) {
  if (cell <= 0 || (kWarp && (threadIdx.x & 31u) != 0u)) return;
  size_t idx = (size_t)cell + ((size_t)g.nCells + 1) * (size_t)(nuP - 1);
  const double v = (double)RMath<R>::div_(dl * deltaE, dV);
  if (out.jlo) {
    flushJ<R>(out, pj);
    pj.old = atomicAdd(out.jste + idx, v);
    pj.v = v;
    pj.idx = idx;
    pj.on = true;
  } else {
    atomicAdd(out.jste + idx, v);
  }
  if (out.hEst) atomicAdd(out.hEst + idx, (double)((dl * deltaE) * costheta / dV));
}

// comptonScatter (source/photon_mod.f90:6805-6848)
template <typename R, typename P>
__device__ __forceinline__ void comptonScatter(const DevGrid& g, const TransportShared<R>& sh, P& p) {
  using M = RMath<R>;
  const float* row = g.KNcdfT + (size_t)(p.nuP - 1) * 180;
  int th = sampleCDF<R>(row, 180, g.nbins, draw(p));
  R newTheta = (R)th * R(3.141592654) / R(180);
  R u = draw(p);
  R w = R(2) * u - R(1);
  R t = M::sqrt_(R(1) - w * w);
  const CosSin<R> cs = scaledCosSin<R>(t, newTheta);
  p.vx = cs.c;
  p.vy = cs.s;
  p.vz = w;
  p.ex = p.vx; p.ey = p.vy; p.ez = p.vz;
  int thc = th > 180 ? 180 : th;
  R newNu = p.nu * (R)__ldg(g.PcompT + (size_t)(p.nuP - 1) * 180 + (thc - 1));
  int newNuP = locateNu<R>(sh.nu, g.nbins, newNu);
  if (newNuP < 1) newNuP = 1;
  p.nu = newNu;
  p.nuP = newNuP;
}

// Volume of cell `cell` in the geometry precision.
template <typename R> __device__ __forceinline__ R cellVolume(const DevGrid& g, int cell);
template <> __device__ __forceinline__ float cellVolume<float>(const DevGrid& g, int cell) { return __ldg(g.volF + cell); }
template <> __device__ __forceinline__ double cellVolume<double>(const DevGrid& g, int cell) { return __ldg(g.volD + cell); }

// The outcome of the interaction in hand: absorbed (p.type says what re-emits
// it), or not, in which case it is scattered (source/photon_mod.f90:2560-2700).
template <typename P>
__device__ __forceinline__ bool absorbs(const DevGrid& g, P& p, LocalCounters& lc) {
  using R = typename P::Real;
  const R rnd = R(1) - draw(p);
  if (g.lgDust ? !(rnd > p.probSca) : rnd <= p.probSca) { ++lc.scatterings; return false; }
  ++lc.absorptions;
  p.type = g.lgDust && !g.lgGas ? PT_DUSTEMI : PT_DIFFUSE;
  return true;
}

// energyPacketRun + newPhotonPacket: create the packet of history step p.type
// at (p.x,p.y,p.z; p.xP,p.yP,p.zP), or scatter it there.  Returns the next state.  Kept out of line:
// with the step code inlined beside it the loop body overflows the
// instruction cache (measured: 11.9 -> 9.5 ms for 1e7 packets at 41^3).
// For a warp history (P::kWarp) the re-emission CDF search is the warp's,
// its first round issued before the line draw; the same draws, the same result.
template <typename R, typename Geo, typename P>
__device__ __forceinline__ int emitBody(const DevGrid& g, const Geo& q, const DevTransportIn& in, const DevTransportOut& out,
                                        const TransportShared<R>& sh, P& p, double deltaE, LocalCounters& lc,
                                        bool scatter) {
  using M = RMath<R>;
  if (scatter && !g.lgDust) {
    comptonScatter<R>(g, sh, p);
    p.origin = activeAt(q, p.xP, p.yP, p.zP);
    p.absTau = R(0);
    p.passProb = drawPassProb(p);
    return ST_STEP;
  }
  if (!scatter) {
    if (p.nEmit >= kRecursionLimit) { ++lc.trapped; return ST_IDLE; }
    ++p.nEmit;
  }
  bool line = false;
  const bool stellar = !scatter && p.type == PT_STELLAR;
  // the frequency first, then one initPacket for every kind of emission (one
  // copy of the direction code keeps the loop within the instruction cache)
  int nuP = 0, ix = p.xP, iy = p.yP, iz = p.zP;
  if (scatter) {
    nuP = p.nuP;          // a grain scatters isotropically and keeps the frequency
  } else if (stellar) {
    nuP = sampleCDF<R>(q.cdf(), g.nbins, g.nbins, draw(p));
    ++lc.emissions;
    p.x = (R)q.starPos(0); p.y = (R)q.starPos(1); p.z = (R)q.starPos(2);
    ix = q.starIdx(0); iy = q.starIdx(1); iz = q.starIdx(2);
  } else {
    if (p.xP < 1 || p.xP > q.nx() || p.yP < 1 || p.yP > q.ny() || p.zP < 1 || p.zP > q.nz()) { ++lc.errors; return ST_IDLE; }
    int cell = activeAt(q, p.xP, p.yP, p.zP);
    if (cell <= 0) { ++lc.errors; return ST_IDLE; }
    const float* cdfTab = p.type == PT_DIFFUSE ? in.recCDFT : in.dustCDFT;
    const float* row = cdfTab ? cdfTab + (size_t)cell * g.nbins : nullptr;
    WarpCdf wc;
    if constexpr (P::kWarp) { if (row && p.cdfShape.x) warpCdfIssue(wc, row, p.cdfShape); }
    auto sample = [&](R u) {
      if constexpr (P::kWarp) {
        if (p.cdfShape.x) return warpCdfFinish<R>(wc, row, g.nbins, g.nbins, u);
      }
      return cellCdf<R>(in, cdfTab, cell, g.nbins, u);
    };
    if (p.type == PT_DIFFUSE) {
      R rnd = R(1) - draw(p);
      if (rnd <= (R)__ldg(in.totalLines + cell)) {
        line = true;
      } else {
        nuP = sample(draw(p));
        ++lc.emissions;
      }
    } else {
      nuP = sample(draw(p));
      ++lc.emissions;
    }
  }
  initPacket<R>(q, sh, p, nuP, line, stellar, ix, iy, iz);
  if (scatter) {
    p.absTau = R(0);
    p.passProb = drawPassProb(p);
    return ST_STEP;
  }
  if (stellar && p.nu >= R(1)) lc.qPhot += deltaE / (2.1799153e-11 * (double)p.nu);
  if (line) {
    ++lc.lineEscapes;
    if (p.nEmit >= kRecursionLimit) ++lc.trapped;
    return ST_IDLE;
  }
  if (!g.lgDust && p.nu < (R)g.ionEdge1) {
    escapeTally<R>(g, out, p, deltaE, lc);
    if (p.nEmit >= kRecursionLimit) ++lc.trapped;
    return ST_IDLE;
  }
  // pathSegment entry (source/photon_mod.f90:1813-1878)
  if (p.xP <= 0 || p.xP > q.nx() || p.yP <= 0 || p.yP > q.ny() || p.zP <= 0 || p.zP > q.nz()) { ++lc.errors; return ST_IDLE; }
  p.absTau = R(0);
  p.passProb = drawPassProb(p);
  p.nStep = 0;
  return ST_STEP;
}

// The same for a slot of the persistent kernel in state st (ST_EMIT, ST_INTERACT):
// the outcome of its interaction first.  A history trapped in its cell is parked
// as it stands before the emission, for the trapped-packet kernel.  Out of line,
// with the packet in registers.
template <typename R, typename Geo>
__device__ __noinline__ int emitSlot(const DevGrid& g, const Geo& q, const DevTransportIn& in, const DevTransportOut& out,
                                     const TransportShared<R>& sh, Slot<R>& slot, int st, uint64_t seed, double deltaE,
                                     LocalCounters& lc, DevTransportCounters* cnt, Packet<R>* parked,
                                     unsigned long long parkedCap, int handoffAt) {
  Packet<R> p = slot.unpack(seed);
  bool scatter = false;
  if (st == ST_INTERACT) scatter = !absorbs(g, p, lc);
  if (!scatter && handoffAt > 0 && p.nEmit >= handoffAt && p.nEmit < kRecursionLimit) {
    const unsigned long long at = atomicAdd(&cnt->handoff, 1ull);
    if (at < parkedCap) { parked[at] = p; return ST_IDLE; }
  }
  st = emitBody<R, Geo>(g, q, in, out, sh, p, deltaE, lc, scatter);
  slot.pack(p);
  return st;
}

// One axis of a step's wall geometry (pathSegment, source/photon_mod.f90:
// 1882-2084), written without branches so that the three axes' arithmetic
// interleaves; every value is the reference's expression, so the results are
// those of its branch-by-branch form.  W(w) is the axis's wall w (axisWall); a
// is a 1-based cell index.

// The wall snap: a packet moving toward the wall ahead whose coordinate is
// within 2 % of it (relative to the signed wall coordinate, as in the
// reference) is given the next cell index.
template <typename R>
__device__ __forceinline__ bool nearWall(R r, R m) {
  return RMath<R>::div_(RMath<R>::abs_(r - m), m) < R(2.e-2);
}

template <typename R, typename W>
__device__ __forceinline__ int axisSnap(W wall, int n, int a, R r, R v) {
  const bool up = v > R(0);
  const bool inside = up ? a < n : (v < R(0) && a > 1);
  const bool near = nearWall<R>(r, wall(up ? a : a - 1));
  return inside && near ? (up ? a + 1 : a - 1) : a;
}

template <typename R>
struct AxisStep { R r, v, dS; int a; bool lost; };

// The reflection at the first plane of a symmetric grid, then the distance to
// the wall ahead; a distance below 1e-5 puts the packet on that wall and in
// the next cell (lost beyond the grid's last plane).  a is the index after the snap.
template <typename R, typename W>
__device__ __forceinline__ AxisStep<R> axisDistance(W wall, int n, int a, R r, R v, bool symmetric, bool plane) {
  using M = RMath<R>;
  const R first = wall(0), last = wall(n);
  const bool refl = symmetric && r <= first;
  v = (refl && v < R(0)) ? -v : v;
  r = refl ? first : r;
  const bool pos = v > R(0), neg = v < R(0);
  const R target = wall(pos ? a : a - 1);
  const R dS = (pos || neg) ? M::div_(target - r, v) : last;
  const bool snap = (pos || neg) && M::abs_(dS) < R(1.e-5);
  AxisStep<R> o;
  o.r = snap ? target : r;
  o.v = v;
  o.dS = dS;
  o.a = snap ? (pos ? (a < n ? a + 1 : a) : (a > 1 ? a - 1 : a)) : a;
  o.lost = snap && pos && a >= n && !plane;   // a plane-parallel slab keeps it (source/photon_mod.f90:2003)
  return o;
}

// One iteration of pathSegment's main loop (source/photon_mod.f90:1880-4036);
// ST_ESCAPE when the packet leaves the grid or R_out (tallied by stepPacket).
template <typename R, typename Geo, typename P, typename Counters>
__device__ __forceinline__ int stepCore(const DevGrid& g, const Geo& q, const DevTransportIn& in,
                                          const DevTransportOut& out, const TransportShared<R>& sh, P& p,
                                          R deltaER, double deltaE, Counters& lc, PendingJ& pj) {
  using M = RMath<R>;
  const int nx = q.nx(), ny = q.ny(), nz = q.nz();
  auto X = [&](int w) { return q.wallX(w); };
  auto Y = [&](int w) { return q.wallY(w); };
  auto Z = [&](int w) { return q.wallZ(w); };
  // safeLimit: 5000 steps per segment for a plane-parallel slab (source/photon_mod.f90:1873-1878)
  if (++p.nStep > (q.plane() ? kSafeLimitPlane : kSafeLimit)) {
    ++lc.trapped;
    if (p.nEmit >= kRecursionLimit) ++lc.trapped;
    return ST_IDLE;
  }
  int xP = p.xP, yP = p.yP, zP = p.zP;
  if (xP < 1 || xP > nx || yP < 1 || yP > ny || zP < 1 || zP > nz) { ++lc.errors; return ST_IDLE; }
  R rx = p.x, ry = p.y, rz = p.z, vx = p.vx, vy = p.vy, vz = p.vz;

  // wall snap (source/photon_mod.f90:1882-1919), one axis at a time without
  // branches so that the three axes' arithmetic interleaves
  xP = axisSnap<R>(X, nx, xP, rx, vx);
  yP = axisSnap<R>(Y, ny, yP, ry, vy);
  zP = axisSnap<R>(Z, nz, zP, rz, vz);

  // the opacity and volume of the cell the snap leaves the packet in, loaded
  // here so that their latency overlaps the wall-distance arithmetic; loaded
  // again below in the rare case that a distance snap moves the index
  const size_t C1 = (size_t)g.nCells + 1;
  int cell = activeAt(q, xP, yP, zP);
  R kap = (R)__ldg(in.opacity + (size_t)cell + C1 * (size_t)(p.nuP - 1));
  R dV = cell > 0 ? cellVolume<R>(g, cell) : R(1);
  const int xS = xP, yS = yP, zS = zP;
  // the symmetric grid's reflection and the distances from the walls
  // (source/photon_mod.f90:1921-2084); with one mother grid the reference's
  // inner loop runs exactly once
  const bool sym = q.symmetric() != 0, plane = q.plane();
  const AxisStep<R> sx = axisDistance<R>(X, nx, xP, rx, vx, sym, plane);
  const AxisStep<R> sy = axisDistance<R>(Y, ny, yP, ry, vy, sym, plane);
  const AxisStep<R> sz = axisDistance<R>(Z, nz, zP, rz, vz, sym, plane);
  if (sx.lost || sy.lost || sz.lost) { if (p.nEmit >= kRecursionLimit) ++lc.trapped; return ST_IDLE; }
  rx = sx.r; vx = sx.v; xP = sx.a;
  ry = sy.r; vy = sy.v; yP = sy.a;
  rz = sz.r; vz = sz.v; zP = sz.a;
  R dSx = sx.dS, dSy = sy.dS, dSz = sz.dS;
  if (xP > nx || xP < 1 || yP > ny || yP < 1 || zP > nz || zP < 1) { ++lc.errors; return ST_IDLE; }

  // nearest wall (source/photon_mod.f90:2087-2137)
  if (M::abs_(dSx) < R(1.e-5)) dSx = X(nx);
  if (M::abs_(dSy) < R(1.e-5)) dSy = Y(ny);
  if (M::abs_(dSz) < R(1.e-5)) dSz = Z(nz);
  dSx = M::abs_(dSx); dSy = M::abs_(dSy); dSz = M::abs_(dSz);
  R dS;
  if (dSx <= R(0)) dS = M::min_(dSy, dSz);
  else if (dSy <= R(0)) dS = M::min_(dSx, dSz);
  else if (dSz <= R(0)) dS = M::min_(dSx, dSy);
  else { dS = M::min_(dSx, dSy); dS = M::min_(dS, dSz); }
  if (!(dS > R(0))) { ++lc.errors; return ST_IDLE; }

  if (xP != xS || yP != yS || zP != zS) {
    cell = activeAt(q, xP, yP, zP);
    kap = (R)__ldg(in.opacity + (size_t)cell + C1 * (size_t)(p.nuP - 1));
    dV = cell > 0 ? cellVolume<R>(g, cell) : R(1);
  }
  const R tauCell = dS * kap;
  R costheta = R(1);
  if (g.radPress && !(rx == R(0) && ry == R(0) && rz == R(0))) {
    costheta = ((rx * vx) + (ry * vy) + (rz * vz)) /
               (R(1.e10) * M::sqrt_((rx / R(1.e10)) * (rx / R(1.e10)) + (ry / R(1.e10)) * (ry / R(1.e10)) +
                                    (rz / R(1.e10)) * (rz / R(1.e10))));
  }

  int next = ST_STEP;
  if ((p.absTau + tauCell > p.passProb) && cell > 0) {
    // interaction within the cell (source/photon_mod.f90:2244-2700)
    R dlLoc = M::div_(p.passProb - p.absTau, kap);
    rx = rx + dlLoc * vx; ry = ry + dlLoc * vy; rz = rz + dlLoc * vz;
    if (q.symmetric()) {
      if (rx <= X(0)) { if (vx < R(0)) vx = -vx; rx = X(0); }
      if (ry <= Y(0)) { if (vy < R(0)) vy = -vy; ry = Y(0); }
      if (rz <= Z(0)) { if (vz < R(0)) vz = -vz; rz = Z(0); }
    }
    deposit<R, P::kWarp>(g, out, cell, p.nuP, dlLoc, dV, deltaER, costheta, pj);
    ++lc.interactions;
    // the radius only matters against an outer radius R_out > 0
    if (q.rOut() > 0.f &&
        M::sqrt_((rx / R(1.e10)) * (rx / R(1.e10)) + (ry / R(1.e10)) * (ry / R(1.e10)) +
                 (rz / R(1.e10)) * (rz / R(1.e10))) * R(1.e10) >= (R)q.rOut()) {
      return ST_ESCAPE;
    }
    // whether it scatters is drawn in a later turn, with the emissions (see emitTurn)
    R probSca = R(0);
    if (g.lgDust) probSca = (R)__ldg(in.scaOpac + (size_t)cell + C1 * (size_t)(p.nuP - 1)) / kap;
    else if (g.lgCompton) probSca = (R)__ldg(g.KNsigmaT + p.nuP - 1) * (R)__ldg(in.ne + cell) / kap;
    p.interacts(probSca);
    next = ST_INTERACT;
  } else {
    // the packet crosses the cell (source/photon_mod.f90:2703-2881)
    deposit<R, P::kWarp>(g, out, cell, p.nuP, dS, dV, deltaER, costheta, pj);
    ++lc.crossings;
    p.absTau = p.absTau + tauCell;
    rx = rx + dS * vx; ry = ry + dS * vy; rz = rz + dS * vz;
    if (dS == dSx && vx > R(0)) xP = xP + 1;
    else if (dS == dSx && vx < R(0)) xP = xP - 1;
    else if (dS == dSy && vy > R(0)) yP = yP + 1;
    else if (dS == dSy && vy < R(0)) yP = yP - 1;
    else if (dS == dSz && vz > R(0)) zP = zP + 1;
    else if (dS == dSz && vz < R(0)) zP = zP - 1;
    bool esc = false;
    if (q.plane()) {
      // plane-parallel slab (source/photon_mod.f90:3249-3611): out through the
      // y planes only, reflected at the x and z planes (the lower z plane puts
      // z at yAxis(1), as the reference does)
      if (ry < Y(0) || yP < 1) { yP = 1; esc = true; }
      if (ry > Y(ny) || yP > ny) { yP = ny; esc = true; }
      if (rx <= X(0) || xP < 1) { xP = 1; rx = X(0); vx = -vx; }
      if (rx >= X(nx) || xP > nx) { xP = nx; rx = X(nx); vx = -vx; }
      if (rz <= Z(0) || zP < 1) { zP = 1; rz = Y(0); vz = -vz; }
      if (rz >= Z(nz) || zP > nz) { zP = nz; rz = Z(nz); vz = -vz; }
      if (esc) return ST_ESCAPE;
    } else {
      if (!q.symmetric()) {
        // full-grid escape (source/photon_mod.f90:2884-3244)
        if (ry < Y(0) || yP < 1) esc = true;
        if (ry > Y(ny) || yP > ny) esc = true;
        if (rx <= X(0) || xP < 1) esc = true;
        if (rx >= X(nx) || xP > nx) esc = true;
        if (rz <= Z(0) || zP < 1) esc = true;
        if (rz >= Z(nz) || zP > nz) esc = true;
      }
      // grid boundary and mirror planes (source/photon_mod.f90:3607-3890)
      if (!esc && ((!q.symmetric() && (rx <= X(0) || ry <= Y(0) || rz <= Z(0))) ||
                   rx >= X(nx) || ry >= Y(ny) || rz >= Z(nz) || xP > nx || yP > ny || zP > nz))
        esc = true;
      if (esc) return ST_ESCAPE;
      if (q.symmetric()) {
        if (rx <= X(0) || xP < 1) { if (vx < R(0)) vx = -vx; xP = 1; rx = X(0); }
        if (ry <= Y(0) || yP < 1) { if (vy < R(0)) vy = -vy; yP = 1; ry = Y(0); }
        if (rz <= Z(0) || zP < 1) { if (vz < R(0)) vz = -vz; zP = 1; rz = Z(0); }
      }
    }
  }
  // source/photon_mod.f90:3951-4036
  if (next == ST_STEP && !q.plane() && (xP > nx || yP > ny || zP > nz)) {
    return ST_ESCAPE;
  }
  p.x = rx; p.y = ry; p.z = rz; p.vx = vx; p.vy = vy; p.vz = vz;
  p.xP = xP; p.yP = yP; p.zP = zP;
  return next;
}

// A step and, for a packet that leaves, its escape tally (one copy of it).
template <typename R, typename Geo, typename P, typename Counters>
__device__ __forceinline__ int stepPacket(const DevGrid& g, const Geo& q, const DevTransportIn& in,
                                          const DevTransportOut& out, const TransportShared<R>& sh, P& p,
                                          R deltaER, double deltaE, Counters& lc, PendingJ& pj) {
  const int st = stepCore<R>(g, q, in, out, sh, p, deltaER, deltaE, lc, pj);
  if (st != ST_ESCAPE) return st;
  escapeTally<R>(g, out, p, deltaE, lc);
  if (p.nEmit >= kRecursionLimit) ++lc.trapped;
  return ST_IDLE;
}

// one atomic per counter per warp
__device__ __forceinline__ void flushCounters(const LocalCounters& lc, DevTransportCounters* cnt) {
  const unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  auto wsum = [&](unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL, v, o);
    return v;
  };
  unsigned long long v;
  v = wsum(lc.crossings);    if (lane == 0 && v) atomicAdd(&cnt->crossings, v);
  v = wsum(lc.interactions); if (lane == 0 && v) atomicAdd(&cnt->interactions, v);
  v = wsum(lc.absorptions);  if (lane == 0 && v) atomicAdd(&cnt->absorptions, v);
  v = wsum(lc.scatterings);  if (lane == 0 && v) atomicAdd(&cnt->scatterings, v);
  v = wsum(lc.escaped);      if (lane == 0 && v) atomicAdd(&cnt->escaped, v);
  v = wsum(lc.lineEscapes);  if (lane == 0 && v) atomicAdd(&cnt->lineEscapes, v);
  v = wsum(lc.trapped);      if (lane == 0 && v) atomicAdd(&cnt->trapped, v);
  v = wsum(lc.emissions);    if (lane == 0 && v) atomicAdd(&cnt->emissions, v);
  v = wsum(lc.errors);       if (lane == 0 && v) atomicAdd(&cnt->errors, v);
  double qp = lc.qPhot;
  for (int o = 16; o > 0; o >>= 1) qp += __shfl_down_sync(FULL, qp, o);
  if (lane == 0 && qp != 0.) atomicAdd(&cnt->qPhot, qp);
}

// Emissions, with the outcomes of interactions, and cell steps take turns by
// warp: an iteration runs the emission code only once emitBatch packets wait for
// it (or no lane is stepping), else it runs one cell step of every stepping
// lane.  They are about one event in ten but long (a draw, a CDF search through
// global memory, the direction draw); run one lane at a time they would stall
// the other 31 lanes on almost every iteration.  Only the order of events
// across lanes changes, not any packet's history.
// Default where a warp has one packet a lane (else 32; the launch may choose another).
// 41^3 lognormal, 1e7 packets, one a lane: 7.5 ms at 4, 6.2 at 12, 6.12 at 16, 6.3 at 24.
constexpr int kEmitBatch = 16;

__device__ __forceinline__ bool emitTurn(int state, int emitBatch) {
  const unsigned FULL = 0xffffffffu;
  const unsigned emit = __ballot_sync(FULL, state == ST_EMIT || state == ST_INTERACT);
  const unsigned step = __ballot_sync(FULL, state == ST_STEP);
  return emit != 0u && (__popc(emit) >= emitBatch || step == 0u);
}

// Idle lanes of the warp take the next packet ids from the work queue with one
// atomic; returns this lane's id (meaningful when the lane was idle).
__device__ __forceinline__ unsigned long long refill(unsigned need, DevTransportCounters* cnt) {
  const unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  const int leader = __ffs(need) - 1;
  unsigned long long first = 0;
  if ((int)lane == leader) first = atomicAdd(&cnt->queue, (unsigned long long)__popc(need));
  first = __shfl_sync(FULL, first, leader);
  return first + (unsigned long long)__popc(need & ((1u << lane) - 1u));
}

// The three axes' walls one after another at w (kWalls = false: none); returns the end.
template <typename R, bool kWalls>
__device__ __forceinline__ R* loadWalls(const DevGrid& g, R* w) {
  if (!kWalls) return w;
  for (int i = threadIdx.x; i <= g.nx; i += blockDim.x) w[i] = axisWall<R>(g.xAxis, g.nx, i);
  w += g.nx + 1;
  for (int i = threadIdx.x; i <= g.ny; i += blockDim.x) w[i] = axisWall<R>(g.yAxis, g.ny, i);
  w += g.ny + 1;
  for (int i = threadIdx.x; i <= g.nz; i += blockDim.x) w[i] = axisWall<R>(g.zAxis, g.nz, i);
  return w + g.nz + 1;
}

// The persistent kernel.  A warp owns `slots` packets in shared memory, up to two
// a lane: a lane whose packet interacts or ends queues it for the emission code and
// goes on with one that is ready, so the steps run with all lanes, and the emissions
// by the 32 once that many wait.  What bounds it: the step's instructions (some 400, six
// FP32 divisions among them) and the latency of the opacity and of the atomics, with 32
// warps a SM at 64 registers.  Packets lie in shared memory for the lanes to take up;
// what they leave is the L1, which holds the opacity and the emission code's local
// memory, so a slot is as small as it can be and 60 a warp, not 64: blocks of eight
// warps then fit the 164 KB split (41^3 x 600 bins).  1e7 packets, 41^3 lognormal gas:
// one packet a lane 6.1 ms (15 of 32 lanes at work), slots of 84 bytes 6.3, of 68
// bytes 5.3; 48 slots 5.7.  61^3 dust shell: 13.8 -> 10.4 ms.
//
// slotLoop is that loop for a warp; Run says what a packet belongs to:
//   bool start(s, id)       packet id of the launch into slot s (false: there is none)
//   int emit(s, st)         the emission code for slot s in state st; the next state
//   void take(s)            this lane steps slot s from here on
//   int step(s)             one step of it; the next state
//   void ended(s)           the history in slot s is over
template <typename S, typename Run>
__device__ __forceinline__ void slotLoop(Run& run, S* slot, uint8_t* waitQ, int slots, int emitBatch,
                                         DevTransportCounters* cnt) {
  const unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  // the two rings of slot numbers: waiting for the emission code, ready to step
  uint8_t* readyQ = waitQ + kSlotRing;
  constexpr unsigned kRing = kSlotRing - 1;
  for (unsigned i = lane; i < (unsigned)slots; i += 32u) {
    slot[i].state = ST_IDLE;
    slot[i].nStep = 0;
    waitQ[i] = (uint8_t)i;
  }
  __syncwarp();
  unsigned wHead = 0, nWait = (unsigned)slots, rHead = 0, nReady = 0;   // the same in every lane
  int cur = -1;               // the slot this lane steps

  for (;;) {
    unsigned idle = __ballot_sync(FULL, cur < 0);
    if (idle != 0u && nReady != 0u) {
      const unsigned rank = (unsigned)__popc(idle & below);
      if (cur < 0 && rank < nReady) {
        cur = readyQ[(rHead + rank) & kRing];
        run.take(cur);
      }
      const unsigned taken = min((unsigned)__popc(idle), nReady);
      rHead += taken;
      nReady -= taken;
      idle = __ballot_sync(FULL, cur < 0);
    }
    if (nWait >= (unsigned)emitBatch || idle == FULL) {
      if (nWait == 0u) break;                    // nothing in flight, nothing left
      const unsigned m = min(nWait, 32u);
      const int s = lane < m ? (int)waitQ[(wHead + lane) & kRing] : -1;
      wHead += m;
      nWait -= m;
      int st = s >= 0 ? (int)slot[s].state : ST_DONE;
      const unsigned need = __ballot_sync(FULL, st == ST_IDLE);
      if (need) {
        const unsigned long long id = refill(need, cnt);
        if (st == ST_IDLE) {
          run.ended(s);
          st = ST_DONE;                          // the slot is given up
          if (run.start(s, id)) {
            slot[s].k = 0u;
            slot[s].type = PT_STELLAR;
            slot[s].nEmit = 0;
            st = ST_EMIT;
          }
        }
      }
      if (st == ST_EMIT || st == ST_INTERACT) st = run.emit(s, st);
      const unsigned ready = __ballot_sync(FULL, st == ST_STEP), again = __ballot_sync(FULL, st == ST_IDLE);
      if (st == ST_STEP) readyQ[(rHead + nReady + (unsigned)__popc(ready & below)) & kRing] = (uint8_t)s;
      if (st == ST_IDLE) {
        slot[s].state = ST_IDLE;
        waitQ[(wHead + nWait + (unsigned)__popc(again & below)) & kRing] = (uint8_t)s;
      }
      nReady += (unsigned)__popc(ready);
      nWait += (unsigned)__popc(again);
      __syncwarp();
      continue;
    }
    int st = ST_STEP;
    if (cur >= 0) st = run.step(cur);
    const unsigned left = __ballot_sync(FULL, st != ST_STEP);
    if (left) {
      if (st != ST_STEP) {
        slot[cur].state = (unsigned)st;
        waitQ[(wHead + nWait + (unsigned)__popc(left & below)) & kRing] = (uint8_t)cur;
        cur = -1;
      }
      nWait += (unsigned)__popc(left);
      __syncwarp();
    }
  }
}

template <typename R, bool kPlane, bool kWalls>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 4 : 1)
transportKernel(const __grid_constant__ DevGrid g, const __grid_constant__ DevTransportIn in,
                const __grid_constant__ DevTransportOut out, DevTransportCounters* cnt,
                uint64_t seed, uint64_t base, unsigned long long n, double deltaE, int emitBatch, int slots,
                Packet<R>* __restrict__ parked, unsigned long long parkedCap, int handoffAt) {
  extern __shared__ __align__(16) unsigned char smem[];
  R* sX = reinterpret_cast<R*>(smem);
  float* sNu = reinterpret_cast<float*>(loadWalls<R, kWalls>(g, sX));
  float* sCdf = sNu + g.nbins;
  for (int i = threadIdx.x; i < g.nbins; i += blockDim.x) { sNu[i] = g.nu[i]; sCdf[i] = g.srcCDF[i]; }
  __syncthreads();
  TransportShared<R> sh{sNu};
  const OneGrid<R, kPlane, kWalls> q{g, sX, sX + g.nx + 1, sX + g.nx + g.ny + 2, sCdf};
  unsigned char* mine = smem + packetStateOffset(transportTableBytes(kWalls ? g.nx + g.ny + g.nz + 3 : 0, g.nbins, sizeof(R) == 8)) +
                        (threadIdx.x >> 5) * transportWarpBytes(slots, sizeof(R) == 8);
  Slot<R>* slot = reinterpret_cast<Slot<R>*>(mine);
  const R deltaER = (R)deltaE;
  LocalCounters lc;
  StepCounters sc;
  PendingJ pj{0., 0., 0, false};
  struct Run {
    const DevGrid& g; const OneGrid<R, kPlane, kWalls>& q; const DevTransportIn& in; const DevTransportOut& out;
    const TransportShared<R>& sh; Slot<R>* slot; LocalCounters& lc; StepCounters& sc; PendingJ& pj;
    DevTransportCounters* cnt; uint64_t seed, base; unsigned long long n; double deltaE; R deltaER;
    Packet<R>* parked; unsigned long long parkedCap; int handoffAt;
    __device__ __forceinline__ bool start(int s, unsigned long long id) {
      if (id >= n) return false;
      const uint64_t pid = base + id;
      slot[s].p0 = (uint32_t)pid;
      slot[s].p1 = (uint32_t)(pid >> 32);
      return true;
    }
    __device__ __forceinline__ int emit(int s, int st) {
      return emitSlot<R>(g, q, in, out, sh, slot[s], st, seed, deltaE, lc, cnt, parked, parkedCap, handoffAt);
    }
    __device__ __forceinline__ void take(int) {}
    __device__ __forceinline__ int step(int s) { return stepPacket<R>(g, q, in, out, sh, slot[s], deltaER, deltaE, sc, pj); }
    __device__ __forceinline__ void ended(int) {}
  } run{g, q, in, out, sh, slot, lc, sc, pj, cnt, seed, base, n, deltaE, deltaER, parked, parkedCap, handoffAt};
  slotLoop(run, slot, reinterpret_cast<uint8_t*>(slot + slots), slots, emitBatch, cnt);
  flushJ<R>(out, pj);
  sc.addTo(lc);
  flushCounters(lc, cnt);
}

// ------------------------------------------------------- trapped histories
//
// A trapped history repeats one event: a re-emission, then an interaction
// within the cell it was emitted in (or the neighbour the wall snap puts it
// in).  Such an event always takes six uniforms (line, frequency, two for the
// direction, optical depth, scattering), so the draws of the next kSpec events
// are known, and so are their directions and optical depths.  The wall snap
// moves an index by the sign of the direction while the wall ahead passes the
// 2 % test, which for a position that hardly moves is a walk clamped to the run
// of passing walls around the index: its composition over the events is a scan.
// So lane e works out event e on its own, from the index the scan gives it and
// the position that the earlier lanes' displacements, added up in order, give
// it, with the step's own expressions; then it checks everything it assumed
// (snaps as predicted, an interaction, no reflection, line, scattering or
// escape).  The events before the first lane whose check fails are what the
// serial history computes, bit for bit, and are committed at once: their
// deposits are one atomic per lane.  The failing lane's emission holds too
// (what came before it does), so only its steps run serially after that.
constexpr int kSpec = 32;            // events per speculation: one per lane
constexpr int kDrawsPerEvent = 6;
// shared memory of a speculating warp: 64 Philox blocks (6 kSpec + 3 draws take 49), the displacements
template <typename R>
struct SpecShared {
  uint4 draws[64];
  R s[3][kSpec], m[3][kSpec];          // [axis][event]
};

// The clamped walk of one axis: x -> min(max(x + s, l), h).
struct Walk { int s, l, h; };
__device__ __forceinline__ Walk then(const Walk& f, const Walk& g) {   // g after f
  return Walk{f.s + g.s, min(max(f.l + g.s, g.l), g.h), min(max(f.h + g.s, g.l), g.h)};
}

// The cells an index can walk to from a while the walls it passes are near r
// (as axisSnap tests them): the run [lo, hi] of cells around it without a wall
// that is not, 32 cells each way at most.  Kept from one speculation to the next
// until one fails, since the position hardly moves (a range that no longer
// holds costs the speculation its events from there on, nothing else).
template <typename R, typename W>
__device__ __forceinline__ int2 walkRange(W wall, int n, int a, R r) {
  const int lane = (int)(threadIdx.x & 31u);
  auto passes = [&](int w) { return w >= 1 && w < n && nearWall<R>(r, wall(min(max(w, 0), n))); };
  const unsigned up = __ballot_sync(0xffffffffu, passes(a + lane));       // bit 0: the wall above a
  const unsigned dn = __ballot_sync(0xffffffffu, passes(a - 1 - lane));   // bit 0: the wall below a
  return make_int2(a - (dn == 0xffffffffu ? 32 : __ffs(~dn) - 1), a + (up == 0xffffffffu ? 32 : __ffs(~up) - 1));
}

// This lane's index offset after its event: from 0, every lane up to this one
// moves it by one in its direction unless that leaves [lo, hi] (offsets).
// Without a clamp it is the sum of the steps; with one end touched, Lindley's
// recursion, a running maximum; with both, the composed clamps.
__device__ __forceinline__ int walkTo(int lo, int hi, bool up) {
  const unsigned FULL = 0xffffffffu;
  if (lo == hi) return 0;
  const int lane = (int)(threadIdx.x & 31u);
  const int s = 2 * __popc(__ballot_sync(FULL, up) & (0xffffffffu >> (31 - lane))) - (lane + 1);
  const bool low = __any_sync(FULL, s < lo), high = __any_sync(FULL, s > hi);
  if (!low && !high) return s;
  if (low != high) {
    int m = low ? max(lo - s, 0) : max(s - hi, 0);      // how far the free walk has been beyond the end
#pragma unroll
    for (int o = 1; o < kSpec; o <<= 1) {
      const int t = __shfl_up_sync(FULL, m, o);
      if (lane >= o) m = max(m, t);
    }
    const int x = low ? s + m : s - m;
    if (!__any_sync(FULL, low ? x > hi : x < lo)) return x;
  }
  Walk w{up ? 1 : -1, lo, hi};
#pragma unroll
  for (int o = 1; o < kSpec; o <<= 1) {
    const Walk f{__shfl_up_sync(FULL, w.s, o), __shfl_up_sync(FULL, w.l, o), __shfl_up_sync(FULL, w.h, o)};
    const Walk c = then(f, w);
    if (lane >= o) w = c;
  }
  return min(max(w.s, w.l), w.h);
}

// What a warp history keeps from one speculation to the next.
struct SpecState {
  int2 x, y, z;     // the cells each axis can walk to (walkRange)
  bool fresh;       // false: to be found at the present position
};

// Up to kSpec events of a history about to be re-emitted as diffuse gas
// radiation; p moves on to where the speculation ended.  Returns the state
// there: ST_STEP with the next emission already made, or ST_EMIT; `ahead` says
// whether that emission is an ordinary one (false: the caller makes it).
template <typename R, typename Geo>
__device__ __forceinline__ int speculate(const DevGrid& g, const Geo& q, const DevTransportIn& in,
                                         const DevTransportOut& out, const TransportShared<R>& sh, WarpPacket<R>& p,
                                         R deltaER, LocalCounters& lc, PendingJ& pj, SpecShared<R>& sp, SpecState& st, bool& ahead) {
  using M = RMath<R>;
  const unsigned FULL = 0xffffffffu;
  const int lane = (int)(threadIdx.x & 31u);
  auto X = [&](int w) { return q.wallX(w); };
  auto Y = [&](int w) { return q.wallY(w); };
  auto Z = [&](int w) { return q.wallZ(w); };
  const int nx = q.nx(), ny = q.ny(), nz = q.nz();
  // this lane's six draws
  p.rng.fill(p.rng.k >> 2);
  __syncwarp();
  sp.draws[lane] = p.rng.b;
  sp.draws[lane + 32] = philoxBlock(p.rng.p0, p.rng.p1, p.rng.blk0 + 32u + (uint32_t)lane, p.rng.k0, p.rng.k1);
  __syncwarp();
  const uint32_t* d = reinterpret_cast<const uint32_t*>(sp.draws) + (p.rng.k & 3u) + kDrawsPerEvent * lane;
  const R uLine = R(1) - uniformFrom<R>(d[0]), uNu = uniformFrom<R>(d[1]);
  const Dir3<R> v = isoDirection<R>(uniformFrom<R>(d[2]), uniformFrom<R>(d[3]));
  const R pass = -M::log_(R(1) - uniformFrom<R>(d[4])), uSca = R(1) - uniformFrom<R>(d[5]);
  // the indices before and after this lane's snap
  if (!st.fresh) {
    st.x = walkRange<R>(X, nx, p.xP, p.x);
    st.y = walkRange<R>(Y, ny, p.yP, p.y);
    st.z = walkRange<R>(Z, nz, p.zP, p.z);
  }
  const int jx = walkTo(st.x.x - p.xP, st.x.y - p.xP, v.x > R(0));
  const int jy = walkTo(st.y.x - p.yP, st.y.y - p.yP, v.y > R(0));
  const int jz = walkTo(st.z.x - p.zP, st.z.y - p.zP, v.z > R(0));
  const int ox = __shfl_up_sync(FULL, jx, 1), oy = __shfl_up_sync(FULL, jy, 1), oz = __shfl_up_sync(FULL, jz, 1);
  const int x0 = p.xP + (lane ? ox : 0), y0 = p.yP + (lane ? oy : 0), z0 = p.zP + (lane ? oz : 0);
  const int x1 = p.xP + jx, y1 = p.yP + jy, z1 = p.zP + jz;
  const size_t C1 = (size_t)g.nCells + 1;
  const int cell = activeAt(q, x1, y1, z1);                    // where it interacts
  const int before = __shfl_up_sync(FULL, cell, 1);
  const int from = lane ? before : activeAt(q, x0, y0, z0);    // where it is emitted
  // the emission
  bool emits = from > 0 && p.nEmit + lane < kRecursionLimit && v.x != R(0) && v.y != R(0) && v.z != R(0);
  emits = emits && !(uLine <= (R)__ldg(in.totalLines + from));
  // the draw that rounds to 1 (FP32) is left to the serial emission: a cell that
  // emits nothing has a row without numbers but its last, and what such a draw
  // finds there depends on the order of the search
  emits = emits && uNu < R(1);
  int nuP = 1;
  if (emits) nuP = cellCdf<R>(in, in.recCDFT, from, g.nbins, uNu);
  const R nu = (R)sh.nu[nuP - 1];
  emits = emits && !(nu < (R)g.ionEdge1);
  // the interaction, from the position that the earlier lanes' displacements give
  R kap = R(1), dV = R(1), probSca = R(0);
  if (emits) {
    kap = (R)__ldg(in.opacity + (size_t)cell + C1 * (size_t)(nuP - 1));
    if (cell > 0) dV = cellVolume<R>(g, cell);
    if (g.lgCompton) probSca = (R)__ldg(g.KNsigmaT + nuP - 1) * (R)__ldg(in.ne + cell) / kap;
  }
  const R dl = M::div_(pass, kap);
  const R sx = dl * v.x, sy = dl * v.y, sz = dl * v.z;
  sp.s[0][lane] = sx; sp.s[1][lane] = sy; sp.s[2][lane] = sz;
  __syncwarp();
  {
    // each axis's sums in the events' order by one lane
    const int ax = min(lane, 2);
    R r = ax == 0 ? p.x : (ax == 1 ? p.y : p.z);
    for (int c = 0; c < kSpec; c += 8) {
      R t[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) t[e] = sp.s[ax][c + e];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const R before = r;
        r = r + t[e];
        t[e] = before;
      }
      if (lane < 3) {
#pragma unroll
        for (int e = 0; e < 8; ++e) sp.m[ax][c + e] = t[e];
      }
    }
  }
  __syncwarp();
  const R mx = sp.m[0][lane], my = sp.m[1][lane], mz = sp.m[2][lane];
  bool ok = emits && cell > 0;
  const R ex = mx + sx, ey = my + sy, ez = mz + sz;      // where it interacts
  if (ok) {
    const bool sym = q.symmetric() != 0, plane = q.plane();
    ok = axisSnap<R>(X, nx, x0, mx, v.x) == x1 && axisSnap<R>(Y, ny, y0, my, v.y) == y1 &&
         axisSnap<R>(Z, nz, z0, mz, v.z) == z1 && !(sym && (mx <= X(0) || my <= Y(0) || mz <= Z(0)));
    const AxisStep<R> a = axisDistance<R>(X, nx, x1, mx, v.x, sym, plane);
    const AxisStep<R> b = axisDistance<R>(Y, ny, y1, my, v.y, sym, plane);
    const AxisStep<R> c = axisDistance<R>(Z, nz, z1, mz, v.z, sym, plane);
    const R ax = M::abs_(a.dS), ay = M::abs_(b.dS), az = M::abs_(c.dS);
    // a distance below 1e-5 is a distance snap: left to the serial step
    ok = ok && ax >= R(1.e-5) && ay >= R(1.e-5) && az >= R(1.e-5);
    const R dS = M::min_(M::min_(ax, ay), az);
    ok = ok && dS * kap > pass;
    ok = ok && !(sym && (ex <= X(0) || ey <= Y(0) || ez <= Z(0)));
    if (q.rOut() > 0.f)
      ok = ok && !(M::sqrt_((ex / R(1.e10)) * (ex / R(1.e10)) + (ey / R(1.e10)) * (ey / R(1.e10)) +
                            (ez / R(1.e10)) * (ez / R(1.e10))) * R(1.e10) >= (R)q.rOut());
    ok = ok && uSca > probSca;
  }
  R costheta = R(1);
  if (g.radPress && !(mx == R(0) && my == R(0) && mz == R(0)))
    costheta = ((mx * v.x) + (my * v.y) + (mz * v.z)) /
               (R(1.e10) * M::sqrt_((mx / R(1.e10)) * (mx / R(1.e10)) + (my / R(1.e10)) * (my / R(1.e10)) +
                                    (mz / R(1.e10)) * (mz / R(1.e10))));
  const unsigned bad = __ballot_sync(FULL, !ok);
  const int f = bad ? __ffs(bad) - 1 : kSpec;
  if (lane < f) deposit<R, false>(g, out, cell, nuP, dl, dV, deltaER, costheta, pj);
  lc.emissions += f; lc.interactions += f; lc.absorptions += f;
  p.nEmit += f;
  p.rng.k += kDrawsPerEvent * f;
  ahead = f == kSpec;
  st.fresh = ahead;
  const int at = ahead ? kSpec - 1 : f;                  // the state before event f, or after the last
  p.x = __shfl_sync(FULL, ahead ? ex : mx, at);
  p.y = __shfl_sync(FULL, ahead ? ey : my, at);
  p.z = __shfl_sync(FULL, ahead ? ez : mz, at);
  p.xP = __shfl_sync(FULL, ahead ? x1 : x0, at);
  p.yP = __shfl_sync(FULL, ahead ? y1 : y0, at);
  p.zP = __shfl_sync(FULL, ahead ? z1 : z0, at);
  if (ahead || !__shfl_sync(FULL, (int)emits, f)) return ST_EMIT;
  // the failing lane's emission
  p.vx = p.ex = __shfl_sync(FULL, v.x, f); p.vy = p.ey = __shfl_sync(FULL, v.y, f); p.vz = p.ez = __shfl_sync(FULL, v.z, f);
  p.nuP = __shfl_sync(FULL, nuP, f);
  p.nu = __shfl_sync(FULL, nu, f);
  p.passProb = __shfl_sync(FULL, pass, f);
  p.absTau = R(0);
  p.origin = __shfl_sync(FULL, from, f);
  p.lgStellar = false;
  p.nStep = 0;
  p.nEmit += 1;
  p.rng.k += kDrawsPerEvent - 1;
  lc.emissions += 1;
  return ST_STEP;
}

// An emission of a warp history that is not speculated, out of line: the state
// is copied around the call so that the caller's stays in registers.
template <typename R, typename Geo>
__device__ __noinline__ int emitWarp(const DevGrid& g, const Geo& q, const DevTransportIn& in, const DevTransportOut& out,
                                     const TransportShared<R>& sh, WarpPacket<R>& p, double deltaE, LocalCounters& lc,
                                     bool scatter) {
  return emitBody<R, Geo>(g, q, in, out, sh, p, deltaE, lc, scatter);
}

// The trapped-packet kernel, launched after transportKernel on the same stream:
// continues every parked history to its end, one history per warp (one warp
// per block, as many blocks as are resident at once, histories handed out
// round-robin).  A trapped history is a serial chain of up to recursionLimit
// emission + step events whose length sets the launch's, so the warp runs up
// to kSpec of its events at a time (speculate); what is left runs in lockstep
// on all lanes (a grain's absorption always).
template <typename R, bool kPlane, bool kWalls>
__global__ void __launch_bounds__(32, 16)   // 16 histories per SM, 2432 at once on 152 SMs: no spills at 128 registers
transportTrappedKernel(const __grid_constant__ DevGrid g, const __grid_constant__ DevTransportIn in,
                const __grid_constant__ DevTransportOut out, DevTransportCounters* cnt, double deltaE,
                       const Packet<R>* __restrict__ parked, unsigned long long parkedCap,
                       unsigned long long warpMax) {
  const unsigned long long written = *reinterpret_cast<volatile unsigned long long*>(&cnt->handoff);
  const unsigned long long count = written < parkedCap ? written : parkedCap;
  // dust, and many more histories than resident warps: transportTrappedLanesKernel runs them
  const bool many = count > warpMax;
  if ((many && g.lgDust) || blockIdx.x >= count) return;
  extern __shared__ __align__(16) unsigned char smem[];
  SpecShared<R>& sp = *reinterpret_cast<SpecShared<R>*>(smem);
  R* sX = reinterpret_cast<R*>(smem + sizeof(SpecShared<R>));
  float* sNu = reinterpret_cast<float*>(loadWalls<R, kWalls>(g, sX));
  for (int i = threadIdx.x; i < g.nbins; i += 32) sNu[i] = g.nu[i];
  __syncwarp();
  TransportShared<R> sh{sNu};
  const OneGrid<R, kPlane, kWalls> q{g, sX, sX + g.nx + 1, sX + g.nx + g.ny + 2, g.srcCDF};
  const R deltaER = (R)deltaE;
  LocalCounters lc;
  PendingJ pj{0., 0., 0, false};
  // the first gridDim.x histories one per warp, the rest from a queue as
  // warps finish (most parked histories end within a few hundred events; a
  // trapped one runs to recursionLimit)
  const int2 cdfShape = many ? make_int2(0, 0) : warpCdfShape(g.nbins);
  for (unsigned long long i = blockIdx.x; i < count;) {
    WarpPacket<R> p;
    p.from(parked[i]);
    p.cdfShape = cdfShape;
    SpecState st{};
    int state = ST_EMIT;
    while (state == ST_EMIT || state == ST_STEP || state == ST_INTERACT) {
      bool scatter = false;
      if (state == ST_INTERACT) { scatter = !absorbs(g, p, lc); state = ST_EMIT; }
      if (state == ST_EMIT) {
        bool ahead = false;
        if (!g.lgDust && !scatter && p.type == PT_DIFFUSE) state = speculate<R>(g, q, in, out, sh, p, deltaER, lc, pj, sp, st, ahead);
        if (state == ST_EMIT && !ahead) {
          WarpPacket<R> t = p;
          LocalCounters tl;
          state = emitWarp<R>(g, q, in, out, sh, t, deltaE, tl, scatter);
          p = t;
          lc.add(tl);
        }
      } else {
        state = stepPacket<R>(g, q, in, out, sh, p, deltaER, deltaE, lc, pj);
      }
    }
    unsigned long long nxt = 0;
    if ((threadIdx.x & 31u) == 0u) nxt = gridDim.x + atomicAdd(&cnt->parkedNext, 1ull);
    i = __shfl_sync(0xffffffffu, nxt, 0);
  }
  flushJ<R>(out, pj);
  if ((threadIdx.x & 31u) != 0u) lc = LocalCounters{};   // every lane counted the same events
  flushCounters(lc, cnt);
}

// The trapped-packet kernel for dust and many parked histories (more than three
// times what the warp kernel holds resident): a grain's events are not
// speculated, so one history per lane, taken from the parked queue as lanes free
// up, with the main kernel's emission batching.  Histories in registers, event
// code inlined, the walls in shared memory.  (For gas the warp kernel is the
// faster one at any count: 28 ms against 410 for 7600 histories of the 27^3
// X-ray gas.)
template <typename R, bool kPlane, bool kWalls>
__global__ void __launch_bounds__(128)
transportTrappedLanesKernel(const __grid_constant__ DevGrid g, const __grid_constant__ DevTransportIn in,
                const __grid_constant__ DevTransportOut out, DevTransportCounters* cnt,
                            double deltaE, const Packet<R>* __restrict__ parked, unsigned long long parkedCap,
                            unsigned long long warpMax, int emitBatch) {
  const unsigned long long written = *reinterpret_cast<volatile unsigned long long*>(&cnt->handoff);
  const unsigned long long count = written < parkedCap ? written : parkedCap;
  if (count <= warpMax || !g.lgDust) return;   // transportTrappedKernel has them, one per warp
  extern __shared__ __align__(16) unsigned char smem[];
  R* sX = reinterpret_cast<R*>(smem);
  loadWalls<R, kWalls>(g, sX);
  __syncthreads();
  TransportShared<R> sh{g.nu};
  const OneGrid<R, kPlane, kWalls> q{g, sX, sX + g.nx + 1, sX + g.nx + g.ny + 2, g.srcCDF};
  const R deltaER = (R)deltaE;
  const unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  LocalCounters lc;
  PendingJ pj{0., 0., 0, false};
  Packet<R> p;
  p.nEmit = 0;
  int state = ST_IDLE;
  for (;;) {
    const unsigned need = __ballot_sync(FULL, state == ST_IDLE);
    if (need) {
      const int leader = __ffs(need) - 1;
      unsigned long long first = 0;
      if ((int)lane == leader) first = atomicAdd(&cnt->parkedNext, (unsigned long long)__popc(need));
      first = __shfl_sync(FULL, first, leader);
      const unsigned long long id = first + (unsigned long long)__popc(need & ((1u << lane) - 1u));
      if (state == ST_IDLE) {
        if (id < count) { p = parked[id]; state = ST_EMIT; }
        else state = ST_DONE;
      }
    }
    if (__ballot_sync(FULL, state != ST_DONE) == 0u) break;
    if (emitTurn(state, emitBatch)) {
      bool scatter = false;
      if (state == ST_INTERACT) { scatter = !absorbs(g, p, lc); state = ST_EMIT; }
      if (state == ST_EMIT) state = emitBody<R, OneGrid<R, kPlane, kWalls>>(g, q, in, out, sh, p, deltaE, lc, scatter);
    } else if (state == ST_STEP) {
      state = stepPacket<R>(g, q, in, out, sh, p, deltaER, deltaE, lc, pj);
    }
  }
  flushJ<R>(out, pj);
  flushCounters(lc, cnt);
}

// A batch of nebulae sharing one frequency mesh and chemistry: their cells are
// numbered batch-wide (the per-cell arrays are the concatenation of the
// nebulae's), and packet ids are handed out batch-wide, nebula b owning
// [pktBegin[b], pktBegin[b+1]).  A packet's nebula is looked up when it goes
// into a slot (bisection over the batch) and kept beside it; the lane that steps
// the slot holds that nebula's geometry, and the same emit / step code runs in it
// with its own deltaE = L*/nPhotons and its own Philox key and counter base, so
// every nebula's histories are those of a run of the nebula alone.
__device__ __forceinline__ unsigned long long globalTimerNs() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The GPU's global timer when the batched launch begins (one thread, launched
// on the same stream just before it).
static __global__ void stampStartKernel(unsigned long long* startNs) { *startNs = globalTimerNs(); }

template <typename R>
__device__ __forceinline__ NebulaGeo<R> nebulaGeo(const NebulaDesc& d, const float* axes, const int32_t* active,
                                                 const float* cdfs) {
  NebulaGeo<R> q;
  q.nx_ = d.nx; q.ny_ = d.ny; q.nz_ = d.nz; q.symmetric_ = d.symmetric; q.rOut_ = d.rOut;
  q.X_ = axes + d.axOff; q.Y_ = q.X_ + d.nx; q.Z_ = q.Y_ + d.ny;
  q.active_ = active + d.actOff;
  q.cdf_ = cdfs + d.cdfOff;
  for (int k = 0; k < 3; ++k) { q.starIdx_[k] = d.starIdx[k]; q.starPos_[k] = d.starPos[k]; }
  return q;
}

// emitSlot in the nebula that the packet belongs to.
template <typename R>
__device__ __noinline__ int emitNebulaSlot(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                                           const TransportShared<R>& sh, Slot<R, int>& slot, int st, const NebulaDesc& d,
                                           const float* axes, const int32_t* active, const float* cdfs, LocalCounters& lc) {
  const NebulaGeo<R> q = nebulaGeo<R>(d, axes, active, cdfs);
  Packet<R> p = slot.unpack(d.seed);
  bool scatter = false;
  if (st == ST_INTERACT) scatter = !absorbs(g, p, lc);
  st = emitBody<R, NebulaGeo<R>>(g, q, in, out, sh, p, d.deltaE, lc, scatter);
  slot.pack(p);
  return st;
}

// (Three blocks an SM in FP32: at four, 64 registers, the nebula's geometry spills.  48
// nebulae, 3e6 packets the largest: one packet a lane 18.5 ms, four blocks 14.1, three
// 12.9; FP64 198 -> 128.)
template <typename R>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 3 : 1)
transportKernelBatched(const __grid_constant__ DevGrid g, const __grid_constant__ DevTransportIn in,
                const __grid_constant__ DevTransportOut out, DevTransportCounters* cnt,
                       const NebulaDesc* __restrict__ neb, const unsigned long long* __restrict__ pktBegin, int nNeb,
                       const float* __restrict__ axes, const int32_t* __restrict__ active,
                       const float* __restrict__ cdfs, int emitBatch, int slots, unsigned long long* __restrict__ doneNs) {
  extern __shared__ __align__(16) unsigned char smem[];
  float* sNu = reinterpret_cast<float*>(smem);
  for (int i = threadIdx.x; i < g.nbins; i += blockDim.x) sNu[i] = g.nu[i];
  __syncthreads();
  TransportShared<R> sh{sNu};
  unsigned char* mine = smem + packetStateOffset((size_t)g.nbins * sizeof(float)) +
                        (threadIdx.x >> 5) * batchWarpBytes(slots, sizeof(R) == 8);
  Slot<R, int>* slot = reinterpret_cast<Slot<R, int>*>(mine);
  uint8_t* rings = reinterpret_cast<uint8_t*>(slot + slots);
  LocalCounters lc;
  StepCounters sc;
  struct Run {
    const DevGrid& g; const DevTransportIn& in; const DevTransportOut& out; const TransportShared<R>& sh;
    Slot<R, int>* slot; int* nebOf;       // [slots] the nebula of each slot's packet, -1: none
    LocalCounters& lc; StepCounters& sc;
    const NebulaDesc* neb; const unsigned long long* pktBegin; int nNeb;
    const float* axes; const int32_t* active; const float* cdfs;
    unsigned long long* doneNs;
    NebulaGeo<R> q;                  // of the packet this lane steps
    int mine;
    double deltaE; R deltaER;
    // the latest finish among this lane's packets of nebula stampNeb, published
    // with one atomic when the lane moves on to another nebula (packet ids, and
    // so the nebulae, are handed out in order) or leaves
    int stampNeb; unsigned long long stampNs;
    PendingJ pj;
    __device__ __forceinline__ bool start(int s, unsigned long long id) {
      if (id >= pktBegin[nNeb]) return false;
      int lo = 0, hi = nNeb - 1;      // last b with pktBegin[b] <= id
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(pktBegin + mid) <= id) lo = mid; else hi = mid - 1;
      }
      nebOf[s] = lo;
      const uint64_t pid = neb[lo].counterBase + (id - __ldg(pktBegin + lo));
      slot[s].p0 = (uint32_t)pid;
      slot[s].p1 = (uint32_t)(pid >> 32);
      return true;
    }
    __device__ __forceinline__ int emit(int s, int st) {
      return emitNebulaSlot<R>(g, in, out, sh, slot[s], st, neb[nebOf[s]], axes, active, cdfs, lc);
    }
    __device__ __forceinline__ void take(int s) {
      const int b = nebOf[s];
      if (b == mine) return;
      mine = b;
      q = nebulaGeo<R>(neb[b], axes, active, cdfs);
      deltaE = neb[b].deltaE;
      deltaER = (R)deltaE;
    }
    __device__ __forceinline__ int step(int s) { return stepPacket<R>(g, q, in, out, sh, slot[s], deltaER, deltaE, sc, pj); }
    __device__ __forceinline__ void ended(int s) {
      const int b = nebOf[s];
      if (b < 0) return;
      if (b != stampNeb) {
        if (stampNeb >= 0) atomicMax(doneNs + stampNeb, stampNs);
        stampNeb = b;
      }
      stampNs = globalTimerNs();
      nebOf[s] = -1;
    }
  } run{g, in, out, sh, slot, reinterpret_cast<int*>(rings + 2 * kSlotRing), lc, sc, neb, pktBegin, nNeb, axes, active, cdfs,
        doneNs, NebulaGeo<R>{}, -1, 0., R(0), -1, 0ull, PendingJ{0., 0., 0, false}};
  for (int i = threadIdx.x & 31; i < slots; i += 32) run.nebOf[i] = -1;
  __syncwarp();
  slotLoop(run, slot, rings, slots, emitBatch, cnt);
  if (run.stampNeb >= 0) atomicMax(doneNs + run.stampNeb, run.stampNs);
  flushJ<R>(out, run.pj);
  sc.addTo(lc);
  flushCounters(lc, cnt);
}

// The guide to the CDFs that re-emissions are drawn from (gas or grains).
inline cudaError_t launchGuide(const DevGrid& g, const DevTransportIn& in, cudaStream_t s) {
  const float* cdf = in.recCDFT && g.lgGas ? in.recCDFT : in.dustCDFT;
  if (!in.guide || !cdf) return cudaSuccess;
  guideKernel<<<(unsigned)(g.nCells + 1), kGuide, (size_t)g.nbins * sizeof(float), s>>>(cdf, g.nbins, in.guide);
  return cudaGetLastError();
}

// The single-grid launch: the persistent kernel, then, when hand-off is on,
// the trapped-packet kernel with one warp per block on every SM (as many
// blocks as are resident at once, so every parked history starts at once).
template <typename R, bool kPlane, bool kWalls>
cudaError_t launchTransportPlane(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                                DevTransportCounters* cnt, uint64_t seed, uint64_t base, unsigned long long n,
                                double deltaE, const TransportLaunch& L, cudaStream_t s) {
  const size_t smem = L.smem;
  cudaError_t e = allowSmem(transportKernel<R, kPlane, kWalls>, smem);
  if (e != cudaSuccess) return e;
  e = launchGuide(g, in, s);
  if (e != cudaSuccess) return e;
  const bool hand = L.parked != nullptr && L.parkedCap > 0 && L.handoffAt > 0 && L.numSMs > 0;
  transportKernel<R, kPlane, kWalls><<<L.blocks, L.threads, smem, s>>>(g, in, out, cnt, seed, base, n, deltaE,
                                                       L.emitBatch > 0 ? L.emitBatch : (L.slots > 32 ? 32 : kEmitBatch),
                                                       L.slots, hand ? static_cast<Packet<R>*>(L.parked) : nullptr,
                                                       hand ? L.parkedCap : 0ull, hand ? L.handoffAt : 0);
  e = cudaGetLastError();
  if (e != cudaSuccess || !hand) return e;
  // the continuation kernel: one history per warp; for dust also the kernel with
  // one per lane, each reading the parked count on the device and only one working
  int perSM = 0, lanesPerSM = 0;
  const size_t wallBytes = (size_t)L.walls * sizeof(R);
  const size_t trappedSmem = sizeof(SpecShared<R>) + wallBytes + (size_t)g.nbins * sizeof(float);
  e = allowSmem(transportTrappedKernel<R, kPlane, kWalls>, trappedSmem);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, transportTrappedKernel<R, kPlane, kWalls>, 32, trappedSmem);
  if (e != cudaSuccess) return e;
  if (perSM < 1) perSM = 1;
  const unsigned long long warpSlots = (unsigned long long)L.numSMs * perSM;
  const unsigned long long warpMax = 3 * warpSlots;
  transportTrappedKernel<R, kPlane, kWalls><<<(unsigned)warpSlots, 32, trappedSmem, s>>>(g, in, out, cnt, deltaE,
                                                               static_cast<const Packet<R>*>(L.parked), L.parkedCap,
                                                               warpMax);
  e = cudaGetLastError();
  if (e != cudaSuccess || !g.lgDust) return e;
  e = allowSmem(transportTrappedLanesKernel<R, kPlane, kWalls>, wallBytes);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&lanesPerSM, transportTrappedLanesKernel<R, kPlane, kWalls>, 128, wallBytes);
  if (e != cudaSuccess) return e;
  transportTrappedLanesKernel<R, kPlane, kWalls><<<L.numSMs * std::max(lanesPerSM, 1), 128, wallBytes, s>>>(
      g, in, out, cnt, deltaE, static_cast<const Packet<R>*>(L.parked), L.parkedCap, warpMax,
      L.emitBatch > 0 ? L.emitBatch : kEmitBatch);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launchTransportImpl(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                                DevTransportCounters* cnt, uint64_t seed, uint64_t base, unsigned long long n,
                                double deltaE, const TransportLaunch& L, cudaStream_t s) {
  if constexpr (sizeof(R) == 8) {
    if (L.walls == 0)
      return g.plane ? launchTransportPlane<R, true, false>(g, in, out, cnt, seed, base, n, deltaE, L, s)
                     : launchTransportPlane<R, false, false>(g, in, out, cnt, seed, base, n, deltaE, L, s);
  }
  return g.plane ? launchTransportPlane<R, true, true>(g, in, out, cnt, seed, base, n, deltaE, L, s)
                 : launchTransportPlane<R, false, true>(g, in, out, cnt, seed, base, n, deltaE, L, s);
}

}  // namespace mcx
