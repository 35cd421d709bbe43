// k_transport_launch.h - host-side launchers of the transport kernel
// instantiations (k_transport_f32.cu, k_transport_f64.cu).
#pragma once
#include "mcx_device.cuh"

namespace mcx {

// Shared memory of the persistent kernel's tables: the axes' walls in the
// geometry precision (walls = 0: not in shared memory), the frequency mesh and the source CDF.
__host__ __device__ constexpr size_t transportTableBytes(int walls, int nbins, bool fp64) {
  return (size_t)walls * (fp64 ? 8 : 4) + (size_t)nbins * 2 * sizeof(float);
}

__host__ __device__ constexpr size_t packetStateOffset(size_t tableBytes) { return (tableBytes + 15) / 16 * 16; }

// After them a warp's packets (slots of the persistent kernel, 32 or kMaxSlots a
// warp) and its two rings of slot numbers.
constexpr int kMaxSlots = 60, kSlotRing = 64;
constexpr size_t kSlotBytesF32 = 68, kSlotBytesF64 = 104;
__host__ __device__ constexpr size_t transportWarpBytes(int slots, bool fp64) {
  return (slots * (fp64 ? kSlotBytesF64 : kSlotBytesF32) + 2 * kSlotRing + 7) / 8 * 8;
}
// In a batch, with indices of 32 bits and the nebula of each slot.
__host__ __device__ constexpr size_t batchWarpBytes(int slots, bool fp64) {
  return (transportWarpBytes(slots, fp64) + slots * 12 + 7) / 8 * 8;
}

struct TransportLaunch {
  int blocks;
  int threads;
  size_t smem;     // transportShape's
  int slots;       // packets of a warp
  int walls;       // walls in shared memory: all the axes', or 0 (see transportShape)
  int emitBatch;   // 0 = the kernel's default
  // Trapped-packet hand-off (single-grid kernel only): a packet about to be
  // re-emitted for the handoffAt-th time is parked in `parked` (room for
  // parkedCap packets) and continued by the trapped-packet kernel launched
  // right after; handoffAt = 0 or parked = null keeps every packet in place.
  void* parked;
  unsigned long long parkedCap;
  int handoffAt;
  int numSMs;
};

cudaError_t launchTransportF32(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                               DevTransportCounters* cnt, uint64_t seed, uint64_t base, unsigned long long n,
                               double deltaE, const TransportLaunch& L, cudaStream_t s);
cudaError_t launchTransportF64(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                               DevTransportCounters* cnt, uint64_t seed, uint64_t base, unsigned long long n,
                               double deltaE, const TransportLaunch& L, cudaStream_t s);
// The batch kernel: every nebula's packets in one launch (pktBegin[nNeb] = total).
cudaError_t launchTransportBatchedF32(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                                      DevTransportCounters* cnt, const NebulaDesc* neb,
                                      const unsigned long long* pktBegin, int nNeb, const float* axes,
                                      const int32_t* active, const float* cdfs, const TransportLaunch& L,
                                      unsigned long long* stamps, cudaStream_t s);
cudaError_t launchTransportBatchedF64(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                                      DevTransportCounters* cnt, const NebulaDesc* neb,
                                      const unsigned long long* pktBegin, int nNeb, const float* axes,
                                      const int32_t* active, const float* cdfs, const TransportLaunch& L,
                                      unsigned long long* stamps, cudaStream_t s);
cudaError_t transportOccupancyBatchedF32(int threads, size_t smem, int* blocksPerSM);
cudaError_t transportOccupancyBatchedF64(int threads, size_t smem, int* blocksPerSM);

// Bytes of one parked packet of the FP32 / FP64 kernel.
size_t parkedPacketBytesF32();
size_t parkedPacketBytesF64();

// Resident blocks per SM of the FP64 (fp64 = true) or FP32 instantiation of
// the persistent kernel (smem: transportShape's), with or without the plane-parallel source.
cudaError_t transportOccupancyF32(int threads, size_t smem, int* blocksPerSM, bool plane);
cudaError_t transportOccupancyF64(int threads, size_t smem, int* blocksPerSM, bool plane, bool walls);

inline cudaError_t transportOccupancy(bool fp64, int threads, size_t smem, int* blocksPerSM, bool plane, bool walls) {
  return fp64 ? transportOccupancyF64(threads, smem, blocksPerSM, plane, walls)
              : transportOccupancyF32(threads, smem, blocksPerSM, plane);
}

// Slots, shared memory and blocks of a transport launch (batch: transportKernelBatched, whose
// table is the mesh alone) over axes with `walls` walls in all for n packets in blocks of
// L.threads, at most gridMult blocks a SM (0: what is resident): kMaxSlots packets a
// warp where there are several times that many and they fit beside the tables, else
// one a lane.  FP64 walls take twice the room of the axes' values; where not even 32
// slots fit beside them (24 000 cells along the axes, 300 bins), the FP64 kernels work
// the walls out from the axes.
inline cudaError_t transportShape(TransportLaunch& L, bool fp64, bool plane, int walls, int nbins, int numSMs,
                                  unsigned long long n, int gridMult, bool batch = false) {
  auto smem = [&](int slots) {
    return packetStateOffset(batch ? (size_t)nbins * sizeof(float) : transportTableBytes(L.walls, nbins, fp64)) +
           L.threads / 32 * (batch ? batchWarpBytes(slots, fp64) : transportWarpBytes(slots, fp64));
  };
  L.walls = batch ? 0 : walls;
  if (fp64 && smem(32) > kMaxBlockSmem) L.walls = 0;
  for (L.slots = kMaxSlots;; L.slots = 32) {
    L.smem = smem(L.slots);
    if (L.slots > 32 && L.smem > kMaxBlockSmem) continue;
    int perSM = 0;
    const cudaError_t e = batch ? (fp64 ? transportOccupancyBatchedF64(L.threads, L.smem, &perSM)
                                        : transportOccupancyBatchedF32(L.threads, L.smem, &perSM))
                                : transportOccupancy(fp64, L.threads, L.smem, &perSM, plane, L.walls > 0);
    if (e != cudaSuccess) return e;
    if (perSM < 1) perSM = 1;
    L.blocks = numSMs * (gridMult > 0 && gridMult < perSM ? gridMult : perSM);
    if (L.slots == 32 || n >= 4ull * (unsigned long long)L.blocks * (unsigned long long)L.threads) break;
  }
  const unsigned long long most = (n + L.threads - 1) / L.threads;
  if (n > 0 && (unsigned long long)L.blocks > most) L.blocks = (int)most;
  return cudaSuccess;
}

}  // namespace mcx
