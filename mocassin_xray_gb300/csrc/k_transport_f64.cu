// k_transport_f64.cu - double-geometry instantiation of the transport kernel.
#include "k_transport.cuh"
#include "k_transport_launch.h"

namespace mcx {

cudaError_t launchTransportF64(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                               DevTransportCounters* cnt, uint64_t seed, uint64_t base, unsigned long long n,
                               double deltaE, const TransportLaunch& L, cudaStream_t s) {
  return launchTransportImpl<double>(g, in, out, cnt, seed, base, n, deltaE, L, s);
}

size_t parkedPacketBytesF64() { return sizeof(Packet<double>); }

cudaError_t launchTransportBatchedF64(const DevGrid& g, const DevTransportIn& in, const DevTransportOut& out,
                                      DevTransportCounters* cnt, const NebulaDesc* neb,
                                      const unsigned long long* pktBegin, int nNeb, const float* axes,
                                      const int32_t* active, const float* cdfs, const TransportLaunch& L,
                                      unsigned long long* stamps, cudaStream_t s) {
  const size_t smem = L.smem;
  cudaError_t e = allowSmem(transportKernelBatched<double>, smem);
  if (e != cudaSuccess) return e;
  e = launchGuide(g, in, s);
  if (e != cudaSuccess) return e;
  // stamps[0]: the global timer at the start; stamps[1 + b]: when nebula b's last packet finished
  stampStartKernel<<<1, 1, 0, s>>>(stamps);
  transportKernelBatched<double><<<L.blocks, L.threads, smem, s>>>(g, in, out, cnt, neb, pktBegin, nNeb, axes, active,
                                                                  cdfs,
                                                                  L.emitBatch > 0 ? L.emitBatch
                                                                                  : (L.slots > 32 ? 32 : kEmitBatch),
                                                                  L.slots,
                                                                  stamps + 1);
  return cudaGetLastError();
}

cudaError_t transportOccupancyBatchedF64(int threads, size_t smem, int* blocksPerSM) {
  const cudaError_t e = allowSmem(transportKernelBatched<double>, smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocksPerSM, transportKernelBatched<double>, threads, smem);
}

template <bool kPlane, bool kWalls>
static cudaError_t occupancyF64(int threads, size_t smem, int* blocksPerSM) {
  const cudaError_t e = allowSmem(transportKernel<double, kPlane, kWalls>, smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocksPerSM, transportKernel<double, kPlane, kWalls>, threads,
                                                       smem);
}

cudaError_t transportOccupancyF64(int threads, size_t smem, int* blocksPerSM, bool plane, bool walls) {
  if (!walls)
    return plane ? occupancyF64<true, false>(threads, smem, blocksPerSM)
                 : occupancyF64<false, false>(threads, smem, blocksPerSM);
  return plane ? occupancyF64<true, true>(threads, smem, blocksPerSM)
               : occupancyF64<false, true>(threads, smem, blocksPerSM);
}

}  // namespace mcx
