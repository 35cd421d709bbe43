// k_opacity.cuh - device tables of the opacity kernel (see k_opacity.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace mcx {

constexpr int kOpBins = 8;    // bins a thread sums at a time

struct OpacityDev {
  int32_t nbins, nCells, nXsec, lgCompton, nSlots, bremsP0;
  const float* nu;            // [nbins]
  const float* log10nu;       // [nbins] log10(nuArray) as the reference's log10nuArray
  const float* xsec;          // [nXsec]
  const float* KNsigmaT;      // [nbins]
  // bound-free terms of the kOpBins bins of group q in [termStart[q], termStart[q+1]),
  // in the summation order: the term's ion slot and its cross section at each
  // bin of the group (0 where the shell is closed)
  const int32_t* termStart;   // [groups+1]
  const int32_t* termSlot;
  const float4* termXs;       // [terms][kOpBins / 4]
  const int32_t* slotPlane;   // [nSlots] ionDen plane (xref-1) + nElemUsed*(ion-1)
  const float* slotAbun;      // [nSlots] elemAbun of the slot's element
  const float* slotFFWeight;  // [nSlots] weight of the slot in the free-free electron sum
};

cudaError_t launchOpacity(const OpacityDev& t, const float* hden, const float* te, const float* ne,
                          const float* ionDen, const float* gauntTe, const uint8_t* compute, float* opacity,
                          cudaStream_t stream);

}  // namespace mcx
