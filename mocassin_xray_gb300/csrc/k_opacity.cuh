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
  const uint8_t* termOpen;    // bit q: bin q of the group is one of the shell's
  const int32_t* slotPlane;   // [nSlots] ionDen plane (xref-1) + nElemUsed*(ion-1)
  const float* slotAbun;      // [nSlots] elemAbun of the slot's element
  const float* slotFFWeight;  // [nSlots] weight of the slot in the free-free electron sum
};

cudaError_t launchOpacity(const OpacityDev& t, const float* hden, const float* te, const float* ne,
                          const float* ionDen, const float* gauntTe, const uint8_t* compute, float* opacity,
                          cudaStream_t stream);

// The skip rule of the opacity and emission loops (source/iteration_mod.f90:131-149,
// :340-356): mask[c] = 1 for the cells to compute, those whose Te or Ne moved by
// at least 0.5 % since the last iteration (every cell when first is set).
// counts[0], counts[1]: cells computed and skipped.
cudaError_t launchSkipMask(const float* te, const float* ne, const float* teOld, const float* neOld, int nCells,
                           bool first, uint8_t* mask, unsigned long long* counts, cudaStream_t stream);

// BoltGaunt's cache (source/ionization_mod.f90:171-175) replayed over the
// computed cells in processing order, from temperature state[b] of grid b:
// gauntTe[c] is the temperature cell c's factors are tabulated at (0 for
// skipped cells) and state[b] the one the grid ends with.  order: the cells in
// processing order (null: 1 .. nCells); grid b's are [gridOff[b], gridOff[b + 1])
// of it (null: one grid of all).  scratch: 3 gauntReplayChunks floats.
int gauntReplayChunks(int nGrids, int nOrdered);
cudaError_t launchGauntReplay(const float* te, const uint8_t* mask, const int32_t* order, const int32_t* gridOff,
                              int nGrids, int nOrdered, float* state, float* scratch, float* gauntTe,
                              cudaStream_t stream);

}  // namespace mcx
