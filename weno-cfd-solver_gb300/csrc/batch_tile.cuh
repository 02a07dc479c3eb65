// Definitions of StageTile (batch_api.h): the fused stage kernel of one tile shape.
#pragma once

#include "batch_api.h"
#include "batch_kernels.cuh"

namespace weno {

inline namespace WENO_TU_NS {
namespace tdetail {

template <class T, bool FAST, bool CHAR, bool BLEND, int TX, int TY>
cudaError_t launch_stage(const SolveDesc* solves, SolveCtl* ctl, const int4* tiles, int ntiles, int grid,
                         const CUtensorMap* tmaps, const T* qn, T* qo, int stage, T gamma, T jp_lo, T jp_hi, T weps,
                         int skip_tile, unsigned long long wait_ns, cudaStream_t st) {
  constexpr size_t sm = tile_smem<T, TX, TY, BLEND>();
  if constexpr (sm > 227 * 1024) {
    return cudaErrorInvalidConfiguration;
  } else {
    auto k = k_stage_tiles<T, FAST, CHAR, BLEND, TX, TY, kTileThreads>;
    // The attribute is per device and cheap to set: set it on every launch (also
    // keeps host threads from racing on a cached flag).
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k<<<grid, kTileThreads, sm, st>>>(solves, ctl, tiles, ntiles, tmaps, qn, qo, stage, gamma, jp_lo, jp_hi, weps, skip_tile,
                             wait_ns);
    return cudaGetLastError();
  }
}

template <class T, bool FAST, bool CHAR, bool BLEND, int TX, int TY>
int occupancy() {
  constexpr size_t sm = tile_smem<T, TX, TY, BLEND>();
  if constexpr (sm > 227 * 1024) {
    return 0;
  } else {
    auto k = k_stage_tiles<T, FAST, CHAR, BLEND, TX, TY, kTileThreads>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kTileThreads, sm) != cudaSuccess) return 0;
    return n;
  }
}

}  // namespace tdetail
}  // inline namespace WENO_TU_NS

template <class H, bool FAST, int TX, int TY>
int StageTile<H, FAST, TX, TY>::ctas_per_sm(bool chr, bool blend) {
  using T = dev_t<H>;
  if (chr && blend) return tdetail::occupancy<T, FAST, true, true, TX, TY>();
  if (chr) return tdetail::occupancy<T, FAST, true, false, TX, TY>();
  if (blend) return tdetail::occupancy<T, FAST, false, true, TX, TY>();
  return tdetail::occupancy<T, FAST, false, false, TX, TY>();
}

template <class H, bool FAST, int TX, int TY>
cudaError_t StageTile<H, FAST, TX, TY>::launch(bool chr, bool blend, const SolveDesc* solves, SolveCtl* ctl,
                                               const void* tiles, int ntiles, int grid, const void* tmaps,
                                               const void* qn, void* qo, int stage, double gamma, double jp_lo,
                                               double jp_hi, double weps, int skip_tile, unsigned long long wait_ns,
                                               cudaStream_t st) {
  using T = dev_t<H>;
  const int4* tl = static_cast<const int4*>(tiles);
  const CUtensorMap* a = static_cast<const CUtensorMap*>(tmaps);
  const T* b = static_cast<const T*>(qn);
  T* o = static_cast<T*>(qo);
  const T g = (T)gamma, lo = (T)jp_lo, hi = (T)jp_hi, w = (T)weps;
#define WENO_TILE(CHAR, BLEND)                                                                                      \
  return tdetail::launch_stage<T, FAST, CHAR, BLEND, TX, TY>(solves, ctl, tl, ntiles, grid, a, b, o, stage, g, lo, \
                                                             hi, w, skip_tile, wait_ns, st)
  if (chr && blend) WENO_TILE(true, true);
  if (chr) WENO_TILE(true, false);
  if (blend) WENO_TILE(false, true);
  WENO_TILE(false, false);
#undef WENO_TILE
}

}  // namespace weno
