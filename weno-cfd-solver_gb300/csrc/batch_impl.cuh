// Batched launcher definitions (see batch_api.h).
#pragma once

#include "batch_api.h"
#include "batch_kernels.cuh"

namespace weno {

// Fused configurations only (0-3); the staged configuration has its own launcher.
#define WENO_TILE_SWITCH(cfg, MACRO) \
  switch (cfg) {                     \
    case 0: MACRO(8, 32); break;     \
    case 1: MACRO(16, 32); break;    \
    case 2: MACRO(16, 16); break;    \
    default: MACRO(8, 64); break;    \
  }

template <class H, bool FAST>
void BatchLaunch<H, FAST>::box(int cfg, bool blend, unsigned* cols, unsigned* rows) {
#define WENO_BOX(TX, TY)                                      \
  *cols = (unsigned)TileGeom<TX, TY, false>::UC;              \
  *rows = blend ? (unsigned)TileGeom<TX, TY, true>::UR : (unsigned)TileGeom<TX, TY, false>::UR;
  WENO_TILE_SWITCH(cfg, WENO_BOX)
#undef WENO_BOX
}

template <class H, bool FAST>
size_t BatchLaunch<H, FAST>::smem_bytes(int cfg, bool blend) {
  using T = dev_t<H>;
  size_t r = 0;
#define WENO_SM(TX, TY) \
  r = blend ? tile_smem<T, TX, TY, true>() : tile_smem<T, TX, TY, false>()
  WENO_TILE_SWITCH(cfg, WENO_SM)
#undef WENO_SM
  return r > 227 * 1024 ? 0 : r;
}

template <class H, bool FAST>
int BatchLaunch<H, FAST>::ctas_per_sm(int cfg, bool chr, bool blend) {
  int r = 0;
#define WENO_OCC(TX, TY) r = StageTile<H, FAST, TX, TY>::ctas_per_sm(chr, blend)
  WENO_TILE_SWITCH(cfg, WENO_OCC)
#undef WENO_OCC
  return r;
}

template <class H, bool FAST>
cudaError_t BatchLaunch<H, FAST>::stage(int cfg, bool chr, bool blend, const SolveDesc* solves, SolveCtl* ctl,
                                        const void* tiles, int ntiles, int grid, const void* tmaps, const void* qn,
                                        void* qo, int stage, double gamma, double jp_lo, double jp_hi,
                                        double weps, int skip_tile, unsigned long long wait_ns, cudaStream_t st) {
  if (ntiles <= 0 || grid <= 0) return cudaSuccess;
  cudaError_t e = cudaSuccess;
#define WENO_ST(TX, TY)                                                                                              \
  e = StageTile<H, FAST, TX, TY>::launch(chr, blend, solves, ctl, tiles, ntiles, grid, tmaps, qn, qo, stage, gamma, \
                                         jp_lo, jp_hi, weps, skip_tile, wait_ns, st)
  WENO_TILE_SWITCH(cfg, WENO_ST)
#undef WENO_ST
  return e;
}

template <class H, bool FAST>
cudaError_t BatchLaunch<H, FAST>::staged(bool chr, bool blend, const SolveDesc* solves, SolveCtl* ctl,
                                         const void* tiles, int ntiles, int grid, const void* qs, const void* qn,
                                         void* qo, void* ws, int stage, double gamma, double jp_lo, double jp_hi,
                                         double weps, cudaStream_t st) {
  using T = dev_t<H>;
  if (ntiles <= 0 || grid <= 0) return cudaSuccess;
  constexpr int TX = kTileTX[kStagedConfig], TY = kTileTY[kStagedConfig], NT = kTileThreads;
  constexpr int NP = kStagedThreads<T, FAST>;
  const int4* tl = static_cast<const int4*>(tiles);
  T* W = static_cast<T*>(ws);
  const T* Qs = static_cast<const T*>(qs);
  if (chr)
    k_staged_pass1<T, FAST, true, TX, TY, NP><<<grid, NP, 0, st>>>(solves, ctl, tl, ntiles, Qs, W, (T)gamma, (T)weps);
  else
    k_staged_pass1<T, FAST, false, TX, TY, NP><<<grid, NP, 0, st>>>(solves, ctl, tl, ntiles, Qs, W, (T)gamma,
                                                                     (T)weps);
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  if (blend)
    k_staged_pass2<T, FAST, true, TX, TY, NP><<<grid, NP, 0, st>>>(solves, ctl, tl, ntiles, W, (T)gamma, (T)weps);
  else
    k_staged_pass2<T, FAST, false, TX, TY, NP><<<grid, NP, 0, st>>>(solves, ctl, tl, ntiles, W, (T)gamma, (T)weps);
  if ((e = cudaGetLastError())) return e;
  const T* Qn = static_cast<const T*>(qn);
  T* Qo = static_cast<T*>(qo);
  if (blend)
    k_staged_residual<T, FAST, true, TX, TY, NT><<<grid, NT, 0, st>>>(solves, ctl, tl, ntiles, W, Qs, Qn, Qo, stage,
                                                                       (T)gamma, (T)jp_lo, (T)jp_hi);
  else
    k_staged_residual<T, FAST, false, TX, TY, NT><<<grid, NT, 0, st>>>(solves, ctl, tl, ntiles, W, Qs, Qn, Qo,
                                                                        stage, (T)gamma, (T)jp_lo, (T)jp_hi);
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t BatchLaunch<H, FAST>::cfl(int cfg, const SolveDesc* solves, SolveCtl* ctl, const void* tiles, int ntiles,
                                      int grid, const void* q, double gamma, cudaStream_t st) {
  using T = dev_t<H>;
  if (ntiles <= 0 || grid <= 0) return cudaSuccess;
  const int tx = kTileTX[cfg < kNumTileConfigs ? cfg : 0], ty = kTileTY[cfg < kNumTileConfigs ? cfg : 0];
  k_cfl_tiles<T, kTileThreads><<<grid, kTileThreads, 0, st>>>(solves, ctl, static_cast<const int4*>(tiles), ntiles,
                                                              tx, ty, static_cast<const T*>(q), (T)gamma);
  return cudaGetLastError();
}

template <class H, bool FAST>
cudaError_t BatchLaunch<H, FAST>::clock(SolveCtl* ctl, int nsolves, int phase, cudaStream_t st) {
  if (nsolves <= 0) return cudaSuccess;
  k_solve_clock<<<(nsolves + 127) / 128, 128, 0, st>>>(ctl, nsolves, phase);
  return cudaGetLastError();
}

#undef WENO_TILE_SWITCH

}  // namespace weno
