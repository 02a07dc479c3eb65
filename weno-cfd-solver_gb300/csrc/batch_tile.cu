// One fused tile shape of one FP64 arithmetic; build.py compiles this file once per
// WENO_TILE_NS (the inline namespace), WENO_TILE_X, WENO_TILE_Y and, for the FAST
// forms, WENO_TILE_FAST.
#ifdef WENO_TILE_FAST
#define WENO_F64_CONTRACT
#define WENO_TILE_ARITH true
#else
#define WENO_TILE_ARITH false
#endif
#define WENO_TU_NS WENO_TILE_NS
#include "batch_tile.cuh"

namespace weno {
template struct StageTile<double, WENO_TILE_ARITH, WENO_TILE_X, WENO_TILE_Y>;
}
