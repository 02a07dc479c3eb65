// Batched stage kernels, float (the FP32 bulk precision), FAST forms.
#define WENO_F64_CONTRACT
#define WENO_TU_NS batch_f32
#include "batch_impl.cuh"
#include "batch_tile.cuh"

namespace weno {
template struct StageTile<float, true, 8, 32>;
template struct StageTile<float, true, 16, 32>;
template struct StageTile<float, true, 16, 16>;
template struct StageTile<float, true, 8, 64>;
template struct BatchLaunch<float, true>;
}
