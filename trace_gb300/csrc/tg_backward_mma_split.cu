// Tensor-core backprojection: float factors as two halves, f16 lengths
// (tg_backward_mma.cuh).
#include "tg_backward_mma.cuh"

namespace tg {

TG_MMA_ENTRY(split, LK_F16, FK_SPLIT, 1)
TG_MMA_MULTI_ENTRY(split, LK_F16, FK_SPLIT, 1)

}  // namespace tg
