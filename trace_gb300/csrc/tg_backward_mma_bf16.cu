// Tensor-core backprojection: TF32 factors, bfloat16 lengths
// (tg_backward_mma.cuh).
#include "tg_backward_mma.cuh"

namespace tg {

TG_MMA_ENTRY(bf16, LK_BF16, FK_TF32, 1)

}  // namespace tg
