// Tensor-core backprojection: TF32 factors, float lengths
// (tg_backward_mma.cuh).
#include "tg_backward_mma.cuh"

namespace tg {

TG_MMA_ENTRY(f32, LK_F32, FK_TF32, 2)

}  // namespace tg
