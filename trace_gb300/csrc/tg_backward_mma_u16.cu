// Tensor-core backprojection: TF32 factors, 16-bit fixed-point lengths
// (tg_backward_mma.cuh).
#include "tg_backward_mma.cuh"

namespace tg {

TG_MMA_ENTRY(u16, LK_U16, FK_TF32, 2)
TG_MMA_MULTI_ENTRY(u16, LK_U16, FK_TF32, 2)

}  // namespace tg
