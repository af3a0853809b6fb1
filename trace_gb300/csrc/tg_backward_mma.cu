// Tensor-core backprojection: half factors, f16 lengths, and the dispatch
// on the kind of factors and lengths
// (tg_backward_mma.cuh).
#include "tg_backward_mma.cuh"

namespace tg {

TG_MMA_ENTRY(half, LK_F16, FK_HALF, 1)
TG_MMA_MULTI_ENTRY(half, LK_F16, FK_HALF, 1)

void launch_backward_mma(const IterArgs& A, int first, int nunits, const float* cur,
                         float* next, float* rep, int epi, cudaStream_t st) {
  if (A.half_factors != FACT_F32)
    launch_backward_mma_half(A, first, nunits, cur, next, rep, epi, st);
  else if (A.M.dlen_kind == LK_F16)
    launch_backward_mma_split(A, first, nunits, cur, next, rep, epi, st);
  else if (A.M.dlen_kind == LK_U16)
    launch_backward_mma_u16(A, first, nunits, cur, next, rep, epi, st);
  else if (A.M.dlen_kind == LK_BF16)
    launch_backward_mma_bf16(A, first, nunits, cur, next, rep, epi, st);
  else
    launch_backward_mma_f32(A, first, nunits, cur, next, rep, epi, st);
}

void launch_backward_mma_multi(const BackItem* items, int n, int64_t blocks, int U,
                               int dlen_kind, int pen, int fh, cudaStream_t st) {
  if (fh)
    launch_backward_mma_multi_half(items, n, blocks, U, pen, st);
  else if (dlen_kind == LK_F16)
    launch_backward_mma_multi_split(items, n, blocks, U, pen, st);
  else
    launch_backward_mma_multi_u16(items, n, blocks, U, pen, st);
}

}  // namespace tg
