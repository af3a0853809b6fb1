// Backprojection at one slice per pass (the default plan): backward_block's
// work (tg_backward.cuh) for several slices per thread. Every slice is a plane
// of its own, so the lengths of a pixel's rays, their columns and the angle's
// coefficients are read and unpacked once, and only the factor gathers and the
// sums are per slice. The factor loads of an angle are in flight while the
// previous angle's sums are taken. The sums run in the same order. Bound by
// instruction issue and the gathers' latency: 1024 x 1024, 720 angles, 16 exact
// slices 5.8 ms, 19.4 one slice per thread without the overlap.
#include <type_traits>

#include "tg_backward.cuh"

namespace tg {

namespace {

template <int NB, int LK, bool EXACT, bool PEN, bool FH>
__global__ void __launch_bounds__(kBlock, NB >= 3 ? 3 : 5)
    k_backward_planes(IterArgs A, int first, int n, const float* __restrict__ cur,
                      float* __restrict__ next, const float* __restrict__ upd,
                      float* __restrict__ rep_num, int epi) {
  static_assert(!(EXACT && FH), "exact mode keeps FP32 factors");
  __shared__ float4 s_coef[kCoefChunk];
  const DevGeom& G = A.G;
  const int g = G.C;
  const int64_t g2 = (int64_t)g * g;
  // consecutive blocks take the same pixels of all groups of slices; the last
  // group starts early if need be and leaves out what is another's (own)
  const int own = blockIdx.x * NB, s0 = min(own, n - NB);
  const int tile = grid_block() * kWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  int x, y;
  tile_pixel(tile, lane, A.M.tiles_x, A.M.tw_shift, &x, &y);
  const bool valid = tile < A.M.ntiles && x < g && y < g;
  const int64_t p = (int64_t)y * g + x;
  const float xf = (float)x, yf = (float)y;
  const float* fsrc = cur + (int64_t)(first + s0 + A.fshift) * g2 + p;
  float rf[NB], acc[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    acc[k] = 0.f;
    rf[k] = PEN && EXACT && valid ? __ldg(fsrc + k * g2) : 0.f;
  }
  // see backward_block
  constexpr bool kScaled = LK == LK_U16 && !EXACT && !FH;
  constexpr int QW = Quad<LK>::kWords;
  const uint32_t qstep = (uint32_t)A.M.ntiles * 32 * QW;
  const uint4* qp = reinterpret_cast<const uint4*>(A.M.dlen) + ((int64_t)tile * 32 + lane) * QW;
  const int C = G.C;
  const int64_t plane = (int64_t)G.P * C;  // factors per slice
  using T = std::conditional_t<FH, unsigned short, float>;
  const T* ua = reinterpret_cast<const T*>(upd) + s0 * plane;
  auto add = [&](int k, bool have, float l, uint32_t lh, T u) {
    if constexpr (FH) {
      asm("{ .reg .b16 l; cvt.u16.u32 l, %2; fma.rn.f32.f16 %0, %1, l, %0; }"
          : "+f"(acc[k]) : "h"(u), "r"(lh));
    } else if constexpr (EXACT && PEN) {
      const float t = fmul(fmul(rf[k], l), u);
      acc[k] = fsub(acc[k], have ? t : 0.f);  // an infinite rf times no length
    } else if constexpr (EXACT) {
      acc[k] = fadd(acc[k], fmul(l, u));
    } else {
      acc[k] = __fmaf_rn(l, u, acc[k]);
    }
  };
  for (int a0 = 0; a0 < A.M.P4; a0 += kCoefChunk) {
    const int na = min(kCoefChunk, A.M.P4 - a0);  // a multiple of 4
    __syncthreads();
    for (int i = threadIdx.x; i < na; i += kBlock) s_coef[i] = A.M.wcoef[a0 + i];
    __syncthreads();
    if (!valid) continue;
    Quad<LK> q;
    load_quad<LK>(qp, q);
    for (int a4 = 0; a4 < na; a4 += 4) {
      Quad<LK> nq;
      if (a4 + 4 < na) load_quad<LK>(qp + qstep, nq);
      float l0[2], l1[2];
      uint32_t lh[2];
      bool h0[2], h1[2];
      T u0[2][NB], u1[2][NB];
      auto issue = [&](int j, int b) {
        if constexpr (FH && LK == LK_F16) {
          lh[b] = pick(q.w[0], j);
          h0[b] = (lh[b] & 0xffffu) != 0u;
          h1[b] = (lh[b] >> 16) != 0u;
        } else {
          quad_pair<LK, kScaled>(q, j, A.M.inv_scale, l0[b], l1[b], h0[b], h1[b]);
          if constexpr (FH) lh[b] = float2_to_half2_bits(l0[b], l1[b]);
        }
        const T* ub = ua + (j * C + window_c0(s_coef[a4 + j], xf, yf));
#pragma unroll
        for (int k = 0; k < NB; ++k) {
          u0[b][k] = u1[b][k] = T(0);
          if (h0[b]) u0[b][k] = __ldg(ub + k * plane);
          if (h1[b]) u1[b][k] = __ldg(ub + k * plane + 1);
        }
      };
      auto consume = [&](int b) {
#pragma unroll
        for (int k = 0; k < NB; ++k) {
          add(k, h0[b], l0[b], lh[b] & 0xffffu, u0[b][k]);
          add(k, h1[b], l1[b], lh[b] >> 16, u1[b][k]);
        }
      };
      issue(0, 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j < 3) issue(j + 1, (j + 1) & 1);
        consume(j & 1);
      }
      q = nq;
      qp += qstep;
      ua += 4 * C;
    }
  }
  if (!valid) return;
  const float Wp = FH ? A.M.Wh[p] : A.M.W[p];
  if constexpr (kScaled) {
#pragma unroll
    for (int k = 0; k < NB; ++k) acc[k] *= A.M.inv_scale;
  }
  // segments outside the pixel's window (stored apart, true lengths)
  for_each_exception(A.M, tile, lane, [&](float l, int ea, int ec) {
    const T* ub = reinterpret_cast<const T*>(upd) + s0 * plane + (int64_t)ea * C + ec;
    uint32_t w = 0;
    if constexpr (FH) w = float2_to_half2_bits(l, 0.f) & 0xffffu;
#pragma unroll
    for (int k = 0; k < NB; ++k) add(k, true, l, w, __ldg(ub + k * plane));
  });
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    if (s0 + k < own) continue;
    float num = acc[k];
    if constexpr (FH) {
      if (A.half_factors == FACT_HALF_M1) num += Wp;
    }
    if (PEN && !EXACT) num = -(__ldg(fsrc + k * g2) * num);
    update_pixel<1, EXACT, PEN>(A, first + s0 + k, x, y, num, Wp, cur, next, rep_num, epi);
  }
}

template <int NB, int LK>
void planes(const IterArgs& A, int first, int n, const float* cur, float* next,
            const float* upd, float* rep_num, int epi, cudaStream_t st) {
  const dim3 blocks = batch_grid((A.M.ntiles + kWarps - 1) / kWarps, (n + NB - 1) / NB);
  const bool pen = A.alg >= 2;
#define TG_PLANES(E, PN, FH)                                                              \
  k_backward_planes<NB, LK, E, PN, FH>                                                    \
      <<<blocks, kBlock, 0, st>>>(A, first, n, cur, next, upd, rep_num, epi)
  if (A.exact) {
    if (pen) TG_PLANES(true, true, false); else TG_PLANES(true, false, false);
  } else if (A.half_factors) {
    if constexpr (LK == LK_F16 || LK == LK_F32) {  // half gathers
      if (pen) TG_PLANES(false, true, true); else TG_PLANES(false, false, true);
    }
  } else {
    if (pen) TG_PLANES(false, true, false); else TG_PLANES(false, false, false);
  }
#undef TG_PLANES
}

template <int NB>
void planes_kind(const IterArgs& A, int first, int n, const float* cur, float* next,
                 const float* upd, float* rep_num, int epi, cudaStream_t st) {
  switch (A.M.dlen_kind) {
    case LK_F32: planes<NB, LK_F32>(A, first, n, cur, next, upd, rep_num, epi, st); break;
    case LK_BF16: planes<NB, LK_BF16>(A, first, n, cur, next, upd, rep_num, epi, st); break;
    case LK_F16: planes<NB, LK_F16>(A, first, n, cur, next, upd, rep_num, epi, st); break;
    default: planes<NB, LK_U16>(A, first, n, cur, next, upd, rep_num, epi, st); break;
  }
}

}  // namespace

void launch_backward_planes(const IterArgs& A, int first, int n, const float* cur, float* next,
                            const float* upd, float* rep_num, int epi, cudaStream_t st) {
  // four slices per thread wherever 13 warps per SM are left (400 columns, 300
  // angles, 4 slices: 0.136 ms with four, 0.147 with two, 0.233 with one; 200
  // columns, 150 angles, 3 slices: 0.049, 0.047, 0.038)
  switch (planes_per_thread(A.M.ntiles, n, 2048, 2048)) {
    case 1: planes_kind<1>(A, first, n, cur, next, upd, rep_num, epi, st); break;
    case 2: planes_kind<2>(A, first, n, cur, next, upd, rep_num, epi, st); break;
    case 3: planes_kind<3>(A, first, n, cur, next, upd, rep_num, epi, st); break;
    default: planes_kind<4>(A, first, n, cur, next, upd, rep_num, epi, st); break;
  }
}

}  // namespace tg
