// Forward projection (ray-driven): one warp per 32-ray group (32 adjacent
// detector columns of one angle), lane = ray. Each lane sums recon[idx]*len
// along its ray in the reference's segment order (CalculateSimdata,
// src/sirt/sirt.cc:4-19) and stores the per-ray factor of the
// backprojection: (ray - sim)/a2 for SIRT (sirt.cc:50-53), ray/sim for
// MLEM/PML/APMLR (mlem.cc:50, pml.cc:234), or sim itself.
//
// K slices share one read of the slice-invariant matrix: slice j of the
// batch is lane j of a K-float vector per pixel, so one gather (a single
// 256-bit load for K = 8) serves all K slices. The matrix rows are streamed
// with evict-first loads so they do not displace the gathered
// reconstruction from L2.
#include "tg_kernels.cuh"

namespace tg {

namespace {

constexpr int kBlock = 256;

template <int LK>
__device__ __forceinline__ float stream_len(const void* base, int64_t e,
                                            float inv_scale) {
  if constexpr (LK == LK_F32)
    return __ldcs(reinterpret_cast<const float*>(base) + e);
  else
    return decode_len<LK>(__ldcs(reinterpret_cast<const uint16_t*>(base) + e),
                          inv_scale);
}

// Per-ray output of the forward kernels: the ray sum (FWD_SIM), SIRT's
// (ray - sim) / a2 (sirt.cc:50) or the ratio ray / sim (mlem.cc:50,
// pml.cc:236, apmlr.cc:1017).
template <int K>
__device__ __forceinline__ void fwd_epilogue(const MatrixDev& M, int64_t r,
                                             const float (&acc)[K], const float* sino,
                                             float* out, int out_mode) {
  Vec<K> o;
  if (out_mode == FWD_SIM) {
#pragma unroll
    for (int j = 0; j < K; ++j) o.v[j] = acc[j];
  } else {
    const Vec<K> ray = load_vec<K>(sino + r * K);
    if (out_mode == FWD_SIRT) {
      const float a2 = M.ra2[r];
#pragma unroll
      for (int j = 0; j < K; ++j) o.v[j] = fdiv(fsub(ray.v[j], acc[j]), a2);
    } else {
#pragma unroll
      for (int j = 0; j < K; ++j) o.v[j] = fdiv(ray.v[j], acc[j]);
    }
  }
  store_vec<K>(out + r * K, o);
}

// Slice batches of one launch: consecutive blocks take the same rays of the nb
// batches, so that all of them read a piece of the matrix while it is in L2.
// Moves the pointers to the block's batch; returns its place in the rays.
template <int K>
__device__ __forceinline__ int batch_block(const DevGeom& G,
                                           const float* __restrict__& recon,
                                           const float* __restrict__& sino,
                                           float* __restrict__& out) {
  const int b = blockIdx.x;
  const int64_t rays = (int64_t)G.P * G.C * K;
  recon += b * ((int64_t)G.C * G.C * K);
  sino += b * rays;
  out += b * rays;
  return grid_block();
}

template <int K, int LK, bool EXACT, bool DELTA>
__global__ void __launch_bounds__(kBlock)
    k_forward(DevGeom G, MatrixDev M, int ngroups,
              const float* __restrict__ recon, const float* __restrict__ sino,
              float* __restrict__ out, int out_mode) {
  // 16 slices per pass: always a single batch (its pointers cost registers: 128
  // columns, 90 angles, 24 exact slices 0.32 ms an iteration, 0.38 with them)
  const int block = K == 16 ? (int)blockIdx.x : batch_block<K>(G, recon, sino, out);
  const int grp = (block * kBlock + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (grp >= ngroups) return;  // warp-uniform
  const int a = grp / G.gpa;
  const int c = (grp - a * G.gpa) * 32 + lane;
  const bool valid = c < G.C;
  const int64_t r = (int64_t)a * G.C + c;
  const int n = valid ? M.rnseg[r] : 0;
  const int cap = M.rcap[grp];
  const int64_t base = M.roff[grp] + lane;
  const int g = G.C;
  float acc[K];
#pragma unroll
  for (int j = 0; j < K; ++j) acc[j] = 0.f;
  int idx = 0;
  int64_t cbase = 0;
  uint32_t word = 0;
  if (DELTA) {
    cbase = M.rcoff[grp] + lane;
    if (n > 0) idx = M.rstart[r];
  }
#pragma unroll 4
  for (int s = 0; s < cap; ++s) {
    if (s < n) {
      const int64_t e = base + (int64_t)s * 32;
      if (DELTA) {
        if ((s & 7) == 0) word = __ldcs(M.rcode + cbase + (int64_t)(s >> 3) * 32);
        if (s > 0) {
          const uint32_t code = (word >> (4 * (s & 7))) & 15u;
          idx += (int)(code & 1u) + ((int)(code >> 1) - 1) * g;
        }
      } else {
        idx = __ldcs(M.ridx + e);
      }
      const float l = stream_len<LK>(M.rlen, e, M.inv_scale);
      const Vec<K> v = load_vec<K>(recon + (int64_t)idx * K);
      if constexpr (EXACT) {
#pragma unroll
        for (int j = 0; j < K; ++j) acc[j] = fadd(acc[j], fmul(v.v[j], l));
      } else {
        fma_slices<K>(acc, l, v.v);
      }
    }
  }
  if (!valid) return;
  fwd_epilogue<K>(M, r, acc, sino, out, out_mode);
}

// On-the-fly forward projection: each ray is traced while it is projected
// (tg::trace_ray, the reference's tracer) instead of read from a stored
// matrix. Lengths are the traced float lengths and the sum runs in the
// reference's segment order, so the exact-mode result equals k_forward's
// with f32 lengths bit for bit. No forward matrix is kept on the device;
// the cost moves from streaming the matrix to tracing (ALU).
template <int K, bool EXACT>
__global__ void __launch_bounds__(kBlock)
    k_forward_otf(DevGeom G, MatrixDev M, int ngroups,
                  const float* __restrict__ recon, const float* __restrict__ sino,
                  float* __restrict__ out, int out_mode) {
  const int grp = (batch_block<K>(G, recon, sino, out) * kBlock + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (grp >= ngroups) return;
  const int a = grp / G.gpa;
  const int c = (grp - a * G.gpa) * 32 + lane;
  if (c >= G.C) return;
  const int64_t r = (int64_t)a * G.C + c;
  float acc[K];
#pragma unroll
  for (int j = 0; j < K; ++j) acc[j] = 0.f;
  trace_ray(G, a, c, [&](int idx, float l, float, int, int) {
    const Vec<K> v = load_vec<K>(recon + (int64_t)idx * K);
    if constexpr (EXACT) {
#pragma unroll
      for (int j = 0; j < K; ++j) acc[j] = fadd(acc[j], fmul(v.v[j], l));
    } else {
      fma_slices<K>(acc, l, v.v);
    }
  });
  fwd_epilogue<K>(M, r, acc, sino, out, out_mode);
}

// One slice per pass (the default plan): NB slices per thread, each a plane of
// its own, so that a segment's index and length are read (or traced) once. The
// gathers bound it: neighbouring rays closer to the horizontal cross pixels
// one above the other, i.e. 32 cache lines per load, so those angles read a
// transposed copy of the planes (tr) when the caller has one. Four segments'
// gathers are in flight at a time, and the next four's indices and lengths.
// 1024 x 1024, 720 angles, 16 exact slices: 13.9 ms; 24.8 without the copy; 32.9
// one slice per thread.
enum PlaneSource { kPlaneIndex, kPlaneDelta, kPlaneTrace };
constexpr int kPlaneChunk = 4;

template <int NB, int LK, bool EXACT, int SRC>
__global__ void __launch_bounds__(kBlock)
    k_forward_planes(DevGeom G, MatrixDev M, int ngroups, int n,
                     const float* __restrict__ recon, const float* __restrict__ turned,
                     const float* __restrict__ sino, float* __restrict__ out, int out_mode) {
  // consecutive blocks take the same rays of all groups of slices; the last
  // group starts early if need be and leaves out what is another's (own)
  const int own = blockIdx.x * NB, s0 = min(own, n - NB);
  const int grp = (grid_block() * kBlock + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (grp >= ngroups) return;  // warp-uniform
  const int a = grp / G.gpa;
  const int c = (grp - a * G.gpa) * 32 + lane;
  const int g = G.C;
  const int64_t r = (int64_t)a * g + c, g2 = (int64_t)g * g, rays = (int64_t)G.P * g;
  const float4 coef = M.wcoef[a];
  const bool tr = turned != nullptr && fabsf(coef.x) < fabsf(coef.y);
  const float* img[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) img[k] = (tr ? turned : recon) + (s0 + k) * g2;
  float acc[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) acc[k] = 0.f;
  auto add = [&](int k, float v, float l) {
    acc[k] = EXACT ? fadd(acc[k], fmul(v, l)) : __fmaf_rn(l, v, acc[k]);
  };
  if constexpr (SRC == kPlaneTrace) {
    if (c >= g) return;
    trace_ray(G, a, c, [&](int idx, float l, float, int ix, int iy) {
      const int at = tr ? ix * g + iy : idx;
#pragma unroll
      for (int k = 0; k < NB; ++k) add(k, __ldg(img[k] + at), l);
    });
  } else {
    const int nseg = c < g ? M.rnseg[r] : 0, cap = M.rcap[grp];
    const int64_t base = M.roff[grp] + lane;
    const float inv_g = 1.0f / (float)g;
    const int dxs = tr ? g : 1, dys = tr ? 1 : g;
    auto turn = [&](int idx) {
      if (!tr) return idx;
      int ix, iy;
      cell_xy(idx, g, inv_g, ix, iy);
      return ix * g + iy;
    };
    int at = 0;
    const uint32_t* codes = nullptr;
    if (SRC == kPlaneDelta) {
      codes = M.rcode + M.rcoff[grp] + lane;
      if (nseg > 0) at = turn(M.rstart[r]);
    }
    struct Chunk {
      int idx[SRC == kPlaneIndex ? kPlaneChunk : 1];
      uint32_t word;
      float len[kPlaneChunk];
    };
    auto load = [&](int s, Chunk& q) {
      if (SRC == kPlaneDelta) q.word = s < nseg ? __ldg(codes + (int64_t)(s >> 3) * 32) : 0u;
#pragma unroll
      for (int i = 0; i < kPlaneChunk; ++i) {
        const int64_t e = base + (int64_t)(s + i) * 32;
        q.len[i] = 0.f;
        if (SRC == kPlaneIndex) q.idx[i] = 0;
        if (s + i < nseg) {
          q.len[i] = stream_len<LK>(M.rlen, e, M.inv_scale);
          if (SRC == kPlaneIndex) q.idx[i] = __ldcs(M.ridx + e);
        }
      }
    };
    Chunk q, nq;
    load(0, q);
    for (int s = 0; s < cap; s += kPlaneChunk) {
      load(s + kPlaneChunk, nq);
      float v[kPlaneChunk][NB];
#pragma unroll
      for (int i = 0; i < kPlaneChunk; ++i) {
        int e;
        if (SRC == kPlaneDelta) {
          const uint32_t code = (q.word >> (4 * ((s + i) & 7))) & 15u;
          if (s + i > 0) at += (int)(code & 1u) * dxs + ((int)(code >> 1) - 1) * dys;
          e = at;
        } else {
          e = turn(q.idx[i]);
        }
#pragma unroll
        for (int k = 0; k < NB; ++k) {
          v[i][k] = 0.f;
          if (s + i < nseg) v[i][k] = __ldg(img[k] + e);
        }
      }
#pragma unroll
      for (int i = 0; i < kPlaneChunk; ++i)
#pragma unroll
        for (int k = 0; k < NB; ++k) add(k, v[i][k], q.len[i]);
      q = nq;
    }
    if (c >= g) return;
  }
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    if (s0 + k < own) continue;
    const float one[1] = {acc[k]};
    fwd_epilogue<1>(M, r, one, sino + (s0 + k) * rays, out + (s0 + k) * rays, out_mode);
  }
}

// n planes of g x g pixels, rows and columns exchanged.
__global__ void __launch_bounds__(256)
    k_turn_planes(const float* __restrict__ in, float* __restrict__ out, int g) {
  __shared__ float t[32][33];
  const int64_t plane = (int64_t)blockIdx.z * g * g;
  const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 32 + threadIdx.y;
  for (int j = 0; j < 32; j += 8)
    if (x < g && y + j < g) t[threadIdx.y + j][threadIdx.x] = __ldg(in + plane + (int64_t)(y + j) * g + x);
  __syncthreads();
  const int tx = blockIdx.y * 32 + threadIdx.x, ty = blockIdx.x * 32 + threadIdx.y;
  for (int j = 0; j < 32; j += 8)
    if (tx < g && ty + j < g) out[plane + (int64_t)(ty + j) * g + tx] = t[threadIdx.x][threadIdx.y + j];
}

template <int NB, int LK>
void planes_launch(const IterArgs& A, int n, const float* recon, const float* turned,
                   const float* sino, float* out, int out_mode, cudaStream_t st) {
  const int ngroups = A.G.P * A.G.gpa, groups = (n + NB - 1) / NB;
  const dim3 blocks = batch_grid(((int64_t)ngroups * 32 + kBlock - 1) / kBlock, groups);
#define TG_PLANES(E, SRC)                                                                 \
  k_forward_planes<NB, LK, E, SRC><<<blocks, kBlock, 0, st>>>(A.G, A.M, ngroups, n, recon, \
                                                              turned, sino, out, out_mode)
  if (A.M.rlen == nullptr) {  // no stored forward matrix: float lengths, traced
    if constexpr (LK == LK_F32) {
      if (A.exact) TG_PLANES(true, kPlaneTrace); else TG_PLANES(false, kPlaneTrace);
    }
  } else if (A.delta_index) {
    if (A.exact) TG_PLANES(true, kPlaneDelta); else TG_PLANES(false, kPlaneDelta);
  } else {
    if (A.exact) TG_PLANES(true, kPlaneIndex); else TG_PLANES(false, kPlaneIndex);
  }
#undef TG_PLANES
}

template <int NB>
void planes_kind(const IterArgs& A, int n, const float* recon, const float* turned,
                 const float* sino, float* out, int out_mode, cudaStream_t st) {
  switch (A.M.rlen ? A.M.len_kind : (int)LK_F32) {
    case LK_F32: planes_launch<NB, LK_F32>(A, n, recon, turned, sino, out, out_mode, st); break;
    case LK_BF16: planes_launch<NB, LK_BF16>(A, n, recon, turned, sino, out, out_mode, st); break;
    case LK_F16: planes_launch<NB, LK_F16>(A, n, recon, turned, sino, out, out_mode, st); break;
    default: planes_launch<NB, LK_U16>(A, n, recon, turned, sino, out, out_mode, st); break;
  }
}

void forward_planes(const IterArgs& A, int n, const float* recon, const float* sino, float* out,
                    int out_mode, cudaStream_t st) {
  // one slice alone is bound by the matrix, not by its gathers (700 columns,
  // 500 angles, one slice: 0.48 ms without the copy, 0.49 with it; five slices
  // 1.80 and 1.36)
  float* turned = n > 1 ? A.turned : nullptr;
  if (turned) {
    const int t = (A.G.C + 31) / 32;
    k_turn_planes<<<dim3(t, t, n), dim3(32, 8), 0, st>>>(recon, turned, A.G.C);
  }
  // Several slices per thread want more registers, so fewer warps are there to
  // hide the loads: four where warps are plenty (1024 columns, 720 angles, 16
  // slices: 13.9 ms with four, 15.0 with two, 18.4 with one), two on a grid that
  // fills the GPU once or twice (400 columns, 300 angles, 4 slices: 0.31, 0.26,
  // 0.30); traced rays take four as soon as those fill the GPU (512 columns, 360
  // angles, 8 slices: 1.34, 1.53, 2.64).
  const int64_t warps = (int64_t)A.G.P * A.G.gpa;
  switch (A.M.rlen ? planes_per_thread(warps, n, 30000, 7000)
                   : planes_per_thread(warps, n, 4800, 4800)) {
    case 1: planes_kind<1>(A, n, recon, turned, sino, out, out_mode, st); break;
    case 2: planes_kind<2>(A, n, recon, turned, sino, out, out_mode, st); break;
    case 3: planes_kind<3>(A, n, recon, turned, sino, out, out_mode, st); break;
    default: planes_kind<4>(A, n, recon, turned, sino, out, out_mode, st); break;
  }
}

template <int K, int LK>
void fwd_launch(const IterArgs& A, int nb, const float* recon, const float* sino,
                float* out, int out_mode, cudaStream_t st) {
  const int ngroups = A.G.P * A.G.gpa;
  const int64_t all = ((int64_t)ngroups * 32 + kBlock - 1) / kBlock;
  const dim3 blocks = K == 16 ? dim3((unsigned)all) : batch_grid(all, nb);
#define TG_FWD(E, D) \
  k_forward<K, LK, E, D><<<blocks, kBlock, 0, st>>>(A.G, A.M, ngroups, recon, sino, out, out_mode)
  if (A.delta_index) {
    if (A.exact) TG_FWD(true, true); else TG_FWD(false, true);
  } else {
    if (A.exact) TG_FWD(true, false); else TG_FWD(false, false);
  }
#undef TG_FWD
}

template <int K>
void fwd_kind(const IterArgs& A, int nb, const float* recon, const float* sino,
              float* out, int out_mode, cudaStream_t st) {
  if (A.M.rlen == nullptr) {  // no stored forward matrix: trace on the fly
    const int ngroups = A.G.P * A.G.gpa;
    const dim3 blocks = batch_grid(((int64_t)ngroups * 32 + kBlock - 1) / kBlock, nb);
    if (A.exact)
      k_forward_otf<K, true><<<blocks, kBlock, 0, st>>>(A.G, A.M, ngroups, recon, sino,
                                                         out, out_mode);
    else
      k_forward_otf<K, false><<<blocks, kBlock, 0, st>>>(A.G, A.M, ngroups, recon, sino,
                                                          out, out_mode);
    return;
  }
  switch (A.M.len_kind) {
    case LK_F32: fwd_launch<K, LK_F32>(A, nb, recon, sino, out, out_mode, st); break;
    case LK_BF16: fwd_launch<K, LK_BF16>(A, nb, recon, sino, out, out_mode, st); break;
    case LK_F16: fwd_launch<K, LK_F16>(A, nb, recon, sino, out, out_mode, st); break;
    default: fwd_launch<K, LK_U16>(A, nb, recon, sino, out, out_mode, st); break;
  }
}

}  // namespace

void launch_forward(const IterArgs& A, int nb, const float* recon_batch,
                    const float* sino_batch, float* out, int out_mode,
                    cudaStream_t st) {
  switch (A.K) {
    case 1: forward_planes(A, nb, recon_batch, sino_batch, out, out_mode, st); break;
    case 2: fwd_kind<2>(A, nb, recon_batch, sino_batch, out, out_mode, st); break;
    case 4: fwd_kind<4>(A, nb, recon_batch, sino_batch, out, out_mode, st); break;
    case 8: fwd_kind<8>(A, nb, recon_batch, sino_batch, out, out_mode, st); break;
    default: fwd_kind<16>(A, nb, recon_batch, sino_batch, out, out_mode, st); break;
  }
}

}  // namespace tg
