// Backprojection on the tensor cores (fast mode, tile-staged plans), with the
// algorithms' UpdateRecon fused into its epilogue.
//
// The backprojection of one 4x4 pixel tile over four angles is a small sparse
// matrix product: D[16 pixels x slices] += A[16 x 32] B[32 x slices], where
// the 32 columns of A are the tile's windows of 8 detector columns at each of
// the four angles and every row of A holds the (at most two, adjacent)
// lengths of its pixel at each angle. Two nonzeros in any four columns is the
// 2:4 sparsity that mma.sp takes, so A goes to the tensor cores as one 32-bit
// word per pixel, angle and half window, and a metadata word that the lanes
// build from the stored lengths: one mma.sp.m16n8k32 serves 16 pixels x 4
// angles x 8 slices. A does not depend on the slice and serves all 8 * NT
// slices of a unit (NT = 1, 2 or 4 accumulator tiles), so its cost and the
// matrix's bytes are paid once per unit instead of once per 8 slices.
//
// Why this shape: four angles by 4x4 pixels is the largest block whose
// windows fit 32 columns: the columns of a 4x4 tile span 3 (|sin| + |cos|)
// <= 4.25, i.e. at most 7 columns.
//
// A block covers 16x8 pixels, one tile per warp. Stages of 16 angles (the
// pixels' length pairs, and the block's windows of at most 21 columns of the
// unit's factors) are copied to shared memory with cp.async, the next stage
// while one is consumed; a warp's B operand is one ldmatrix (4 wavefronts)
// per accumulator tile. Gathered from global memory instead, every 8 lanes
// of a B load touch four cache lines: 16 wavefronts.
//
// Window columns to sparse groups: columns {0, 1, 4, 5} of an angle are its
// lower group and {2, 3, 6, 7} its upper one. With o the pixel's first column
// in the window, the pair (l0, l1) sits at positions o, o + 1 (mod 4) of the
// ring [lower lo, lower hi, upper lo, upper hi], and each group's metadata is
// one of two codes: its columns (0, 1) or (2, 3). o depends on the geometry
// only: construction stores it, with the metadata bits, as one byte per pixel
// and angle (place_byte), in the order the lanes read them; computing it here
// took 40 of 124 instructions per warp and four angles.
//
// The tensor core truncates its sums, which biases them: accumulators run over
// few angles (32 with half factors, 16 split, 8 in TF32 parts, whatever the unit's
// size) and are then added to FP32 sums with a rounded add. f32 lengths, error of
// one MLEM iteration against 64 bits at 160 columns: 4.8e-7 over 32 angles, 1.6e-7
// over 8, in the same time; 1.8e-7 by the scalar kernel.
//
// Factors (FK): halves (FK_HALF: MLEM/PML/APMLR, see k_fwd_finish) or floats.
// With f16 lengths a float is the sum of two halves of its slice's scale
// (FK_SPLIT: k_split_factors puts the slice's largest factor near 2^14; both
// parts rounded, so what is left is below 2^-23 of the factor, or below 2^-39
// of the largest), one more product with the same A. Other lengths take TF32
// (FK_TF32): two parts of each factor (hi rounded, lo the exact rest,
// truncated below 2^-22 of the factor) and mma.sp.m16n8k16, whose sparsity is
// one in two, so the groups are columns {4h, 4h + 2} and {4h + 1, 4h + 3}, and
// four angles are two products (h = 0, 1). Of o and o + 1 exactly one has the
// group's parity. Lengths that TF32 does not hold exactly (more than 11 bits)
// are split too, the two low parts' product left out.
//
// A zero of A times a non-finite factor would reach pixels that the ray does
// not cross: the finish kernel marks the slice when it stores a non-finite
// factor for a ray with segments, and the kernel then takes that slice's sums
// per crossed ray (slow_sum), as the scalar kernel does. The columns of a
// product are independent, so the other slices' stay. The same goes for
// FK_SPLIT's wide slices: where one hot ray's factor stands 2^15 and more over
// most others, two halves of one scale keep less of these than FP32 does.
//
// Measured (1024 x 1024, 720 angles, ms per 8 slices; the scalar kernel of
// tg_backward.cuh before the arrow): MLEM half factors 1.15 -> 0.96 in units
// of 8 slices, 0.61 of 16, 0.39 of 32; PML 1.16 -> 0.44 (32); SIRT 1.93 ->
// 1.10 (8), 0.60 (32). Bound by issue in small units (75 instructions per
// warp, tile and four angles, half of them on the integer pipe), by the
// shared-memory wavefronts (64 %) and issue (66 %) together in units of 32;
// the tensor pipe is 24 % busy.
#pragma once
#include "tg_kernels.cuh"

namespace tg {

namespace {

constexpr int kMmaTiles = 8;  // 4 x 2 tiles of 4x4 pixels per block, one per warp
constexpr int kMmaBlock = kMmaTiles * 32;
// Columns staged per angle: the tiles' window starts span 12 |cos| + 4 |sin|
// (or the other way round) <= 12.7 columns, and a window has 8.
constexpr int kMmaCols = 21;

constexpr int kMmaStarts = 32;  // angles whose window starts are computed at once

// Shared memory of one block: two stages of length pairs, place bytes and
// factors, and two sets of window starts.
enum { FK_HALF = 0, FK_SPLIT = 1, FK_TF32 = 2 };
template <int NT, int LK, int FK>
struct MmaStage {
  static constexpr int U = 8 * NT;
  static constexpr int NC = FK == FK_SPLIT ? 2 * NT : NT;  // 16-byte chunks of halves
  static constexpr int W = LK == LK_F32 ? 2 : 1;  // words per stored pair
  static constexpr int AS = FK == FK_TF32 || NC == 8 ? 8 : 16;  // angles per stage
  static constexpr int kElem = FK == FK_HALF ? 2 : 4;  // bytes per factor
  // bytes between staged columns: halves are swizzled (row_swizzle); floats
  // are padded to 8 words mod 32, so that 4 columns x 8 slices fill the banks
  static constexpr int kCol = FK != FK_TF32 ? NC * 16 : (U == 8 ? 32 : (U + 8) * 4);
  static constexpr int kQuad = kMmaTiles * 16 * 16 * W;  // bytes of 4 angles' pairs
  static constexpr int kPairs = AS / 4 * kQuad;
  static constexpr int kFactors = AS * kMmaCols * kCol;
  static constexpr int kPlaces = AS / 4 * kMmaTiles * 64;
  // [tiles][kMmaStarts] staged row of the tile's window, [kMmaStarts] block start
  static constexpr int kMeta = (kMmaTiles + 1) * kMmaStarts * 4;
  static constexpr int kBytes = 2 * (kPairs + kPlaces + kFactors + kMeta);
};

// 16-byte chunk swizzle of staged half column r: 8 consecutive columns of
// one chunk fall in 8 different bank groups.
template <int NC>
__device__ __forceinline__ int row_swizzle(int r) {
  return NC == 1 ? 0 : NC == 2 ? (r >> 2) & 1 : NC == 4 ? (r >> 1) & 3 : r & 7;
}

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(a));
  return v;
}

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4],
                                        const uint32_t (&b)[4], uint32_t e) {
  asm("mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.f16.f16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9,%10,%11}, {%0,%1,%2,%3}, %12, 0x0;"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]),
        "r"(e));
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4],
                                         const uint32_t (&b)[4], uint32_t e) {
  asm("mma.sp::ordered_metadata.sync.aligned.m16n8k16.row.col.f32.tf32.tf32.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9,%10,%11}, {%0,%1,%2,%3}, %12, 0x0;"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]),
        "r"(e));
}

__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&b)[4], uint32_t smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
               : "r"(smem));
}

// The TF32 part of a float (rounded to nearest, ties away) and the exact rest.
__device__ __forceinline__ uint32_t tf32_hi(float v) {
  return (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
}
__device__ __forceinline__ uint32_t tf32_lo(float v, uint32_t hi) {
  return __float_as_uint(__fsub_rn(v, __uint_as_float(hi)));
}

// NT words of shared memory in one load.
template <int NT>
__device__ __forceinline__ void lds_words(uint32_t (&w)[NT], uint32_t at) {
  if constexpr (NT == 1) {
    w[0] = lds32(at);
  } else if constexpr (NT == 2) {
    const uint2 v = lds64(at);
    w[0] = v.x; w[1] = v.y;
  } else {
    const uint4 v = lds128(at);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  }
}

// The stored pair of one (pixel, angle): 16-bit storages one word, f32 two.
template <int LK>
struct PairWord {
  uint32_t v[LK == LK_F32 ? 2 : 1];
};

// Both lengths as floats (16-bit fixed point unscaled: scaled once, at the end).
template <int LK>
__device__ __forceinline__ void pair_lengths(const PairWord<LK>& w, float& l0, float& l1) {
  if constexpr (LK == LK_F32) {
    l0 = __uint_as_float(w.v[0]);
    l1 = __uint_as_float(w.v[1]);
  } else if constexpr (LK == LK_U16) {
    l0 = u16_to_float(w.v[0] & 0xffffu);
    l1 = u16_to_float(w.v[0] >> 16);
  } else {
    l0 = decode_len<LK>((uint16_t)(w.v[0] & 0xffffu), 1.f);
    l1 = decode_len<LK>((uint16_t)(w.v[0] >> 16), 1.f);
  }
}

// Sum over the pixel's crossed rays of one slice, one product at a time, of
// every other angle quad from q0 on: for slices that a matrix product does not
// serve. `at` is the pixel's first pair. The four angles' factors are in flight
// together.
template <int LK, bool HALF>
__device__ __noinline__ float slow_sum(const IterArgs& A, const uint32_t* at, int x, int y, int q0,
                                       int64_t unit_base, int su) {
  constexpr int W = LK == LK_F32 ? 2 : 1;
  const int U = A.F.U, RP = A.F.RP;
  float acc = 0.f;
  for (int q = q0; q < A.M.P4 / 4; q += 2) {
    const uint4* w = reinterpret_cast<const uint4*>(at + (int64_t)q * A.M.ntiles * (128 * W));
    uint32_t v[4 * W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const uint4 t = __ldg(w + k);
      v[4 * k] = t.x; v[4 * k + 1] = t.y; v[4 * k + 2] = t.z; v[4 * k + 3] = t.w;
    }
    float l[8], f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      PairWord<LK> p;
#pragma unroll
      for (int k = 0; k < W; ++k) p.v[k] = v[j * W + k];
      const bool h0 = LK == LK_F32 ? p.v[0] != 0u : (p.v[0] & 0xffffu) != 0u;
      const bool h1 = LK == LK_F32 ? p.v[W - 1] != 0u : (p.v[0] >> 16) != 0u;
      pair_lengths<LK>(p, l[2 * j], l[2 * j + 1]);
      const int a = q * 4 + j, c0 = window_c0(__ldg(A.M.wcoef + a), (float)x, (float)y);
      const int64_t e = factor_at(unit_base, RP, U, a, c0, su);
      f[2 * j] = f[2 * j + 1] = 0.f;
      if constexpr (HALF) {
        const __half* b = reinterpret_cast<const __half*>(A.F.base) + e;
        if (h0) f[2 * j] = __half2float(b[0]);
        if (h1) f[2 * j + 1] = __half2float(b[U]);
      } else {
        const float* b = reinterpret_cast<const float*>(A.F.base) + e;
        if (h0) f[2 * j] = b[0];
        if (h1) f[2 * j + 1] = b[U];
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) acc = fmaf(l[i], f[i], acc);
  }
  return acc;
}

// A bit per slice of the unit: those that the products do not serve. bad: a
// non-finite factor. Wide (split plans): most factors lie below 2^-15 of the largest
// one, with which they share a scale (or none is in the sample).
template <bool SPLIT>
__device__ __forceinline__ unsigned redo_slices(const IterArgs& A, int unit, int lane) {
  const int s = unit * A.F.U + lane;
  bool redo = false;
  if (lane < A.F.U && s < A.S) {
    const FactorStat t = A.F.stat[s];
    redo = t.bad != 0 ||
           (SPLIT && (t.small > t.nonzero / 2 || (t.nonzero == 0u && t.most != 0u)));
  }
  return __ballot_sync(0xffffffffu, redo);
}

// n <= N consecutive slots' values of one pixel, slot s's at `r` (one vector
// load when they are contiguous and aligned in the batched layout).
template <int N>
__device__ __forceinline__ void load_slots(float (&v)[N], const float* r, int s, int n,
                                           int64_t g2, int K, bool vec) {
  if (vec) {
    const Vec<N> t = load_vec<N>(r);
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = t.v[j];
  } else {
    const int64_t a0 = slot_addr(s, 0, g2, K);
#pragma unroll
    for (int j = 0; j < N; ++j)
      v[j] = j < n ? __ldg(r + (slot_addr(s + j, 0, g2, K) - a0)) : 0.f;
  }
}

// Penalty F and G of N consecutive slices of one pixel (penalty_fg's
// operations in penalty_fg's order for each slice). base: slot s0 + vshift's
// pixel 0, K floats per pixel.
template <int N>
__device__ __forceinline__ void penalty_slices(const IterArgs& A, const float* cur,
                                               const float* base, int s0, int n, int x, int y,
                                               int p, int64_t g2, bool vec, float (&F)[N],
                                               float (&Gv)[N]) {
  const int g = A.G.C, K = A.K, s = s0 + A.vshift;
  if (A.alg != 3) {
    int region;
    const int cls = nbr_class(x, y, g, &region);
    float r0[N];
    load_slots<N>(r0, base + (int64_t)p * K, s, n, g2, K, vec);
    const float twob = fmul(2.f, A.pw.beta);
    float f = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) Gv[j] = 0.f;
    auto neighbour = [&](int dx, int dy, float w) {
      const float tw = fmul(twob, w);
      float rq[N];
      load_slots<N>(rq, base + (int64_t)(p + dx + dy * g) * K, s, n, g2, K, vec);
      f = fadd(f, tw);
#pragma unroll
      for (int j = 0; j < N; ++j) Gv[j] = fsub(Gv[j], fmul(tw, fadd(r0[j], rq[j])));
    };
    if (cls == 0) {  // the interior, unrolled: the table's order
      const float wo = A.pw.pml[0][0], wd = A.pw.pml[0][1];
      neighbour(1, 0, wo);
      neighbour(-1, 0, wo);
      neighbour(0, 1, wo);
      neighbour(0, -1, wo);
      neighbour(1, 1, wd);
      neighbour(-1, 1, wd);
      neighbour(1, -1, wd);
      neighbour(-1, -1, wd);
    } else {
      for (int q = 0; q < c_nbr.n[cls]; ++q)
        neighbour(c_nbr.dx[cls][q], c_nbr.dy[cls][q], A.pw.pml[region][c_nbr.kind[cls][q]]);
    }
#pragma unroll
    for (int j = 0; j < N; ++j) F[j] = f;
  } else {
    for (int j = 0; j < N; ++j) F[j] = Gv[j] = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if (j >= n) continue;
      int up = 0, down = 0;
      apmlr_axial(A, s0 + j, &up, &down);
      const float* at[3];  // slices one below, own, one above
#pragma unroll
      for (int dz = 0; dz < 3; ++dz)
        at[dz] = (dz == 0 && !down) || (dz == 2 && !up)
                     ? cur
                     : cur + slot_addr(s + j + dz - 1, 0, g2, K);
      penalty_fg(true, A.pw, x, y, g, up, down,
                 [&](int dx, int dy, int dz) {
                   return at[dz + 1][(int64_t)(p + dx + dy * g) * K];
                 },
                 F[j], Gv[j]);
    }
  }
}

// One block's work: 16x8 pixels of unit `unit`.
// LK: kind of the stored lengths (f16 unless FK_TF32). LP: TF32 parts of a
// length (1: exact in 11 bits).
template <int NT, int LK, int FK, int LP, bool PEN>
__device__ __forceinline__ void backward_mma_block(const IterArgs& A, int unit, int block,
                                                   const float* __restrict__ cur,
                                                   float* __restrict__ next,
                                                   float* __restrict__ rep_num, int epi) {
  using St = MmaStage<NT, LK, FK>;
  constexpr bool F16 = FK != FK_TF32;  // operands are halves
  constexpr int W = St::W, U = St::U, AS = St::AS, kCol = St::kCol;
  extern __shared__ __align__(128) uint4 smem_mma[];
  // [2] pairs, [2] places, [2] factors, [2] starts
  constexpr int kPlace = 2 * St::kPairs, kFac = kPlace + 2 * St::kPlaces;
  constexpr int kMeta = kFac + 2 * St::kFactors;
  constexpr int kPerStart = kMmaStarts / AS;  // stages per set of starts
  // stages whose products the accumulators take: 32 angles with half factors, 16
  // split, 8 in TF32 parts
  constexpr int kPerFold = (FK == FK_HALF ? 32 : FK == FK_SPLIT ? 16 : 8) / AS;
  char* const sm = reinterpret_cast<char*>(smem_mma);
  const uint32_t sm32 = (uint32_t)__cvta_generic_to_shared(smem_mma);
  const int g = A.G.C;
  const int64_t g2 = (int64_t)g * g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = lane >> 2, t = lane & 3;  // A row (pixels row, row + 8), group
  const int bx = block % A.F.blocks_x, by = block / A.F.blocks_x;
  const int X0 = bx * 16, Y0 = by * 8;
  // the lane's two pixels
  const int x = X0 + (warp & 3) * 4 + (row & 3), ya = Y0 + (warp >> 2) * 4 + (row >> 2);
  const int yb = ya + 2;
  const bool va = x < g && ya < g, vb = x < g && yb < g;
  const uint32_t* dl = reinterpret_cast<const uint32_t*>(A.M.dlen);
  const int64_t unit_base = (int64_t)(unit % A.F.ring) * A.F.unit_elems;
  const int P4 = A.M.P4, RP = A.F.RP;
  // the slices that the products do not serve: looked up now or after the products,
  // what suits the kernel's registers (PML, half factors, 2048 x 2048, 1500 angles, 64
  // slices 26.4 ms, after them 27.1)
  unsigned redo = 0u;
  if constexpr (FK == FK_HALF) redo = redo_slices<false>(A, unit, lane);

  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;

  {
    // length pairs: the thread copies one pixel (rows of 16 pixels, the
    // matrix's order), of every other angle quad
    const int cx = X0 + (tid & 15), cy = Y0 + ((tid >> 4) & 7);
    const bool cv = cx < g && cy < g;
    int ctile = 0, clane = 0;
    if (cv) pixel_tile(cx, cy, A.M.tiles_x, A.M.tw_shift, &ctile, &clane);
    const int64_t qstep = (int64_t)A.M.ntiles * 128 * W;  // words per four angles
    const int cq = tid >> 7;
    const uint32_t* cpair = dl + ((int64_t)ctile * 128 + clane * 4) * W + cq * qstep;
    const uint32_t cdst =
        sm32 + cq * St::kQuad +
        ((((tid >> 6) & 1) * 4 + ((tid >> 2) & 3)) * 16 + ((tid >> 4) & 3) * 4 + (tid & 3)) * 16 * W;
    // place bytes: 32 threads per angle quad, each one 16-byte chunk of a tile
    const int ptx = bx * 4 + ((tid >> 2) & 3), pty = by * 2 + ((tid >> 4) & 1);
    const bool pv = (tid >> 5) < AS / 4 && ptx < A.M.tiles4 && pty < A.M.tiles4;
    const int64_t pstep = (int64_t)A.M.tiles4 * A.M.tiles4 * 16;  // words per four angles
    const uint32_t* cplace = A.M.place + (tid >> 5) * pstep +
                             ((int64_t)pty * A.M.tiles4 + ptx) * 16 + (tid & 3) * 4;
    const uint32_t pdst = sm32 + kPlace + tid * 16;
    // factors: kThreads threads per angle, each one 16-byte chunk of every
    // kStep-th column
    constexpr int kThreads = kMmaBlock / AS, kChunks = U * St::kElem / 16;
    constexpr int kStep = kThreads / kChunks, kCopies = (kMmaCols + kStep - 1) / kStep;
    const int fj = tid / kThreads, fk = tid % kThreads;
    const int fr = fk / kChunks, fc = fk % kChunks;
    const char* fac = reinterpret_cast<const char*>(FK == FK_SPLIT ? A.F.split : A.F.base) +
                      unit_base * St::kElem + fk * 16;
    uint32_t fdst[2];  // columns fr + kStep i for even and odd i
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = fj * kMmaCols + fr + i * kStep;
      fdst[i] = sm32 + kFac + r * kCol + ((F16 ? fc ^ row_swizzle<St::NC>(r) : fc) << 4);
    }

    // window starts of angles S * kMmaStarts + lane: the warp's tile's (its
    // row in the staged columns) and the block's
    auto starts = [&](int S) {
      const int a = S * kMmaStarts + lane;
      if (a >= P4) return;
      const float4 cf = __ldg(A.M.wcoef + a);
      // the block's first staged column, counted from the padding's start;
      // windows outside the detector hold no lengths: any columns will do
      const int ws = min(max(window_low(cf, X0, Y0, 16, 8) - kWindowBias + kRayPad, 0),
                         RP - kMmaCols);
      const int lo = window_low(cf, X0 + (warp & 3) * 4, Y0 + (warp >> 2) * 4, 4, 4);
      const int r = min(max(lo - kWindowBias + kRayPad - ws, 0), kMmaCols - 8);
      int* m = reinterpret_cast<int*>(sm + kMeta + (S & 1) * St::kMeta);
      m[warp * kMmaStarts + lane] = (lane % AS) * kMmaCols + r;
      if (warp == 0) m[kMmaTiles * kMmaStarts + lane] = ws;
    };
    // copies of stage s (its block starts are in shared memory)
    auto copy = [&](int s) {
      const uint32_t pd = cdst + (s & 1) * St::kPairs;
#pragma unroll
      for (int q = 0; q < AS / 4; q += 2) {
        if (cv && s * AS + (q + cq) * 4 < P4) {
#pragma unroll
          for (int w = 0; w < W; ++w) cp_async16(pd + q * St::kQuad + w * 16, cpair + q * qstep + w * 4);
        }
      }
      cpair += (AS / 4) * qstep;
      if (pv && s * AS + (tid >> 5) * 4 < P4) cp_async16(pdst + (s & 1) * St::kPlaces, cplace);
      cplace += (AS / 4) * pstep;
      const int a = s * AS + fj;
      if (a < P4) {
        const int ws = (int)lds32(sm32 + kMeta + ((s / kPerStart) & 1) * St::kMeta +
                                  (kMmaTiles * kMmaStarts + a % kMmaStarts) * 4);
        const char* src = fac + ((int64_t)a * RP + ws) * (U * St::kElem);
        const uint32_t fo = (s & 1) * St::kFactors;
#pragma unroll
        for (int i = 0; i < kCopies; ++i)
          if ((i + 1) * kStep <= kMmaCols || fr + i * kStep < kMmaCols)
            cp_async16(fdst[i & 1] + fo + (i & ~1) * kStep * kCol, src + i * kStep * (U * St::kElem));
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int half = t & 1, pr = t >> 1;  // the lane's group of angles 2 pr and 2 pr + 1
    const int nstages = (P4 + AS - 1) / AS;
    // the lane's shared-memory addresses of angle quad 0
    const uint32_t l_pairs = sm32 + warp * (256 * W) + row * 16 * W + pr * 8 * W;
    const uint32_t l_place = sm32 + kPlace + warp * 64 + row * 8;
    // halves: B register i holds angle {0, 2, 1, 3}[i], its columns in the
    // order 0, 1, 4, 5, 2, 3, 6, 7; the lane names column lane & 7 of
    // register lane >> 3 for ldmatrix
    const uint32_t l_row = sm32 + kMeta + warp * (kMmaStarts * 4) +
                           (F16 ? (lane >> 4) | ((lane >> 2) & 2) : 0) * 4;
    const int rl = (lane & 1) | ((lane & 2) << 1) | ((lane & 4) >> 1);
    // the ring of byte selectors, turned by the lane's half (two bytes)
    const uint32_t ring = half ? 0x32104444u : 0x44443210u;
    // metadata word `half`: the place bytes of angles half and half + 2
    const uint32_t pick = half ? 0x7531u : 0x6420u;
    float d[NT][4];
    if (!cv) {  // pixels outside the grid: no lengths, in any stage
#pragma unroll
      for (int q = 0; q < 2 * AS / 4; q += 2)
        for (int w = 0; w < W; ++w)
          *reinterpret_cast<uint4*>(sm + (cdst - sm32) + q * St::kQuad + w * 16) =
              make_uint4(0u, 0u, 0u, 0u);
    }
    starts(0);
    __syncthreads();
    copy(0);
    for (int s = 0; s < nstages; ++s) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      if (s + 1 < nstages) copy(s + 1);
      if (s % kPerStart == 0) starts(s / kPerStart + 1);
      const uint32_t q_pairs = l_pairs + (s & 1) * St::kPairs;
      const uint32_t q_place = l_place + (s & 1) * St::kPlaces;
      const uint32_t q_row = l_row + ((s / kPerStart) & 1) * St::kMeta + s % kPerStart * AS * 4;
      const uint32_t q_fac = sm32 + kFac + (s & 1) * St::kFactors +
                             (F16 ? 0 : (pr + 2 * half) * kCol + row * (NT * 4));
      if (s % kPerFold == 0) {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) d[j][i] = 0.f;
      }
      auto quad = [&](int q) {
        // pairs and place bytes of the lane's two pixels
        PairWord<LK> w[2][2];  // [pixel][angle]
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if constexpr (LK == LK_F32) {
            const uint4 v = lds128(q_pairs + q * St::kQuad + h * 128 * W);
            w[h][0].v[0] = v.x; w[h][0].v[1] = v.y;
            w[h][1].v[0] = v.z; w[h][1].v[1] = v.w;
          } else {
            const uint2 v = lds64(q_pairs + q * St::kQuad + h * 128);
            w[h][0].v[0] = v.x;
            w[h][1].v[0] = v.y;
          }
        }
        const uint2 pl = lds64(q_place + q * (kMmaTiles * 64));
        uint32_t o8[2][2];  // the low bits: 8 x the pair's place
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          o8[0][k] = pl.x >> (16 * pr + 8 * k);
          o8[1][k] = pl.y >> (16 * pr + 8 * k);
        }
        // metadata bits of the two groups of two angles, for both pixels
        const uint32_t px = __byte_perm(pl.x, pl.y, pick);
        const uint32_t bits = F16 ? ((px >> 6) & 0x01010101u) | ((px >> 1) & 0x10101010u)
                                   : ((px >> 7) & 0x01010101u) | (px & 0x10101010u);
        const uint32_t code = 0x44444444u + bits * 10u;
        float v[2][2];
        if constexpr (!F16) {
          // of the pair's two columns, the one of the group's parity and its
          // length
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              float l0, l1;
              pair_lengths<LK>(w[h][k], l0, l1);
              const uint32_t second = (o8[h][k] ^ (half << 3)) & 8u;
              v[h][k] = second ? l1 : l0;
              o8[h][k] = (o8[h][k] & 0x38u) + second;
            }
        }
        if constexpr (F16) {
          uint32_t a[4];
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              a[2 * k + h] =
                  __byte_perm(w[h][k].v[0], 0u, __funnelshift_l(ring, ring, o8[h][k]));
          const int r = (int)lds32(q_row + q * 16) + rl;
          const uint32_t at = q_fac + r * kCol + (row_swizzle<St::NC>(r) << 4);
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            uint32_t b[4];
            if constexpr (FK == FK_SPLIT) {  // the low parts
              ldmatrix4_trans(b, at ^ ((NT + j) << 4));
              mma_f16(d[j], a, b, code);
            }
            ldmatrix4_trans(b, at ^ (j << 4));
            mma_f16(d[j], a, b, code);
          }
        } else {
          // B register i holds angle {0, 2, 1, 3}[i], column
          // 4 hh + t / 2 + 2 (t & 1) of product hh
          const uint4 rr = lds128(q_row + q * 16);
          const uint32_t f[4] = {q_fac + rr.x * kCol, q_fac + rr.z * kCol, q_fac + rr.y * kCol,
                                 q_fac + rr.w * kCol};
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            uint32_t ah[4], al[4];
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float l = ((o8[h][k] >> 5) & 1) == hh ? v[h][k] : 0.f;
                ah[2 * k + h] = LP == 1 ? __float_as_uint(l) : tf32_hi(l);
                if constexpr (LP == 2) al[2 * k + h] = tf32_lo(l, ah[2 * k + h]);
              }
            uint32_t fw[4][NT];
#pragma unroll
            for (int i = 0; i < 4; ++i) lds_words<NT>(fw[i], f[i] + hh * 4 * kCol);
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              uint32_t bh[4], bl[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float fv = __uint_as_float(fw[i][j]);
                bh[i] = tf32_hi(fv);
                bl[i] = tf32_lo(fv, bh[i]);
              }
              mma_tf32(d[j], ah, bl, code);
              if constexpr (LP == 2) mma_tf32(d[j], al, bh, code);
              mma_tf32(d[j], ah, bh, code);
            }
          }
        }
      };
      const int nq = min(AS, P4 - s * AS) / 4;  // angle quads of the stage
#pragma unroll
      for (int q = 0; q < AS / 4; ++q)
        if (q == 0 || q < nq) quad(q);
      if ((s + 1) % kPerFold == 0 || s + 1 == nstages) {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[j][i] = fadd(acc[j][i], d[j][i]);
      }
    }
  }

  // Slices that the products do not serve: their sums again, ray by ray, into shared
  // memory ([warp][16 pixels][U]; kept out of the accumulators' registers). A lane
  // takes one of the tile's 16 pixels and half of the angle quads.
  if constexpr (FK != FK_HALF) redo = redo_slices<FK == FK_SPLIT>(A, unit, lane);
  float* const again = reinterpret_cast<float*>(sm) + warp * 16 * U;
  static_assert(kMmaTiles * 16 * U * 4 <= St::kBytes, "the sums fit the stages");
  if (redo) {
    __syncthreads();  // the stages' last reads
    for (unsigned left = redo; left; left &= left - 1) {
      const int su = __ffs(left) - 1;
      const int px = X0 + (warp & 3) * 4 + (lane & 3);
      const int py = Y0 + (warp >> 2) * 4 + ((lane >> 2) & 3);
      float sum = 0.f;
      if (px < g && py < g) {
        int tile, tl;
        pixel_tile(px, py, A.M.tiles_x, A.M.tw_shift, &tile, &tl);
        sum = slow_sum<LK, FK == FK_HALF>(A, dl + ((int64_t)tile * 128 + tl * 4) * W, px, py,
                                          lane >> 4, unit_base, su);
      }
      sum = fadd(sum, __shfl_xor_sync(0xffffffffu, sum, 16));
      if (lane < 16) again[lane * U + su] = sum;
    }
    __syncwarp();
  }

  // ---- epilogue: the lane holds columns 2 t and 2 t + 1 of every accumulator
  // tile for its two pixels; column n of tile j is slice 8 j + n of the unit
  // with halves (NV vectors of N = 2 slices), n * NT + j with TF32 (one vector
  // of N = 2 NT)
  constexpr int N = F16 ? 2 : 2 * NT, NV = F16 ? NT : 1;
  // one loop body for the lane's 2 NV vectors (the sums move up to acc[0]):
  // unrolled, the penalties' code no longer fits the instruction cache
#pragma unroll 1
  for (int i = 0; i < 2 * NV; ++i) {
    const int v = i >> 1, h = i & 1;
    float num[N];
    if constexpr (F16) {
      num[0] = acc[0][0];
      num[1] = acc[0][1];
      float* f = &acc[0][0];
#pragma unroll
      for (int k = 0; k + 2 < 4 * NT; ++k) f[k] = f[k + 2];
    } else {
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        num[j] = acc[j][0];
        num[NT + j] = acc[j][1];
        acc[j][0] = acc[j][2];
        acc[j][1] = acc[j][3];
      }
    }
    const int su = F16 ? 8 * v + 2 * t : t * N;
    const int s0 = unit * U + su;
    const int n = min(N, A.S - s0);
    if (!(h ? vb : va) || n <= 0) continue;
    const int y = h ? yb : ya;
    const int p = y * g + x;  // g <= 32768
    int tile, tl;
    pixel_tile(x, y, A.M.tiles_x, A.M.tw_shift, &tile, &tl);
    const float Wp = FK == FK_HALF ? A.M.Wh[p] : A.M.W[p];
    const bool vecv = A.K >= N && ((s0 + A.vshift) & (N - 1)) == 0;
    const bool vecf = A.K >= N && ((s0 + A.fshift) & (N - 1)) == 0;
    if constexpr (FK == FK_SPLIT) {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (j < n) num[j] *= 1.f / split_scale(A.F.stat[s0 + j].most);
    }
    if (redo) {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (redo >> (su + j) & 1u) num[j] = again[(row + 8 * h) * U + su + j];
    }
    if constexpr (LK == LK_U16) {
#pragma unroll
      for (int j = 0; j < N; ++j) num[j] *= A.M.inv_scale;
    }
    for_each_exception(A.M, tile, tl, [&](float l, int ea, int ec) {
#pragma unroll
      for (int j = 0; j < N; ++j) {
        if (j >= n) continue;
        const int64_t e = factor_at(unit_base, RP, U, ea, ec, su + j);
        if constexpr (FK == FK_HALF)
          num[j] = fmaf(__half2float(__float2half_rn(l)),
                        __half2float(reinterpret_cast<const __half*>(A.F.base)[e]), num[j]);
        else
          num[j] = fmaf(l, reinterpret_cast<const float*>(A.F.base)[e], num[j]);
      }
    });
    if constexpr (FK == FK_HALF) {
      if (A.half_factors == FACT_HALF_M1) {
#pragma unroll
        for (int j = 0; j < N; ++j) num[j] += Wp;
      }
    }
    if constexpr (PEN) {  // the reconstruction factor, applied once per pixel
      float r[N];
      load_slots<N>(r, cur + slot_addr(s0 + A.fshift, p, g2, A.K), s0 + A.fshift, n, g2, A.K,
                    vecf);
#pragma unroll
      for (int j = 0; j < N; ++j) num[j] = -(r[j] * num[j]);
    }
    if (epi == EPI_REPLICA) {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (j < n) rep_num[(int64_t)(s0 + j) * g2 + p] = num[j];
      continue;
    }
    const int64_t base = slot_addr(s0 + A.vshift, 0, g2, A.K);
    float nv[N];
    if constexpr (!PEN) {
      float old[N];
      load_slots<N>(old, cur + base + (int64_t)p * A.K, s0 + A.vshift, n, g2, A.K, vecv);
#pragma unroll
      for (int j = 0; j < N; ++j)
        nv[j] = A.alg == 0 ? fadd(old[j], fdiv(num[j], Wp)) : fmul(old[j], fdiv(num[j], Wp));
    } else {
      float F[N], Gv[N];
      penalty_slices<N>(A, cur, cur + base, s0, n, x, y, p, g2, vecv, F, Gv);
#pragma unroll
      for (int j = 0; j < N; ++j)
        nv[j] = penalised_root_stable(F[j], fadd(Gv[j], Wp), num[j]);
    }
    float* out = next + base + (int64_t)p * A.K;
    if (vecv && n == N) {
      Vec<N> o;
#pragma unroll
      for (int j = 0; j < N; ++j) o.v[j] = nv[j];
      store_vec<N>(out, o);
    } else {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (j < n) out[slot_addr(s0 + j + A.vshift, 0, g2, A.K) - base] = nv[j];
    }
  }
}

// Resident blocks per SM that registers and shared memory are sized for.
template <int NT, int FK>
constexpr int mma_blocks_per_sm() {
  return NT == 1 ? 4 : FK == FK_TF32 && NT == 4 ? 2 : 3;
}

// Units first..first + nunits - 1 of the slices; a region's units are
// adjacent blocks, so that they read its matrix rows together (from L2).
template <int NT, int LK, int FK, int LP, bool PEN>
__global__ void __launch_bounds__(kMmaBlock, mma_blocks_per_sm<NT, FK>())
    k_backward_mma(const __grid_constant__ IterArgs A, int first, int nunits,
                   const float* __restrict__ cur, float* __restrict__ next,
                   float* __restrict__ rep_num, int epi) {
  const int region = blockIdx.x / nunits, unit = first + (int)blockIdx.x - region * nunits;
  backward_mma_block<NT, LK, FK, LP, PEN>(A, unit, region, cur, next, rep_num, epi);
}

// Many plans' fused backprojection + update in one launch.
template <int NT, int LK, int FK, int LP, bool PEN>
__global__ void __launch_bounds__(kMmaBlock, mma_blocks_per_sm<NT, FK>())
    k_backward_mma_multi(const BackItem* __restrict__ items, int nitems) {
  const BackItem& it = items[item_of(items, nitems, blockIdx.x)];
  const int b = (int)(blockIdx.x - it.first);
  const int region = b / it.nunits, unit = b - region * it.nunits;
  backward_mma_block<NT, LK, FK, LP, PEN>(it.A, unit, region, it.cur, it.next, nullptr,
                                            EPI_UPDATE);
}

template <int NT, int LK, int FK, int LP, bool PEN>
void mma_launch_pen(const IterArgs& A, int first, int nunits, const float* cur, float* next,
                    float* rep_num, int epi, cudaStream_t st) {
  constexpr int smem = MmaStage<NT, LK, FK>::kBytes;
  cudaFuncSetAttribute(k_backward_mma<NT, LK, FK, LP, PEN>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k_backward_mma<NT, LK, FK, LP, PEN>
      <<<(unsigned)(mma_regions(A.G.C) * nunits), kMmaBlock, smem, st>>>(A, first, nunits, cur,
                                                                         next, rep_num, epi);
}

template <int NT, int LK, int FK, int LP>
void mma_launch(const IterArgs& A, int first, int nunits, const float* cur, float* next,
                float* rep_num, int epi, cudaStream_t st) {
  if (A.alg >= 2)
    mma_launch_pen<NT, LK, FK, LP, true>(A, first, nunits, cur, next, rep_num, epi, st);
  else
    mma_launch_pen<NT, LK, FK, LP, false>(A, first, nunits, cur, next, rep_num, epi, st);
}

template <int NT, int LK, int FK, int LP, bool PEN>
void mma_multi_pen(const BackItem* items, int n, int64_t blocks, cudaStream_t st) {
  constexpr int smem = MmaStage<NT, LK, FK>::kBytes;
  cudaFuncSetAttribute(k_backward_mma_multi<NT, LK, FK, LP, PEN>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k_backward_mma_multi<NT, LK, FK, LP, PEN>
      <<<(unsigned)blocks, kMmaBlock, smem, st>>>(items, n);
}

template <int NT, int LK, int FK, int LP>
void mma_multi(const BackItem* items, int n, int64_t blocks, int pen, cudaStream_t st) {
  if (pen)
    mma_multi_pen<NT, LK, FK, LP, true>(items, n, blocks, st);
  else
    mma_multi_pen<NT, LK, FK, LP, false>(items, n, blocks, st);
}

}  // namespace

// Launches of one kind of factors and lengths, each in its own translation
// unit (tg_backward_mma_*.cu) so that the instances build in parallel; the
// multi-plan launches (TG_MMA_MULTI_ENTRY) serve plans with 16-bit fixed-point
// lengths.
#define TG_MMA_ENTRY(KIND, LK, FK, LP)                                                      \
  void launch_backward_mma_##KIND(const IterArgs& A, int first, int nunits,                \
                                  const float* recon_cur, float* recon_next,               \
                                  float* rep_num, int epi, cudaStream_t st) {              \
    if (A.F.U == 8)                                                                         \
      mma_launch<1, LK, FK, LP>(A, first, nunits, recon_cur, recon_next, rep_num, epi, st); \
    else if (A.F.U == 16)                                                                   \
      mma_launch<2, LK, FK, LP>(A, first, nunits, recon_cur, recon_next, rep_num, epi, st); \
    else                                                                                    \
      mma_launch<4, LK, FK, LP>(A, first, nunits, recon_cur, recon_next, rep_num, epi, st); \
  }
#define TG_MMA_MULTI_ENTRY(KIND, LK, FK, LP)                                                \
  void launch_backward_mma_multi_##KIND(const BackItem* items, int n, int64_t blocks,      \
                                        int U, int pen, cudaStream_t st) {                 \
    if (U == 8)                                                                             \
      mma_multi<1, LK, FK, LP>(items, n, blocks, pen, st);                                  \
    else if (U == 16)                                                                       \
      mma_multi<2, LK, FK, LP>(items, n, blocks, pen, st);                                  \
    else                                                                                    \
      mma_multi<4, LK, FK, LP>(items, n, blocks, pen, st);                                  \
  }

}  // namespace tg
