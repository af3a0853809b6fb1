// Strip-ordered forward projection on the tensor cores (half-gather plans with
// many slices).
//
// Rays of neighbouring angles run side by side for a while: within a chunk of
// R rows, the rays of four consecutive angles whose positions at the chunk's
// middle row fall into a strip of four pixels (at most four per angle, rays
// being at least a pixel apart) stay within eight pixels of one another. Such
// a bundle of 16 rays walks its strip four rows at a time, and each step is a
// small sparse matrix product: D[16 rays x slices] += A[16 x 32] B[32 x
// slices], the 32 columns of A being the strip's windows of eight pixels in
// the four rows. A ray takes at most three neighbouring pixels of a row, so
// with the even and the odd pixels of a window as the groups every group
// holds at most two lengths: the 2:4 sparsity of mma.sp.m16n8k32. The 16-bit
// length codes are two exact halves (high and low byte), i.e. two products
// per step with the same B; the sums stay with the bundle for the whole
// chunk.
//
// Rows are pixel rows for rays closer to the vertical, pixel columns for the
// others (cls). A block is 4 strips x 4 quads of angles: the 16 warps share
// the pixels of 24 columns by 8 rows per stage, copied to shared memory as
// halves with cp.async; A comes from memory as the lanes need it (one 512-byte
// row of codes and 64 bytes of metadata per bundle and step). Each bundle
// stores its 16 x U sums once per chunk; the finish kernel adds a ray's chunks
// in order.
//
// The tile-staged forward (tg_tiles.cu) reads a 16-byte pixel vector from
// shared memory per segment and 8 slices and is bound by those wavefronts
// (94 %) and issue (77 %). 1024 x 1024, 720 angles, 64 slices: 7.8 ms there
// with 0.4 for its finish, 4.0 and 0.73 here; 2048 x 2048, 1500 angles: 56 and
// 3 there, 29.8 and 3.0 here. Here one block of 16 warps fills an SM (128
// registers a thread); tensor pipe 38 %, shared memory 59 %, DRAM 41 %, and the
// rest waits: the stage's barrier and the chain ldmatrix - product - sum.
//
// Segments that do not fit (stray ones, far from their ray) are kept apart in
// a list per ray and added by the finish kernel.
#include <algorithm>
#include <climits>

#include "tg_segments.cuh"

namespace tg {

namespace {

constexpr int kStripWarps = 16;  // 4 strips x 4 quads of angles
constexpr int kStripBlock = kStripWarps * 32;
constexpr int kStripStage = 8;   // rows per stage (two steps, two rows per warp pair)
constexpr int kStripBufs = 4;
constexpr int kFinishWarps = 8;

// Byte address of pixel column `col` in staged row rr, chunk 0 of 16 bytes;
// chunk c is at this address ^ 16 c. The eight pixels of one ldmatrix matrix
// are every other pixel of two neighbouring rows: the row's parity and the
// pixel's bits 1 and 2 put them in eight different bank groups.
template <int NT>
__device__ __forceinline__ uint32_t staged(int rr, int col) {
  const uint32_t p = (col >> 1) & 3;
  if constexpr (NT == 8)
    return (uint32_t)(rr * kStripCols + col) * 128u + ((p | ((rr & 1) << 2)) << 4);
  else
    return (uint32_t)((rr >> 1) * kStripCols + col) * 128u + ((rr & 1) << 6) + (p << 4);
}

// First pixel of the window of `width` strips' worth of positions starting at
// strip `strip`, in row m of a chunk whose middle is mid: positions at m spread
// by the slopes' half range.
__device__ __forceinline__ int strip_base(const StripSlopes& s, int strip, float mid, int m) {
  const float d = (float)m + 0.5f - mid;
  return __float2int_rd(__fmaf_rn(d, s.mid, (float)(strip * 4)) - __fmaf_rn(fabsf(d), s.half, s.ext));
}

// Strip (relative to the first) and slot 0..3 of ray (a, c) in chunk j: rays
// are numbered along the strip's 2^22 positions, |sigma| >= 2^20 apart.
__device__ __forceinline__ void ray_strip(const StripDev& S, int j, int a, int c, int* strip,
                                          int* slot) {
  const int64_t sg = S.sigma[a], at = S.alpha[(int64_t)j * S.P + a] + sg * c;
  const int64_t k = at >> 22;
  const int p = (int)(at - (k << 22)), d = (int)(sg < 0 ? -sg : sg);
  *slot = (p >= d) + (p >= 2 * d) + (p >= 3 * d);
  *strip = (int)(k - S.strip0);
}

__device__ __forceinline__ int64_t bundle_of(const StripDev& S, int j, int a, int strip) {
  const int hq = S.place[a];  // (block of 16 angles) * 16 + quad * 4 + angle
  return (((int64_t)j * S.nblk16 + (hq >> 4)) * S.nstrips + strip) * 4 + ((hq >> 2) & 3);
}

// ---- construction -------------------------------------------------------------
// A warp's 32 rays (one group of the ray-ordered matrix), row by row from its
// first row on, so that the lanes stay within a few segments of one another:
// the next 64 segments' codes and step codes wait in shared memory, in pieces
// of 8, and a lane that is not within them reads the matrix itself. (One lane
// per ray, segment by segment, ran every lane's row ends at another time: 9.1
// ms at 1024 x 1024, 720 angles, 6.2 so.)
constexpr int kFillWarps = 4;
constexpr int kPieces = 8;

struct FillRing {
  unsigned short len[kPieces][8][32];
  uint32_t word[kPieces][32];
};

// One row's window of eight pixels: 16-bit codes of the even (x, y) and the
// odd (z, w) ones.
struct FillRow {
  uint32_t x, y, z, w;
};

// The pair of columns of a group's two words (four codes) and its metadata
// nibble; what lies off that pair comes back in `rest`.
__device__ __forceinline__ uint32_t group_pair(uint32_t lo, uint32_t hi, uint32_t* nibble,
                                               uint2* rest) {
  const bool mid = (lo >> 16) && (hi & 0xffffu), upper = !lo;
  *nibble = mid ? 9u : upper ? 14u : 4u;
  *rest = mid ? make_uint2(lo & 0xffffu, hi & 0xffff0000u) : make_uint2(0u, upper ? 0u : hi);
  return mid ? __funnelshift_r(lo, hi, 16) : upper ? hi : lo;
}

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}

template <bool DELTA>
__global__ void __launch_bounds__(kFillWarps * 32)
    k_strips_fill(DevGeom G, MatrixDev M, StripDev S, uint2* codes, unsigned short* meta,
                  uint8_t* grazed, StripExc* exc, int exc_cap, int* nexc) {
  __shared__ __align__(16) FillRing s_ring[DELTA ? kFillWarps : 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * kFillWarps + warp;
  if (grp >= G.P * G.gpa) return;  // a whole warp
  FillRing& ring = s_ring[DELTA ? warp : 0];
  const int a = grp / G.gpa, c = (grp - a * G.gpa) * 32 + lane;
  const int g = G.C;
  const int64_t r = (int64_t)a * g + c;
  const int n = c < g ? M.rnseg[r] : 0;
  const int cap = M.rcap[grp];
  const int64_t lbase = M.roff[grp], cbase = DELTA ? M.rcoff[grp] : 0;
  const unsigned short* lens = reinterpret_cast<const unsigned short*>(M.rlen);
  const float inv_g = 1.0f / (float)g;
  const int cls = S.cls[a];
  const StripSlopes sl = S.quad[S.place[a] >> 2];
  const int dir = cls ? 1 : G.quad[a] ? 1 : -1;  // rows along the path

  int loaded = 0, ready = 0;  // pieces asked for, pieces here
  auto ask = [&](int upto) {
    if constexpr (DELTA) {
      for (; loaded < upto && loaded * 8 < cap; ++loaded) {
        const int k = loaded & (kPieces - 1);
        if (loaded * 8 + (lane >> 2) < cap)
          cp_async16((uint32_t)__cvta_generic_to_shared(&ring.len[k][lane >> 2][(lane & 3) * 8]),
                     lens + lbase + (int64_t)loaded * 256 + lane * 8);
        if (lane < 8)
          cp_async16((uint32_t)__cvta_generic_to_shared(&ring.word[k][lane * 4]),
                     M.rcode + cbase + (int64_t)loaded * 32 + lane * 4);
      }
    }
  };
  // the current segment
  int s = 0, ix = 0, iy = 0;
  uint32_t code = 0;
  auto fetch = [&]() {
    const int64_t e = lbase + lane + (int64_t)s * 32;
    if constexpr (DELTA) {
      const int k = s >> 3;
      uint32_t word;
      if (k < ready) {
        code = ring.len[k & (kPieces - 1)][s & 7][lane];
        word = ring.word[k & (kPieces - 1)][lane];
      } else {
        code = lens[e];
        word = M.rcode[cbase + lane + (int64_t)k * 32];
      }
      if (s > 0) {
        const uint32_t st = (word >> (4 * (s & 7))) & 15u;
        ix += (int)(st & 1u);
        iy += (int)(st >> 1) - 1;
      }
    } else {
      code = lens[e];
      cell_xy(M.ridx[e], g, inv_g, ix, iy);
    }
  };
  auto except = [&](int idx, uint32_t l) {
    const int k = atomicAdd(nexc, 1);
    if (k < exc_cap) exc[k] = StripExc{(int)r, idx, (int)l, 0};
  };

  ask(kPieces);
  if (n > 0) {
    if constexpr (DELTA) cell_xy(M.rstart[r], g, inv_g, ix, iy);
    fetch();
  }
  // row m and the one after it: their windows' first pixels and codes. Rows
  // start with a whole step of four. Two rows are open at a time: the
  // reference's tracer can return to the previous row for a segment (float
  // jitter in the crossing points).
  const int m0 = cls ? ix : iy;
  int m = dir > 0 ? m0 & ~3 : m0 | 3;
  int chunk = -1, strip = 0, slot = 0, base = 0;  // of row m + dir
  auto next_row = [&](int row) {
    const int j = (int)__umulhi((uint32_t)min(max(row, 0), g - 1), S.rmul);
    if (j != chunk) {
      chunk = j;
      ray_strip(S, j, a, c, &strip, &slot);
    }
    base = strip_base(sl, strip + S.strip0, ((float)j + 0.5f) * (float)S.R, row);
  };
  if (n > 0) next_row(m);
  FillRow w1{0, 0, 0, 0};
  auto open = [&]() { return s < n || (w1.x | w1.y | w1.z | w1.w) != 0u; };
  while (__any_sync(0xffffffffu, open())) {
    if constexpr (DELTA) {
      // what was asked for a step ago is here; slots before the hindmost lane
      // are free
      const int low = __reduce_min_sync(0xffffffffu, s < n ? s : INT_MAX);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      ready = loaded;
      if (low != INT_MAX) ask((low >> 3) + kPieces);
    }
    if (open()) {
      const int step_chunk = chunk, step_strip = strip, step_slot = slot, step_m = m;
      uint32_t word[4][2];
      uint32_t me = 0x4444u, mo = 0x4444u;
      bool any = false;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        FillRow w0 = w1;
        w1 = FillRow{0, 0, 0, 0};
        const int base0 = base, strip0 = strip;
        next_row(m + dir);
        while (s < n) {
          const int k = ((cls ? ix : iy) - m) * dir;
          if (k > 1) break;
          const int o = (cls ? iy : ix) - (k == 1 ? base : base0);
          const int st = k == 1 ? strip : strip0;
          const bool in = k >= 0 && (unsigned)o <= 7u && (unsigned)st < (unsigned)S.nstrips;
          // into word (o & 1, o >> 2) of the row
          const int sh = (o & 2) << 3;
          const uint32_t add = code << sh;
          const uint32_t e0 = k == 1 ? w1.x : w0.x, e1 = k == 1 ? w1.y : w0.y;
          const uint32_t e2 = k == 1 ? w1.z : w0.z, e3 = k == 1 ? w1.w : w0.w;
          const uint32_t had = (o & 4) ? ((o & 1) ? e3 : e1) : ((o & 1) ? e2 : e0);
          const bool fits = in && ((had >> sh) & 0xffffu) + code <= 0xffffu;
          if (code == 0u) {
            grazed[iy * g + ix] = 1;
          } else if (!fits) {
            except(iy * g + ix, code);
          } else if (k == 1) {
            w1.x += (o & 5) == 0 ? add : 0u;
            w1.y += (o & 5) == 4 ? add : 0u;
            w1.z += (o & 5) == 1 ? add : 0u;
            w1.w += (o & 5) == 5 ? add : 0u;
          } else {
            w0.x += (o & 5) == 0 ? add : 0u;
            w0.y += (o & 5) == 4 ? add : 0u;
            w0.z += (o & 5) == 1 ? add : 0u;
            w0.w += (o & 5) == 5 ? add : 0u;
          }
          if (++s < n) fetch();
        }
        if (w0.x | w0.y | w0.z | w0.w) {
          any = true;
          uint32_t ce, co;
          uint2 re, ro;
          word[i][0] = group_pair(w0.x, w0.y, &ce, &re);
          word[i][1] = group_pair(w0.z, w0.w, &co, &ro);
          me ^= (4u ^ ce) << (4 * (m & 3));
          mo ^= (4u ^ co) << (4 * (m & 3));
          if (re.x | re.y | ro.x | ro.y) {  // a third code of a group
            const uint32_t left[4] = {re.x, re.y, ro.x, ro.y};
            for (int q = 0; q < 8; ++q) {
              const uint32_t l = (left[q >> 1] >> (16 * (q & 1))) & 0xffffu;
              const int v = base0 + 2 * (q & 3) + (q >> 2);
              if (l) except(cls ? v * g + m : m * g + v, l);
            }
          }
        } else {
          word[i][0] = word[i][1] = 0u;
        }
        m += dir;
      }
      if (any) {
        // 32 bytes of codes per ray and step; metadata word (row16 & 7,
        // parity), upper half for rays 8..15
        const int row16 = (S.place[a] & 3) * 4 + step_slot;
        const int64_t step = bundle_of(S, step_chunk, a, step_strip) * (S.R / 4) +
                             ((step_m - step_chunk * S.R) >> 2);
        uint4* d = reinterpret_cast<uint4*>(codes + (step * 16 + row16) * 4);
        const bool up = dir > 0;
        d[up ? 0 : 1] = up ? make_uint4(word[0][0], word[0][1], word[1][0], word[1][1])
                           : make_uint4(word[1][0], word[1][1], word[0][0], word[0][1]);
        d[up ? 1 : 0] = up ? make_uint4(word[2][0], word[2][1], word[3][0], word[3][1])
                           : make_uint4(word[3][0], word[3][1], word[2][0], word[2][1]);
        unsigned short* q = meta + step * 32 + ((row16 & 7) * 2) * 2 + (row16 >> 3);
        q[0] = (unsigned short)me;
        q[2] = (unsigned short)mo;
      }
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Pixel indices and length codes of the rays' segments in the ray-ordered
// matrix's layout, for a plan that does not keep it.
__global__ void __launch_bounds__(128)
    k_strips_trace(DevGeom G, MatrixDev M, int* ridx, uint16_t* rlen) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= (int64_t)G.P * G.C) return;
  const int a = (int)(r / G.C), c = (int)(r - (int64_t)a * G.C);
  int64_t e = M.roff[a * G.gpa + (c >> 5)] + (c & 31);
  ray_segments<kSrcTrace, kLenCode>(G, M, r, [&](int idx, int, int, float, uint16_t code) {
    ridx[e] = idx;
    rlen[e] = code;
    e += 32;
  });
}

// FP32 reconstruction slots -> halves [pixel][U]; one thread per pixel
// and 8 slices. A product runs over whole windows, so a non-finite pixel would
// reach rays beside it: one that no ray crosses, not even with a zero length
// (0 / 0 in the updates), becomes 0; any other marks its slice in `bad`, and the
// rays of that slice are then walked. Resets the stat of nstat slices.
__global__ void k_strips_image(const float* __restrict__ recon, __half* __restrict__ img,
                               int64_t g2, int K, int U, int S, int first_slot, int first,
                               int64_t n, const float* __restrict__ W,
                               const uint8_t* __restrict__ grazed, int* bad,
                               FactorStat* stat, int nstat) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.x == 0 && threadIdx.x < nstat) stat[threadIdx.x] = FactorStat{};
  if (i >= n) return;
  const int oct = U / 8;
  const int o = (int)(i % oct);
  const int64_t p = i / oct;
  const int s0 = first + o * 8;
  Vec<8> v;
  if (K >= 8 && s0 < S) {  // first_slot is a multiple of K
    v = load_vec<8>(recon + slot_addr(s0 + first_slot, p, g2, K));
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (s0 + j >= S) v.v[j] = 0.f;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      v.v[j] = s0 + j < S ? __ldg(recon + slot_addr(s0 + j + first_slot, p, g2, K)) : 0.f;
  }
  bool finite = true;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v.v[j] = __half2float(__float2half_rn(v.v[j]));
    finite &= fabsf(v.v[j]) < 7e4f;
  }
  if (!finite) {
    const bool crossed = W[p] != 0.f || grazed[p];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (fabsf(v.v[j]) < 7e4f) continue;
      if (crossed) bad[o * 8 + j] = 1;
      else v.v[j] = 0.f;
    }
  }
  store_hvec<8>(img + p * U + o * 8, v);
}

// One ray's sum of one slice, segment by segment.
__device__ __noinline__ float walk_ray(const DevGeom& G, const MatrixDev& M, int src, int64_t r,
                                       const __half* im, int U) {
  float s = 0.f;
  auto add = [&](int idx, int, int, float, uint16_t code) {
    s = fmaf((float)code * M.inv_scale, __half2float(im[(int64_t)idx * U]), s);
  };
  if (src == kSrcDelta) ray_segments<kSrcDelta, kLenCode>(G, M, r, add);
  else if (src == kSrcIndex) ray_segments<kSrcIndex, kLenCode>(G, M, r, add);
  else ray_segments<kSrcTrace, kLenCode>(G, M, r, add);
  return s;
}

__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&b)[4], uint32_t smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
               : "r"(smem));
}
__device__ __forceinline__ void mma_sp(float (&d)[4], const uint32_t (&a)[4],
                                       const uint32_t (&b)[4], uint32_t e) {
  asm("mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.f16.f16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9,%10,%11}, {%0,%1,%2,%3}, %12, 0x0;"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]),
        "r"(e));
}

// Two 16-bit codes as halves: the high bytes, and the low bytes / 256.
__device__ __forceinline__ uint32_t high_halves(uint32_t w) {
  const uint32_t v = __byte_perm(w, 0x64646464u, 0x4341);  // 1024 + byte
  __half2 h;
  memcpy(&h, &v, 4);
  h = __hsub2(h, __float2half2_rn(1024.f));
  uint32_t o;
  memcpy(&o, &h, 4);
  return o;
}
__device__ __forceinline__ uint32_t low_halves(uint32_t w) {
  const uint32_t v = __byte_perm(w, 0x64646464u, 0x4240);
  __half2 h;
  memcpy(&h, &v, 4);
  h = __hfma2(h, __float2half2_rn(1.f / 256.f), __float2half2_rn(-4.f));  // exact
  uint32_t o;
  memcpy(&o, &h, 4);
  return o;
}

// Bytes of one stage: the block's pixels, then each warp's codes and metadata
// of two steps.
template <int NT>
struct StripStage {
  static constexpr int kPix = kStripStage * kStripCols * NT * 16;
  static constexpr int kCodes = kStripWarps * 1024, kMeta = kStripWarps * 128;
  static constexpr int kBytes = kPix + kCodes + kMeta;
};

// One block: 4 strips x 4 quads of one block of 16 angles, 8 NT slices, down
// all rows of the grid: the stages run on across the chunks, at whose ends the
// sums go out.
template <int NT>
__global__ void __launch_bounds__(kStripBlock, 1)
    k_forward_strips(const __grid_constant__ StripDev S, int g, float scale,
                     const __half* __restrict__ img, float* __restrict__ part) {
  using St = StripStage<NT>;
  constexpr int U = 8 * NT;
  extern __shared__ __align__(128) uint4 smem_strip[];
  const uint32_t sm = (uint32_t)__cvta_generic_to_shared(smem_strip);
  const int per16 = S.nstrips / 4;
  const int sg = blockIdx.x % per16, h16 = blockIdx.x / per16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = lane >> 2, t = lane & 3;
  const int sw = warp >> 2, quad = warp & 3;  // strip of the block, quad of angles
  // the warp's bundle in chunk 0, and from one chunk to the next
  const int64_t bundle0 = ((int64_t)h16 * S.nstrips + sg * 4 + sw) * 4 + quad;
  const int64_t bstep = (int64_t)S.nblk16 * S.nstrips * 4;
  const int cls = S.cls16[h16];
  const StripSlopes s16 = S.blk16[h16], sq = S.quad[h16 * 4 + quad];
  const int strip_b = S.strip0 + sg * 4, strip_w = strip_b + sw;
  const int nst = (g + kStripStage - 1) / kStripStage, per_chunk = S.R / kStripStage;
  const int nks = S.R / 4;

  // copies: a warp half a row (14 pixels), lanes chunks of 16 bytes
  constexpr int kPer = 32 / NT, kCopies = (kStripCols / 2 + kPer - 1) / kPer;
  const int crow = warp >> 1, cpix = lane / NT, cchunk = lane % NT;
  const int ccol = (warp & 1) * (kStripCols / 2) + cpix;
  uint32_t cdst[kCopies];
#pragma unroll
  for (int i = 0; i < kCopies; ++i)
    cdst[i] = sm + (staged<NT>(crow, ccol + i * kPer) ^ (cchunk << 4));
  const int sm_m = cls ? 1 : g, sm_n = cls ? g : 1;  // pixel index strides
  const char* im = reinterpret_cast<const char*>(img) + cchunk * 16;
  const char* codes = reinterpret_cast<const char*>(S.codes);
  const char* meta = reinterpret_cast<const char*>(S.meta);
  const uint32_t a_dst = sm + St::kPix + warp * 1024 + lane * 16;
  const uint32_t m_dst = sm + St::kPix + St::kCodes + warp * 128 + lane * 16;
  int copy_j = 0, copy_s = 0;  // chunk and its stage of the next copy
  auto copy = [&](int s) {
    const uint32_t buf = (s % kStripBufs) * St::kBytes;
    const float mid = ((float)copy_j + 0.5f) * (float)S.R;
    const int m = s * kStripStage + crow;
    // pixels outside the grid hold no lengths: any pixel will do
    const int n0 = strip_base(s16, strip_b, mid, m) + ccol;
    const int pm = min(m, g - 1) * sm_m;
#pragma unroll
    for (int i = 0; i < kCopies; ++i)
      if ((i + 1) * kPer <= kStripCols / 2 || cpix + i * kPer < kStripCols / 2) {
        const int p = pm + min(max(n0 + i * kPer, 0), g - 1) * sm_n;
        cp_async16(cdst[i] + buf, im + (int64_t)p * (U * 2));
      }
    const int64_t step = (bundle0 + copy_j * bstep) * nks + copy_s * 2;
    const char* c = codes + step * 512 + lane * 16;
    cp_async16(a_dst + buf, c);
    cp_async16(a_dst + buf + 512, c + 512);
    if (lane < 8) cp_async16(m_dst + buf, meta + step * 64 + lane * 16);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++copy_s == per_chunk) {
      copy_s = 0;
      ++copy_j;
    }
  };

  float acc[NT][4], d[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = d[n][i] = 0.f;
  // B: register lane >> 3 holds the columns 8 (lane >> 3) ..: row (lane >> 2) & 3
  // of the step, pixels of parity lane >> 4
  const int lq = (lane >> 2) & 3, lpos = 2 * (lane & 3) + (lane >> 4);
  const uint32_t a_src = sm + St::kPix + warp * 1024 + (row * 4 + t) * 8;
  const uint32_t m_src = sm + St::kPix + St::kCodes + warp * 128 + (row * 2 + (t & 1)) * 4;
#pragma unroll
  for (int s = 0; s < kStripBufs - 1; ++s)
    if (s < nst) copy(s);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  int j = 0, js = 0;  // chunk, and its stage
  for (int s = 0; s < nst; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStripBufs - 2) : "memory");
    __syncthreads();
    if (s + kStripBufs - 1 < nst) copy(s + kStripBufs - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const uint32_t buf = (s % kStripBufs) * St::kBytes;
    // the warp's window in the staged columns of the stage's eight rows
    const float mid = ((float)j + 0.5f) * (float)S.R;
    const int m = s * kStripStage + (lane & 7);
    const int off = min(max(strip_base(sq, strip_w, mid, m) - strip_base(s16, strip_b, mid, m), 0),
                        kStripCols - 8);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      // A: rays row and row + 8, window row t: even pixels' pair, odd pixels'
      uint32_t w[4], code, ah[4], al[4];
      asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w[0]), "=r"(w[2]) : "r"(a_src + buf + q * 512));
      asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w[1]), "=r"(w[3]) : "r"(a_src + buf + q * 512 + 256));
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(code) : "r"(m_src + buf + q * 64));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ah[i] = high_halves(w[i]);
        al[i] = low_halves(w[i]);
      }
      const int o = __shfl_sync(0xffffffffu, off, q * 4 + lq);
      const uint32_t at = sm + buf + staged<NT>(q * 4 + lq, o + lpos);
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        uint32_t b[4];
        ldmatrix4_trans(b, at ^ (n << 4));
        mma_sp(d[n], al, b, code);
        mma_sp(d[n], ah, b, code);
      }
    }
    ++js;
    const bool last = js == per_chunk || s + 1 == nst;
    if (last || (js & 3) == 0) {  // every 8 steps
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[n][i] = fadd(acc[n][i], d[n][i]);
          d[n][i] = 0.f;
        }
    }
    if (last) {
      // column n of accumulator tile k is slice 8 k + n
      float* out = part + ((bundle0 + j * bstep) * 16 + row) * U + 2 * t;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          __stcs(reinterpret_cast<float2*>(out + 8 * i * U + n * 8),
                 make_float2(acc[n][2 * i] * scale, acc[n][2 * i + 1] * scale));
          acc[n][2 * i] = acc[n][2 * i + 1] = 0.f;
        }
      js = 0;
      ++j;
    }
  }
}

// Stores the per-ray value of slice s from its sum v (b: the sinogram's value, at:
// its place there); returns |factor|.
template <bool FH>
__device__ __forceinline__ float ray_value(const FactorDev& F, float* sim, int64_t at, int a,
                                           int c, int n, int s, float v, float b, float a2,
                                           int out_mode, float fofs) {
  if (out_mode == FWD_SIM) {
    sim[at] = v;
    return 0.f;
  }
  float o = 0.f;
  if (n > 0) {
    o = out_mode == FWD_SIRT ? fdiv(fsub(b, v), a2) : fdiv(b, v);
    if constexpr (FH) o -= fofs;
  }
  const int u = s / F.U;
  const int64_t e = factor_at((int64_t)(u % F.ring) * F.unit_elems, F.RP, F.U, a, c, s % F.U);
  if constexpr (FH) {
    const __half h = __float2half_rn(o);
    reinterpret_cast<__half*>(F.base)[e] = h;
    if (!(fabsf(__half2float(h)) < 7e4f)) F.stat[s].bad = 1;
  } else {
    reinterpret_cast<float*>(F.base)[e] = o;
    if (!(fabsf(o) < 1e38f)) F.stat[s].bad = 1;
  }
  return fabsf(o);
}

// The marked slices' rays, walked: one of a warp's 32 rays per lane. The last
// block clears the marks for the next launch.
template <bool FH>
__global__ void __launch_bounds__(kFinishWarps * 32)
    k_strips_walk(const __grid_constant__ DevGeom G, const __grid_constant__ MatrixDev M,
                  const __grid_constant__ FactorDev F, int src, int* bad,
                  const __half* __restrict__ img, const float* __restrict__ sino,
                  float* __restrict__ sim, int U, int first, int nslices, int64_t K, int out_mode,
                  float fofs) {
  const int lane = threadIdx.x & 31;
  const int64_t nrays = (int64_t)G.P * G.C;
  for (int k = 0; k < U; k += 32)
    for (unsigned left = __ballot_sync(0xffffffffu, bad[k + lane] != 0); left; left &= left - 1) {
      const int su = k + __ffs(left) - 1, s = first + su;
      if (s >= nslices) continue;
      float most = 0.f;
      for (int64_t grp = (int64_t)blockIdx.x * kFinishWarps + (threadIdx.x >> 5);
           grp < (int64_t)G.P * G.gpa; grp += (int64_t)gridDim.x * kFinishWarps) {
        const int a = (int)(grp / G.gpa), c = (int)(grp - (int64_t)a * G.gpa) * 32 + lane;
        if (c >= G.C) continue;
        const int64_t r = (int64_t)a * G.C + c, at = s / K * nrays * K + r * K + s % K;
        most = fmaxf(most, ray_value<FH>(F, sim, at, a, c, M.rnseg[r], s,
                                         walk_ray(G, M, src, r, img + su, U),
                                         out_mode != FWD_SIM ? __ldg(sino + at) : 0.f,
                                         out_mode == FWD_SIRT ? M.ra2[r] : 1.f, out_mode, fofs));
      }
      if (!FH && out_mode != FWD_SIM && F.split && most > 0.f)
        atomicMax(&F.stat[s].most, __float_as_uint(most));
    }
  __syncthreads();  // the block has read the marks
  if (threadIdx.x == 0 && atomicAdd(bad + 64, 1) == (int)gridDim.x - 1)
    for (int i = 0; i <= 64; ++i) bad[i] = 0;
}

// One warp per ray (grid-strided): its chunks' sums in order (lane = U / 32
// slices), the exceptions, then the per-ray value of every slice: factors into
// F's units (half or float, with the stat of finish_units_ray), or the ray sums
// (sim). Slices marked in `bad` are k_strips_walk's.
template <int U, bool FH>
__global__ void __launch_bounds__(kFinishWarps * 32)
    k_strips_finish(const __grid_constant__ DevGeom G, const __grid_constant__ MatrixDev M,
                    const __grid_constant__ StripDev S, const __grid_constant__ FactorDev F,
                    const int* __restrict__ bad, const float* __restrict__ part,
                    const __half* __restrict__ img, const float* __restrict__ sino,
                    float* __restrict__ sim, int first, int nslices, int K, int out_mode,
                    float fofs) {
  constexpr int N = U / 32;
  const int lane = threadIdx.x & 31;
  const int64_t nrays = (int64_t)G.P * G.C;
  const int s0 = first + lane * N;  // the lane's slices
  float most[N];
  unsigned walk = 0;  // a bit per slice of the lane
#pragma unroll
  for (int k = 0; k < N; ++k) {
    most[k] = 0.f;
    walk |= bad[lane * N + k] ? 1u << k : 0u;
  }
  const int64_t w0 = (int64_t)blockIdx.x * kFinishWarps + (threadIdx.x >> 5);
  for (int64_t r = w0; r < nrays; r += (int64_t)gridDim.x * kFinishWarps) {
    const int a = (int)(r / G.C), c = (int)(r - (int64_t)a * G.C);
    float v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = 0.f;
    const int n = M.rnseg[r];
    float b[N];  // the sinogram's values, in flight with the sums
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int s = s0 + k;
      b[k] = s < nslices && out_mode != FWD_SIM
                 ? __ldg(sino + (int64_t)(s / K) * nrays * K + r * K + s % K)
                 : 0.f;
    }
    for (int j0 = 0; n > 0 && j0 < S.nchunks; j0 += 32) {
      // the ray's row of sums in chunk j0 + lane
      int64_t at = -1;
      if (j0 + lane < S.nchunks) {
        int strip, slot;
        ray_strip(S, j0 + lane, a, c, &strip, &slot);
        if ((unsigned)strip < (unsigned)S.nstrips)
          at = bundle_of(S, j0 + lane, a, strip) * 16 + (S.place[a] & 3) * 4 + slot;
      }
      const int nj = min(32, S.nchunks - j0);
      for (int j = 0; j < nj; j += 8) {  // eight rows in flight
        Vec<N> q[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int64_t x = __shfl_sync(0xffffffffu, at, (j + i) & 31);
#pragma unroll
          for (int k = 0; k < N; ++k) q[i].v[k] = 0.f;
          if (j + i < nj && x >= 0) q[i] = load_vec_cs<N>(part + x * U + lane * N);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int k = 0; k < N; ++k) v[k] = fadd(v[k], q[i].v[k]);
      }
    }
    if (S.exc_first) {
      for (int e = S.exc_first[r]; e < S.exc_first[r + 1]; ++e) {
        const StripExc x = S.exc[e];
        const float l = (float)x.code * M.inv_scale;
#pragma unroll
        for (int k = 0; k < N; ++k)
          v[k] = fmaf(l, __half2float(img[(int64_t)x.idx * U + lane * N + k]), v[k]);
      }
    }
    const float a2 = out_mode == FWD_SIRT ? M.ra2[r] : 1.f;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int s = s0 + k;
      if (s >= nslices || (walk >> k & 1u)) continue;
      const int64_t at = (int64_t)(s / K) * nrays * K + r * K + s % K;
      const float f = ray_value<FH>(F, sim, at, a, c, n, s, v[k], b[k], a2, out_mode, fofs);
      if constexpr (!FH) most[k] = fmaxf(most[k], f);
    }
  }
  if constexpr (!FH) {
    if (out_mode != FWD_SIM && F.split) {
      // one atomic per block and slice (the order of floats' bits)
      __shared__ float s_most[kFinishWarps][U];
#pragma unroll
      for (int k = 0; k < N; ++k) s_most[threadIdx.x >> 5][lane * N + k] = most[k];
      __syncthreads();
      for (int k = threadIdx.x; k < U; k += blockDim.x) {
        float m = 0.f;
        for (int w = 0; w < kFinishWarps; ++w) m = fmaxf(m, s_most[w][k]);
        const int s = first + k;
        if (s < nslices && m > 0.f) atomicMax(&F.stat[s].most, __float_as_uint(m));
      }
    }
  }
}

template <int NT>
void forward_strips(const StripDev& S, int g, float scale, const __half* img, float* part,
                    cudaStream_t st) {
  constexpr int smem = kStripBufs * StripStage<NT>::kBytes;
  cudaFuncSetAttribute(k_forward_strips<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k_forward_strips<NT><<<(unsigned)(S.nblk16 * (S.nstrips / 4)), kStripBlock, smem, st>>>(
      S, g, scale, img, part);
}

}  // namespace

void launch_strips_trace(const DevGeom& G, const MatrixDev& M, int* ridx, uint16_t* rlen,
                         cudaStream_t st) {
  const int64_t R = (int64_t)G.P * G.C;
  k_strips_trace<<<(unsigned)((R + 127) / 128), 128, 0, st>>>(G, M, ridx, rlen);
}

void launch_strips_fill(const DevGeom& G, const MatrixDev& M, const StripDev& S, uint2* codes,
                        uint32_t* meta, uint8_t* grazed, StripExc* exc, int exc_cap, int* nexc,
                        cudaStream_t st) {
  const unsigned blocks = (unsigned)(((int64_t)G.P * G.gpa + kFillWarps - 1) / kFillWarps);
  unsigned short* m = reinterpret_cast<unsigned short*>(meta);
  if (M.rcode)
    k_strips_fill<true><<<blocks, kFillWarps * 32, 0, st>>>(G, M, S, codes, m, grazed, exc,
                                                            exc_cap, nexc);
  else
    k_strips_fill<false><<<blocks, kFillWarps * 32, 0, st>>>(G, M, S, codes, m, grazed, exc,
                                                             exc_cap, nexc);
}

void launch_strips_forward(const IterArgs& A, const StripDev& S, int first, int U,
                           const float* recon, __half* img, float* part, int reset,
                           cudaStream_t st) {
  const int g = A.G.C;
  const int64_t g2 = (int64_t)g * g;
  const int64_t n = g2 * (U / 8);
  k_strips_image<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(recon, img, g2, A.K, U, A.S,
                                                             A.fshift, first, n, A.M.W, S.grazed, S.bad,
                                                             A.F.stat + first,
                                                             reset ? min(U, A.S - first) : 0);
  const float scale = A.M.inv_scale * 256.f;
  if (U == 64)
    forward_strips<8>(S, g, scale, img, part, st);
  else
    forward_strips<4>(S, g, scale, img, part, st);
}

void launch_strips_finish(const IterArgs& A, const StripDev& S, int first, int U,
                          const __half* img, const float* part, const float* sino, float* sim,
                          int out_mode, cudaStream_t st) {
  const int64_t rays = (int64_t)A.G.P * A.G.C;
  // a few rays per warp: the largest factors cost one atomic per block and slice
  const unsigned bx = (unsigned)std::min<int64_t>((rays + kFinishWarps - 1) / kFinishWarps, 152 * 32);
#define TG_FIN(UU, FH)                                                                       \
  k_strips_finish<UU, FH><<<bx, kFinishWarps * 32, 0, st>>>(                                 \
      A.G, A.M, S, A.F, S.bad, part, img, sino, sim, first, A.S, A.K, out_mode,              \
      factor_offset(A.half_factors))
  const bool fh = A.half_factors != FACT_F32 && out_mode == FWD_RATIO;
  if (U == 64) {
    if (fh) TG_FIN(64, true); else TG_FIN(64, false);
  } else {
    if (fh) TG_FIN(32, true); else TG_FIN(32, false);
  }
#undef TG_FIN
#define TG_WALK(FH)                                                                        \
  k_strips_walk<FH><<<(unsigned)std::min<int64_t>(bx, 152 * 4), kFinishWarps * 32, 0, st>>>( \
      A.G, A.M, A.F, seg_source(A.M), S.bad, img, sino, sim, U, first, A.S, A.K, out_mode,   \
      factor_offset(A.half_factors))
  if (fh) TG_WALK(true); else TG_WALK(false);
#undef TG_WALK
}

}  // namespace tg
