// The segments of one ray, read back from the stored ray-ordered matrix (or
// traced again), for the kernels that build the other forward matrices from it.
#pragma once
#include "tg_kernels.cuh"

namespace tg {

namespace {

// The segments of one ray, in order, as f(idx, ix, iy, length, 16-bit length
// code), idx = iy * g + ix:
// read back from the ray-ordered forward matrix when the plan keeps one
// (delta-coded or explicit indices; the stored code is the one encode16 gives
// the traced length, so both sources yield the same tile stream), traced
// again otherwise (forward traced on the fly, or a stray step the 4-bit code
// cannot hold). LEN: which length the caller takes - none (0 and 0 are
// passed; the matrix's lengths are not read), the 16-bit code (the plan's
// 16-bit storage) or the float length (f32 storage).
enum SegSource { kSrcTrace = 0, kSrcDelta = 1, kSrcIndex = 2 };
enum SegLen { kLenNone = 0, kLenCode = 1, kLenFloat = 2 };

template <int SRC, int LEN, class F>
__device__ __forceinline__ void ray_segments(const DevGeom& G, const MatrixDev& M,
                                             int64_t r, F&& f) {
  const int a = (int)(r / G.C), c = (int)(r - (int64_t)a * G.C);
  if constexpr (SRC == kSrcTrace) {
    trace_ray(G, a, c, [&](int idx, float l, float, int ix, int iy) {
      f(idx, ix, iy, l, LEN == kLenCode ? encode16(l, M.len_kind, M.scale) : (uint16_t)0);
    });
  } else {
    const int g = G.C;
    const int grp = a * G.gpa + (c >> 5), lane = c & 31;
    const int n = M.rnseg[r];
    const int64_t base = M.roff[grp] + lane;
    const int64_t cbase = SRC == kSrcDelta ? M.rcoff[grp] + lane : 0;
    const float inv_g = 1.0f / (float)g;
    int idx = (SRC == kSrcDelta && n > 0) ? M.rstart[r] : 0;
    int ix = 0, iy = 0;
    if (SRC == kSrcDelta && n > 0) cell_xy(idx, g, inv_g, ix, iy);
    if constexpr (SRC == kSrcDelta) {
      // chunks of 8 steps (one step-code word, 8 lengths), the next chunk's
      // loads issued before the current one is walked: the walk is a chain
      // of dependent steps, so a load issued at its step would stall it
      struct Chunk {
        uint32_t word;
        uint32_t len[LEN == kLenNone ? 1 : 8];
      };
      auto load = [&](int ch, Chunk& k) {
        const int s0 = ch * 8;
        k.word = __ldcs(M.rcode + cbase + (int64_t)ch * 32);
        if constexpr (LEN != kLenNone) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int64_t e = base + (int64_t)(s0 + j) * 32;
            k.len[j] = 0u;
            if (s0 + j < n) {
              if constexpr (LEN == kLenCode)
                k.len[j] = __ldcs(reinterpret_cast<const uint16_t*>(M.rlen) + e);
              else
                k.len[j] = __float_as_uint(__ldcs(reinterpret_cast<const float*>(M.rlen) + e));
            }
          }
        }
      };
      Chunk cur{}, nxt{};
      if (n > 0) load(0, cur);
      for (int ch = 0; ch * 8 < n; ++ch) {
        if ((ch + 1) * 8 < n) load(ch + 1, nxt);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int st = ch * 8 + j;
          if (st >= n) break;
          if (st > 0) {
            const uint32_t code = (cur.word >> (4 * j)) & 15u;
            const int dx = (int)(code & 1u), dy = (int)(code >> 1) - 1;
            ix += dx;
            iy += dy;
            idx += dx + dy * g;
          }
          if constexpr (LEN == kLenCode)
            f(idx, ix, iy, 0.f, (uint16_t)cur.len[j]);
          else if constexpr (LEN == kLenFloat)
            f(idx, ix, iy, __uint_as_float(cur.len[j]), (uint16_t)0);
          else
            f(idx, ix, iy, 0.f, (uint16_t)0);
        }
        cur = nxt;
      }
    } else {
      for (int st = 0; st < n; ++st) {
        const int64_t e = base + (int64_t)st * 32;
        idx = __ldcs(M.ridx + e);
        cell_xy(idx, g, inv_g, ix, iy);
        if constexpr (LEN == kLenCode)
          f(idx, ix, iy, 0.f, __ldcs(reinterpret_cast<const uint16_t*>(M.rlen) + e));
        else if constexpr (LEN == kLenFloat)
          f(idx, ix, iy, __ldcs(reinterpret_cast<const float*>(M.rlen) + e), (uint16_t)0);
        else
          f(idx, ix, iy, 0.f, (uint16_t)0);
      }
    }
  }
}

inline int seg_source(const MatrixDev& M) {
  if (M.rlen == nullptr) return kSrcTrace;
  return M.rcode != nullptr ? kSrcDelta : kSrcIndex;
}

}  // namespace

}  // namespace tg
