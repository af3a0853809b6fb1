// Kernel launchers shared between the kernel translation units and the plan
// (host) code.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tg_device.cuh"
#include "tg_penalty.cuh"

namespace tg {

// Device view of the traced system matrix of one geometry.
struct MatrixDev {
  // forward matrix, ray-major, one 32-ray group (32 adjacent columns of one
  // angle) per warp; entry (group, step, lane) at roff[group] + step*32 + lane
  const int64_t* roff;
  const int* rcap;     // steps per group (max segment count of its rays)
  const int* rnseg;    // [P*C] segments per ray
  const int* ridx;     // pixel index per entry (explicit form)
  const uint32_t* rcode;  // delta form: 8 x 4-bit steps per word per lane
  const int64_t* rcoff;   // delta form: word offset per group
  const int* rstart;      // delta form: [P*C] first pixel of each ray
  const void* rlen;    // length per entry (float or 16-bit code)
  const float* ra2;    // [P*C] sum of squared lengths (SIRT's a2)
  // backward matrix, angle-major over 32-pixel tiles (pixel_tile: 16x2, 8x4
  // or 4x8 pixels): for pixel (x, y) in tile t at lane l, the pair of angle a
  // at dense_pair(ntiles, a, t, l) holds the lengths of rays (a, window_c0)
  // and (a, window_c0 + 1) through the pixel
  const void* dlen;
  const float4* wcoef; // [P4] window coefficients {-sin, cos, D, 0}
  // tensor-core backprojection: per angle quad and 4x4 pixel tile (tiles4 per
  // row and column) 16 words, of pixels 0, 8, 1, 9, ..., 7, 15 of the tile;
  // byte a & 3 of a word is the pixel's place_byte at angle a
  const uint32_t* place;
  int tiles4;
  // segments outside their pixel's two-column window (rare: the reference's
  // tracer puts a stray segment far from its ray at some near-vertical
  // angles): per pixel tile t, entries exc[exc_first[t] .. exc_first[t+1]) =
  // {lane, angle, column, length bits}; exc_first == nullptr when none
  const int* exc_first;
  const int4* exc;
  int tiles_x, ntiles;
  int tw_shift;        // backward tiles are 2^tw_shift pixels wide
  int P4;              // angles rounded up to a multiple of 4 (padding empty)
  const float* W;      // [g*g] total length through each pixel
  const float* Wh;     // [g*g] the same over half-rounded lengths (half_gathers)
  int len_kind;        // LenKind of the forward matrices
  // LenKind of the backward matrix: IEEE halves with half gathers (the
  // backprojection's mixed-precision FMAs take them as stored), else len_kind
  int dlen_kind;
  float scale, inv_scale;
};

// Tile-staged forward matrix (tg_tiles.cu): per ts x ts tile, groups of 32
// runs (consecutive segments of one ray inside the tile), lane = run. The
// tile side ts is a plan choice (32 to 96 in steps of 16; a step inside a
// tile is one signed byte dx + dy * (ts + 1), so ts + 1 <= 127).
constexpr int kTileSide = 64;

// Division by the tile side without an integer divide (the construction
// kernels take it for every segment): q = umulhi(v, m), m = ceil(2^32 / ts),
// exact for 0 <= v < 2^32 / ts, because v * (m * ts - 2^32) < 2^32 keeps
// the error of v * m / 2^32 below 1 / ts, the smallest distance from v / ts
// up to the next integer.
struct TileDiv {
  int ts;
  uint32_t m;
};
inline TileDiv make_tile_div(int ts) {
  return TileDiv{ts, 0xFFFFFFFFu / (uint32_t)(ts > 0 ? ts : 1) + 1u};
}
__device__ __forceinline__ int tdiv(int v, TileDiv d) {
  return (int)__umulhi((uint32_t)v, d.m);
}
__device__ __forceinline__ int tile_of_pixel(int ix, int iy, int tiles_x, TileDiv d) {
  return tdiv(iy, d) * tiles_x + tdiv(ix, d);
}

// A 4-bit step code holds (dx, dy) in {0,1} x {-1,0,1}. The reference's
// tracer can emit a segment far from the previous one (float rounding with
// the source a million units away, at near-vertical angles on the edge
// columns): such a step starts a new run, as a tile change does.
__device__ __forceinline__ bool unit_step(int ix, int iy, int px, int py) {
  const int dx = ix - px, dy = iy - py;
  return dx >= 0 && dx <= 1 && dy >= -1 && dy <= 1;
}
// Each run's partial sums (K floats) go to a slot fixed at construction:
// rays are taken in groups of 32 (ray r in group r / 32 at lane r % 32), and
// run k of ray r (k-th in the order its path crosses the tiles) has slot
// pbase[r / 32] + k * 32 + r % 32, so the finish kernel's warp reads one
// contiguous row of 32 slots per run ordinal while each lane adds its ray's
// runs in path order. No atomics: the forward projection is bit-reproducible.
struct TileMatrixDev {
  int tiles_x, ntiles;
  int ts;                   // tile side (pixels); shared-memory row stride ts + 1
  int bw;                   // warps per tile block (8, 16 or 32)
  const int* group_first;   // [ntiles + 1] first group of each tile
  const int* gpart;         // [groups * 32] partial-sum slot of each lane's
                            // run, -1 if the lane is empty
  const int* rnrun;         // [P*C] runs of each ray
  const int* pbase;         // [ceil(P*C / 32)] first slot of each ray group
  const uint16_t* glp;      // [groups * 32] first pixel, tile-local (y*ts + x)
  const uint16_t* glen;     // [groups * 32] run length (segments)
  const int* gsteps;        // [groups] longest run of the group
  const int64_t* gseg_off;  // [groups] entry offset of the group's lengths
  const int64_t* gcode_off; // [groups] word offset of the step codes
  const void* tlen;         // lengths, entry (group, step/8, lane, step%8)
  const uint32_t* tcode;    // 8 x 4-bit step codes per word per lane
};

// Strip-ordered forward matrix (tg_strips.cu). The slope of a ray is its shift
// in pixels per row (class 0: rows are pixel rows; class 1: pixel columns);
// positions of a group of angles lie within mid x d +- half x |d| at d rows
// from a chunk's middle, and a ray's pixels in a row within +- ext.
constexpr int kStripCols = 28;  // pixels staged per row by a block
struct StripSlopes {
  float mid, half, ext;
};
struct StripExc {
  int ray, idx, code, pad;
};
struct StripDev {
  int P, R, nchunks;       // rows per chunk
  uint32_t rmul;           // m / R = umulhi(m, rmul), as TileDiv's
  int strip0, nstrips;     // first strip's index; strips (a multiple of 4)
  int nblk16;              // blocks of 16 angles of one class
  int64_t nbundles;        // nchunks x nblk16 x nstrips x 4 quads
  const int* cls;          // [P]
  const int* place;        // [P] block x 16 + quad x 4 + angle of the quad
  const int64_t* alpha;    // [nchunks][P] position of column 0 at the chunk's
                           // middle row, in 2^-20 pixels
  const int64_t* sigma;    // [P] and its step per column (at least a pixel)
  const int* cls16;        // [nblk16]
  const StripSlopes* blk16;  // [nblk16]
  const StripSlopes* quad;   // [nblk16 * 4]
  const uint2* codes;      // [bundle][R / 4][16 rays][4 rows] even and odd
                           // pixels' pairs of 16-bit codes
  const uint32_t* meta;    // [bundle][R / 4][8][2]
  const int* exc_first;    // [P*C + 1] exceptions per ray, or nullptr
  const StripExc* exc;
  const uint8_t* grazed;   // [C*C] 1: a ray's zero-length segment lies in the pixel
  int* bad;                // [64] slices of the launch: a crossed pixel's half is not
                           // finite; [1] blocks that are done with these marks
};

// Which per-ray value the forward kernel stores.
enum FwdOut { FWD_SIRT = 0, FWD_RATIO = 1, FWD_SIM = 2 };
// What the backward kernel does with its per-pixel sums.
enum BackEpi { EPI_UPDATE = 0, EPI_REPLICA = 1 };

// Per-ray factors as the tensor-core backprojection (tg_backward_mma.cuh)
// reads them: units of U = 8, 16 or 32 slices, each [P4][RP][U] floats or
// halves with kRayPad zero columns before column 0 of an angle and twice as
// many after the last (windows may start and end outside the detector).
// Per slice, reset by the slice's forward launch and raised by its finish: bad
// != 0 where a factor of a ray with segments is not finite; on split plans the
// bits of the largest |factor|, and (counted by the split, in a sample) the
// factors that are not zero and those of them below about 2^-15 of the largest.
constexpr int kRayPad = 8;
struct __align__(16) FactorStat {
  unsigned most;
  int bad;
  unsigned nonzero, small;
};
// Float factors of plans with f16 lengths are also kept as two halves each,
// [P4][RP][2][U] (high parts, then low), scaled per slice by
// split_scale(stat[slice].most): every factor from 2^-15 of the largest on keeps
// FP32's 24 bits, smaller ones what is above 2^-39 of the largest. A slice most
// of whose factors are smaller (one hot ray) is summed ray by ray instead
// (redo_slices).
struct FactorDev {
  void* base;
  __half* split;
  int64_t unit_elems;  // P4 * RP * U
  int U, RP;
  int ring;            // units held; unit u is at u % ring
  FactorStat* stat;    // [slices, rounded up to whole batches]
  int blocks_x;        // 16 x 8 pixel blocks per row
};
// at least the 21 columns that a block stages
inline int factor_row(int C) { return C + 3 * kRayPad; }
inline int64_t mma_regions(int C) { return (int64_t)((C + 15) / 16) * ((C + 7) / 8); }

// The power of two that takes a largest |factor| (its float bits) to [2^13,
// 2^14): 1 for zero; kept finite, with a finite inverse, at the ends.
__host__ __device__ __forceinline__ float split_scale(unsigned bits) {
  const int e = (int)(bits >> 23);  // biased exponent
  if (e == 0) return 1.f;
  const int b = 127 + 13 - (e - 127);  // biased exponent of the scale
  const unsigned u = (unsigned)(b < 1 ? 1 : b > 253 ? 253 : b) << 23;
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}

// Element of column c, angle a, slice su of the unit at unit_base.
__device__ __forceinline__ int64_t factor_at(int64_t unit_base, int RP, int U, int a, int c,
                                             int su) {
  return unit_base + ((int64_t)a * RP + c + kRayPad) * U + su;
}

struct IterArgs {
  DevGeom G;
  MatrixDev M;
  FactorDev F;        // tensor-core backprojection (U = 0: the scalar kernels)
  int K;              // slices per pass
  int S;              // sinogram slices
  int alg;            // 0..3
  int exact;          // TG_MODE_EXACT
  int delta_index;
  // reconstruction slots: slot(true slice t) = t + vshift; layout
  // [nslots/K][g*g][K]
  int vshift;
  int fshift;         // forward source slot of sinogram slice s = s + fshift
  int nslots;
  int slice_id, num_total_slices;  // APMLR top/bottom
  PenaltyWeights pw;
  // 16-bit gather operands (fast mode, set per launch sequence):
  // half_tile - the tile-staged forward keeps its shared-memory tile as
  //             halves; half_factors - storage of the per-ray ratio
  //             factors (FACT_*)
  int half_tile;
  int half_factors;
  // compensated (Kahan) summation of the ray and pixel sums (fast mode,
  // tile-staged forward, L1 backprojection)
  int comp;
  // one slice per pass: room for a launch's planes with rows and columns
  // exchanged, or null
  float* turned;
};

// Work items of the launches that serve many plans at once (tg_batch): one
// item is one plan's slice batch, `first` its first block in the launch
// (items ascending by it).
struct FwdItem {
  TileMatrixDev T;
  const float* recon;   // the batch's reconstruction slots
  float* part;          // the plan's partial-sum slots
  FactorStat* stat;     // of the batch's slices (nullptr: none), reset here
  int g;
  float inv_scale;
  int64_t first;
};
// Storage of the per-ray ratio factors between the forward finish and the
// backprojection. FACT_HALF_M1: halves of (factor - 1), exact to a half's
// precision relative to the factor's distance from 1, so the steady state
// (factors near 1) loses least; the backprojection adds the pixel's total
// length back. FACT_HALF: halves of the factor itself, a half's relative
// precision whatever the factor, for the first iteration after a reset,
// where factors lie anywhere between 0 and their largest value.
enum { FACT_F32 = 0, FACT_HALF_M1 = 1, FACT_HALF = 2 };

__host__ __device__ inline float factor_offset(int half_factors) {
  return half_factors == FACT_HALF_M1 ? 1.f : 0.f;
}

struct FinItem {
  const int* rnrun;
  const int* pbase;
  const float* ra2;
  const float* part;
  const float* sino;    // the batch's sinogram rows
  float* out;           // per-ray factors [rays][K], or F when F.U != 0
  FactorDev F;
  int batch, C;
  int P4, S;            // launch_split_factors_multi
  int64_t nrays;        // there: blocks per unit
  int64_t first;        // 256 rays a block
  int out_mode;
  int fh;               // factor storage (FACT_*)
};
struct BackItem {
  IterArgs A;
  int batch;
  int nunits;           // tensor-core backprojection: units of the plan
  const float* cur;
  float* next;
  const float* upd;
  int64_t first;
};

// The item a block belongs to.
template <class Item>
__device__ __forceinline__ int item_of(const Item* items, int n, int64_t block) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (items[mid].first <= block) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Address of (slot, pixel) in the batched reconstruction layout.
__device__ __forceinline__ int64_t slot_addr(int slot, int64_t p, int64_t g2,
                                             int K) {
  return ((int64_t)(slot / K) * g2 + p) * K + (slot % K);
}

// APMLR's axial neighbours of slice s: the first slice of the dataset has
// none above, the last none below (apmlr.cc:937-967).
__device__ __forceinline__ void apmlr_axial(const IterArgs& A, int s, int* up,
                                            int* down) {
  const int beg = A.slice_id, end = A.slice_id + A.S - 1;
  const int final_index = A.slice_id + A.num_total_slices - 1;
  const bool top = (beg == 0 && s == 0);
  const bool bottom =
      !top && (final_index == end && final_index != 0 && s == A.S - 1);
  *up = !bottom;
  *down = !top;
}

// tg_trace.cu
// ray_nruns (optional): runs per ray of the tile-ordered forward matrix
// (a new run at each tile change and non-unit step), counted in the same pass
void launch_trace_count(const DevGeom& G, int* nseg, int* rcap,
                        unsigned* maxlen_bits, int tiles_x, int ts, int* ray_nruns,
                        cudaStream_t st);
void launch_trace_fill(const DevGeom& G, const MatrixDev& M, int* ridx,
                       uint32_t* rcode, int* rstart, void* rlen, float* ra2,
                       double* ra2d, void* dlen, unsigned long long* overflow,
                       int4* exc, int* exc_tile, int exc_cap, cudaStream_t st);

// Adds the window exceptions of the calling lane's pixel: f(l, angle,
// column) for each, after the regular angle loop.
template <typename F>
__device__ __forceinline__ void for_each_exception(const MatrixDev& M, int tile,
                                                   int lane, F&& f) {
  if (M.exc_first == nullptr) return;
  const int e1 = M.exc_first[tile + 1];
  for (int e = M.exc_first[tile]; e < e1; ++e) {
    const int4 x = M.exc[e];
    if (x.x == lane) f(__int_as_float(x.w), x.y, x.z);
  }
}
// the place words of MatrixDev::place (P4 / 4 x tiles4^2 x 16)
void launch_places(const DevGeom& G, const MatrixDev& M, uint32_t* place, cudaStream_t st);
// W (and, when Wh is given, the total of the half-rounded lengths) per pixel
void launch_weights(const DevGeom& G, const MatrixDev& M, int exact, float* W,
                    float* Wh, cudaStream_t st);
void launch_trace_export(const DevGeom& G, const int64_t* offsets, int* idx,
                         float* len, float* len2, cudaStream_t st);

// Grid of `blocks` blocks for each of nb slice batches, those of one block
// next to one another: the batch is blockIdx.x (uniform, without a division),
// the block grid_block().
inline dim3 batch_grid(int64_t blocks, int nb) {
  const unsigned y = (unsigned)(blocks < 65535 ? blocks : 65535);
  return dim3((unsigned)nb, y, (unsigned)((blocks + y - 1) / y));
}
__device__ __forceinline__ int grid_block() { return (int)(blockIdx.z * gridDim.y + blockIdx.y); }

// tg_forward.cu
// nb consecutive slice batches in one launch (sinogram rows and outputs P*C*K
// values apart)
void launch_forward(const IterArgs& A, int nb, const float* recon_batch,
                    const float* sino_batch, float* out, int out_mode,
                    cudaStream_t st);
// tg_backward.cu
// per-K instances of launch_backward (tg_backward*.cu)
#define TG_BACKWARD_DECL(KK)                                                      \
  void launch_backward_k##KK(const IterArgs& A, int first, int nb,                 \
                             const float* recon_cur, float* recon_next,            \
                             const float* upd, float* rep_num, int epi,            \
                             cudaStream_t st);                                     \
  void launch_backward_multi_k##KK(const BackItem* items, int n, int64_t blocks,   \
                                   int dlen_kind, int pen, int fh, int comp,        \
                                   cudaStream_t st);
TG_BACKWARD_DECL(1)
TG_BACKWARD_DECL(2)
TG_BACKWARD_DECL(4)
TG_BACKWARD_DECL(8)
#undef TG_BACKWARD_DECL
void launch_backward_k16(const IterArgs& A, int first, int nb, const float* recon_cur,
                         float* recon_next, const float* upd, float* rep_num, int epi,
                         cudaStream_t st);
// batches first .. first + nb - 1 in one launch, their factors (P*C*K values
// each) one behind the other at upd
void launch_backward(const IterArgs& A, int first, int nb, const float* recon_cur,
                     float* recon_next, const float* upd, float* rep_num,
                     int epi, cudaStream_t st);
// tg_backward_planes.cu: the same at one slice per pass, sums not compensated
void launch_backward_planes(const IterArgs& A, int first, int n, const float* cur, float* next,
                            const float* upd, float* rep_num, int epi, cudaStream_t st);
// Slices (at most four) a thread of a launch over n slices takes at one slice
// per pass, where one slice's launch has `warps` warps: four, two or one, the
// first with need4 (need2) warps left, evened out over the groups.
inline int planes_per_thread(int64_t warps, int n, int64_t need4, int64_t need2) {
  const int most = warps * ((n + 3) / 4) >= need4 ? 4 : warps * ((n + 1) / 2) >= need2 ? 2 : 1;
  const int groups = (n + most - 1) / most;
  return (n + groups - 1) / groups;
}
// tg_backward_mma*.cu: units first .. first + nunits - 1 of A.F (half_factors
// != FACT_F32: halves; else floats, split: A.F.split); the multi launch serves
// items of one (unit size, length kind, penalty, factor kind)
void launch_backward_mma(const IterArgs& A, int first, int nunits, const float* recon_cur,
                         float* recon_next, float* rep_num, int epi, cudaStream_t st);
void launch_backward_mma_multi(const BackItem* items, int n, int64_t blocks, int U,
                               int dlen_kind, int pen, int fh, cudaStream_t st);
#define TG_MMA_DECL(KIND)                                                                  \
  void launch_backward_mma_##KIND(const IterArgs& A, int first, int nunits,               \
                                  const float* recon_cur, float* recon_next,              \
                                  float* rep_num, int epi, cudaStream_t st);
#define TG_MMA_MULTI_DECL(KIND)                                                            \
  void launch_backward_mma_multi_##KIND(const BackItem* items, int n, int64_t blocks,     \
                                        int U, int pen, cudaStream_t st);
TG_MMA_DECL(half)
TG_MMA_DECL(split)
TG_MMA_DECL(u16)
TG_MMA_DECL(bf16)
TG_MMA_DECL(f32)
TG_MMA_MULTI_DECL(half)
TG_MMA_MULTI_DECL(split)
TG_MMA_MULTI_DECL(u16)
#undef TG_MMA_MULTI_DECL
#undef TG_MMA_DECL
// tg_backward_staged.cu (fast mode)
void launch_backward_staged(const IterArgs& A, int batch, const float* recon_cur,
                            float* recon_next, const float* upd, float* rep_num,
                            int epi, cudaStream_t st);
// tg_fp64.cu
void launch_forward64(const IterArgs& A, const double* ra2d, const double* recon,
                      const float* sino, double* out, int out_mode,
                      cudaStream_t st);
void launch_backward64(const IterArgs& A, int s, const double* cur,
                       double* next, const double* upd, const double* W,
                       cudaStream_t st);
void launch_weights64(const DevGeom& G, const MatrixDev& M, double* W,
                      cudaStream_t st);
void launch_convert(const float* in, double* out, int64_t n, cudaStream_t st);
void launch_narrow(const double* in, float* out, int64_t n, cudaStream_t st);
void launch_fill64(double* p, int64_t n, double v, cudaStream_t st);
// tg_tiles.cu
// Run sort key: tile | chunk-count class | ray | ordinal (RunKey).
struct RunKey {
  int ray_bits;  // bits of the ray id field
  __host__ __device__ int class_shift() const { return 8 + ray_bits; }
  __host__ __device__ int tile_shift() const { return 13 + ray_bits; }
};
// Run emission and the tile-stream fill read each ray's segments back from
// the ray-ordered forward matrix M when it is stored (M.rlen), else trace them.
void launch_runs_emit(const DevGeom& G, const MatrixDev& M, int tiles_x, int ts, RunKey rk,
                      const int64_t* ray_run_off, unsigned long long* key, int* val,
                      uint16_t* run_lp, uint16_t* run_len, cudaStream_t st);
// Construction prefix sums (tg_tiles.cu): tmp == nullptr asks for the
// temporary bytes; counts (int) to int64 offsets, or int64 to int64.
cudaError_t scan_counts(void* tmp, size_t* tmp_bytes, const int* in, int64_t* out, int n,
                        cudaStream_t st);
cudaError_t scan_i64(void* tmp, size_t* tmp_bytes, const int64_t* in, int64_t* out, int n,
                     cudaStream_t st);
// gslots[g] = 32 x the longest run count of ray group g (32 rays)
void launch_group_slots(const int* nruns, int64_t R, int64_t* gslots, cudaStream_t st);
// out[g] = tile-stream entries of run group g (256 per 8-step chunk)
void launch_group_entries(const int* gsteps, int groups, int64_t* out, cudaStream_t st);
// out[i] = in[i] >> shift (as int, or int64)
void launch_shift_narrow_i32(const int64_t* in, int* out, int64_t n, int shift,
                             cudaStream_t st);
void launch_shift_i64(const int64_t* in, int64_t* out, int64_t n, int shift,
                      cudaStream_t st);
// tile_first[t] = first sorted run of tile t, tile_first[ntiles] = nruns
void launch_tile_bounds(RunKey rk, const unsigned long long* skey, int64_t nruns,
                        int ntiles, int* tile_first, cudaStream_t st);
int sort_runs(unsigned long long* key_in, unsigned long long* key_out,
              int* val_in, int* val_out, int64_t n, int end_bit,
              cudaStream_t st);
void launch_runs_group(RunKey rk, const unsigned long long* skey, const int* sval,
                       int64_t nruns, const int* tile_first_run,
                       const int* group_first, const uint16_t* run_lp,
                       const uint16_t* run_len, const int64_t* ray_run_off,
                       const int* pbase, int* gpart, uint16_t* glp,
                       uint16_t* glen, int* gsteps, int* run_slot, cudaStream_t st);
void launch_runs_fill(const DevGeom& G, const MatrixDev& M, int tiles_x, int ts,
                      const int64_t* ray_run_off, const int* run_slot,
                      const int64_t* gseg_off, const int64_t* gcode_off,
                      void* tlen, uint32_t* tcode, cudaStream_t st);
// part: [runs][K] partial sums, written (not accumulated) by each launch;
// stat (optional): of the batch's slices, reset; width: A.K slices, or the 8 of
// 8 / A.K batches (half tile, not compensated)
void launch_forward_tiled(const IterArgs& A, const TileMatrixDev& T,
                          const float* recon_batch, float* part, FactorStat* stat,
                          int width, cudaStream_t st);
// ray sums from the partial sums (fixed order) -> per-ray values `out`
void launch_fwd_finish(const IterArgs& A, const TileMatrixDev& T, const float* part,
                       const float* sino, float* out, int out_mode, cudaStream_t st);
// the same, factors of the `width` slices from slice batch `batch` on into A.F
void launch_fwd_finish_units(const IterArgs& A, const TileMatrixDev& T, const float* part,
                             const float* sino, int batch, int out_mode, int width,
                             cudaStream_t st);
// units first .. first + nunits - 1 of A.F: floats -> scaled halves (A.F.split)
void launch_split_factors(const IterArgs& A, int first, int nunits, cudaStream_t st);
void launch_split_factors_multi(const FinItem* items, int n, int64_t blocks, cudaStream_t st);
// blocks per unit of a plan's item in the multi launch
int64_t split_blocks(const FactorDev& F, int P4);
// the same over many plans' slice batches in one launch each (device item
// arrays; blocks = the launch's total blocks; all items of one launch share
// K, the tile side and precision and the summation; 16-bit fixed-point
// lengths)
void launch_forward_tiled_multi(const FwdItem* items, int n, int64_t blocks, int K, int ts,
                                int bw, int half_tile, int comp, cudaStream_t st);
void launch_fwd_finish_multi(const FinItem* items, int n, int64_t blocks, int K, int comp,
                             cudaStream_t st);
// plans with 16-bit fixed-point lengths (backward matrix u16, or f16 with
// half gathers), compensated or of few slices per unit; pen: PML/APMLR;
// fh: half factors
void launch_backward_multi(const BackItem* items, int n, int64_t blocks, int K,
                           int dlen_kind, int pen, int fh, int comp, cudaStream_t st);
// blocks (of 256 threads) a plan's backprojection launch uses
int64_t backward_blocks(const IterArgs& A);
// tg_strips.cu
// the rays' pixel indices and length codes (16-bit storage) in the layout of
// the ray-ordered matrix
void launch_strips_trace(const DevGeom& G, const MatrixDev& M, int* ridx, uint16_t* rlen,
                         cudaStream_t st);
void launch_strips_fill(const DevGeom& G, const MatrixDev& M, const StripDev& S, uint2* codes,
                        uint32_t* meta, uint8_t* grazed, StripExc* exc, int exc_cap, int* nexc,
                        cudaStream_t st);
// U (32 or 64) slices from slice `first`: their halves into img ([pixel][U]),
// then every bundle's sums into part ([bundle][16][U]); reset: their
// factors' stat too
void launch_strips_forward(const IterArgs& A, const StripDev& S, int first, int U,
                           const float* recon, __half* img, float* part, int reset,
                           cudaStream_t st);
// their per-ray values: factors into A.F, or the sums ([S/K][P*C][K]) into sim
void launch_strips_finish(const IterArgs& A, const StripDev& S, int first, int U,
                          const __half* img, const float* part, const float* sino, float* sim,
                          int out_mode, cudaStream_t st);
// tg_iter.cu
void launch_fg(const IterArgs& A, const float* recon, const float* W, float* F,
               float* Gv, cudaStream_t st);
void launch_update(const IterArgs& A, float* recon, const float* W,
                   const float* F, const float* Gv, const float* rep_num,
                   cudaStream_t st);
void launch_sino_pack(const float* in, float* out, int P, int S, int C, int K,
                      int apply_abs, int clip, float clip_min, cudaStream_t st);
void launch_sino_unpack(const float* in, float* out, int P, int S, int C,
                        int K, cudaStream_t st);
void launch_recon_pack(const float* in, float* out, int nuser, int g2, int K,
                       int slot0, int nslots, cudaStream_t st);
void launch_recon_unpack(const float* in, float* out, int nuser, int g2, int K,
                         int slot0, cudaStream_t st);
void launch_fill(float* p, size_t n, float v, cudaStream_t st);
void launch_replica_interleave(const float* rep_num, const float* W,
                               float* out, int S, int g2, cudaStream_t st);

}  // namespace tg
