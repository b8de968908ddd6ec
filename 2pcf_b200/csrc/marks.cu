// marks.cu -- xi from precomputed per-lens marks (calculate_tpcf_from_marks,
// src/main.f90:1017-1139): for each foreground map m and field i,
//   g_t[b] = sum_j xi_E[j][b] val_mj w_mj / sum_j K[j][b] w_mj,
//   g_x[b] = sum_j xi_B[j][b] val_mj w_mj / sum_j K[j][b] w_mj,
//   weights = sum_j mw_j w_mj,
// over the lenses j with mw_j w_mj > 0 (the reference packs the others away,
// :1089-1104), and the fields stacked by summing numerators and K
// (:1127-1135).  The marks were computed once with val = w = 1; each new map
// only re-weights them, so this is a streaming pass over the marks: 12 bytes
// per lens and bin plus 8 bytes per lens and map against 2 FP64 FLOP per lens,
// row and map, which puts 16 maps per pass on both the HBM and the FP64
// roofline.
//
// One block = a run of lenses of one field and up to kMapGroup maps
// (register-tiled FP64 sums, rows x maps), per-block partial sums in scratch,
// then a fixed-order reduction over blocks (deterministic).

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "philox.cuh"
#include "tpcf_b200.h"
#include "tpcf_ctx.h"
#include "tpcf_device.cuh"
#include "tpcf_internal.cuh"
#include "tpcf_kernels.h"

namespace tpcf {

constexpr int kMapGroup = 16;     // maps or resamples per pass over the marks

struct MarksField {
  long long n;
  int n_bin;
  int chunk0;               // first block of this field
  long long lens0;          // index of the field's first lens among all fields
  const float* mw;          // marks weight [n]
  const float* xiE;         // [n][n_bin]
  const float* xiB;
  const float* K;
  const float* val;         // maps: [n_map][n]
  const float* w;           // maps: [n_map][n]
};

// Asynchronous copies global -> shared (cp.async) of 4 or 16 bytes; with
// valid == false nothing is read and the destination is zero-filled.
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(valid ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Raw factor inputs of a tile in shared memory: one row of 64 lenses per map
// or resample, rows kRawStride floats apart (16-byte aligned rows; the
// conversion's warps read 16 maps x 2 lenses, at most two lanes per bank).
constexpr int kRawStride = 68;

// Copies `rows` runs of 64 consecutive 4-byte values, run k from src(k) (a
// device pointer to the run's first value), into dst rows kRawStride values
// apart, by all threads of the block: valid values are the first nt of each
// run of the first live_rows runs, the rest is zero-filled.  16-byte chunks
// when the tile is whole and every run starts on a 16-byte boundary (vec),
// else 4-byte copies.
template <class SrcOf>
__device__ __forceinline__ void stage_runs(void* dst, int rows, int live_rows, int nt, bool vec, SrcOf src, int tid,
                                           int nthr) {
  unsigned char* d = reinterpret_cast<unsigned char*>(dst);
  if (vec) {
    for (int e = tid; e < rows * 16; e += nthr) {
      const int k = e >> 4, c = e & 15;
      const bool v = k < live_rows;
      cp_async16(d + (size_t)(k * kRawStride + 4 * c) * 4,
                 v ? reinterpret_cast<const unsigned char*>(src(k)) + 16 * c
                   : reinterpret_cast<const unsigned char*>(src(0)), v);
    }
  } else {
    for (int e = tid; e < rows * 64; e += nthr) {
      const int k = e >> 6, jj = e & 63;
      const bool v = k < live_rows && jj < nt;
      cp_async4(d + (size_t)(k * kRawStride + jj) * 4,
                v ? reinterpret_cast<const unsigned char*>(src(k)) + 4 * jj
                  : reinterpret_cast<const unsigned char*>(src(0)), v);
    }
  }
}

// Four values p[0 .. 3] of which the first n exist (the others read as 0);
// vec: all four exist and p is 16-byte aligned.
template <class V4, class T>
__device__ __forceinline__ V4 load4(const T* p, int n, bool vec) {
  if (vec) return __ldg(reinterpret_cast<const V4*>(p));
  V4 v = {0, 0, 0, 0};
  if (n > 0) v.x = __ldg(p);
  if (n > 1) v.y = __ldg(p + 1);
  if (n > 2) v.z = __ldg(p + 2);
  if (n > 3) v.w = __ldg(p + 3);
  return v;
}
template <class V4>
__device__ __forceinline__ auto comp4(const V4& v, int s) {
  return s == 0 ? v.x : s == 1 ? v.y : s == 2 ? v.z : v.w;
}

// Lens factors: the numerator factor vw and the K factor wm of one lens and
// map or resample, both 0 for a lens that takes no part.  stage() starts the
// copies of a tile's raw inputs into shared memory (all threads) and factors()
// reads a landed value; load() reads four lenses' raw inputs of two maps (g,
// g + 8) into registers and factor() turns one of them into its factors.
struct MapFactors {  // foreground maps: vw = val w, wm = w
  static constexpr bool kSame = false;  // vw and wm differ: two factor arrays
  int map0;
  static constexpr size_t kRawBytes = sizeof(float) * (2 * kMapGroup + 1) * kRawStride;
  // moves to the p-th 16 of n maps: how many they are
  __device__ __forceinline__ int pass(int p, int n) {
    map0 += p * kMapGroup;
    return min(kMapGroup, n - p * kMapGroup);
  }
  static __device__ __forceinline__ void of(float v, float w, float mw, double& vw, double& wm) {
    wm = (double)w;
    vw = (double)v * wm;
    // calculate_tpcf_from_marks drops lenses with marks weight x weight <= 0
    if (!((double)mw * wm > 0.0)) vw = wm = 0.0;
  }
  // raw rows: val of the kMapGroup maps, w of the kMapGroup maps, marks weight
  __device__ __forceinline__ void stage(const MarksField& F, long long t0, int nt, int n_g, unsigned char* raw,
                                        int tid, int nthr) const {
    float* rv = reinterpret_cast<float*>(raw);
    const bool vec = nt == 64 && al16(F.val) && al16(F.w) && al16(F.mw) && (F.n & 3) == 0 && (t0 & 3) == 0;
    const size_t o = (size_t)map0 * (size_t)F.n + (size_t)t0;
    const float* val = F.val;
    const float* w = F.w;
    const long long n = F.n;
    stage_runs(rv, kMapGroup, n_g, nt, vec, [&](int k) { return val + o + (size_t)k * n; }, tid, nthr);
    stage_runs(rv + kMapGroup * kRawStride, kMapGroup, n_g, nt, vec, [&](int k) { return w + o + (size_t)k * n; },
               tid, nthr);
    const float* mw = F.mw + t0;
    stage_runs(rv + 2 * kMapGroup * kRawStride, 1, 1, nt, vec, [&](int) { return mw; }, tid, nthr);
  }
  __device__ __forceinline__ void factors(const unsigned char* raw, int g, int jj, double& vw, double& wm) const {
    const float* rv = reinterpret_cast<const float*>(raw);
    of(rv[g * kRawStride + jj], rv[(kMapGroup + g) * kRawStride + jj], rv[2 * kMapGroup * kRawStride + jj], vw, wm);
  }
  struct Raw {
    float4 v[2], w[2];
  };
  __device__ __forceinline__ bool vec_ok(const MarksField& F) const {
    return al16(F.val) && al16(F.w) && (F.n & 3) == 0;
  }
  // Lenses l0 .. l0 + n - 1, n <= 4; vec (the same for the whole warp): n = 4
  // and l0 a multiple of 4.  Maps past n_g read the last one: their sums are
  // dropped.
  __device__ __forceinline__ void load(const MarksField& F, long long l0, int n, bool vec, int n_g, int g,
                                       Raw& r) const {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const size_t o = (size_t)(map0 + min(g + 8 * k, n_g - 1)) * (size_t)F.n + (size_t)l0;
      r.v[k] = load4<float4>(F.val + o, n, vec);
      r.w[k] = load4<float4>(F.w + o, n, vec);
    }
  }
  __device__ __forceinline__ void factor(const Raw& r, int k, int s, float mw, double& vw, double& wm) const {
    of(comp4(r.v[k], s), comp4(r.w[k], s), mw, vw, wm);
  }
};
struct MultFactors {  // resamples: vw = wm = multiplicity of the lens's unit
  static constexpr bool kSame = true;  // one factor array serves every row
  const int* mult;    // [G][n_units]
  const int* unit;    // unit of each lens (all fields concatenated), or nullptr: the lens itself
  long long n_units;
  static constexpr size_t kRawBytes = sizeof(int) * kMapGroup * kRawStride;
  __device__ __forceinline__ int pass(int p, int n) {
    mult += (size_t)p * kMapGroup * (size_t)n_units;
    return min(kMapGroup, n - p * kMapGroup);
  }
  // the bootstraps take every drawn lens (src/tpcf.f90:601, :917, :1248)
  static __device__ __forceinline__ double of(int m) { return m > 0 ? (double)m : 0.0; }
  __device__ __forceinline__ void stage(const MarksField& F, long long t0, int nt, int n_g, unsigned char* raw,
                                        int tid, int nthr) const {
    int* rm = reinterpret_cast<int*>(raw);
    const long long gl0 = F.lens0 + t0;
    if (!unit) {  // each lens its own unit: runs of consecutive multiplicities
      const bool vec = nt == 64 && al16(mult) && (n_units & 3) == 0 && (gl0 & 3) == 0;
      const int* m = mult + gl0;
      const long long nu = n_units;
      stage_runs(rm, kMapGroup, n_g, nt, vec, [&](int k) { return m + (size_t)k * nu; }, tid, nthr);
      return;
    }
    for (int e = tid; e < kMapGroup * 64; e += nthr) {  // gathered through the unit labels
      const int g = e >> 6, jj = e & 63;
      const bool v = g < n_g && jj < nt;
      const size_t o = v ? (size_t)g * (size_t)n_units + (size_t)__ldg(unit + gl0 + jj) : 0;
      cp_async4(rm + g * kRawStride + jj, mult + o, v);
    }
  }
  __device__ __forceinline__ void factors(const unsigned char* raw, int g, int jj, double& vw, double& wm) const {
    vw = wm = of(reinterpret_cast<const int*>(raw)[g * kRawStride + jj]);
  }
  struct Raw {
    int4 m[2];
  };
  __device__ __forceinline__ bool vec_ok(const MarksField& F) const {
    return !unit && al16(mult) && (n_units & 3) == 0 && (F.lens0 & 3) == 0;
  }
  __device__ __forceinline__ void load(const MarksField& F, long long l0, int n, bool vec, int n_g, int g,
                                       Raw& r) const {
    const long long gl = F.lens0 + l0;
    const int4 u = unit ? load4<int4>(unit + gl, n, false) : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int* m = mult + (size_t)min(g + 8 * k, n_g - 1) * (size_t)n_units;
      if (unit)
        r.m[k] = make_int4(n > 0 ? __ldg(m + u.x) : 0, n > 1 ? __ldg(m + u.y) : 0, n > 2 ? __ldg(m + u.z) : 0,
                           n > 3 ? __ldg(m + u.w) : 0);
      else
        r.m[k] = load4<int4>(m + gl, n, vec);
    }
  }
  __device__ __forceinline__ void factor(const Raw& r, int k, int s, float, double& vw, double& wm) const {
    vw = wm = of(comp4(r.m[k], s));
  }
};

// partial[(blk * n_g + g) * R + r], R = 3 n_bin + 1 (E, B, K rows, weight):
// a split-K product of the marks [lens][R] with the lens factors [lens][n_g]
// over the block's lenses.  This FP64 FMA form serves wide binnings
// (n_bin > 32, marks read from HBM by the summing loop); narrower ones run on
// the FP64 tensor cores (k_marks_dmma below).
//
// The rows come in quads: four consecutive bins of one quantity (xi_E, xi_B
// or K; the last quad of a quantity padded with zero bins) and one quad for
// the marks weight (the weight and three zeros).  A lens group is tg
// threads, lane 2 quad + half owning rows quad x maps 8 half .. 8 half + 7 as
// 32 FP64 register sums; per lens it loads its quad's marks (four values)
// and its 8 factors (four 16-byte shared-memory loads) and adds the 32
// products (FP64 FMA).
// The block takes `chunk` lenses of one field in tiles of kTileL; while it
// sums one tile the factors' raw inputs of the next are being copied
// (cp.async) into shared memory, and after a barrier they become the FP64
// factors (zero for lenses left out).  Group k takes the tile's lenses k,
// k + NG, ...; the groups are summed in fixed order at the end
// (deterministic, no atomics).
//
// The factors of one lens are stored as [vw of the 16 maps | 2 pad | wm of
// the 16 maps | 2 pad] (kLensStride doubles): the four 16-byte loads of a
// warp touch at most four distinct chunks (vw or wm, half 0 or 1), on
// disjoint banks.
constexpr int kTileL = 64;
constexpr int kLensStride = 2 * (kMapGroup + 2);
constexpr int kWmOffset = kMapGroup + 2;
// Threads per block at most (whole lens groups); two blocks per SM leave 128
// registers per thread for the 32 FP64 sums and the loads in flight.
constexpr int kMarksThreads = 256;
// Blocks the lenses of a call are spread over: two per SM of a 148-SM part,
// one wave.  A constant, so the summation order (and the result) depends
// only on the input.
constexpr int kMarksBlocks = 2 * 148;
static_assert(kTileL == 64, "the raw staging areas hold 64 lenses");
__host__ __device__ inline int marks_quad_bins(int n_bin) { return (n_bin + 3) / 4 * 4; }
// Factors of one tile: raw inputs -> FP64 vw, wm in fac_s, all threads.
// Consecutive lanes take consecutive maps of one lens, so each warp's stores
// fill whole 128-byte rows.
template <class Fac>
__device__ __forceinline__ void convert_factors(const Fac& fac, const unsigned char* raw, double* fac_s, int tid,
                                                int nthr) {
  static_assert(kMapGroup == 16, "maps are the low 4 bits of the element index");
  for (int e = tid; e < kTileL * kMapGroup; e += nthr) {
    const int g = e & 15, jj = e >> 4;
    double vw, wm;
    fac.factors(raw, g, jj, vw, wm);
    fac_s[jj * kLensStride + g] = vw;
    if (!Fac::kSame) fac_s[jj * kLensStride + kWmOffset + g] = wm;
  }
}

template <class Fac>
__global__ void __launch_bounds__(kMarksThreads, 2) k_marks_partials(const MarksField* __restrict__ fields, int n_field,
                                                            Fac fac, int n_maps, int n_bin, int tg,
                                                            long long chunk, double* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr int TF = kTileL * kLensStride;
  const int R = 3 * n_bin + 1;
  const int n_g = fac.pass(blockIdx.y, n_maps);
  partial += (size_t)blockIdx.y * gridDim.x * kMapGroup * R;
  const int nbp = marks_quad_bins(n_bin), nbq = nbp / 4;
  const int ng = blockDim.x / tg;
  double* fac_s = reinterpret_cast<double*>(sm);  // [kTileL][kLensStride] factors of every row
  unsigned char* raw = sm + TF * sizeof(double);
  const int blk = blockIdx.x;
  int fi = 0;
  while (fi + 1 < n_field && fields[fi + 1].chunk0 <= blk) ++fi;
  const MarksField& F = fields[fi];  // read where used: its pointers need no registers across the loop
  const long long j0 = (long long)(blk - F.chunk0) * chunk;
  const long long j1 = min(F.n, j0 + chunk);
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int grp = tid / tg, l = tid % tg;
  const int quad = l >> 1, half = l & 1;
  const bool live = quad <= 3 * nbq;
  const int k = quad / nbq, c = quad - k * nbq;  // k = 3: the marks weight quad
  const double* fsel = ((k < 2 || Fac::kSame) ? fac_s : fac_s + kWmOffset) + 8 * half;
  // this lane's quad in HBM: bins 4 c .. of quantity k of lens j, or the marks weight
  const float* qrow = k == 0 ? F.xiE : k == 1 ? F.xiB : k == 2 ? F.K : F.mw;

  auto stage_tile = [&](long long t0) { fac.stage(F, t0, (int)min((long long)kTileL, j1 - t0), n_g, raw, tid, nthr); };
  auto convert_tile = [&]() { convert_factors(fac, raw, fac_s, tid, nthr); };

  double acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int g = 0; g < 8; ++g) acc[i][g] = 0.0;
  if (j0 < j1) stage_tile(j0);
  cp_async_wait_all();
  __syncthreads();
  if (j0 < j1) convert_tile();
  __syncthreads();
  for (long long t0 = j0; t0 < j1; t0 += kTileL) {
    const int nt = (int)min((long long)kTileL, j1 - t0);
    const bool more = t0 + kTileL < j1;
    // the raw area was read before the last barrier
    if (more) stage_tile(t0 + kTileL);
    if (live) {
#pragma unroll 1
      for (int jj = grp; jj < nt; jj += ng) {
        double m[4];
        const long long j = t0 + jj;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool v = k < 3 ? 4 * c + i < n_bin : i == 0;
          m[i] = v ? (double)__ldg(k < 3 ? qrow + j * n_bin + 4 * c + i : qrow + j) : 0.0;
        }
        const double2* f2 = reinterpret_cast<const double2*>(fsel + jj * kLensStride);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const double2 f = f2[h];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            acc[i][2 * h] = fma(m[i], f.x, acc[i][2 * h]);
            acc[i][2 * h + 1] = fma(m[i], f.y, acc[i][2 * h + 1]);
          }
        }
      }
    }
    cp_async_wait_all();
    __syncthreads();  // the next tile's copies landed; this tile's factors are no longer read
    if (more) {
      convert_tile();
      __syncthreads();
    }
  }
  // groups 1.. add their sums into group 0's, in group order
  double* red = reinterpret_cast<double*>(sm);  // [tg][32]
  for (int kk = 1; kk < ng; ++kk) {
    __syncthreads();
    if (grp == kk) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int g = 0; g < 8; ++g) red[l * 32 + i * 8 + g] = acc[i][g];
    }
    __syncthreads();
    if (grp == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int g = 0; g < 8; ++g) acc[i][g] += red[l * 32 + i * 8 + g];
    }
  }
  if (grp == 0 && live) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int b = 4 * c + i;
      if (k < 3 ? b >= n_bin : i > 0) continue;
      const int r = k < 3 ? k * n_bin + b : 3 * n_bin;
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        const int map = 8 * half + g;
        if (map < n_g) partial[((size_t)blk * n_g + map) * R + r] = acc[i][g];
      }
    }
  }
}

// FP64 tensor-core form for n_bin <= 32 (tcgen05 has no FP64 kind; the FP64
// tensor instruction of sm_100 is mma.sync .f64, here m16n8k16: D[16][8] +=
// A[16][16] B[16][8], maps by rows by lenses, 2048 FMA per warp instruction
// against 32 for a warp FFMA64).
//
// The rows of the marks (B's N dimension) are grouped so that no tile of 8 mixes
// the two factor kinds: the xi_E, xi_B rows (vw factors) fill the first
// MV = ceil(2 n_bin / 8) tiles, the K rows and the marks weight row (wm
// factors) the next MK = ceil((n_bin + 1) / 8); padding rows are zeros.  The 16
// maps are A's rows, so a tile needs one kind of factors.
//
// Bound by the FP64 tensor pipe (57 us for 10^6 lenses, 61 rows and 16 maps,
// as long as the 370 MB of marks and maps take from HBM), so everything else
// has to stay below it.  Each warp therefore takes lenses of its own (16 at a
// time, k, k + kDmmaWarps, ... of the block's) and all row tiles of them: a
// factor is needed by one lane only, which loads its inputs from HBM into
// registers one group ahead and converts them there; the marks come by bulk
// copies into the warp's own ring of buffers; no barrier until the end, where
// the block's warps are summed in order.  With one row tile per warp instead,
// every warp read all factors from shared memory, written there in a pass
// between block barriers: 6 wavefronts of shared memory for 2 tensor
// instructions, where this form has 1.4, and the m8n8k4 form of the instruction
// instead of m16n8k16: 130 us for that case against 91 now (pipe 67 % busy; 16
// warps a SM instead of 12 need spills: 114 us; a third buffer: 93).
//
// Within a group of 16 the K index 4 s + tq (tq: the lane's index in the
// fragment) is lens 4 tq + s: any bijection serves, and with this one a lane's
// four lenses are consecutive, so its inputs are one 16-byte load a map.
//
// Staged marks: quantity q of lens jj, bin b at q QS + jj n_bin + b
// (QS = 16 n_bin).  Groups that are short or not 16-byte aligned in HBM are
// copied value by value (cp.async, zeros past the end).  Every wait is
// bounded: a copy that does not land sets kErrTimeout in *err and the warp
// stops.
constexpr int kDmmaLens = 16;   // lenses per group of a warp
constexpr int kDmmaWarps = 4;
constexpr int kDmmaRing = 2;    // buffers per warp
static_assert(kTileL % kDmmaLens == 0, "chunks hold whole groups");
__host__ __device__ inline int marks_dmma_buffer(int n_bin) { return 3 * kDmmaLens * n_bin; }
__host__ __device__ inline int marks_vw_tiles(int n_bin) { return (2 * n_bin + 7) / 8; }
__host__ __device__ inline int marks_m_tiles(int n_bin) { return marks_vw_tiles(n_bin) + (n_bin + 1 + 7) / 8; }
constexpr int kDmmaMaxBins = 32;
// Blocks a SM: 3 up to 8 row tiles (168 registers, 64 of them sums), 2 beyond.
__host__ __device__ constexpr int marks_dmma_per_sm(int tiles) { return tiles <= 8 ? 3 : 2; }
// Output row of row i of the tiles: 0 .. R - 1, or -1 (padding).
__device__ __forceinline__ int marks_row(int i, int n_bin) {
  const int v = 8 * marks_vw_tiles(n_bin);
  if (i < v) return i < 2 * n_bin ? i : -1;
  return i - v <= n_bin ? 2 * n_bin + i - v : -1;
}

// d[16][8] += A[16][16] B[16][8]; a[2 s + h]: row gq + 8 h, K 4 s + tq; b[s]: K
// 4 s + tq, column gq; d[2 h + c]: row gq + 8 h, column 2 tq + c.
__device__ __forceinline__ void dmma_16816(double (&d)[4], const double (&a)[8], const double (&b)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7, %8, %9, %10, %11}, "
      "{%12, %13, %14, %15}, {%0, %1, %2, %3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
        "d"(b[2]), "d"(b[3]));
}

template <class Fac, int MV, int MK>
__global__ void __launch_bounds__(32 * kDmmaWarps, marks_dmma_per_sm(MV + MK))
k_marks_dmma(const MarksField* __restrict__ fields, int n_field, Fac fac, int n_maps, int n_bin, long long chunk,
             double* __restrict__ partial, unsigned* __restrict__ err, int skip_tile, unsigned wait_limit) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ __align__(8) uint64_t full_s[kDmmaWarps][kDmmaRing];
  const int nb = n_bin, R = 3 * nb + 1;
  const int n_g = fac.pass(blockIdx.y, n_maps);
  partial += (size_t)blockIdx.y * gridDim.x * kMapGroup * R;
  const int QS = kDmmaLens * nb, BS = marks_dmma_buffer(nb);
  constexpr int NM = MV + MK;  // tiles of the vw and of the wm rows
  const int blk = blockIdx.x;
  int fi = 0;
  while (fi + 1 < n_field && fields[fi + 1].chunk0 <= blk) ++fi;
  const MarksField F = fields[fi];
  const long long j0 = (long long)(blk - F.chunk0) * chunk;
  const int n_len = (int)min(F.n - j0, chunk);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  float* mk = reinterpret_cast<float*>(sm) + warp * kDmmaRing * BS;
  uint64_t* full = full_s[warp];
  // this lane's row of the marks (row gq of each tile): staged offset of its
  // value for lens 4 tq.  Padding is in the last vw tile, the marks weight row
  // and padding in the last wm tile.
  int off[NM];
#pragma unroll
  for (int i = 0; i < NM; ++i) {
    const int r = marks_row(8 * i + gq, nb), q = r < 0 ? 0 : r / nb;
    off[i] = 4 * tq * nb + (r < 0 || q > 2 ? 0 : q * QS + (r - q * nb));
  }
  const bool vpad = marks_row(8 * (MV - 1) + gq, nb) < 0, wpad = marks_row(8 * (NM - 1) + gq, nb) < 0;
  const bool wrow = marks_row(8 * (NM - 1) + gq, nb) == 3 * nb;
  if (lane == 0) {
#pragma unroll
    for (int b = 0; b < kDmmaRing; ++b) mbar_init(&full[b], 1);
    mbar_fence_init();
  }
  __syncwarp();
  const bool mbulk = al16(F.xiE) && al16(F.xiB) && al16(F.K);
  const bool lvec = al16(F.mw) && fac.vec_ok(F);
  // fault injection for tests (tpcf_debug_inject): the bulk copies of each
  // block's lenses 64 skip_tile .. + 63 are never issued, so the wait on them
  // runs out after wait_limit polls (both off in every product call)
  const uint32_t polls = wait_limit ? wait_limit : kWaitPolls;
  // groups of this warp: group k starts at lens j0 + first(k)
  const int n_group = (n_len + kDmmaLens - 1) / kDmmaLens;
  const int mine = n_group > warp ? (n_group - warp + kDmmaWarps - 1) / kDmmaWarps : 0;
  auto first = [&](int k) { return (warp + k * kDmmaWarps) * kDmmaLens; };
  auto bulk = [&](int k) { return mbulk && first(k) + kDmmaLens <= n_len; };
  // starts the copies of group k into its buffer (bulk copies complete on
  // full[buffer], others in the warp's k-th cp.async group)
  auto stage = [&](int k) {
    const int f = first(k), b = k % kDmmaRing;
    float* dst = mk + b * BS;
    const size_t o = (size_t)(j0 + f) * nb;
    if (bulk(k)) {
      if (lane == 0 && f / kTileL != skip_tile) {
        mbar_arrive_tx(&full[b], 4u * BS);
        bulk_g2s(dst, F.xiE + o, 4u * QS, &full[b]);
        bulk_g2s(dst + QS, F.xiB + o, 4u * QS, &full[b]);
        bulk_g2s(dst + 2 * QS, F.K + o, 4u * QS, &full[b]);
      }
    } else {
      const int nq = min(kDmmaLens, n_len - f) * nb;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const float* src = (q == 0 ? F.xiE : q == 1 ? F.xiB : F.K) + o;
        for (int e = lane; e < QS; e += 32) cp_async4(dst + q * QS + e, e < nq ? src + e : src, e < nq);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // waits for group k, with at most kDmmaRing - 1 later groups begun
  auto land = [&](int k) -> bool {
    if (bulk(k)) {
      const bool ok = mbar_wait_bounded(&full[k % kDmmaRing], (uint32_t)(k / kDmmaRing) & 1u, polls);
      return __all_sync(0xffffffffu, ok);
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(kDmmaRing - 1) : "memory");
    __syncwarp();
    return true;
  };
  // the lane's raw factor inputs and marks weights of group k
  auto inputs = [&](int k, typename Fac::Raw& r, float4& mw) {
    const int f = first(k) + 4 * tq, n = min(4, max(0, n_len - f));
    const bool vec = lvec && first(k) + kDmmaLens <= n_len;
    fac.load(F, j0 + f, n, vec, n_g, gq, r);
    mw = load4<float4>(F.mw + j0 + f, n, vec);
  };

  double acc[NM][4];
#pragma unroll
  for (int i = 0; i < NM; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0;
#pragma unroll
  for (int k = 0; k < kDmmaRing; ++k) {
    if (k < mine) stage(k);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  typename Fac::Raw raw, raw_n;
  float4 mw, mw_n;
  if (mine > 0) inputs(0, raw, mw);
  for (int k = 0; k < mine; ++k) {
    if (k + 1 < mine) inputs(k + 1, raw_n, mw_n);
    if (!land(k)) {  // flag it, give the warp's copies one more bounded wait, leave
      if (lane == 0) atomicOr(err, kErrTimeout);
      for (int q = k; q < min(mine, k + kDmmaRing); ++q) land(q);
      break;
    }
    const float* ma = mk + (k % kDmmaRing) * BS;
    double vw[8], wm[8];
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h) fac.factor(raw, h, s, comp4(mw, s), vw[2 * s + h], wm[2 * s + h]);
#pragma unroll
    for (int i = 0; i < NM; ++i) {
      double m[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        float v = ma[off[i] + s * nb];
        if (i == NM - 1 && wrow) v = comp4(mw, s);
        if ((i == NM - 1 && wpad) || (i == MV - 1 && vpad)) v = 0.f;
        m[s] = (double)v;
      }
      dmma_16816(acc[i], Fac::kSame || i < MV ? vw : wm, m);
    }
    __syncwarp();  // all lanes have read the buffer
    if (k + kDmmaRing < mine) stage(k + kDmmaRing);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    raw = raw_n;
    mw = mw_n;
  }
  // the warps' sums, added in warp order
  __syncthreads();
  double* red = reinterpret_cast<double*>(sm);  // [warp][NM * 4][32]
#pragma unroll
  for (int i = 0; i < NM; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) red[((warp * NM + i) * 4 + c) * 32 + lane] = acc[i][c];
  __syncthreads();
  for (int e = tid; e < NM * 128; e += 32 * kDmmaWarps) {
    const int l = e & 31, c = (e >> 5) & 3;
    const int r = marks_row(8 * (e >> 7) + 2 * (l & 3) + (c & 1), nb), map = (l >> 2) + 8 * (c >> 1);
    if (r < 0 || map >= n_g) continue;
    double t = red[e];
#pragma unroll
    for (int v = 1; v < kDmmaWarps; ++v) t += red[v * NM * 128 + e];
    partial[((size_t)blk * n_g + map) * R + r] = t;
  }
}
size_t marks_dmma_smem(int n_bin) {
  const size_t ring = sizeof(float) * kDmmaWarps * kDmmaRing * (size_t)marks_dmma_buffer(n_bin);
  return std::max(ring, sizeof(double) * 128 * kDmmaWarps * marks_m_tiles(n_bin));
}
// The kernel compiled for n_bin's numbers of row tiles (they are compile-time so
// that the loads, conversions and products of all tiles interleave).
template <class Fac>
using MarksDmma = void (*)(const MarksField*, int, Fac, int, int, long long, double*, unsigned*, int, unsigned);
template <class Fac, int NB = 1>
MarksDmma<Fac> marks_dmma_kernel(int n_bin) {
  if constexpr (NB > kDmmaMaxBins) {
    return nullptr;
  } else {
    return n_bin == NB ? k_marks_dmma<Fac, (2 * NB + 7) / 8, (NB + 1 + 7) / 8> : marks_dmma_kernel<Fac, NB + 1>(n_bin);
  }
}

// Threads per lens group (two per row quad, whole warps) and per block: as
// many groups as fit in kMarksThreads.
int marks_group_threads(int n_bin) { return (2 * (3 * marks_quad_bins(n_bin) / 4 + 1) + 31) / 32 * 32; }
int marks_block_threads(int n_bin) {
  const int tg = marks_group_threads(n_bin);
  return std::max(1, kMarksThreads / tg) * tg;
}
size_t marks_smem(int n_bin) {
  const size_t fac = sizeof(double) * kTileL * kLensStride + std::max(MapFactors::kRawBytes, MultFactors::kRawBytes);
  const size_t red = sizeof(double) * (size_t)marks_group_threads(n_bin) * 32;
  return std::max(fac, red);
}
// Blocks of a pass: as many as fit on a 148-SM part at once (by the shared
// memory and threads of the form used for n_bin), so the pass is one wave.
// A function of n_bin only, so the summation order (and the result) depends
// only on the input.
int marks_blocks(int n_bin) {
  if (n_bin > kDmmaMaxBins) return kMarksBlocks;
  return 148 * marks_dmma_per_sm(marks_m_tiles(n_bin));
}
// Lenses per block for n_lens lenses in all: marks_blocks blocks, whole tiles.
long long marks_chunk(long long n_lens, int n_bin) {
  const long long nbk = marks_blocks(n_bin);
  const long long per = (n_lens + nbk - 1) / nbk;
  return std::max<long long>(kTileL, (per + kTileL - 1) / kTileL * kTileL);
}
// The partial sums of n_maps maps or resamples over all fields, 16 to a pass
// (blockIdx.y; partial sums of a pass follow those of the one before): the FP64 tensor-core form for
// n_bin <= 32, the FP64 FMA form for wider binnings.
template <class Fac>
cudaError_t launch_marks_partials(const MarksField* fields, int n_field, int nblk, long long chunk, const Fac& fac,
                                  int n_maps, int nb, double* part, unsigned* err, int skip_tile, unsigned wait_limit,
                                  cudaStream_t st) {
  const dim3 grid(nblk, (n_maps + kMapGroup - 1) / kMapGroup);
  if (nb <= kDmmaMaxBins) {
    const MarksDmma<Fac> k = marks_dmma_kernel<Fac>(nb);
    const size_t msm = marks_dmma_smem(nb);
    cudaError_t e = allow_dynamic_smem(k);
    if (e != cudaSuccess) return e;
    k<<<grid, 32 * kDmmaWarps, msm, st>>>(fields, n_field, fac, n_maps, nb, chunk, part, err, skip_tile, wait_limit);
    return cudaGetLastError();
  }
  const size_t msm = marks_smem(nb);
  const int bt = marks_block_threads(nb), tg = marks_group_threads(nb);
  cudaError_t e = allow_dynamic_smem(k_marks_partials<Fac>);
  if (e != cudaSuccess) return e;
  k_marks_partials<Fac><<<grid, bt, msm, st>>>(fields, n_field, fac, n_maps, nb, tg, chunk, part);
  return cudaGetLastError();
}

// Multiplicities of G resamples s0.. over n_units units: n_draw draws each,
// counter (d/4, s, 0x2BCF, 0), word d%4, index by multiply-shift (the stream
// of the patch bootstrap).  mult must be zeroed.
__global__ void k_unit_mult(unsigned long long seed, long long n_units, long long n_draw, int s0, int G,
                            int* mult) {
  const long long nq = (n_draw + 3) / 4;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nq * G;
       t += (long long)gridDim.x * blockDim.x) {
    const int g = (int)(t / nq);
    const long long q = t % nq;
    uint32_t c[4] = {(uint32_t)q, (uint32_t)(s0 + g), 0x2BCFu, 0u};
    philox4x32(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    for (int u = 0; u < 4; ++u) {
      const long long d = 4 * q + u;
      if (d < n_draw) {
        const long long idx = (long long)(((unsigned long long)c[u] * (unsigned long long)n_units) >> 32);
        atomicAdd(&mult[(size_t)g * (size_t)n_units + (size_t)idx], 1);
      }
    }
  }
}

// Field sums of several passes: pass p (of blockIdx.z), map or resample g of the
// pass: out[((p MG + g) * n_field + fi) * R + r] = sum over the field's blocks.
// A block covers 32 consecutive outputs of one field: warp v adds blocks v,
// v + 16, ... (256-byte loads of a block's row), then the warps' sums are added in
// warp order (the same order every run).  One warp per output, each lane on
// another block's row, read 32 bytes for every 8 it used: 7.1 us a pass at 435
// blocks x 976 outputs.
constexpr int kMarksReduceWarps = 16;
__global__ void __launch_bounds__(32 * kMarksReduceWarps) k_marks_reduce(const double* __restrict__ partial,
                                                                        const MarksField* __restrict__ fields,
                                                                        int n_field, int n_blocks, int n_map_g, int R,
                                                                        double* __restrict__ out) {
  __shared__ double part[kMarksReduceWarps][32];
  const int lane = threadIdx.x & 31, v = threadIdx.x >> 5;
  // n_map_g: maps of the last pass; the others hold kMapGroup
  const int p = blockIdx.z, g_p = p + 1 < (int)gridDim.z ? kMapGroup : n_map_g;
  const int fi = blockIdx.y, e = blockIdx.x * 32 + lane, ne = g_p * R;
  partial += (size_t)p * n_blocks * kMapGroup * R;
  out += (size_t)p * kMapGroup * n_field * R;
  const int c0 = fields[fi].chunk0;
  const int c1 = fi + 1 < n_field ? fields[fi + 1].chunk0 : n_blocks;
  double s = 0.0;
  if (e < ne) {
#pragma unroll 8
    for (int c = c0 + v; c < c1; c += kMarksReduceWarps) s += partial[(size_t)c * ne + e];
  }
  part[v][lane] = s;
  __syncthreads();
  if (v == 0 && e < ne) {
    double t = part[0][lane];
#pragma unroll
    for (int k = 1; k < kMarksReduceWarps; ++k) t += part[k][lane];
    out[((size_t)(e / R) * n_field + fi) * R + e % R] = t;
  }
}
// g: maps of the last of the n_pass passes.
cudaError_t launch_marks_reduce(const double* part, const MarksField* df, int n_field, int nblk, int n_pass, int g,
                                int R, double* out, cudaStream_t st) {
  const int e = (n_pass > 1 ? kMapGroup : g) * R;
  k_marks_reduce<<<dim3((e + 31) / 32, n_field, n_pass), 32 * kMarksReduceWarps, 0, st>>>(part, df, n_field, nblk, g, R,
                                                                                         out);
  return cudaGetLastError();
}
// Passes whose partial sums are kept (up to 64 MiB) before one reduction of all
// of them: a reduction of one pass is all latency (6 us).
int marks_passes_kept(int nblk, int R, int n_pass) {
  const size_t one = sizeof(double) * (size_t)std::max(nblk, 1) * kMapGroup * R;
  // at most 32768: a grid dimension holds 65535
  return (int)std::max<size_t>(1, std::min<size_t>(std::min<size_t>((size_t)n_pass, 32768), ((size_t)64 << 20) / one));
}

// Multiplicities of the passes of one launch: what stays in L2 between the
// draws and the sums.
constexpr size_t kDrawBytes = (size_t)64 << 20;

// With timing enabled (tpcf_set_timing), CUDA events on the call's stream
// around every partial-sum launch; total() after the stream has synchronised
// is their summed device time, kept as the call's kernel time.
struct PassTimer {
  tpcf_ctx* c;
  std::vector<cudaEvent_t> ev;
  explicit PassTimer(tpcf_ctx* ctx) : c(ctx) {}
  ~PassTimer() {
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
  }
  void mark(cudaStream_t st) {
    if (!c->time_pairs) return;
    cudaEvent_t e = nullptr;
    check(cudaEventCreate(&e), "event");
    ev.push_back(e);
    check(cudaEventRecord(e, st), "event record");
  }
  void total() {
    if (!c->time_pairs) return;
    double ms = 0.0;
    for (size_t i = 0; i + 1 < ev.size(); i += 2) {
      float t = 0.f;
      check(cudaEventElapsedTime(&t, ev[i], ev[i + 1]), "event time");
      ms += t;
    }
    c->last_pair_ms = ms;
  }
};

// Order of the draws and the sums of a marks bootstrap.  With overlap the
// draws run on the context's second stream: a buffer is drawn into once the
// sums over its last contents are done, and summed once it is drawn.  Without,
// everything is on the call's stream.  The destructor waits for the second
// stream, so a call that fails midway leaves nothing running on the workspace.
struct DrawStream {
  tpcf_ctx* c;
  cudaStream_t aux = nullptr;
  std::unique_ptr<Event> drawn[2], free_[2];
  bool busy[2] = {false, false};
  DrawStream(tpcf_ctx* ctx, bool overlap) : c(ctx) {
    if (!overlap) return;
    for (int b = 0; b < 2; ++b) drawn[b].reset(new Event), free_[b].reset(new Event);
    cudaStream_t a = aux_stream(c);
    check(cudaEventRecord(free_[0]->e, c->stream), "event record");
    check(cudaStreamWaitEvent(a, free_[0]->e, 0), "stream wait");  // after all earlier work of the call
    aux = a;
  }
  ~DrawStream() {
    if (aux) cudaStreamSynchronize(aux);
  }
  cudaStream_t begin(int b) {
    if (!aux) return c->stream;
    if (busy[b]) check(cudaStreamWaitEvent(aux, free_[b]->e, 0), "stream wait");
    return aux;
  }
  void end(int b) {
    if (!aux) return;
    check(cudaEventRecord(drawn[b]->e, aux), "event record");
    check(cudaStreamWaitEvent(c->stream, drawn[b]->e, 0), "stream wait");
  }
  void used(int b) {
    if (!aux) return;
    check(cudaEventRecord(free_[b]->e, c->stream), "event record");
    busy[b] = true;
  }
};

// A call's field descriptors, error word and n sums in one piece of device
// memory: one copy up (descriptors and a cleared word) and one down (word and
// sums) in place of two each, which is 10 % of a call on 30 k lenses.
struct MarksCall {
  MarksField* fields;
  unsigned* err;
  double* sums;
  std::vector<double> host;  // [descriptors][error word][sums]
  size_t head;
  MarksCall(tpcf_ctx* c, const std::vector<MarksField>& f, size_t n, cudaStream_t st) {
    static_assert(sizeof(MarksField) % sizeof(double) == 0, "descriptors fill whole doubles");
    head = f.size() * (sizeof(MarksField) / sizeof(double));
    host.assign(head + 1 + n, 0.0);
    std::memcpy(host.data(), f.data(), f.size() * sizeof(MarksField));
    double* d = (double*)ws_alloc(c, sizeof(double) * host.size());
    fields = reinterpret_cast<MarksField*>(d);
    err = reinterpret_cast<unsigned*>(d + head);
    sums = d + head + 1;
    check(cudaMemcpyAsync(d, host.data(), sizeof(double) * (head + 1), cudaMemcpyHostToDevice, st), "H2D fields");
  }
  // waits for the call's stream; the sums
  const double* read(cudaStream_t st) {
    check(cudaMemcpyAsync(host.data() + head, err, sizeof(double) * (host.size() - head), cudaMemcpyDeviceToHost, st),
          "D2H sums");
    check(cudaStreamSynchronize(st), "sync marks");
    unsigned e;
    std::memcpy(&e, host.data() + head, sizeof(e));
    if (e & kErrTimeout) throw Failure(TPCF_ERR_TIMEOUT, "a bounded device wait timed out in the marks kernel");
    return host.data() + head + 1;
  }
};

// Flags a unit label outside [0, n_units).
__global__ void k_check_units(const int* __restrict__ unit, long long n, long long n_units, int* bad) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (unit[i] < 0 || (long long)unit[i] >= n_units) atomicOr(bad, 1);
}

// max |a - b| over n entries, as order-preserving bits of a non-negative float.
__global__ void k_max_absdiff(const float* __restrict__ a, const float* __restrict__ b, long long n, int* out) {
  float m = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float d = fabsf(a[i] - b[i]);
    m = fmaxf(m, d != d ? INFINITY : d);
  }
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_int(m));
}

}  // namespace tpcf

using namespace tpcf;

extern "C" tpcf_status tpcf_xi_from_marks(tpcf_ctx* c, int32_t n_field, const tpcf_marks_field* marks,
                                          int32_t n_map, const float* const* val, const float* const* w,
                                          const float* const* lens_x, const float* const* lens_y, double* g_t,
                                          double* g_x, double* weights, double* g_t_stacked,
                                          double* g_x_stacked, double* weights_stacked) {
  if (!c || n_field < 1 || !marks || n_map < 1 || !val || !w) return TPCF_ERR_INVALID_ARG;
  const int nb = (int)marks[0].n_bin;
  if (nb < 1 || nb > kMaxBins) return TPCF_ERR_INVALID_ARG;
  for (int i = 0; i < n_field; ++i) {
    const tpcf_marks_field& m = marks[i];
    if (m.n_bin != nb || m.n < 0 || m.n > (1ll << 31) - 2 || !val[i] || !w[i]) return TPCF_ERR_INVALID_ARG;
    if (m.n > 0 && (!m.w || !m.xi_E || !m.xi_B || !m.K)) return TPCF_ERR_INVALID_ARG;
  }
  try {
    Phase ph_nvtx("tpcf: marks");
    begin_call(c);
    cudaStream_t st = c->stream;
    std::vector<MarksField> hf(n_field);
    int nblk = 0;
    int64_t n_all = 0;
    for (int i = 0; i < n_field; ++i) n_all += marks[i].n;
    const long long chunk = marks_chunk(n_all, nb);
    for (int i = 0; i < n_field; ++i) {
      const tpcf_marks_field& m = marks[i];
      const int64_t n = m.n;
      MarksField& F = hf[i];
      F.n = n;
      F.n_bin = nb;
      F.chunk0 = nblk;
      F.lens0 = 0;
      nblk += (int)((n + chunk - 1) / chunk);
      F.mw = stage(c, m.w, n);
      F.xiE = stage(c, m.xi_E, n * nb);
      F.xiB = stage(c, m.xi_B, n * nb);
      F.K = stage(c, m.K, n * nb);
      F.val = stage(c, val[i], n * n_map);
      F.w = stage(c, w[i], n * n_map);
      // the lenses must be the ones the marks were computed for (main.f90:1036-1049)
      if (lens_x && lens_y && lens_x[i] && lens_y[i] && n > 0) {
        if (!m.x || !m.y) throw Failure(TPCF_ERR_INVALID_ARG, "marks positions missing for the check");
        const float* a[2] = {stage(c, m.x, n), stage(c, m.y, n)};
        const float* b[2] = {stage(c, lens_x[i], n), stage(c, lens_y[i], n)};
        int* dm = (int*)ws_alloc(c, sizeof(int) * 2);
        check(cudaMemsetAsync(dm, 0, sizeof(int) * 2, st), "memset");
        for (int k = 0; k < 2; ++k) {
          k_max_absdiff<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, st>>>(a[k], b[k], n, dm + k);
          counted(c, cudaGetLastError(), "position check");
        }
        int hm[2];
        check(cudaMemcpyAsync(hm, dm, sizeof(hm), cudaMemcpyDeviceToHost, st), "D2H check");
        check(cudaStreamSynchronize(st), "sync check");
        for (int k = 0; k < 2; ++k) {
          float d;
          std::memcpy(&d, &hm[k], 4);
          if (!(d <= 1.0e-5f))
            throw Failure(TPCF_ERR_INVALID_ARG, std::string(k ? "Y" : "X") + "-coordinates of lenses do not match in field " +
                                                    std::to_string(i));
        }
      }
    }
    const int R = 3 * nb + 1;
    const size_t n_sum = (size_t)n_map * n_field * R;
    const size_t part_pass = (size_t)std::max(nblk, 1) * kMapGroup * R;
    const int n_keep = marks_passes_kept(nblk, R, (n_map + kMapGroup - 1) / kMapGroup);
    double* part = (double*)ws_alloc(c, sizeof(double) * part_pass * n_keep);
    // the sums of every pass stay on the device until one copy after the
    // last pass, so the host queues all passes without waiting on any
    MarksCall call(c, hf, n_sum, st);
    const MarksField* df = call.fields;
    double* dout = call.sums;
    PassTimer timer(c);
    if (nblk == 0) check(cudaMemsetAsync(dout, 0, sizeof(double) * n_sum, st), "memset");
    // all passes whose partial sums are kept in one launch: their first and last
    // blocks overlap
    for (int m0 = 0; m0 < n_map && nblk > 0; m0 += n_keep * kMapGroup) {
      const int g = std::min(n_keep * kMapGroup, n_map - m0), n_pass = (g + kMapGroup - 1) / kMapGroup;
      timer.mark(st);
      counted(c, launch_marks_partials(df, n_field, nblk, chunk, MapFactors{m0}, g, nb, part, call.err, c->skip_tile,
                                       c->wait_limit, st),
              "marks partials");
      timer.mark(st);
      counted(c, launch_marks_reduce(part, df, n_field, nblk, n_pass, g - (n_pass - 1) * kMapGroup, R,
                                     dout + (size_t)m0 * n_field * R, st),
              "marks reduce");
    }
    const double* sums = call.read(st);
    timer.total();
    // normalisation (main.f90:1118-1133): plain quotients, as the reference
    for (int m = 0; m < n_map; ++m) {
      std::vector<double> sE(nb, 0.0), sB(nb, 0.0), sK(nb, 0.0);
      double sw = 0.0;
      for (int i = 0; i < n_field; ++i) {
        const double* s = sums + ((size_t)m * n_field + i) * R;
        for (int b = 0; b < nb; ++b) {
          if (g_t) g_t[((size_t)m * n_field + i) * nb + b] = s[b] / s[2 * nb + b];
          if (g_x) g_x[((size_t)m * n_field + i) * nb + b] = s[nb + b] / s[2 * nb + b];
          sE[b] += s[b];
          sB[b] += s[nb + b];
          sK[b] += s[2 * nb + b];
        }
        if (weights) weights[(size_t)m * n_field + i] = s[3 * nb];
        sw += s[3 * nb];
      }
      for (int b = 0; b < nb; ++b) {
        if (g_t_stacked) g_t_stacked[(size_t)m * nb + b] = sE[b] / sK[b];
        if (g_x_stacked) g_x_stacked[(size_t)m * nb + b] = sB[b] / sK[b];
      }
      if (weights_stacked) weights_stacked[m] = sw;
    }
    return TPCF_OK;
  } catch (...) {
    const Failure f = caught();
    c->err = f.msg;
    return f.status;
  }
}

extern "C" tpcf_status tpcf_marks_bootstrap(tpcf_ctx* c, int32_t n_field, const tpcf_marks_field* marks,
                                            const int32_t* unit, int64_t n_units, const int32_t* multiplicity,
                                            uint64_t seed, int32_t n_boot, double supersampling, int32_t k_guard,
                                            double* g_t, double* g_x, double* weights, double* cov_gt,
                                            double* cov_gx) {
  if (!c || n_field < 1 || !marks || n_boot < 1 || !(supersampling > 0)) return TPCF_ERR_INVALID_ARG;
  const int nb = (int)marks[0].n_bin;
  if (nb < 1 || nb > kMaxBins) return TPCF_ERR_INVALID_ARG;
  int64_t n_lens = 0;
  for (int i = 0; i < n_field; ++i) {
    const tpcf_marks_field& m = marks[i];
    if (m.n_bin != nb || m.n < 0 || (m.n > 0 && (!m.w || !m.xi_E || !m.xi_B || !m.K))) return TPCF_ERR_INVALID_ARG;
    n_lens += m.n;
  }
  if (n_lens > (1ll << 31) - 2) return TPCF_ERR_INVALID_ARG;
  if (!unit) n_units = n_lens;
  if (n_units < 1) return TPCF_ERR_INVALID_ARG;
  try {
    Phase ph_nvtx("tpcf: marks bootstrap");
    begin_call(c);
    cudaStream_t st = c->stream;
    std::vector<MarksField> hf(n_field);
    int nblk = 0;
    int64_t off = 0;
    const long long chunk = marks_chunk(n_lens, nb);
    for (int i = 0; i < n_field; ++i) {
      const tpcf_marks_field& m = marks[i];
      MarksField& F = hf[i];
      F.n = m.n;
      F.n_bin = nb;
      F.chunk0 = nblk;
      F.lens0 = off;
      off += m.n;
      nblk += (int)((m.n + chunk - 1) / chunk);
      F.mw = stage(c, m.w, m.n);
      F.xiE = stage(c, m.xi_E, m.n * nb);
      F.xiB = stage(c, m.xi_B, m.n * nb);
      F.K = stage(c, m.K, m.n * nb);
      F.val = F.w = nullptr;
    }
    const int* dunit = unit ? stage(c, (const int*)unit, n_lens) : nullptr;
    if (dunit) {  // labels must lie in [0, n_units): checked on the device before use
      int* bad = (int*)ws_alloc(c, sizeof(int));
      check(cudaMemsetAsync(bad, 0, sizeof(int), st), "memset");
      k_check_units<<<(unsigned)std::min<int64_t>((n_lens + 255) / 256, 148 * 8), 256, 0, st>>>(dunit, n_lens, n_units,
                                                                                                   bad);
      counted(c, cudaGetLastError(), "unit check");
      int hb = 0;
      check(cudaMemcpyAsync(&hb, bad, sizeof(int), cudaMemcpyDeviceToHost, st), "D2H check");
      check(cudaStreamSynchronize(st), "sync check");
      if (hb) throw Failure(TPCF_ERR_INVALID_ARG, "unit label outside [0, n_units)");
    }
    const int* dmult_all = multiplicity ? stage(c, (const int*)multiplicity, (int64_t)n_boot * n_units) : nullptr;
    // n_samples = int(n_objects * supersampling_factor) (src/tpcf.f90:1234, :894)
    const long long n_draw = (long long)((double)n_units * supersampling);
    if (!multiplicity && n_draw < 1) throw Failure(TPCF_ERR_INVALID_ARG, "no draws per resample");
    const int R = 3 * nb + 1;
    // Multiplicities drawn here (16 M scattered atomic increments per pass of 16
    // resamples of 1 M lenses, bound by L2 atomics) run on a second stream into
    // one of two buffers while the other is summed (bound by FP64).  The draws and
    // sums of as many passes as kDrawBytes holds go in one launch each, so that
    // the passes' first and last blocks overlap.  250 k lenses, 1000 resamples:
    // 3.33 ms for the call; one pass a launch 3.49, two 3.40, eight 3.61; in line
    // 3.45 (the two kernels share the SMs' registers and mostly take turns; fewer
    // draw blocks, to leave the sums room, are slower: 592: 3.74, and drawing
    // inside the sum kernel: 4.9).  One buffer, and no overlap, beyond 1 GiB.
    const size_t part_pass = (size_t)std::max(nblk, 1) * kMapGroup * R;
    const int n_pass_all = (n_boot + kMapGroup - 1) / kMapGroup;
    const size_t mpass = sizeof(int) * (size_t)kMapGroup * n_units;
    int n_keep = marks_passes_kept(nblk, R, n_pass_all);
    const int n_launch = (int)std::max<size_t>(1, std::min<size_t>(n_keep, kDrawBytes / mpass));
    n_keep = n_keep / n_launch * n_launch;
    const size_t mbytes = mpass * n_launch;
    const int n_buf = multiplicity ? 0 : mbytes <= ((size_t)1 << 30) ? 2 : 1;
    int* mbuf[2] = {nullptr, nullptr};
    for (int b = 0; b < n_buf; ++b) mbuf[b] = (int*)ws_alloc(c, mbytes);
    DrawStream draws(c, n_buf == 2);
    int kept = 0;
    double* part = (double*)ws_alloc(c, sizeof(double) * part_pass * n_keep);
    const size_t n_sum = (size_t)n_boot * n_field * R;
    // the sums of every pass stay on the device until one copy after the
    // last pass, so the host queues all passes without waiting on any
    MarksCall call(c, hf, n_sum, st);
    const MarksField* df = call.fields;
    double* dout = call.sums;
    if (nblk == 0) check(cudaMemsetAsync(dout, 0, sizeof(double) * n_sum, st), "memset");
    PassTimer timer(c);
    const int MG = n_launch * kMapGroup;
    for (int s0 = 0; s0 < n_boot; s0 += MG) {
      const int G = std::min(MG, n_boot - s0), n_pass = (G + kMapGroup - 1) / kMapGroup;
      const int* mult;
      if (multiplicity) {
        mult = dmult_all + (size_t)s0 * n_units;
      } else {
        const int b = n_buf == 2 ? (s0 / MG) & 1 : 0;
        cudaStream_t ds = draws.begin(b);
        check(cudaMemsetAsync(mbuf[b], 0, sizeof(int) * (size_t)G * n_units, ds), "memset mult");
        const long long work = (n_draw + 3) / 4 * G;
        k_unit_mult<<<(unsigned)std::min<long long>((work + 255) / 256, 148 * 16), 256, 0, ds>>>(seed, n_units, n_draw,
                                                                                                 s0, G, mbuf[b]);
        counted(c, cudaGetLastError(), "bootstrap draws");
        draws.end(b);
        mult = mbuf[b];
      }
      if (nblk > 0) {
        timer.mark(st);
        counted(c,
                launch_marks_partials(df, n_field, nblk, chunk, MultFactors{mult, dunit, n_units}, G, nb,
                                      part + part_pass * kept, call.err,
                                      c->skip_tile, c->wait_limit, st),
                "bootstrap partials");
        timer.mark(st);
        if (!multiplicity) draws.used((n_buf == 2 ? (s0 / MG) & 1 : 0));
        kept += n_pass;
        if (kept == n_keep || s0 + G == n_boot) {
          counted(c, launch_marks_reduce(part, df, n_field, nblk, kept, G - (n_pass - 1) * kMapGroup, R,
                                         dout + (size_t)(s0 / kMapGroup + n_pass - kept) * kMapGroup * n_field * R, st),
                  "bootstrap reduce");
          kept = 0;
        }
      }
    }
    const double* sums = call.read(st);
    timer.total();
    // all fields together (src/tpcf.f90:1245-1262); K > 0 guard of the point
    // bootstraps, plain quotients for the pair-weighted block bootstrap (:929-930)
    std::vector<double> gt((size_t)n_boot * nb), gx((size_t)n_boot * nb);
    for (int s = 0; s < n_boot; ++s) {
      double W = 0.0;
      for (int b = 0; b < nb; ++b) {
        double E = 0.0, B = 0.0, K = 0.0;
        for (int i = 0; i < n_field; ++i) {
          const double* r = sums + ((size_t)s * n_field + i) * R;
          E += r[b];
          B += r[nb + b];
          K += r[2 * nb + b];
        }
        const bool zero = k_guard && !(K > 0.0);
        gt[(size_t)s * nb + b] = zero ? 0.0 : E / K;
        gx[(size_t)s * nb + b] = zero ? 0.0 : B / K;
      }
      for (int i = 0; i < n_field; ++i) W += sums[((size_t)s * n_field + i) * R + 3 * nb];
      if (weights) weights[s] = W;
    }
    if (g_t) std::memcpy(g_t, gt.data(), sizeof(double) * gt.size());
    if (g_x) std::memcpy(g_x, gx.data(), sizeof(double) * gx.size());
    if ((cov_gt || cov_gx) && n_boot >= 2) {
      double* dg = (double*)ws_alloc(c, sizeof(double) * gt.size());
      double* dc = (double*)ws_alloc(c, sizeof(double) * (size_t)nb * nb);
      for (int q = 0; q < 2; ++q) {
        double* user = q == 0 ? cov_gt : cov_gx;
        if (!user) continue;
        check(cudaMemcpyAsync(dg, (q == 0 ? gt : gx).data(), sizeof(double) * gt.size(), cudaMemcpyHostToDevice, st),
              "H2D g");
        counted(c, launch_cov(dg, n_boot, nb, dc, st), "covariance");
        check(cudaMemcpyAsync(user, dc, sizeof(double) * nb * nb, cudaMemcpyDefault, st), "D2H cov");
        check(cudaStreamSynchronize(st), "sync cov");
      }
    }
    return TPCF_OK;
  } catch (...) {
    const Failure f = caught();
    c->err = f.msg;
    return f.status;
  }
}
