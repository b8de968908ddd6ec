// pairs.cu -- the pair-summing kernels of libtpcf_b200 (sm_100a).
//
// Replaces the OpenMP pair loops of tangential_shear_tpcf
// (src/tpcf.f90:261-363) and scalar_kappa_tpcf (src/tpcf.f90:451-535).
//
// Every warp works on its own: it takes work items of 32 lenses (one per
// lane) from an atomic queue and walks the source rows of the items'
// theta_max neighbourhood.  The source grid is stored in HBM as 32-source
// sub-chunks already in the pair-interleaved form of the packed FP32
// instructions (SrcPair), each with its bounding box and sums (ChunkMeta), so
// a tile is copied into shared memory by the bulk-copy engine (cp.async.bulk
// + mbarrier, issued by lane 0) and used as it lands.  Each warp owns a ring
// of tile buffers; no barrier or shared state ties it to the other warps of
// its block.  Every lane reads the same source (broadcast) and bins its
// pairs into its own FP32 histogram column in shared memory, laid out
// [bin][quantity][thread] so that a warp's 32 read-modify-writes fall in 32
// distinct banks whatever bins the lanes pick, with no atomics.  Every ~4096
// sources (1024 with per-lens output) the warp folds its 32 columns into its
// FP64 sums (times the lens factors val*w or w) and, when per-lens output is
// requested, into per-lens FP64 columns.
//
// Most pairs never touch the histogram: per 32-source sub-chunk a lens whose
// bin range (from the sub-chunk's box) spans at most three bins sums in
// registers and adds once per sub-chunk.  Those register paths run on sm_100's
// packed FP32 instructions (two pairs per instruction).
//
// Binning.  The pair arithmetic is FP32.  For log spacing the bin comes from
// t = log2(d2)*A + B (one MUFU.LG2 and one FFMA): bin = floor(t).  When t is
// within `eps` of an integer the pair is re-binned in FP64 by the canonical
// rule (squared FP64 edges, d2 from the FP32 inputs without contraction), so
// n_pairs is identical to the FP64 rule of tpcf_canonical_edges.  Other
// spacings binary-search the FP32 squared edges with a relative guard band.

#include <algorithm>
#include <cub/cub.cuh>
#include <cstdio>

#include "pair_hist.cuh"
#include "pair_tiles.cuh"
#include "tpcf_device.cuh"
#include "tpcf_internal.cuh"
#include "tpcf_kernels.h"

#ifndef TPCF_DUAL_UNROLL
#define TPCF_DUAL_UNROLL 4
#endif
#ifndef TPCF_SINGLE_UNROLL
#define TPCF_SINGLE_UNROLL 8
#endif

namespace tpcf {

constexpr int kDualUnroll = TPCF_DUAL_UNROLL;      // source-loop unrolling of the edge paths
constexpr int kSingleUnroll = TPCF_SINGLE_UNROLL;  // and of the single-bin path
// Warps per SM that the pair kernel is compiled for: the shared-memory
// occupancy of 128 threads at 20 bins (51 KB histogram + tiles).  Declaring it
// gives the compiler a register budget (up to 168 per thread) that it spends
// on overlapping the packed FP32 chains of the register paths.
constexpr int kPairWarps = 12;
// Coordinate of the null source that pads the last sub-chunk of a grid: its
// d2 (~2e36) stays finite in FP32 and its weight and values are zero.
constexpr float kNullPos = 1.0e18f;
// Tile buffers per warp: TCH sub-chunks (1 KB each) plus their ChunkMeta each.
constexpr int kPairBuf = 2;
constexpr int kRowsPerPass = 32;  // cell rows whose spans a warp holds at once (one per lane)

// ------------------------------------------------------- shared-memory map --
struct PairSmem {
  size_t ring, hist, bsum, e2s, fvw, fw, e2f, mbar, misc, total;
};
__host__ __device__ inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
// Bytes of one ring buffer: TCH sub-chunks and their metadata.
__host__ __device__ inline size_t ring_buffer_bytes(int tch) {
  return (size_t)tch * (kChunk * sizeof(SrcRec) + sizeof(ChunkMeta));
}
// bt is the number of threads (histogram columns), tch the sub-chunks per tile.
__host__ __device__ inline PairSmem pair_smem_layout(int nb, int qa, int bt, int tch) {
  const int nw = bt / 32;
  const int nbuf = kPairBuf;
  PairSmem s;
  size_t o = 0;
  s.ring = o;  o += (size_t)nw * nbuf * ring_buffer_bytes(tch);
  s.hist = o;  o += (size_t)nb * qa * bt * sizeof(float);
  o = align_up(o, 16);
  s.bsum = o;  o += (size_t)nw * kQ * nb * sizeof(double);
  s.e2s = o;   o += (size_t)(nb + 1) * sizeof(double);
  s.fvw = o;   o += (size_t)bt * sizeof(double);
  s.fw = o;    o += (size_t)bt * sizeof(double);
  s.e2f = o;   o += (size_t)(nb + 1) * sizeof(float);
  o = align_up(o, 8);
  s.mbar = o;  o += (size_t)nw * nbuf * sizeof(uint64_t);
  s.misc = o;  o += 16;
  s.total = align_up(o, 128);
  return s;
}

// One pair: lens (lx, ly, lz) against source record (a, b).  hcol points at
// this lens's histogram column; row (bin*QA + q) is at hcol[(bin*QA+q)*NC].
template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB, int NC, int QA>
__device__ __forceinline__ void do_pair(float lx, float ly, float lz, const float4 a, const float4 b,
                                        float* __restrict__ hcol, const BinCtx& C) {
  if (HAS_Z) {
    if (lz > b.z) return;  // src/tpcf.f90:322
  }
  const float dx = lx - a.x;
  const float dy = ly - a.y;
  const float dx2 = dx * dx;
  const float d2 = fmaf(dy, dy, dx2);
  const int bin = pair_bin<LOGB>(d2, lx, ly, a.x, a.y, C);
  if ((unsigned)bin >= (unsigned)C.nb) return;
  // d and 1/d^2 from one MUFU.RSQ.  Generic spacings may have x_min = 0, where
  // d2 = 0 is in range: there d = sqrt(0) = 0 exactly (as in the reference).
  float d, r;
  if (LOGB) {
    const float rs = rsqrt_ftz(d2);
    d = d2 * rs;
    r = rs * rs;
  } else {
    d = sqrtf(d2);
    r = __frcp_rn(d2);
  }
  float* h = hcol + bin * (QA * NC);
  if (MODE == 0) {
    // cos 2phi = (dx^2 - dy^2)/d^2, sin 2phi = 2 dx dy / d^2 (src/tpcf.f90:343-344)
    const float c2 = fmaf(-dy, dy, dx2) * r;
    const float qq = dx * dy;
    const float s2 = (qq + qq) * r;
    // a.z = -e1*w, a.w = -e2*w:  g_t term = a.z*c2 + a.w*s2,  g_x term = a.w*c2 - a.z*s2
    const float gt = fmaf(a.z, c2, a.w * s2);
    const float gx = fmaf(a.w, c2, -(a.z * s2));
    h[QGT * NC] += gt;
    h[QGX * NC] += gx;
  } else {
    h[QGT * NC] += a.z;
    h[QGX * NC] += a.w;
  }
  h[QW * NC] += b.x;
  h[QDW * NC] = fmaf(d, b.x, h[QDW * NC]);
  h[QN * NC] += 1.0f;
  if (MODE == 0 && HAS_M) h[QK * NC] += b.y;
}

// ---------------------------------------------------- sub-chunk fast paths --
// Each sub-chunk holds 32 consecutive sources of the cell-sorted order
// (spatially compact: cells in rows, Hilbert order inside a cell).  For each
// lens and sub-chunk the bin range of the chunk's bounding box is bounded
// conservatively (guard band eps on both ends):
//   0  no pair of the chunk is in range        -> nothing to do
//   1  every pair is in one bin `blo`           -> register sums, no binning
//   2  pairs fall in bins blo, blo+1            -> register sums split at the
//   3  pairs fall in bins blo .. blo+2             one or two edges, FP64
//                                                  re-binning inside a guard
//                                                  band
//   4  anything else                           -> per-pair binning (do_pair)
// The path is chosen per warp (the largest class of its lanes), so lanes never
// diverge inside a source loop.  Every pair still lands in its canonical bin:
// in classes 1 to 3 the box bounds prove which bins are possible.
//
// A row span of the grid starts and ends anywhere inside a sub-chunk; its
// first and last sub-chunks are "partial": only the sources [lo, hi) of the
// sub-chunk belong to the span (the others belong to other cells and are
// either out of reach or counted through another span).  The box of a partial
// sub-chunk covers all its sources, so the bounds stay conservative; its pairs
// carry a per-pair mask, as does a z cut (z_A > z_B skips the pair).

// Per-pair quantities shared by the register paths, for the two sources of
// one SrcPair at once (packed FP32: one instruction per operation for both
// pairs).  Shear: with P = dx^2 - dy^2, u = 2 dx dy and r = 1/d^2,
// cos 2phi = P r, sin 2phi = u r (src/tpcf.f90:343-344), so the g_t, g_x
// terms are r*X and r*Y with X = p P + q u, Y = q P - p u (p = -e1 w,
// q = -e2 w).  Scalar-scalar: X = kE w, Y = kB w, r = 1.  Each half of a
// packed operation rounds like the scalar operation (x - lx = -(lx - x));
// the compiler may fuse a product into a following add, as it may in scalar
// code, so a term agrees with a scalar evaluation to within one FMA rounding.
struct LensP {
  float2 nlx, nly;  // (-lx, -lx), (-ly, -ly)
};

template <int MODE, bool LOGB>
__device__ __forceinline__ void pair_terms2(const LensP& L, const float4 xy, const float4 pq, float2& d2, float2& d,
                                            float2& r, float2& X, float2& Y) {
  const float2 dxp = add2(lo2(xy), L.nlx);  // x - lx
  const float2 dyp = add2(hi2(xy), L.nly);  // y - ly
  const float2 dx2 = mul2(dxp, dxp);
  d2 = fma2(dyp, dyp, dx2);
  if (LOGB) {
    const float2 rs = make_float2(rsqrt_ftz(d2.x), rsqrt_ftz(d2.y));
    d = mul2(d2, rs);
    r = mul2(rs, rs);
  } else {
    d = make_float2(sqrtf(d2.x), sqrtf(d2.y));
    r = make_float2(__frcp_rn(d2.x), __frcp_rn(d2.y));
  }
  if (MODE == 0) {
    const float2 P = fma2(make_float2(-dyp.x, -dyp.y), dyp, dx2);  // dx^2 - dy^2
    const float2 qq = mul2(dxp, dyp);
    const float2 u = add2(qq, qq);                                 // 2 dx dy
    X = fma2(lo2(pq), P, mul2(hi2(pq), u));
    const float2 pu = mul2(lo2(pq), u);
    Y = fma2(hi2(pq), P, make_float2(-pu.x, -pu.y));
  } else {
    r = dup2(1.f);
    X = lo2(pq);
    Y = hi2(pq);
  }
}

// Source j of a sub-chunk in SrcPair form, as the (a, b) records of do_pair.
__device__ __forceinline__ void src_of(const SrcPair* __restrict__ S, int j, float4& a, float4& b) {
  const float* f = reinterpret_cast<const float*>(S + (j >> 1)) + (j & 1);
  a = make_float4(f[0], f[2], f[4], f[6]);
  b = make_float4(f[8], f[10], f[12], 0.f);
}

// Which of the two sources of pair block k take part: the z cut and, in a
// partial sub-chunk, the span [lo, hi).
template <bool HAS_Z, bool PART>
__device__ __forceinline__ float2 pair_mask(const SrcPair* __restrict__ S, int k, float lz, int lo, int hi, bool& a0,
                                            bool& a1) {
  a0 = true;
  a1 = true;
  if (HAS_Z) {
    const float4 zn = S[k].zn;
    a0 = lz <= zn.x;  // src/tpcf.f90:322 (a NaN z of a null source fails)
    a1 = lz <= zn.y;
  }
  if (PART) {
    a0 = a0 && (2 * k >= lo);
    a1 = a1 && (2 * k + 1 < hi);
  }
  return make_float2(a0 ? 1.f : 0.f, a1 ? 1.f : 0.f);
}

// The register paths share the sub-chunk sums ss = {sum p, sum q, sum w,
// sum K} over its sources: for a whole sub-chunk without a z cut, the w and K
// sums of every lens are these (and, for scalar-scalar, so are the g_t and
// g_x sums, r = 1), so they are not accumulated per pair.
//
// Class 1: every pair of the chunk is in bin `blo`.  A masked pair (z cut,
// outside the span) adds nothing.
template <int MODE, bool HAS_M, bool HAS_Z, bool PART, bool LOGB, int NC, int QA>
__device__ __forceinline__ void chunk_single(const SrcPair* __restrict__ S, int lo, int hi, const LensP& L, float lz,
                                             int cls, int blo, float* __restrict__ hcol, const float4 ss) {
  constexpr bool MK = HAS_Z || PART;
  constexpr bool LI = !MK;  // lens-independent sums come from ss
  float2 sgt = dup2(0.f), sgx = dup2(0.f), sw = dup2(0.f), sdw = dup2(0.f), sk = dup2(0.f), sn = dup2(0.f);
  const int k0 = PART ? (lo >> 1) : 0;
  const int k1 = PART ? ((hi + 1) >> 1) : kChunk / 2;
#pragma unroll kSingleUnroll
  for (int k = k0; k < k1; ++k) {
    const float4 xy = S[k].xy, pq = S[k].pq, wk = S[k].wk;
    float2 d2, d, r, X, Y;
    pair_terms2<MODE, LOGB>(L, xy, pq, d2, d, r, X, Y);
    float2 w = lo2(wk), K = hi2(wk);
    if (MK) {
      bool a0, a1;
      const float2 zm = pair_mask<HAS_Z, PART>(S, k, lz, lo, hi, a0, a1);
      r = mul2(r, zm);
      w = mul2(w, zm);
      if (MODE == 0 && HAS_M) K = mul2(K, zm);
      sn = add2(sn, zm);
    }
    if (!(LI && MODE == 1)) {
      sgt = fma2(r, X, sgt);
      sgx = fma2(r, Y, sgx);
    }
    if (!LI) sw = add2(sw, w);
    sdw = fma2(d, w, sdw);
    if (MODE == 0 && HAS_M && !LI) sk = add2(sk, K);
  }
  if (cls != 1) return;
  float acc[QA];
  acc[QGT] = (LI && MODE == 1) ? ss.x : sum2(sgt);
  acc[QGX] = (LI && MODE == 1) ? ss.y : sum2(sgx);
  acc[QW] = LI ? ss.z : sum2(sw);
  acc[QDW] = sum2(sdw);
  acc[QN] = MK ? sum2(sn) : (float)kChunk;
  if (MODE == 0 && HAS_M) acc[QK] = LI ? ss.w : sum2(sk);
  hist_add<QA, NC>(hcol, blo, acc);
}

// Classes 2 and 3: the pairs of the chunk fall in bins blo .. blo + NE across
// NE = 1 or 2 edges (a bin outside [0, nb) is dropped); edge e is
// e2f[blo + 1 + e].  Sums over all pairs (s*) and, per edge, over the pairs on
// its far side (h*[e]: d2 >= E_e); bin blo + j receives h[j-1] - h[j] with
// h[-1] = all and h[NE] = 0.  The side of a pair is a 1.0/0.0 mask from the sign
// of d2 - E, applied by multiplication.  The smallest |d2 - E| is kept per
// edge: when it lies within the guard band, or a sum is not finite (a pair with
// d = 0), this lane drops its register sums and bins the sub-chunk pair by pair by
// the canonical rule (rare).  A lane with fewer edges than NE
// (class 1, or class 2 in a class-3 warp) keeps 3e38 on its unused edges (its
// |d2 - E| is then 3e38 too: out of the band).
template <int MODE, bool HAS_M, bool HAS_Z, bool PART, bool LOGB, int NC, int QA, int NE>
__device__ __forceinline__ void chunk_edges(const SrcPair* __restrict__ S, int lo, int hi, const LensP& L, float lx,
                                            float ly, float lz, int cls, int blo, float* __restrict__ hcol,
                                            const BinCtx& C, const float4 ss) {
  constexpr bool MK = HAS_Z || PART;
  constexpr bool LI = !MK;
  float2 sgt = dup2(0.f), sgx = dup2(0.f), sw = dup2(0.f), sdw = dup2(0.f), sk = dup2(0.f), sn = dup2(0.f);
  float2 hgt[NE], hgx[NE], hw[NE], hdw[NE], hk[NE], hn[NE];
  float E[NE], close[NE];  // edges and the smallest |d2 - E|
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    hgt[e] = hgx[e] = hw[e] = hdw[e] = hk[e] = hn[e] = dup2(0.f);
    E[e] = e < cls - 1 ? C.e2f[min(max(blo + 1 + e, 0), C.nb)] : 3.0e38f;
    close[e] = 3.0e38f;
  }
  const int k0 = PART ? (lo >> 1) : 0;
  const int k1 = PART ? ((hi + 1) >> 1) : kChunk / 2;
#pragma unroll kDualUnroll
  for (int k = k0; k < k1; ++k) {
    const float4 xy = S[k].xy, pq = S[k].pq, wk = S[k].wk;
    float2 d2, d, r, X, Y;
    pair_terms2<MODE, LOGB>(L, xy, pq, d2, d, r, X, Y);
    float2 w = lo2(wk), K = hi2(wk);
    float2 zm = dup2(1.f);
    if (MK) {
      bool a0, a1;
      zm = pair_mask<HAS_Z, PART>(S, k, lz, lo, hi, a0, a1);
      r = mul2(r, zm);
      w = mul2(w, zm);
      if (MODE == 0 && HAS_M) K = mul2(K, zm);
      sn = add2(sn, zm);
    }
    // products folded into the sums: one packed FFMA per quantity and side
    if (!(LI && MODE == 1)) {
      sgt = fma2(r, X, sgt);
      sgx = fma2(r, Y, sgx);
    }
    if (!LI) sw = add2(sw, w);
    sdw = fma2(d, w, sdw);
    if (MODE == 0 && HAS_M && !LI) sk = add2(sk, K);
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const float2 t = add2(d2, dup2(-E[e]));
      close[e] = fminf(close[e], fminf(fabsf(t.x), fabsf(t.y)));
      float2 mh = make_float2(t.x >= 0.f ? 1.f : 0.f, t.y >= 0.f ? 1.f : 0.f);
      if (MK) mh = mul2(mh, zm);
      const float2 rm = mul2(r, mh);
      const float2 wm = mul2(w, mh);
      hgt[e] = fma2(rm, X, hgt[e]);
      hgx[e] = fma2(rm, Y, hgx[e]);
      hw[e] = add2(hw[e], wm);
      hdw[e] = fma2(d, wm, hdw[e]);
      hn[e] = add2(hn[e], mh);
      if (MODE == 0 && HAS_M) hk[e] = fma2(K, mh, hk[e]);
    }
  }
  if (cls == 0) return;
  // a pair with d = 0 (1/d^2 infinite, d NaN for log bins) is on a side of its own:
  // its 0/1 mask does not keep it out of the other sums
  bool band = !(fabsf(sum2(sdw)) <= kMaxFinite) || (MODE == 0 && !(fabsf(sum2(sgt)) <= kMaxFinite));
#pragma unroll
  for (int e = 0; e < NE; ++e) band = band || close[e] <= E[e] * C.eps_rel;
  if (band) {
    for (int j = lo; j < hi; ++j) {
      float4 a, b;
      src_of(S, j, a, b);
      do_pair<MODE, HAS_M, HAS_Z, LOGB, NC, QA>(lx, ly, lz, a, b, hcol, C);
    }
    return;
  }
  float prev[QA];
  prev[QGT] = (LI && MODE == 1) ? ss.x : sum2(sgt);
  prev[QGX] = (LI && MODE == 1) ? ss.y : sum2(sgx);
  prev[QW] = LI ? ss.z : sum2(sw);
  prev[QDW] = sum2(sdw);
  prev[QN] = MK ? sum2(sn) : (float)kChunk;
  if (MODE == 0 && HAS_M) prev[QK] = LI ? ss.w : sum2(sk);
#pragma unroll
  for (int j = 0; j <= NE; ++j) {
    float up[QA];
    if (j < NE) {
      up[QGT] = sum2(hgt[j]);
      up[QGX] = sum2(hgx[j]);
      up[QW] = sum2(hw[j]);
      up[QDW] = sum2(hdw[j]);
      up[QN] = sum2(hn[j]);
      if (MODE == 0 && HAS_M) up[QK] = sum2(hk[j]);
    } else {
#pragma unroll
      for (int q = 0; q < QA; ++q) up[q] = 0.f;
    }
    const int bin = blo + j;
    if (j <= cls - 1 && bin >= 0 && bin < C.nb) {
      float v[QA];
#pragma unroll
      for (int q = 0; q < QA; ++q) v[q] = prev[q] - up[q];
      hist_add<QA, NC>(hcol, bin, v);
    }
#pragma unroll
    for (int q = 0; q < QA; ++q) prev[q] = up[q];
  }
}

#ifdef TPCF_MODE_STATS
// Diagnostic build only: warp-level path counts [4], lane-pairs per warp path
// [4], and lane-pairs per lane class [4] (active lanes only).
__device__ unsigned long long g_mode_stats[15];
extern "C" int tpcf_debug_mode_stats(unsigned long long* out) {
  return (int)cudaMemcpyFromSymbol(out, g_mode_stats, sizeof(g_mode_stats));
}
#endif

// ------------------------------------------------------------ pair kernel --
// Every warp is independent: it takes its own work items (32 lenses, one per
// lane, against every source row the group's theta_max neighbourhood touches)
// from the queue and streams their tiles through its own ring of NBUF buffers
// in shared memory (bulk copies issued by lane 0, one mbarrier per buffer,
// bounded waits); no barrier and no shared state ties it to the other warps
// of the block, so a warp never waits for another's share of work.  The
// block's warps share only the launch (occupancy, the bin edges).
// PATH 0: sub-chunk classification with the register paths (default);
// PATH 1: per-pair binning for every pair in reach (for A/B measurement).
template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB, int BT, int TCH, int PATH>
__global__ void __launch_bounds__(BT, kPairWarps * 32 / BT) k_pairs(const PairParams P) {
  constexpr int QA = (MODE == 0 && HAS_M) ? 6 : 5;
  constexpr int NBUF = kPairBuf;
  constexpr size_t BUFB = (size_t)TCH * (kChunk * sizeof(SrcRec) + sizeof(ChunkMeta));
  const int nb = P.nb;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  extern __shared__ __align__(128) unsigned char smem[];
  const PairSmem L = pair_smem_layout(nb, QA, BT, TCH);
  unsigned char* wring = smem + L.ring + (size_t)warp * NBUF * BUFB;
  float* hist = reinterpret_cast<float*>(smem + L.hist);
  double* bsum = reinterpret_cast<double*>(smem + L.bsum);
  double* e2s = reinterpret_cast<double*>(smem + L.e2s);
  double* fvw = reinterpret_cast<double*>(smem + L.fvw);
  double* fw = reinterpret_cast<double*>(smem + L.fw);
  float* e2f = reinterpret_cast<float*>(smem + L.e2f);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.mbar) + (size_t)warp * NBUF;
  auto tile_ptr = [&](int b) { return reinterpret_cast<SrcPair*>(wring + (size_t)b * BUFB); };
  auto meta_ptr = [&](int b) {
    return reinterpret_cast<ChunkMeta*>(wring + (size_t)b * BUFB + (size_t)TCH * kChunk * sizeof(SrcRec));
  };

  if (lane == 0) {
    for (int b = 0; b < NBUF; ++b) mbar_init(&full[b], 1);
    mbar_fence_init();
  }
  for (int i = tid; i <= nb; i += BT) {
    e2s[i] = P.e2[i];
    e2f[i] = P.e2f[i];
  }
  __syncthreads();
  BinCtx C;
  C.A = P.binA; C.B = P.binB; C.eps = P.eps; C.one_m_eps = 1.f - P.eps;
  C.nb = nb; C.e2s = e2s; C.e2f = e2f;
  C.eps_rel = 4e-6f;
  C.lo_g = e2f[0] * (1.f - P.eps);
  C.hi_g = e2f[nb] * (1.f + P.eps);

  const uint32_t wait_limit = P.wait_limit ? P.wait_limit : kWaitPolls;
  int ring_t = 0;         // ring index of the next tile this warp consumes
  int issued_end = 0;     // ring index one past the last tile this warp issued
  bool aborted = false;   // a bounded wait ran out: consume and issue nothing more
  float* __restrict__ hcol = hist + tid;
  double* wsum = bsum + (size_t)warp * kQ * nb;
#ifdef TPCF_MODE_STATS
  __shared__ unsigned long long sh_stats[15];
  if (tid < 15) sh_stats[tid] = 0ull;
  __syncthreads();
#endif
  for (int e = 0; e < nb * QA; ++e) hcol[e * BT] = 0.f;

  int item = 0, run_i = 0, run_n = 0;
  while (!aborted) {
    if (run_i == run_n) {  // this item's parts are done: the next item
      if (lane == 0) item = atomicAdd(P.queue_head, 1);
      item = __shfl_sync(0xffffffffu, item, 0);
      if (item >= P.n_items) break;
      run_i = 0;
    }
    const int2 it = P.items[item];
    const TaskDesc T = P.tasks[it.x];
    run_n = T.run;
    const LensDesc LD = P.lenses[T.lens_cat];
    const GridDesc G = P.grids[T.src_cat];
    const int per = T.split / T.run, g = it.y / per;
    const int part = (it.y - g * per) * T.run + run_i++;
    const int gs = LD.group_start[g];
    const int nl = LD.group_start[g + 1] - gs;
    const bool act = lane < nl;
    float lx = 0.f, ly = 0.f, lz = 0.f;
    double vw = 0.0, w = 0.0;
    double* lens_col = nullptr;
    if (act) {
      const float4 r = LD.rec[gs + lane];
      lx = r.x; ly = r.y;
      vw = (double)r.z * (double)r.w;
      w = (double)r.w;
      if (HAS_Z) lz = LD.z[gs + lane];
      if (P.lens_acc && T.lens_acc_off >= 0)
        lens_col = P.lens_acc + T.lens_acc_off + (size_t)(T.run > 1 ? 0 : part) * kQ * nb * LD.n_valid + gs + lane;
    }
    LensP LP;
    LP.nlx = dup2(-lx);
    LP.nly = dup2(-ly);
    fvw[tid] = vw;
    fw[tid] = w;
    const size_t lens_stride = (size_t)LD.n_valid;
    for (int e = lane; e < kQ * nb; e += 32) wsum[e] = 0.0;
    int since_flush = 0;
    const float4 box = LD.group_box[g];
    int cy0, cy1;
    row_range(G, box, P.R, T.margin, cy0, cy1);

    for (int c0 = cy0 + part; c0 <= cy1 && !aborted; c0 += kRowsPerPass * T.split) {
      int s0 = 0, s1 = 0;
      const int row = c0 + lane * T.split;
      if (row <= cy1) {
        const int2 sp = row_span(G, box, P.R, T.margin, row);
        s0 = sp.x;
        s1 = sp.y > sp.x ? sp.y : sp.x;
      }
      const int ntr = tiles_of_span<TCH>(s0, s1);
      int incl = ntr;  // inclusive prefix of the tile counts over the lanes (rows)
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const int ntiles = __shfl_sync(0xffffffffu, incl, 31);
      // Ring: the tile with ring index t lives in buffer t % NBUF and completes
      // phase (t / NBUF) & 1 of that buffer's barrier.  The pass's tile k has
      // ring index ring_t + k; each consumed buffer is refilled at once with
      // the tile NBUF places ahead.
      auto issue = [&](int k) {
        const TileGeom tg = tile_of<TCH>(k, incl, ntr, s0, s1);  // all lanes (shuffles)
        const int t = ring_t + k;
        issued_end = t + 1;
        if (t + 1 == P.debug_skip_tile) return;  // fault injection (tests): this tile never lands
        if (lane == 0) {
          const int b = t % NBUF;
          mbar_arrive_tx(&full[b], (uint32_t)(tg.n * (kChunk * sizeof(SrcRec) + sizeof(ChunkMeta))));
          bulk_g2s(tile_ptr(b), G.pairs + (size_t)tg.c0 * (kChunk / 2), (uint32_t)tg.n * kChunk * sizeof(SrcRec),
                   &full[b]);
          bulk_g2s(meta_ptr(b), G.meta + tg.c0, (uint32_t)tg.n * sizeof(ChunkMeta), &full[b]);
        }
      };
      for (int k = 0; k < NBUF && k < ntiles; ++k) issue(k);
      for (int k = 0; k < ntiles; ++k) {
        const int t = ring_t + k;
        const int b = t % NBUF;
        const TileGeom tg = tile_of<TCH>(k, incl, ntr, s0, s1);
        const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[b], (uint32_t)(t / NBUF) & 1u, wait_limit));
        if (!ok) {  // stop: drain this warp's copies in flight below, report the timeout
          aborted = true;
          ring_t = t;
          break;
        }
        const SrcPair* Tb = tile_ptr(b);
        const ChunkMeta* Mb = meta_ptr(b);
        for (int j = 0; j < tg.n; ++j) {
          const int lo = j == 0 ? tg.lo0 : 0;
          const int hi = j == tg.n - 1 ? tg.hiL : kChunk;
          if (since_flush >= T.flush_src) {
            warp_fold<QA, BT>(hist, hcol, wsum, fvw, fw, nb, lens_col, lens_stride, warp, lane);
            since_flush = 0;
          }
          since_flush += hi - lo;
          const bool part = lo > 0 || hi < kChunk;
          const SrcPair* __restrict__ Sc = Tb + j * (kChunk / 2);
          const float4 cbox = Mb[j].box;
          int blo = 0;
          int cls = act ? classify_edges<LOGB>(lx, ly, cbox, C, blo) : 0;
          if (PATH == 1 && cls) cls = 4;
          const int m = (int)__reduce_max_sync(0xffffffffu, (unsigned)cls);
#ifdef TPCF_MODE_STATS
          {
            const unsigned nact = __popc(__ballot_sync(0xffffffffu, act));
            unsigned ncls[5];
            for (int cc = 0; cc < 5; ++cc) ncls[cc] = __popc(__ballot_sync(0xffffffffu, act && cls == cc));
            if (lane == 0) {
              atomicAdd(&sh_stats[m], 1ull);
              atomicAdd(&sh_stats[5 + m], (unsigned long long)((hi - lo) * nact));
              for (int cc = 0; cc < 5; ++cc)
                atomicAdd(&sh_stats[10 + cc], (unsigned long long)((hi - lo) * ncls[cc]));
            }
          }
#endif
          if (m == 0) continue;
          const float4 ss = Mb[j].sum;
          if (m == 1) {
            if (part)
              chunk_single<MODE, HAS_M, HAS_Z, true, LOGB, BT, QA>(Sc, lo, hi, LP, lz, cls, blo, hcol, ss);
            else
              chunk_single<MODE, HAS_M, HAS_Z, false, LOGB, BT, QA>(Sc, 0, kChunk, LP, lz, cls, blo, hcol, ss);
          } else if (m == 2) {
            if (part)
              chunk_edges<MODE, HAS_M, HAS_Z, true, LOGB, BT, QA, 1>(Sc, lo, hi, LP, lx, ly, lz, cls, blo, hcol, C,
                                                                     ss);
            else
              chunk_edges<MODE, HAS_M, HAS_Z, false, LOGB, BT, QA, 1>(Sc, 0, kChunk, LP, lx, ly, lz, cls, blo, hcol,
                                                                      C, ss);
          } else if (m == 3) {
            if (part)
              chunk_edges<MODE, HAS_M, HAS_Z, true, LOGB, BT, QA, 2>(Sc, lo, hi, LP, lx, ly, lz, cls, blo, hcol, C,
                                                                     ss);
            else
              chunk_edges<MODE, HAS_M, HAS_Z, false, LOGB, BT, QA, 2>(Sc, 0, kChunk, LP, lx, ly, lz, cls, blo, hcol,
                                                                      C, ss);
          } else if (act) {
            for (int jj = lo; jj < hi; ++jj) {
              float4 a, bb;
              src_of(Sc, jj, a, bb);
              do_pair<MODE, HAS_M, HAS_Z, LOGB, BT, QA>(lx, ly, lz, a, bb, hcol, C);
            }
          }
        }
        __syncwarp();  // every lane is done reading buffer b
        if (k + NBUF < ntiles) issue(k + NBUF);
      }
      if (!aborted) ring_t += ntiles;
    }
    if (aborted) break;
    warp_fold<QA, BT>(hist, hcol, wsum, fvw, fw, nb, lens_col, lens_stride, warp, lane);
    double* out = P.item_sums + (size_t)(T.item_base + g * T.split + part) * kQ * nb;
    for (int e = lane; e < kQ * nb; e += 32) {
      const int src = (e / nb == QK && QA == 5) ? e - (QK - QW) * nb : e;
      out[e] = wsum[src];
    }
    __syncwarp();
  }
  if (aborted) {
    // No tile is consumed or issued any more; wait (bounded) for the copies
    // this warp issued and did not consume, so that none is in flight when
    // the block's shared memory is released.
    for (int t = ring_t; t < issued_end; ++t)
      if (t + 1 != P.debug_skip_tile) mbar_wait_bounded(&full[t % NBUF], (uint32_t)(t / NBUF) & 1u, wait_limit);
    if (lane == 0) atomicOr(P.err, kErrTimeout);
  }
#ifdef TPCF_MODE_STATS
  __syncthreads();
  if (tid < 15) atomicAdd(&g_mode_stats[tid], sh_stats[tid]);
#endif
}

// ------------------------------------------------------------ prep kernels --
__device__ __forceinline__ int f2ord(float f) {
  int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// Bounding box, z range and count of the valid objects of one catalogue.
// box_ord = {minx, miny, maxx, maxy, minz, maxz} as order-preserving ints;
// prange = {min, max} of the patch labels of valid lenses.
// kind 0 = source (z < 0 masked, src/tpcf.f90:306); kind 1 = lens (w == 0
// skipped, src/tpcf.f90:285; z < 0 masked).
__global__ void k_bbox(const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z,
                       const float* __restrict__ w, const int* __restrict__ patch, const float* __restrict__ m,
                       long long n, int kind, int* box_ord, unsigned long long* count, int* prange) {
  float mnx = INFINITY, mny = INFINITY, mxx = -INFINITY, mxy = -INFINITY, mnz = INFINITY, mxz = -INFINITY;
  float mxm = 0.f;
  int pmn = INT_MAX, pmx = INT_MIN;
  unsigned long long c = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float xi = x[i], yi = y[i];
    const float zi = z ? z[i] : 0.f;
    bool v = isfinite(xi) && isfinite(yi) && zi >= 0.f;
    if (kind == 1) {
      if (w[i] == 0.f) v = false;
      if (v && patch) { pmn = min(pmn, patch[i]); pmx = max(pmx, patch[i]); }
    }
    if (v) {
      mnx = fminf(mnx, xi); mxx = fmaxf(mxx, xi);
      mny = fminf(mny, yi); mxy = fmaxf(mxy, yi);
      mnz = fminf(mnz, zi); mxz = fmaxf(mxz, zi);
      if (m) mxm = fmaxf(mxm, fabsf(m[i]));
      ++c;
    }
  }
  typedef cub::BlockReduce<float, 256> BRf;
  typedef cub::BlockReduce<unsigned long long, 256> BRu;
  typedef cub::BlockReduce<int, 256> BRi;
  __shared__ union {
    typename BRf::TempStorage f;
    typename BRu::TempStorage u;
    typename BRi::TempStorage i;
  } tmp;
  const float mins[3] = {mnx, mny, mnz};
  const float maxs[3] = {mxx, mxy, mxz};
  const int slot_min[3] = {0, 1, 4};
  const int slot_max[3] = {2, 3, 5};
  for (int k = 0; k < 3; ++k) {
    float r = BRf(tmp.f).Reduce(mins[k], cub::Min());
    __syncthreads();
    if (threadIdx.x == 0) atomicMin(&box_ord[slot_min[k]], f2ord(r));
    r = BRf(tmp.f).Reduce(maxs[k], cub::Max());
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&box_ord[slot_max[k]], f2ord(r));
  }
  {
    const float r = BRf(tmp.f).Reduce(mxm, cub::Max());
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&box_ord[6], f2ord(r));
  }
  const unsigned long long cs = BRu(tmp.u).Sum(c);
  __syncthreads();
  if (threadIdx.x == 0) atomicAdd(count, cs);
  int pi = BRi(tmp.i).Reduce(pmn, cub::Min());
  __syncthreads();
  if (threadIdx.x == 0) atomicMin(&prange[0], pi);
  pi = BRi(tmp.i).Reduce(pmx, cub::Max());
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(&prange[1], pi);
}

__global__ void k_bbox_init(int* box_ord, unsigned long long* count, int* prange, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    box_ord[8 * i + 0] = f2ord(INFINITY);
    box_ord[8 * i + 1] = f2ord(INFINITY);
    box_ord[8 * i + 2] = f2ord(-INFINITY);
    box_ord[8 * i + 3] = f2ord(-INFINITY);
    box_ord[8 * i + 4] = f2ord(INFINITY);
    box_ord[8 * i + 5] = f2ord(-INFINITY);
    box_ord[8 * i + 6] = f2ord(0.f);
    box_ord[8 * i + 7] = 0;
    count[i] = 0;
    prange[2 * i] = INT_MAX;
    prange[2 * i + 1] = INT_MIN;
  }
}

__global__ void k_bbox_finish(const int* box_ord, float* box, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) box[i] = ord2f(box_ord[i]);
}


// Sort key of each source: (cell << mb) | Hilbert index of its position inside
// the cell on a 2^(mb/2) grid, so that consecutive sources of one cell are
// spatially compact (32-source sub-chunks get small bounding boxes).  Invalid
// sources get ncells << mb and sort last.
__global__ void k_src_keys(const float* __restrict__ x, const float* __restrict__ y,
                           const float* __restrict__ z, long long n, float x0, float y0, float inv_cell,
                           int ncx, int ncy, int mb, unsigned* keys, int* idx) {
  const unsigned ncells = (unsigned)ncx * (unsigned)ncy;
  const int half = mb >> 1;
  const float q = (float)(1u << half);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float xi = x[i], yi = y[i];
    bool v = isfinite(xi) && isfinite(yi);
    if (z && z[i] < 0.f) v = false;
    unsigned key = ncells << mb;
    if (v) {
      const float fx = (xi - x0) * inv_cell, fy = (yi - y0) * inv_cell;
      const int cx = clamp_floor(fx, 0, ncx - 1);
      const int cy = clamp_floor(fy, 0, ncy - 1);
      key = ((unsigned)cy * (unsigned)ncx + (unsigned)cx) << mb;
      if (half > 0) {
        const unsigned qx = (unsigned)clamp_floor((fx - (float)cx) * q, 0, (1 << half) - 1);
        const unsigned qy = (unsigned)clamp_floor((fy - (float)cy) * q, 0, (1 << half) - 1);
        key |= hilbert_index(qx, qy, half);
      }
    }
    keys[i] = key;
    idx[i] = (int)i;
  }
}

// cell_start[c] = first sorted position with key >= c << mb, for c in [0, ncells].
__global__ void k_cell_start(const unsigned* __restrict__ keys, long long n, unsigned ncells, int mb,
                             int* cell_start) {
  const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > ncells) return;
  const unsigned t = c << mb;
  long long lo = 0, hi = n;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (keys[mid] < t) lo = mid + 1; else hi = mid;
  }
  cell_start[c] = (int)lo;
}

// Cell-sorted source records in sub-chunk form: one warp per 32-source
// sub-chunk gathers its sources (sorted positions 32c .. 32c+31, null sources
// past n_valid) into 16 SrcPair blocks -- sources 2k and 2k+1 with their
// fields interleaved, {x0 x1 y0 y1}{p0 p1 q0 q1}{w0 w1 K0 K1}{z0 z1 0 0} --
// and writes the sub-chunk's bounding box and {p, q, w, K} sums.  Shear:
// p = -e1 w, q = -e2 w, K = (1+m) w; scalar-scalar (mode 1): p = kE w,
// q = kB w, K = w.
__global__ void k_src_pairs(const int* __restrict__ idx, int n_valid, int n_chunks, int mode,
                            const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z,
                            const float* __restrict__ f1, const float* __restrict__ f2,
                            const float* __restrict__ w, const float* __restrict__ m, SrcPair* pairs,
                            ChunkMeta* meta) {
  const int c = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= n_chunks) return;  // whole warps
  const int s = c * kChunk + lane;
  float4 a = make_float4(kNullPos, kNullPos, 0.f, 0.f);
  float4 b = make_float4(0.f, 0.f, __int_as_float(0x7fc00000), 0.f);
  float mnx = INFINITY, mny = INFINITY, mxx = -INFINITY, mxy = -INFINITY;
  if (s < n_valid) {
    const int i = idx[s];
    const float wi = w[i];
    if (mode == 0) {
      a = make_float4(x[i], y[i], -(f1[i] * wi), -(f2[i] * wi));
      const float mi = m ? m[i] : 0.f;
      b = make_float4(wi, wi * (1.0f + mi), z ? z[i] : 0.f, 0.f);
    } else {
      a = make_float4(x[i], y[i], f1[i] * wi, f2[i] * wi);
      b = make_float4(wi, wi, 0.f, 0.f);
    }
    mnx = mxx = a.x;
    mny = mxy = a.y;
  }
  const bool odd = lane & 1;
  // lanes 2k, 2k+1 trade halves: the even lane writes {x, y, p, q} of both,
  // the odd lane {w, K, z}
  const float r0 = __shfl_xor_sync(0xffffffffu, odd ? a.x : b.x, 1);
  const float r1 = __shfl_xor_sync(0xffffffffu, odd ? a.y : b.y, 1);
  const float r2 = __shfl_xor_sync(0xffffffffu, odd ? a.z : b.z, 1);
  const float r3 = __shfl_xor_sync(0xffffffffu, a.w, 1);
  float4* dst = reinterpret_cast<float4*>(pairs + (size_t)c * (kChunk / 2) + (lane >> 1));
  if (!odd) {
    dst[0] = make_float4(a.x, r0, a.y, r1);
    dst[1] = make_float4(a.z, r2, a.w, r3);
  } else {
    dst[2] = make_float4(r0, b.x, r1, b.y);
    dst[3] = make_float4(r2, b.z, 0.f, 0.f);
  }
  float s0 = a.z, s1 = a.w, s2 = b.x, s3 = b.y;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
    mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
    mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
    mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    s3 += __shfl_xor_sync(0xffffffffu, s3, o);
  }
  if (lane == 0) {
    meta[c].box = make_float4(mnx, mny, mxx, mxy);
    meta[c].sum = make_float4(s0, s1, s2, s3);
  }
}


// Lens sort keys: (patch << 2 half) | Hilbert index of (x, y) on a 2^half grid
// over the box (groups of consecutive lenses of one patch: a third less box
// diagonal than Morton order on the tomography lenses); invalid lenses get
// patch n_patch and sort last.
template <class Key>
__global__ void k_lens_keys(const float* __restrict__ x, const float* __restrict__ y,
                            const float* __restrict__ z, const float* __restrict__ w,
                            const int* __restrict__ patch, long long n, float4 box, int half, int n_patch,
                            Key* keys, int* idx) {
  const int top = (1 << half) - 1;
  const float sx = (float)top / fmaxf(box.z - box.x, 1e-30f);
  const float sy = (float)top / fmaxf(box.w - box.y, 1e-30f);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float xi = x[i], yi = y[i];
    bool v = isfinite(xi) && isfinite(yi) && (!w || w[i] != 0.f);
    if (z && z[i] < 0.f) v = false;
    Key key = (Key)n_patch << (2 * half);
    if (v) {
      const unsigned qx = (unsigned)clamp_floor((xi - box.x) * sx, 0, top);
      const unsigned qy = (unsigned)clamp_floor((yi - box.y) * sy, 0, top);
      const Key p = patch ? (Key)(unsigned)patch[i] : (Key)0;
      key = (p << (2 * half)) | (Key)hilbert_index(qx, qy, half);
    }
    keys[i] = key;
    idx[i] = (int)i;
  }
}

__global__ void k_lens_gather(const int* __restrict__ idx, int n_valid, const float* __restrict__ x,
                              const float* __restrict__ y, const float* __restrict__ z,
                              const float* __restrict__ val, const float* __restrict__ w, float4* rec,
                              float* zs, int* perm) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_valid) return;
  const int i = idx[s];
  rec[s] = make_float4(x[i], y[i], val[i], w[i]);
  if (zs) zs[s] = z ? z[i] : 0.f;
  perm[s] = i;
}

// off[p] = first sorted lens with patch >= p, for p in [0, n_patch].
template <class Key>
__global__ void k_patch_offsets(const Key* __restrict__ keys, int n_valid, int n_patch, int shift, int* off) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > n_patch) return;
  const Key t = (Key)(unsigned)p << shift;
  int lo = 0, hi = n_valid;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (keys[mid] < t) lo = mid + 1; else hi = mid;
  }
  off[p] = lo;
}

// Groups of `size` consecutive lenses of one patch: starts [n_groups + 1] and
// the patch's group range {0, n_groups}.
__global__ void k_uniform_groups(int n_groups, int n_valid, int size, int* start, int* patch_groups) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g <= n_groups) start[g] = min(g * size, n_valid);
  if (g == 0) {
    patch_groups[0] = 0;
    patch_groups[1] = n_groups;
  }
}

// One warp per group: bounding box of its lenses.
__global__ void k_group_box(const float4* __restrict__ rec, const int* __restrict__ gstart, int n_groups,
                            float4* box) {
  const int g = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x & 31;
  if (g >= n_groups) return;
  float mnx = INFINITY, mny = INFINITY, mxx = -INFINITY, mxy = -INFINITY;
  for (int i = gstart[g] + lane; i < gstart[g + 1]; i += 32) {
    const float4 r = rec[i];
    mnx = fminf(mnx, r.x); mxx = fmaxf(mxx, r.x);
    mny = fminf(mny, r.y); mxy = fmaxf(mxy, r.y);
  }
  for (int o = 16; o; o >>= 1) {
    mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
    mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
    mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
    mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
  }
  if (lane == 0) box[g] = make_float4(mnx, mny, mxx, mxy);
}

// Work items and their cost bands (cost = lenses x sources in the item's
// rows); 8 threads per item share its rows.
__global__ void k_item_cost(const int2* __restrict__ ranges, int n_ranges, int n_items,
                            const TaskDesc* __restrict__ tasks, const LensDesc* __restrict__ lenses,
                            const GridDesc* __restrict__ grids, float R, int2* __restrict__ items,
                            unsigned* __restrict__ band) {
  const int i = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 3), v = threadIdx.x & 7;
  const bool live = i < n_items;
  const int2 it = item_at(ranges, n_ranges, live ? i : n_items - 1);
  const TaskDesc T = tasks[it.x];
  const LensDesc L = lenses[T.lens_cat];
  const GridDesc G = grids[T.src_cat];
  const int per = T.split / T.run, g = it.y / per, part = it.y - g * per;
  const float4 box = L.group_box[g];
  int cy0, cy1;
  row_range(G, box, R, T.margin, cy0, cy1);
  unsigned long long s = 0;
  for (int cy = cy0 + part + v * per; cy <= cy1; cy += 8 * per) {
    const int2 sp = row_span(G, box, R, T.margin, cy);
    if (sp.y > sp.x) s += (unsigned long long)(sp.y - sp.x);
  }
#pragma unroll
  for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (!live || v) return;
  const unsigned long long nl = (unsigned long long)(L.group_start[g + 1] - L.group_start[g]);
  items[i] = it;
  band[i] = cost_band(s * nl + 1);
}

// Items by descending cost band in one block (up to kOrderMax items; five
// launches of a radix sort otherwise, 58 us against 6 us for 5000 items).  The
// order inside a band is not fixed: every item sums into its own slot, so the
// order changes no result (shards, which must agree on it, sort instead).
constexpr int kOrderMax = 16384;
__global__ void __launch_bounds__(1024) k_item_order(const int2* __restrict__ items, const unsigned* __restrict__ band,
                                                     int n, int2* __restrict__ out) {
  __shared__ int count[kCostBands], base[kCostBands];
  __shared__ int wsum[kCostBands / 32];
  const int t = threadIdx.x;
  if (t < kCostBands) count[t] = 0;
  __syncthreads();
  for (int i = t; i < n; i += 1024) atomicAdd(&count[kCostBands - 1 - band[i]], 1);
  __syncthreads();
  int v = 0, incl = 0;
  if (t < kCostBands) {  // exclusive scan, highest band first
    v = incl = count[t];
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if ((t & 31) >= o) incl += u;
    }
    if ((t & 31) == 31) wsum[t >> 5] = incl;
  }
  __syncthreads();
  if (t < kCostBands) {
    int add = 0;
    for (int k = 0; k < (t >> 5); ++k) add += wsum[k];
    base[t] = incl - v + add;
  }
  __syncthreads();
  for (int i = t; i < n; i += 1024) out[atomicAdd(&base[kCostBands - 1 - band[i]], 1)] = items[i];
}
__global__ void k_iota32(int* v, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = i;
}

// out[j] = items[order[j*count + index]]: shard `index` of `count`, taking every
// count-th item of the cost-descending order (balanced shards).
__global__ void k_permute_items(const int2* __restrict__ items, const int* __restrict__ order, int n, int index,
                                int count, int2* out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const long long i = (long long)j * count + index;
  if (i < n) out[j] = items[order[i]];
}

// FP32 FMA throughput probe: 8 independent FFMA chains per thread.
__global__ void k_ffma_peak(float* out, int iters, float a, float b) {
  float r[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) r[k] = threadIdx.x * 1e-3f + k;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = fmaf(r[k], a, b);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += r[k];
  if (s == 12345.678f) out[0] = s;  // keeps the loop alive, never true in practice
}

// FP64 FMA throughput probe: 8 independent DFMA chains per thread.
__global__ void k_dfma_peak(double* out, int iters, double a, double b) {
  double r[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) r[k] = threadIdx.x * 1e-3 + k;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = fma(r[k], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += r[k];
  if (s == 12345.678) out[0] = s;  // keeps the loop alive, never true in practice
}

// Per-patch FP64 sums from item sums, fixed order (deterministic).
// patch_groups[p] .. patch_groups[p+1] are the groups of patch p, `split` items each.  Block
// (p, c) covers the 32 sums e = 32 c + lane of patch p: warp w adds the items
// g0 + w, g0 + w + kReduceWarps, ... (lane-contiguous loads), then the warp sums
// are added in warp order.
constexpr int kReduceWarps = 32;  // 5000 items of one patch: 63 us with 8 warps
__global__ void __launch_bounds__(32 * kReduceWarps) k_patch_reduce(const double* __restrict__ item_sums, int item_base,
                                                                   int split, const int* __restrict__ patch_groups, int n_patch,
                                                                   int nb, double* patch_sums) {
  __shared__ double part[kReduceWarps][32];
  const int p = blockIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int e = blockIdx.y * 32 + lane;
  const int ne = kQ * nb;
  const int g0 = patch_groups[p] * split, g1 = patch_groups[p + 1] * split;
  double s = 0.0;
  if (e < ne) {
#pragma unroll 8
    for (int g = g0 + w; g < g1; g += kReduceWarps) s += item_sums[(size_t)(item_base + g) * ne + e];
  }
  part[w][lane] = s;
  __syncthreads();
  if (w == 0 && e < ne) {
    double t = part[0][lane];
    for (int k = 1; k < kReduceWarps; ++k) t += part[k][lane];
    patch_sums[(size_t)p * ne + e] = t;
  }
}

// Per-lens outputs in input order from per-lens FP64 sums [kQ][nb][n_valid]
// (sorted order, no lens factors), the `split` parts of the task added in
// order.  Outputs must be zeroed beforehand (masked lenses keep 0, as in the
// reference).
//
// Bound by HBM (the sums once, the outputs once).  The sums lie lens by lens and
// the outputs bin by bin, so a block turns 32 lenses x kOutBins bins around in
// shared memory and both sides are runs of 160 to 256 bytes; with one thread per
// lens every store of a warp touched 32 sectors: 60 k lenses in 4 parts, 15 bins,
// raw FP64 sums: 195 us, against 50 now (32 at 6650 GB/s; 71 with the parts loaded
// one after the other).  20 bins a chunk keep seven blocks on an SM: 100 k
// lenses in 2 parts, 20 / 24 / 31 / 32 bins 96 / 127 / 152 / 147 us, against 121 / 131 /
// 160 / 196 with chunks of 31.
constexpr int kOutBins = 20;
__global__ void __launch_bounds__(128) k_lens_outputs(const double* __restrict__ acc, int split,
                                                      const float4* __restrict__ rec, const int* __restrict__ perm,
                                                      int n_valid, int nb, float* xi_E, float* xi_B, float* K_m,
                                                      float* w_m, float* marks_weight, double* lens_sums,
                                                      double* lens_raw) {
  __shared__ double tile[32][kQ * kOutBins + 1];  // odd stride: no bank conflicts across lenses
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s0 = blockIdx.x * 32, ns = min(32, n_valid - s0);
  const size_t part = (size_t)kQ * nb * n_valid;
  const int quantity[6] = {QDW, QGT, QGX, QW, QK, QN};  // in the order of lens_sums
  double mw = 0.0;
  for (int b0 = 0; b0 < nb; b0 += kOutBins) {
    const int cb = min(kOutBins, nb - b0);
    if (lane < ns) {
#pragma unroll
      for (int j = 0; j < 6; ++j) {
#pragma unroll 2
        for (int b = warp; b < cb; b += 4) {
          const double* a = acc + (size_t)(quantity[j] * nb + b0 + b) * n_valid + s0 + lane;
          double v[kMaxSplit];  // loaded together, added in order
#pragma unroll
          for (int p = 0; p < kMaxSplit; ++p) v[p] = p < split ? a[p * part] : 0.0;
#pragma unroll
          for (int p = 1; p < kMaxSplit; ++p) v[0] += p < split ? v[p] : 0.0;
          tile[lane][j * kOutBins + b] = v[0];
        }
      }
    }
    __syncthreads();
    if (marks_weight && threadIdx.x < ns) {
      const double w = (double)rec[s0 + threadIdx.x].w;
      for (int b = 0; b < cb; ++b) mw += tile[threadIdx.x][3 * kOutBins + b] * w;
    }
    for (int l = warp; l < ns; l += 4) {
      const float4 r = rec[s0 + l];
      const double w = (double)r.w, vw = (double)r.z * w;
      const size_t i = (size_t)perm[s0 + l];
      if (lane < cb) {
        const int b = b0 + lane;
        double v[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) v[j] = tile[l][j * kOutBins + lane];
        const double o[6] = {v[0] * w, v[1] * vw, v[2] * vw, v[3] * w, v[4] * w, v[5]};
        if (xi_E) {
          xi_E[i * nb + b] = (float)o[1];
          xi_B[i * nb + b] = (float)o[2];
          K_m[i * nb + b] = (float)o[4];
          w_m[i * nb + b] = (float)o[3];
        }
#pragma unroll
        for (int j = 0; j < 6; ++j) {
          if (lens_sums) lens_sums[(i * 6 + j) * nb + b] = o[j];
          if (lens_raw) lens_raw[(i * 6 + j) * nb + b] = v[j];
        }
      }
    }
    __syncthreads();
  }
  if (marks_weight && threadIdx.x < ns) marks_weight[perm[s0 + threadIdx.x]] = (float)mw;
}
static_assert(kOutBins <= 32, "a warp's lanes are the bins of a chunk");

// --------------------------------------------------------- host launchers --
// prepare_*: sets the kernel's shared-memory attribute and sizes its grid
// (persistent: the occupancy times the SM count, at most one warp per work
// item); the launch itself is a plain cudaLaunchKernel of the result, so that
// a prepared launch can be recorded into a CUDA graph.
template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB, int BT, int TCH, int PATH>
static cudaError_t prepare_pairs_t(const PairParams& P, int num_sms, PairLaunch* L) {
  constexpr int QA = (MODE == 0 && HAS_M) ? 6 : 5;
  const size_t smem = pair_smem_layout(P.nb, QA, BT, TCH).total;
  auto kern = k_pairs<MODE, HAS_M, HAS_Z, LOGB, BT, TCH, PATH>;
  cudaError_t e = allow_dynamic_smem(kern);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BT, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  int grid = per_sm * num_sms;
  const int need = (P.n_items + BT / 32 - 1) / (BT / 32);  // each warp takes items of its own
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  L->func = reinterpret_cast<const void*>(kern);
  L->grid = grid;
  L->block = BT;
  L->smem = smem;
  return cudaSuccess;
}

// Tile shapes: bt threads per block (128, 64 or 32; each warp takes 32-lens
// work items of its own) and tch sub-chunks per source tile (two
// buffers of tch x 1.1 KB per warp).  variant 1 forces per-pair binning
// (A/B measurement).
template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB>
static cudaError_t prepare_pairs_bt(const PairParams& P, int bt, int tch, int variant, int num_sms, PairLaunch* L) {
  if (bt == 128) {
    if (variant == 1 && MODE == 0 && !HAS_M && !HAS_Z && LOGB)
      return prepare_pairs_t<MODE, HAS_M, HAS_Z, LOGB, 128, 2, 1>(P, num_sms, L);
    if (tch == 1) return prepare_pairs_t<MODE, HAS_M, HAS_Z, LOGB, 128, 1, 0>(P, num_sms, L);
    return prepare_pairs_t<MODE, HAS_M, HAS_Z, LOGB, 128, 2, 0>(P, num_sms, L);
  }
  if (bt == 64) return prepare_pairs_t<MODE, HAS_M, HAS_Z, LOGB, 64, 2, 0>(P, num_sms, L);
  return prepare_pairs_t<MODE, HAS_M, HAS_Z, LOGB, 32, 2, 0>(P, num_sms, L);
}

size_t pair_smem_bytes(int nb, int qa, int bt, int tch) { return pair_smem_layout(nb, qa, bt, tch).total; }

// Tile shape of a call that sets none, at most *bt threads: the one that keeps
// the most warps on an SM (228 KB of shared memory, 1 KB of it per block; 12 warps
// by registers); among equals the one with the longest tiles and largest blocks,
// whose per-tile work is least.  128 threads x 2 sub-chunks keep 12 warps up to 20
// bins and 8 beyond or, with shear calibration (a sixth sum per bin), from 18 bins
// on; there 128 x 1 or 64 x 2 keep 10 or 12: 100 k lenses x 500 k sources, 20
// bins, shear calibration: kernel 7.91 -> 7.17 ms with 128 x 1; 60 k x
// 300 k, 35 bins: 4.6 -> 3.34 ms.
void pair_tile_shape(int nb, int qa, int* bt, int* tch) {
  const int shapes[4][2] = {{128, 2}, {128, 1}, {64, 2}, {32, 2}};
  const int bt_max = *bt;
  int best = 0;
  for (const auto& s : shapes) {
    if (s[0] > bt_max) continue;
    const int blocks = (int)((size_t)(228 * 1024) / (pair_smem_bytes(nb, qa, s[0], s[1]) + 1024));
    const int warps = std::min(blocks * s[0] / 32, kPairWarps);
    if (warps > best) best = warps, *bt = s[0], *tch = s[1];
  }
}

cudaError_t prepare_pairs(const PairParams& P, int mode, bool has_m, bool has_z, bool logb, int bt, int tch,
                          int variant, int num_sms, PairLaunch* L) {
  if (mode == 1) {
    return logb ? prepare_pairs_bt<1, false, false, true>(P, bt, tch, variant, num_sms, L)
                : prepare_pairs_bt<1, false, false, false>(P, bt, tch, variant, num_sms, L);
  }
  if (has_m) {
    if (has_z) return logb ? prepare_pairs_bt<0, true, true, true>(P, bt, tch, variant, num_sms, L)
                           : prepare_pairs_bt<0, true, true, false>(P, bt, tch, variant, num_sms, L);
    return logb ? prepare_pairs_bt<0, true, false, true>(P, bt, tch, variant, num_sms, L)
                : prepare_pairs_bt<0, true, false, false>(P, bt, tch, variant, num_sms, L);
  }
  if (has_z) return logb ? prepare_pairs_bt<0, false, true, true>(P, bt, tch, variant, num_sms, L)
                         : prepare_pairs_bt<0, false, true, false>(P, bt, tch, variant, num_sms, L);
  return logb ? prepare_pairs_bt<0, false, false, true>(P, bt, tch, variant, num_sms, L)
              : prepare_pairs_bt<0, false, false, false>(P, bt, tch, variant, num_sms, L);
}

cudaError_t launch_prepared(const PairLaunch& L, const PairParams& P, cudaStream_t st) {
  void* args[] = {const_cast<PairParams*>(&P)};
  return cudaLaunchKernel(L.func, dim3((unsigned)L.grid), dim3((unsigned)L.block), args, L.smem, st);
}

cudaError_t launch_pairs(const PairParams& P, int mode, bool has_m, bool has_z, bool logb, int bt, int tch,
                         int variant, int num_sms, cudaStream_t st, int* grid) {
  PairLaunch L;
  cudaError_t e = prepare_pairs(P, mode, has_m, has_z, logb, bt, tch, variant, num_sms, &L);
  if (e != cudaSuccess) return e;
  *grid = L.grid;
  return launch_prepared(L, P, st);
}

static inline unsigned gdim(long long n, int b) {
  long long g = (n + b - 1) / b;
  if (g < 1) g = 1;
  if (g > 148 * 32) g = 148 * 32;
  return (unsigned)g;
}

cudaError_t launch_bbox(const float* x, const float* y, const float* z, const float* w, const int* patch,
                        const float* m, long long n, int kind, int* box_ord, unsigned long long* count,
                        int* prange, cudaStream_t st) {
  if (n > 0) k_bbox<<<gdim(n, 256), 256, 0, st>>>(x, y, z, w, patch, m, n, kind, box_ord, count, prange);
  return cudaGetLastError();
}
cudaError_t launch_bbox_init(int* box_ord, unsigned long long* count, int* prange, int n, cudaStream_t st) {
  k_bbox_init<<<1, 1024, 0, st>>>(box_ord, count, prange, n);
  return cudaGetLastError();
}
cudaError_t launch_bbox_finish(const int* box_ord, float* box, int n, cudaStream_t st) {
  k_bbox_finish<<<(n + 255) / 256, 256, 0, st>>>(box_ord, box, n);
  return cudaGetLastError();
}
cudaError_t launch_src_keys(const float* x, const float* y, const float* z, long long n, float x0, float y0,
                            float inv_cell, int ncx, int ncy, int mb, unsigned* keys, int* idx, cudaStream_t st) {
  if (n > 0) k_src_keys<<<gdim(n, 256), 256, 0, st>>>(x, y, z, n, x0, y0, inv_cell, ncx, ncy, mb, keys, idx);
  return cudaGetLastError();
}
cudaError_t launch_cell_start(const unsigned* keys, long long n, unsigned ncells, int mb, int* cell_start,
                              cudaStream_t st) {
  k_cell_start<<<(ncells + 1 + 255) / 256, 256, 0, st>>>(keys, n, ncells, mb, cell_start);
  return cudaGetLastError();
}
cudaError_t launch_src_pairs(const int* idx, int n_valid, int mode, const float* x, const float* y, const float* z,
                             const float* f1, const float* f2, const float* w, const float* m, SrcPair* pairs,
                             ChunkMeta* meta, cudaStream_t st) {
  const int n_chunks = (n_valid + kChunk - 1) / kChunk;
  if (n_chunks > 0)
    k_src_pairs<<<(n_chunks + 7) / 8, 256, 0, st>>>(idx, n_valid, n_chunks, mode, x, y, z, f1, f2, w, m, pairs,
                                                     meta);
  return cudaGetLastError();
}
template <class Key>
cudaError_t launch_lens_keys(const float* x, const float* y, const float* z, const float* w, const int* patch,
                             long long n, float4 box, int half, int n_patch, Key* keys, int* idx, cudaStream_t st) {
  if (n > 0) k_lens_keys<Key><<<gdim(n, 256), 256, 0, st>>>(x, y, z, w, patch, n, box, half, n_patch, keys, idx);
  return cudaGetLastError();
}
template cudaError_t launch_lens_keys<unsigned>(const float*, const float*, const float*, const float*, const int*,
                                                long long, float4, int, int, unsigned*, int*, cudaStream_t);
template cudaError_t launch_lens_keys<unsigned long long>(const float*, const float*, const float*, const float*,
                                                          const int*, long long, float4, int, int,
                                                          unsigned long long*, int*, cudaStream_t);
cudaError_t launch_lens_gather(const int* idx, int n_valid, const float* x, const float* y, const float* z,
                               const float* val, const float* w, float4* rec, float* zs, int* perm, cudaStream_t st) {
  if (n_valid > 0) k_lens_gather<<<(n_valid + 255) / 256, 256, 0, st>>>(idx, n_valid, x, y, z, val, w, rec, zs, perm);
  return cudaGetLastError();
}
template <class Key>
cudaError_t launch_patch_offsets(const Key* keys, int n_valid, int n_patch, int shift, int* off, cudaStream_t st) {
  k_patch_offsets<Key><<<(n_patch + 1 + 255) / 256, 256, 0, st>>>(keys, n_valid, n_patch, shift, off);
  return cudaGetLastError();
}
template cudaError_t launch_patch_offsets<unsigned>(const unsigned*, int, int, int, int*, cudaStream_t);
template cudaError_t launch_patch_offsets<unsigned long long>(const unsigned long long*, int, int, int, int*,
                                                              cudaStream_t);
cudaError_t launch_uniform_groups(int n_groups, int n_valid, int size, int* start, int* patch_groups,
                                  cudaStream_t st) {
  k_uniform_groups<<<(n_groups + 1 + 255) / 256, 256, 0, st>>>(n_groups, n_valid, size, start, patch_groups);
  return cudaGetLastError();
}
cudaError_t launch_group_box(const float4* rec, const int* gstart, int n_groups, float4* box, cudaStream_t st) {
  if (n_groups > 0) k_group_box<<<(n_groups + 7) / 8, 256, 0, st>>>(rec, gstart, n_groups, box);
  return cudaGetLastError();
}
cudaError_t launch_item_cost(const int2* ranges, int n_ranges, int n_items, const TaskDesc* tasks,
                             const LensDesc* lenses, const GridDesc* grids, float R, int2* items, unsigned* band,
                             cudaStream_t st) {
  if (n_items > 0)
    k_item_cost<<<(n_items + 31) / 32, 256, 0, st>>>(ranges, n_ranges, n_items, tasks, lenses, grids, R, items, band);
  return cudaGetLastError();
}
int item_order_max() { return kOrderMax; }
cudaError_t launch_item_order(const int2* items, const unsigned* band, int n, int2* out, cudaStream_t st) {
  k_item_order<<<1, 1024, 0, st>>>(items, band, n, out);
  return cudaGetLastError();
}
cudaError_t launch_iota32(int* v, int n, cudaStream_t st) {
  k_iota32<<<(n + 255) / 256, 256, 0, st>>>(v, n);
  return cudaGetLastError();
}
cudaError_t launch_permute_items(const int2* items, const int* order, int n, int index, int count, int2* out,
                                 cudaStream_t st) {
  if (n > 0) k_permute_items<<<(n + 255) / 256, 256, 0, st>>>(items, order, n, index, count, out);
  return cudaGetLastError();
}
cudaError_t launch_ffma_peak(float* out, int blocks, int threads, int iters, cudaStream_t st) {
  k_ffma_peak<<<blocks, threads, 0, st>>>(out, iters, 0.999999f, 1e-7f);
  return cudaGetLastError();
}
cudaError_t launch_dfma_peak(double* out, int blocks, int threads, int iters, cudaStream_t st) {
  k_dfma_peak<<<blocks, threads, 0, st>>>(out, iters, 0.999999999, 1e-13);
  return cudaGetLastError();
}
cudaError_t launch_patch_reduce(const double* item_sums, int item_base, int split, const int* patch_groups, int n_patch,
                                int nb, double* patch_sums, cudaStream_t st) {
  if (n_patch > 0)
    k_patch_reduce<<<dim3(n_patch, (kQ * nb + 31) / 32), 32 * kReduceWarps, 0, st>>>(item_sums, item_base, split, patch_groups,
                                                                                    n_patch, nb, patch_sums);
  return cudaGetLastError();
}
cudaError_t launch_lens_outputs(const double* acc, int split, const float4* rec, const int* perm, int n_valid, int nb,
                                float* xi_E, float* xi_B, float* K_m, float* w_m, float* marks_weight,
                                double* lens_sums, double* lens_raw, cudaStream_t st) {
  if (n_valid > 0)
    k_lens_outputs<<<(n_valid + 31) / 32, 128, 0, st>>>(acc, split, rec, perm, n_valid, nb, xi_E, xi_B, K_m, w_m,
                                                          marks_weight, lens_sums, lens_raw);
  return cudaGetLastError();
}

// CUB radix sorts (temp storage supplied by the caller).
cudaError_t sort_pairs_u32(void* tmp, size_t& tmp_bytes, const unsigned* kin, unsigned* kout, const int* vin,
                           int* vout, int n, int end_bit, cudaStream_t st) {
  return cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, kin, kout, vin, vout, n, 0, end_bit, st);
}
cudaError_t sort_pairs_u64(void* tmp, size_t& tmp_bytes, const unsigned long long* kin, unsigned long long* kout,
                           const int* vin, int* vout, int n, int end_bit, cudaStream_t st) {
  return cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, kin, kout, vin, vout, n, 0, end_bit, st);
}
cudaError_t sort_bands_desc(void* tmp, size_t& tmp_bytes, const unsigned* kin, unsigned* kout, const int* vin,
                            int* vout, int n, cudaStream_t st) {
  static_assert(kCostBands == 512, "nine key bits");
  return cub::DeviceRadixSort::SortPairsDescending(tmp, tmp_bytes, kin, kout, vin, vout, n, 0, 9, st);
}

}  // namespace tpcf
