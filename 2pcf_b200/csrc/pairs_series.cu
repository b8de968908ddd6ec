// pairs_series.cu -- the planar pair kernel for calls without per-lens outputs
// (the totals and per-patch sums of tangential_shear_tpcf, src/tpcf.f90:261-363,
// and scalar_kappa_tpcf, src/tpcf.f90:451-535).
//
// Work items, queue, cell rows and the per-warp tile ring are those of k_pairs
// (pairs.cu).  What differs is what a warp does with a 32-source sub-chunk.
// Most (lens, sub-chunk) combinations lie in one bin and far apart (the
// sub-chunk's radius is a few percent of the distance); their 32 pairs need not
// be formed one by one:
//
//   far     the sums over the sub-chunk's sources come from a series about its
//           centre.  With Z = centre - lens (complex), delta_j = source -
//           centre, t = s / Z (s = the sub-chunk's radius, |t| <= kFarRatio)
//           and A = p + i q (p = -e1 w, q = -e2 w):
//             sum A conj(z)/z  = conj(Z)/Z sum_k M_k (-t)^k + t sum_k N_k (-t)^k,
//             M_k = sum A (delta/s)^k,  N_k = sum A conj(delta/s) (delta/s)^k
//           (conj(z)/z = exp(-2 i phi), so the real and imaginary parts are the
//           g_t and g_x terms of src/tpcf.f90:343-344), to order 6; and with
//           |1 + tau| = sum_ab c_a c_b tau^a conj(tau)^b, c = binomial(1/2, .),
//             sum w |z| = |Z| sum_ab c_a c_b W_ab t^a conj(t)^b,
//             W_ab = sum w (delta/s)^a conj(delta/s)^b,
//           to order 5.  The moments are formed once per catalogue in FP64
//           (k_src_series) and held in FP32.
//   direct  everything else: the lenses of the group that need it are listed,
//           lane = source, two lenses per iteration of packed FP32 arithmetic.
//           A lens whose pairs span one or two bin edges is summed on both
//           sides of each edge by compares with the squared edge; a pair inside
//           the guard band of an edge is decided by the canonical FP64 rule, so
//           n_pairs is that rule's.  Since a lane keeps its source, p, q, w and
//           K multiply once per list and not once per pair.
//
// Truncation at |t| = kFarRatio = 0.08, the worst of any 32 sources: 2 |t|^7 / (1 - |t|)
// = 4.6e-8 of sum |A| and 2e-8 of sum w |z| (formulas evaluated in FP64: two knots at
// opposite ends of the sub-chunk reach 4.2e-8 and 1.6e-8, random sub-chunks 9e-9 and
// 2.5e-9), below the FP32 rounding of a directly formed term (6e-8).  One order less
// each leaves 5.2e-7 and 2.8e-7 for the two knots.

#include <cstdio>

#include "pair_hist.cuh"
#include "pair_tiles.cuh"
#include "tpcf_device.cuh"
#include "tpcf_internal.cuh"
#include "tpcf_kernels.h"

namespace tpcf {

namespace {

// At least 14 warps per SM, at most 144 registers: the tomography call (25 tasks,
// 1.24e12 pairs) took 869 ms against 952 ms with 12 warps at 168 registers (874 now,
// with one more order in both series); where the compiler needs 128 or less, as without
// z cut and calibration, 16 warps fit and gain nothing more.
constexpr int kSeriesThreads = 64, kSeriesBlocks = 7;
constexpr float kFarRatio = 0.08f;
constexpr float kNullPos = 1.0e18f;  // coordinate of a source that takes no part: every term stays finite
constexpr float kMinNormal = 1.17549435e-38f;
constexpr int kRows = 32;            // cell rows whose spans a warp holds at once (one per lane)
constexpr int kTch = 3;              // sub-chunks per tile
// Lenses per lane (a work item holds 64 lenses): the per-sub-chunk work and the
// lists are shared by twice as many pairs and the two lenses' chains overlap
// (32 lenses: 1097 ms for the tomography, 64: 952 ms; 128: 905 ms, but 9% slower on
// sparse lenses).
constexpr int kLpl = 2;
constexpr int kNbuf = 2;             // tiles in flight per warp
constexpr int kOrder = 6;            // M_0 .. M_6, N_0 .. N_5
// Guard band around a squared edge, relative: FP32 d2 is within 3e-7 of its
// exact value and the FP32 edge within 6e-8.
constexpr float kEdgeBand = 1.0e-6f;
// Lists whose one-edge sums a warp keeps in registers before it adds them to its FP64
// sums: FP32 sums of at most 8 x 64 pairs per lane (a list holds up to 64 lenses), in
// runs of 32 and 8, then a tree over the 32 lanes.
constexpr int kKeep = 8;

// One sub-chunk record: {cx cy s (s / kFarRatio)^2}{P Q W K sums}{zmin zmax 0 0},
// shear: kOrder + 1 times {M_re N_re M_im N_im}, then the distance series
// {W00 W11/4 W22/64 0}{W10, -W21/8}{-W20/4, W31/16}{W30/8, -5/128 W41}
// {-5/64 W40, 7/128 W50}{-W32/64, 0}, then the fields of the 32 sources, each [32]:
// x y p q w (K) (z).
struct RecShape {
  int g, d, src, fields, floats;
};
__host__ __device__ constexpr RecShape rec_shape(int mode, bool has_m, bool has_z) {
  RecShape r{};
  r.g = 12;
  r.d = r.g + (mode == 0 ? 4 * (kOrder + 1) : 0);
  r.src = r.d + 24;
  r.fields = 5 + (has_m ? 1 : 0) + (has_z ? 1 : 0);
  r.floats = r.src + kChunk * r.fields;
  return r;
}

// Shared memory of one warp; nt = bins of the far sums.
struct WarpSmem {
  size_t ring, hist, wsum, lxy, lf, lz, mbar, total;
};
__host__ __device__ inline WarpSmem warp_smem(int nb, int nt, int qa, int rec_floats) {
  WarpSmem s{};
  size_t o = 0;
  s.ring = o; o += (size_t)kNbuf * kTch * rec_floats * sizeof(float);
  s.hist = o; o += (size_t)nt * qa * 32 * sizeof(float);
  s.wsum = o; o += ((size_t)kQ * nb + 2) * sizeof(double);  // then the scales of the lens factors
  o = (o + 15) / 16 * 16;
  s.lxy = o;  o += 16 * kLpl * sizeof(float4);
  s.lf = o;   o += 16 * kLpl * sizeof(float4);
  s.lz = o;   o += 16 * kLpl * sizeof(float2);
  s.mbar = o; o += kNbuf * sizeof(uint64_t);
  s.total = (o + 15) / 16 * 16;
  return s;
}
__host__ __device__ inline size_t edge_smem(int nb) { return ((size_t)(nb + 1) * 12 + 15) / 16 * 16; }

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Lowest and highest bin (clamped to [-1, nb]) of the distances dc - rad ..
// dc + rad; false when none is in range.
template <bool LOGB>
__device__ __forceinline__ bool bin_range(float dc, float rad, const BinCtx& C, int& b0, int& b1) {
  const float lo = fmaxf(dc - rad, 0.f), hi = dc + rad;
  if (LOGB) {
    b0 = __float2int_rd(fmaf(lg2_ftz(lo), 2.f * C.A, C.B - C.eps));
    b1 = __float2int_rd(fmaf(lg2_ftz(hi), 2.f * C.A, C.B + C.eps));
  } else {
    b0 = edge_index_f32(lo * lo * (1.f - C.eps), C.e2f, C.nb);
    b1 = edge_index_f32(hi * hi * (1.f + C.eps), C.e2f, C.nb);
  }
  const bool in = b1 >= 0 && b0 < C.nb;
  b0 = max(b0, -1);
  b1 = min(b1, C.nb);
  return in;
}

// Whether the pair lies at or above edge e by the canonical FP64 rule (the
// last edge belongs to the last bin).
__device__ __noinline__ bool above_edge(float lx, float ly, float sx, float sy, const double* e2, int e, int nb) {
  const double dx = __dsub_rn((double)lx, (double)sx);
  const double dy = __dsub_rn((double)ly, (double)sy);
  const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
  return e == nb ? d2 > e2[e] : d2 >= e2[e];
}

// Biased exponent of v, 0 for an infinity or NaN.
__device__ __forceinline__ unsigned exponent_of(double v) {
  const unsigned e = ((unsigned)__double2hiint(v) >> 20) & 0x7ffu;
  return e == 0x7ffu ? 0u : e;
}
// The power of two with biased exponent e (1 .. 2046).
__device__ __forceinline__ double pow2_biased(unsigned e) { return __hiloint2double((int)(e << 20), 0); }

struct LaneSrc {
  float x, y, p, q, w, K, z;
  bool ok;
};

// Terms of this lane's source with two lenses (packed): Pn = dy^2 - dx^2,
// qq = dx dy, rv = vw / d^2 (scalar fields: vw), wv = w, zero where the z cut
// drops the pair.
struct Terms {
  float2 d2, d, Pn, qq, rv, wv, one;
};
template <int MODE, bool HAS_Z, bool LOGB>
__device__ __forceinline__ Terms pair_terms(const float4 a, const float4 f, const float2 lz, const LaneSrc& S,
                                            float tiny) {
  Terms T;
  const float2 dx = add2(dup2(S.x), lo2(a));
  const float2 dy = add2(dup2(S.y), hi2(a));
  const float2 dx2 = mul2(dx, dx);
  T.d2 = fma2(dy, dy, dx2);
  float2 r;
  if (LOGB) {
    // d2 = 0 is below the first edge; the offset (1e-9 of that edge) only keeps its
    // terms finite
    const float2 e2 = add2(T.d2, dup2(tiny));
    const float2 rs = make_float2(rsqrt_ftz(e2.x), rsqrt_ftz(e2.y));
    T.d = mul2(T.d2, rs);
    r = mul2(rs, rs);
  } else {
    // one Newton step each on sqrt and 1/d^2 (within 1 ulp); d2 = 0 gives
    // d = 0 and r = 0 (the caller sees to its 0/0)
    const float2 rs = make_float2(T.d2.x >= kMinNormal ? rsqrt_ftz(T.d2.x) : 0.f,
                                  T.d2.y >= kMinNormal ? rsqrt_ftz(T.d2.y) : 0.f);
    const float2 dd = mul2(T.d2, rs);
    T.d = fma2(fma2(make_float2(-dd.x, -dd.y), dd, T.d2), mul2(rs, dup2(0.5f)), dd);
    const float2 r0 = mul2(rs, rs);
    r = fma2(r0, fma2(make_float2(-T.d2.x, -T.d2.y), r0, dup2(1.f)), r0);
  }
  T.rv = MODE == 0 ? mul2(r, lo2(f)) : lo2(f);
  T.wv = hi2(f);
  T.one = dup2(1.f);
  if (HAS_Z) {
    T.one = make_float2(lz.x <= S.z ? 1.f : 0.f, lz.y <= S.z ? 1.f : 0.f);  // src/tpcf.f90:322
    T.rv = mul2(T.rv, T.one);
    T.wv = mul2(T.wv, T.one);
  }
  if (MODE == 0) {
    T.Pn = fma2(dx2, dup2(-2.f), T.d2);
    T.qq = mul2(dx, dy);
  } else {
    T.Pn = T.qq = dup2(0.f);
  }
  return T;
}

struct Acc {
  float2 c, s, w, d, n;
};
template <int MODE>
__device__ __forceinline__ void acc_add(Acc& A, const Terms& T, float2 r, float2 w) {
  if (MODE == 0) {
    A.c = fma2(r, T.Pn, A.c);
    A.s = fma2(r, T.qq, A.s);
  } else {
    A.c = add2(A.c, r);
  }
  A.w = add2(A.w, w);
  A.d = fma2(T.d, w, A.d);
}

// Sums of this lane's source with the cnt listed lenses, apart for the NE + 1
// sides of the NE edges e0, e0 + 1: v[k] belongs to bin e0 - 1 + k (masks of
// one compare per edge; every term is added on its own side only).
// lxy: {-x0 -x1 -y0 -y1}, lf: {vw0 vw1 w0 w1} of two lenses per entry; an odd
// list ends in a copy of its last lens with zero factors.  `zero` tells
// whether a counted pair has d = 0 (other than log spacing).
template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB, int NE>
__device__ __forceinline__ void direct_sums(const float4* lxy, const float4* lf, const float2* lz, int cnt,
                                            const LaneSrc& S, int e0, const BinCtx& C, float (&v)[NE + 1][6],
                                            bool& zero) {
  Acc A[NE + 1];
  float E[NE > 0 ? NE : 1], last[NE > 0 ? NE : 1], close = 3.0e38f, dmin = 3.0e38f, last_one = 1.f;
#pragma unroll
  for (int k = 0; k <= NE; ++k) A[k].c = A[k].s = A[k].w = A[k].d = A[k].n = dup2(0.f);
#pragma unroll
  for (int k = 0; k < NE; ++k) E[k] = C.e2f[e0 + k], last[k] = 0.f;
  const int np = (cnt + 1) >> 1;
#pragma unroll(NE < 2 ? 4 : 1)
  for (int i = 0; i < np; ++i) {
    const Terms T = pair_terms<MODE, HAS_Z, LOGB>(lxy[i], lf[i], HAS_Z ? lz[i] : make_float2(0.f, 0.f), S, C.tiny);
    if (HAS_Z) A[0].n = add2(A[0].n, T.one), last_one = T.one.x;
    if (!LOGB) dmin = fminf(dmin, fminf(T.one.x > 0.f ? T.d2.x : 1.f, T.one.y > 0.f ? T.d2.y : 1.f));
    float2 ra = T.rv, wa = T.wv;  // at or above the edge below side k
#pragma unroll
    for (int k = 0; k <= NE; ++k) {
      float2 rk = ra, wk = wa;
      if (k < NE) {
        const float2 t = add2(T.d2, dup2(-E[k]));
        close = fminf(close, fminf(fabsf(t.x), fabsf(t.y)));
        float2 m = make_float2(t.x >= 0.f ? 1.f : 0.f, t.y >= 0.f ? 1.f : 0.f);
        ra = mul2(T.rv, m);
        wa = mul2(T.wv, m);
        rk = fma2(ra, dup2(-1.f), rk);  // exactly 0 or the value
        wk = fma2(wa, dup2(-1.f), wk);
        if (HAS_Z) m = mul2(m, T.one);
        last[k] = m.x;
        A[k + 1].n = add2(A[k + 1].n, m);
      }
      acc_add<MODE>(A[k], T, rk, wk);
    }
  }
  if (NE > 0 && close <= E[NE > 0 ? NE - 1 : 0] * C.eps_rel) {
    // a pair inside the guard band: where the canonical FP64 rule puts it on
    // the other side of an edge than its FP32 distance, move its terms
#pragma unroll 1
    for (int i = 0; i < np; ++i) {
      const float4 a = lxy[i];
      const Terms T = pair_terms<MODE, HAS_Z, LOGB>(a, lf[i], HAS_Z ? lz[i] : make_float2(0.f, 0.f), S, C.tiny);
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const float2 t = add2(T.d2, dup2(-E[k]));
        const float band = E[k] * C.eps_rel;
        float2 m = dup2(0.f);
        if (fabsf(t.x) <= band)
          m.x = (above_edge(-a.x, -a.z, S.x, S.y, C.e2s, e0 + k, C.nb) ? 1.f : 0.f) - (t.x >= 0.f ? 1.f : 0.f);
        if (fabsf(t.y) <= band)
          m.y = (above_edge(-a.y, -a.w, S.x, S.y, C.e2s, e0 + k, C.nb) ? 1.f : 0.f) - (t.y >= 0.f ? 1.f : 0.f);
        const float2 rm = mul2(T.rv, m), wm = mul2(T.wv, m);
        acc_add<MODE>(A[k + 1], T, rm, wm);
        acc_add<MODE>(A[k], T, mul2(rm, dup2(-1.f)), mul2(wm, dup2(-1.f)));
        m = mul2(T.one, m);
        A[k + 1].n = add2(A[k + 1].n, m);
        if (i == np - 1) last[k] += m.x;
      }
    }
  }
  zero = !LOGB && dmin == 0.f;
  // (__fmul_rn: products that the callers' additions must not fuse with, so that every
  // variant of the kernel rounds alike)
  // A[k].n counts the pairs at or above edge k - 1 (k = 0: all)
  float n[NE + 2];
#pragma unroll
  for (int k = 0; k <= NE; ++k) {
    // the pad of an odd list was counted on its last lens's side
    n[k] = (k == 0 && !HAS_Z) ? (float)cnt : sum2(A[k].n);
    if ((k > 0 || HAS_Z) && (cnt & 1)) n[k] -= k == 0 ? last_one : last[k > 0 ? k - 1 : 0];
  }
  n[NE + 1] = 0.f;
#pragma unroll
  for (int k = 0; k <= NE; ++k) {
    const float c = sum2(A[k].c), w = sum2(A[k].w);
    if (MODE == 0) {
      const float sn = -2.f * sum2(A[k].s);  // c and sn carry the sign of Pn
      v[k][QGT] = -fmaf(S.p, c, S.q * sn);
      v[k][QGX] = -fmaf(S.q, c, -(S.p * sn));
    } else {
      v[k][QGT] = __fmul_rn(S.p, c);
      v[k][QGX] = __fmul_rn(S.q, c);
    }
    v[k][QW] = __fmul_rn(S.w, w);
    v[k][QDW] = __fmul_rn(S.w, sum2(A[k].d));
    v[k][QN] = S.ok ? n[k] - n[k + 1] : 0.f;
    v[k][QK] = (MODE == 0 && HAS_M) ? __fmul_rn(S.K, w) : 0.f;
  }
}

// Adds the warp's sum of v (one row per lane) to the warp's FP64 sums of `bin`.
__device__ __forceinline__ void add_bin(const float (&v)[6], int bin, int nb, double* wsum, int lane) {
  if (bin < 0 || bin >= nb) return;
  const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
  float k0 = h16 ? v[4] : v[0], k1 = h16 ? v[5] : v[1], k2 = h16 ? 0.f : v[2], k3 = h16 ? 0.f : v[3];
  k0 += __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[4], 16);
  k1 += __shfl_xor_sync(0xffffffffu, h16 ? v[1] : v[5], 16);
  k2 += __shfl_xor_sync(0xffffffffu, h16 ? v[2] : 0.f, 16);
  k3 += __shfl_xor_sync(0xffffffffu, h16 ? v[3] : 0.f, 16);
  float m0 = h8 ? k2 : k0, m1 = h8 ? k3 : k1;
  m0 += __shfl_xor_sync(0xffffffffu, h8 ? k0 : k2, 8);
  m1 += __shfl_xor_sync(0xffffffffu, h8 ? k1 : k3, 8);
  float s = h4 ? m1 : m0;
  s += __shfl_xor_sync(0xffffffffu, h4 ? m0 : m1, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  const int q = (h16 ? 4 : 0) + (h8 ? 2 : 0) + (h4 ? 1 : 0);
  if ((lane & 3) == 0 && q < kQ) wsum[q * nb + bin] += (double)s;
}

}  // namespace

#ifdef TPCF_MODE_STATS
// Diagnostic build only: (lens, sub-chunk) combinations [out of range, far, direct with
// 0, 1, 2, more edges], lists, lenses listed.
__device__ unsigned long long g_series_stats[8];
extern "C" int tpcf_debug_series_stats(unsigned long long* out) {
  return (int)cudaMemcpyFromSymbol(out, g_series_stats, sizeof(g_series_stats));
}
#endif

// Far sums of the warp's 32 columns into its FP64 sums; the columns are cleared.
template <int QA>
__device__ __forceinline__ void fold_far(float* hist, double* wsum, int nb, int tb, int lane) {
  __syncwarp();
  const int nt = nb - tb;
  for (int e = lane; e < nt * QA; e += 32) {
    const float* row = hist + e * 32;
    double s = 0.0;
#pragma unroll 8
    for (int l = 0; l < 32; ++l) s += (double)row[(l + lane) & 31];
    const int b = e / QA, q = e - b * QA;
    wsum[q * nb + tb + b] += s;
  }
  __syncwarp();
  for (int e = 0; e < nt * QA; ++e) hist[e * 32 + lane] = 0.f;
}

template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB>
__global__ void __launch_bounds__(kSeriesThreads, kSeriesBlocks) k_pairs_series(const PairParams P) {
  constexpr int QA = (MODE == 0 && HAS_M) ? 6 : 5;
  constexpr RecShape R = rec_shape(MODE, HAS_M, HAS_Z);
  const int nb = P.nb, tb = P.far_bin;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  extern __shared__ __align__(128) unsigned char smem[];
  double* e2s = reinterpret_cast<double*>(smem);
  float* e2f = reinterpret_cast<float*>(e2s + nb + 1);
  const WarpSmem W = warp_smem(nb, nb - tb, QA, R.floats);
  unsigned char* wb = smem + edge_smem(nb) + (size_t)warp * W.total;
  float* ring = reinterpret_cast<float*>(wb + W.ring);
  float* hist = reinterpret_cast<float*>(wb + W.hist);
  double* wsum = reinterpret_cast<double*>(wb + W.wsum);
  float4* lxy = reinterpret_cast<float4*>(wb + W.lxy);
  float4* lf = reinterpret_cast<float4*>(wb + W.lf);
  float2* lzs = reinterpret_cast<float2*>(wb + W.lz);
  uint64_t* full = reinterpret_cast<uint64_t*>(wb + W.mbar);

  if (lane == 0) {
    for (int b = 0; b < kNbuf; ++b) mbar_init(&full[b], 1);
    mbar_fence_init();
  }
  for (int i = tid; i <= nb; i += blockDim.x) {
    e2s[i] = P.e2[i];
    e2f[i] = P.e2f[i];
  }
#ifdef TPCF_MODE_STATS
  __shared__ unsigned long long sh_stats[8];
  if (tid < 8) sh_stats[tid] = 0ull;
#endif
  for (int e = 0; e < (nb - tb) * QA; ++e) hist[e * 32 + lane] = 0.f;
  __syncthreads();
  BinCtx C;
  C.A = P.binA; C.B = P.binB; C.eps = P.eps; C.one_m_eps = 1.f - P.eps;
  C.nb = nb; C.e2s = e2s; C.e2f = e2f;
  C.eps_rel = kEdgeBand;
  C.lo_g = e2f[0] * (1.f - P.eps);
  C.hi_g = e2f[nb] * (1.f + P.eps);
  C.tiny = e2f[0] * 1e-9f;

  const uint32_t wait_limit = P.wait_limit ? P.wait_limit : kWaitPolls;
  int ring_t = 0;        // ring index of the next tile this warp consumes
  int issued_end = 0;    // ring index one past the last tile this warp issued
  bool aborted = false;  // a bounded wait ran out: consume and issue nothing more

  while (!aborted) {
    int item = 0;
    if (lane == 0) item = atomicAdd(P.queue_head, 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= P.n_items) break;
    const int2 it = P.items[item];
    const TaskDesc T = P.tasks[it.x];
    const LensDesc LD = P.lenses[T.lens_cat];
    const GridDesc G = P.grids[T.src_cat];
    const int g = it.y / T.split, part_i = it.y - g * T.split;
    const int gs = LD.group_start[g], nl = LD.group_start[g + 1] - gs;
    // lenses lane and lane + 32 of the group.  Their factors val w (formed in FP64)
    // and w enter the FP32 terms, so the group's are scaled by a power of two to at
    // most 2 and the item's FP64 sums scaled back: products of very small or very
    // large lens and source weights stay in range.
    float lx[kLpl], ly[kLpl], lz[kLpl], vw[kLpl], w[kLpl];
    double fv[kLpl], fw[kLpl];
    unsigned xv = 0, xw = 0;
    bool act[kLpl];
#pragma unroll
    for (int l = 0; l < kLpl; ++l) {
      const int i = lane + 32 * l;
      act[l] = i < nl;
      lx[l] = ly[l] = lz[l] = 0.f;
      fv[l] = fw[l] = 0.0;
      if (act[l]) {
        const float4 r = LD.rec[gs + i];
        lx[l] = r.x;
        ly[l] = r.y;
        fv[l] = (double)r.z * (double)r.w;
        fw[l] = (double)r.w;
        if (HAS_Z) lz[l] = LD.z[gs + i];
      }
      xv = max(xv, exponent_of(fv[l]));
      xw = max(xw, exponent_of(fw[l]));
    }
    xv = __reduce_max_sync(0xffffffffu, xv);
    xw = __reduce_max_sync(0xffffffffu, xw);
    xv = xv ? xv : 1023u;
    xw = xw ? xw : 1023u;
#pragma unroll
    for (int l = 0; l < kLpl; ++l) {
      vw[l] = (float)(fv[l] * pow2_biased(2046u - xv));
      w[l] = (float)(fw[l] * pow2_biased(2046u - xw));
    }
    if (lane == 0) {
      wsum[kQ * nb] = pow2_biased(xv);
      wsum[kQ * nb + 1] = pow2_biased(xw);
    }
    for (int e = lane; e < kQ * nb; e += 32) wsum[e] = 0.0;
    __syncwarp();
    int since_flush = 0;
    const float4 box = LD.group_box[g];
    int cy0, cy1;
    row_range(G, box, P.R, T.margin, cy0, cy1);

    // sums of the passes at one edge, kept in registers: bins keep_e - 1, keep_e
    float keep[2][6];
    int keep_e = -1, keep_n = 0;
#pragma unroll
    for (int q = 0; q < 6; ++q) keep[0][q] = keep[1][q] = 0.f;
    auto flush_keep = [&]() {
      if (keep_n == 0) return;
      add_bin(keep[0], keep_e - 1, nb, wsum, lane);
      add_bin(keep[1], keep_e, nb, wsum, lane);
#pragma unroll
      for (int q = 0; q < 6; ++q) keep[0][q] = keep[1][q] = 0.f;
      keep_n = 0;
    };

    for (int c0 = cy0 + part_i; c0 <= cy1 && !aborted; c0 += kRows * T.split) {
      int s0 = 0, s1 = 0;
      const int row = c0 + lane * T.split;
      if (row <= cy1) {
        const int2 sp = row_span(G, box, P.R, T.margin, row);
        s0 = sp.x;
        s1 = sp.y > sp.x ? sp.y : sp.x;
      }
      const int ntr = tiles_of_span<kTch>(s0, s1);
      int incl = ntr;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const int ntiles = __shfl_sync(0xffffffffu, incl, 31);
      // Ring: the tile with ring index t lives in buffer t % kNbuf and completes
      // phase (t / kNbuf) & 1 of that buffer's barrier.
      auto issue = [&](int k) {
        const TileGeom tg = tile_of<kTch>(k, incl, ntr, s0, s1);
        const int t = ring_t + k;
        issued_end = t + 1;
        if (t + 1 == P.debug_skip_tile) return;  // fault injection (tests): this tile never lands
        if (lane == 0) {
          const int b = t % kNbuf;
          const uint32_t bytes = (uint32_t)tg.n * R.floats * (uint32_t)sizeof(float);
          mbar_arrive_tx(&full[b], bytes);
          bulk_g2s(ring + (size_t)b * kTch * R.floats, G.series + (size_t)tg.c0 * R.floats, bytes, &full[b]);
        }
      };
      for (int k = 0; k < kNbuf && k < ntiles; ++k) issue(k);
      for (int k = 0; k < ntiles; ++k) {
        const int t = ring_t + k;
        const int b = t % kNbuf;
        const TileGeom tg = tile_of<kTch>(k, incl, ntr, s0, s1);
        const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[b], (uint32_t)(t / kNbuf) & 1u, wait_limit));
        if (!ok) {  // stop: drain this warp's copies in flight below, report the timeout
          aborted = true;
          ring_t = t;
          break;
        }
#pragma unroll 1
        for (int j = 0; j < tg.n; ++j) {
          const int lo = j == 0 ? tg.lo0 : 0;
          const int hi = j == tg.n - 1 ? tg.hiL : kChunk;
          const bool whole = lo == 0 && hi == kChunk;
          const float* __restrict__ rec = ring + (size_t)(b * kTch + j) * R.floats;
          const float4 cen = ld4(rec);
          float Zx[kLpl], Zy[kLpl], Z2[kLpl], rs[kLpl], dc[kLpl];
          int b0[kLpl], b1[kLpl];
          bool in[kLpl], far[kLpl], any_in = false, any_far = false, any_dir = false;
          float2 zr = make_float2(0.f, 0.f);
          if (HAS_Z) zr = *reinterpret_cast<const float2*>(rec + 8);
#pragma unroll
          for (int l = 0; l < kLpl; ++l) {
            Zx[l] = cen.x - lx[l];
            Zy[l] = cen.y - ly[l];
            Z2[l] = fmaf(Zy[l], Zy[l], Zx[l] * Zx[l]);
            rs[l] = rsqrt_ftz(fmaxf(Z2[l], kMinNormal));
            dc[l] = __fmul_rn(Z2[l], rs[l]);
            in[l] = bin_range<LOGB>(dc[l], cen.z, C, b0[l], b1[l]) && act[l];
            bool zall = true;
            if (HAS_Z) {
              in[l] = in[l] && lz[l] <= zr.y;  // else every source is in front of the lens
              zall = lz[l] <= zr.x;
            }
            far[l] = in[l] && b0[l] == b1[l] && b0[l] >= tb && whole && zall && Z2[l] >= cen.w;
            any_in = any_in || in[l];
            any_far = any_far || far[l];
            any_dir = any_dir || (in[l] && !far[l]);
          }
#ifdef TPCF_MODE_STATS
#pragma unroll
          for (int l = 0; l < kLpl; ++l) {
            const int cls = !act[l] ? -1 : !in[l] ? 0 : far[l] ? 1 : 2 + min(b1[l] - b0[l], 3);
            for (int q = 0; q < 6; ++q) {
              const unsigned n = __popc(__ballot_sync(0xffffffffu, cls == q));
              if (lane == 0 && n) atomicAdd(&sh_stats[q], (unsigned long long)n);
            }
          }
#endif
          if (!__any_sync(0xffffffffu, any_in)) continue;
          if (__any_sync(0xffffffffu, any_far)) {
            const float4 sums = ld4(rec + 4);
            float r[kLpl], tx[kLpl], ty[kLpl], gt[kLpl], gx[kLpl], dw[kLpl];
#pragma unroll
            for (int l = 0; l < kLpl; ++l) {
              r[l] = rs[l] * rs[l];
              const float sr = cen.z * r[l];
              tx[l] = sr * Zx[l];
              ty[l] = -(sr * Zy[l]);
            }
            if (MODE == 0) {
              // Horner in -t for M (x halves) and N (y halves) at once
              float4 m = ld4(rec + R.g + 4 * kOrder);
              float2 re[kLpl], im[kLpl];
#pragma unroll
              for (int l = 0; l < kLpl; ++l) re[l] = lo2(m), im[l] = hi2(m);
#pragma unroll
              for (int o = kOrder - 1; o >= 0; --o) {
                m = ld4(rec + R.g + 4 * o);
#pragma unroll
                for (int l = 0; l < kLpl; ++l) {
                  const float2 nre = fma2(dup2(-tx[l]), re[l], fma2(dup2(ty[l]), im[l], lo2(m)));
                  im[l] = fma2(dup2(-tx[l]), im[l], fma2(dup2(-ty[l]), re[l], hi2(m)));
                  re[l] = nre;
                }
              }
#pragma unroll
              for (int l = 0; l < kLpl; ++l) {
                const float c2 = fmaf(-Zy[l], Zy[l], Zx[l] * Zx[l]) * r[l];
                const float zz = __fmul_rn(Zx[l], Zy[l]);
                const float s2 = (zz + zz) * r[l];
                gt[l] = fmaf(c2, re[l].x, fmaf(s2, im[l].x, fmaf(tx[l], re[l].y, -(ty[l] * im[l].y))));
                gx[l] = fmaf(c2, im[l].x, fmaf(-s2, re[l].x, fmaf(tx[l], im[l].y, ty[l] * re[l].y)));
              }
            } else {
#pragma unroll
              for (int l = 0; l < kLpl; ++l) gt[l] = sums.x, gx[l] = sums.y;
            }
            const float4 q0 = ld4(rec + R.d), q1 = ld4(rec + R.d + 4), q2 = ld4(rec + R.d + 8), q3 = ld4(rec + R.d + 12),
                         q4 = ld4(rec + R.d + 16);
            const float2 q5 = *reinterpret_cast<const float2*>(rec + R.d + 20);
#pragma unroll
            for (int l = 0; l < kLpl; ++l) {
              const float tt = fmaf(tx[l], tx[l], ty[l] * ty[l]);
              const float2 tt2 = dup2(tt);
              // (acc.re, acc.im) <- c + t acc
              auto step = [&](float2 a, float2 c) {
                return fma2(dup2(tx[l]), a, fma2(make_float2(-ty[l], ty[l]), make_float2(a.y, a.x), c));
              };
              float2 a = step(hi2(q4), lo2(q4));
              a = step(a, fma2(tt2, hi2(q3), lo2(q3)));
              a = step(a, fma2(tt2, hi2(q2), lo2(q2)));
              a = step(a, fma2(tt2, fma2(tt2, q5, hi2(q1)), lo2(q1)));
              const float p0 = fmaf(tt, fmaf(tt, q0.z, q0.y), q0.x);
              dw[l] = dc[l] * (p0 + fmaf(tx[l], a.x, -(ty[l] * a.y)));
            }
#pragma unroll
            for (int l = 0; l < kLpl; ++l) {
              if (far[l]) {
                float* h = hist + (b0[l] - tb) * (QA * 32) + lane;
                h[QGT * 32] = fmaf(gt[l], vw[l], h[QGT * 32]);
                h[QGX * 32] = fmaf(gx[l], vw[l], h[QGX * 32]);
                h[QW * 32] = fmaf(sums.z, w[l], h[QW * 32]);
                h[QDW * 32] = fmaf(dw[l], w[l], h[QDW * 32]);
                h[QN * 32] += (float)kChunk;
                if (MODE == 0 && HAS_M) h[QK * 32] = fmaf(sums.w, w[l], h[QK * 32]);
              }
            }
          }
          if (!__any_sync(0xffffffffu, any_dir)) continue;
          // direct: the lens's pairs span the bins db .. dt; lenses with the same
          // bins are listed together.  Up to two edges are summed in one pass; a
          // lens with more takes the two lowest bins first, then one bin per pass
          // (from its lower edge on), the last two together.
          LaneSrc S;
          {
            const float* f = rec + R.src + lane;
            S.x = f[0];
            S.y = f[32];
            S.p = f[64];
            S.q = f[96];
            S.w = f[128];
            S.K = (MODE == 0 && HAS_M) ? f[160] : 0.f;
            S.z = HAS_Z ? f[32 * (R.fields - 1)] : 0.f;
            S.ok = true;
            if (!whole) {
              S.ok = lane >= lo && lane < hi;
              if (!S.ok) {
                S.x = S.y = kNullPos;
                S.p = S.q = S.w = S.K = 0.f;
              }
            }
          }
          int key[kLpl];  // (lowest bin not summed yet + 1) * 8 + pass type; -1: nothing left
#pragma unroll
          for (int l = 0; l < kLpl; ++l)
            key[l] = in[l] && !far[l] ? (b0[l] + 1) * 8 + min(b1[l] - b0[l], 3) : -1;
          for (;;) {
            int kmax = key[0];
#pragma unroll
            for (int l = 1; l < kLpl; ++l) kmax = max(kmax, key[l]);
            const int kkey = (int)__reduce_max_sync(0xffffffffu, kmax);
            if (kkey < 0) break;
            unsigned mem[kLpl];  // the listed lenses
            int cnt = 0;
#pragma unroll
            for (int l = 0; l < kLpl; ++l) {
              mem[l] = __ballot_sync(0xffffffffu, key[l] == kkey);
              cnt += __popc(mem[l]);
            }
            const int kb = (kkey >> 3) - 1, kt = kkey & 7;
#ifdef TPCF_MODE_STATS
            if (lane == 0) {
              atomicAdd(&sh_stats[6], 1ull);
              atomicAdd(&sh_stats[7], (unsigned long long)cnt);
            }
#endif
            __syncwarp();
            int base = 0;
#pragma unroll
            for (int l = 0; l < kLpl; ++l) {
              if (key[l] == kkey) {
                const int rank = base + __popc(mem[l] & ((1u << lane) - 1u));
                float* a = reinterpret_cast<float*>(lxy + (rank >> 1)) + (rank & 1);
                float* f = reinterpret_cast<float*>(lf + (rank >> 1)) + (rank & 1);
                a[0] = -lx[l];
                a[2] = -ly[l];
                f[0] = vw[l];
                f[2] = w[l];
                if (HAS_Z) reinterpret_cast<float*>(lzs)[rank] = lz[l];
                if (rank == cnt - 1 && (cnt & 1)) {  // pad: the same lens with zero factors
                  a[1] = -lx[l];
                  a[3] = -ly[l];
                  f[1] = 0.f;
                  f[3] = 0.f;
                  if (HAS_Z) reinterpret_cast<float*>(lzs)[rank + 1] = lz[l];
                }
                const int db = kt == 3 ? kb + 2 : kt == 6 ? kb + 1 : nb;
                key[l] = db < nb ? (db + 1) * 8 + 4 + min(b1[l] - db, 2) : -1;
              }
              base += __popc(mem[l]);
            }
            __syncwarp();
            bool zero = false;
            if (kt == 0) {
              float v[1][6];
              direct_sums<MODE, HAS_M, HAS_Z, LOGB, 0>(lxy, lf, lzs, cnt, S, 0, C, v, zero);
              add_bin(v[0], kb, nb, wsum, lane);
            } else if (kt == 1 || kt == 4) {
              float v[2][6];
              const int e = kt == 1 ? kb + 1 : kb;
              direct_sums<MODE, HAS_M, HAS_Z, LOGB, 1>(lxy, lf, lzs, cnt, S, e, C, v, zero);
              if (kt == 4) {
                add_bin(v[1], kb, nb, wsum, lane);
              } else {
                if (keep_e != e || keep_n == kKeep) flush_keep();
                keep_e = e;
                ++keep_n;
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                  keep[0][q] += v[0][q];
                  keep[1][q] += v[1][q];
                }
              }
            } else {
              float v[3][6];
              const int e = kt < 4 ? kb + 1 : kb;
              direct_sums<MODE, HAS_M, HAS_Z, LOGB, 2>(lxy, lf, lzs, cnt, S, e, C, v, zero);
              if (kt < 4) add_bin(v[0], e - 1, nb, wsum, lane);
              add_bin(v[1], e, nb, wsum, lane);
              if (kt == 2 || kt == 5) add_bin(v[2], e + 1, nb, wsum, lane);
            }
            // d = 0 is in bin 0 when x_min = 0: its g terms are 0/0, as in the reference
            if (!LOGB && MODE == 0 && kt < 4 && kb <= 0 && C.e2f[0] <= 0.f && __any_sync(0xffffffffu, zero && S.ok) &&
                lane == 0)
              wsum[QGT * nb] = wsum[QGX * nb] = __longlong_as_double(0x7ff8000000000000ll);
          }
        }
        since_flush += tg.n * kChunk - tg.lo0 - (kChunk - tg.hiL);
        __syncwarp();  // every lane is done reading buffer b
        if (k + kNbuf < ntiles) issue(k + kNbuf);
        if (since_flush >= kFlushSrc) {
          fold_far<QA>(hist, wsum, nb, tb, lane);
          since_flush = 0;
        }
      }
      if (!aborted) ring_t += ntiles;
    }
    if (aborted) break;
    flush_keep();
    fold_far<QA>(hist, wsum, nb, tb, lane);
    double* out = P.item_sums + (size_t)(T.item_base + it.y) * kQ * nb;
    for (int e = lane; e < kQ * nb; e += 32) {
      const int q = e / nb;
      const int src = (q == QK && QA == 5) ? e - (QK - QW) * nb : e;
      out[e] = wsum[src] * (q == QN ? 1.0 : wsum[kQ * nb + (q == QGT || q == QGX ? 0 : 1)]);
    }
    __syncwarp();
  }
  if (aborted) {
    // No tile is consumed or issued any more; wait (bounded) for the copies
    // this warp issued and did not consume, so that none is in flight when
    // the block's shared memory is released.
    for (int t = ring_t; t < issued_end; ++t)
      if (t + 1 != P.debug_skip_tile) mbar_wait_bounded(&full[t % kNbuf], (uint32_t)(t / kNbuf) & 1u, wait_limit);
    if (lane == 0) atomicOr(P.err, kErrTimeout);
  }
#ifdef TPCF_MODE_STATS
  __syncthreads();
  if (tid < 8) atomicAdd(&g_series_stats[tid], sh_stats[tid]);
#endif
}

// Sub-chunk records of the cell-sorted sources: one warp per 32-source
// sub-chunk, moments in FP64 (about 200 shuffles and FP64 adds per sub-chunk).
__global__ void k_src_series(const int* __restrict__ idx, int n_valid, int n_chunks, int mode, bool has_m, bool has_z,
                             const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z,
                             const float* __restrict__ f1, const float* __restrict__ f2, const float* __restrict__ w,
                             const float* __restrict__ m, float* __restrict__ rec) {
  const int c = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= n_chunks) return;  // whole warps
  const RecShape R = rec_shape(mode, has_m, has_z);
  float* out = rec + (size_t)c * R.floats;
  const int s = c * kChunk + lane;
  const bool real = s < n_valid;
  float px = kNullPos, py = kNullPos, p = 0.f, q = 0.f, wi = 0.f, K = 0.f, zi = 0.f;
  float mnx = INFINITY, mny = INFINITY, mxx = -INFINITY, mxy = -INFINITY, mnz = INFINITY, mxz = -INFINITY;
  if (real) {
    const int i = idx[s];
    wi = w[i];
    px = x[i];
    py = y[i];
    if (mode == 0) {
      p = -(f1[i] * wi);
      q = -(f2[i] * wi);
      K = wi * (1.0f + (m ? m[i] : 0.f));
      zi = z ? z[i] : 0.f;
    } else {
      p = f1[i] * wi;
      q = f2[i] * wi;
      K = wi;
    }
    mnx = mxx = px;
    mny = mxy = py;
    mnz = zi != zi ? -INFINITY : zi;  // a NaN z takes part in no pair: never "every source"
    mxz = zi;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
    mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
    mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
    mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
    mnz = fminf(mnz, __shfl_xor_sync(0xffffffffu, mnz, o));
    mxz = fmaxf(mxz, __shfl_xor_sync(0xffffffffu, mxz, o));
  }
  float* f = out + R.src + lane;
  f[0] = px;
  f[32] = py;
  f[64] = p;
  f[96] = q;
  f[128] = wi;
  if (has_m) f[160] = K;
  if (has_z) f[32 * (R.fields - 1)] = real ? zi : __int_as_float(0x7fc00000);
  const float cx = 0.5f * mnx + 0.5f * mxx, cy = 0.5f * mny + 0.5f * mxy;
  const double dx = real ? (double)px - (double)cx : 0.0, dy = real ? (double)py - (double)cy : 0.0;
  float rad = (float)(sqrt(dx * dx + dy * dy) * (1.0 + 1e-6));
#pragma unroll
  for (int o = 16; o; o >>= 1) rad = fmaxf(rad, __shfl_xor_sync(0xffffffffu, rad, o));
  const double inv = rad > 0.f ? 1.0 / (double)rad : 0.0;
  const double ux = dx * inv, uy = dy * inv;  // delta / s
  auto red = [&](double v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  const double dp = p, dq = q, dw = wi;
  const double sp = red(dp), sq = red(dq), sw = red(dw), sk = red((double)K);
  if (lane == 0) {
    float4* o4 = reinterpret_cast<float4*>(out);
    // never 0: a lens on the centre of a sub-chunk without extent has no series
    const float far2 = (float)((double)rad * rad / ((double)kFarRatio * kFarRatio));
    o4[0] = make_float4(cx, cy, rad, fmaxf(far2, kMinNormal));
    o4[1] = make_float4((float)sp, (float)sq, (float)sw, (float)sk);
    o4[2] = make_float4(mnz, mxz, 0.f, 0.f);
  }
  const double uu = ux * ux + uy * uy;
  double re = 1.0, im = 0.0;  // (delta / s)^k
  double W[6][2];             // w (delta/s)^k
  for (int k = 0; k <= kOrder; ++k) {
    const double Mr = dp * re - dq * im, Mi = dp * im + dq * re;
    if (mode == 0) {
      // N_k: A conj(u) u^k; the highest order is not kept
      const double Nr = k < kOrder ? Mr * ux + Mi * uy : 0.0, Ni = k < kOrder ? Mi * ux - Mr * uy : 0.0;
      const double a = red(Mr), b = red(Nr), e = red(Mi), g = red(Ni);
      if (lane == 0)
        *reinterpret_cast<float4*>(out + R.g + 4 * k) = make_float4((float)a, (float)b, (float)e, (float)g);
    }
    if (k < 6) {
      W[k][0] = dw * re;
      W[k][1] = dw * im;
    }
    const double nr = re * ux - im * uy;
    im = re * uy + im * ux;
    re = nr;
  }
  const double w11 = red(dw * uu), w22 = red(dw * uu * uu);
  double v[18];
  v[0] = red(W[1][0]), v[1] = red(W[1][1]);
  v[2] = red(W[1][0] * uu), v[3] = red(W[1][1] * uu);
  v[4] = red(W[2][0]), v[5] = red(W[2][1]);
  v[6] = red(W[2][0] * uu), v[7] = red(W[2][1] * uu);
  v[8] = red(W[3][0]), v[9] = red(W[3][1]);
  v[10] = red(W[4][0]), v[11] = red(W[4][1]);
  v[12] = red(W[3][0] * uu), v[13] = red(W[3][1] * uu);
  v[14] = red(W[5][0]), v[15] = red(W[5][1]);
  v[16] = red(W[1][0] * uu * uu), v[17] = red(W[1][1] * uu * uu);
  if (lane == 0) {
    float4* o4 = reinterpret_cast<float4*>(out + R.d);
    o4[0] = make_float4((float)sw, (float)(w11 / 4), (float)(w22 / 64), 0.f);
    o4[1] = make_float4((float)v[0], (float)v[1], (float)(-v[2] / 8), (float)(-v[3] / 8));
    o4[2] = make_float4((float)(-v[4] / 4), (float)(-v[5] / 4), (float)(v[6] / 16), (float)(v[7] / 16));
    o4[3] = make_float4((float)(v[8] / 8), (float)(v[9] / 8), (float)(-5 * v[12] / 128), (float)(-5 * v[13] / 128));
    o4[4] = make_float4((float)(-5 * v[10] / 64), (float)(-5 * v[11] / 64), (float)(7 * v[14] / 128),
                        (float)(7 * v[15] / 128));
    o4[5] = make_float4((float)(-v[16] / 64), (float)(-v[17] / 64), 0.f, 0.f);
  }
}

// --------------------------------------------------------- host launchers --
template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB>
static cudaError_t prepare_t(const PairParams& P, int bt, int num_sms, PairLaunch* L) {
  constexpr int QA = (MODE == 0 && HAS_M) ? 6 : 5;
  bt = min(bt, kSeriesThreads);
  const size_t per = warp_smem(P.nb, P.nb - P.far_bin, QA, rec_shape(MODE, HAS_M, HAS_Z).floats).total;
  while (bt > 32 && edge_smem(P.nb) + per * (bt / 32) > 110 * 1024) bt /= 2;
  const size_t smem = edge_smem(P.nb) + per * (bt / 32);
  auto kern = k_pairs_series<MODE, HAS_M, HAS_Z, LOGB>;
  cudaError_t e = allow_dynamic_smem(kern);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, bt, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const int need = (P.n_items + bt / 32 - 1) / (bt / 32);  // each warp takes items of its own
  L->func = reinterpret_cast<const void*>(kern);
  L->grid = max(1, min(per_sm * num_sms, need));
  L->block = bt;
  L->smem = smem;
  return cudaSuccess;
}

cudaError_t prepare_pairs_series(const PairParams& P, int mode, bool has_m, bool has_z, bool logb, int bt, int num_sms,
                                 PairLaunch* L) {
  if (mode == 1)
    return logb ? prepare_t<1, false, false, true>(P, bt, num_sms, L)
                : prepare_t<1, false, false, false>(P, bt, num_sms, L);
  if (has_m) {
    if (has_z)
      return logb ? prepare_t<0, true, true, true>(P, bt, num_sms, L)
                  : prepare_t<0, true, true, false>(P, bt, num_sms, L);
    return logb ? prepare_t<0, true, false, true>(P, bt, num_sms, L)
                : prepare_t<0, true, false, false>(P, bt, num_sms, L);
  }
  if (has_z)
    return logb ? prepare_t<0, false, true, true>(P, bt, num_sms, L)
                : prepare_t<0, false, true, false>(P, bt, num_sms, L);
  return logb ? prepare_t<0, false, false, true>(P, bt, num_sms, L)
              : prepare_t<0, false, false, false>(P, bt, num_sms, L);
}

int series_lens_group() { return 32 * kLpl; }

// First bin of the far sums: the bins within a factor of 8 of theta_max (98%
// of the disc), and at most 20, so that a warp's sums stay small in shared
// memory; nearer sub-chunks are summed directly.
int series_far_bin(const double* e2, int nb) {
  int b = nb;
  while (b > 0 && nb - b < 20 && e2[b] > e2[nb] / 64.0) --b;
  return b;
}

size_t series_bytes(int n_valid, int mode, bool has_m, bool has_z) {
  const int n_chunks = max((n_valid + kChunk - 1) / kChunk, 1);
  return (size_t)n_chunks * rec_shape(mode, has_m, has_z).floats * sizeof(float);
}

cudaError_t launch_src_series(const int* idx, int n_valid, int mode, bool has_m, bool has_z, const float* x,
                              const float* y, const float* z, const float* f1, const float* f2, const float* w,
                              const float* m, float* rec, cudaStream_t st) {
  const int n_chunks = (n_valid + kChunk - 1) / kChunk;
  if (n_chunks > 0)
    k_src_series<<<(n_chunks + 7) / 8, 256, 0, st>>>(idx, n_valid, n_chunks, mode, has_m, has_z, x, y, z, f1, f2, w, m,
                                                     rec);
  return cudaGetLastError();
}

}  // namespace tpcf
