// sphere.cu -- pair sums on the sphere: the spherical_coords branch of
// tangential_shear_tpcf / scalar_kappa_tpcf (src/tpcf.f90:297-359, with
// distance_sphere src/utils.f90:512-528 and angles_sphere :618-639).
//
// Positions are FP32 (lambda, phi) in radians.  Each object becomes its unit
// vector u, computed in FP64 by canon_sincos (sph_canon.cuh) and split into
// FP32 hi + lo parts.  For a pair (lens A, source B):
//   chord^2  c^2 = |u_B - u_A|^2, binned against (2 sin(e_i/2))^2 of the FP64
//            angle edges e_i (monotone in the angle, so the same bins);
//   angle    theta = 2 asin(c/2) (the reference's acos of the dot product);
//   position angle at the lens, A = (u_B - u_A).east_A and
//            B = (u_B - u_A).north_A.  These are the numerators of
//            angles_sphere, so cos 2phi = (A^2 - B^2)/(A^2 + B^2) and
//            sin 2phi = 2AB/(A^2 + B^2), the same as 2 cs1^2 - 1, 2 cs1 cs2.
// The pair arithmetic is FP32 on hi + lo differences (relative error ~1e-7
// at any separation).  The FP64 guard band re-bins a pair by the canonical
// rule: u = hi + lo in FP64, c^2 = (dx^2 + dy^2) + dz^2 rounded as written.
// The one-bin and one-edge sub-chunk paths run on packed FP32 instructions
// (two pairs per instruction) over sub-chunks laid out in pair form in HBM (ChunkS).
//
// Pruning: a cell grid over (lambda reduced to [0, 2 pi), phi).  The rows of a
// work item are the phi rows within R of the lens box (angular distance
// >= |dphi|).  In each row the cells lie within the lambda reach
// asin(sin R / cos phi*) of the box, phi* being its largest |phi|, taken
// modulo 2 pi as up to three disjoint cell runs.  A pole within reach scans
// the whole row.  The reference aborts near poles and the prime meridian
// (src/kdtree.f90:398-413); here every position is valid.

#include <cstdio>

#include "pair_hist.cuh"
#include "pair_tiles.cuh"
#include "sph_canon.cuh"
#include "tpcf_device.cuh"
#include "tpcf_internal.cuh"
#include "tpcf_kernels.h"

namespace tpcf {

// --------------------------------------------------- canonical unit vector --
// u = (cos phi cos lambda, cos phi sin lambda, sin phi), hi = fl32(u),
// lo = fl32(u - hi).
__device__ __forceinline__ void canon_unit(float lam, float phi, float4& hi, float4& lo) {
  double sl, cl, sp, cp;
  canon_sincos((double)lam, sl, cl);
  canon_sincos((double)phi, sp, cp);
  const double ux = __dmul_rn(cp, cl), uy = __dmul_rn(cp, sl), uz = sp;
  hi = make_float4(__double2float_rn(ux), __double2float_rn(uy), __double2float_rn(uz), 0.f);
  lo = make_float4(__double2float_rn(__dsub_rn(ux, (double)hi.x)), __double2float_rn(__dsub_rn(uy, (double)hi.y)),
                   __double2float_rn(__dsub_rn(uz, (double)hi.z)), 0.f);
}

// Canonical FP64 bin of a pair on the sphere (the guard-band path).
__device__ __forceinline__ int slow_bin_s(float4 ha, float4 la, float4 hb, float4 lb, const double* e2,
                                              int nb) {
  const double dx = __dsub_rn(__dadd_rn((double)hb.x, (double)lb.x), __dadd_rn((double)ha.x, (double)la.x));
  const double dy = __dsub_rn(__dadd_rn((double)hb.y, (double)lb.y), __dadd_rn((double)ha.y, (double)la.y));
  const double dz = __dsub_rn(__dadd_rn((double)hb.z, (double)lb.z), __dadd_rn((double)ha.z, (double)la.z));
  const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  if (!(d2 >= e2[0]) || d2 > e2[nb]) return -1;
  if (d2 == e2[nb]) return nb - 1;
  int lo = 0, hi = nb;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (d2 >= e2[mid]) lo = mid; else hi = mid;
  }
  return lo;
}

// ------------------------------------------------------------ pair terms ----
// One source in scalar form: a = {hi, p}, b = {lo, q}, c = {w, K, z, 0}.
struct __align__(16) SrcRecS {
  float4 a, b, c;
};

// One lens: unit vector hi/lo and its local east/north basis.
struct LensS {
  float4 h, l;
  float ex, ey, nx, ny, nz;
};

__device__ __forceinline__ LensS lens_frame(float4 h, float4 l) {
  LensS L;
  L.h = h;
  L.l = l;
  const double ux = (double)h.x + (double)l.x, uy = (double)h.y + (double)l.y, uz = (double)h.z + (double)l.z;
  const double rho = sqrt(ux * ux + uy * uy);
  if (rho > 0.0) {
    L.ex = (float)(-uy / rho); L.ey = (float)(ux / rho);
    L.nx = (float)(-uz * ux / rho); L.ny = (float)(-uz * uy / rho); L.nz = (float)rho;
  } else {  // exactly on a pole: any tangent basis
    L.ex = 0.f; L.ey = 1.f; L.nx = uz > 0 ? -1.f : 1.f; L.ny = 0.f; L.nz = 0.f;
  }
  return L;
}

// theta = 2 asin(c/2) from c^2 and c.  SMALL (c <= 0.25): the series
// c (1 + c^2/24 + 3 c^4/640 + 5 c^6/7168), truncation < 2e-9 relative.
template <bool SMALL>
__device__ __forceinline__ float chord_theta(float d2, float c) {
  if (SMALL) return c * fmaf(d2, fmaf(d2, fmaf(d2, 6.9754464e-4f, 4.6875e-3f), 4.16666679e-2f), 1.f);
  return 2.f * asinf(fminf(0.5f * c, 1.f));
}
// theta^2 / c^2 by the same series (log-spaced binning in theta^2).
__device__ __forceinline__ float chord_theta2(float d2) {
  const float g = fmaf(d2, fmaf(d2, fmaf(d2, 6.9754464e-4f, 4.6875e-3f), 4.16666679e-2f), 1.f);
  return d2 * g * g;
}

// d2 = c^2, th = theta, r = 1/(A^2+B^2), X = p P + q U, Y = q P - p U with
// P = A^2 - B^2, U = 2AB (shear); scalar: r = 1, X = p, Y = q.
template <int MODE, bool SMALL>
__device__ __forceinline__ void sph_terms(const LensS& L, const float4 a, const float4 b, float& d2, float& th,
                                          float& r, float& X, float& Y) {
  const float dx = (a.x - L.h.x) + (b.x - L.l.x);
  const float dy = (a.y - L.h.y) + (b.y - L.l.y);
  const float dz = (a.z - L.h.z) + (b.z - L.l.z);
  d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
  // series path: binned pairs have d2 > 0; otherwise c = 0 exactly at d2 = 0
  const float c = SMALL ? d2 * rsqrt_ftz(d2) : sqrtf(d2);
  th = chord_theta<SMALL>(d2, c);
  if (MODE == 0) {
    const float A = fmaf(dy, L.ey, dx * L.ex);
    const float B = fmaf(dz, L.nz, fmaf(dy, L.ny, dx * L.nx));
    const float A2 = A * A;
    const float P = fmaf(-B, B, A2);
    const float s = fmaf(B, B, A2);
    const float ab = A * B;
    const float U = ab + ab;
    r = __fdividef(1.f, s);
    X = fmaf(a.w, P, b.w * U);
    Y = fmaf(b.w, P, -(a.w * U));
  } else {
    r = 1.f;
    X = a.w;
    Y = b.w;
  }
}

template <bool LOGB>
__device__ __forceinline__ int pair_bin_s(float d2, const LensS& L, const float4 a, const float4 b,
                                          const BinCtx& C) {
  if (LOGB) {
    const float t = fmaf(lg2_ftz(chord_theta2(d2)), C.A, C.B);
    const float tf = floorf(t);
    const float fr = t - tf;
    int bin = __float2int_rz(tf);
    if (fr < C.eps || fr > C.one_m_eps) bin = slow_bin_s(L.h, L.l, a, b, C.e2s, C.nb);
    return bin;
  } else {
    if (d2 < C.lo_g || d2 > C.hi_g) return -1;
    int lo = 0, hi = C.nb;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (d2 >= C.e2f[mid]) lo = mid; else hi = mid;
    }
    const float el = C.e2f[lo], eh = C.e2f[lo + 1];
    if (d2 <= el * (1.f + C.eps) || d2 >= eh * (1.f - C.eps)) lo = slow_bin_s(L.h, L.l, a, b, C.e2s, C.nb);
    return lo;
  }
}

// Conservative bin class of a 3-D box (min mn, max mx of the chunk's hi parts,
// already widened by the hi/lo split error) for one lens; classes as in the
// planar kernel.
template <bool LOGB>
__device__ __forceinline__ int classify_s(const LensS& L, const float4 mn, const float4 mx, const BinCtx& C,
                                          int& blo) {
  const float dxl = fmaxf(fmaxf(mn.x - L.h.x, L.h.x - mx.x), 0.f);
  const float dyl = fmaxf(fmaxf(mn.y - L.h.y, L.h.y - mx.y), 0.f);
  const float dzl = fmaxf(fmaxf(mn.z - L.h.z, L.h.z - mx.z), 0.f);
  const float dxh = fmaxf(L.h.x - mn.x, mx.x - L.h.x);
  const float dyh = fmaxf(L.h.y - mn.y, mx.y - L.h.y);
  const float dzh = fmaxf(L.h.z - mn.z, mx.z - L.h.z);
  const float dmin2 = fmaf(dzl, dzl, fmaf(dyl, dyl, dxl * dxl));
  const float dmax2 = fmaf(dzh, dzh, fmaf(dyh, dyh, dxh * dxh));
  int b0, b1;
  if (LOGB) {
    b0 = __float2int_rd(fmaf(lg2_ftz(chord_theta2(dmin2)), C.A, C.B) - C.eps);
    b1 = __float2int_rd(fmaf(lg2_ftz(chord_theta2(dmax2)), C.A, C.B) + C.eps);
  } else {
    b0 = edge_index_f32(dmin2 * (1.f - C.eps), C.e2f, C.nb);
    b1 = edge_index_f32(dmax2 * (1.f + C.eps), C.e2f, C.nb);
  }
  if (b1 < 0 || b0 >= C.nb) return 0;
  b0 = max(b0, -1);  // every bin below 0 or from nb up is dropped alike
  b1 = min(b1, C.nb);
  blo = b0;
  const int e = b1 - b0;  // bin edges in range; a z cut is applied inside the register paths
  return e <= 2 ? 1 + e : 4;
}

template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB, bool SMALL, int NC, int QA>
__device__ __forceinline__ void do_pair_s(const LensS& L, float lz, const SrcRecS& s, float* __restrict__ hcol,
                                          const BinCtx& C) {
  if (HAS_Z) {
    if (lz > s.c.z) return;  // src/tpcf.f90:322
  }
  float d2, th, r, X, Y;
  sph_terms<MODE, SMALL>(L, s.a, s.b, d2, th, r, X, Y);
  const int bin = pair_bin_s<LOGB>(d2, L, s.a, s.b, C);
  if ((unsigned)bin >= (unsigned)C.nb) return;
  float* h = hcol + bin * (QA * NC);
  h[QGT * NC] = fmaf(r, X, h[QGT * NC]);
  h[QGX * NC] = fmaf(r, Y, h[QGX * NC]);
  h[QW * NC] += s.c.x;
  h[QDW * NC] = fmaf(th, s.c.x, h[QDW * NC]);
  h[QN * NC] += 1.0f;
  if (MODE == 0 && HAS_M) h[QK * NC] += s.c.y;
}

// Two consecutive sources (2k, 2k+1) of a 32-source sub-chunk with their fields
// interleaved, so that a 64-bit register pair holds one field of both (the
// operand form of the sm_100 packed FP32 instructions).  The source grid is
// stored in this form.  hi, lo: parts of the unit vector; p = -e1 w, q = -e2 w
// (scalar-scalar kE w, kB w), K = (1 + m) w.
struct __align__(16) SrcPairS {
  float4 hxy;  // hi.x0 hi.x1 hi.y0 hi.y1
  float4 hzp;  // hi.z0 hi.z1 p0 p1
  float4 lxy;  // lo.x0 lo.x1 lo.y0 lo.y1
  float4 lzq;  // lo.z0 lo.z1 q0 q1
  float4 wk;   // w0 w1 K0 K1
  float4 zz;   // z0 z1 0 0
};
// A sub-chunk as it lies in HBM and is copied into shared memory: the 3-D box
// of its hi parts widened by 2^-23 per side (the hi/lo split of both ends moves
// u_B - u_A by at most 2^-24), its {p, q, w, K} sums, its sources.
struct __align__(16) ChunkS {
  float4 mn, mx, sum;
  SrcPairS src[kChunk / 2];
};
static_assert(sizeof(ChunkS) % 16 == 0, "copied in 16-byte units");
// Source j of a sub-chunk in SrcPairS form, as a SrcRecS.
__device__ __forceinline__ SrcRecS src_of_s(const SrcPairS* __restrict__ S, int j) {
  const float* f = reinterpret_cast<const float*>(S + (j >> 1)) + (j & 1);
  SrcRecS r;
  r.a = make_float4(f[0], f[2], f[4], f[6]);
  r.b = make_float4(f[8], f[10], f[12], f[14]);
  r.c = make_float4(f[16], f[18], f[20], 0.f);
  return r;
}

// A lens's constants in packed form: -hi, -lo and the east/north basis.
struct LensS2 {
  float2 nhx, nhy, nhz, nlx, nly, nlz, ex, ey, nx, ny, nz;
};
__device__ __forceinline__ LensS2 lens_pack(const LensS& L) {
  LensS2 P;
  P.nhx = dup2(-L.h.x); P.nhy = dup2(-L.h.y); P.nhz = dup2(-L.h.z);
  P.nlx = dup2(-L.l.x); P.nly = dup2(-L.l.y); P.nlz = dup2(-L.l.z);
  P.ex = dup2(L.ex); P.ey = dup2(L.ey);
  P.nx = dup2(L.nx); P.ny = dup2(L.ny); P.nz = dup2(L.nz);
  return P;
}

// sph_terms for the two sources of one SrcPairS (packed FP32; each half
// equals the scalar computation: a.x - h.x = a.x + (-h.x)).
template <int MODE, bool SMALL>
__device__ __forceinline__ void sph_terms2(const LensS2& L, const SrcPairS& s, float tiny, float2& d2, float2& th,
                                           float2& r, float2& X, float2& Y) {
  const float2 dx = add2(add2(lo2(s.hxy), L.nhx), add2(lo2(s.lxy), L.nlx));
  const float2 dy = add2(add2(hi2(s.hxy), L.nhy), add2(hi2(s.lxy), L.nly));
  const float2 dz = add2(add2(lo2(s.hzp), L.nhz), add2(lo2(s.lzq), L.nlz));
  // series path (log bins): d2 = 0 is below the first edge; the offsets (1e-9 of
  // that edge) only keep its masked terms finite
  d2 = fma2(dz, dz, fma2(dy, dy, SMALL ? fma2(dx, dx, dup2(tiny)) : mul2(dx, dx)));
  if (SMALL) {
    const float2 c = mul2(d2, make_float2(rsqrt_ftz(d2.x), rsqrt_ftz(d2.y)));
    th = mul2(c, fma2(d2, fma2(d2, fma2(d2, dup2(6.9754464e-4f), dup2(4.6875e-3f)), dup2(4.16666679e-2f)),
                      dup2(1.f)));
  } else {
    th = make_float2(chord_theta<false>(d2.x, sqrtf(d2.x)), chord_theta<false>(d2.y, sqrtf(d2.y)));
  }
  if (MODE == 0) {
    const float2 A = fma2(dy, L.ey, mul2(dx, L.ex));
    const float2 B = fma2(dz, L.nz, fma2(dy, L.ny, mul2(dx, L.nx)));
    const float2 A2 = SMALL ? fma2(A, A, dup2(tiny)) : mul2(A, A);
    const float2 P = fma2(make_float2(-B.x, -B.y), B, A2);
    const float2 sq = fma2(B, B, A2);
    const float2 ab = mul2(A, B);
    const float2 U = add2(ab, ab);
    r = make_float2(__fdividef(1.f, sq.x), __fdividef(1.f, sq.y));
    X = fma2(hi2(s.hzp), P, mul2(hi2(s.lzq), U));
    const float2 pU = mul2(hi2(s.hzp), U);
    Y = fma2(hi2(s.lzq), P, make_float2(-pU.x, -pU.y));
  } else {
    r = dup2(1.f);
    X = hi2(s.hzp);
    Y = hi2(s.lzq);
  }
}

// Register sums of one lens over a sub-chunk.  One edge: all pairs (s*) and the
// upper side (h*).  Two edges: each side on its own (s*, h*[0], h*[1]), since a bin
// between two edges may hold one pair of a sub-chunk whose others are far beyond: a
// difference of sums would carry their rounding (1.8e-5 of a bin's d w).  Counts are at or above each edge.
template <int NE>
struct SphAcc {
  float2 sgt, sgx, sw, sdw, sk, sn;
  float close[NE ? NE : 1];  // smallest |d2 - E|
  float2 hgt[NE ? NE : 1], hgx[NE ? NE : 1], hw[NE ? NE : 1], hdw[NE ? NE : 1], hk[NE ? NE : 1], hn[NE ? NE : 1];
};
template <int NE>
__device__ __forceinline__ void sph_acc_zero(SphAcc<NE>& A) {
  A.sgt = A.sgx = A.sw = A.sdw = A.sk = A.sn = dup2(0.f);
#pragma unroll
  for (int e = 0; e < NE; ++e) A.close[e] = 3.0e38f, A.hgt[e] = A.hgx[e] = A.hw[e] = A.hdw[e] = A.hk[e] = A.hn[e] = dup2(0.f);
}

// The two pairs of one SrcPairS against a lens; in a partial sub-chunk (PART)
// a0, a1 tell which of the two belong to the row span.  With a z cut a pair with z_A > z_B
// (src/tpcf.f90:322) adds nothing.  For each of the NE edges the upper-side
// sums are formed too (pairs with d2 >= E, the side a 1.0/0.0 mask from the sign
// of d2 - E, applied by multiplication) and the smallest |d2 - E| is kept.
// Without a z cut the w and K sums of all pairs (and, scalar-scalar, the g sums)
// are the sub-chunk's totals, so they are not accumulated here.
template <int MODE, bool HAS_M, bool HAS_Z, bool SMALL, int NE, bool PART>
__device__ __forceinline__ void sph_step(const LensS2& L, float lz, const SrcPairS& s, bool a0, bool a1,
                                         float tiny, const float* E, SphAcc<NE>& A) {
  constexpr bool LI = !(HAS_Z || PART);
  float2 d2, th, r, X, Y;
  sph_terms2<MODE, SMALL>(L, s, tiny, d2, th, r, X, Y);
  float2 w = lo2(s.wk), K = hi2(s.wk);
  bool v0 = true, v1 = true;
  if (HAS_Z) {
    v0 = lz <= s.zz.x;
    v1 = lz <= s.zz.y;
  }
  if (PART) {
    v0 = v0 && a0;
    v1 = v1 && a1;
  }
  const float2 vm = make_float2(v0 ? 1.f : 0.f, v1 ? 1.f : 0.f);
  if (!LI) {
    r = mul2(r, vm);
    w = mul2(w, vm);
    if (MODE == 0 && HAS_M) K = mul2(K, vm);
    A.sn = add2(A.sn, vm);
  }
  if (NE == 2) {
    const float2 one_neg = dup2(-1.f);
    float2 m[2], rk[3], wk[3], kk[3];
    rk[0] = r; wk[0] = w; kk[0] = K;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 t = add2(d2, dup2(-E[NE ? e : 0]));
      A.close[e] = fminf(A.close[e], fminf(fabsf(t.x), fabsf(t.y)));
      m[e] = make_float2(t.x >= 0.f ? 1.f : 0.f, t.y >= 0.f ? 1.f : 0.f);
      rk[e + 1] = mul2(r, m[e]);  // r, w, K carry the validity mask already
      wk[e + 1] = mul2(w, m[e]);
      rk[e] = fma2(rk[e + 1], one_neg, rk[e]);  // exactly 0 or the value
      wk[e] = fma2(wk[e + 1], one_neg, wk[e]);
      if (MODE == 0 && HAS_M) {
        kk[e + 1] = mul2(K, m[e]);
        kk[e] = fma2(kk[e + 1], one_neg, kk[e]);
      }
      A.hn[e] = add2(A.hn[e], LI ? m[e] : mul2(m[e], vm));
    }
    A.sgt = fma2(rk[0], X, A.sgt);
    A.sgx = fma2(rk[0], Y, A.sgx);
    A.sw = add2(A.sw, wk[0]);
    A.sdw = fma2(th, wk[0], A.sdw);
    if (MODE == 0 && HAS_M) A.sk = add2(A.sk, kk[0]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      A.hgt[e] = fma2(rk[e + 1], X, A.hgt[e]);
      A.hgx[e] = fma2(rk[e + 1], Y, A.hgx[e]);
      A.hw[e] = add2(A.hw[e], wk[e + 1]);
      A.hdw[e] = fma2(th, wk[e + 1], A.hdw[e]);
      if (MODE == 0 && HAS_M) A.hk[e] = add2(A.hk[e], kk[e + 1]);
    }
    return;
  }
  if (!(LI && MODE == 1)) {
    A.sgt = fma2(r, X, A.sgt);
    A.sgx = fma2(r, Y, A.sgx);
  }
  if (!LI) A.sw = add2(A.sw, w);
  A.sdw = fma2(th, w, A.sdw);
  if (MODE == 0 && HAS_M && !LI) A.sk = add2(A.sk, K);
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const float2 t = add2(d2, dup2(-E[e]));
    A.close[e] = fminf(A.close[e], fminf(fabsf(t.x), fabsf(t.y)));
    float2 mh = make_float2(t.x >= 0.f ? 1.f : 0.f, t.y >= 0.f ? 1.f : 0.f);
    if (!LI) mh = mul2(mh, vm);
    const float2 rm = mul2(r, mh);  // r, w, K carry the validity mask already
    const float2 wm = mul2(w, mh);
    A.hgt[e] = fma2(rm, X, A.hgt[e]);
    A.hgx[e] = fma2(rm, Y, A.hgx[e]);
    A.hw[e] = add2(A.hw[e], wm);
    A.hdw[e] = fma2(th, wm, A.hdw[e]);
    A.hn[e] = add2(A.hn[e], mh);
    if (MODE == 0 && HAS_M) A.hk[e] = fma2(K, mh, A.hk[e]);
  }
}

// Sums over all pairs of a sub-chunk; ss = {sum p, sum q, sum w, sum K}.
template <int MODE, bool HAS_M, bool LI, int QA, int NE>
__device__ __forceinline__ void sph_totals(const SphAcc<NE>& A, const float4 ss, float* tot) {
  tot[QGT] = (LI && MODE == 1) ? ss.x : sum2(A.sgt);
  tot[QGX] = (LI && MODE == 1) ? ss.y : sum2(A.sgx);
  tot[QW] = LI ? ss.z : sum2(A.sw);
  tot[QDW] = sum2(A.sdw);
  tot[QN] = LI ? (float)kChunk : sum2(A.sn);
  if (MODE == 0 && HAS_M) tot[QK] = LI ? ss.w : sum2(A.sk);
}

// The sources [lo, hi) of a sub-chunk (all 32 unless PART) against a lens.
template <int MODE, bool HAS_M, bool HAS_Z, bool SMALL, bool PART, int NE>
__device__ __forceinline__ void sph_loop(const SrcPairS* __restrict__ S, int lo, int hi, const LensS2& L, float lz,
                                         float tiny, const float* E, SphAcc<NE>& A) {
  const int k0 = PART ? lo >> 1 : 0, k1 = PART ? (hi + 1) >> 1 : kChunk / 2;
#pragma unroll 2
  for (int k = k0; k < k1; ++k)
    sph_step<MODE, HAS_M, HAS_Z, SMALL, NE, PART>(L, lz, S[k], !PART || 2 * k >= lo, !PART || 2 * k + 1 < hi, tiny, E, A);
}

// Class 1: every pair of the chunk is in bin `blo`.
template <int MODE, bool HAS_M, bool HAS_Z, bool SMALL, bool PART, int NC, int QA>
__device__ __forceinline__ void chunk_single_s(const SrcPairS* __restrict__ S, int lo, int hi, const LensS2& L,
                                               float lz, float tiny, int cls, int blo, float* __restrict__ hcol,
                                               const float4 ss) {
  SphAcc<0> A;
  sph_acc_zero(A);
  sph_loop<MODE, HAS_M, HAS_Z, SMALL, PART, 0>(S, lo, hi, L, lz, tiny, nullptr, A);
  if (cls != 1) return;
  float acc[QA];
  sph_totals<MODE, HAS_M, !(HAS_Z || PART), QA>(A, ss, acc);
  hist_add<QA, NC>(hcol, blo, acc);
}

// Classes 2 and 3: pairs in bins blo .. blo + NE across NE = 1 or 2 edges (a bin
// outside [0, nb) is dropped); edge e is e2f[blo + 1 + e].  One edge: bin blo + j receives
// h[j-1] - h[j] with h[-1] = all and h[1] = 0, as in the planar kernel; two: its own sums.
template <int MODE, bool HAS_M, bool HAS_Z, bool SMALL, bool PART, int NC, int QA, int NE>
__device__ __forceinline__ void chunk_edges_s(const SrcPairS* __restrict__ S, int lo, int hi, const LensS& Lf,
                                              const LensS2& L, float lz, int cls, int blo, float* __restrict__ hcol,
                                              const BinCtx& C, const float4 ss) {
  float E[NE];
#pragma unroll
  for (int e = 0; e < NE; ++e)  // lanes with fewer edges keep one no pair reaches
    E[e] = e < cls - 1 ? C.e2f[min(max(blo + 1 + e, 0), C.nb)] : 3.0e38f;
  SphAcc<NE> A;
  sph_acc_zero(A);
  sph_loop<MODE, HAS_M, HAS_Z, SMALL, PART, NE>(S, lo, hi, L, lz, C.tiny, E, A);
  if (cls == 0) return;
  // without the offsets of the series path a pair with d = 0 makes the sums infinite
  // or NaN whatever its mask
  bool band = MODE == 0 && !SMALL && !(fabsf(sum2(A.sgt)) <= kMaxFinite);
#pragma unroll
  for (int e = 0; e < NE; ++e) band = band || A.close[e] <= E[e] * C.eps_rel;
  if (band) {  // rare: a pair inside the guard band or at d = 0; the sub-chunk is binned pair by pair
    for (int j = lo; j < hi; ++j) do_pair_s<MODE, HAS_M, HAS_Z, SMALL, SMALL, NC, QA>(Lf, lz, src_of_s(S, j), hcol, C);
    return;
  }
  float prev[QA];
  sph_totals<MODE, HAS_M, NE == 1 && !(HAS_Z || PART), QA>(A, ss, prev);
  if (NE == 2 && !(HAS_Z || PART)) prev[QN] = (float)kChunk;
#pragma unroll
  for (int j = 0; j <= NE; ++j) {
    float up[QA];
#pragma unroll
    for (int q = 0; q < QA; ++q) up[q] = 0.f;
    if (j < NE) {
      up[QGT] = sum2(A.hgt[j < NE ? j : 0]);
      up[QGX] = sum2(A.hgx[j < NE ? j : 0]);
      up[QW] = sum2(A.hw[j < NE ? j : 0]);
      up[QDW] = sum2(A.hdw[j < NE ? j : 0]);
      up[QN] = sum2(A.hn[j < NE ? j : 0]);
      if (MODE == 0 && HAS_M) up[QK] = sum2(A.hk[j < NE ? j : 0]);
    }
    const int bin = blo + j;
    if (j <= cls - 1 && bin >= 0 && bin < C.nb) {
      float v[QA];
#pragma unroll
      for (int q = 0; q < QA; ++q) v[q] = NE == 2 && q != QN ? prev[q] : prev[q] - up[q];
      hist_add<QA, NC>(hcol, bin, v);
    }
#pragma unroll
    for (int q = 0; q < QA; ++q) prev[q] = up[q];
  }
}

// ------------------------------------------------------------ cell runs -----
constexpr float kTwoPiF = 6.28318548f;      // 2 pi rounded up to FP32
constexpr int kRowsS = 10;  // rows whose (up to three) runs a warp holds at once: lane 3 r + j
constexpr int kNbufS = 3;   // sub-chunks in flight per warp

// Lambda reach of a work item: full = every cell of a row, else the interval
// [box.x - dl, box.z + dl] modulo 2 pi.
__device__ __forceinline__ void sph_reach(const GridDesc& G, float4 box, float R, float m, float& dl, bool& full) {
  const float ps = fmaxf(fabsf(box.y), fabsf(box.w)) + m;
  full = false;
  dl = 0.f;
  if (ps + R >= 1.5707f) { full = true; return; }
  const float sr = sinf(R) / cosf(ps);
  if (!(sr < 0.999f)) { full = true; return; }
  dl = asinf(sr) * 1.0001f + m;
  if ((box.z - box.x) + 2.f * dl + 2.f * G.cell + 4.f * m >= 6.2831f) full = true;
}

// The runs of sorted sources in row cy whose cells may hold a source within R
// of the box; returns how many (0..3).  The shifted intervals are more than
// two cells apart, so no cell appears in two runs.
__device__ __forceinline__ int sph_row_spans(const GridDesc& G, float4 box, float R, float m, int cy, float dl,
                                             bool full, int2* out) {
  const float ylo = G.y0 + (float)cy * G.cell - m;
  const float yhi = G.y0 + (float)(cy + 1) * G.cell + m;
  const float dyr = fmaxf(0.f, fmaxf(ylo - box.w, box.y - yhi));
  if (dyr > R) return 0;
  const int base = cy * G.ncx;
  if (full) {
    out[0] = make_int2(G.cell_start[base], G.cell_start[base + G.ncx]);
    return 1;
  }
  const float a = box.x - dl, b = box.z + dl;
  const float xmax = G.x0 + (float)G.ncx * G.cell;
  int n = 0;
#pragma unroll
  for (int k = -1; k <= 1; ++k) {
    const float s = (float)k * kTwoPiF;
    if (b + s < G.x0 - m || a + s > xmax + m) continue;
    const int cx0 = clamp_floor((a + s - G.x0) * G.inv_cell, 0, G.ncx - 1);
    const int cx1 = clamp_floor((b + s - G.x0) * G.inv_cell, 0, G.ncx - 1);
    out[n++] = make_int2(G.cell_start[base + cx0], G.cell_start[base + cx1 + 1]);
  }
  return n;
}

// ------------------------------------------------------------ the kernel ----
// Shared memory of one warp.
struct SphWarpSmem {
  size_t ring, hist, wsum, fvw, fw, mbar, total;
};
__host__ __device__ inline SphWarpSmem sph_warp_smem(int nb, int qa) {
  SphWarpSmem s{};
  size_t o = 0;
  s.ring = o; o += kNbufS * sizeof(ChunkS);
  s.hist = o; o += (size_t)nb * qa * 32 * sizeof(float);
  s.wsum = o; o += (size_t)kQ * nb * sizeof(double);
  s.fvw = o;  o += 32 * sizeof(double);
  s.fw = o;   o += 32 * sizeof(double);
  s.mbar = o; o += kNbufS * sizeof(uint64_t);
  s.total = (o + 15) / 16 * 16;
  return s;
}
__host__ __device__ inline size_t sph_edge_smem(int nb) { return ((size_t)(nb + 1) * 12 + 15) / 16 * 16; }

// Persistent, every warp on its own as in the planar kernel: it takes items of
// 32 lenses from the queue and streams the sub-chunks of the item's source runs
// through its own ring of buffers (bulk copies, bounded waits).  The tiles were
// copied for a block of 128 lenses and rewritten into pair form there, between
// two barriers (barrier stall 1.1 per issued instruction).  Twelve warps per SM
// (the shared-memory occupancy at 20 bins), up to 168 registers.
// 100 k x 500 k on the sky, theta_max 200': 13.7 ms for the call with the block-wide form, 10.34 now
// (two-edge path and items split by cell rows 10.8, warps on their own 10.67, the
// d2 - E form of the edge paths 10.34).
template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB>
__global__ void __launch_bounds__(64, 6) k_pairs_sph(const PairParams P) {
  constexpr int QA = (MODE == 0 && HAS_M) ? 6 : 5;
  constexpr bool SMALL = LOGB;  // log spacing on the sphere is only chosen with chord(x_max) <= 0.25
  const int nb = P.nb;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  extern __shared__ __align__(128) unsigned char smem[];
  double* e2s = reinterpret_cast<double*>(smem);
  float* e2f = reinterpret_cast<float*>(e2s + nb + 1);
  const SphWarpSmem W = sph_warp_smem(nb, QA);
  unsigned char* wb = smem + sph_edge_smem(nb) + (size_t)warp * W.total;
  ChunkS* ring = reinterpret_cast<ChunkS*>(wb + W.ring);
  float* hist = reinterpret_cast<float*>(wb + W.hist);
  double* wsum = reinterpret_cast<double*>(wb + W.wsum);
  double* fvw = reinterpret_cast<double*>(wb + W.fvw);
  double* fw = reinterpret_cast<double*>(wb + W.fw);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(wb + W.mbar);

  if (lane == 0) {
    for (int b = 0; b < kNbufS; ++b) mbar_init(&full_bar[b], 1);
    mbar_fence_init();
  }
  for (int i = tid; i <= nb; i += blockDim.x) {
    e2s[i] = P.e2[i];
    e2f[i] = P.e2f[i];
  }
  float* __restrict__ hcol = hist + lane;
  for (int e = 0; e < nb * QA; ++e) hcol[e * 32] = 0.f;
  __syncthreads();
  BinCtx C;
  C.A = P.binA; C.B = P.binB; C.eps = P.eps; C.one_m_eps = 1.f - P.eps;
  C.nb = nb; C.e2s = e2s; C.e2f = e2f;
  C.eps_rel = 4e-6f;
  C.lo_g = e2f[0] * (1.f - P.eps);
  C.hi_g = e2f[nb] * (1.f + P.eps);
  C.tiny = e2f[0] * 1e-9f;

  const uint32_t wait_limit = P.wait_limit ? P.wait_limit : kWaitPolls;
  int ring_t = 0;        // ring index of the next sub-chunk this warp consumes
  int issued_end = 0;    // ring index one past the last sub-chunk this warp issued
  bool aborted = false;  // a bounded wait ran out: consume and issue nothing more

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
    const ChunkS* __restrict__ src = reinterpret_cast<const ChunkS*>(G.sph);
    const int per = T.split / T.run, g = it.y / per;
    const int part = (it.y - g * per) * T.run + run_i++;  // its rows: every T.split-th
    const int gs = LD.group_start[g];
    const bool act = lane < LD.group_start[g + 1] - gs;
    LensS Lf;
    float lz = 0.f;
    double vw = 0.0, w = 0.0;
    double* lens_col = nullptr;
    if (act) {
      const float4 r = LD.rec[gs + lane];
      Lf = lens_frame(LD.pos[2 * (gs + lane)], LD.pos[2 * (gs + lane) + 1]);
      vw = (double)r.z * (double)r.w;
      w = (double)r.w;
      if (HAS_Z) lz = LD.z[gs + lane];
      if (P.lens_acc && T.lens_acc_off >= 0)
        lens_col = P.lens_acc + T.lens_acc_off + (size_t)(T.run > 1 ? 0 : part) * kQ * nb * LD.n_valid + gs + lane;
    } else {
      Lf = lens_frame(make_float4(1.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f));
    }
    const LensS2 LP = lens_pack(Lf);
    fvw[lane] = vw;
    fw[lane] = w;
    const size_t lens_stride = (size_t)LD.n_valid;
    for (int e = lane; e < kQ * nb; e += 32) wsum[e] = 0.0;
    int since_flush = 0;
    const float4 box = LD.group_box[g];
    int cy0, cy1;
    row_range(G, box, P.R, T.margin, cy0, cy1);
    float dl;
    bool full;
    sph_reach(G, box, P.R, T.margin, dl, full);

    for (int c0 = cy0 + part; c0 <= cy1 && !aborted; c0 += kRowsS * T.split) {
      int s0 = 0, s1 = 0;
      const int r = lane / 3, row = c0 + r * T.split;
      if (r < kRowsS && row <= cy1) {
        int2 sp[3];
        const int k = sph_row_spans(G, box, P.R, T.margin, row, dl, full, sp);
        const int j = lane - 3 * r;
        if (j < k) {
          const int2 v = j == 0 ? sp[0] : j == 1 ? sp[1] : sp[2];
          s0 = v.x;
          s1 = v.y > v.x ? v.y : v.x;
        }
      }
      const int ntr = tiles_of_span<1>(s0, s1);
      int incl = ntr;  // inclusive prefix of the sub-chunk counts over the lanes (runs)
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const int ntiles = __shfl_sync(0xffffffffu, incl, 31);
      auto issue = [&](int k) {
        const TileGeom tg = tile_of<1>(k, incl, ntr, s0, s1);
        const int t = ring_t + k;
        issued_end = t + 1;
        if (t + 1 == P.debug_skip_tile) return;  // fault injection (tests): this copy never lands
        if (lane == 0) {
          const int b = t % kNbufS;
          mbar_arrive_tx(&full_bar[b], (uint32_t)sizeof(ChunkS));
          bulk_g2s(ring + b, src + tg.c0, (uint32_t)sizeof(ChunkS), &full_bar[b]);
        }
      };
      for (int k = 0; k < kNbufS && k < ntiles; ++k) issue(k);
      for (int k = 0; k < ntiles; ++k) {
        const int t = ring_t + k;
        const int b = t % kNbufS;
        const TileGeom tg = tile_of<1>(k, incl, ntr, s0, s1);
        const bool ok = __all_sync(0xffffffffu,
                                   mbar_wait_bounded(&full_bar[b], (uint32_t)(t / kNbufS) & 1u, wait_limit));
        if (!ok) {  // stop: drain this warp's copies in flight below, report the timeout
          aborted = true;
          ring_t = t;
          break;
        }
        const ChunkS* ch = ring + b;
        const SrcPairS* __restrict__ Sc = ch->src;
        const int lo = tg.lo0, hi = tg.hiL;
        const bool partial = lo > 0 || hi < kChunk;
        int blo = 0;
        const int cls = act ? classify_s<LOGB>(Lf, ch->mn, ch->mx, C, blo) : 0;
        const int m = (int)__reduce_max_sync(0xffffffffu, (unsigned)cls);
        const float4 ss = ch->sum;
        if (m == 1) {
          if (partial)
            chunk_single_s<MODE, HAS_M, HAS_Z, SMALL, true, 32, QA>(Sc, lo, hi, LP, lz, C.tiny, cls, blo, hcol, ss);
          else
            chunk_single_s<MODE, HAS_M, HAS_Z, SMALL, false, 32, QA>(Sc, 0, kChunk, LP, lz, C.tiny, cls, blo, hcol, ss);
        } else if (m == 2) {
          if (partial)
            chunk_edges_s<MODE, HAS_M, HAS_Z, SMALL, true, 32, QA, 1>(Sc, lo, hi, Lf, LP, lz, cls, blo, hcol, C, ss);
          else
            chunk_edges_s<MODE, HAS_M, HAS_Z, SMALL, false, 32, QA, 1>(Sc, 0, kChunk, Lf, LP, lz, cls, blo, hcol, C,
                                                                       ss);
        } else if (m == 3) {
          if (partial)
            chunk_edges_s<MODE, HAS_M, HAS_Z, SMALL, true, 32, QA, 2>(Sc, lo, hi, Lf, LP, lz, cls, blo, hcol, C, ss);
          else
            chunk_edges_s<MODE, HAS_M, HAS_Z, SMALL, false, 32, QA, 2>(Sc, 0, kChunk, Lf, LP, lz, cls, blo, hcol, C,
                                                                       ss);
        } else if (m == 4 && act) {
          for (int j = lo; j < hi; ++j)
            do_pair_s<MODE, HAS_M, HAS_Z, LOGB, SMALL, 32, QA>(Lf, lz, src_of_s(Sc, j), hcol, C);
        }
        since_flush += hi - lo;
        __syncwarp();  // every lane is done reading buffer b
        if (k + kNbufS < ntiles) issue(k + kNbufS);
        if (since_flush >= T.flush_src) {
          warp_fold<QA, 32>(hist, hcol, wsum, fvw, fw, nb, lens_col, lens_stride, 0, lane);
          since_flush = 0;
        }
      }
      if (!aborted) ring_t += ntiles;
    }
    if (aborted) break;
    warp_fold<QA, 32>(hist, hcol, wsum, fvw, fw, nb, lens_col, lens_stride, 0, lane);
    double* out = P.item_sums + (size_t)(T.item_base + g * T.split + part) * kQ * nb;
    for (int e = lane; e < kQ * nb; e += 32) {
      const int from = (e / nb == QK && QA == 5) ? e - (QK - QW) * nb : e;
      out[e] = wsum[from];
    }
    __syncwarp();
  }
  if (aborted) {
    // wait (bounded) for the copies this warp issued and did not consume, so that
    // none is in flight when the block's shared memory is released
    for (int t = ring_t; t < issued_end; ++t)
      if (t + 1 != P.debug_skip_tile) mbar_wait_bounded(&full_bar[t % kNbufS], (uint32_t)(t / kNbufS) & 1u, wait_limit);
    if (lane == 0) atomicOr(P.err, kErrTimeout);
  }
}

// ------------------------------------------------------------ prep kernels --
// lambda reduced to [0, 2 pi) (FP32; used only for the cell grid and the
// lens ordering, never in the pair arithmetic).
__global__ void k_wrap_lambda(const float* __restrict__ x, long long n, float* out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = x[i];
    float t = v - kTwoPiF * floorf(v * 0.159154937f);
    if (t < 0.f) t += kTwoPiF;
    if (t >= kTwoPiF) t -= kTwoPiF;
    out[i] = t;
  }
}

// Cell-sorted sub-chunks: one warp per 32 sources (lanes 2k, 2k+1 trade halves
// with one shuffle round).  Past the last source the last one is repeated; such
// copies are outside every row span.
__global__ void k_src_gather_sph(const int* __restrict__ idx, int n_valid, int n_chunks, int mode,
                                 const float* __restrict__ lam, const float* __restrict__ phi,
                                 const float* __restrict__ z, const float* __restrict__ f1,
                                 const float* __restrict__ f2, const float* __restrict__ w,
                                 const float* __restrict__ m, ChunkS* __restrict__ out) {
  const int ch = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (ch >= n_chunks) return;  // whole warps
  const int s = ch * kChunk + lane;
  const bool real = s < n_valid;
  const int i = idx[real ? s : n_valid - 1];
  const float wi = w[i];
  float4 a, b;
  canon_unit(lam[i], phi[i], a, b);
  float K = wi, zi = 0.f;
  if (mode == 0) {
    a.w = -(f1[i] * wi);
    b.w = -(f2[i] * wi);
    K = wi * (1.0f + (m ? m[i] : 0.f));
    zi = z ? z[i] : 0.f;
  } else {
    a.w = f1[i] * wi;
    b.w = f2[i] * wi;
  }
  const bool odd = lane & 1;
  // even lane keeps {hi.x, hi.y, hi.z, p, lo.x, lo.y} of both, odd lane {lo.z, q, w, K, z}
  const float r0 = __shfl_xor_sync(0xffffffffu, odd ? a.x : b.z, 1);
  const float r1 = __shfl_xor_sync(0xffffffffu, odd ? a.y : b.w, 1);
  const float r2 = __shfl_xor_sync(0xffffffffu, odd ? a.z : wi, 1);
  const float r3 = __shfl_xor_sync(0xffffffffu, odd ? a.w : K, 1);
  const float r4 = __shfl_xor_sync(0xffffffffu, odd ? b.x : zi, 1);
  const float r5 = __shfl_xor_sync(0xffffffffu, b.y, 1);
  SrcPairS* dst = out[ch].src + (lane >> 1);
  if (!odd) {
    dst->hxy = make_float4(a.x, r0, a.y, r1);
    dst->hzp = make_float4(a.z, r2, a.w, r3);
    dst->lxy = make_float4(b.x, r4, b.y, r5);
  } else {
    dst->lzq = make_float4(r0, b.z, r1, b.w);
    dst->wk = make_float4(r2, wi, r3, K);
    dst->zz = make_float4(r4, zi, 0.f, 0.f);
  }
  float s0 = real ? a.w : 0.f, s1 = real ? b.w : 0.f, s2 = real ? wi : 0.f, s3 = real ? K : 0.f;
  float mnx = a.x, mny = a.y, mnz = a.z, mxx = a.x, mxy = a.y, mxz = a.z;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    s3 += __shfl_xor_sync(0xffffffffu, s3, o);
    mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
    mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
    mnz = fminf(mnz, __shfl_xor_sync(0xffffffffu, mnz, o));
    mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
    mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
    mxz = fmaxf(mxz, __shfl_xor_sync(0xffffffffu, mxz, o));
  }
  if (lane == 0) {
    const float d = 1.1920929e-7f;
    out[ch].mn = make_float4(mnx - d, mny - d, mnz - d, 0.f);
    out[ch].mx = make_float4(mxx + d, mxy + d, mxz + d, 0.f);
    out[ch].sum = make_float4(s0, s1, s2, s3);
  }
}

// Unit vectors (hi, lo) of the sorted lenses; perm[s] = input index.
__global__ void k_lens_pos_sph(const int* __restrict__ perm, int n_valid, const float* __restrict__ lam,
                               const float* __restrict__ phi, float4* pos) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_valid) return;
  const int i = perm[s];
  float4 hi, lo;
  canon_unit(lam[i], phi[i], hi, lo);
  pos[2 * s] = hi;
  pos[2 * s + 1] = lo;
}

// Unit vectors (hi, lo) in input order (tests and diagnostics).
__global__ void k_unit_vectors(const float* __restrict__ lam, const float* __restrict__ phi, long long n,
                               float* hi, float* lo) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float4 h, l;
    canon_unit(lam[i], phi[i], h, l);
    hi[3 * i] = h.x; hi[3 * i + 1] = h.y; hi[3 * i + 2] = h.z;
    lo[3 * i] = l.x; lo[3 * i + 1] = l.y; lo[3 * i + 2] = l.z;
  }
}

__global__ void k_item_cost_sph(const int2* __restrict__ ranges, int n_ranges, int n_items,
                                const TaskDesc* __restrict__ tasks, const LensDesc* __restrict__ lenses,
                                const GridDesc* __restrict__ grids, float R, int2* __restrict__ items,
                                unsigned* __restrict__ band) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_items) return;
  const int2 it = item_at(ranges, n_ranges, i);
  const TaskDesc T = tasks[it.x];
  const LensDesc L = lenses[T.lens_cat];
  const GridDesc G = grids[T.src_cat];
  const int per = T.split / T.run, g = it.y / per, part = it.y - g * per;
  const float4 box = L.group_box[g];
  int cy0, cy1;
  row_range(G, box, R, T.margin, cy0, cy1);
  float dl;
  bool full;
  sph_reach(G, box, R, T.margin, dl, full);
  unsigned long long s = 0;
  for (int cy = cy0 + part; cy <= cy1; cy += per) {
    int2 sp[3];
    const int k = sph_row_spans(G, box, R, T.margin, cy, dl, full, sp);
    for (int j = 0; j < k; ++j)
      if (sp[j].y > sp[j].x) s += (unsigned long long)(sp[j].y - sp[j].x);
  }
  const unsigned long long nl = (unsigned long long)(L.group_start[g + 1] - L.group_start[g]);
  items[i] = it;
  band[i] = cost_band(s * nl + 1);
}

// --------------------------------------------------------- host launchers --
template <int MODE, bool HAS_M, bool HAS_Z, bool LOGB>
static cudaError_t launch_sph_t(const PairParams& P, int num_sms, cudaStream_t st, int* grid_out) {
  constexpr int QA = (MODE == 0 && HAS_M) ? 6 : 5;
  const size_t per = sph_warp_smem(P.nb, QA).total;
  const int bt = sph_edge_smem(P.nb) + 2 * per <= 113 * 1024 ? 64 : 32;  // two blocks per SM at least
  const size_t smem = sph_edge_smem(P.nb) + per * (bt / 32);
  auto kern = k_pairs_sph<MODE, HAS_M, HAS_Z, LOGB>;
  cudaError_t e = allow_dynamic_smem(kern);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, bt, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const int need = (P.n_items + bt / 32 - 1) / (bt / 32);  // each warp takes items of its own
  const int grid = max(1, min(per_sm * num_sms, need));
  *grid_out = grid;
  kern<<<grid, bt, smem, st>>>(P);
  return cudaGetLastError();
}

cudaError_t launch_pairs_sph(const PairParams& P, int mode, bool has_m, bool has_z, bool logb, int num_sms,
                             cudaStream_t st, int* grid) {
  if (mode == 1)
    return logb ? launch_sph_t<1, false, false, true>(P, num_sms, st, grid)
                : launch_sph_t<1, false, false, false>(P, num_sms, st, grid);
  if (has_m) {
    if (has_z) return logb ? launch_sph_t<0, true, true, true>(P, num_sms, st, grid)
                           : launch_sph_t<0, true, true, false>(P, num_sms, st, grid);
    return logb ? launch_sph_t<0, true, false, true>(P, num_sms, st, grid)
                : launch_sph_t<0, true, false, false>(P, num_sms, st, grid);
  }
  if (has_z) return logb ? launch_sph_t<0, false, true, true>(P, num_sms, st, grid)
                         : launch_sph_t<0, false, true, false>(P, num_sms, st, grid);
  return logb ? launch_sph_t<0, false, false, true>(P, num_sms, st, grid)
              : launch_sph_t<0, false, false, false>(P, num_sms, st, grid);
}

size_t sph_src_bytes(int n_valid) { return sizeof(ChunkS) * (size_t)max((n_valid + kChunk - 1) / kChunk, 1); }

static inline unsigned gdim_s(long long n, int b) {
  long long g = (n + b - 1) / b;
  if (g < 1) g = 1;
  if (g > 148 * 32) g = 148 * 32;
  return (unsigned)g;
}

cudaError_t launch_wrap_lambda(const float* x, long long n, float* out, cudaStream_t st) {
  if (n > 0) k_wrap_lambda<<<gdim_s(n, 256), 256, 0, st>>>(x, n, out);
  return cudaGetLastError();
}
cudaError_t launch_src_gather_sph(const int* idx, int n_valid, int mode, const float* lam, const float* phi,
                                  const float* z, const float* f1, const float* f2, const float* w, const float* m,
                                  void* out, cudaStream_t st) {
  const int n_chunks = (n_valid + kChunk - 1) / kChunk;
  if (n_chunks > 0)
    k_src_gather_sph<<<(n_chunks + 7) / 8, 256, 0, st>>>(idx, n_valid, n_chunks, mode, lam, phi, z, f1, f2, w, m,
                                                          static_cast<ChunkS*>(out));
  return cudaGetLastError();
}
cudaError_t launch_lens_pos_sph(const int* perm, int n_valid, const float* lam, const float* phi, float4* pos,
                                cudaStream_t st) {
  if (n_valid > 0) k_lens_pos_sph<<<(n_valid + 255) / 256, 256, 0, st>>>(perm, n_valid, lam, phi, pos);
  return cudaGetLastError();
}
cudaError_t launch_unit_vectors(const float* lam, const float* phi, long long n, float* hi, float* lo,
                                cudaStream_t st) {
  if (n > 0) k_unit_vectors<<<gdim_s(n, 256), 256, 0, st>>>(lam, phi, n, hi, lo);
  return cudaGetLastError();
}
cudaError_t launch_item_cost_sph(const int2* ranges, int n_ranges, int n_items, const TaskDesc* tasks,
                                 const LensDesc* lenses, const GridDesc* grids, float R, int2* items, unsigned* band,
                                 cudaStream_t st) {
  if (n_items > 0)
    k_item_cost_sph<<<(n_items + 127) / 128, 128, 0, st>>>(ranges, n_ranges, n_items, tasks, lenses, grids, R, items,
                                                            band);
  return cudaGetLastError();
}

}  // namespace tpcf
