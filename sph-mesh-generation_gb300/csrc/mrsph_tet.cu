// mrsph_tet.cu — 3D tetrahedralisation of the particles and tet quality (row F3).
//
//   Graphmeshcls::Reconstruct_tets (graph_mesh.cpp:981-1100) hands every
//   particle to TetGen (a Delaunay tetrahedralisation of the convex hull) and
//   drops the tets Check_whether_this_tet_should_be_delete (:675-979) names:
//   all four particles not REAL and aspect ratio above tet_delete_thres = 10
//   (its phi tests are commented out).
//     -> k_tet_star: local Delaunay stars, one warp per particle.  Particle
//        i gift-wraps the tets around itself over its neighbour row, which
//        holds every particle within cutoff * h_i, walking its whole star in
//        the row's Delaunay tetrahedralisation.  A tet is certified when its
//        circumsphere lies inside that ball and no row particle lies inside
//        or on it; then no particle at all does, so it is a Delaunay tet of
//        the whole set and the unique one through its four particles.  Each
//        certified tet is emitted once, by the lowest-id particle whose ball
//        holds it.  Tets that no ball holds (across concavities of the body
//        and on the convex hull, where TetGen keeps large tets) are not
//        produced.
//   Graphmeshcls::Tet_quality_statistics (:1967-2400) -> k_tet_quality: the
//   volume, edge, aspect-ratio, radius-ratio and dihedral-angle statistics
//   and histograms of the kept tets.
// Positions are snapped to the grid 2^(e-52), e the exponent that bounds the
// domain, so that every coordinate is both an exact double and an exact
// integer.  Predicate signs come from an FP64 evaluation with a conservative
// error bound (the permanent bounds of Shewchuk, "Adaptive Precision
// Floating-Point Arithmetic and Fast Robust Geometric Predicates", 1997) and,
// when the bound cannot decide, from exact 320-bit integer arithmetic, so the
// tets do not depend on evaluation order.  Compiled with -fmad=false.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "handle.h"

namespace mrsph {
namespace {

// ------------------------------------------------------------ 320-bit integers
// Two's complement, little-endian 64-bit limbs; wide enough for the insphere
// determinant of 54-bit coordinate differences (< 2^277).
constexpr int BL = 5;
struct BI {
  unsigned long long w[BL];
};

__device__ inline BI bi_from(long long v) {
  BI r;
  const unsigned long long s = v < 0 ? ~0ull : 0ull;
  r.w[0] = (unsigned long long)v;
  for (int k = 1; k < BL; k++) r.w[k] = s;
  return r;
}
__device__ inline BI bi_add(const BI& a, const BI& b) {
  BI r;
  unsigned long long c = 0;
  for (int k = 0; k < BL; k++) {
    const unsigned long long s = a.w[k] + b.w[k];
    const unsigned long long c1 = s < a.w[k];
    r.w[k] = s + c;
    c = c1 | (r.w[k] < s);
  }
  return r;
}
__device__ inline BI bi_neg(const BI& a) {
  BI r;
  unsigned long long c = 1;
  for (int k = 0; k < BL; k++) {
    r.w[k] = ~a.w[k] + c;
    c = (c && r.w[k] == 0) ? 1 : 0;
  }
  return r;
}
__device__ inline BI bi_sub(const BI& a, const BI& b) { return bi_add(a, bi_neg(b)); }
__device__ inline bool bi_negative(const BI& a) { return (long long)a.w[BL - 1] < 0; }
__device__ inline int bi_sign(const BI& a) {
  if (bi_negative(a)) return -1;
  for (int k = 0; k < BL; k++)
    if (a.w[k]) return 1;
  return 0;
}
// a * b, both |.| < 2^(64 BL - 1) with the product in range
__device__ BI bi_mul(const BI& a, const BI& b) {
  const bool na = bi_negative(a), nb = bi_negative(b);
  const BI ua = na ? bi_neg(a) : a, ub = nb ? bi_neg(b) : b;
  BI r;
  for (int k = 0; k < BL; k++) r.w[k] = 0;
  for (int i = 0; i < BL; i++) {
    if (!ua.w[i]) continue;
    unsigned long long carry = 0;
    for (int j = 0; i + j < BL; j++) {
      const unsigned long long lo = ua.w[i] * ub.w[j], hi = __umul64hi(ua.w[i], ub.w[j]);
      unsigned long long s = r.w[i + j] + lo;
      unsigned long long c = s < lo;
      s += carry;
      c += s < carry;
      r.w[i + j] = s;
      carry = hi + c;
    }
  }
  return (na != nb) ? bi_neg(r) : r;
}

// ------------------------------------------------------------ predicates
// Points are snapped doubles; I = integer coordinates (x / grid).
struct Pt {
  double x, y, z;
};
constexpr double kEps = 1.1102230246251565e-16;  // 2^-53
// Conservative error-bound factors of the FP64 evaluations below (the
// published bounds are 7 eps and 16 eps of the same permanents).
constexpr double kO3Bound = 16.0 * kEps;
constexpr double kIsBound = 64.0 * kEps;

__device__ inline long long ival(double v, double inv_g) { return __double2ll_rn(v * inv_g); }

// orient3d(a, b, c, d) = det[a - d; b - d; c - d]: > 0 when d lies below the
// plane of a, b, c seen counter-clockwise from above.
__device__ __noinline__ int orient_x(const Pt& a, const Pt& b, const Pt& c, const Pt& d, double ig) {
  const long long adx = ival(a.x, ig) - ival(d.x, ig), ady = ival(a.y, ig) - ival(d.y, ig),
                  adz = ival(a.z, ig) - ival(d.z, ig);
  const long long bdx = ival(b.x, ig) - ival(d.x, ig), bdy = ival(b.y, ig) - ival(d.y, ig),
                  bdz = ival(b.z, ig) - ival(d.z, ig);
  const long long cdx = ival(c.x, ig) - ival(d.x, ig), cdy = ival(c.y, ig) - ival(d.y, ig),
                  cdz = ival(c.z, ig) - ival(d.z, ig);
  const BI m1 = bi_sub(bi_mul(bi_from(bdy), bi_from(cdz)), bi_mul(bi_from(bdz), bi_from(cdy)));
  const BI m2 = bi_sub(bi_mul(bi_from(cdy), bi_from(adz)), bi_mul(bi_from(cdz), bi_from(ady)));
  const BI m3 = bi_sub(bi_mul(bi_from(ady), bi_from(bdz)), bi_mul(bi_from(adz), bi_from(bdy)));
  const BI det = bi_add(bi_add(bi_mul(bi_from(adx), m1), bi_mul(bi_from(bdx), m2)), bi_mul(bi_from(cdx), m3));
  return bi_sign(det);
}
__device__ __noinline__ int orient3d(const Pt& a, const Pt& b, const Pt& c, const Pt& d, double ig) {
  const double adx = a.x - d.x, ady = a.y - d.y, adz = a.z - d.z;
  const double bdx = b.x - d.x, bdy = b.y - d.y, bdz = b.z - d.z;
  const double cdx = c.x - d.x, cdy = c.y - d.y, cdz = c.z - d.z;
  const double p1 = bdy * cdz, p2 = bdz * cdy, p3 = cdy * adz, p4 = cdz * ady, p5 = ady * bdz, p6 = adz * bdy;
  const double det = adx * (p1 - p2) + bdx * (p3 - p4) + cdx * (p5 - p6);
  const double perm = fabs(adx) * (fabs(p1) + fabs(p2)) + fabs(bdx) * (fabs(p3) + fabs(p4)) +
                      fabs(cdx) * (fabs(p5) + fabs(p6));
  const double bound = kO3Bound * perm;
  if (det > bound) return 1;
  if (-det > bound) return -1;
  return orient_x(a, b, c, d, ig);
}

// insphere(a, b, c, d, e) > 0 when e lies inside the sphere through a, b, c,
// d and orient3d(a, b, c, d) > 0 (the sign flips with the orientation).
__device__ __noinline__ int insphere_x(const Pt& a, const Pt& b, const Pt& c, const Pt& d, const Pt& e, double ig) {
  const long long ex = ival(e.x, ig), ey = ival(e.y, ig), ez = ival(e.z, ig);
  const long long aex = ival(a.x, ig) - ex, aey = ival(a.y, ig) - ey, aez = ival(a.z, ig) - ez;
  const long long bex = ival(b.x, ig) - ex, bey = ival(b.y, ig) - ey, bez = ival(b.z, ig) - ez;
  const long long cex = ival(c.x, ig) - ex, cey = ival(c.y, ig) - ey, cez = ival(c.z, ig) - ez;
  const long long dex = ival(d.x, ig) - ex, dey = ival(d.y, ig) - ey, dez = ival(d.z, ig) - ez;
  auto M = [](long long p, long long q) { return bi_mul(bi_from(p), bi_from(q)); };
  auto lift = [&](long long x, long long y, long long z) { return bi_add(bi_add(M(x, x), M(y, y)), M(z, z)); };
  const BI ab = bi_sub(M(aex, bey), M(bex, aey)), bc = bi_sub(M(bex, cey), M(cex, bey));
  const BI cd = bi_sub(M(cex, dey), M(dex, cey)), da = bi_sub(M(dex, aey), M(aex, dey));
  const BI ac = bi_sub(M(aex, cey), M(cex, aey)), bd = bi_sub(M(bex, dey), M(dex, bey));
  const BI az = bi_from(aez), bz = bi_from(bez), cz = bi_from(cez), dz = bi_from(dez);
  const BI abc = bi_add(bi_sub(bi_mul(az, bc), bi_mul(bz, ac)), bi_mul(cz, ab));
  const BI bcd = bi_add(bi_sub(bi_mul(bz, cd), bi_mul(cz, bd)), bi_mul(dz, bc));
  const BI cda = bi_add(bi_add(bi_mul(cz, da), bi_mul(dz, ac)), bi_mul(az, cd));
  const BI dab = bi_add(bi_add(bi_mul(dz, ab), bi_mul(az, bd)), bi_mul(bz, da));
  const BI det = bi_add(bi_sub(bi_mul(lift(dex, dey, dez), abc), bi_mul(lift(cex, cey, cez), dab)),
                        bi_sub(bi_mul(lift(bex, bey, bez), cda), bi_mul(lift(aex, aey, aez), bcd)));
  return bi_sign(det);
}
__device__ __noinline__ int insphere(const Pt& a, const Pt& b, const Pt& c, const Pt& d, const Pt& e, double ig) {
  const double aex = a.x - e.x, aey = a.y - e.y, aez = a.z - e.z;
  const double bex = b.x - e.x, bey = b.y - e.y, bez = b.z - e.z;
  const double cex = c.x - e.x, cey = c.y - e.y, cez = c.z - e.z;
  const double dex = d.x - e.x, dey = d.y - e.y, dez = d.z - e.z;
  const double ab1 = aex * bey, ab2 = bex * aey, bc1 = bex * cey, bc2 = cex * bey;
  const double cd1 = cex * dey, cd2 = dex * cey, da1 = dex * aey, da2 = aex * dey;
  const double ac1 = aex * cey, ac2 = cex * aey, bd1 = bex * dey, bd2 = dex * bey;
  const double ab = ab1 - ab2, bc = bc1 - bc2, cd = cd1 - cd2, da = da1 - da2, ac = ac1 - ac2, bd = bd1 - bd2;
  const double abc = aez * bc - bez * ac + cez * ab;
  const double bcd = bez * cd - cez * bd + dez * bc;
  const double cda = cez * da + dez * ac + aez * cd;
  const double dab = dez * ab + aez * bd + bez * da;
  const double al = aex * aex + aey * aey + aez * aez, bl = bex * bex + bey * bey + bez * bez;
  const double cl = cex * cex + cey * cey + cez * cez, dl = dex * dex + dey * dey + dez * dez;
  const double det = (dl * abc - cl * dab) + (bl * cda - al * bcd);
  const double Pab = fabs(ab1) + fabs(ab2), Pbc = fabs(bc1) + fabs(bc2), Pcd = fabs(cd1) + fabs(cd2);
  const double Pda = fabs(da1) + fabs(da2), Pac = fabs(ac1) + fabs(ac2), Pbd = fabs(bd1) + fabs(bd2);
  const double Pabc = fabs(aez) * Pbc + fabs(bez) * Pac + fabs(cez) * Pab;
  const double Pbcd = fabs(bez) * Pcd + fabs(cez) * Pbd + fabs(dez) * Pbc;
  const double Pcda = fabs(cez) * Pda + fabs(dez) * Pac + fabs(aez) * Pcd;
  const double Pdab = fabs(dez) * Pab + fabs(aez) * Pbd + fabs(bez) * Pda;
  const double perm = dl * Pabc + cl * Pdab + bl * Pcda + al * Pbcd;
  const double bound = kIsBound * perm;
  if (det > bound) return 1;
  if (-det > bound) return -1;
  return insphere_x(a, b, c, d, e, ig);
}

// ------------------------------------------------------------ tet geometry
// Canonical evaluation over the ascending ids p[0] < p[1] < p[2] < p[3]:
// A_k = P_k - P_3, det = A_0 . (A_1 x A_2), circumcentre P_3 + c.
struct TetGeo {
  double A[3][3], det, c[3], rc, vol_scale;
};
__device__ inline void cross3(const double* u, const double* v, double* w) {
  w[0] = u[1] * v[2] - u[2] * v[1];
  w[1] = u[2] * v[0] - u[0] * v[2];
  w[2] = u[0] * v[1] - u[1] * v[0];
}
__device__ inline double dot3(const double* u, const double* v) { return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]; }

__device__ __noinline__ void tet_geo(const Pt* P, TetGeo& g) {
  const double* p3 = &P[3].x;
  for (int k = 0; k < 3; k++) {
    const double* pk = &P[k].x;
    for (int q = 0; q < 3; q++) g.A[k][q] = pk[q] - p3[q];
  }
  double x12[3], x20[3], x01[3];
  cross3(g.A[1], g.A[2], x12);
  cross3(g.A[2], g.A[0], x20);
  cross3(g.A[0], g.A[1], x01);
  g.det = dot3(g.A[0], x12);
  const double r0 = 0.5 * dot3(g.A[0], g.A[0]), r1 = 0.5 * dot3(g.A[1], g.A[1]), r2 = 0.5 * dot3(g.A[2], g.A[2]);
  for (int q = 0; q < 3; q++) g.c[q] = (r0 * x12[q] + r1 * x20[q] + r2 * x01[q]) / g.det;
  g.rc = sqrt(dot3(g.c, g.c));
  g.vol_scale = sqrt(dot3(g.A[0], g.A[0])) * sqrt(dot3(g.A[1], g.A[1])) * sqrt(dot3(g.A[2], g.A[2]));
}

// Circumsphere inside the certificate ball of the particle at x with
// smoothing length h; flat tets (|det| below 1e-6 of the edge-length
// product) are never certified.
__device__ inline bool tet_in_ball(const TetGeo& g, const Pt* P, const double* x, double h, double cutoff) {
  if (!(fabs(g.det) >= 1.e-6 * g.vol_scale)) return false;
  double v[3];
  const double* p3 = &P[3].x;
  for (int q = 0; q < 3; q++) v[q] = p3[q] + g.c[q] - x[q];
  return sqrt(dot3(v, v)) + g.rc <= cutoff * h * (1.0 - 1.e-6);
}

__device__ inline void sort4(int* v) {
  for (int a = 1; a < 4; a++)
    for (int b = a; b > 0 && v[b - 1] > v[b]; b--) {
      const int t = v[b];
      v[b] = v[b - 1];
      v[b - 1] = t;
    }
}

struct TetIn {
  long long n;
  int cap;
  const double* x;  // snapped positions (n x 3)
  const int* type;
  const double* h;
  const float* rf;  // FP32 radius of the certificate ball, cutoff h (1 - 1e-6)
  const int* rows;  // n x cap ids (list order; self may appear)
  const int* cnt;
  double inv_g;  // 1 / grid
  double cutoff;
  double thres;  // tet_delete_thres
};

__device__ inline Pt load_pt(const TetIn& T, int j) {
  const double* p = T.x + 3 * (long long)j;
  return Pt{p[0], p[1], p[2]};
}

// aspect = longest edge / smallest height (Check_whether_this_tet_should_be_delete,
// graph_mesh.cpp:900-970): longest edge * max_k |grad lambda_k|
__device__ double tet_aspect(const TetGeo& g, const Pt* P) {
  double n[4][3];
  cross3(g.A[1], g.A[2], n[0]);
  cross3(g.A[2], g.A[0], n[1]);
  cross3(g.A[0], g.A[1], n[2]);
  for (int k = 0; k < 3; k++)
    for (int q = 0; q < 3; q++) n[k][q] /= g.det;
  for (int q = 0; q < 3; q++) n[3][q] = -n[0][q] - n[1][q] - n[2][q];
  double hmax = 0.0;
  for (int k = 0; k < 4; k++) hmax = fmax(hmax, sqrt(dot3(n[k], n[k])));
  double e[3], longlen = 0.0;
  for (int k = 0; k < 3; k++) longlen = fmax(longlen, dot3(g.A[k], g.A[k]));
  const double* p0 = &P[0].x;
  const double* p1 = &P[1].x;
  const double* p2 = &P[2].x;
  for (int q = 0; q < 3; q++) e[q] = p1[q] - p0[q];
  longlen = fmax(longlen, dot3(e, e));
  for (int q = 0; q < 3; q++) e[q] = p2[q] - p1[q];
  longlen = fmax(longlen, dot3(e, e));
  for (int q = 0; q < 3; q++) e[q] = p0[q] - p2[q];
  longlen = fmax(longlen, dot3(e, e));
  return sqrt(longlen) * hmax;
}

constexpr int kMaxStar = 128;  // tets around one particle
constexpr int kMaxLink = 224;  // link edges around one particle
constexpr int kMaxOut = kMaxStar;  // tets emitted by one particle (at most its star)
// flags: 4 spilled neighbour row (a star that outgrows kMaxStar / kMaxLink stops
// its walk and is counted in stats[3])

constexpr unsigned kFull = 0xffffffffu;

// ------------------------------------------------------------ FP32 geometry
// The star is walked in FP32 relative to particle i (w = x_j - x_i, rounded
// once, kept in shared memory for the whole star), with an error bound beside
// every value: a decision is taken from FP32 only when it clears its bound, and
// from the exact predicates otherwise, so every decision equals the exact one.
// Lengths are taken in units of the power of two at the radius of i's ball: up
// to six of them are multiplied, and in the body's own units a spacing of 3e-8
// would already leave FP32's range.  Points far closer to one another than to
// the ball's size can still do so: products that come near it decide nothing.
// FP64 runs at 1/60 of the FP32 rate on this part: with the candidates' FP64
// differences, an FP64 circumcentre per tet and a second scan of the row per
// tet the pass took 142.9 ms for 150,001 particles (830,000 tets); in this
// form it takes 7.5 ms, bound by instruction issue and latency.
constexpr float kE = 0x1p-24f;
constexpr int kRowS = 256;  // row entries kept in shared memory; longer rows read the rest from the positions

struct V3 {
  float x, y, z;
};
__device__ inline V3 vcross(const V3& a, const V3& b) {
  return V3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ inline float vdot(const V3& a, const V3& b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); }

struct Star {  // one warp's particle
  float4 w[kRowS];  // (w, |w|); x is NaN for the particle itself
  int tet[kMaxStar][3];  // row slots
  float rc2[kMaxStar], band[kMaxStar];  // circumsphere diameter and its error bound
  int le[kMaxLink][2];
  unsigned char done[kMaxLink], cert[kMaxStar];
};

struct StarRow {
  const TetIn& T;
  const int* S;  // the row's ids
  int i, m;
  Pt pi;
  float sc;  // the unit of length, inverted
  const Star& sm;
  __device__ float4 make(int q) const {
    const int j = S[q];
    const Pt p = load_pt(T, j);
    const float x = (float)(p.x - pi.x) * sc, y = (float)(p.y - pi.y) * sc, z = (float)(p.z - pi.z) * sc;
    return make_float4(j == i ? __int_as_float(0x7fffffff) : x, y, z, sqrtf(fmaf(z, z, fmaf(y, y, x * x))));
  }
  __device__ float4 at(int q) const { return q < kRowS ? sm.w[q] : make(q); }
  __device__ Pt pt(int q) const { return load_pt(T, S[q]); }
};

// Orders floats as ints do (for __reduce_min_sync).
__device__ inline int ford(float v) {
  const int b = __float_as_int(v);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
// 2^-k for v in [2^k, 2^(k + 1)); 1 where FP32 has no such number
__device__ inline float inv_pow2(float v) {
  const int e = (__float_as_int(v) >> 23) & 0xff;
  return e >= 1 && e <= 253 ? __int_as_float((254 - e) << 23) : 1.f;
}
__device__ inline float funord(int b) { return __int_as_float(b >= 0 ? b : b ^ 0x7fffffff); }

struct Face {  // the pencil of spheres through i, u, v: centres c0 + sigma t n
  V3 n, c0;
  float sigma, nn, cO, cP, dc0, L;  // |n|; bounds per |w| of n . w and of the power; of c0; |A| + |B|
};
// Bounds, with e = 2^-24, k = |A||B| / |n| and L = |A| + |B|: n is off by at most
// 4 e |A||B|, c0 by 22 e k^2 L (its formula's rounding 14, the rounding of A and
// B 8), n . w by 8 e |A||B||w|, the power |w|^2 - 2 w . c0 by e (8 |w|^2 + 48 k^2 L |w|).
// The constants below are at least a third larger.  They are relative to the
// products they bound, so a face whose products come near FP32's smallest numbers
// has no bound: |n|^2 above 1e-22 keeps both lengths above 1e-12 (rows reach a few
// radii of the ball), and no bound on n . w is one on nothing else either.
constexpr float kTiny = 1.e-22f;
__device__ inline Face face_of(const float4& A4, const float4& B4, float sigma) {
  Face F;
  const V3 A{A4.x, A4.y, A4.z}, B{B4.x, B4.y, B4.z};
  F.n = vcross(A, B);
  const float n2 = vdot(F.n, F.n), a2 = A4.w * A4.w, b2 = B4.w * B4.w;
  const V3 p = vcross(B, F.n), q = vcross(F.n, A);
  const float inv = 0.5f / n2;
  F.c0 = V3{(a2 * p.x + b2 * q.x) * inv, (a2 * p.y + b2 * q.y) * inv, (a2 * p.z + b2 * q.z) * inv};
  F.sigma = sigma;
  F.nn = sqrtf(n2);
  const float ab = A4.w * B4.w, k = ab / F.nn;
  F.L = A4.w + B4.w;
  F.cO = n2 > kTiny ? 16.f * kE * ab : __int_as_float(0x7f800000);
  F.cP = 64.f * kE * k * k * F.L;
  F.dc0 = 32.f * kE * k * k * F.L;
  return F;
}

struct Wrap {
  int d;         // row slot of the winner, -1 when no row particle lies on the side
  float t, et;   // its place on the pencil, and the bound
  float o;       // sigma n . w
  bool tie;      // another row particle lies on its sphere
};

// Gift-wraps the face (i, u, v) to side s (s * orient3d(i, u, v, d) > 0), one
// warp over the row: the candidate whose sphere through i, u, v holds no other
// candidate.  Along the pencil "e inside the sphere of d" is t_e < t_d, t =
// power / (2 sigma n . w), so the winner is the smallest t.  FP32 gives each
// candidate an interval; when only one reaches below the smallest upper end it
// has won, else the exact insphere signs decide among those that do.
__device__ Wrap wrap(const StarRow& R, const Face& F, int u, int v, int s, int lane) {
  const float INF = __int_as_float(0x7f800000);
  float lo1 = INF, lo2 = INF, H = INF;
  int q1 = -1;
  // interval of candidate q; false when it lies on the other side
  auto interval = [&](int q, float& lo, float& hi) -> bool {
    if (q == u || q == v) return false;
    const float4 w = R.at(q);
    const V3 w3{w.x, w.y, w.z};
    const float o = F.sigma * vdot(F.n, w3), eo = F.cO * w.w;
    if (!(o > -eo)) {
      if (o <= -eo || w.x != w.x) return false;  // certainly beyond the face; the particle itself
    }
    if (!(o > 2.f * eo)) {
      if (w.x != w.x) return false;
      const Pt pu = R.pt(u), pv = R.pt(v), pd = R.pt(q);
      if (s * orient3d(R.pi, pu, pv, pd, R.T.inv_g) <= 0) return false;
      lo = -INF;
      hi = INF;
      return true;
    }
    const float n2 = w.w * w.w;
    const float p = fmaf(-2.f, vdot(w3, F.c0), n2);
    const float r = __fdividef(0.5f, o);
    const float t = p * r;
    const float et = 2.f * (fmaf(16.f * kE, n2, F.cP * w.w) * r + 2.f * fabsf(t) * eo * r) + 4.f * kE * fabsf(t);
    lo = t - et;
    hi = t + et;
    if (!(lo <= hi)) { lo = -INF; hi = INF; }  // no usable bound (a face too thin for FP32)
    return true;
  };
  for (int q = lane; q < R.m; q += 32) {
    float lo, hi;
    if (!interval(q, lo, hi)) continue;
    if (q1 < 0 || lo < lo1) { lo2 = q1 < 0 ? INF : lo1; lo1 = lo; q1 = q; }
    else lo2 = fminf(lo2, lo);
    H = fminf(H, hi);
  }
  Wrap W;
  W.tie = false;
  const float Hm = funord(__reduce_min_sync(kFull, ford(H)));
  const unsigned cand = __ballot_sync(kFull, q1 >= 0 && lo1 <= Hm);
  const bool more = __any_sync(kFull, lo2 <= Hm && q1 >= 0 && lo2 < INF);
  if (!cand) {
    W.d = -1;
    return W;
  }
  int best;
  if (__popc(cand) == 1 && !more) {
    best = __shfl_sync(kFull, q1, __ffs(cand) - 1);
  } else {
    // exact: every candidate that reaches below the smallest upper end, in row order
    best = -1;
    const Pt pu = R.pt(u), pv = R.pt(v);
    for (int q0 = 0; q0 < R.m; q0 += 32) {
      const int q = q0 + lane;
      float lo = INF, hi;
      bool in = q < R.m && interval(q, lo, hi);
      in = in && lo <= Hm;
      unsigned mask = __ballot_sync(kFull, in);
      while (mask) {
        const int d = q0 + __ffs(mask) - 1;
        mask &= mask - 1u;
        if (best < 0) {
          best = d;
          continue;
        }
        const int sg = s * insphere(R.pi, pu, pv, R.pt(best), R.pt(d), R.T.inv_g);
        if (sg > 0) { best = d; W.tie = false; }
        else if (sg == 0) W.tie = true;
      }
    }
  }
  W.d = best;
  const float4 w = R.at(best);
  const V3 w3{w.x, w.y, w.z};
  const float eo = F.cO * w.w, n2 = w.w * w.w;
  W.o = F.sigma * vdot(F.n, w3);
  const float r = __fdividef(0.5f, W.o);
  W.t = fmaf(-2.f, vdot(w3, F.c0), n2) * r;
  W.et = W.o > 2.f * eo
             ? 2.f * (fmaf(16.f * kE, n2, F.cP * w.w) * r + 2.f * fabsf(W.t) * eo * r) + 4.f * kE * fabsf(W.t)
             : INF;
  return W;
}

// Whether the circumsphere of (i, u, v, d) lies inside i's ball and the tet is
// not flat (certified: a Delaunay tet of all particles once its sphere is
// empty); rc2, band: the sphere's diameter and its error bound.  All lanes
// agree.  The sphere passes through i, so it lies inside the ball when its
// diameter does not exceed the radius.  FP32 decides outside its bound, else
// the canonical FP64 evaluation (tet_in_ball) that the emission uses as well.
__device__ bool certified(const StarRow& R, const Face& F, const Wrap& W, int u, int v, float Ri, float& rc2,
                          float& band) {
  const float4 w = R.at(W.d);
  const float tn = W.t * F.nn, c2 = vdot(F.c0, F.c0);
  const float rc = sqrtf(fmaf(tn, tn, c2));
  rc2 = 2.f * rc;
  band = 2.f * (F.dc0 + F.nn * W.et + fabsf(W.t) * F.cO + 8.f * kE * rc) + 4.e-6f * Ri;
  const float Lm = fmaxf(F.L, w.w);
  const bool solid = W.o - F.cO * w.w > 1.e-5f * Lm * Lm * Lm;  // |det| above 1e-6 of the longest possible edge product
  if (solid && rc2 + band < Ri) return true;
  if (solid && rc2 - band > Ri) return false;
  int id[4] = {R.i, R.S[u], R.S[v], R.S[W.d]};
  sort4(id);
  Pt P[4];
  for (int k = 0; k < 4; k++) P[k] = load_pt(R.T, id[k]);
  TetGeo g;
  tet_geo(P, g);
  if (!solid) band = __int_as_float(0x7f800000);  // the emission decides in FP64 as well
  const double xi[3] = {R.pi.x, R.pi.y, R.pi.z};
  return tet_in_ball(g, P, xi, R.T.h[R.i], R.T.cutoff);
}

// No row particle inside or on the sphere of the star's first tet (i, u, v, d)
// (the faces of later tets border an empty sphere, see k_tet_star); *degen is
// set when row particles lie on it and none inside.
__device__ bool first_empty(const StarRow& R, const Face& F, const Wrap& W, int u, int v, int s, bool* degen, int lane) {
  const float st = F.sigma * W.t;
  const V3 c{fmaf(st, F.n.x, F.c0.x), fmaf(st, F.n.y, F.c0.y), fmaf(st, F.n.z, F.c0.z)};
  const float cn = sqrtf(vdot(c, c));
  const float dc = F.dc0 + F.nn * W.et + fabsf(W.t) * F.cO + 8.f * kE * cn;
  const Pt pu = R.pt(u), pv = R.pt(v), pd = R.pt(W.d);
  bool inside = false, on = false;
  for (int q = lane; q < R.m && !inside; q += 32) {
    if (q == u || q == v || q == W.d) continue;
    const float4 w = R.at(q);
    if (w.x != w.x) continue;
    const V3 w3{w.x, w.y, w.z};
    const float n2 = w.w * w.w, p = fmaf(-2.f, vdot(w3, c), n2);
    const float e = 16.f * kE * n2 + 2.f * w.w * (dc + 8.f * kE * cn);
    // insphere(i, u, v, d) is positive inside when orient3d(i, u, v, d) > 0, that is s > 0
    const int sg = p > e ? -1 : (p < -e ? 1 : s * insphere(R.pi, pu, pv, pd, R.pt(q), R.T.inv_g));
    if (sg > 0) inside = true;
    else if (sg == 0) on = true;
  }
  const bool any_in = __any_sync(kFull, inside), any_on = __any_sync(kFull, on);
  if (any_on && !any_in) *degen = true;
  return !any_in && !any_on;
}

constexpr int kStarWarps = 4;  // warps (particles) per block of k_tet_star

// One warp per particle (grid-stride): its certified star, the tets it
// emits (ascending ids, in star order) into out[i * kMaxOut ...], their
// number into count[i].  stats: [0] open stars, [1] deleted tets, [2] ties,
// [3] stars cut at the per-particle limits.
//
// A tet's sphere is scanned for row particles only once, for the first tet.
// Every later one is wrapped from a face of a tet whose sphere holds no row
// particle inside or on it: on the far side of the face the new sphere lies
// inside that one, on the near side no candidate lies inside the winner's, and
// one lies on it exactly when the wrap saw a tie.
//
// Four blocks of four warps per SM (128 registers): 7.5 ms for 150,001
// particles, 10.6 ms at six blocks (spills), 7.9 ms at three.
__global__ void __launch_bounds__(32 * kStarWarps, 4) k_tet_star(TetIn T, int* __restrict__ out,
                                                              int* __restrict__ count, unsigned long long* stats) {
  __shared__ Star s_star[kStarWarps];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Star& sm = s_star[wib];
  const long long nwarps = (long long)gridDim.x * kStarWarps;
  for (long long i64 = (long long)blockIdx.x * kStarWarps + wib; i64 < T.n; i64 += nwarps) {
    const int i = (int)i64;
    const float sc = inv_pow2(T.rf[i]);
    const StarRow R{T, T.rows + i64 * T.cap, i, T.cnt[i], load_pt(T, i), sc, sm};
    const int m = R.m;
    const float Ri = T.rf[i] * sc;
    bool degen = false, open = false, trunc = false;
    int ns = 0, nl = 0;
    for (int q = lane; q < min(m, kRowS); q += 32) sm.w[q] = R.make(q);
    __syncwarp();
    // 1. nearest neighbour a (ties: lower id) and the third point c of the
    // smallest circumcircle through i and a (ties: lower id), by FP64
    // values, which only the candidates near the FP32 minimum need
    const float INF = __int_as_float(0x7f800000);
    float dm = INF;
    for (int q = lane; q < m; q += 32) {
      const float4 w = R.at(q);
      if (w.x == w.x) dm = fminf(dm, w.w);
    }
    dm = __int_as_float(__reduce_min_sync(kFull, __float_as_int(dm)));
    double best = 1.e300;
    int a = 0x7fffffff, qa = -1;
    for (int q = lane; q < m; q += 32) {
      const float4 w = R.at(q);
      if (!(w.x == w.x) || w.w > dm * (1.f + 0x1p-18f)) continue;
      const int j = R.S[q];
      const Pt pj = load_pt(T, j);
      const double dx = pj.x - R.pi.x, dy = pj.y - R.pi.y, dz = pj.z - R.pi.z;
      const double d2 = dx * dx + dy * dy + dz * dz;
      if (d2 < best || (d2 == best && j < a)) { a = j; best = d2; qa = q; }
    }
    for (int off = 16; off > 0; off >>= 1) {
      const double ob = __shfl_down_sync(kFull, best, off);
      const int oa = __shfl_down_sync(kFull, a, off), oq = __shfl_down_sync(kFull, qa, off);
      if (ob < best || (ob == best && oa < a)) { a = oa; best = ob; qa = oq; }
    }
    qa = __shfl_sync(kFull, qa, 0);
    int c = 0x7fffffff, qc = -1;
    if (qa >= 0) {
      const float4 u4 = R.at(qa);
      const V3 u3{u4.x, u4.y, u4.z};
      // squared circumradius |u|^2 |v|^2 |v - u|^2 / (4 |u x v|^2), at least a
      // quarter of the longest edge's square; its relative error is below
      // 40 e |u||v| / |u x v|
      auto radius = [&](int q, float& lo, float& hi) -> bool {
        if (q == qa) return false;
        const float4 w = R.at(q);
        if (w.x != w.x) return false;
        const V3 v3{w.x, w.y, w.z}, d3{w.x - u4.x, w.y - u4.y, w.z - u4.z};
        const V3 x = vcross(u3, v3);
        const float xx = vdot(x, x), dd = vdot(d3, d3), vv = w.w * w.w, uu = u4.w * u4.w;
        const float floor_ = 0.25f * fmaxf(vv, fmaxf(uu, dd)) * (1.f - 0x1p-16f);
        const float top = uu * vv * dd, r2 = top / (4.f * xx), rel = 64.f * kE * u4.w * w.w / sqrtf(xx);
        // |v - u| relative to its own rounding: d3 is off by at most 3 e (|u| + |v|)
        const float rd = 8.f * kE * (u4.w + w.w) / sqrtf(dd);
        const float er = rel + 2.f * rd;
        // (top above 1e-17 keeps |u||v| above 1e-10, and er below 1/4 then |u x v|^2 above 1e-30)
        if (!(top > 1.e-17f) || !(er < 0.25f) || !(r2 < 3.e38f)) { lo = floor_; hi = INF; }
        else { lo = fmaxf(r2 * (1.f - 2.f * er), floor_); hi = r2 * (1.f + 2.f * er); }
        return true;
      };
      float H = INF;
      for (int q = lane; q < m; q += 32) {
        float lo, hi;
        if (radius(q, lo, hi)) H = fminf(H, hi);
      }
      H = __int_as_float(__reduce_min_sync(kFull, __float_as_int(H)));
      const Pt pa = R.pt(qa);
      const double u[3] = {pa.x - R.pi.x, pa.y - R.pi.y, pa.z - R.pi.z};
      const double uu = dot3(u, u);
      double bestr = 1.e300;
      for (int q = lane; q < m; q += 32) {
        float lo, hi;
        if (!radius(q, lo, hi) || lo > H) continue;
        const int j = R.S[q];
        const Pt pj = load_pt(T, j);
        const double v[3] = {pj.x - R.pi.x, pj.y - R.pi.y, pj.z - R.pi.z}, w[3] = {v[0] - u[0], v[1] - u[1], v[2] - u[2]};
        double x[3];
        cross3(u, v, x);
        const double xx = dot3(x, x);
        if (!(xx > 0.0)) continue;
        const double r2 = uu * dot3(v, v) * dot3(w, w) / (4.0 * xx);
        if (r2 < bestr || (r2 == bestr && j < c)) { c = j; bestr = r2; qc = q; }
      }
      for (int off = 16; off > 0; off >>= 1) {
        const double ob = __shfl_down_sync(kFull, bestr, off);
        const int oc = __shfl_down_sync(kFull, c, off), oq = __shfl_down_sync(kFull, qc, off);
        if (ob < bestr || (ob == bestr && oc < c)) { c = oc; bestr = ob; qc = oq; }
      }
      qc = __shfl_sync(kFull, qc, 0);
    }
    // 2. first tet: the face (i, a, c) wrapped to either side
    if (qc >= 0) {
      const float4 A = R.at(qa), B = R.at(qc);
      for (int s = 1; s >= -1 && ns == 0; s -= 2) {
        const Face F = face_of(A, B, (float)-s);  // orient3d(i, a, c, d) = -n . w
        const Wrap W = wrap(R, F, qa, qc, s, lane);
        if (W.d >= 0 && first_empty(R, F, W, qa, qc, s, &degen, lane)) {
          float rc2, band;
          const bool cert = certified(R, F, W, qa, qc, Ri, rc2, band);
          if (lane == 0) {
            sm.tet[0][0] = s > 0 ? qa : qc;
            sm.tet[0][1] = s > 0 ? qc : qa;
            sm.tet[0][2] = W.d;
            sm.cert[0] = cert;
            sm.rc2[0] = rc2;
            sm.band[0] = band;
          }
          ns = 1;
        }
      }
    }
    __syncwarp();
    if (ns == 0) open = true;
    // 3. breadth-first over the link, through every tet of the row's
    // Delaunay tetrahedralisation around i (certified or not, so that the
    // whole star is reached): every tet (x, y, z) is stored with
    // orient3d(i, x, y, z) > 0; its link edges (x, y), (y, z), (z, x) lead
    // to the tets across the faces (i, x, y) ...  (warp-uniform; lane 0 writes)
    int head = 0, first = 0;  // first: no open link edge before it
    while (true) {
      for (; head < ns && !trunc; head++) {
        const int t0 = sm.tet[head][0], t1 = sm.tet[head][1], t2 = sm.tet[head][2];
        const int eu[3] = {t0, t1, t2}, ev[3] = {t1, t2, t0};
        int at[3] = {-1, -1, -1};  // the tet's link edges already in the list
        for (int q0 = 0; q0 < nl; q0 += 32) {
          const int q = q0 + lane;
          const int x = q < nl ? sm.le[q][0] : -1, y = q < nl ? sm.le[q][1] : -1;
          for (int k = 0; k < 3; k++) {
            const unsigned hit = __ballot_sync(kFull, (x == eu[k] && y == ev[k]) || (x == ev[k] && y == eu[k]));
            if (hit && at[k] < 0) at[k] = q0 + __ffs(hit) - 1;
          }
        }
        __syncwarp();
        for (int k = 0; k < 3; k++) {
          if (at[k] >= 0) {
            if (lane == 0) sm.done[at[k]] = 1;
          } else if (nl < kMaxLink) {
            if (lane == 0) { sm.le[nl][0] = eu[k]; sm.le[nl][1] = ev[k]; sm.done[nl] = 0; }
            nl++;
          } else {
            trunc = true;
          }
        }
        __syncwarp();
      }
      if (trunc) break;
      int f = -1;
      for (; first < nl; first += 32) {
        const int q = first + lane;
        const unsigned todo = __ballot_sync(kFull, q < nl && !sm.done[q]);
        if (todo) { f = first + __ffs(todo) - 1; break; }
        if (first + 32 > nl) break;  // edges appended later may land in this group
      }
      if (f < 0) break;
      const int u = sm.le[f][0], v = sm.le[f][1];
      __syncwarp();
      if (lane == 0) sm.done[f] = 1;
      __syncwarp();
      // the stored tet (u, v, w) has orient3d(i, u, v, w) > 0: wrap to the other side
      const Face F = face_of(R.at(u), R.at(v), 1.f);
      const Wrap W = wrap(R, F, u, v, -1, lane);
      if (W.d >= 0 && W.tie) degen = true;
      if (W.d < 0 || W.tie) {
        open = true;
        continue;
      }
      const int d = W.d;
      bool dup = false;
      for (int q0 = 0; q0 < ns && !dup; q0 += 32) {
        const int q = q0 + lane;
        bool same = false;
        if (q < ns) {
          const int* t = sm.tet[q];
          same = (t[0] == u || t[1] == u || t[2] == u) && (t[0] == v || t[1] == v || t[2] == v) &&
                 (t[0] == d || t[1] == d || t[2] == d);
        }
        dup = __any_sync(kFull, same);
      }
      if (dup) continue;
      if (ns == kMaxStar) {
        trunc = true;
        break;
      }
      float rc2, band;
      const bool cert = certified(R, F, W, u, v, Ri, rc2, band);
      if (lane == 0) {  // orient3d(i, v, u, d) > 0
        sm.tet[ns][0] = v;
        sm.tet[ns][1] = u;
        sm.tet[ns][2] = d;
        sm.cert[ns] = cert;
        sm.rc2[ns] = rc2;
        sm.band[ns] = band;
      }
      ns++;
      __syncwarp();
    }
    __syncwarp();
    // 4. emit the tets whose lowest-id holding ball is i's (lanes over the
    // star, compacted in star order); apply the deletion rule
    int ne = 0;
    unsigned long long ndel = 0;
    for (int base = 0; base < ns; base += 32) {
      const int q = base + lane;
      bool emit = false, del = false;
      int v[4] = {0, 0, 0, 0};
      if (q < ns && sm.cert[q]) {
        v[0] = i; v[1] = R.S[sm.tet[q][0]]; v[2] = R.S[sm.tet[q][1]]; v[3] = R.S[sm.tet[q][2]];
        sort4(v);
        // every corner lies on the sphere, so its ball holds the sphere when
        // the diameter is at most its radius
        const float rc2 = sm.rc2[q], band = sm.band[q];
        int owner = -1;
        bool sure = band < INF;
        for (int k = 0; k < 4 && owner < 0 && sure; k++) {
          const float Rk = T.rf[v[k]] * sc;
          if (v[k] == i || rc2 + band < Rk) owner = v[k];
          else if (!(rc2 - band > Rk)) sure = false;
        }
        bool all_boundary = false;
        if (!sure || owner == i)
          all_boundary = T.type[v[0]] != 0 && T.type[v[1]] != 0 && T.type[v[2]] != 0 && T.type[v[3]] != 0;
        if (!sure || all_boundary) {
          Pt P[4];
          for (int k = 0; k < 4; k++) P[k] = load_pt(T, v[k]);
          TetGeo g;
          tet_geo(P, g);
          if (!sure) {
            owner = -1;
            for (int k = 0; k < 4 && owner < 0; k++) {
              const double xv[3] = {P[k].x, P[k].y, P[k].z};
              if (tet_in_ball(g, P, xv, T.h[v[k]], T.cutoff)) owner = v[k];
            }
          }
          if (owner == i) del = all_boundary && tet_aspect(g, P) > T.thres;
        }
        emit = owner == i && !del;
      }
      const unsigned em = __ballot_sync(kFull, emit);
      ndel += __popc(__ballot_sync(kFull, del));
      if (emit) {
        int* o = out + (i64 * kMaxOut + ne + __popc(em & ((1u << lane) - 1u))) * 4;
        for (int k = 0; k < 4; k++) o[k] = v[k];
      }
      ne += __popc(em);
    }
    if (lane == 0) {
      count[i] = ne;
      if (open) atomicAdd(&stats[0], 1ull);
      if (ndel) atomicAdd(&stats[1], ndel);
      if (degen) atomicAdd(&stats[2], 1ull);
      if (trunc) atomicAdd(&stats[3], 1ull);
    }
    __syncwarp();
  }
}

// Snap to the grid: x' = rint(x / g) g (g a power of two, |x / g| < 2^52).
// Also the FP32 ball radii (the first n threads).
__global__ void k_tet_snap(long long n, double* __restrict__ x, double inv_g, double g, const double* __restrict__ h,
                           double cutoff, float* __restrict__ rf) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < 3 * n) x[k] = rint(x[k] * inv_g) * g;
  if (k < n) rf[k] = (float)(cutoff * h[k] * (1.0 - 1.e-6));
}

__global__ void k_tet_compact(long long n, const int* __restrict__ src, const int* __restrict__ count,
                              const int* __restrict__ off, int* __restrict__ tets) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = count[i];
  const long long o = off[i];
  for (int k = 0; k < 4 * c; k++) tets[4 * o + k] = src[i * kMaxOut * 4 + k];
}

// ------------------------------------------------------------ quality
struct TetStat {
  double vol, vmin, vmax, emin2, emax2, amin, amax, asum, rmin, rmax, rsum, dsum;
  double cdmin, cdmax;  // cosines of the smallest and the largest dihedral angle
};
struct TetQIn {
  const double* x;
  const int* tets;
  long long ntet;
  const double* cos_dihed;  // cos(4 k degrees), k = 0..45
  const double* cos_small;  // cos(10, 20, 30, 40 degrees)
  unsigned long long* hist;  // aspect 12, radius 56, dihedral 45, small-dihedral 4
};
constexpr int kQualHist = 12 + 56 + 45 + 4;
constexpr int kAspectBins = 12, kRadiusBins = 56, kDihedBins = 45;
// degrees as the reference converts them: acos(x) / PI * 180 with its PI (glbparam.h:186)
constexpr double kPiRef = 3.1415926;

__host__ __device__ inline double dihed_degrees(double c) { return acos(c) / kPiRef * 180.0; }

__device__ void tet_quality_one(const TetQIn& Q, long long t, TetStat& s, unsigned* hist) {
  Pt P[4];
  for (int k = 0; k < 4; k++) {
    const double* p = Q.x + 3 * (long long)Q.tets[4 * t + k];
    P[k] = Pt{p[0], p[1], p[2]};
  }
  TetGeo g;
  tet_geo(P, g);
  double n[4][3], H[4];
  cross3(g.A[1], g.A[2], n[0]);
  cross3(g.A[2], g.A[0], n[1]);
  cross3(g.A[0], g.A[1], n[2]);
  for (int k = 0; k < 3; k++)
    for (int q = 0; q < 3; q++) n[k][q] /= g.det;
  for (int q = 0; q < 3; q++) n[3][q] = -n[0][q] - n[1][q] - n[2][q];
  double hsum = 0.0, hmax = 0.0;
  for (int k = 0; k < 4; k++) {
    H[k] = sqrt(dot3(n[k], n[k]));
    hsum += H[k];
    hmax = fmax(hmax, H[k]);
    for (int q = 0; q < 3; q++) n[k][q] /= H[k];
  }
  double e2[6], e[3];
  for (int k = 0; k < 3; k++) e2[k] = dot3(g.A[k], g.A[k]);
  const double* p0 = &P[0].x;
  const double* p1 = &P[1].x;
  const double* p2 = &P[2].x;
  for (int q = 0; q < 3; q++) e[q] = p1[q] - p0[q];
  e2[3] = dot3(e, e);
  for (int q = 0; q < 3; q++) e[q] = p2[q] - p1[q];
  e2[4] = dot3(e, e);
  for (int q = 0; q < 3; q++) e[q] = p0[q] - p2[q];
  e2[5] = dot3(e, e);
  double lo = e2[0], hi = e2[0];
  for (int k = 1; k < 6; k++) { lo = fmin(lo, e2[k]); hi = fmax(hi, e2[k]); }
  const double vol = fabs(g.det) / 6.0;
  const double aspect = sqrt(hi) * hmax;
  const double ratio = 3.0 * (1.0 / hsum) / g.rc;
  s.vol += vol;
  s.vmin = fmin(s.vmin, vol);
  s.vmax = fmax(s.vmax, vol);
  s.emin2 = fmin(s.emin2, lo);
  s.emax2 = fmax(s.emax2, hi);
  s.amin = fmin(s.amin, aspect);
  s.amax = fmax(s.amax, aspect);
  s.asum += aspect;
  s.rmin = fmin(s.rmin, ratio);
  s.rmax = fmax(s.rmax, ratio);
  s.rsum += ratio;
  // aspect histogram (aspectratiotable, graph_mesh.cpp:2037-2042, 2349-2353)
  const double tab[11] = {1.5, 2.0, 2.5, 3.0, 4.0, 6.0, 10.0, 15.0, 25.0, 50.0, 100.0};
  int ai = 0;
  while (ai < 11 && aspect > tab[ai]) ai++;
  atomicAdd(&hist[ai], 1u);
  const double rq = floor(ratio / 0.02);
  const int ri = rq >= 0.0 ? (rq < kRadiusBins - 1 ? (int)rq : kRadiusBins - 1) : 0;
  atomicAdd(&hist[kAspectBins + ri], 1u);
  // dihedral angles at the six edges: cos = -n_a . n_b
  const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {1, 2, 3, 2, 3, 3};
  double cmax = -2.0, cmin = 2.0;
  for (int k = 0; k < 6; k++) {
    double cs = -dot3(n[pa[k]], n[pb[k]]);
    cs = fmin(1.0, fmax(-1.0, cs));
    cmax = fmax(cmax, cs);  // smallest angle
    cmin = fmin(cmin, cs);  // largest angle
    // the bin is the number of table cosines at or above cs: an FP32 angle is
    // within one bin, the FP64 comparisons settle it
    int b = min(max((int)(acosf((float)cs) * (45.f / 3.14159265f)), 0), kDihedBins - 1);
    while (b < kDihedBins - 1 && cs <= Q.cos_dihed[b + 1]) b++;
    while (b > 0 && !(cs <= Q.cos_dihed[b])) b--;
    atomicAdd(&hist[kAspectBins + kRadiusBins + b], 1u);
  }
  for (int k = 0; k < 4; k++)
    if (cmax > Q.cos_small[k]) atomicAdd(&hist[kAspectBins + kRadiusBins + kDihedBins + k], 1u);
  s.cdmin = fmax(s.cdmin, cmax);
  s.cdmax = fmin(s.cdmax, cmin);
  s.dsum += dihed_degrees(cmax);
}

__device__ inline void stat_init(TetStat& s) {
  s.vol = s.asum = s.rsum = s.dsum = 0.0;
  s.vmin = s.emin2 = s.amin = s.rmin = 1.e300;
  s.vmax = s.emax2 = s.amax = s.rmax = 0.0;
  s.cdmin = -2.0;
  s.cdmax = 2.0;
}
__device__ inline void stat_fold(TetStat& a, const TetStat& b) {
  a.vol += b.vol; a.asum += b.asum; a.rsum += b.rsum; a.dsum += b.dsum;
  a.vmin = fmin(a.vmin, b.vmin); a.emin2 = fmin(a.emin2, b.emin2); a.amin = fmin(a.amin, b.amin);
  a.rmin = fmin(a.rmin, b.rmin); a.cdmin = fmax(a.cdmin, b.cdmin);
  a.vmax = fmax(a.vmax, b.vmax); a.emax2 = fmax(a.emax2, b.emax2); a.amax = fmax(a.amax, b.amax);
  a.rmax = fmax(a.rmax, b.rmax); a.cdmax = fmin(a.cdmax, b.cdmax);
}

// 256 threads, one partial per block folded in a fixed order (deterministic).
// The histograms are counted in shared memory and added once per block: on
// global memory every tet's nine counts met on a few dozen words.  With that, the
// search for a dihedral's bin from an FP32 angle and the extreme angles kept
// as cosines, 830,000 tets take 1.07 ms instead of 1.78; FP64 divisions and
// square roots bound it.
__global__ void __launch_bounds__(256) k_tet_quality(TetQIn Q, TetStat* part) {
  __shared__ TetStat sh[256];
  __shared__ unsigned s_hist[kQualHist];
  for (int b = threadIdx.x; b < kQualHist; b += blockDim.x) s_hist[b] = 0u;
  __syncthreads();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  TetStat s;
  stat_init(s);
  if (t < Q.ntet) tet_quality_one(Q, t, s, s_hist);
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int b = threadIdx.x; b < kQualHist; b += blockDim.x)
    if (s_hist[b]) atomicAdd(&Q.hist[b], (unsigned long long)s_hist[b]);
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) stat_fold(sh[threadIdx.x], sh[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}
// one block over the partials, in a fixed order (one thread took 2.70 ms for 3,244)
__global__ void __launch_bounds__(256) k_tet_quality_fold(const TetStat* part, int nblk, TetStat* out) {
  __shared__ TetStat sh[256];
  TetStat s;
  stat_init(s);
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) stat_fold(s, part[b]);
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) stat_fold(sh[threadIdx.x], sh[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

int tfail(mrsph_handle* h, int code, const std::string& m) {
  h->err = m;
  return code;
}

}  // namespace
}  // namespace mrsph

using namespace mrsph;

extern "C" int mrsph_tetrahedralize(mrsph_handle* h, int* tets, long long cap, long long* ntet_out,
                                    mrsph_tet_quality* q) {
  if (!h) return MRSPH_ERR_ARG;
  if (!h->eng) return tfail(h, MRSPH_ERR_STATE, "mrsph_set_levelset must come first");
  if (h->prm.dim != 3) return tfail(h, MRSPH_ERR_ARG, "tetrahedralisation is 3D only");
  if (cudaSetDevice(h->prm.device) != cudaSuccess) return tfail(h, MRSPH_ERR_CUDA, "cudaSetDevice failed");
  const long long n = h->eng->num_particles();
  if (n <= 0) return tfail(h, MRSPH_ERR_STATE, "no particles");
  if (n > 0x7fffffffLL / kMaxOut) return tfail(h, MRSPH_ERR_RANGE, "too many particles for one tetrahedralisation");
  const int rowcap = h->eng->neighbor_capacity();
  cudaStream_t s = h->stream;
  std::vector<void*> mem;
  int rc = 0;
  auto A = [&](void** p, size_t bytes) -> bool {
    if (cudaMalloc(p, bytes) != cudaSuccess) return false;
    mem.push_back(*p);
    return true;
  };
  // grid 2^(e-52) with 2^e above every |coordinate| of the domain
  double M = 1.0;
  for (int d = 0; d < 3; d++) M = std::fmax(M, std::fmax(std::fabs(h->prm.box_l[d]), std::fabs(h->prm.box_r[d])));
  int e = 0;
  std::frexp(M, &e);  // M < 2^e
  e += 1;
  const double g = std::ldexp(1.0, e - 52), inv_g = std::ldexp(1.0, 52 - e);
  double *d_x = nullptr, *d_phi = nullptr, *d_h = nullptr, *d_cos = nullptr;
  float* d_rf = nullptr;
  int *d_type = nullptr, *d_rows = nullptr, *d_cnt = nullptr, *d_out = nullptr, *d_count = nullptr;
  int *d_off = nullptr, *d_blk = nullptr, *d_tets = nullptr;
  unsigned* d_flags = nullptr;
  unsigned long long *d_stats = nullptr, *d_hist = nullptr;
  TetStat *d_part = nullptr, *d_tq = nullptr;
  const size_t NC = (size_t)n * rowcap;
  constexpr int kHist = kAspectBins + kRadiusBins + kDihedBins + 4;
  unsigned long long st[4] = {0, 0, 0, 0}, hist[kHist];
  std::memset(hist, 0, sizeof(hist));
  TetStat tq;
  std::memset(&tq, 0, sizeof(tq));
  long long ntet = 0;
  unsigned flags = 0;
  double cosv[50];
  for (int k = 0; k <= kDihedBins; k++) cosv[k] = std::cos(4.0 * k * kPiRef / 180.0);
  for (int k = 0; k < 4; k++) cosv[46 + k] = std::cos(10.0 * (k + 1) * kPiRef / 180.0);
  if (!A((void**)&d_x, sizeof(double) * 3 * n) || !A((void**)&d_phi, sizeof(double) * n) ||
      !A((void**)&d_h, sizeof(double) * n) || !A((void**)&d_rf, sizeof(float) * n) || !A((void**)&d_type, sizeof(int) * n) ||
      !A((void**)&d_rows, sizeof(int) * NC) || !A((void**)&d_cnt, sizeof(int) * n) ||
      !A((void**)&d_out, sizeof(int) * 4 * kMaxOut * (size_t)n) || !A((void**)&d_count, sizeof(int) * (n + 1)) ||
      !A((void**)&d_off, sizeof(int) * (n + 1)) || !A((void**)&d_blk, sizeof(int) * scan_blocksums_size(n)) ||
      !A((void**)&d_flags, sizeof(unsigned)) || !A((void**)&d_stats, sizeof(st)) ||
      !A((void**)&d_hist, sizeof(hist)) || !A((void**)&d_cos, sizeof(cosv))) {
    rc = tfail(h, MRSPH_ERR_OOM, "cudaMalloc failed");
    goto done;
  }
  cudaMemsetAsync(d_flags, 0, sizeof(unsigned), s);
  cudaMemsetAsync(d_stats, 0, sizeof(st), s);
  cudaMemsetAsync(d_hist, 0, sizeof(hist), s);
  cudaMemcpyAsync(d_cos, cosv, sizeof(cosv), cudaMemcpyHostToDevice, s);
  rc = h->eng->export_tri(d_x, d_type, d_phi, d_rows, d_cnt, rowcap, d_flags, d_h, false);
  if (rc) { h->err = h->eng->err; goto done; }
  {
    const int nbN = (int)std::min<long long>((n + kStarWarps - 1) / kStarWarps, 152LL * 64);
    k_tet_snap<<<(int)((3 * n + 255) / 256), 256, 0, s>>>(n, d_x, inv_g, g, d_h, h->prm.cutoff, d_rf);
    TetIn T;
    T.n = n; T.cap = rowcap; T.x = d_x; T.type = d_type; T.h = d_h; T.rf = d_rf; T.rows = d_rows; T.cnt = d_cnt;
    T.inv_g = inv_g; T.cutoff = h->prm.cutoff; T.thres = 10.0;
    k_tet_star<<<nbN, 32 * kStarWarps, 0, s>>>(T, d_out, d_count, d_stats);
    cell_scan(d_count, d_off, d_blk, n, 0, s);
    int tot = 0, last = 0;
    cudaMemcpyAsync(&tot, d_off + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&last, d_count + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&flags, d_flags, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(st, d_stats, sizeof(st), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) { rc = tfail(h, MRSPH_ERR_CUDA, "tetrahedralisation failed"); goto done; }
    ntet = (long long)tot + last;
    if (flags & 4u) { rc = tfail(h, MRSPH_ERR_RANGE, "neighbour list spilled; raise neighbor_cap"); goto done; }
    if (ntet > 0) {
      if (!A((void**)&d_tets, sizeof(int) * 4 * ntet)) { rc = tfail(h, MRSPH_ERR_OOM, "cudaMalloc failed"); goto done; }
      k_tet_compact<<<(int)((n + 255) / 256), 256, 0, s>>>(n, d_out, d_count, d_off, d_tets);
      const int nbT = (int)((ntet + 255) / 256);
      if (!A((void**)&d_part, sizeof(TetStat) * nbT) || !A((void**)&d_tq, sizeof(TetStat))) {
        rc = tfail(h, MRSPH_ERR_OOM, "cudaMalloc failed");
        goto done;
      }
      TetQIn Q;
      Q.x = d_x; Q.tets = d_tets; Q.ntet = ntet; Q.cos_dihed = d_cos; Q.cos_small = d_cos + 46; Q.hist = d_hist;
      k_tet_quality<<<nbT, 256, 0, s>>>(Q, d_part);
      k_tet_quality_fold<<<1, 256, 0, s>>>(d_part, nbT, d_tq);
      cudaMemcpyAsync(&tq, d_tq, sizeof(TetStat), cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(hist, d_hist, sizeof(hist), cudaMemcpyDeviceToHost, s);
      if (tets && cap >= ntet) cudaMemcpyAsync(tets, d_tets, sizeof(int) * 4 * ntet, cudaMemcpyDeviceToHost, s);
    }
    cudaError_t err = cudaStreamSynchronize(s);
    if (err == cudaSuccess) err = cudaGetLastError();
    if (err != cudaSuccess) { rc = tfail(h, MRSPH_ERR_CUDA, std::string("tetrahedralisation: ") + cudaGetErrorString(err)); goto done; }
  }
  if (ntet_out) *ntet_out = ntet;
  if (q) {
    std::memset(q, 0, sizeof(*q));
    q->ntet = ntet;
    q->nopen = (long long)st[0];
    q->ndeleted = (long long)st[1];
    q->ntie = (long long)st[2];
    q->ntrunc = (long long)st[3];
    q->grid = g;
    if (ntet > 0) {
      q->total_volume = tq.vol; q->min_volume = tq.vmin; q->max_volume = tq.vmax;
      q->min_edge = std::sqrt(tq.emin2); q->max_edge = std::sqrt(tq.emax2);
      q->min_aspect = tq.amin; q->max_aspect = tq.amax; q->avg_aspect = tq.asum / ntet;
      q->min_radius_ratio = tq.rmin; q->max_radius_ratio = tq.rmax; q->avg_radius_ratio = tq.rsum / ntet;
      q->min_dihedral = dihed_degrees(tq.cdmin); q->max_dihedral = dihed_degrees(tq.cdmax); q->avg_min_dihedral = tq.dsum / ntet;
    }
    for (int k = 0; k < kAspectBins; k++) q->aspect_hist[k] = (long long)hist[k];
    for (int k = 0; k < kRadiusBins; k++) q->radius_hist[k] = (long long)hist[kAspectBins + k];
    for (int k = 0; k < kDihedBins; k++) q->dihedral_hist[k] = (long long)hist[kAspectBins + kRadiusBins + k];
    for (int k = 0; k < 4; k++) q->nsmall_dihedral[k] = (long long)hist[kAspectBins + kRadiusBins + kDihedBins + k];
  }
done:
  for (void* p : mem) cudaFree(p);
  return rc;
}
