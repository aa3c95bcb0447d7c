// mrsph_tri.cu — 2D neighbour-graph triangulation and mesh quality (row A14).
//
//   Voronoi_construction::Local_VD_generation (voronoi_construction.cpp:6-127)
//     -> k_tri_mark / k_tri_mark_exact: j is an edge of i when j is a Voronoi
//        neighbour of i among i's neighbour set (voro++ replaced by exact
//        orient2d / incircle signs: FP32 intervals, then an FP64 filter, then
//        expansion arithmetic); k_tri_adj: the edges as one short list per particle
//   Graphmeshcls::Reconstruct_tris (graph_mesh.cpp:37-409)
//     -> k_tri_pass1 (3-cycles i > j > k, longest-edge deletion for all-boundary
//        triangles whose centroid phi <= 1e-4 of the vertex mean), k_tri_alive
//        (rebuild from the kept triangles), k_tri_mirror, k_tri_pass2 (final 3-cycles,
//        non-manifold and crossing checks)
//   Tri_quality_statistics (graph_mesh.cpp:411-670) -> k_tri_quality
// Exact predicate signs make the edge set independent of evaluation order, so
// it matches the oracle exactly.  Compiled with -fmad=false.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <initializer_list>
#include <vector>

#include "handle.h"

namespace mrsph {
namespace {

// ------------------------------------------------------------ expansions
__device__ inline void two_sum(double a, double b, double& x, double& y) {
  x = a + b;
  double bv = x - a, av = x - bv, br = b - bv, ar = a - av;
  y = ar + br;
}
__device__ inline void two_diff(double a, double b, double& x, double& y) {
  x = a - b;
  double bv = a - x, av = x + bv, br = bv - b, ar = a - av;
  y = ar + br;
}
__device__ inline void two_prod(double a, double b, double& x, double& y) {
  x = a * b;
  y = fma(a, b, -x);
}
__device__ int xgrow(const double* e, int m, double b, double* h) {
  double Q = b;
  int k = 0;
  for (int i = 0; i < m; i++) {
    double Qn, hh;
    two_sum(Q, e[i], Qn, hh);
    Q = Qn;
    if (hh != 0.0) h[k++] = hh;
  }
  if (Q != 0.0 || k == 0) h[k++] = Q;
  return k;
}
__device__ int xscale(const double* e, int m, double b, double* h) {
  double Q, hh;
  int k = 0;
  two_prod(e[0], b, Q, hh);
  if (hh != 0.0) h[k++] = hh;
  for (int i = 1; i < m; i++) {
    double T, t, Q2, s;
    two_prod(e[i], b, T, t);
    two_sum(Q, t, Q2, s);
    if (s != 0.0) h[k++] = s;
    double x = T + Q2, bv = x - T;
    s = Q2 - bv;
    Q = x;
    if (s != 0.0) h[k++] = s;
  }
  if (Q != 0.0 || k == 0) h[k++] = Q;
  return k;
}
constexpr int XCAP = 256;
// acc += sign * p*q*r*s exactly; returns false when the accumulator would overflow
__device__ bool xacc4(double* acc, int* n, double* tmp, double p, double q, double r, double s, double sign) {
  double e[8], f[8];
  two_prod(p, q, e[1], e[0]);
  int m = xscale(e, 2, r, f);
  m = xscale(f, m, s * sign, e);
  for (int i = 0; i < m; i++) {
    if (*n + 1 > XCAP) return false;
    int l = xgrow(acc, *n, e[i], tmp);
    for (int t = 0; t < l; t++) acc[t] = tmp[t];
    *n = l;
  }
  return true;
}
__device__ int xsign(const double* e, int n) {
  for (int i = n - 1; i >= 0; i--)
    if (e[i] != 0.0) return e[i] > 0 ? 1 : -1;
  return 0;
}

// ------------------------------------------------------------ predicates
// Filtered: returns 2 when the FP64 sign is not certain.
__device__ int orient_f(const double* a, const double* b, const double* c) {
  double acx = a[0] - c[0], bcx = b[0] - c[0], acy = a[1] - c[1], bcy = b[1] - c[1];
  double l = acx * bcy, r = acy * bcx;
  double det = l - r;
  double bound = 1.0e-15 * (fabs(l) + fabs(r));
  if (det > bound) return 1;
  if (-det > bound) return -1;
  return 2;
}
__device__ int incircle_f(const double* a, const double* b, const double* c, const double* d) {
  double adx = a[0] - d[0], ady = a[1] - d[1], bdx = b[0] - d[0], bdy = b[1] - d[1];
  double cdx = c[0] - d[0], cdy = c[1] - d[1];
  double al = adx * adx + ady * ady, bl = bdx * bdx + bdy * bdy, cl = cdx * cdx + cdy * cdy;
  double t1 = bdx * cdy, t2 = cdx * bdy, t3 = cdx * ady, t4 = adx * cdy, t5 = adx * bdy, t6 = bdx * ady;
  double det = al * (t1 - t2) + bl * (t3 - t4) + cl * (t5 - t6);
  double perm = (fabs(t1) + fabs(t2)) * al + (fabs(t3) + fabs(t4)) * bl + (fabs(t5) + fabs(t6)) * cl;
  double bound = 2.0e-14 * perm;
  if (det > bound) return 1;
  if (-det > bound) return -1;
  return 2;
}
// Exact signs (expansion arithmetic); *ok = false on accumulator overflow.
__device__ int orient_x(const double* a, const double* b, const double* c, double* acc, double* tmp, bool* ok) {
  int f = orient_f(a, b, c);
  if (f != 2) return f;
  double ax[2], ay[2], bx[2], by[2];
  two_diff(a[0], c[0], ax[1], ax[0]);
  two_diff(a[1], c[1], ay[1], ay[0]);
  two_diff(b[0], c[0], bx[1], bx[0]);
  two_diff(b[1], c[1], by[1], by[0]);
  int n = 0;
  for (int u = 0; u < 2; u++)
    for (int v = 0; v < 2; v++) {
      *ok = *ok && xacc4(acc, &n, tmp, ax[u], by[v], 1.0, 1.0, 1.0);
      *ok = *ok && xacc4(acc, &n, tmp, ay[u], bx[v], 1.0, 1.0, -1.0);
    }
  return xsign(acc, n);
}
__device__ int incircle_x(const double* a, const double* b, const double* c, const double* d, double* acc,
                          double* tmp, bool* ok) {
  int f = incircle_f(a, b, c, d);
  if (f != 2) return f;
  double X[3][2], Y[3][2];
  const double* P[3] = {a, b, c};
  for (int q = 0; q < 3; q++) {
    two_diff(P[q][0], d[0], X[q][1], X[q][0]);
    two_diff(P[q][1], d[1], Y[q][1], Y[q][0]);
  }
  int n = 0;
  for (int q = 0; q < 3; q++) {
    int r = (q + 1) % 3, s = (q + 2) % 3;
    for (int u = 0; u < 2; u++)
      for (int v = 0; v < 2; v++)
        for (int w = 0; w < 2; w++)
          for (int z = 0; z < 2; z++) {
            *ok = *ok && xacc4(acc, &n, tmp, X[q][u], X[q][v], X[r][w], Y[s][z], 1.0);
            *ok = *ok && xacc4(acc, &n, tmp, Y[q][u], Y[q][v], X[r][w], Y[s][z], 1.0);
            *ok = *ok && xacc4(acc, &n, tmp, X[q][u], X[q][v], X[s][w], Y[r][z], -1.0);
            *ok = *ok && xacc4(acc, &n, tmp, Y[q][u], Y[q][v], X[s][w], Y[r][z], -1.0);
          }
  }
  return xsign(acc, n);
}

// Local Delaunay test of edge (i, j) among row S, exact: 1 edge, 0 none.
__device__ int local_delaunay(const double* xyz, int i, int j, const int* S, int ns, double* acc, double* tmp,
                              bool* ok) {
  const double pi[2] = {xyz[3 * (long long)i], xyz[3 * (long long)i + 1]};
  const double pj[2] = {xyz[3 * (long long)j], xyz[3 * (long long)j + 1]};
  int lstar = -1, rstar = -1;
  double pl[2] = {0, 0}, pr[2] = {0, 0};
  for (int q = 0; q < ns; q++) {
    int k = S[q];
    if (k == i || k == j) continue;
    const double pk[2] = {xyz[3 * (long long)k], xyz[3 * (long long)k + 1]};
    int o = orient_x(pi, pj, pk, acc, tmp, ok);
    if (o == 0) {
      double t = (pk[0] - pi[0]) * (pj[0] - pi[0]) + (pk[1] - pi[1]) * (pj[1] - pi[1]);
      double L = (pj[0] - pi[0]) * (pj[0] - pi[0]) + (pj[1] - pi[1]) * (pj[1] - pi[1]);
      if (t > 0 && t < L) return 0;
      continue;
    }
    if (o > 0) {
      int c = 1;
      if (lstar >= 0) c = incircle_x(pi, pj, pl, pk, acc, tmp, ok);
      if (lstar < 0 || c > 0) { lstar = k; pl[0] = pk[0]; pl[1] = pk[1]; }
    } else {
      int c = 1;
      if (rstar >= 0) c = incircle_x(pj, pi, pr, pk, acc, tmp, ok);
      if (rstar < 0 || c > 0) { rstar = k; pr[0] = pk[0]; pr[1] = pk[1]; }
    }
  }
  if (lstar < 0 || rstar < 0) return 1;
  return incircle_x(pi, pj, pl, pr, acc, tmp, ok) < 0 ? 1 : 0;
}

struct TriIn {
  long long n;
  int cap;
  const double* xyz;
  const int* type;
  const double* phi;
  int* rows;  // n x cap, sorted ids incl. self
  const int* cnt;
  // edges: particle i's deg[i] neighbours, ascending ids, in adj + i * cap
  int* deg;
  int* adj;
};

__device__ inline int row_find(const TriIn& T, int a, int b) {
  const int* S = T.rows + (long long)a * T.cap;
  int lo = 0, hi = T.cnt[a] - 1;
  while (lo <= hi) {
    int m = (lo + hi) >> 1;
    int v = S[m];
    if (v == b) return m;
    if (v < b) lo = m + 1; else hi = m - 1;
  }
  return -1;
}

// mark[i*cap+q]: 1 edge, 0 none; slots FP32 cannot decide are queued.  One
// warp per particle: the row is sorted by id (by rank, in shared memory) and
// written back, its positions relative to i are rounded to FP32 once, and
// every lane tests its slots j against all of the row.  A circle through i and
// j holds k on its side of the edge when the angle at k is larger, i.e. its
// cotangent smaller, so (i, j) is an edge when the smallest cotangents of
// the two sides have a positive sum; an interval per cotangent decides almost
// every slot, and a negative sum of upper ends decides "no edge" whatever the
// other points are.  With e = 2^-24 the cross product |e_j x w| is off by at most
// 8 e |e_j||w| and the dot product w . (w - e_j) by 10 e (|w|^2 + |w||e_j|) (each
// position rounded once); the constants below are larger.  All of this in FP64
// (rate 1/60), an incircle determinant per point, took 9.9 ms for 77,551
// particles; now 0.16 ms.
constexpr float kTE = 0x1p-24f;
__host__ __device__ inline size_t mark_smem(int cap) { return (sizeof(float4) + 2 * sizeof(int)) * (size_t)cap; }  // per warp
__global__ void k_tri_mark(TriIn T, unsigned char* mark, long long* queue, unsigned long long* nqueue) {
  extern __shared__ float4 s_dyn[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  float4* w = s_dyn + (size_t)wid * T.cap;  // (x, y, |w|^2, |w|)
  int* raw = reinterpret_cast<int*>(s_dyn + (size_t)nw * T.cap) + (size_t)wid * 2 * T.cap;
  int* id = raw + T.cap;
  const long long i64 = (long long)blockIdx.x * nw + wid;
  if (i64 >= T.n) return;  // whole warps
  const int i = (int)i64, m = T.cnt[i];
  int* S = T.rows + i64 * T.cap;
  for (int q = lane; q < m; q += 32) raw[q] = S[q];
  __syncwarp();
  for (int q = lane; q < m; q += 32) {
    const int v = raw[q];
    int r = 0;
    for (int k = 0; k < m; k++) r += raw[k] < v;
    id[r] = v;
  }
  __syncwarp();
  const double px = T.xyz[3 * i64], py = T.xyz[3 * i64 + 1];
  // the bounds are relative to products of two lengths: a row whose products leave
  // FP32's range (a length below 1e-15 or above 1e15) is decided exactly
  bool fits = true;
  for (int q = lane; q < m; q += 32) {
    const long long j = id[q];
    S[q] = (int)j;
    const float x = (float)(T.xyz[3 * j] - px), y = (float)(T.xyz[3 * j + 1] - py);
    const float n2 = fmaf(y, y, x * x);
    w[q] = make_float4(x, y, n2, sqrtf(n2));
    if (j != i64) fits = fits && n2 > 1.e-30f && n2 < 1.e30f;
  }
  __syncwarp();
  fits = __all_sync(0xffffffffu, fits);
  const float INF = __int_as_float(0x7f800000);
  for (int q = lane; q < m; q += 32) {
    unsigned char* out = mark + i64 * T.cap + q;
    if (id[q] == i) {
      *out = 0;
      continue;
    }
    const float4 e = w[q];
    const float es0 = 16.f * kTE * e.w, ed0 = 16.f * kTE;
    float loL = INF, hiL = INF, loR = INF, hiR = INF;
    bool undecided = !fits, cut = false;
    for (int k = 0; fits && k < m; k++) {
      if (k == q || id[k] == i) continue;
      const float4 p = w[k];
      const float s = e.x * p.y - e.y * p.x, d = p.z - fmaf(e.y, p.y, e.x * p.x);
      const float es = es0 * p.w, a = fabsf(s);
      if (!(a > 2.f * es)) {
        undecided = true;
        continue;
      }
      const float r = __fdividef(1.f, a), c = d * r;
      const float er = 2.f * r * (ed0 * (p.z + p.w * e.w) + fabsf(c) * es) + 8.f * kTE * fabsf(c);
      const float lo = c - er, hi = c + er;
      if (!(hi < INF) || !(lo > -INF)) undecided = true;
      if (s > 0.f) { loL = fminf(loL, lo); hiL = fminf(hiL, hi); }
      else { loR = fminf(loR, lo); hiR = fminf(hiR, hi); }
      if (hiL + hiR < 0.f) {
        cut = true;
        break;
      }
    }
    // loL + loR is infinite when a side has no point: an edge, as in the exact test
    const bool edge = !cut && !undecided && loL + loR > 0.f;
    *out = edge ? 1 : 0;
    if (!cut && !edge) queue[atomicAdd(nqueue, 1ull)] = i64 * T.cap + q;
  }
}

// rows too long for k_tri_mark's shared memory: every slot goes to the exact test
__global__ void k_tri_mark_all(TriIn T, unsigned char* mark, long long* queue, unsigned long long* nqueue) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T.n * T.cap) return;
  const int i = (int)(t / T.cap), q = (int)(t % T.cap);
  if (q >= T.cnt[i]) return;
  mark[t] = 0;
  if (T.rows[t] != i) queue[atomicAdd(nqueue, 1ull)] = t;
}

// Exact test of the queued slots (grid-stride).
// scratch: 2 * XCAP doubles per thread of the launch.
__global__ void __launch_bounds__(64) k_tri_mark_exact(TriIn T, unsigned char* mark, const long long* queue,
                                                         const unsigned long long* nqueue, unsigned* flags,
                                                         double* scratch) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double* acc = scratch + tid * (2 * XCAP);
  double* tmp = acc + XCAP;
  const long long nq = (long long)*nqueue;
  for (long long u = tid; u < nq; u += (long long)gridDim.x * blockDim.x) {
    const long long t = queue[u];
    int i = (int)(t / T.cap), q = (int)(t % T.cap);
    const int* S = T.rows + (long long)i * T.cap;
    bool ok = true;
    int r = local_delaunay(T.xyz, i, S[q], S, T.cnt[i], acc, tmp, &ok);
    if (!ok) atomicOr(flags, 2u);
    mark[t] = (unsigned char)(r == 1 ? 1 : 0);
  }
}

// The edges of particle i in either direction (one warp per particle) as a list
// of ascending ids, with cleared deletion and alive flags: a handful of
// entries, where the passes below went over the row's bytes for every pair of
// slots and searched the partner's whole row.
__global__ void __launch_bounds__(256) k_tri_adj(TriIn T, const unsigned char* mark, unsigned* del, unsigned* alive) {
  const int lane = threadIdx.x & 31;
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= T.n) return;
  const int m = T.cnt[i];
  int n = 0;
  for (int q0 = 0; q0 < m; q0 += 32) {
    const int q = q0 + lane;
    int j = -1;
    bool e = false;
    if (q < m) {
      j = T.rows[i * T.cap + q];
      if (j != i) {
        e = mark[i * T.cap + q] != 0;
        if (!e) {
          const int p = row_find(T, j, (int)i);
          e = p >= 0 && mark[(long long)j * T.cap + p] != 0;
        }
      }
    }
    const unsigned b = __ballot_sync(0xffffffffu, e);
    if (e) {
      const long long o = i * T.cap + n + __popc(b & ((1u << lane) - 1u));
      T.adj[o] = j;
      del[o] = 0u;
      alive[o] = 0u;
    }
    n += __popc(b);
  }
  if (lane == 0) T.deg[i] = n;
}

// position of edge (a, b) in a's list, -1 if there is none; eight entries are in
// flight at a time (lists have about six)
__device__ inline long long edge_find(const TriIn& T, int a, int b) {
  const long long o = (long long)a * T.cap;
  const int n = T.deg[a];
  for (int q0 = 0; q0 < n; q0 += 8) {
    int v[8], hit = -1;
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = T.adj[o + min(q0 + u, n - 1)];
#pragma unroll
    for (int u = 7; u >= 0; u--)
      if (v[u] == b) hit = min(q0 + u, n - 1);
    if (hit >= 0) return o + hit;
  }
  return -1;
}

// deletion rule of Reconstruct_tris (graph_mesh.cpp:144-205): -1 when kept, else
// the longest edge: 0 (I, j), 1 (j, k), 2 (I, k)
__device__ int tri_rule(const TriIn& T, const LsSet& ls, int I, int j, int k) {
  if (T.type[I] == REAL_P || T.type[j] == REAL_P || T.type[k] == REAL_P) return -1;
  const double* p1 = T.xyz + 3 * (long long)I;
  const double* p2 = T.xyz + 3 * (long long)j;
  const double* p3 = T.xyz + 3 * (long long)k;
  double cen[3] = {1. / 3. * (p1[0] + p2[0] + p3[0]), 1. / 3. * (p1[1] + p2[1] + p3[1]),
                   1. / 3. * (p1[2] + p2[2] + p3[2])};
  double pc, nn[3], cv;
  ls_sample<2, double>(ls, cen, pc, nn, cv);
  double phi_size = 1. / 3. * (T.phi[I] + T.phi[j] + T.phi[k]);
  if (pc > 0.0001 * phi_size) return -1;
  double v1[2] = {p2[0] - p1[0], p2[1] - p1[1]};
  double v2[2] = {p3[0] - p2[0], p3[1] - p2[1]};
  double v3[2] = {p1[0] - p3[0], p1[1] - p3[1]};
  double d = sqrt(v1[0] * v1[0] + v1[1] * v1[1]);
  int e = 0;
  double d2 = sqrt(v2[0] * v2[0] + v2[1] * v2[1]);
  if (d2 > d) { d = d2; e = 1; }
  double d3 = sqrt(v3[0] * v3[0] + v3[1] * v3[1]);
  if (d3 > d) { d = d3; e = 2; }
  return e;
}

// The passes over the triangles i > j > k run on kTG lanes per particle, which
// share its pairs of edges; flags of an edge are kept at its larger end while
// they are formed, where a triangle already knows their places.  One thread per
// particle left each SM a chain of dependent loads: 231 (k_tri_pass1), 347
// (k_tri_alive), 136 and 120 us (k_tri_pass2) for 77,551 particles; now 125, 54,
// 60 and 45, and 25 for k_tri_mirror.
constexpr int kTG = 8;

// pass 1a: deleted edges
__global__ void __launch_bounds__(256) k_tri_pass1(TriIn T, LsSet ls, unsigned* del) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = t / kTG;
  const int g = (int)(t % kTG);
  if (i >= T.n) return;
  const long long o = i * T.cap;
  const int* A = T.adj + o;
  const int c = T.deg[i];
  int p = 0;
  for (int a = 0; a < c; a++) {
    const int j = A[a];
    if (j >= i) break;
    for (int b = 0; b < a; b++, p++) {
      if (p % kTG != g) continue;
      const int k = A[b];
      const long long jk = edge_find(T, j, k);
      if (jk < 0) continue;
      const int e = tri_rule(T, ls, (int)i, j, k);
      if (e >= 0) del[e == 0 ? o + a : (e == 1 ? jk : o + b)] = 1u;
    }
  }
}

// pass 1b: edges of kept triangles without a deleted edge are alive.  A triangle
// that the rule does not keep has its longest edge deleted, so the rule is not
// asked again.
__global__ void __launch_bounds__(256) k_tri_alive(TriIn T, const unsigned* del, unsigned* alive) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = t / kTG;
  const int g = (int)(t % kTG);
  if (i >= T.n) return;
  const long long o = i * T.cap;
  const int* A = T.adj + o;
  const int c = T.deg[i];
  int p = 0;
  for (int a = 0; a < c; a++) {
    const int j = A[a];
    if (j >= i) break;
    for (int b = 0; b < a; b++, p++) {
      if (p % kTG != g || del[o + a] || del[o + b]) continue;
      const long long jk = edge_find(T, j, A[b]);
      if (jk < 0 || del[jk]) continue;
      alive[o + a] = 1u;
      alive[o + b] = 1u;
      alive[jk] = 1u;
    }
  }
}

// the alive flags of the smaller ends; edges and deleted edges of the first pass
__global__ void __launch_bounds__(256) k_tri_mirror(TriIn T, const unsigned* del, unsigned* alive,
                                                    unsigned long long* stats) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = t / kTG;
  unsigned e1 = 0, nd = 0;
  if (i < T.n) {
    const long long o = i * T.cap;
    const int c = T.deg[i];
    for (int a = (int)(t % kTG); a < c; a += kTG) {
      const int j = T.adj[o + a];
      if (j < i) continue;
      const long long p = edge_find(T, j, (int)i);
      e1++;
      if (p >= 0 && del[p]) nd++;
      if (p >= 0 && alive[p]) alive[o + a] = 1u;
    }
  }
  e1 = __reduce_add_sync(0xffffffffu, e1);
  nd = __reduce_add_sync(0xffffffffu, nd);
  if ((threadIdx.x & 31) == 0) {
    if (e1) atomicAdd(&stats[2], (unsigned long long)e1);
    if (nd) atomicAdd(&stats[3], (unsigned long long)nd);
  }
}

__device__ inline bool is_alive(const TriIn& T, const unsigned* alive, int a, int b) {
  const long long p = edge_find(T, a, b);
  return p >= 0 && alive[p];
}

// pass 2: final triangles (count or fill) and edge checks (graph_mesh.cpp:300-365).
// The lanes of a particle test the third vertices of one edge together; ballots
// give their order.
template <bool FILL>
__global__ void __launch_bounds__(256) k_tri_pass2(TriIn T, const unsigned* alive, int* count, const int* offset,
                                                   int* tris, unsigned long long* stats) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = t / kTG;
  const int g = (int)(t % kTG), lane = threadIdx.x & 31, g0 = lane - g;
  const unsigned gm = ((1u << kTG) - 1u) << g0;
  unsigned nerr = 0, nedge = 0;
  if (i < T.n) {
    const int* S = T.adj + i * T.cap;
    const unsigned* A = alive + i * T.cap;
    const int c = T.deg[i];
    int ntri = 0;
    const int base = FILL ? offset[i] : 0;
    for (int a = 0; a < c; a++) {
      const int j = S[a];
      if (j >= i) break;
      if (!A[a]) continue;
      nedge++;
      int total = 0, c0 = -1, c1 = -1;  // third vertices, the first two of them
      for (int b0 = 0; b0 < c; b0 += kTG) {
        const int b = b0 + g;
        const int k = b < c ? S[b] : j;
        const bool hit = k != j && A[b] && is_alive(T, alive, j, k);
        const unsigned all = __ballot_sync(gm, hit) >> g0;
        const unsigned low = __ballot_sync(gm, hit && k < j) >> g0;
        int seen = total;
        for (unsigned m = all; m && seen < 2; m &= m - 1u, seen++) (seen ? c1 : c0) = S[b0 + __ffs(m) - 1];
        if (FILL && hit && k < j) {
          int* o = tris + 3 * (long long)(base + ntri + __popc(low & ((1u << g) - 1u)));
          o[0] = (int)i; o[1] = j; o[2] = k;
        }
        ntri += __popc(low);
        total += __popc(all);
      }
      if (!FILL && g == 0 && (total > 2 || (total == 2 && is_alive(T, alive, c0, c1)))) nerr++;
    }
    if (!FILL && g == 0) count[i] = ntri;
    if (g) nedge = 0;
  }
  if (!FILL) {
    nerr = __reduce_add_sync(0xffffffffu, nerr);
    nedge = __reduce_add_sync(0xffffffffu, nedge);
    if (lane == 0) {
      if (nerr) atomicAdd(&stats[0], (unsigned long long)nerr);
      if (nedge) atomicAdd(&stats[1], (unsigned long long)nedge);
    }
  }
}

// per-triangle quality terms (graph_mesh.cpp:445-520)
struct TriStat {
  double max_angle, min_angle, max_aspect, max_edge, min_edge, max_area, min_area, G_min;
  double sum_G, sum_minangle, sum_area;
  unsigned long long theta30;
};

__device__ inline void stat_init(TriStat& s) {
  s.max_angle = 0.; s.min_angle = 1.e15; s.max_aspect = 0.; s.max_edge = 0.; s.min_edge = 1.e15;
  s.max_area = 0.; s.min_area = 1.e15; s.G_min = 1.e20; s.sum_G = 0.; s.sum_minangle = 0.; s.sum_area = 0.;
  s.theta30 = 0;
}
__device__ inline void stat_fold(TriStat& r, const TriStat& q) {
  r.max_angle = fmax(r.max_angle, q.max_angle);
  r.min_angle = fmin(r.min_angle, q.min_angle);
  r.max_aspect = fmax(r.max_aspect, q.max_aspect);
  r.max_edge = fmax(r.max_edge, q.max_edge);
  r.min_edge = fmin(r.min_edge, q.min_edge);
  r.max_area = fmax(r.max_area, q.max_area);
  r.min_area = fmin(r.min_area, q.min_area);
  r.G_min = fmin(r.G_min, q.G_min);
  r.sum_G += q.sum_G;
  r.sum_minangle += q.sum_minangle;
  r.sum_area += q.sum_area;
  r.theta30 += q.theta30;
}
// the 256 entries of sh folded into sh[0] in a fixed order
__device__ inline void block_fold(TriStat* sh) {
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) stat_fold(sh[threadIdx.x], sh[threadIdx.x + w]);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_tri_quality(const double* __restrict__ xyz, long long ntri,
                                                     const int* __restrict__ tris, TriStat* part,
                                                     unsigned long long* hist) {
  __shared__ TriStat sh[256];
  __shared__ unsigned s_hist[45];
  if (threadIdx.x < 45) s_hist[threadIdx.x] = 0u;
  __syncthreads();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  TriStat s;
  stat_init(s);
  if (t < ntri) {
    const double rad = 180. / acos(-1.);
    const double* v0 = xyz + 3 * (long long)tris[3 * t];
    const double* v1 = xyz + 3 * (long long)tris[3 * t + 1];
    const double* v2 = xyz + 3 * (long long)tris[3 * t + 2];
    double a1[2] = {v1[0] - v0[0], v1[1] - v0[1]}, a2[2] = {v2[0] - v1[0], v2[1] - v1[1]},
           a3[2] = {v0[0] - v2[0], v0[1] - v2[1]};
    double d1 = sqrt(a1[0] * a1[0] + a1[1] * a1[1]);
    double d2 = sqrt(a2[0] * a2[0] + a2[1] * a2[1]);
    double d3 = sqrt(a3[0] * a3[0] + a3[1] * a3[1]);
    double dmax = fmax(d1, fmax(d2, d3)), dmin = fmin(d1, fmin(d2, d3));
    s.max_edge = dmax;
    s.min_edge = dmin;
    s.max_aspect = dmax / (dmin + 1.e-20);
    double c13 = -(a1[0] * a3[0] + a1[1] * a3[1]) / (d3 * d1 + 1.e-20);
    double al1 = rad * acos(c13);
    double al2 = rad * acos(-(a1[0] * a2[0] + a1[1] * a2[1]) / (d2 * d1 + 1.e-20));
    double al3 = rad * acos(-(a2[0] * a3[0] + a2[1] * a3[1]) / (d3 * d2 + 1.e-20));
    al1 = fmax(0., fmin(al1, 180.));
    al2 = fmax(0., fmin(al2, 180.));
    al3 = fmax(0., fmin(al3, 180.));
    s.max_angle = fmax(al1, fmax(al2, al3));
    double mm = fmin(al1, fmin(al2, al3));
    s.min_angle = mm;
    atomicAdd(&s_hist[min(44, (int)(al1 / 4.0))], 1u);
    atomicAdd(&s_hist[min(44, (int)(al2 / 4.0))], 1u);
    atomicAdd(&s_hist[min(44, (int)(al3 / 4.0))], 1u);
    s.theta30 = mm < 30. ? 1 : 0;
    s.sum_minangle = mm;
    double area = 0.5 * (d3 * d1) * sin(acos(c13));
    s.sum_area = area;
    s.max_area = area;
    s.min_area = area;
    double G = 2. * sqrt(3.) * area / (dmax * (d1 + d2 + d3) / 2.);
    s.G_min = G;
    s.sum_G = G;
  }
  sh[threadIdx.x] = s;
  block_fold(sh);
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
  if (threadIdx.x < 45 && s_hist[threadIdx.x]) atomicAdd(&hist[threadIdx.x], (unsigned long long)s_hist[threadIdx.x]);
}

// one block over the partials, in a fixed order
__global__ void __launch_bounds__(256) k_tri_quality_fold(const TriStat* part, int nblk, TriStat* out) {
  __shared__ TriStat sh[256];
  TriStat r;
  stat_init(r);
  for (int k = threadIdx.x; k < nblk; k += blockDim.x) stat_fold(r, part[k]);
  sh[threadIdx.x] = r;
  block_fold(sh);
  if (threadIdx.x == 0) *out = sh[0];
}

int tfail(mrsph_handle* h, int code, const std::string& msg) {
  h->err = msg;
  return code;
}

}  // namespace
}  // namespace mrsph

using namespace mrsph;

extern "C" int mrsph_triangulate(mrsph_handle* h, int* tris, long long cap, long long* ntri_out,
                                 mrsph_tri_quality* q) {
  if (!h) return MRSPH_ERR_ARG;
  if (!h->eng) return tfail(h, MRSPH_ERR_STATE, "mrsph_set_levelset must come first");
  if (h->prm.dim != 2) return tfail(h, MRSPH_ERR_ARG, "triangulation is 2D only");
  if (cudaSetDevice(h->prm.device) != cudaSuccess) return tfail(h, MRSPH_ERR_CUDA, "cudaSetDevice failed");
  const long long n = h->eng->num_particles();
  if (n <= 0) return tfail(h, MRSPH_ERR_STATE, "no particles");
  const int rowcap = h->eng->neighbor_capacity();
  cudaStream_t s = h->stream;
  std::vector<void*> mem;
  int rc = 0;
  // one allocation for the buffers of known size (each 256-byte aligned), one for
  // those of the mesh
  struct Part { void** p; size_t bytes; };
  auto A = [&](std::initializer_list<Part> parts) -> bool {
    size_t all = 0;
    for (const Part& q : parts) all += (q.bytes + 255) & ~(size_t)255;
    char* base = nullptr;
    if (cudaMalloc(&base, all) != cudaSuccess) return false;
    mem.push_back(base);
    for (const Part& q : parts) {
      *q.p = base;
      base += (q.bytes + 255) & ~(size_t)255;
    }
    return true;
  };
  double *d_xyz = nullptr, *d_phi = nullptr;
  int *d_type = nullptr, *d_rows = nullptr, *d_cnt = nullptr, *d_count = nullptr, *d_off = nullptr;
  int *d_blk = nullptr, *d_tris = nullptr;
  unsigned char* d_mark = nullptr;
  int *d_deg = nullptr, *d_adj = nullptr;
  long long* d_queue = nullptr;
  unsigned *d_del = nullptr, *d_alive = nullptr, *d_flags = nullptr;  // flags per entry of d_adj
  unsigned long long *d_stats = nullptr, *d_hist = nullptr;  // stats[4]: queued slots
  TriStat *d_part = nullptr, *d_tq = nullptr;
  double* d_scratch = nullptr;
  constexpr size_t kMarkSmem = 200 * 1024;
  int wpb = 0;
  const int XB = 152, XT = 64;  // exact-predicate launch: a block per SM, 40 MB of scratch
  const size_t NC = (size_t)n * rowcap;
  long long ntri = 0;
  unsigned flags = 0;
  unsigned long long st[4] = {0, 0, 0, 0}, hist[45];
  TriStat tq;
  std::memset(&tq, 0, sizeof(tq));
  if (!A({{(void**)&d_xyz, sizeof(double) * 3 * n}, {(void**)&d_phi, sizeof(double) * n},
          {(void**)&d_type, sizeof(int) * n}, {(void**)&d_rows, sizeof(int) * NC}, {(void**)&d_cnt, sizeof(int) * n},
          {(void**)&d_count, sizeof(int) * (n + 1)}, {(void**)&d_off, sizeof(int) * (n + 1)},
          {(void**)&d_blk, sizeof(int) * scan_blocksums_size(n)}, {(void**)&d_mark, NC},
          {(void**)&d_adj, sizeof(int) * NC}, {(void**)&d_deg, sizeof(int) * n},
          {(void**)&d_queue, sizeof(long long) * NC}, {(void**)&d_flags, sizeof(unsigned)},
          {(void**)&d_stats, sizeof(unsigned long long) * 5}, {(void**)&d_hist, sizeof(unsigned long long) * 45},
          {(void**)&d_scratch, sizeof(double) * 2 * XCAP * XB * XT}})) {
    rc = tfail(h, MRSPH_ERR_OOM, "cudaMalloc failed");
    goto done;
  }
  // the flags of the edge lists take the queue's place: it is spent by then
  d_del = reinterpret_cast<unsigned*>(d_queue);
  d_alive = d_del + NC;
  cudaMemsetAsync(d_flags, 0, sizeof(unsigned), s);
  cudaMemsetAsync(d_stats, 0, sizeof(unsigned long long) * 5, s);
  cudaMemsetAsync(d_hist, 0, sizeof(unsigned long long) * 45, s);
  // k_tri_mark sorts the rows itself when a warp's row fits the shared memory
  // (kMarkSmem: below the 227 KB a block may have)
  wpb = (int)std::min<size_t>(8, kMarkSmem / mark_smem(rowcap));
  rc = h->eng->export_tri(d_xyz, d_type, d_phi, d_rows, d_cnt, rowcap, d_flags, nullptr, wpb == 0);
  if (rc) { h->err = h->eng->err; goto done; }
  {
    TriIn T;
    T.n = n; T.cap = rowcap; T.xyz = d_xyz; T.type = d_type; T.phi = d_phi; T.rows = d_rows; T.cnt = d_cnt;
    T.deg = d_deg; T.adj = d_adj;
    const int nbE = (int)((NC + 255) / 256), nbN = (int)((n * kTG + 255) / 256);
    if (wpb > 0) {
      const size_t sm = wpb * mark_smem(rowcap);
      cudaFuncSetAttribute(k_tri_mark, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMarkSmem);
      k_tri_mark<<<(unsigned)((n + wpb - 1) / wpb), 32 * wpb, sm, s>>>(T, d_mark, d_queue, d_stats + 4);
    } else {
      k_tri_mark_all<<<nbE, 256, 0, s>>>(T, d_mark, d_queue, d_stats + 4);
    }
    k_tri_mark_exact<<<XB, XT, 0, s>>>(T, d_mark, d_queue, d_stats + 4, d_flags, d_scratch);
    k_tri_adj<<<(unsigned)((n + 7) / 8), 256, 0, s>>>(T, d_mark, d_del, d_alive);
    k_tri_pass1<<<nbN, 256, 0, s>>>(T, h->ls, d_del);
    k_tri_alive<<<nbN, 256, 0, s>>>(T, d_del, d_alive);
    k_tri_mirror<<<nbN, 256, 0, s>>>(T, d_del, d_alive, d_stats);
    k_tri_pass2<false><<<nbN, 256, 0, s>>>(T, d_alive, d_count, nullptr, nullptr, d_stats);
    cell_scan(d_count, d_off, d_blk, n, 0, s);
    int tot = 0;
    if (cudaMemcpyAsync(&tot, d_off + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) {
      rc = tfail(h, MRSPH_ERR_CUDA, "copy failed");
      goto done;
    }
    int last = 0;
    cudaMemcpyAsync(&last, d_count + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&flags, d_flags, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) { rc = tfail(h, MRSPH_ERR_CUDA, "triangulation failed"); goto done; }
    ntri = (long long)tot + last;
    if (flags & 4u) { rc = tfail(h, MRSPH_ERR_RANGE, "neighbour list spilled; raise neighbor_cap"); goto done; }
    if (flags) { rc = tfail(h, MRSPH_ERR_DEVICE, "exact predicate accumulator overflow"); goto done; }
    if (ntri > 0) {
      const int nbT = (int)((ntri + 255) / 256);
      if (!A({{(void**)&d_tris, sizeof(int) * 3 * ntri}, {(void**)&d_part, sizeof(TriStat) * nbT},
              {(void**)&d_tq, sizeof(TriStat)}})) {
        rc = tfail(h, MRSPH_ERR_OOM, "cudaMalloc failed");
        goto done;
      }
      k_tri_pass2<true><<<nbN, 256, 0, s>>>(T, d_alive, nullptr, d_off, d_tris, nullptr);
      k_tri_quality<<<nbT, 256, 0, s>>>(d_xyz, ntri, d_tris, d_part, d_hist);
      k_tri_quality_fold<<<1, 256, 0, s>>>(d_part, nbT, d_tq);
      cudaMemcpyAsync(&tq, d_tq, sizeof(TriStat), cudaMemcpyDeviceToHost, s);
      if (tris && cap >= ntri)
        cudaMemcpyAsync(tris, d_tris, sizeof(int) * 3 * ntri, cudaMemcpyDeviceToHost, s);
    }
    cudaMemcpyAsync(st, d_stats, sizeof(st), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(hist, d_hist, sizeof(hist), cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { rc = tfail(h, MRSPH_ERR_CUDA, std::string("triangulation: ") + cudaGetErrorString(e)); goto done; }
  }
  if (ntri_out) *ntri_out = ntri;
  if (q) {
    std::memset(q, 0, sizeof(*q));
    q->ntri = ntri;
    q->nedge = (long long)st[1];
    q->nedge_first = (long long)st[2];
    q->ndeleted = (long long)st[3];
    q->nerror = (long long)st[0];
    if (ntri > 0) {
      q->max_angle = tq.max_angle; q->min_angle = tq.min_angle; q->max_aspect = tq.max_aspect;
      q->max_edge = tq.max_edge; q->min_edge = tq.min_edge; q->max_area = tq.max_area; q->min_area = tq.min_area;
      q->G_min = tq.G_min;
      q->G_avg = tq.sum_G / ntri;
      q->min_angle_avg = tq.sum_minangle / ntri;
      q->theta_30 = (double)tq.theta30 / (double)ntri;
      q->total_area = tq.sum_area;
    } else {  // the statistics' initial values (graph_mesh.cpp:433-443)
      q->min_angle = 1.e15;
      q->min_edge = 1.e15;
      q->min_area = 1.e15;
      q->G_min = 1.e20;
    }
    for (int b = 0; b < 45; b++) q->hist[b] = (long long)hist[b];
  }
done:
  for (void* p : mem) cudaFree(p);
  return rc;
}
