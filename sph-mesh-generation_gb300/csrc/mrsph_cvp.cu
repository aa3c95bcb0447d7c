// mrsph_cvp.cu — centroidal Voronoi partitioning of the particles (row A13),
// Voronoi::Partitioning (CVP/voronoi.cpp:1376-1446) on the GPU.
//
// One iteration = eight kernels:
//   k_cvp_assign    nearest VP per point, strict '<' (Get_CPU_id, voronoi.cpp:480-493)
//   k_cvp_partials  per (VP, 2048-point chunk) mass, mass centre and energy,
//                   points in order (voronoi.cpp:617-631); one block per chunk
//                   groups its points by VP first
//   k_cvp_reduce    per VP: chunk partials in order, centroid, pressure, error
//   k_cvp_planes    bisector plane of every VP pair
//   k_cvp_face_cull per (VP, plane) an FP32 clip of the plane's polygon, enough
//                   to drop the pairs that share no face
//   k_cvp_faces     the exact Voronoi face inside the box of the pairs left: the
//                   plane's polygon clipped by every other bisector half-space
//                   (replaces voro++, voronoi.cpp:724-790)
//   k_cvp_force     face pressure force and h per VP, faces in order
//   k_cvp_update    Update_position (voronoi.cpp:830-897), Update_position_CVT
//                   (:901-992), Check_partition_error (:1228-1262)
// The level-set partition (Voronoi_lset::Partitioning_for_initial_VP_distribution,
// voronoi_lset.cpp:824-889) adds, before the assignment, k_cvp_flags and
// k_cvp_ghosts: the ghost VPs (Ghost_VP_generation, :250-308), which take
// part in the assignment (a point nearest a ghost belongs to no VP, label -1)
// and bound the VPs' cells like walls.
// Compiled with -fmad=false: every operation rounds as written, in the same
// order as the oracle, so labels and VP positions match it bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "handle.h"
#include "mrsph_cvp_clip.cuh"

namespace mrsph {
namespace {

constexpr int CVP_CHUNK = 2048;
constexpr int CVP_MAX_K = 1024;

// K VPs; the points that bound their cells are the K VPs, then GM ghost
// slots (0 without a level set, else K), then the 2 D box walls: NP planes
// per VP.  Bisector planes are stored per VP for the K + GM points.
struct CvpGeo {
  int dim, K, GM, NP;
  double box_l[3], box_r[3];
};

struct CvpState {  // device-resident iteration state
  double relax, error_record, error_max, total_energy, target;
  int converged, iter;
  int nghost;  // ghosts of the current iteration (in slots K .. K + nghost - 1)
  int nface;   // (VP, plane) pairs queued for k_cvp_faces
};

__device__ inline double cdot(const double* a, const double* b) {
  double s = 0.0;
  s += a[0] * b[0];
  s += a[1] * b[1];
  s += a[2] * b[2];
  return s;
}

__device__ inline double cdist(int D, const double* a, const double* b) {
  double s = 0.0;
  s += (a[0] - b[0]) * (a[0] - b[0]);
  s += (a[1] - b[1]) * (a[1] - b[1]);
  if (D == 3) s += (a[2] - b[2]) * (a[2] - b[2]);
  return sqrt(s);
}

__device__ inline double cmin(double a, double b) { return a <= b ? a : b; }
__device__ inline double cmax(double a, double b) { return a >= b ? a : b; }

// plane p of VP k: a bisector with point p (p < K + GM; vp holds the VPs and
// the ghost slots) or wall p - K - GM
__device__ void cplane(const CvpGeo& G, const double* vp, int k, int p, double* n, double* d) {
  if (p < G.K + G.GM) {
    const double* ck = vp + 3 * k;
    const double* cm = vp + 3 * p;
    double e[3] = {cm[0] - ck[0], cm[1] - ck[1], cm[2] - ck[2]};
    double len = sqrt(cdot(e, e));
    double mid[3] = {0.5 * (ck[0] + cm[0]), 0.5 * (ck[1] + cm[1]), 0.5 * (ck[2] + cm[2])};
    for (int q = 0; q < 3; q++) n[q] = e[q] / len;
    *d = cdot(n, mid);
  } else {
    int w = p - G.K - G.GM, ax = w / 2, hi = w % 2;
    n[0] = n[1] = n[2] = 0.0;
    n[ax] = hi ? 1.0 : -1.0;
    *d = hi ? G.box_r[ax] : -G.box_l[ax];
  }
}

// Nearest VP, strict '<' on the FP64 distance (lowest index wins a tie).  An
// FP32 pass finds the smallest FP32 distance first; only VPs within twice the
// FP32 error bound of it (1e-6 x (coordinate magnitude + distance), several
// times the bound) are then compared in FP64, in index order.  Every VP whose
// FP64 distance ties the minimum is among them, so the label is the one the
// full FP64 scan gives.  vp holds the K VPs and then st->nghost ghost VPs
// (st NULL: none); a point nearest a ghost gets label -1.
__global__ void k_cvp_assign(long long n, const double* __restrict__ xyz, int KV, const double* __restrict__ vp,
                             int D, int* __restrict__ label, const CvpState* st) {
  __shared__ double s_vp[3 * CVP_MAX_K];
  __shared__ float4 s_vf[CVP_MAX_K];
  __shared__ int s_lvp;  // largest |VP coordinate| (FP32 bits)
  const int K = KV + (st ? st->nghost : 0);
  if (threadIdx.x == 0) s_lvp = 0;
  __syncthreads();
  float lm = 0.f;
  for (int t = threadIdx.x; t < 3 * K; t += blockDim.x) {
    const double v = vp[t];
    s_vp[t] = v;
    lm = fmaxf(lm, fabsf((float)v));
  }
  const int wm = __reduce_max_sync(0xffffffffu, __float_as_int(lm));
  if ((threadIdx.x & 31) == 0) atomicMax(&s_lvp, wm);
  __syncthreads();
  for (int t = threadIdx.x; t < K; t += blockDim.x)
    s_vf[t] = make_float4((float)s_vp[3 * t], (float)s_vp[3 * t + 1], (float)s_vp[3 * t + 2], 0.f);
  __syncthreads();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double x[3] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
  const float xf[3] = {(float)x[0], (float)x[1], D == 3 ? (float)x[2] : 0.f};
  float bf = 3.4e38f, b2 = 3.4e38f;  // smallest and second smallest FP32 distance
  int bk = 0;
#pragma unroll 4
  for (int k = 0; k < K; k++) {
    const float4 v = s_vf[k];
    const float dx = xf[0] - v.x, dy = xf[1] - v.y, dz = D == 3 ? xf[2] - v.z : 0.f;
    const float dd = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    b2 = fminf(b2, fmaxf(bf, dd));
    if (dd < bf) { bf = dd; bk = k; }
  }
  const float L = fmaxf(__int_as_float(s_lvp), fmaxf(fabsf(xf[0]), fmaxf(fabsf(xf[1]), fabsf(xf[2]))));
  const float df = sqrtf(bf);
  const float thr = df + 2.e-6f * (L + df) + 1.e-30f;
  const float T = thr * thr * 1.0001f;
  if (b2 > T) {  // no other VP within the bound: the FP64 scan would pick bk
    label[i] = bk < KV ? bk : -1;
    return;
  }
  double best = 1.e20;
  int idx = 0;
  for (int k = 0; k < K; k++) {
    const float4 v = s_vf[k];
    const float dx = xf[0] - v.x, dy = xf[1] - v.y, dz = D == 3 ? xf[2] - v.z : 0.f;
    if (fmaf(dz, dz, fmaf(dy, dy, dx * dx)) > T) continue;
    double dd = cdist(D, x, s_vp + 3 * k);
    if (dd < best) { best = dd; idx = k; }
  }
  label[i] = idx < KV ? idx : -1;
}

// VPs k > 0 that hold a point with surface mass (the reference's
// contains_cutcell, colour > 0, voronoi_lset.cpp:256-266)
__global__ void k_cvp_flags(long long n, const double* __restrict__ psurf, const int* __restrict__ label,
                            unsigned char* flag) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int l = label[i];
  if (l > 0 && psurf[i] > 0.) flag[l] = 1;
}

// One block: the VPs copied to the point array, then thread 0 makes the ghost
// VPs in VP order (Ghost_VP_generation, voronoi_lset.cpp:276-301): x - 2 phi n
// with phi and the interpolated normal at the VP, when phi >= 1e-6 there;
// the flags are cleared for the next iteration.
template <int D>
__global__ void k_cvp_ghosts(LsSet ls, int K, const double* __restrict__ vp, unsigned char* flag, double* src,
                             CvpState* st) {
  for (int t = threadIdx.x; t < 3 * K; t += blockDim.x) src[t] = vp[t];
  __syncthreads();
  if (threadIdx.x != 0) return;
  int G = 0;
  for (int k = 0; k < K; k++) {
    if (!flag[k]) continue;
    flag[k] = 0;
    double phi, nn[3], cv;
    ls_sample<D, double>(ls, vp + 3 * k, phi, nn, cv);
    if (phi >= 1.e-6) {
      double* g = src + 3 * (K + G);
      for (int q = 0; q < 3; q++) g[q] = q < D ? vp[3 * k + q] - 2. * phi * nn[q] : vp[3 * k + q];
      G++;
    }
  }
  st->nghost = G;
}

// total point mass in chunked order (Set_target_mass, voronoi.cpp:495-510):
// a block loads its chunk, one thread adds it up in point order
__global__ void __launch_bounds__(256) k_cvp_chunk_mass(long long n, const double* __restrict__ pm, double* out) {
  __shared__ double s_m[CVP_CHUNK];
  const long long b = (long long)blockIdx.x * CVP_CHUNK;
  const int m = (int)min((long long)CVP_CHUNK, n - b);
  for (int t = threadIdx.x; t < m; t += blockDim.x) s_m[t] = pm[b + t];
  __syncthreads();
  if (threadIdx.x != 0) return;
  double s = 0.0;
#pragma unroll 8
  for (int t = 0; t < m; t++) s += s_m[t];
  out[blockIdx.x] = s;
}

__global__ void __launch_bounds__(256) k_cvp_target(long long nchunk, const double* tm, int K, CvpState* st) {
  __shared__ double s_m[CVP_CHUNK];
  double s = 0.0;
  for (long long c0 = 0; c0 < nchunk; c0 += CVP_CHUNK) {
    const int m = (int)min((long long)CVP_CHUNK, nchunk - c0);
    for (int t = threadIdx.x; t < m; t += blockDim.x) s_m[t] = tm[c0 + t];
    __syncthreads();
    if (threadIdx.x == 0)
      for (int t = 0; t < m; t++) s += s_m[t];
    __syncthreads();
  }
  if (threadIdx.x == 0) st->target = s / K;
}

// Per 2048-point chunk (one block): the chunk's points grouped by VP in point
// order (a stable counting sort in shared memory, each warp over its own 256
// points), every point's five summands computed in parallel, then each (VP,
// component) added up over the VP's points in order, so every (VP, chunk)
// partial adds the same values in the same order as a scan of the chunk per
// VP would, in O(chunk) work instead of O(K x chunk).  The sums' threads only
// read and add shared memory: the FP64 distances (a square root each) run on
// all lanes instead of inside the uneven per-VP loops, and no thread waits on
// a gather (80 -> 36 us for 301,270 points and 128 VPs).
// part: [chunk][component][VP].
constexpr int kPartWarps = 8;
inline size_t partials_smem(int K) {
  return sizeof(double) * 5 * CVP_CHUNK + sizeof(int) * (K + 1) + sizeof(unsigned short) * ((size_t)kPartWarps * K + CVP_CHUNK);
}
__global__ void __launch_bounds__(32 * kPartWarps) k_cvp_partials(long long n, const double* __restrict__ xyz,
                                                                  const double* __restrict__ pm,
                                                                  const int* __restrict__ label, int K,
                                                                  const double* __restrict__ vp, int D,
                                                                  double* __restrict__ part) {
  extern __shared__ double s_term[];  // 5 x CVP_CHUNK
  int* s_start = reinterpret_cast<int*>(s_term + 5 * CVP_CHUNK);                  // K + 1
  unsigned short* s_cnt = reinterpret_cast<unsigned short*>(s_start + (K + 1));  // [warp][VP]
  unsigned short* s_list = s_cnt + (size_t)kPartWarps * K;                        // CVP_CHUNK
  const long long c = blockIdx.x;
  const long long b = c * (long long)CVP_CHUNK;
  const int m = (int)min((long long)CVP_CHUNK, n - b);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int k = tid; k < kPartWarps * K; k += blockDim.x) s_cnt[k] = 0;
  __syncthreads();
  constexpr int SEG = CVP_CHUNK / kPartWarps;  // points per warp
  unsigned short* cnt = s_cnt + (size_t)wid * K;
  int lab[SEG / 32];
#pragma unroll
  for (int r = 0; r < SEG / 32; r++) {
    const int t = wid * SEG + r * 32 + lane;
    const int l = t < m ? __ldg(&label[b + t]) : -1;  // -1: nearest a ghost, no VP
    lab[r] = l;
    const unsigned act = __ballot_sync(0xffffffffu, l >= 0);
    if (l >= 0) {
      const long long i = b + t;
      const double w = pm[i];
      const double p[3] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
      const double ck[3] = {vp[3 * l], vp[3 * l + 1], vp[3 * l + 2]};
      s_term[t] = w;
      s_term[CVP_CHUNK + t] = p[0] * w;
      s_term[2 * CVP_CHUNK + t] = p[1] * w;
      s_term[3 * CVP_CHUNK + t] = p[2] * w;
      s_term[4 * CVP_CHUNK + t] = w * cdist(D, ck, p);
      const unsigned peers = __match_any_sync(act, l);
      if ((peers & ((1u << lane) - 1u)) == 0) cnt[l] += (unsigned short)__popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
  if (wid == 0) {  // exclusive scan, VP by VP and warp by warp: counts become fill cursors
    int run = 0;
    for (int k0 = 0; k0 < K; k0 += 32) {
      const int k = k0 + lane;
      int v = 0;
      if (k < K)
        for (int w = 0; w < kPartWarps; w++) v += s_cnt[(size_t)w * K + k];
      int inc = v;
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (k < K) {
        int at = run + inc - v;
        s_start[k] = at;
        for (int w = 0; w < kPartWarps; w++) {
          const int cw = s_cnt[(size_t)w * K + k];
          s_cnt[(size_t)w * K + k] = (unsigned short)at;
          at += cw;
        }
      }
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_start[K] = run;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < SEG / 32; r++) {
    const int l = lab[r];
    const unsigned act = __ballot_sync(0xffffffffu, l >= 0);
    if (l >= 0) {
      const unsigned peers = __match_any_sync(act, l);
      const int rank = __popc(peers & ((1u << lane) - 1u));
      s_list[cnt[l] + rank] = (unsigned short)(wid * SEG + r * 32 + lane);
      __syncwarp(act);
      if (rank == 0) cnt[l] += (unsigned short)__popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
  for (int q = tid; q < 5 * K; q += blockDim.x) {
    const int j = q / K, k = q - j * K;
    const double* term = s_term + j * CVP_CHUNK;
    double v = 0.0;
    for (int t = s_start[k]; t < s_start[k + 1]; t++) v += term[s_list[t]];
    part[(size_t)c * 5 * K + q] = v;
  }
}

// 32 VPs x 5 components per block, each thread over the chunks in order (the
// loads of a batch of chunks are independent of the running sum)
__global__ void __launch_bounds__(160) k_cvp_reduce(long long nchunk, int K, int D, const double* __restrict__ part,
                                                    const CvpState* st, const double* __restrict__ vp, double* mass,
                                                    double* mc, double* energy, double* P, double* err) {
  __shared__ double s_v[5][32];
  const int kl = threadIdx.x & 31, j = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + kl;
  double v = 0.0;
  if (k < K) {
    const double* q = part + (size_t)j * K + k;
    const size_t step = (size_t)5 * K;
    long long c = 0;
    for (; c + 16 <= nchunk; c += 16) {
      double t[16];
#pragma unroll
      for (int u = 0; u < 16; u++) t[u] = q[(size_t)(c + u) * step];
#pragma unroll
      for (int u = 0; u < 16; u++) v += t[u];
    }
    for (; c < nchunk; c++) v += q[(size_t)c * step];
  }
  s_v[j][kl] = v;
  __syncthreads();
  if (j != 0 || k >= K) return;
  const double m = s_v[0][kl], x = s_v[1][kl], y = s_v[2][kl], z = s_v[3][kl], e = s_v[4][kl];
  mass[k] = m;
  energy[k] = e;
  double target = st->target;
  if (m > 0.) {
    double inv = 1. / m;
    mc[3 * k] = x * inv;
    mc[3 * k + 1] = y * inv;
    mc[3 * k + 2] = (D == 3) ? z * inv : 0.0;
    P[k] = target / m;
  } else {
    // a cell without points (the reference divides by its zero mass):
    // centroid = its position, no pressure; it does not move (k_cvp_update)
    for (int q = 0; q < 3; q++) mc[3 * k + q] = vp[3 * k + q];
    P[k] = 0.;
  }
  err[k] = fabs(m - target) / target;
}

// bisector planes of every (VP, point) pair, computed once per iteration
// (row stride K + GM; slots of absent ghosts are left alone)
__global__ void k_cvp_planes(CvpGeo G, const double* __restrict__ vp, double* __restrict__ planes,
                             float4* __restrict__ planes_f, CvpState* st) {
  const int PS = G.K + G.GM;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) st->nface = 0;
  if (t >= (long long)G.K * PS) return;
  int k = (int)(t / PS), m = (int)(t % PS);
  if (k == m || m >= G.K + st->nghost) return;
  double n[3], d;
  cplane(G, vp, k, m, n, &d);
  double* o = planes + 4 * t;
  o[0] = n[0]; o[1] = n[1]; o[2] = n[2]; o[3] = d;
  planes_f[t] = make_float4((float)n[0], (float)n[1], (float)n[2], (float)d);
}

// The polygon of plane (n, d) before any clip: a square of half side S (twice
// the box diagonal) around the foot of the box centre, one corner per lane
// 0..3; and the box (z from -0.5 to 0.5 in 2D).
template <class T>
__device__ void face_square(const CvpGeo& G, const Lanes& g, const T* n, T d, T* lo, T* hi, T& S, T (*A)[3]) {
  for (int q = 0; q < 3; q++) {
    lo[q] = q < G.dim ? (T)G.box_l[q] : (T)-0.5;
    hi[q] = q < G.dim ? (T)G.box_r[q] : (T)0.5;
  }
  auto dot = [](const T* a, const T* b) {
    T t = 0;
    t += a[0] * b[0];
    t += a[1] * b[1];
    t += a[2] * b[2];
    return t;
  };
  const T h = (T)0.5;
  T c[3] = {h * (lo[0] + hi[0]), h * (lo[1] + hi[1]), h * (lo[2] + hi[2])};
  S = 0;
  for (int q = 0; q < 3; q++) S += (hi[q] - lo[q]) * (hi[q] - lo[q]);
  S = (T)2.0 * sqrt(S);
  int ax = 0;
  if (fabs(n[1]) < fabs(n[ax])) ax = 1;
  if (fabs(n[2]) < fabs(n[ax])) ax = 2;
  T e[3] = {0, 0, 0};
  e[ax] = 1;
  T u[3] = {n[1] * e[2] - n[2] * e[1], n[2] * e[0] - n[0] * e[2], n[0] * e[1] - n[1] * e[0]};
  T ul = sqrt(dot(u, u));
  for (int q = 0; q < 3; q++) u[q] = u[q] / ul;
  T w[3] = {n[1] * u[2] - n[2] * u[1], n[2] * u[0] - n[0] * u[2], n[0] * u[1] - n[1] * u[0]};
  T off = d - dot(n, c);
  T p0[3] = {c[0] + n[0] * off, c[1] + n[1] * off, c[2] + n[2] * off};
  const int a = g.gl;
  if (a < 4) {
    const T su = (a == 1 || a == 2) ? (T)1 : (T)-1, sw = a >= 2 ? (T)1 : (T)-1;  // (-,-) (+,-) (+,+) (-,+)
    for (int q = 0; q < 3; q++) A[a][q] = p0[q] + u[q] * (su * S) + w[q] * (sw * S);
  }
  __syncwarp();
}

// Whether plane (n, d) may cut the polygon v (FP32): no when every vertex
// lies more than margin inside.  Undecidable values (NaN) count as cutting.
__device__ inline bool face_may_cut(const float (*v)[3], int nv, const float4& pl, float margin) {
  bool cut = false;
  for (int a = 0; a < nv; a++)
    cut = cut || !((pl.x * v[a][0] + pl.y * v[a][1] + pl.z * v[a][2]) - pl.w <= -margin);
  return cut;
}

// Pass 1 of the faces, kGroup lanes per (VP k, plane p): the polygon clipped
// in FP32 by every other plane moved outwards by 4e-5 of the magnitudes
// (|d| + box coordinates + S), hundreds of times the rounding a vertex
// collects over the clips.  The result then holds the exact polygon, so an
// empty one proves that the pair has no face; the others (about one in six)
// are queued for the FP64 pass.  FP64 runs at 1/60 of the FP32 rate here, and
// most pairs are far apart.  49 us for 128 VPs in 3D (17,152 pairs).
constexpr float kCullMargin = 4.e-5f;
__global__ void __launch_bounds__(128) k_cvp_face_cull(CvpGeo G, const double* __restrict__ vp,
                                                       const float4* __restrict__ planes_f,
                                                       double* __restrict__ face, int* __restrict__ queue,
                                                       CvpState* st) {
  __shared__ float s_v[128 / kGroup][2][CVP_MAXV][3];
  __shared__ float s_s[128 / kGroup][CVP_MAXV];
  const Lanes g;
  const int grp = threadIdx.x / kGroup;
  const long long t = (long long)blockIdx.x * (128 / kGroup) + grp;
  const int PS = G.K + G.GM, NPT = G.K + st->nghost;  // plane row stride, points present
  bool live = t < (long long)G.K * G.NP;
  const int k = live ? (int)(t / G.NP) : 0, p = live ? (int)(t % G.NP) : 0;
  if (live && g.gl == 0) face[6 * t] = 0.0;
  live = live && !(p < G.K && p == k) && !(p >= NPT && p < PS);  // not a VP with itself, not an unused ghost slot
  const float4* pkf = planes_f + (long long)k * PS;
  float n[3] = {1.f, 0.f, 0.f}, d = 0.f;
  if (live && p < PS) {
    const float4 pl = pkf[p];
    n[0] = pl.x; n[1] = pl.y; n[2] = pl.z; d = pl.w;
  } else if (live) {
    double nd[3], dd;
    cplane(G, vp, k, p, nd, &dd);
    for (int q = 0; q < 3; q++) n[q] = (float)nd[q];
    d = (float)dd;
  }
  float lo[3], hi[3], S;
  float (*A)[3] = s_v[grp][0], (*B)[3] = s_v[grp][1];
  face_square<float>(G, g, n, d, lo, hi, S, A);
  float mag = S;
  for (int q = 0; q < 3; q++) mag += fmaxf(fabsf(lo[q]), fabsf(hi[q]));
  int nv = live ? 4 : 0;
  // left to the FP64 pass: a box whose squares leave FP32's range (S is then 0 or
  // infinite), or more vertices than are kept
  bool full = !(mag > 1.e-15f && mag < 1.e15f);
  auto clip = [&](const float* cn, float cd, bool act) {
    const int no = gclip<float>(g, A, act ? nv : 0, cn, cd + kCullMargin * (mag + fabsf(cd)), B, s_s[grp]);
    if (no < 0) return;
    full = full || no > CVP_MAXV;
    nv = min(no, CVP_MAXV);
    float (*tmp)[3] = A;
    A = B;
    B = tmp;
  };
  for (int wq = 0; wq < 6; wq++) {
    float wn[3] = {0.f, 0.f, 0.f};
    wn[wq / 2] = (wq & 1) ? 1.f : -1.f;
    clip(wn, (wq & 1) ? hi[wq / 2] : -lo[wq / 2], !(p >= PS && wq == p - PS));
  }
  // the groups test planes on their own and clip together
  float4 pl = make_float4(0.f, 0.f, 0.f, 0.f);
  unsigned cm = 0;
  int m0 = 0;
  while (true) {
    while (__any_sync(0xffffffffu, cm == 0 && nv > 0 && !full && m0 < NPT)) {
      const bool look = cm == 0 && nv > 0 && !full && m0 < NPT;
      const int m = m0 + g.gl;
      bool cut = false;
      if (look && m < NPT && m != k && m != p) {
        pl = __ldg(&pkf[m]);
        cut = face_may_cut(A, nv, pl, -kCullMargin * (mag + fabsf(pl.w)));
      }
      const unsigned b = g.ballot(cut);
      if (look) { cm = b; m0 += kGroup; }
    }
    const bool act = cm != 0 && nv > 0 && !full;
    if (!__any_sync(0xffffffffu, act)) break;
    const int q = g.shift + (act ? __ffs(cm) - 1 : 0);
    cm &= cm - 1u;
    const float cn[3] = {__shfl_sync(0xffffffffu, pl.x, q), __shfl_sync(0xffffffffu, pl.y, q),
                         __shfl_sync(0xffffffffu, pl.z, q)};
    clip(cn, __shfl_sync(0xffffffffu, pl.w, q), act);
  }
  if (live && g.gl == 0 && (full || nv > 0)) queue[atomicAdd(&st->nface, 1)] = (int)t;
}

// Pass 2, kGroup lanes per queued pair: face of VP k on plane p; out: exists,
// area, n (3), dist.  The clips run in plane order; a plane is skipped only
// when an FP32 test with a margin (4e-6 of the magnitudes, far above its
// rounding) shows every vertex inside, which would keep the polygon as it is,
// so the result is the one of clipping by every plane in turn.
__global__ void __launch_bounds__(64) k_cvp_faces(CvpGeo G, const double* __restrict__ vp,
                                                  const double* __restrict__ planes,
                                                  const float4* __restrict__ planes_f, double* __restrict__ face,
                                                  const int* __restrict__ queue, const CvpState* st) {
  __shared__ double s_v[64 / kGroup][2][CVP_MAXV][3];
  __shared__ double s_s[64 / kGroup][CVP_MAXV];
  __shared__ float s_f[64 / kGroup][CVP_MAXV][3];
  const Lanes g;
  const int grp = threadIdx.x / kGroup, nq = st->nface;
  const int PS = G.K + G.GM, NPT = G.K + st->nghost;
  double* s = s_s[grp];
  float (*vf)[3] = s_f[grp];
  for (int it0 = blockIdx.x * (64 / kGroup) + (grp & ~3); it0 < nq; it0 += gridDim.x * (64 / kGroup)) {  // warp-uniform
    const int it = it0 + (grp & 3);
    const bool live = it < nq;
    const int t = queue[live ? it : it0];
    const int k = t / G.NP, p = t % G.NP;
    double* out = face + 6 * (long long)t;
    double n[3], d;
    if (p < PS) {
      const double* pl = planes + 4 * ((long long)k * PS + p);
      n[0] = pl[0]; n[1] = pl[1]; n[2] = pl[2]; d = pl[3];
    } else {
      cplane(G, vp, k, p, n, &d);
    }
    double lo[3], hi[3], S;
    double (*A)[3] = s_v[grp][0], (*B)[3] = s_v[grp][1];
    face_square<double>(G, g, n, d, lo, hi, S, A);
    int nv = live ? 4 : 0;
    auto clip = [&](const double* cn, double cd, bool act) {
      const int no = gclip<double>(g, A, act ? nv : 0, cn, cd, B, s);
      if (no < 0) return;
      nv = min(no, CVP_MAXV);
      double (*tmp)[3] = A;
      A = B;
      B = tmp;
      for (int a = g.gl; a < nv; a += kGroup)
        for (int q = 0; q < 3; q++) vf[a][q] = (float)A[a][q];
    };
    for (int a = g.gl; a < nv; a += kGroup)
      for (int q = 0; q < 3; q++) vf[a][q] = (float)A[a][q];
    for (int wq = 0; wq < 6; wq++) {
      double wn[3] = {0, 0, 0};
      wn[wq / 2] = (wq & 1) ? 1.0 : -1.0;
      clip(wn, (wq & 1) ? hi[wq / 2] : -lo[wq / 2], !(p >= PS && wq == p - PS));
    }
    float mag = (float)S;
    for (int q = 0; q < 3; q++) mag += fmaxf(fabsf((float)lo[q]), fabsf((float)hi[q]));
    const double* pk = planes + 4 * (long long)k * PS;
    const float4* pkf = planes_f + (long long)k * PS;
    // the groups look for their next cutting plane on their own and clip together
    int m0 = 0, cur = -1;  // next plane to test; the plane to clip by
    while (true) {
      __syncwarp();
      while (__any_sync(0xffffffffu, cur < 0 && nv > 0 && m0 < NPT)) {
        const bool look = cur < 0 && nv > 0 && m0 < NPT;
        const int m = m0 + g.gl;
        bool cut = false;
        if (look && m < NPT && m != k && m != p) {
          const float4 pl = __ldg(&pkf[m]);
          cut = face_may_cut(vf, nv, pl, 4.001e-6f * (mag + fabsf(pl.w)));
        }
        const unsigned cm = g.ballot(cut);
        if (look) {
          if (cm) cur = m0 + __ffs(cm) - 1;
          m0 = cm ? cur + 1 : m0 + kGroup;
        }
      }
      if (!__any_sync(0xffffffffu, cur >= 0)) break;
      const double* bn = pk + 4 * (cur >= 0 ? cur : 0);
      clip(bn, bn[3], cur >= 0);
      cur = -1;
    }
    if (nv >= 3) {
      for (int a = 1 + g.gl; a + 1 < nv; a += kGroup) {
        double x[3] = {A[a][0] - A[0][0], A[a][1] - A[0][1], A[a][2] - A[0][2]};
        double y[3] = {A[a + 1][0] - A[0][0], A[a + 1][1] - A[0][1], A[a + 1][2] - A[0][2]};
        double cr[3] = {x[1] * y[2] - x[2] * y[1], x[2] * y[0] - x[0] * y[2], x[0] * y[1] - x[1] * y[0]};
        s[a] = cdot(cr, n);
      }
    }
    __syncwarp();
    if (nv >= 3) {
      double ar = 0.0;
      for (int a = 1; a + 1 < nv; a++) ar += s[a];
      ar = 0.5 * fabs(ar);
      double ext = S * S;
      if (g.gl == 0 && ar > 1.e-13 * ext) {
        const double* ck = vp + 3 * k;
        double dx[3] = {A[0][0] - ck[0], A[0][1] - ck[1], A[0][2] - ck[2]};
        out[0] = 1.0;
        out[1] = ar;
        out[2] = n[0];
        out[3] = n[1];
        out[4] = n[2];
        out[5] = fabs(cdot(dx, n)) * 2.;
      }
    }
    __syncwarp();
  }
}

// Face pressure force and length scale h of every VP, one warp per VP: the
// lanes read 32 planes' faces at a time, the sums run over the faces in plane
// order.
__global__ void __launch_bounds__(128) k_cvp_force(CvpGeo G, const double* __restrict__ face,
                                                   const double* __restrict__ P, double* f, double* hk,
                                                   const CvpState* st) {
  const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (k >= G.K) return;
  const int K = G.K, NP = G.NP;
  double fx = 0.0, fy = 0.0, fz = 0.0, sr = 0.0;
  int nnb = 0;
  for (int p0 = 0; p0 < NP; p0 += 32) {
    const int p = p0 + lane;
    const double* fc = face + 6 * ((size_t)k * NP + p);
    const bool has = p < NP && fc[0] != 0.0;
    double vx = 0.0, vy = 0.0, vz = 0.0, vr = 0.0;
    if (has) {
      double nP = (p < K) ? P[p] : P[k];
      double pmid = 0.5 * (P[k] + nP);
      double coef = -1 * pmid * fc[1];
      vx = fc[2] * coef;
      vy = fc[3] * coef;
      vz = fc[4] * coef;
      vr = fc[5];
    }
    unsigned m = __ballot_sync(0xffffffffu, has);
    nnb += __popc(m);
    while (m) {
      const int q = __ffs(m) - 1;
      m &= m - 1u;
      sr += __shfl_sync(0xffffffffu, vr, q);
      fx = fx + __shfl_sync(0xffffffffu, vx, q);
      fy = fy + __shfl_sync(0xffffffffu, vy, q);
      fz = fz + __shfl_sync(0xffffffffu, vz, q);
    }
  }
  if (lane == 0) {
    const double scale_coeff = 0.25 + 1.75 * (1. - cmin((st->iter - 1) / 500., 1.));
    f[3 * k] = fx; f[3 * k + 1] = fy; f[3 * k + 2] = fz;
    hk[k] = scale_coeff * sr / (double)nnb;
  }
}

// minimum of v over the block (cmin is exact; no thread's value is NaN)
__device__ double block_cmin(double v, double* s_w) {
  for (int o = 16; o > 0; o >>= 1) v = cmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  double r = s_w[0];
  for (int w = 1; w < nw; w++) r = cmin(r, s_w[w]);
  __syncthreads();
  return r;
}

// VP update, one block: per-VP work in parallel (thread k handles VPs
// k, k + blockDim, ...), the order-sensitive scalars (error and energy sums)
// on thread 0 in VP order from shared memory, as the reference loops do.
__global__ void __launch_bounds__(1024) k_cvp_update(CvpGeo G, double* vp, const double* mass, const double* mc,
                                                     const double* energy, const double* err, const double* f,
                                                     const double* hk, double* shift, CvpState* st,
                                                     double error_tolerance, int pressure_step) {
  __shared__ double s_en[CVP_MAX_K], s_er[CVP_MAX_K];
  __shared__ double s_w[32];
  __shared__ int s_conv;
  const int K = G.K, D = G.dim;
  const int iter = st->iter;
  const double relax = st->relax;  // read by every thread before thread 0 updates it
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    s_en[k] = energy[k];
    s_er[k] = err[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double error_max = 0.0, total_energy = 0.0;
#pragma unroll 4
    for (int k = 0; k < K; k++) {
      error_max = cmax(error_max, s_er[k]);
      total_energy += s_en[k];
    }
    st->error_record = st->error_record + error_max;
    if (iter % 40 == 0) {
      st->error_record /= 40.;
      if (error_max <= error_tolerance && st->error_record <= error_tolerance) st->converged = 1;
      st->error_record = 0.;
    }
    st->error_max = error_max;
    st->total_energy = total_energy;
    s_conv = st->converged;
  }
  __syncthreads();
  if (s_conv == 0) {
    double gdt = 1.e20;
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
      if (!(mass[k] > 0.)) continue;  // an empty cell neither moves nor limits the step
      double inv = 1. / mass[k];
      double acc = 0.0;
      for (int q = 0; q < D; q++) {
        double a = f[3 * k + q] * inv;
        acc += a * a;
      }
      acc = sqrt(acc);
      gdt = cmin(0.25 * sqrt(hk[k] / (acc + 1.e-20)), gdt);
    }
    gdt = block_cmin(gdt, s_w);
    double gcvt = 1.e20;
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
      const bool full = mass[k] > 0.;
      double inv = full ? 1. / mass[k] : 0.;
      double fac = gdt * gdt * 0.5 * relax;
      for (int q = 0; q < D; q++) {
        double a = full ? f[3 * k + q] * inv : 0.0;
        double v = pressure_step ? vp[3 * k + q] + a * fac : vp[3 * k + q];
        vp[3 * k + q] = cmax(G.box_l[q] + 1.e-20, cmin(v, G.box_r[q] - 1.e-20));
      }
      double sh = 0.0;
      for (int q = 0; q < D; q++) {
        shift[3 * k + q] = mc[3 * k + q] - vp[3 * k + q];
        sh += shift[3 * k + q] * shift[3 * k + q];
      }
      sh = sqrt(sh);
      double sc = cmin(sh, 1. / 32. * hk[k]);
      if (full) gcvt = cmin(sc / (sh + 1.e-20), gcvt);
    }
    gcvt = block_cmin(gcvt, s_w);
    for (int k = threadIdx.x; k < K; k += blockDim.x)
      for (int q = 0; q < D; q++) {
        double v = vp[3 * k + q] + shift[3 * k + q] * (gcvt * (1 - relax));
        vp[3 * k + q] = cmax(G.box_l[q] + 1.e-20, cmin(v, G.box_r[q] - 1.e-20));
      }
  }
  if (threadIdx.x == 0) {
    double r = relax;
    if (iter % 600 == 0) r = 1.02 * r;
    st->relax = cmin(r, 0.90);
    st->iter = iter + 1;
  }
}

int cfail(mrsph_handle* h, int code, const std::string& msg) {
  h->err = msg;
  return code;
}

#define CV_CK(call)                                                                     \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) { rc = cfail(h, MRSPH_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); goto done; } \
  } while (0)

// Core loop on device points (xyz n x 3, pm n), id order.  d_ps (surface
// mass per point) not NULL: the level-set partition with ghost VPs on the
// handle's level set; ghost_xyz (K x 3) / nghost (may be NULL) receive the
// last iteration's ghosts.
int cvp_run(mrsph_handle* h, long long n, double* d_xyz, double* d_pm, const mrsph_cvp_params* p, double* vp_xyz,
            int* labels, double* vp_mass, mrsph_cvp_result* res, const double* d_ps = nullptr,
            double* ghost_xyz = nullptr, int* nghost = nullptr) {
  const int K = p->num_vp, D = h->prm.dim;
  const bool ghosts = d_ps != nullptr;
  CvpGeo G;
  G.dim = D;
  G.K = K;
  G.GM = ghosts ? K : 0;
  G.NP = K + G.GM + 2 * D;
  for (int q = 0; q < 3; q++) {
    G.box_l[q] = h->prm.box_l[q];
    G.box_r[q] = h->prm.box_r[q];
  }
  const long long nchunk = (n + CVP_CHUNK - 1) / CVP_CHUNK;
  cudaStream_t s = h->stream;
  int rc = 0;
  std::vector<void*> mem;
  double *d_vp = nullptr, *d_part = nullptr, *d_face = nullptr, *d_k = nullptr, *d_tm = nullptr, *d_planes = nullptr;
  double* d_src = nullptr;  // VPs then ghost VPs (level-set partition)
  unsigned char* d_flag = nullptr;
  float4* d_planes_f = nullptr;
  int *d_label = nullptr, *d_queue = nullptr;
  const size_t PS = (size_t)K + G.GM;
  CvpState* d_st = nullptr;
  CvpState hs;
  std::memset(&hs, 0, sizeof(hs));
  hs.relax = p->relax_ratio;
  auto A = [&](void** ptr, size_t bytes) -> cudaError_t {
    cudaError_t e = cudaMalloc(ptr, bytes);
    if (e == cudaSuccess) mem.push_back(*ptr);
    return e;
  };
  CV_CK(A((void**)&d_vp, sizeof(double) * 3 * K));
  CV_CK(A((void**)&d_part, sizeof(double) * 5 * K * nchunk));
  CV_CK(A((void**)&d_face, sizeof(double) * 6 * (size_t)K * G.NP));
  CV_CK(A((void**)&d_queue, sizeof(int) * (size_t)K * G.NP));
  CV_CK(A((void**)&d_planes, sizeof(double) * 4 * (size_t)K * PS));
  CV_CK(A((void**)&d_planes_f, sizeof(float4) * (size_t)K * PS));
  if (ghosts) {
    CV_CK(A((void**)&d_src, sizeof(double) * 3 * PS));
    CV_CK(A((void**)&d_flag, (size_t)K));
    CV_CK(cudaMemsetAsync(d_flag, 0, (size_t)K, h->stream));
  }
  CV_CK(A((void**)&d_k, sizeof(double) * 12 * K));  // mass, mc(3), energy, P, err, f(3), hk, pad
  CV_CK(A((void**)&d_tm, sizeof(double) * nchunk));
  CV_CK(A((void**)&d_label, sizeof(int) * n));
  CV_CK(A((void**)&d_st, sizeof(CvpState)));
  {
    double* vp3 = nullptr;
    CV_CK(A((void**)&vp3, sizeof(double) * 3 * K));  // shift
    CV_CK(cudaMemcpyAsync(d_vp, vp_xyz, sizeof(double) * 3 * K, cudaMemcpyHostToDevice, s));
    CV_CK(cudaMemcpyAsync(d_st, &hs, sizeof(hs), cudaMemcpyHostToDevice, s));
    double *mass = d_k, *mc = d_k + K, *energy = d_k + 4 * K, *P = d_k + 5 * K, *err = d_k + 6 * K,
           *f = d_k + 7 * K, *hk = d_k + 10 * K;
    k_cvp_chunk_mass<<<(unsigned)nchunk, 256, 0, s>>>(n, d_pm, d_tm);
    k_cvp_target<<<1, 256, 0, s>>>(nchunk, d_tm, K, d_st);
    const size_t psm = partials_smem(K);
    CV_CK(cudaFuncSetAttribute(k_cvp_partials, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)partials_smem(CVP_MAX_K)));
    const int nb = (int)((n + 255) / 256);
    const int ftot = K * G.NP;
    const int fgrid = std::min((ftot + 64 / kGroup - 1) / (64 / kGroup), 152 * 4);  // FP64 faces: the queue's length is known on the device only
    const double* pts = ghosts ? d_src : d_vp;  // the points that bound the cells
    // Voronoi_lset::Initialize: points coloured by their nearest VP
    if (ghosts) k_cvp_assign<<<nb, 256, 0, s>>>(n, d_xyz, K, d_vp, D, d_label, nullptr);
    int it = 0;
    for (; it <= p->max_iter; it++) {
      if (ghosts) {
        k_cvp_flags<<<nb, 256, 0, s>>>(n, d_ps, d_label, d_flag);
        if (D == 3) k_cvp_ghosts<3><<<1, 256, 0, s>>>(h->ls, K, d_vp, d_flag, d_src, d_st);
        else k_cvp_ghosts<2><<<1, 256, 0, s>>>(h->ls, K, d_vp, d_flag, d_src, d_st);
      }
      k_cvp_assign<<<nb, 256, 0, s>>>(n, d_xyz, K, pts, D, d_label, d_st);
      k_cvp_partials<<<(unsigned)nchunk, 32 * kPartWarps, psm, s>>>(n, d_xyz, d_pm, d_label, K, d_vp, D, d_part);
      k_cvp_reduce<<<(K + 31) / 32, 160, 0, s>>>(nchunk, K, D, d_part, d_st, d_vp, mass, mc, energy, P, err);
      k_cvp_planes<<<(int)((K * PS + 255) / 256), 256, 0, s>>>(G, pts, d_planes, d_planes_f, d_st);
      k_cvp_face_cull<<<(ftot + 128 / kGroup - 1) / (128 / kGroup), 128, 0, s>>>(G, pts, d_planes_f, d_face, d_queue,
                                                                              d_st);
      k_cvp_faces<<<fgrid, 64, 0, s>>>(G, pts, d_planes, d_planes_f, d_face, d_queue, d_st);
      k_cvp_force<<<(K + 3) / 4, 128, 0, s>>>(G, d_face, P, f, hk, d_st);
      k_cvp_update<<<1, (K + 31) / 32 * 32, 0, s>>>(G, d_vp, mass, mc, energy, err, f, hk, vp3, d_st,
                                                   p->error_tolerance, p->pressure_step);
      CV_CK(cudaGetLastError());
      // the convergence test falls due every 40 iterations (k_cvp_update); between
      // two of them the host has nothing to decide and does not wait
      if (it % 40 != 0 && it != p->max_iter) continue;
      CV_CK(cudaMemcpyAsync(&hs, d_st, sizeof(hs), cudaMemcpyDeviceToHost, s));
      CV_CK(cudaStreamSynchronize(s));
      if (hs.converged) { it++; break; }
    }
    CV_CK(cudaMemcpyAsync(vp_xyz, d_vp, sizeof(double) * 3 * K, cudaMemcpyDeviceToHost, s));
    if (labels) CV_CK(cudaMemcpyAsync(labels, d_label, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
    if (vp_mass) CV_CK(cudaMemcpyAsync(vp_mass, mass, sizeof(double) * K, cudaMemcpyDeviceToHost, s));
    if (ghosts && ghost_xyz)
      CV_CK(cudaMemcpyAsync(ghost_xyz, d_src + 3 * (size_t)K, sizeof(double) * 3 * K, cudaMemcpyDeviceToHost, s));
    CV_CK(cudaStreamSynchronize(s));
    if (nghost) *nghost = ghosts ? hs.nghost : 0;
    if (res) {
      res->iterations = it;
      res->converged = hs.converged;
      res->error_max = hs.error_max;
      res->total_energy = hs.total_energy;
    }
  }
done:
  for (void* q : mem) cudaFree(q);
  return rc;
}

}  // namespace
}  // namespace mrsph

using namespace mrsph;

static int cvp_check(mrsph_handle* h, const mrsph_cvp_params* p, double* vp_xyz) {
  if (!h) return MRSPH_ERR_ARG;
  if (!p || !vp_xyz) return cfail(h, MRSPH_ERR_ARG, "null argument");
  if (p->num_vp < 1 || p->num_vp > CVP_MAX_K) return cfail(h, MRSPH_ERR_RANGE, "num_vp must be 1..1024");
  if (p->max_iter < 0) return cfail(h, MRSPH_ERR_ARG, "max_iter must be >= 0");
  return 0;
}

extern "C" int mrsph_cvp_points(mrsph_handle* h, long long n, const double* xyz, const double* mass,
                                const mrsph_cvp_params* p, double* vp_xyz, int* labels, double* vp_mass,
                                mrsph_cvp_result* res) {
  int rc = cvp_check(h, p, vp_xyz);
  if (rc) return rc;
  if (n <= 0 || !xyz) return cfail(h, MRSPH_ERR_ARG, "no points");
  if (cudaSetDevice(h->prm.device) != cudaSuccess) return cfail(h, MRSPH_ERR_CUDA, "cudaSetDevice failed");
  double *d_xyz = nullptr, *d_pm = nullptr;
  if (cudaMalloc(&d_xyz, sizeof(double) * 3 * n) != cudaSuccess ||
      cudaMalloc(&d_pm, sizeof(double) * n) != cudaSuccess) {
    cudaFree(d_xyz);
    return cfail(h, MRSPH_ERR_OOM, "cudaMalloc failed");
  }
  std::vector<double> ones;
  const double* pm = mass;
  if (!pm) { ones.assign(n, 1.0); pm = ones.data(); }
  cudaMemcpyAsync(d_xyz, xyz, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, h->stream);
  cudaMemcpyAsync(d_pm, pm, sizeof(double) * n, cudaMemcpyHostToDevice, h->stream);
  rc = cvp_run(h, n, d_xyz, d_pm, p, vp_xyz, labels, vp_mass, res);
  cudaFree(d_xyz);
  cudaFree(d_pm);
  return rc;
}

extern "C" int mrsph_cvp_lset(mrsph_handle* h, long long n, const double* xyz, const double* mass,
                              const double* mass_surface, const mrsph_cvp_params* p, double* vp_xyz, int* labels,
                              double* vp_mass, double* ghost_xyz, int* num_ghost, mrsph_cvp_result* res) {
  int rc = cvp_check(h, p, vp_xyz);
  if (rc) return rc;
  if (n <= 0 || !xyz || !mass || !mass_surface) return cfail(h, MRSPH_ERR_ARG, "no points or masses");
  if (2 * p->num_vp > CVP_MAX_K) return cfail(h, MRSPH_ERR_RANGE, "num_vp must be 1..512 with ghost VPs");
  if (h->nls < 1) return cfail(h, MRSPH_ERR_STATE, "mrsph_set_levelset must come first");
  if (cudaSetDevice(h->prm.device) != cudaSuccess) return cfail(h, MRSPH_ERR_CUDA, "cudaSetDevice failed");
  double *d_xyz = nullptr, *d_pm = nullptr, *d_ps = nullptr;
  if (cudaMalloc(&d_xyz, sizeof(double) * 3 * n) != cudaSuccess || cudaMalloc(&d_pm, sizeof(double) * n) != cudaSuccess ||
      cudaMalloc(&d_ps, sizeof(double) * n) != cudaSuccess) {
    cudaFree(d_xyz);
    cudaFree(d_pm);
    return cfail(h, MRSPH_ERR_OOM, "cudaMalloc failed");
  }
  cudaMemcpyAsync(d_xyz, xyz, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, h->stream);
  cudaMemcpyAsync(d_pm, mass, sizeof(double) * n, cudaMemcpyHostToDevice, h->stream);
  cudaMemcpyAsync(d_ps, mass_surface, sizeof(double) * n, cudaMemcpyHostToDevice, h->stream);
  rc = cvp_run(h, n, d_xyz, d_pm, p, vp_xyz, labels, vp_mass, res, d_ps, ghost_xyz, num_ghost);
  cudaFree(d_xyz);
  cudaFree(d_pm);
  cudaFree(d_ps);
  return rc;
}

extern "C" int mrsph_cvp(mrsph_handle* h, const mrsph_cvp_params* p, double* vp_xyz, int* labels, double* vp_mass,
                         mrsph_cvp_result* res) {
  int rc = cvp_check(h, p, vp_xyz);
  if (rc) return rc;
  if (!h->eng) return cfail(h, MRSPH_ERR_STATE, "no particles");
  if (cudaSetDevice(h->prm.device) != cudaSuccess) return cfail(h, MRSPH_ERR_CUDA, "cudaSetDevice failed");
  long long n = h->eng->num_particles();
  if (n <= 0) return cfail(h, MRSPH_ERR_STATE, "no particles");
  double *d_xyz = nullptr, *d_pm = nullptr;
  if (cudaMalloc(&d_xyz, sizeof(double) * 3 * n) != cudaSuccess ||
      cudaMalloc(&d_pm, sizeof(double) * n) != cudaSuccess) {
    cudaFree(d_xyz);
    return cfail(h, MRSPH_ERR_OOM, "cudaMalloc failed");
  }
  rc = h->eng->world_positions(d_xyz);  // particle mass 1 (Particle_mesh_generation::Initialize)
  if (rc) { h->err = h->eng->err; cudaFree(d_xyz); cudaFree(d_pm); return rc; }
  std::vector<double> ones(n, 1.0);
  cudaMemcpyAsync(d_pm, ones.data(), sizeof(double) * n, cudaMemcpyHostToDevice, h->stream);
  rc = cvp_run(h, n, d_xyz, d_pm, p, vp_xyz, labels, vp_mass, res);
  cudaFree(d_xyz);
  cudaFree(d_pm);
  return rc;
}
