// engine.cuh — the relaxation step as CUDA kernels, templated on dimension D
// and arithmetic type R (double: FP64-plain, float: FP32-split).  Included by
// mrsph_fp64.cu (compiled without FMA contraction: FP64 follows the reference's
// operation order but for the Wendland gradient and the kernel sum, whose
// divisions share one reciprocal, kernel_dW and quot, within 1e-12 of the
// reference's value) and mrsph_fp32.cu.
//
// One step (SPH_mesh_generation::SPH_run_mesh_generation,
// sph_mesh_generation.cpp:1371-1463) is 11 launches on one stream (15 where the
// lists are made in brick order), replayed as a CUDA graph:
//   k_begin_step   scalars of the step
//   k_map          A1 advect + A2 sample + A3 surface map/re-seed + A4 spacing
//                  + scale/level refresh + cell key + cell histogram
//   scan, scatter  A5 counting sort into (level, cell) order
//   k_reorder      rank inside the cell, gather of the persistent state into the
//                  sorted order, search radii
//   k_brick_*      the work order of a large graded 3D handle's list builder
//   k_density_(group, lane, tile)  A6 neighbour search over the cell table: the neighbour lists
//   k_force<1>     A7 kernel sum + A8 stage 1 + A9 dt/max|v| grid reduction (FP64
//                  bit atomics), k_force_spill for particles whose list spilled
//   k_force<2>     A8 stage 2 + A9 + A10 (stage-1 kick folded in; the stage-2
//                  kick is folded into the next k_map)
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "engine_iface.h"

namespace mrsph {

using std::max;
using std::min;

// ---------------------------------------------------------------------------
// device data
// ---------------------------------------------------------------------------
template <class R>
struct Buf {  // persistent per-particle state, one ping-pong half
  typename V4<R>::T* posh;  // FP64: (x, y, z, h); FP32: (offset in anchor cell, h)
  typename V4<R>::T* nr;    // (nx, ny, nz, rho)
  typename V4<R>::T* v1;    // velocity after the stage-1 kick
  typename V4<R>::T* a2;    // stage-2 acceleration
  int* key;                 // FP32 anchor cell, packed (FP64: unused)
  int* meta;                // type | level << 8
  int* id;
  R* nu;                    // viscosity read by stage 2
  R* nu_next;               // viscosity written by stage 2
  R* phi;
  R* curv;
  int* cellkey;             // (level, cell) table index
  typename V4<R>::T* rec;   // packed neighbour-pass record, 2 words per particle
};

// Neighbour-list layout: blocks of 32 particles (one warp); inside a block,
// chunks of 8 consecutive entries (one 32-byte sector) per particle,
// interleaved over the 32 particles.  A particle's appends fill whole sectors
// in turn (as a row-major list would), and the lanes of a warp reading their
// q-th entries touch 8 lines instead of 32.  cap is a multiple of 8.
__host__ __device__ inline long long nb_slot(long long s, int q, int cap) {
  return (((((s >> 5) * (cap >> 3) + (q >> 3)) << 5) + (s & 31)) << 3) + (q & 7);
}

template <class R>
struct Work {  // per-step arrays in sorted order
  R* sum;
  typename V4<R>::T* a1;
  int* cnt;
  int* nbl;  // neighbour lists, entry q < cap of particle s at nbl[nb_slot(s, q, cap)]
  R* pc;     // stage-1 pair coefficients aw * (1/rho_i^2 + 1/rho_j^2), 0 for a skipped pair; nbl's layout
  int cap;
  int* counts;
  unsigned* lhmax;  // [level][level-0 cell]: largest h (FP32 bits, rounded up) this step, 0 if none
  int* bcount;      // particles per brick, then (bstart) their exclusive sums; the work order
  int* bstart;
  int* order;       // storage slots in work order: bricks, Z-order of half cells inside a brick
  float* rlev;      // [level][particle]: search radius on the level (level_radius), 0 if none
  int* cstart;
  int* perm;  // the counting sort's particles, cells in order, and their ids
  int* pid;
  int* blocksums;
  int* slot_of_id;
  int* spillq;  // particles whose list spilled (count sc->nspill)
};

// FP32-split decisions.  Three decisions of a step must come out as the
// reference's FP64 arithmetic on the world positions makes them: the cell of
// a particle (get_cell_id, glbfunc.h:196-208), the neighbour criterion
// r <= h cutoff + 1e-10 for h_i or h_j (level_infor.cpp:491-500) and the
// surface filter |n_i . n_j| > cos(angle_thres) (particle_mesh_generation.cpp:
// 719, 747, 937).  Each is made in FP32 with a band around its threshold that
// is wider than the FP32 error, and inside the band in FP64 with the
// reference's operation order on the world coordinates the position taps
// report.  Bands: the half-cell coordinate of the sort key, 2^-16 of a half
// cell; the squared distance, 2^-15 of the squared cut-off radius (the
// +1e-10 moves the radius by at most 2^-18.9 for radii of at least 1e-4,
// which mrsph_create enforces for FP32-split handles); the cosine, 2^-16.
constexpr float kBandKey = 1.0f / 65536.0f;
constexpr float kD2Accept = 1.0f + 1.0f / 32768.0f;  // FP32 d2 above R^2 * this: certainly not a neighbour
constexpr float kD2Sure = 1.0f - 1.0f / 32768.0f;    // FP32 d2 below R^2 * this: certainly a neighbour
constexpr float kBandCos = 1.0f / 65536.0f;

// Warp-aggregated append of val to queue q (counter *cnt); every lane of the
// warp calls it.
__device__ inline void queue_push(bool pred, unsigned* cnt, int* q, int val) {
  const unsigned m = __ballot_sync(0xffffffffu, pred);
  if (!m) return;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(cnt, (unsigned)__popc(m));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (pred) q[base + __popc(m & ((1u << lane) - 1u))] = val;
}

struct KCtx {
  Params prm;
  CellGeo geo;
  LsSet ls;
  long long n;
  DevScalars* sc;
};

// One FP32-split geometry of a batch as the batch kernels (mrsph_persist.cu)
// see it: the handle's context, both state buffers, its per-step arrays, the
// size of its cell table and the buffer that holds its state when the batch
// launch starts.
struct BatchSlot {
  KCtx c;
  Buf<float> buf[2];
  Work<float> w;
  long long ncells;
  int dim;
  int cur;
};

enum { MAP_STEP = 0, MAP_PRE = 1 };

// The forms of the neighbour passes.  All give the same lists and the same bits.
enum ListForm {
  LIST_GROUP,  // kG lanes per particle (list_group)
  LIST_LANE,   // one lane per particle (list_lanes), FP32-split
  LIST_TILE,   // a tile per warp, particles in storage order (list_warp), FP32-split in 3D
  LIST_BRICK   // the same in brick order
};
struct Forms {
  ListForm list = LIST_GROUP;
  bool force_group = true;  // kG lanes per particle in the force passes, else one
  bool operator==(const Forms& o) const { return list == o.list && force_group == o.force_group; }
};
// A group shortens the chain of gathers that bounds a pass while the chip is not
// full, at three times the instructions; so what counts is total, the particles of
// all handles that step at the same time (n: this handle's).  Force passes: stage
// 1 of 20,000 in 3D 37 us by groups, 67 by lanes, of 77,551 in 2D 39 and 26.
// In FP64 the line lies higher in 3D (seeded graded bodies, ms: 41,000 3.08 and 4.11,
// 160,000 8.91 and 10.20) and about there in 2D (50,000 0.299 and 0.315 in stage 1, 0.180
// and 0.138 in stage 2).
// Lists, by levels of the cell list and by row length (dense: more than kDenseRow
// neighbours on average, as uniformly seeded bodies have), us of 4 steps with
// upload and download, groups / lanes / tiles / tiles in brick order:
//   2D, one level    20,000 363/387, 30,000 449/444, 97,000 597/505
//   2D, graded       60,000 625/672, 85,000 -/681, 110,000 799/734
//   3D, one level    50,000 937/967/1018/1043, 60,000 992/974/1013/-,
//                    150,000 1641/1320/1506/1482, 1,000,000 -/6671/6683/6726
//   3D, graded       90,000 2389/2600/2594/2744, 111,500 2743/-/2600/2430,
//                    165,000 3598/2906/2704/3385, 200,000 4207/3034/3749/3202,
//                    600,000 10434/6802/5863/5622, 2,410,164 34445/-/18862/18848
//   3D, graded dense 30,000 3197/4831/3384/3594, 60,000 5212/6430/4971/5137,
//                    160,000 7953/7079/6084/7052, 301,270 13017/-/8262/8626
// Graded bodies want tiles because the candidates of coarse particles near fine
// ones are many; brick order saves a quarter of the instructions there but makes
// the longest warps longer, which shows until some 200,000 particles hide them.
// Many handles side by side (24 bodies of 2,000 to 60,000 particles on streams of
// their own, 4 steps): 1608 us in 2D and 3076 in 3D chosen by their total, 2515
// and 5156 each by its own number.
constexpr long long kGroupMax = 40960;
constexpr int kDenseRow = 160;
inline Forms choose_forms(int D, bool fp32, int ncl, bool dense, long long n, long long total) {
  Forms f;
  f.force_group = total <= kGroupMax;
  if (!fp32) return f;
  if (D == 2) {
    if (total > (ncl == 1 ? 24576 : 73728)) f.list = LIST_LANE;
  } else if (ncl == 1) {
    if (total > 57344) f.list = LIST_LANE;
  } else if (total > (dense ? 49152 : 98304)) {
    f.list = dense || n <= 196608 ? LIST_TILE : LIST_BRICK;
  }
  return f;
}

// Tuning of the FP32 map and neighbour passes: resident blocks per SM the
// register allocation must allow (density: of kDensityThreads threads, else 256).
#ifndef MRSPH_DENSITY_MIN_BLOCKS
#define MRSPH_DENSITY_MIN_BLOCKS 6
#endif
#ifndef MRSPH_FORCE_MIN_BLOCKS
#define MRSPH_FORCE_MIN_BLOCKS 5
#endif
#ifndef MRSPH_FORCE2_MIN_BLOCKS
#define MRSPH_FORCE2_MIN_BLOCKS 6
#endif
// the list builder's tile: candidates, and the spread in half cells within which
// a warp's lanes share it
#ifndef MRSPH_TILE_SIZE
#define MRSPH_TILE_SIZE 256
#endif
#ifndef MRSPH_TILE_SPAN_X
#define MRSPH_TILE_SPAN_X 15
#endif
#ifndef MRSPH_TILE_SPAN_YZ
#define MRSPH_TILE_SPAN_YZ 1
#endif
#ifndef MRSPH_MAP_MIN_BLOCKS
#define MRSPH_MAP_MIN_BLOCKS 4
#endif
// ---------------------------------------------------------------------------
// position representations
// ---------------------------------------------------------------------------
template <int D, class R> struct PosOps;

template <int D>
struct PosOps<D, double> {
  using T4 = double4;
  __device__ static void world(const KCtx&, const T4& p, int, double* x) { x[0] = p.x; x[1] = p.y; x[2] = (D == 3) ? p.z : 0.0; }
  __device__ static void set_world(const KCtx&, T4& p, int&, const double* x) { p.x = x[0]; p.y = x[1]; p.z = (D == 3) ? x[2] : 0.0; }
  // x = x + d  (the reference's coord + delta, component-wise)
  __device__ static void add(const KCtx&, T4& p, int&, const double* d) {
    p.x = p.x + d[0];
    p.y = p.y + d[1];
    if (D == 3) p.z = p.z + d[2];
  }
  // get_cell_id, glbfunc.h:196-208 (_NON_SYM_: [0, num_cell))
  __device__ static void cell(const KCtx& c, int L, const T4& p, int, int* cc) {
    double x[3] = {p.x, p.y, p.z};
    cc[2] = 0;
    for (int d = 0; d < D; d++) {
      int q = (int)floor((x[d] - c.geo.box_l[d]) / c.geo.dcell[L][d]);
      cc[d] = max(0, min(q, c.geo.n[L][d] - 1));
    }
  }
  // box-relative position (the operand of get_cell_id)
  __device__ static void xrel(const KCtx& c, const T4& p, int, double* xr) {
    xr[0] = p.x - c.geo.box_l[0];
    xr[1] = p.y - c.geo.box_l[1];
    xr[2] = (D == 3) ? p.z - c.geo.box_l[2] : 0.0;
  }
  __device__ static void rel(const KCtx&, const T4& pi, int, const T4& pj, int, double* dr) {
    dr[0] = pi.x - pj.x;
    dr[1] = pi.y - pj.y;
    dr[2] = (D == 3) ? pi.z - pj.z : 0.0;
  }
};

// FP32-split: position = anchor cell (finest cell-list cell) + FP32 offset.
template <int D>
struct PosOps<D, float> {
  using T4 = float4;
  __device__ static void unpack(int key, int* k) {
    unsigned u = (unsigned)key;
    if (D == 2) { k[0] = u & 0xFFFF; k[1] = (u >> 16) & 0xFFFF; k[2] = 0; }
    else { k[0] = u & 0x7FF; k[1] = (u >> 11) & 0x7FF; k[2] = (u >> 22) & 0x3FF; }
  }
  __device__ static int pack(const int* k) {
    if (D == 2) return (int)((unsigned)k[0] | ((unsigned)k[1] << 16));
    return (int)((unsigned)k[0] | ((unsigned)k[1] << 11) | ((unsigned)k[2] << 22));
  }
  // world coordinate box_l + (k A + o): one fused multiply-add and one add,
  // both explicit, so every kernel (and the position taps) gets the same bits
  __device__ static double world1(const KCtx& c, int d, int k, float o) {
    return __dadd_rn(c.geo.box_l[d], __fma_rn((double)k, c.geo.A[d], (double)o));
  }
  __device__ static void world(const KCtx& c, const T4& p, int key, double* x) {
    int k[3];
    unpack(key, k);
    float o[3] = {p.x, p.y, p.z};
    x[2] = 0.0;
    for (int d = 0; d < D; d++) x[d] = world1(c, d, k[d], o[d]);
  }
  __device__ static void set_world(const KCtx& c, T4& p, int& key, const double* x) {
    int k[3] = {0, 0, 0};
    float o[3] = {0.f, 0.f, 0.f};
    const int lm = c.geo.ncl - 1;
    for (int d = 0; d < D; d++) {
      double rel = x[d] - c.geo.box_l[d];
      int q = (int)floor(rel / c.geo.A[d]);
      q = max(0, min(q, c.geo.n[lm][d] - 1));
      k[d] = q;
      o[d] = (float)(rel - (double)q * c.geo.A[d]);
    }
    p.x = o[0]; p.y = o[1]; p.z = o[2];
    key = pack(k);
  }
  __device__ static void add(const KCtx& c, T4& p, int& key, const float* dlt) {
    int k[3];
    unpack(key, k);
    float o[3] = {p.x, p.y, p.z};
    const int lm = c.geo.ncl - 1;
    for (int d = 0; d < D; d++) {
      o[d] = o[d] + dlt[d];
      float q = floorf(o[d] / c.geo.Af[d]);
      if (q != 0.f) {
        int kn = max(0, min(k[d] + (int)q, c.geo.n[lm][d] - 1));
        o[d] -= (float)(kn - k[d]) * c.geo.Af[d];
        k[d] = kn;
      }
    }
    p.x = o[0]; p.y = o[1]; p.z = o[2];
    key = pack(k);
  }
  __device__ static void cell(const KCtx& c, int L, const T4&, int key, int* cc) {
    int k[3];
    unpack(key, k);
    int sh = c.geo.ncl - 1 - L;
    cc[2] = 0;
    for (int d = 0; d < D; d++) cc[d] = k[d] >> sh;
  }
  __device__ static void xrel(const KCtx& c, const T4& p, int key, double* xr) {
    int k[3];
    unpack(key, k);
    const float o[3] = {p.x, p.y, p.z};
    xr[2] = 0.0;
    for (int d = 0; d < D; d++) xr[d] = (double)k[d] * c.geo.A[d] + (double)o[d];
  }
  __device__ static void rel(const KCtx& c, const T4& pi, int ki, const T4& pj, int kj, float* dr) {
    int a[3], b[3];
    unpack(ki, a);
    unpack(kj, b);
    dr[0] = (float)(a[0] - b[0]) * c.geo.Af[0] + (pi.x - pj.x);
    dr[1] = (float)(a[1] - b[1]) * c.geo.Af[1] + (pi.y - pj.y);
    dr[2] = (D == 3) ? (float)(a[2] - b[2]) * c.geo.Af[2] + (pi.z - pj.z) : 0.f;
  }
};

// Packed record j (two 16-byte halves, 32-byte aligned; 64 bytes in FP64)
// read through the read-only path with 256-bit loads (sm_100 and later):
// one load instruction per FP32 record instead of two.
__device__ __forceinline__ void ld_rec(const float4* rec, long long j, float4& b0, float4& b1) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(b0.x), "=f"(b0.y), "=f"(b0.z), "=f"(b0.w), "=f"(b1.x), "=f"(b1.y), "=f"(b1.z), "=f"(b1.w)
      : "l"(rec + 2 * j));
}
__device__ __forceinline__ void ld_rec(const double4* rec, long long j, double4& b0, double4& b1) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(b0.x), "=d"(b0.y), "=d"(b0.z), "=d"(b0.w) : "l"(rec + 2 * j));
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(b1.x), "=d"(b1.y), "=d"(b1.z), "=d"(b1.w) : "l"(rec + 2 * j + 1));
}

// Load policies of the step's device functions.  LdNC: the read-only data
// path (ld.global.nc, __ldg) for the per-handle kernels, which never write
// what they read this way.  LdPlain: ordinary global loads for the persistent
// batch kernel, where a buffer read in one phase was written by other blocks
// in an earlier phase of the same launch (after a grid barrier whose fences
// make those writes visible).  The pointers reach the batch kernel through a
// shared-memory copy of the geometry's slot, never as const __restrict__
// kernel parameters, so these loads are not turned into read-only ones.
struct LdNC {
  __device__ static void rec(const float4* r, long long j, float4& b0, float4& b1) { ld_rec(r, j, b0, b1); }
  __device__ static void rec(const double4* r, long long j, double4& b0, double4& b1) { ld_rec(r, j, b0, b1); }
  template <class T> __device__ static T ld(const T* p) { return __ldg(p); }
};
struct LdPlain {
  __device__ static void rec(const float4* r, long long j, float4& b0, float4& b1) {
    b0 = r[2 * j];
    b1 = r[2 * j + 1];
  }
  __device__ static void rec(const double4* r, long long j, double4& b0, double4& b1) {
    b0 = r[2 * j];
    b1 = r[2 * j + 1];
  }
  template <class T> __device__ static T ld(const T* p) { return *p; }
};

template <class R> __device__ inline typename V4<R>::T mk4(R a, R b, R c, R d);
template <> __device__ inline double4 mk4<double>(double a, double b, double c, double d) { return make_double4(a, b, c, d); }
template <> __device__ inline float4 mk4<float>(float a, float b, float c, float d) { return make_float4(a, b, c, d); }

template <int D, class R>
__device__ inline R dot3(const R* a, const R* b) {
  R s = a[0] * b[0];
  s = madd(a[1], b[1], s);
  if (D == 3) s = madd(a[2], b[2], s);
  return s;
}

// Set_particle_info, particle_mesh_generation.cpp:361-381 (mass = 1)
template <int D, class R>
__device__ inline void set_info(const KCtx& c, R phi, R curv, R& h, R& rho) {
  R h_tmp = get_scale<R>(c.ls, phi, curv);
  h = h_tmp * pick<R>(c.prm.cell_ratio, c.prm.cell_ratio_f) / pick<R>(c.prm.cutoff, c.prm.cutoff_f);
  R vol;
  if constexpr (std::is_same<R, float>::value) vol = (D == 2) ? h_tmp * h_tmp : h_tmp * h_tmp * h_tmp;
  else vol = (D == 2) ? h_tmp * h_tmp : pow(h_tmp, 3.0);  // pow(h, DIM) as the reference
  rho = (R)1.0 / vol;
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__device__ inline void begin_step_body(DevScalars* sc, int inc) {
  sc->dt_adv = sc->dt2;
  sc->dt_adv_f = (float)bitsd(sc->dt2);
  sc->hdt_adv_f = (float)(0.5 * bitsd(sc->dt2));
  sc->dt1 = 0x7FF0000000000000ull;  // +inf
  sc->dt2 = 0x7FF0000000000000ull;
  sc->vmax1 = 0;
  sc->vmax2 = 0;
  sc->pairs = 0;
  sc->remap = 0;
  sc->nsurf = 0;
  sc->maxcnt = 0;
  sc->nspill = 0;
  for (int l = 0; l < MAX_CL; l++) {
    sc->hmax[l] = 0;
    sc->lcount[l] = 0;
  }
  sc->step += inc;
}
// scalars of the step, and the step's per-level h maxima (n words) cleared
static __global__ void k_begin_step(DevScalars* sc, int inc, unsigned* lhmax, long long n) {
  chain_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) begin_step_body(sc, inc);
  if (i < n) lhmax[i] = 0u;
}

// Random_particle_distribution, sph_mesh_generation.cpp:1302-1367 (one rank)
template <int D, class R>
__global__ void k_seed(KCtx c, Buf<R> b, unsigned max_att) {
  using P = PosOps<D, R>;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.n) return;
  const LsLevel& L0 = c.ls.lv[0];
  double padding = L0.dpkg[0];
  R phi = 0, n[3] = {0, 0, 0}, curv = 0, h = 0, rho = 0;
  double x[3] = {0, 0, 0};
  bool ok = false;
  for (unsigned att = 0; att < max_att && !ok; att++) {
    for (int d = 0; d < D; d++) {
      U4 r = philox((uint32_t)i, 0u, att, (RNG_SEED << 8) | d, c.prm.seed);
      double u1 = u53(r.v[0], r.v[1]), u2 = u53(r.v[2], r.v[3]);
      double box = c.prm.box_r[d] - c.prm.box_l[d];
      double lbl = L0.box_l[d], lbr = L0.box_l[d] + L0.dpkg[d] * L0.num_pkg[d];
      double xd = u1 * box + u2 * 1.e-3 + c.prm.box_l[d];
      xd = AMAX1(c.prm.box_l[d] + 1.e-10, AMIN1(xd, c.prm.box_r[d] - 1.e-10));
      xd = AMAX1(lbl + padding, AMIN1(lbr - padding, xd));
      x[d] = xd;
    }
    ls_sample<D, R>(c.ls, x, phi, n, curv);
    set_info<D, R>(c, phi, curv, h, rho);
    if (phi > h) ok = true;
  }
  if (!ok) atomicOr(&c.sc->flags, (unsigned)FLAG_SEED);
  typename V4<R>::T p = mk4<R>(0, 0, 0, h);
  int key = 0;
  P::set_world(c, p, key, x);
  b.posh[i] = p;
  if (b.key) b.key[i] = key;
  b.nr[i] = mk4<R>(n[0], n[1], n[2], rho);
  b.meta[i] = REAL_P;  // level 0: scale = max_scale (Particle_mesh_generation::Initialize)
  b.id[i] = (int)i;
  b.nu[i] = 0;
  b.nu_next[i] = 0;
  b.phi[i] = phi;
  b.curv[i] = curv;
  b.v1[i] = mk4<R>(0, 0, 0, 0);
  b.a2[i] = mk4<R>(0, 0, 0, 0);
}

// A1-A4 + scale refresh + cell key (see file header).  mode MAP_PRE is the
// map part of Pre_run (sph_mesh_generation.cpp:1010-1050): no advection,
// Set_particle_info before Find_and_map.
template <int D, class R>
__device__ inline void map_block(const KCtx& c, const Buf<R>& b, int* counts, unsigned* lhmax, int mode,
                                 unsigned max_att, long long blk) {
  using P = PosOps<D, R>;
  constexpr bool F32 = std::is_same<R, float>::value;
  __shared__ unsigned long long s_hmax[MAX_CL];
  __shared__ unsigned s_lcount[MAX_CL];
  if (threadIdx.x < MAX_CL) {
    s_hmax[threadIdx.x] = 0;
    s_lcount[threadIdx.x] = 0;
  }
  __syncthreads();
  long long i = blk * blockDim.x + threadIdx.x;
  unsigned surf = 0;
  if (i < c.n) {
    int meta = b.meta[i];
    int type = meta & 0xFF;
    int e = (int)(signed char)((meta >> 8) & 0xFF);
    typename V4<R>::T p = b.posh[i];
    int key = b.key ? b.key[i] : 0;
    const int id = b.id[i];
    R h = p.w;
    // A1 Update_coord_full_step (particle_mesh_generation.cpp:1139-1179), with
    // the stage-2 half kick of the previous step folded in (:1130-1135)
    if (mode == MAP_STEP && type != SINGULARITY_P) {
      typename V4<R>::T v1 = b.v1[i], a2 = b.a2[i];
      R hdt, dtr;
      if constexpr (F32) {
        hdt = c.sc->hdt_adv_f;
        dtr = c.sc->dt_adv_f;
      } else {
        const double dt2 = bitsd(c.sc->dt_adv);
        hdt = (R)(0.5 * dt2);
        dtr = (R)dt2;
      }
      R v[3] = {v1.x + a2.x * hdt, v1.y + a2.y * hdt, v1.z + a2.z * hdt};
      R dl[3] = {v[0] * dtr, v[1] * dtr, (D == 3) ? v[2] * dtr : (R)0};
      P::add(c, p, key, dl);
    }
    // A2 at the particle's position: from FP64 world coordinates (FP64-plain)
    // or in FP32 from the anchor representation (FP32-split)
    auto sample_here = [&](R& ph, R* nn, R& cv) {
      if constexpr (F32) {
        int k[3];
        P::unpack(key, k);
        const float o[3] = {p.x, p.y, p.z};
        ls_sample_anchor<D>(c.ls, k, o, ph, nn, cv);
      } else {
        double xw[3];
        P::world(c, p, key, xw);
        ls_sample<D, R>(c.ls, xw, ph, nn, cv);
      }
    };
    auto tag_here = [&](int* chr) -> int {
      if constexpr (F32) {
        // the cell in FP32 unless a cell face lies within the band, then
        // the reference's FP64 lookup of the world position
        int k[3];
        P::unpack(key, k);
        const float o[3] = {p.x, p.y, p.z};
        bool near = false;
        const int t = ls_tag_anchor<D>(c.ls, k, o, chr, &near);
        if (!near) return t;
        double xw[3];
        P::world(c, p, key, xw);
        return ls_tag<D, double>(c.ls, xw, chr);
      } else {
        double xw[3];
        P::world(c, p, key, xw);
        return ls_tag<D, R>(c.ls, xw, chr);
      }
    };
    R phi, n[3], curv, rho = 0;
    sample_here(phi, n, curv);  // A2 Get_particle_info
    if (mode == MAP_PRE) set_info<D, R>(c, phi, curv, h, rho);
    // A3 Find_and_map_particle (:408-467) + driver loop (sph_mesh_generation.cpp:1506-1545)
    int chr = 0;  // characteristic cell: k + 1 on segment k, -(k + 1) at singularity k
    int tag = tag_here(&chr);
    R nl = r_sqrt(dot3<D, R>(n, n));
    if (tag == CUT_CELL && (type == REAL_P || type == SURFACE_P) && chr == 0) {
      type = SURFACE_P;
      R dist = r_fabs(phi);
      R div = (R)1.0 / (nl + (R)1.0e-15);
      R dl[3] = {0, 0, 0};
      for (int d = 0; d < D; d++) {
        R nn = n[d] * div;
        R nd = phi < (R)0 ? nn : -nn;
        dl[d] = nd * dist;
      }
      P::add(c, p, key, dl);
    } else if (chr > 0) {
      // SEGMENT: onto the segment's line (:439-455), in FP64 on the world
      // position: e = (p2 - p1) / max(|p2 - p1|, 1e-15), x = p1 + e ((x - p1) . e)
      type = SEGMENT_P;
      const double* p1 = c.ls.seg + 6 * (chr - 1);
      const double* p2 = p1 + 3;
      double xw[3];
      P::world(c, p, key, xw);
      double Pv[3] = {0.0, 0.0, 0.0}, Nv[3] = {0.0, 0.0, 0.0};
      for (int d = 0; d < D; d++) {
        Pv[d] = __dsub_rn(p2[d], p1[d]);
        Nv[d] = __dsub_rn(xw[d], p1[d]);
      }
      double len = __dmul_rn(Pv[0], Pv[0]);
      len = __dadd_rn(len, __dmul_rn(Pv[1], Pv[1]));
      if (D == 3) len = __dadd_rn(len, __dmul_rn(Pv[2], Pv[2]));
      const double inv = __ddiv_rn(1.0, fmax(__dsqrt_rn(len), 1.e-15));
      double e[3] = {0.0, 0.0, 0.0};
      for (int d = 0; d < D; d++) e[d] = __dmul_rn(Pv[d], inv);
      double dist = __dmul_rn(Nv[0], e[0]);
      dist = __dadd_rn(dist, __dmul_rn(Nv[1], e[1]));
      if (D == 3) dist = __dadd_rn(dist, __dmul_rn(Nv[2], e[2]));
      for (int d = 0; d < D; d++) xw[d] = __dadd_rn(p1[d], __dmul_rn(e[d], dist));
      P::set_world(c, p, key, xw);
    } else if (chr < 0) {
      // SINGULARITY: at the point (:456-465)
      type = SINGULARITY_P;
      const double* ps = c.ls.sing + 3 * (-chr - 1);
      double xw[3] = {ps[0], ps[1], D == 3 ? ps[2] : 0.0};
      P::set_world(c, p, key, xw);
    } else {
      type = REAL_P;
    }
    if (type == SURFACE_P || type == SEGMENT_P) {  // Get_dispersed_position(0.00001*h), :385-404
      R dx = (R)0.00001 * h;
      R div = (R)1.0 / (nl + (R)1.0e-15);
      R dl[3] = {0, 0, 0};
      for (int d = 0; d < D; d++) {
        R nn = n[d] * div;
        R nd = phi < (R)0 ? nn : -nn;
        dl[d] = nd * dx;
      }
      P::add(c, p, key, dl);
    }
    sample_here(phi, n, curv);
    if (phi < (R)0 && type == REAL_P) {
      double x[3];
      // Remap_this_particle_to_positive_phase, sph_mesh_generation.cpp:1885-1928
      atomicAdd(&c.sc->remap, 1u);
      bool ok = false;
      for (unsigned att = 0; att < max_att && !ok; att++) {
        for (int d = 0; d < D; d++) {
          U4 r = philox((uint32_t)id, c.sc->step, att, (RNG_REMAP << 8) | d, c.prm.seed);
          double u1 = u53(r.v[0], r.v[1]), u2 = u53(r.v[2], r.v[3]);
          double bl = c.prm.box_l[d], br = c.prm.box_r[d], box = br - bl;
          double xd = u1 * box + u2 * 1.e-3 + bl;
          x[d] = AMAX1(bl + 1.e-10, AMIN1(xd, br - 1.e-10));
        }
        ls_sample<D, R>(c.ls, x, phi, n, curv);
        if (phi > h) ok = true;
      }
      if (!ok) atomicOr(&c.sc->flags, (unsigned)FLAG_REMAP);
      P::set_world(c, p, key, x);
      type = REAL_P;
      set_info<D, R>(c, phi, curv, h, rho);
    }
    // A4 Set_particle_scale (:361-381)
    if (mode == MAP_STEP) set_info<D, R>(c, phi, curv, h, rho);
    // Particle_base::Set_particle_scale, particle.cpp:957-975 (scale = max_scale*2^-e)
    {
      R sc = F32 ? (R)ldexpf(c.geo.max_scale_f, -e) : (R)ldexp(c.geo.max_scale, -e);
      R hc = h * pick<R>(c.prm.cutoff, c.prm.cutoff_f);
      for (int it = 0; it < 64; it++) {
        if (hc > sc + (R)1.e-15) { sc *= 2; e--; }
        else if (hc < sc / 2 - (R)1.e-15) { sc /= 2; e++; }
        else break;
      }
    }
    int L = e;
    if (L < 0 || L >= c.geo.ncl) {
      atomicOr(&c.sc->flags, (unsigned)FLAG_LEVEL);
      L = max(0, min(L, c.geo.ncl - 1));
      e = L;
    }
    // sort key: level-L half cell (get_cell_id, glbfunc.h:196-208, at dcell/2)
    int hq[3] = {0, 0, 0};
    long long c0 = 0;  // level-0 cell, for the local h maximum of level L
    if constexpr (F32) {
      // a level-L cell is 2^sh anchor cells: the half cell follows from the
      // anchor index and the FP32 position inside the level-L cell
      int k[3];
      P::unpack(key, k);
      const float o[3] = {p.x, p.y, p.z};
      const int sh = c.geo.ncl - 1 - L;
      bool near_edge = false;
      for (int d = 0; d < D; d++) {
        const int cc = k[d] >> sh;
        const float pos = fmaf((float)(k[d] - (cc << sh)), c.geo.Af[d], o[d]);
        const float u = pos * c.geo.ihs_f[L][d];
        const float fl = floorf(u);
        const float fr = u - fl;
        near_edge = near_edge || fr < kBandKey || fr > 1.f - kBandKey;
        hq[d] = max(0, min(2 * cc + (int)fl, c.geo.hn[L][d] - 1));
      }
      if (near_edge) {
        // within the band of a half-cell face: the reference's FP64 binning,
        // floor((x - box_l) / dcell), of the world position.  Half cells are
        // dcell / 2 exactly, so floor((x - box_l) / (dcell / 2)) >> 1 is that
        // cell.
        for (int d = 0; d < D; d++) {
          const double rel = __dsub_rn(P::world1(c, d, k[d], o[d]), c.geo.box_l[d]);
          const double u = floor(__ddiv_rn(rel, c.geo.hs[L][d]));
          hq[d] = (int)fmax(0.0, fmin(u, (double)(c.geo.hn[L][d] - 1)));
        }
      }
      for (int d = D - 1; d >= 0; d--) c0 = c0 * c.geo.n[0][d] + (k[d] >> (c.geo.ncl - 1));
    } else {
      double xr[3];
      P::xrel(c, p, key, xr);
      for (int d = 0; d < D; d++) {
        double u = floor(xr[d] / c.geo.hs[L][d]);
        u = fmax(0.0, fmin(u, (double)(c.geo.hn[L][d] - 1)));
        hq[d] = (int)u;
      }
      for (int d = D - 1; d >= 0; d--) {
        int q0 = (int)fmax(0.0, fmin(floor(xr[d] * c.geo.idc0[d]), (double)(c.geo.n[0][d] - 1)));
        c0 = c0 * c.geo.n[0][d] + q0;
      }
    }
    int ck = (int)(c.geo.hoff[L] + ((long long)hq[2] * c.geo.hn[L][1] + hq[1]) * c.geo.hn[L][0] + hq[0]);
    atomicAdd(&counts[ck], 1);
    atomicMax(&lhmax[L * c.geo.nc0 + c0], __float_as_uint(F32 ? (float)h : __double2float_ru((double)h)));
    atomicMax(&s_hmax[L], dbits((double)h));
    atomicAdd(&s_lcount[L], 1u);
    p.w = h;
    b.posh[i] = p;
    if (b.key) b.key[i] = key;
    b.nr[i] = mk4<R>(n[0], n[1], n[2], rho);
    b.meta[i] = type | ((e & 0xFF) << 8);
    b.phi[i] = phi;
    b.curv[i] = curv;
    b.cellkey[i] = ck;
    surf = (type == SURFACE_P) ? 1u : 0u;
  }
  unsigned ws = __popc(__ballot_sync(0xffffffffu, surf != 0));
  if ((threadIdx.x & 31) == 0 && ws) atomicAdd(&c.sc->nsurf, ws);
  __syncthreads();
  if (threadIdx.x < MAX_CL && s_lcount[threadIdx.x]) {
    atomicMax(&c.sc->hmax[threadIdx.x], s_hmax[threadIdx.x]);
    atomicAdd(&c.sc->lcount[threadIdx.x], s_lcount[threadIdx.x]);
  }
}

template <int D, class R>
__global__ void __launch_bounds__(256, (std::is_same<R, float>::value ? MRSPH_MAP_MIN_BLOCKS : 1))
k_map(KCtx c, Buf<R> b, int* counts, unsigned* lhmax, int mode, unsigned max_att) {
  chain_wait();
  map_block<D, R>(c, b, counts, lhmax, mode, max_att, blockIdx.x);
}

// Packed record read by the neighbour passes, two V4 words per particle so
// that one candidate costs one 32-byte sector (FP32):
//   FP32: w0 = (offset x, y, z, h), w1 = (anchor x, y, z as exact floats, +-1/rho^2)
//   FP64: w0 = (x, y, z, h),        w1 = (box-relative x, y, z, h as four
//         floats in the first 16 bytes, 0, +-1/rho^2)
// The sign carries the type: negative for a particle that is not REAL.  1/rho^2 is the
// neighbour's share of the pair coefficient of the force stages, computed once
// per particle (as 1 / (rho * rho), the forces' own expression).
template <int D, class R> struct RecOps;
template <int D>
struct RecOps<D, double> {
  __device__ static void pack(const KCtx& c, const double4& p, int, int type, double rho, double4& w0, double4& w1) {
    w0 = p;
    const double vol = r_rcp(rho * rho);
    const float x = (float)(p.x - c.geo.box_l[0]), y = (float)(p.y - c.geo.box_l[1]);
    const float z = D == 3 ? (float)(p.z - c.geo.box_l[2]) : 0.f, h = (float)p.w;
    w1 = make_double4(__hiloint2double(__float_as_int(y), __float_as_int(x)),
                      __hiloint2double(__float_as_int(h), __float_as_int(z)), 0.0, type != REAL_P ? -vol : vol);
  }
  // box-relative position and h in FP32 (the first 16 bytes of w1)
  __device__ static float4 filter(const double4& w1) {
    return make_float4(__int_as_float(__double2loint(w1.x)), __int_as_float(__double2hiint(w1.x)),
                       __int_as_float(__double2loint(w1.y)), __int_as_float(__double2hiint(w1.y)));
  }
  template <class LD>
  __device__ static float4 load_filter(const double4* rec, long long j) {
    return LD::ld(reinterpret_cast<const float4*>(rec + 2 * j + 1));
  }
  __device__ static void rel(const KCtx&, const double4& a0, const double4&, const double4& b0, const double4&,
                             double* dr) {
    dr[0] = a0.x - b0.x;
    dr[1] = a0.y - b0.y;
    dr[2] = (D == 3) ? a0.z - b0.z : 0.0;
  }
};
template <int D>
struct RecOps<D, float> {
  __device__ static void pack(const KCtx&, const float4& p, int key, int type, float rho, float4& w0, float4& w1) {
    int k[3];
    PosOps<D, float>::unpack(key, k);
    w0 = p;
    const float vol = r_rcp(rho * rho);
    w1 = make_float4((float)k[0], (float)k[1], (float)k[2], type != REAL_P ? -vol : vol);
  }
  __device__ static void rel(const KCtx& c, const float4& a0, const float4& a1, const float4& b0, const float4& b1,
                             float* dr) {
    dr[0] = fmaf(a1.x - b1.x, c.geo.Af[0], a0.x - b0.x);
    dr[1] = fmaf(a1.y - b1.y, c.geo.Af[1], a0.y - b0.y);
    dr[2] = (D == 3) ? fmaf(a1.z - b1.z, c.geo.Af[2], a0.z - b0.z) : 0.f;
  }
};

// The reference's neighbour criterion in FP64 for two FP32-split records
// (w0 = offset, h; w1 = anchor index): world coordinates as the position taps
// compute them, dr = x_i - x_j, dist = sqrt(dr.dr) summed in axis order, and
// dist <= h cutoff + 1e-10 for h_i or h_j (level_infor.cpp:491-500).
template <int D>
__device__ __noinline__ bool exact_neighbor(const KCtx& c, const float4& a0, const float4& a1, const float4& b0,
                                            const float4& b1) {
  const float ao[3] = {a0.x, a0.y, a0.z}, bo[3] = {b0.x, b0.y, b0.z};
  const float ak[3] = {a1.x, a1.y, a1.z}, bk[3] = {b1.x, b1.y, b1.z};
  double d2 = 0.0;
  for (int d = 0; d < D; d++) {
    const double xi = PosOps<D, float>::world1(c, d, (int)ak[d], ao[d]);
    const double xj = PosOps<D, float>::world1(c, d, (int)bk[d], bo[d]);
    const double dr = __dsub_rn(xi, xj);
    d2 = (d == 0) ? __dmul_rn(dr, dr) : __dadd_rn(d2, __dmul_rn(dr, dr));
  }
  const double dist = __dsqrt_rn(d2);
  const double ri = __dadd_rn(__dmul_rn((double)a0.w, c.prm.cutoff), 1.e-10);
  const double rj = __dadd_rn(__dmul_rn((double)b0.w, c.prm.cutoff), 1.e-10);
  return (dist <= ri) || (dist <= rj);
}

// The surface filter |n_i . n_j| > cos(angle_thres) in FP64, products summed
// in axis order (particle_mesh_generation.cpp:719, 747, 937).
template <int D>
__device__ __noinline__ bool exact_cos(const KCtx& c, const float* ni, const float* nj) {
  double ca = __dmul_rn((double)ni[0], (double)nj[0]);
  ca = __dadd_rn(ca, __dmul_rn((double)ni[1], (double)nj[1]));
  if (D == 3) ca = __dadd_rn(ca, __dmul_rn((double)ni[2], (double)nj[2]));
  return fabs(ca) > c.prm.cos_thres;
}

// ---------------------------------------------------------------- work order
// Storage is by rows of half cells, so the 32 particles of a warp lie along a
// row, and where rows are short (a shell of one level, the end of a body) in
// several of them: 2.2 segments per level on a relaxed torus.  The list builder
// of a large graded handle therefore takes its particles in another order, by bricks
// of 4 half cells per axis and by Z-order of the half cells inside a brick; what
// is computed for a particle does not depend on it.
__device__ inline void brick_of(const CellGeo& g, long long t, int& L, int* q) {
  L = 0;
  while (L + 1 < g.ncl && t >= g.boff[L + 1]) L++;
  long long r = t - g.boff[L];
  q[0] = (int)(r % g.bn[L][0]);
  r /= g.bn[L][0];
  q[1] = (int)(r % g.bn[L][1]);
  q[2] = (int)(r / g.bn[L][1]);
}
// one thread per brick: its particles, from the start table (D = 3)
template <int D>
__global__ void __launch_bounds__(256) k_brick_count(KCtx c, const int* __restrict__ cstart, int* __restrict__ bcount) {
  chain_wait();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= c.geo.boff[c.geo.ncl]) return;
  int L, q[3], n = 0;
  brick_of(c.geo, t, L, q);
  if (c.sc->lcount[L]) {
    const int* hn = c.geo.hn[L];
    const int x0 = 4 * q[0], x1 = min(x0 + 4, hn[0]);
    for (int z = 4 * q[2]; z < min(4 * q[2] + 4, hn[2]); z++)
      for (int y = 4 * q[1]; y < min(4 * q[1] + 4, hn[1]); y++) {
        const long long rb = c.geo.hoff[L] + ((long long)z * hn[1] + y) * hn[0];
        n += cstart[rb + x1] - cstart[rb + x0];
      }
  }
  bcount[t] = n;
}
// A warp takes per (1 to 32) bricks one after the other, those with particles:
// their half cells' particles in Z-order.  A brick is a chain of some 1.4 us, so
// few bricks are spread over many warps: 32 to a warp take 47 us for the 27,000
// of a one-level body of 150,000 particles, one or two to a warp 10 us for those of
// a graded one of 200,000.
template <int D>
__global__ void __launch_bounds__(256) k_brick_order(KCtx c, const int* __restrict__ cstart,
                                                     const int* __restrict__ bcount, const int* __restrict__ bstart,
                                                     int* __restrict__ order, int per) {
  chain_wait();
  const int lane = threadIdx.x & 31;
  const long long base = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per, nb = c.geo.boff[c.geo.ncl];
  const long long mine = base + lane;
  unsigned todo = __ballot_sync(0xffffffffu, lane < per && mine < nb && bcount[mine] > 0);
  while (todo) {
    const long long t = base + __ffs(todo) - 1;
    todo &= todo - 1u;
    int L, q[3];
    brick_of(c.geo, t, L, q);
    const int* hn = c.geo.hn[L];
    int at = bstart[t];
#pragma unroll
    for (int z0 = 0; z0 < 64; z0 += 32) {
      const int zc = z0 + lane;  // Z-order index of the half cell
      int h[3];
      bool ok = true;
      for (int d = 0; d < 3; d++) {
        h[d] = 4 * q[d] + (((zc >> d) & 1) | (((zc >> (3 + d)) & 1) << 1));
        ok = ok && h[d] < hn[d];
      }
      int s0 = 0, s1 = 0;
      if (ok) {
        const long long cell = c.geo.hoff[L] + ((long long)h[2] * hn[1] + h[1]) * hn[0] + h[0];
        s0 = cstart[cell];
        s1 = cstart[cell + 1];
      }
      int inc = s1 - s0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      int o = at + inc - (s1 - s0);
      for (int u = s0; u < s1; u++) order[o++] = u;
      at += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

// Largest h of level-L particles (lhmax entries) over the level-0 cells
// lo..hi (0: none).
template <class LD = LdNC>
__device__ inline float lhmax_over(const KCtx& c, const unsigned* __restrict__ lhmax, int L, const int* lo,
                                   const int* hi) {
  const unsigned* o = lhmax + (long long)L * c.geo.nc0;
  unsigned m = 0;
  for (int z = lo[2]; z <= hi[2]; z++)
    for (int y = lo[1]; y <= hi[1]; y++)
      for (int x = lo[0]; x <= hi[0]; x++)
        m = max(m, LD::ld(&o[((long long)z * c.geo.n[0][1] + y) * c.geo.n[0][0] + x]));
  return __uint_as_float(m);
}

// Search origin of a particle: its box-relative FP64 position (FP64-plain) or
// its anchor cell and FP32 offset (FP32-split).
template <int D, class R> struct SOrigin;
template <int D> struct SOrigin<D, double> {
  double xr[3];
  __device__ SOrigin(const KCtx& c, const double4& p, int key) { PosOps<D, double>::xrel(c, p, key, xr); }
};
template <int D> struct SOrigin<D, float> {
  int k[3];
  float o[3];
  __device__ SOrigin(const KCtx&, const float4& p, int key) {
    PosOps<D, float>::unpack(key, k);
    o[0] = p.x; o[1] = p.y; o[2] = p.z;
  }
};

// Level L of the candidate search from origin so with smoothing length hi.
// level_radius: R_L = cutoff * max(hi, local h maximum of level L) + 1e-10 with
// a relative pad (1e-5 FP64, 3e-5 FP32-split; 0 when no level-L particle can
// pair with the origin).  The local h maximum is the largest lhmax entry over
// the level-0 cells overlapping the cube of the level-wide bound (every level-L
// particle that can pair with the origin lies in one of them).  level_position:
// the origin's half-cell coordinate q + fr on level L.
// FP64-plain keeps the box-relative FP64 arithmetic; FP32-split works in FP32
// relative to the anchor: a level-L cell is 2^(finest - L) anchor cells, so the
// position inside the origin's level-L (or level-0) cell is (anchor index -
// cell's first anchor) * A + offset.
template <int D, class LD = LdNC>
__device__ inline float level_radius(const KCtx& c, const unsigned* __restrict__ lhmax, int L,
                                     const SOrigin<D, double>& so, double hi) {
  const double hic = hi * c.prm.cutoff;
  const double Rg = (fmax(hic, bitsd(c.sc->hmax[L]) * c.prm.cutoff) + 1.e-10) * (1.0 + 1.e-5);
  int lo[3] = {0, 0, 0}, up[3] = {0, 0, 0};
  for (int d = 0; d < D; d++) {
    const double top = (double)(c.geo.n[0][d] - 1);
    lo[d] = (int)fmax(0.0, fmin(floor((so.xr[d] - Rg) * c.geo.idc0[d]), top));
    up[d] = (int)fmax(0.0, fmin(floor((so.xr[d] + Rg) * c.geo.idc0[d]), top));
  }
  const float hloc = lhmax_over<LD>(c, lhmax, L, lo, up);
  if (!(hloc > 0.f)) return 0.f;
  const double Rw = fmax(hic, (double)hloc * c.prm.cutoff) + 1.e-10;
  return (float)(Rw * (1.0 + 1.e-5));
}
template <int D>
__device__ inline void level_position(const KCtx& c, int L, const SOrigin<D, double>& so, int* q, float* fr) {
  for (int d = 0; d < D; d++) {
    double u = so.xr[d] / c.geo.hs[L][d];
    u = fmax(-1.0e6, fmin(u, 1.0e9));
    const double fl = floor(u);
    q[d] = (int)fl;
    fr[d] = (float)(u - fl);
  }
}
template <int D, class LD = LdNC>
__device__ inline float level_radius(const KCtx& c, const unsigned* __restrict__ lhmax, int L,
                                     const SOrigin<D, float>& so, float hi) {
  const float cut = c.prm.cutoff_f;
  const float hic = hi * cut;
  const float Rg = (fmaxf(hic, (float)bitsd(c.sc->hmax[L]) * cut) + 1.e-10f) * (1.f + 3.e-5f);
  const int sh0 = c.geo.ncl - 1;
  int lo[3] = {0, 0, 0}, up[3] = {0, 0, 0};
  for (int d = 0; d < D; d++) {
    const int c0 = so.k[d] >> sh0;
    const float u0 = fmaf((float)(so.k[d] - (c0 << sh0)), c.geo.Af[d], so.o[d]) * c.geo.idc0_f[d];
    const float r0 = Rg * c.geo.idc0_f[d];
    const int top = c.geo.n[0][d] - 1;
    lo[d] = max(0, min(c0 + (int)floorf(fmaxf(u0 - r0, -1.0e6f)), top));
    up[d] = max(0, min(c0 + (int)floorf(fminf(u0 + r0, 1.0e6f)), top));
  }
  const float hloc = lhmax_over<LD>(c, lhmax, L, lo, up);
  if (!(hloc > 0.f)) return 0.f;
  return (fmaxf(hic, hloc * cut) + 1.e-10f) * (1.f + 3.e-5f);
}
template <int D>
__device__ inline void level_position(const KCtx& c, int L, const SOrigin<D, float>& so, int* q, float* fr) {
  const int sh = c.geo.ncl - 1 - L;
  for (int d = 0; d < D; d++) {
    const int cc = so.k[d] >> sh;
    float u = fmaf((float)(so.k[d] - (cc << sh)), c.geo.Af[d], so.o[d]) * c.geo.ihs_f[L][d];
    u = fmaxf(-1.0e6f, fminf(u, 1.0e6f));
    const float fl = floorf(u);
    q[d] = 2 * cc + (int)fl;
    fr[d] = u - fl;
  }
}
// the half cells the sphere of radius R around q + fr reaches, per axis
template <int D>
__device__ inline void level_box(const KCtx& c, int L, float R, const int* q, const float* fr, int* lo, int* up) {
  for (int d = 0; d < D; d++) {
    const float rr = R * c.geo.ihs_f[L][d];
    lo[d] = max(q[d] + (int)floorf(fr[d] - rr), 0);
    up[d] = min(q[d] + (int)floorf(fr[d] + rr), c.geo.hn[L][d] - 1);
  }
}
// Particles [s0, e0) of row (z, y) of level L inside the sphere; false when the
// row lies outside.
template <int D, class LD = LdNC>
__device__ inline bool row_range(const KCtx& c, const int* __restrict__ cstart, int L, float R, const int* q,
                                 const float* fr, int z, int y, int& s0, int& e0) {
  const int* hn = c.geo.hn[L];
  float gz = 0.f;
  if (D == 3) {
    const int m = z - q[2];
    if (z > 0) gz = fmaxf(gz, (float)m - fr[2]);
    if (z < hn[2] - 1) gz = fmaxf(gz, fr[2] - (float)(m + 1));
    gz *= c.geo.hs_f[L][2];
  }
  const int m = y - q[1];
  float gy = 0.f;
  if (y > 0) gy = fmaxf(gy, (float)m - fr[1]);
  if (y < hn[1] - 1) gy = fmaxf(gy, fr[1] - (float)(m + 1));
  gy *= c.geo.hs_f[L][1];
  const float rem = R * R - gy * gy - gz * gz;
  if (rem < 0.f) return false;
  const float w = sqrtf(rem) * c.geo.ihs_f[L][0];
  const int xl = max(q[0] + (int)floorf(fr[0] - w), 0);
  const int xh = min(q[0] + (int)floorf(fr[0] + w), hn[0] - 1);
  if (xl > xh) return false;
  const long long rb = c.geo.hoff[L] + ((long long)z * hn[1] + y) * hn[0];
  s0 = LD::ld(&cstart[rb + xl]);
  e0 = LD::ld(&cstart[rb + xh + 1]);
  return true;
}

// The last step of the counting sort, the gather into storage order and the
// per-level search radii, one thread per entry of perm: perm holds each cell's
// particles in arbitrary order, the canonical order inside a cell is ascending
// id, so the thread counts the lower ids of its cell and writes its particle
// there.  (A separate ranking pass wrote and read back the permutation: 25 us
// and a launch for 2.4 M particles.)
template <int D, class R, class LD = LdNC>
__device__ inline void reorder_block(const Buf<R>& src, const Buf<R>& dst, const KCtx& c, const Work<R>& w,
                                     int partial, long long blk) {
  const long long t = blk * blockDim.x + threadIdx.x;
  const long long n = c.n;
  if (t >= n) return;
  const int o = w.perm[t];
  const int ck = src.cellkey[o], id = w.pid[t];
  const int c0 = LD::ld(&w.cstart[ck]), c1 = LD::ld(&w.cstart[ck + 1]);
  long long s = c0;
  for (int u = c0; u < c1; u++) s += w.pid[u] < id ? 1 : 0;
  const auto p = src.posh[o];
  const int key = src.key ? src.key[o] : 0;
  const auto nr = src.nr[o];
  const int meta = src.meta[o];
  dst.posh[s] = p;
  if (src.key) dst.key[s] = key;
  dst.nr[s] = nr;
  dst.meta[s] = meta;
  typename V4<R>::T w0, w1;
  RecOps<D, R>::pack(c, p, key, meta & 0xFF, nr.w, w0, w1);
  dst.rec[2 * s] = w0;
  dst.rec[2 * s + 1] = w1;
  dst.id[s] = id;
  dst.nu[s] = src.nu_next[o];
  dst.phi[s] = src.phi[o];
  dst.curv[s] = src.curv[o];
  dst.cellkey[s] = ck;
  if (partial) {  // a step that stops before stage 2 keeps these consistent
    dst.nu_next[s] = src.nu_next[o];
    dst.v1[s] = src.v1[o];
    dst.a2[s] = src.a2[o];
  }
  w.slot_of_id[id] = (int)s;
  const SOrigin<D, R> so(c, p, key);
  for (int L = 0; L < c.geo.ncl; L++)
    w.rlev[(long long)L * n + s] = c.sc->lcount[L] ? level_radius<D, LD>(c, w.lhmax, L, so, p.w) : 0.f;
}

template <int D, class R>
__global__ void k_reorder(Buf<R> src, Buf<R> dst, KCtx c, Work<R> w, int partial) {
  chain_wait();
  reorder_block<D, R>(src, dst, c, w, partial, blockIdx.x);
}

// Candidates of particle i over all cell-list levels.  The reference walks
// the 3^D cells of i's level, whose lists hold the particles of that level and
// of every finer one, and links i and j when r <= 2 h_i or r <= 2 h_j
// (level_infor.cpp:407-506).  The same relation is found here per level L
// among the level-L particles within R_L = cutoff * max(h_i, hmax_L) + 1e-10
// of x_i, hmax_L being the largest h on level L this step: only the half cells
// of the sort table that the sphere of radius R_L reaches are read.  Each
// (z, y) row of half cells is one contiguous range of the sorted arrays; rows
// farther than R_L are skipped and the x range of each row is cut to the
// sphere.  Edge rows extend to infinity (keys are clamped into the table).
// R_L carries a relative pad for the rounding of the keys and of the row
// arithmetic (FP64: 1e-5; FP32-split: 3e-5, which also covers the FP32
// test's acceptance band of 2^-15 on R^2, so the per-lane and the warp-tile
// scans accept the same candidates); the candidate test decides membership.
// The candidates by a group of kG lanes per particle.  The lanes take the rows of the particle's spheres
// kG at a time, one row range each; the ranges of up to kRowTile non-empty rows
// stand in shared memory as one run of candidates, which the lanes then walk
// kG at a time: visit(j, in) is called by the whole group, in = false past the
// end.  The search radii come from w.rlev (one thread per particle and level
// filled them in the reorder pass).
constexpr int kG = 8;
constexpr int kRowTile = 48;
struct RowTile {
  int off[kRowTile];  // first particle of the row - its place in the run
  int end[kRowTile];  // end of the row in the run
};
struct GroupLanes {
  unsigned mask, below;
  int gl, shift;
  __device__ GroupLanes() {
    const int lane = threadIdx.x & 31;
    gl = lane & (kG - 1);
    shift = lane - gl;
    mask = ((1u << kG) - 1u) << shift;
    below = (1u << gl) - 1u;
  }
  __device__ unsigned ballot(bool p) const { return (__ballot_sync(mask, p) >> shift) & ((1u << kG) - 1u); }
};
template <int D, class R, class LD, class F>
__device__ inline void group_scan(const KCtx& c, const Work<R>& w, const GroupLanes& g, RowTile& rt, long long i,
                                  const SOrigin<D, R>& so, F&& visit) {
  int nrow = 0, T = 0;
  auto flush = [&]() {
    __syncwarp(g.mask);
    int r = 0;
    for (int t0 = 0; t0 < T; t0 += kG) {
      const int t = t0 + g.gl;
      const bool in = t < T;
      int j = 0;
      if (in) {
        while (t >= rt.end[r]) r++;
        j = rt.off[r] + t;
      }
      visit(j, in);
    }
    __syncwarp(g.mask);
    nrow = 0;
    T = 0;
  };
  for (int L = 0; L < c.geo.ncl; L++) {
    const float R_ = LD::ld(&w.rlev[(long long)L * c.n + i]);
    if (!(R_ > 0.f)) continue;  // group-uniform
    int q[3] = {0, 0, 0}, lo[3] = {0, 0, 0}, up[3] = {0, 0, 0};
    float fr[3] = {0.f, 0.f, 0.f};
    level_position<D>(c, L, so, q, fr);
    level_box<D>(c, L, R_, q, fr, lo, up);
    const int ny = up[1] - lo[1] + 1, nz = up[2] - lo[2] + 1;
    if (ny <= 0 || nz <= 0) continue;
    const int nr = ny * nz;
    for (int b = 0; b < nr; b += kG) {
      const int rr = b + g.gl;
      int s0 = 0, e0 = 0;
      if (rr < nr) {
        const int iz = D == 3 ? rr / ny : 0;
        row_range<D, LD>(c, w.cstart, L, R_, q, fr, lo[2] + iz, lo[1] + rr - iz * ny, s0, e0);
      }
      const int len = max(e0 - s0, 0);
      int inc = len;
#pragma unroll
      for (int o = 1; o < kG; o <<= 1) {
        const int t = __shfl_up_sync(g.mask, inc, o, kG);
        if (g.gl >= o) inc += t;
      }
      const unsigned full = g.ballot(len > 0);
      if (!full) continue;
      if (nrow + __popc(full) > kRowTile) flush();
      if (len > 0) {
        const int at = nrow + __popc(full & g.below);
        rt.off[at] = s0 - (T + inc - len);
        rt.end[at] = T + inc;
      }
      nrow += __popc(full);
      T += __shfl_sync(g.mask, inc, kG - 1, kG);
    }
  }
  if (T > 0) flush();
}

// Neighbour criterion, level_infor.cpp:491-500.
__device__ inline bool nb_test(double d2, double hi, double hj, double cutoff, double& dist) {
  double R = fmax(hi, hj) * cutoff + 1.e-10;
  if (d2 > R * R * (1.0 + 1.e-9)) return false;  // conservative pre-reject
  dist = sqrt(d2);
  return (dist <= (hi * cutoff + 1.e-10)) || (dist <= (hj * cutoff + 1.e-10));
}

// pair distance of the force passes: IEEE square root in FP32 (see wendland_aw)
__device__ inline double force_dist(double d2) { return sqrt(d2); }
__device__ inline float force_dist(float d2) { return sqrtf(d2); }

template <class R> __device__ inline R d2_of(const R* dr, int D) {
  R d2 = dr[0] * dr[0];
  d2 = madd(dr[1], dr[1], d2);
  if (D == 3) d2 = madd(dr[2], dr[2], d2);
  return d2;
}

// How a SURFACE or SEGMENT particle i pairs with a neighbour j that is not
// REAL, in the kernel sum (particle_mesh_generation.cpp:717-759) and the
// forces (:769-991): 1 = through the normal-angle filter (j of i's own type),
// 2 = without the filter, 0 = not at all.  A SURFACE particle takes SURFACE,
// SEGMENT and SINGULARITY neighbours; a SEGMENT particle SEGMENT and
// SINGULARITY neighbours.  Both skip REAL neighbours.
__device__ inline int char_pair(int ti, int tj) {
  if (ti == SURFACE_P) return tj == SURFACE_P ? 1 : 2;
  return tj == SEGMENT_P ? 1 : (tj == SINGULARITY_P ? 2 : 0);
}

// The neighbour criterion of a pair (A6, Refresh_neighbor_info,
// level_infor.cpp:469-506), decided as the reference's FP64 arithmetic decides
// it.  FP32-split: in FP32 outside the band, else on the world positions.
// FP64-plain: in FP32 on box-relative positions (two words of the record) when
// the distance clears the radius by the rounding of the positions (2^-21 of
// their magnitude, above the 3.5 * 2^-24 that three coordinate differences can
// be off by) and of the test (1e-5), else by the FP64 test itself; an FP64
// instruction costs 60 FP32 ones here, and nearly every candidate clears it.
template <int D, class R> struct PairTest;
template <int D> struct PairTest<D, float> {
  float4 a0, a1;
  float cut, R2i;
  __device__ PairTest(const KCtx& c, const float4* rec, long long i) {
    a0 = rec[2 * i];
    a1 = rec[2 * i + 1];
    cut = c.prm.cutoff_f;
    R2i = (a0.w * cut) * (a0.w * cut);
  }
  template <class LD>
  __device__ bool near(const KCtx& c, const float4* rec, int j) const {
    float4 b0, b1;
    LD::rec(rec, j, b0, b1);
    float dr[3];
    RecOps<D, float>::rel(c, a0, a1, b0, b1, dr);
    const float d2 = d2_of(dr, D);
    const float rj = b0.w * cut;
    const float Rm = fmaxf(R2i, rj * rj);
    if (d2 > Rm * kD2Accept) return false;
    return d2 < Rm * kD2Sure || exact_neighbor<D>(c, a0, a1, b0, b1);
  }
  // in FP32 alone: accepts the band, and notes in close that a pair lies in it
  __device__ bool near32(const KCtx& c, const float4& b0, const float4& b1, bool& close) const {
    float dr[3];
    RecOps<D, float>::rel(c, a0, a1, b0, b1, dr);
    const float d2 = d2_of(dr, D);
    const float rj = b0.w * cut;
    const float Rm = fmaxf(R2i, rj * rj);
    if (d2 > Rm * kD2Accept) return false;
    close = close || !(d2 < Rm * kD2Sure);
    return true;
  }
};
template <int D>
__device__ __noinline__ bool exact_neighbor64(const KCtx& c, const double4* rec, long long i, int j) {
  const double4 a0 = rec[2 * i], b0 = rec[2 * (long long)j];
  double dr[3], dist;
  RecOps<D, double>::rel(c, a0, a0, b0, b0, dr);
  return nb_test(d2_of(dr, D), a0.w, b0.w, c.prm.cutoff, dist);
}
template <int D> struct PairTest<D, double> {
  float4 f;  // box-relative position, h
  float cut, pad;
  long long i;
  __device__ PairTest(const KCtx& c, const double4* rec, long long i_) : i(i_) {
    f = RecOps<D, double>::filter(rec[2 * i + 1]);
    cut = c.prm.cutoff_f;
    pad = 0x1p-21f * (c.geo.ext_f + fabsf(f.x) + fabsf(f.y) + fabsf(f.z)) + 2.e-10f;
  }
  template <class LD>
  __device__ bool near(const KCtx& c, const double4* rec, int j) const {
    const float4 q = RecOps<D, double>::template load_filter<LD>(rec, j);
    const float dx = f.x - q.x, dy = f.y - q.y, dz = D == 3 ? f.z - q.z : 0.f;
    const float d2 = dx * dx + dy * dy + dz * dz, Rm = fmaxf(f.w, q.w) * cut;
    const float far = Rm * 1.00001f + pad, sure = Rm * 0.99999f - pad;
    if (d2 > far * far) return false;
    return (sure > 0.f && d2 < sure * sure) || exact_neighbor64<D>(c, rec, i, j);
  }
};

// Neighbour list of particle i by its group of kG lanes, in the fixed scan
// order.  Returns the number of neighbours (itself included); the list keeps the
// first cap.
template <int D, class R, class LD>
__device__ inline int list_group(const KCtx& c, const Buf<R>& b, const Work<R>& w, const GroupLanes& g, RowTile& rt,
                                 long long i) {
  const PairTest<D, R> pt(c, b.rec, i);
  const SOrigin<D, R> so(c, b.posh[i], b.key ? b.key[i] : 0);
  int* row = w.nbl + nb_slot(i, 0, w.cap);  // entry q at row[(q >> 3) * 256 + (q & 7)]
  int cnt = 0;
  group_scan<D, R, LD>(c, w, g, rt, i, so, [&](int j, bool in) {
    const bool ok = in && pt.template near<LD>(c, b.rec, j);
    const unsigned m = g.ballot(ok);
    const int pos = cnt + __popc(m & g.below);
    if (ok && pos < w.cap) row[((pos >> 3) << 8) + (pos & 7)] = j;
    cnt += __popc(m);
  });
  return cnt;
}

// Neighbour lists of 32 particles by one warp (FP32-split, 3D), lane l's particle i.
// The lanes that sit in neighbouring half cells (a segment: all 32 in the work
// order, a few groups in storage order) reach nearly the same rows of the
// sort table.  The lanes take one row each of the segment's bounding box, the
// rows' particles are loaded once, coalesced, those within reach of the box are
// put into a tile of 256 candidates in shared memory, and every lane tests
// the whole tile: with the positions relative to the segment's frame, |p|^2 +
// |c|^2 - 2 p . c - max(R_i, R_j)^2 takes two candidates at a time (packed FP32:
// three fused multiply-adds, two additions), and its sign bits shift into a
// mask.  The expanded form is off by at most 2^-20 (|p|^2 + |c|^2) (four fused
// operations on values of at most twice that, and the rounding of c); when a
// candidate of 32 comes closer to zero than that and the criterion's band of
// 2^-15 R^2, the lane decides the 32 again one by one, else the mask is the
// decision and the lane appends its set bits.  The tile is kept over rows and
// levels, so its words are full.  Lanes walking their own rows (430 candidates
// for 86 neighbours in the relaxed state) ran at a third of the warp's width.
constexpr int kTile = MRSPH_TILE_SIZE, kTileRows = 64, kSegX = MRSPH_TILE_SPAN_X, kSegYZ = MRSPH_TILE_SPAN_YZ;
template <int TILE>
struct WarpTile {
  static_assert(TILE % 64 == 0 && TILE <= 1024, "whole mask words, at most 32 of them");
  float4 xy[TILE / 2];  // (x0, x1, y0, y1) of two candidates
  float4 zq[TILE / 2];  // (z0, z1, |c|^2_0, |c|^2_1)
  float2 nr2[TILE / 2];  // squared cut-off radii, negated
  int id[TILE];
  unsigned mask[TILE / 32][32];
  int off[kTileRows], end[kTileRows];
};
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ inline float warp_fmin(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ inline float warp_fmax(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <class LD, int TILE>
__device__ inline int list_warp(const KCtx& c, const Buf<float>& b, const Work<float>& w, WarpTile<TILE>& wt, long long i,
                                bool act) {
  constexpr int D = 3;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, BIG = 0x3fffffff;
  float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f);
  int k[3] = {0, 0, 0}, own = 0;
  if (act) {
    a0 = b.rec[2 * i];
    PosOps<D, float>::unpack(b.key[i], k);
    own = (int)(signed char)((b.meta[i] >> 8) & 0xFF);
  }
  const float cut = c.prm.cutoff_f, nR2i = -((a0.w * cut) * (a0.w * cut));
  const int cap = w.cap;
  int* row = w.nbl + nb_slot(act ? i : 0, 0, cap);  // entry q at row[(q >> 3) * 256 + (q & 7)]
  int cnt = 0;
  unsigned rem = __ballot_sync(FULL, act);
  while (rem) {
    // the segment: the lanes within kSegX half cells of the first left, in x,
    // and kSegYZ in y and z (of its level; anchor cells are 2^-sh of a level's cell)
    const int seed = __ffs(rem) - 1;
    bool in = (rem >> lane) & 1u;
    const int sh = c.geo.ncl - 1 - __shfl_sync(FULL, own, seed);
    const int span = ((kSegX + 1) << sh) >> 1, span1 = ((kSegYZ + 1) << sh) >> 1;
    int ks[3];
    for (int d = 0; d < 3; d++) {
      ks[d] = __shfl_sync(FULL, k[d], seed);
      in = in && abs(k[d] - ks[d]) <= (d == 0 ? span : span1);
    }
    rem &= ~__ballot_sync(FULL, in);
    // frame: the middle anchor in x, the seed's in y and z; bounding box
    ks[0] = (__reduce_min_sync(FULL, in ? k[0] : BIG) + __reduce_max_sync(FULL, in ? k[0] : -1)) >> 1;
    float p[3] = {0.f, 0.f, 0.f}, lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
    const float ao[3] = {a0.x, a0.y, a0.z};
    for (int d = 0; d < D; d++) {
      p[d] = fmaf((float)(k[d] - ks[d]), c.geo.Af[d], ao[d]);
      lo[d] = warp_fmin(in ? p[d] : 3.e38f);
      hi[d] = warp_fmax(in ? p[d] : -3.e38f);
    }
    const float Rm2 = __int_as_float(__reduce_max_sync(FULL, in ? __float_as_int(-nR2i) : 0));  // largest R_i^2
    const float fk[3] = {(float)ks[0], (float)ks[1], (float)ks[2]};
    const float pp = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
    const unsigned long long pp2 = pack2(pp, pp);
    const unsigned long long mx = pack2(-2.f * p[0], -2.f * p[0]), my = pack2(-2.f * p[1], -2.f * p[1]);
    const unsigned long long mz = pack2(-2.f * p[2], -2.f * p[2]);
    int tn = 0;         // candidates in the tile
    float qmax = 0.f;   // this lane's largest |c|^2 and R_j^2 among those it put there
    float rmax = 0.f;
    // tests the tile's candidates, appends the hits, empties the tile
    auto drain = [&]() {
      const int nw = (tn + 31) >> 5, pad = (nw << 5) - tn;
      if (lane < pad) {
        const int t = tn + lane, s2 = 4 * (t >> 1) + (t & 1);
        float* xy = reinterpret_cast<float*>(wt.xy);
        float* zq = reinterpret_cast<float*>(wt.zq);
        xy[s2] = xy[s2 + 2] = zq[s2] = 0.f;
        zq[s2 + 2] = 3.e38f;  // |c|^2: never in reach
        reinterpret_cast<float*>(wt.nr2)[t] = 0.f;
      }
      const float qm = __int_as_float(__reduce_max_sync(FULL, __float_as_int(qmax)));
      const float rm = __int_as_float(__reduce_max_sync(FULL, __float_as_int(rmax)));
      const float band = fmaf(fmaxf(-nR2i, rm), 0x1.1p-15f, 0x1p-20f * (pp + qm));
      __syncwarp();
      unsigned slow = 0u, hits = 0u;
      for (int v = 0; v < nw; v++) {
        unsigned mask = 0u;
        float close = 3.e38f;
#pragma unroll
        for (int t = 0; t < 16; t++) {
          const ulonglong2 xy = *reinterpret_cast<const ulonglong2*>(&wt.xy[v * 16 + t]);
          const ulonglong2 zq = *reinterpret_cast<const ulonglong2*>(&wt.zq[v * 16 + t]);
          const float2 nr = wt.nr2[v * 16 + t];
          unsigned long long s = add2(zq.y, pp2);
          s = fma2(zq.x, mz, s);
          s = fma2(xy.y, my, s);
          s = fma2(xy.x, mx, s);
          s = add2(s, pack2(fminf(nR2i, nr.x), fminf(nR2i, nr.y)));
          const unsigned s0 = (unsigned)s, s1 = (unsigned)(s >> 32);
          mask = __funnelshift_l(s0, mask, 1);
          mask = __funnelshift_l(s1, mask, 1);
          close = fminf(close, fminf(fabsf(__uint_as_float(s0)), fabsf(__uint_as_float(s1))));
        }
        if (in) {
          if (close <= band) slow |= 1u << v;
          if (mask) hits |= 1u << v;
          wt.mask[v][lane] = mask;
        }
      }
      // a candidate within the band: its 32 again one by one, decided as the reference does
      while (slow) {
        const int v = __ffs(slow) - 1;
        slow &= slow - 1u;
        const PairTest<D, float> pt(c, b.rec, i);
        unsigned mask = 0u;
        for (int t = 0; t < min(32, tn - 32 * v); t++)
          if (pt.template near<LD>(c, b.rec, wt.id[32 * v + t])) mask |= 0x80000000u >> t;
        wt.mask[v][lane] = mask;
        hits = mask ? hits | (1u << v) : hits & ~(1u << v);
      }
      __syncwarp();
      // accept: candidate 32 v + t is bit 31 - t of word v; a lane goes on to its
      // next word as soon as one is used up
      unsigned mk = 0u;
      const int* id = wt.id;
      while (hits | mk) {
        if (!mk) {
          const int v = __ffs(hits) - 1;
          hits &= hits - 1u;
          mk = wt.mask[v][lane];
          id = wt.id + 32 * v;
        }
        const int t = __clz(mk);
        mk &= ~(0x80000000u >> t);
        if (cnt < cap) row[((cnt >> 3) << 8) + (cnt & 7)] = id[t];
        cnt++;
      }
      __syncwarp();
      tn = 0;
      qmax = 0.f;
      rmax = 0.f;
    };
    int nrow = 0, T = 0;
    // puts the rows' candidates that lie within reach of the box into the tile
    auto take_rows = [&]() {
      __syncwarp();
      int r = 0;
      for (int t0 = 0; t0 < T; t0 += 32) {
        const int t = t0 + lane;
        float e[3] = {0.f, 0.f, 0.f}, rr = 0.f;
        int j = 0;
        bool keep = false;
        if (t < T) {
          while (t >= wt.end[r]) r++;
          j = wt.off[r] + t;
          float4 b0, b1;
          LD::rec(b.rec, j, b0, b1);
          e[0] = fmaf(b1.x - fk[0], c.geo.Af[0], b0.x);
          e[1] = fmaf(b1.y - fk[1], c.geo.Af[1], b0.y);
          e[2] = fmaf(b1.z - fk[2], c.geo.Af[2], b0.z);
          const float rj = b0.w * cut;
          rr = rj * rj;
          float d2 = 0.f;
          for (int d = 0; d < D; d++) {
            const float gd = fmaxf(fmaxf(lo[d] - e[d], e[d] - hi[d]), 0.f);
            d2 = fmaf(gd, gd, d2);
          }
          keep = d2 <= fmaxf(Rm2, rr) * 1.0002f;
        }
        const unsigned m = __ballot_sync(FULL, keep);
        if (keep) {
          const int at = tn + __popc(m & ((1u << lane) - 1u)), s2 = 4 * (at >> 1) + (at & 1);
          const float q = fmaf(e[2], e[2], fmaf(e[1], e[1], e[0] * e[0]));
          float* xy = reinterpret_cast<float*>(wt.xy);
          float* zq = reinterpret_cast<float*>(wt.zq);
          xy[s2] = e[0];
          xy[s2 + 2] = e[1];
          zq[s2] = e[2];
          zq[s2 + 2] = q;
          reinterpret_cast<float*>(wt.nr2)[at] = -rr;
          wt.id[at] = j;
          qmax = fmaxf(qmax, q);
          rmax = fmaxf(rmax, rr);
        }
        tn += __popc(m);
        if (tn > TILE - 32) drain();
      }
      __syncwarp();
      nrow = 0;
      T = 0;
    };
    for (int L = 0; L < c.geo.ncl; L++) {
      if (c.sc->lcount[L] == 0) continue;
      const float R = warp_fmax(in ? LD::ld(&w.rlev[(long long)L * c.n + i]) : 0.f);
      if (!(R > 0.f)) continue;
      const float R2 = R * R;
      // half cell h of axis d covers [(h - h0) hs - f0, + hs) of the frame
      const int shl = c.geo.ncl - 1 - L;
      int h0[3] = {0, 0, 0}, r0[3] = {0, 0, 0}, r1[3] = {0, 0, 0};
      float f0[3] = {0.f, 0.f, 0.f};
      for (int d = 0; d < D; d++) {
        if (shl == 0) h0[d] = 2 * ks[d];
        else {
          h0[d] = ks[d] >> (shl - 1);
          f0[d] = (float)(ks[d] & ((1 << (shl - 1)) - 1)) * c.geo.Af[d];
        }
        const float ih = c.geo.ihs_f[L][d];
        r0[d] = max(h0[d] + (int)floorf((lo[d] - R + f0[d]) * ih), 0);
        r1[d] = min(h0[d] + (int)floorf((hi[d] + R + f0[d]) * ih), c.geo.hn[L][d] - 1);
      }
      if (r1[0] < r0[0] || r1[1] < r0[1] || r1[2] < r0[2]) continue;
      if (w.bstart && (r1[1] - r0[1] + 1) * (r1[2] - r0[2] + 1) > 64) {
        // many rows (a finer level): cut them to the bricks that hold particles
        const int b0y = r0[1] >> 2, b0z = r0[2] >> 2;
        const int nby = (r1[1] >> 2) - b0y + 1, nbz = (r1[2] >> 2) - b0z + 1;
        int ymin = BIG, ymax = -1, zmin = BIG, zmax = -1;
        for (int t = lane; t < nby * nbz; t += 32) {
          const int z = b0z + t / nby, y = b0y + t % nby;
          const long long at = c.geo.boff[L] + ((long long)z * c.geo.bn[L][1] + y) * c.geo.bn[L][0];
          if (LD::ld(&w.bstart[at + (r1[0] >> 2) + 1]) > LD::ld(&w.bstart[at + (r0[0] >> 2)])) {
            ymin = min(ymin, y); ymax = max(ymax, y);
            zmin = min(zmin, z); zmax = max(zmax, z);
          }
        }
        ymax = __reduce_max_sync(FULL, ymax);
        if (ymax < 0) continue;
        ymin = __reduce_min_sync(FULL, ymin);
        r0[1] = max(r0[1], 4 * ymin);
        r1[1] = min(r1[1], 4 * ymax + 3);
        r0[2] = max(r0[2], 4 * __reduce_min_sync(FULL, zmin));
        r1[2] = min(r1[2], 4 * __reduce_max_sync(FULL, zmax) + 3);
      }
      const int ny = r1[1] - r0[1] + 1, nr = ny * (r1[2] - r0[2] + 1);
      for (int rb = 0; rb < nr; rb += 32) {
        const int rr = rb + lane;
        int s0 = 0, e0 = 0;
        if (rr < nr) {
          const int iz = rr / ny;
          const int z = r0[2] + iz, y = r0[1] + rr - iz * ny;
          float gz = 0.f, gy = 0.f;
          const float zl = fmaf((float)(z - h0[2]), c.geo.hs_f[L][2], -f0[2]);
          if (z > 0) gz = fmaxf(gz, zl - hi[2]);
          if (z < c.geo.hn[L][2] - 1) gz = fmaxf(gz, lo[2] - (zl + c.geo.hs_f[L][2]));
          const float yl = fmaf((float)(y - h0[1]), c.geo.hs_f[L][1], -f0[1]);
          if (y > 0) gy = fmaxf(gy, yl - hi[1]);
          if (y < c.geo.hn[L][1] - 1) gy = fmaxf(gy, lo[1] - (yl + c.geo.hs_f[L][1]));
          const float left = R2 - gy * gy - gz * gz;
          if (left >= 0.f) {
            const float wd = sqrtf(left), ih = c.geo.ihs_f[L][0];
            const int xl = max(h0[0] + (int)floorf((lo[0] - wd + f0[0]) * ih), 0);
            const int xh = min(h0[0] + (int)floorf((hi[0] + wd + f0[0]) * ih), c.geo.hn[L][0] - 1);
            if (xl <= xh) {
              const long long at = c.geo.hoff[L] + ((long long)z * c.geo.hn[L][1] + y) * c.geo.hn[L][0];
              s0 = LD::ld(&w.cstart[at + xl]);
              e0 = LD::ld(&w.cstart[at + xh + 1]);
            }
          }
        }
        const int len = max(e0 - s0, 0);
        const unsigned full = __ballot_sync(FULL, len > 0);
        if (!full) continue;
        int inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(FULL, inc, o);
          if (lane >= o) inc += t;
        }
        if (nrow + __popc(full) > kTileRows) take_rows();
        if (len > 0) {
          const int at = nrow + __popc(full & ((1u << lane) - 1u));
          wt.off[at] = s0 - (T + inc - len);
          wt.end[at] = T + inc;
        }
        nrow += __popc(full);
        T += __shfl_sync(FULL, inc, 31);
      }
    }
    if (T > 0) take_rows();
    if (tn > 0) drain();
  }
  return cnt;
}

// Neighbour list of particle i by one lane (FP32-split), its rows one after the
// other, two candidates in flight, decided in FP32: -1 when a pair lies in the
// criterion's band (the hot loop has no registers for the exact test).
template <int D, class LD>
__device__ inline int list_lane(const KCtx& c, const Buf<float>& b, const Work<float>& w, long long i) {
  const PairTest<D, float> pt(c, b.rec, i);
  const SOrigin<D, float> so(c, b.posh[i], b.key[i]);
  const int cap = w.cap;
  int* row = w.nbl + nb_slot(i, 0, cap);  // entry q at row[(q >> 3) * 256 + (q & 7)]
  int cnt = 0;
  bool close = false;
  auto take = [&](int j) {
    if (cnt < cap) row[((cnt >> 3) << 8) + (cnt & 7)] = j;
    cnt++;
  };
  for (int L = 0; L < c.geo.ncl; L++) {
    const float R_ = LD::ld(&w.rlev[(long long)L * c.n + i]);
    if (!(R_ > 0.f)) continue;
    int q[3] = {0, 0, 0}, lo[3] = {0, 0, 0}, up[3] = {0, 0, 0};
    float fr[3] = {0.f, 0.f, 0.f};
    level_position<D>(c, L, so, q, fr);
    level_box<D>(c, L, R_, q, fr, lo, up);
    for (int z = lo[2]; z <= up[2]; z++)
      for (int y = lo[1]; y <= up[1]; y++) {
        int s0, e0;
        if (!row_range<D, LD>(c, w.cstart, L, R_, q, fr, z, y, s0, e0)) continue;
        for (int j = s0; j < e0; j += 2) {
          float4 b0, b1, c0, c1;
          LD::rec(b.rec, j, b0, b1);
          LD::rec(b.rec, min(j + 1, e0 - 1), c0, c1);
          if (pt.near32(c, b0, b1, close)) take(j);
          if (j + 1 < e0 && pt.near32(c, c0, c1, close)) take(j + 1);
        }
      }
  }
  return close ? -1 : cnt;
}
// Lists of the 32 particles from first, lane l's being first + l.  Those with a
// pair in the band (one particle in 300 of 74 neighbours, so one warp in ten)
// are taken again by groups, which decide as the reference does; a lane taking
// them again made its warp wait for a second whole list.
template <int D, class LD>
__device__ inline int list_lanes(const KCtx& c, const Buf<float>& b, const Work<float>& w, RowTile& rt,
                                 long long first) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int cnt = first + lane < c.n ? list_lane<D, LD>(c, b, w, first + lane) : 0;
  unsigned again = __ballot_sync(FULL, cnt < 0);
  while (again) {
    const GroupLanes g;
    unsigned left = again;  // group k takes the k-th of them
    for (int k = 0; k < lane / kG; k++) left &= left - 1u;
    const int own = left ? __ffs(left) - 1 : -1;
    for (int k = 0; k < 32 / kG; k++) again &= again - 1u;
    int m = 0;
    if (own >= 0) m = list_group<D, float, LD>(c, b, w, g, rt, first + own);
    __syncwarp();
    for (int k = 0; k < 32; k += kG) {
      const int to = __shfl_sync(FULL, own, k), v = __shfl_sync(FULL, m, k);
      if (lane == to) cnt = v;
    }
  }
  return cnt;
}

// what follows a list: its length, the spill queue, the step's totals
template <int D, class R>
__device__ inline void list_done(const KCtx& c, const Work<R>& w, long long i, int cnt, bool lead) {
  if (lead) {
    w.cnt[i] = cnt;
    if (cnt > w.cap) atomicOr(&c.sc->flags, (unsigned)FLAG_SPILL);
  }
  queue_push(lead && cnt > w.cap, &c.sc->nspill, w.spillq, (int)i);
  const unsigned mc = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
  const unsigned ps = __reduce_add_sync(0xffffffffu, lead ? (unsigned)(cnt - 1) : 0u);
  if ((threadIdx.x & 31) == 0) {
    if (mc > 1) atomicMax(&c.sc->maxcnt, mc);
    if (ps) atomicAdd(&c.sc->pairs, (unsigned long long)ps);
  }
}

// particles [first, first + blockDim.x / kG), a group each
template <int D, class R, class LD = LdNC>
__device__ inline void density_group_block(const KCtx& c, const Buf<R>& b, const Work<R>& w, RowTile* tiles,
                                           long long first) {
  const GroupLanes g;
  const long long i = first + threadIdx.x / kG;
  int cnt = 0;
  if (i < c.n) cnt = list_group<D, R, LD>(c, b, w, g, tiles[threadIdx.x / kG], i);
  __syncwarp();
  list_done<D, R>(c, w, i, cnt, i < c.n && g.gl == 0);
}

// particles [first, first + blockDim.x), one warp per 32
template <class LD = LdNC, int TILE>
__device__ inline void density_warp_block(const KCtx& c, const Buf<float>& b, const Work<float>& w, WarpTile<TILE>* tiles,
                                          long long first) {
  const long long t = first + threadIdx.x;
  const bool act = t < c.n;
  const long long i = act && w.order ? w.order[t] : t;
  const int cnt = list_warp<LD>(c, b, w, tiles[threadIdx.x >> 5], i, act);
  list_done<3, float>(c, w, i, cnt, act);
}

// particles [first, first + blockDim.x), a lane each
template <int D, class LD = LdNC>
__device__ inline void density_lane_block(const KCtx& c, const Buf<float>& b, const Work<float>& w, RowTile* tiles,
                                          long long first) {
  const long long i = first + threadIdx.x;
  const int cnt = list_lanes<D, LD>(c, b, w, tiles[threadIdx.x / kG], i - (threadIdx.x & 31));
  list_done<D, float>(c, w, i, cnt, i < c.n);
}

constexpr int kDensityThreads = 128;
template <int D>
__global__ void __launch_bounds__(kDensityThreads, D == 2 ? 8 : 10) k_density_lane(KCtx c, Buf<float> b, Work<float> w) {
  chain_wait();
  __shared__ RowTile tiles[kDensityThreads / kG];
  density_lane_block<D>(c, b, w, tiles, (long long)blockIdx.x * kDensityThreads);
}
template <int D, class R>
__global__ void __launch_bounds__(kDensityThreads, 10) k_density_group(KCtx c, Buf<R> b, Work<R> w) {
  chain_wait();
  __shared__ RowTile tiles[kDensityThreads / kG];
  density_group_block<D, R>(c, b, w, tiles, (long long)blockIdx.x * (kDensityThreads / kG));
}
template <int D>
__global__ void __launch_bounds__(kDensityThreads, MRSPH_DENSITY_MIN_BLOCKS) k_density_tile(KCtx c, Buf<float> b, Work<float> w) {
  chain_wait();
  __shared__ WarpTile<kTile> tiles[kDensityThreads / 32];
  density_warp_block<LdNC>(c, b, w, tiles, (long long)blockIdx.x * kDensityThreads);
}

__device__ inline void accum_pairs_body(DevScalars* sc) { sc->pairs_total += sc->pairs; }

// four consecutive pair coefficients (16-byte aligned)
__device__ inline void store4(float* p, const float* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ inline void store4(double* p, const double* v) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}
template <class LD>
__device__ inline void load4(const float* p, float* v) {
  const float4 t = LD::ld(reinterpret_cast<const float4*>(p));
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <class LD>
__device__ inline void load4(const double* p, double* v) {
  const double2 t0 = LD::ld(reinterpret_cast<const double2*>(p)), t1 = LD::ld(reinterpret_cast<const double2*>(p) + 1);
  v[0] = t0.x; v[1] = t0.y; v[2] = t1.x; v[3] = t1.y;
}

// A7 Get_kernel_summation (particle_mesh_generation.cpp:690-765), A8 force
// stages, A9 timestep (Set_timestep(stage), :127-145).
// Stage 1 forms the kernel sum and the pressure force together: the force of a
// pair is sum_i * c_ij dr_ij with the pair coefficient c_ij = aw * (1/rho_i^2 +
// 1/rho_j^2), so the inverted sum scales the accumulated force at the end and
// the distance is computed once.  It stores c_ij in the neighbour list's layout (0
// for a pair the forces skip), and per particle (a1, eta), eta = nu * rho, negated for a
// particle that is not REAL.  The stage-2 viscous term of a pair is c_ij * eta_ij *
// (v_i - v_j) (:1021-1049), so stage 2 reads the coefficient and one vector per
// neighbour; a particle whose list spilled re-scans its cells and recomputes c_ij
// in both stages.  Stage 0 forms the kernel sum alone (a step that stops after
// the density phase).
// A particle is taken by one thread (G = 1) or by a group of kG lanes (G = kG),
// which share its entries kG at a time and hand their terms to lanes 0 to 3,
// one per component, to be added in list order: the sums, and so every bit,
// are the same.  One thread is the cheaper form once the chip is full; below
// that a group shortens the chain of gathers that bounds the kernel (see
// kGroupMax).
// FP32 Wendland C2 gradient over distance in DK dimensions (0 in 1D, the
// reference's quirk), Derivative_kernel_function (particle.cpp:732-750):
// -5 C (1 - s/2)^3 s / h / (r + 1e-15) with C = norm / h^DK and s = r / h,
// which is -5 norm (1 - s/2)^3 / h^(DK+2) for r > 0 in FP32, and 0 at r = 0.
// 1/h is rounded correctly (__frcp_rn): the hardware approximation's error
// is a smooth function of h, so pairs of similar h_ij share it and a
// near-balanced sum of hundreds of pair forces does not average it out (it
// acts as a slightly different kernel); the force passes take the distance
// from an IEEE square root for the same reason (force_dist).
template <int DK>
__device__ inline float wendland_aw(float dist, float h) {
  if (DK == 1) return 0.f;
  const float ih = __frcp_rn(h);
  const float t = fmaxf(fmaf(-0.5f * ih, dist, 1.f), 0.f);
  float ihp = (ih * ih) * (ih * ih);
  if (DK == 3) ihp *= ih;
  return dist > 0.f ? (-5.f * (float)kern_norm(K_WEN, DK)) * ihp * (t * t * t) : 0.f;
}

// Shared memory of a group of kG lanes.
template <class R>
struct GroupTile {
  RowTile rows;       // the candidate scan of a spilled particle
  int vlist[2 * kG];  // its neighbours, kG at a time
  R term[4][kG];      // force components and kernel-sum term of the entries in hand
};

// One particle of a force stage.  SPILL = false: the particle's list is complete
// (cnt <= cap); SPILL = true: it spilled, and its cells are scanned for the
// list's entries in their order, so a spill changes nothing.  my_dt / my_v take
// the min / max (of the group's first lane).
template <int D, class R, int STAGE, int KK, int G, bool SPILL, class LD = LdNC>
__device__ inline void force_particle(const KCtx& c, const Buf<R>& b, const Work<R>& w, const GroupLanes& g,
                                      GroupTile<R>* gt, long long i, double& my_dt, double& my_v) {
  using Q = RecOps<D, R>;
  constexpr bool F32 = std::is_same<R, float>::value;
  constexpr bool WEN32 = F32 && KK == K_WEN;
  constexpr bool GEO = STAGE < 2 || SPILL;  // the pair geometry is needed
  using T4 = typename V4<R>::T;
  const T4 a0 = b.rec[2 * i], a1r = b.rec[2 * i + 1];
  const int ti = b.meta[i] & 0xFF;
  const int kind = KK >= 0 ? KK : c.prm.kernel;
  R ni[3] = {0, 0, 0};
  if (ti != REAL_P) {
    const T4 nri = b.nr[i];
    ni[0] = nri.x; ni[1] = nri.y; ni[2] = nri.z;
  }
  const R rho = b.nr[i].w, h = a0.w;
  const R inv_h = STAGE < 2 ? pair_inv(h) : (R)0;
  R eta_i = 0, hdt1 = 0;
  R vi[3] = {0, 0, 0};
  if (STAGE == 2) {
    hdt1 = (R)(0.5 * bitsd(c.sc->dt1));
    const T4 an = w.a1[i];
    vi[0] = rmul(an.x, hdt1); vi[1] = rmul(an.y, hdt1); vi[2] = rmul(an.z, hdt1);
    eta_i = r_fabs(an.w);
  }
  // FP32-split accumulates a particle's pair forces in groups of four list
  // entries and adds each group's sum into F with compensated (Kahan)
  // summation.  The list is in scan order (levels, then z, y rows), so a plain
  // running sum first collects every same-signed term of one side and reaches
  // about half of sum |terms| before the other side cancels it; rounding at that
  // magnitude, not the terms, dominated the FP32 error.  FP64-plain sums
  // plainly.  G = 1: components 0..2; G = kG: lane d < 3 holds component d in
  // F[0] (and lane 3 the kernel sum in sum).
  R F[3] = {0, 0, 0}, Fb[3] = {0, 0, 0}, Fc[3] = {0, 0, 0};
  R sum = 0;
  int ncount = 0;
  auto accum = [&](int d, R v) {
    if constexpr (F32) Fb[d] = radd(Fb[d], v);
    else F[d] = F[d] + v;
  };
  auto flush = [&](int d) {
    if constexpr (F32) {
      const float y = Fb[d] - Fc[d];
      const float t = F[d] + y;
      Fc[d] = (t - F[d]) - y;
      F[d] = t;
      Fb[d] = 0.f;
    }
  };
  const R vol_i = (R)1.0 / (rho * rho);
  const R CW = (!F32 && STAGE < 2) ? kernel_C<R>(kind, D, h) : (R)0;
  // kernel-sum term of a pair at distance r in dim dimensions
  auto W = [&](int dim, R r) -> R {
    if constexpr (F32) return kernel_W_fast(kind, dim, (float)r, (float)inv_h);
    else return dim == D ? kernel_W_C<R>(kind, dim, quot(r, h, inv_h), CW) : kernel_W<R>(kind, dim, r, h);
  };
  // pair (i, j): the skip rules of :717-759, :904-920 and :1019-1031; its
  // kernel-sum term wt (true when it counts), and the pair coefficient cij and
  // the direction dr its force acts along (cij = 0: no force)
  auto pair = [&](int j, R* dr, R& cij, R& wt) -> bool {
    T4 b0, b1;
    LD::rec(b.rec, j, b0, b1);
    Q::rel(c, a0, a1r, b0, b1, dr);
    const R hij = (R)0.5 * (h + b0.w);
    cij = 0;
    wt = 0;
    if (ti == REAL_P) {
      const R dist = force_dist(dot3<D, R>(dr, dr));
      if (STAGE < 2) {
        if constexpr (WEN32) {
          // (1 - s/2)^4 (1 + 2s), s = r/h, clamped at s = 2; the
          // normalisation C/h^D comes once at the end
          const float s = (float)dist * (float)inv_h;
          const float t = fmaxf(fmaf(-0.5f, s, 1.f), 0.f), t2 = t * t;
          wt = rmul(t2 * t2, fmaf(2.f, s, 1.f));
        } else {
          wt = W(D, dist);
        }
      }
      if (STAGE > 0 && j != (int)i) {
        R aw;
        if constexpr (WEN32) aw = wendland_aw<D>(dist, hij);
        else aw = pair_dW(kind, D, dist, hij);
        cij = aw * (vol_i + r_fabs(b1.w));
      }
      return true;
    }
    if (!(b1.w < (R)0)) return false;  // SURFACE or SEGMENT: j must not be REAL
    const int rule = char_pair(ti, b.meta[j] & 0xFF);
    if (rule == 0) return false;
    const R dn = dot3<D, R>(dr, ni);
    for (int d = 0; d < 3; d++) dr[d] = madd(-ni[d], dn, dr[d]);
    if (rule == 1) {
      const T4 nrj = b.nr[j];
      const R nj[3] = {nrj.x, nrj.y, nrj.z};
      const R ca = r_fabs(dot3<D, R>(ni, nj)), cos_t = pick<R>(c.prm.cos_thres, c.prm.cos_thres_f);
      bool ok = ca > cos_t;
      if constexpr (F32) {
        if (fabsf(ca - cos_t) <= kBandCos) ok = exact_cos<D>(c, (const float*)ni, (const float*)nj);
      }
      if (!ok) return false;
    }
    const R dist = force_dist(dot3<D, R>(dr, dr));
    if (STAGE > 0 && j != (int)i) {
      R aw;
      if (ti == SEGMENT_P) {  // the 1D kernel gradient in 3D, none in 2D (:769-879)
        if constexpr (WEN32) aw = wendland_aw<1>(dist, hij);
        else aw = (D == 3) ? pair_dW(kind, 1, dist, hij) : (R)0;
      } else {
        if constexpr (WEN32) aw = wendland_aw<D - 1>(dist, hij);
        else aw = pair_dW(kind, D - 1, dist, hij);
      }
      cij = aw * (vol_i + r_fabs(b1.w));
    }
    if (STAGE == 2 || !(ti == SURFACE_P || D == 3)) return false;  // a SEGMENT particle sums in 3D only (:740-759)
    wt = W(ti == SEGMENT_P ? 1 : D - 1, dist);
    return true;
  };
  // viscous term of neighbour j
  auto visc = [&](int j, R cij, R* t) {
    const T4 anj = w.a1[j];
    const bool char_j = signbit(anj.w);  // j is not REAL
    R vj[3];
    if (ti == REAL_P && char_j) {
      vj[0] = vi[0] * (R)-1.0; vj[1] = vi[1] * (R)-1.0; vj[2] = vi[2] * (R)-1.0;
    } else {
      vj[0] = rmul(anj.x, hdt1); vj[1] = rmul(anj.y, hdt1); vj[2] = rmul(anj.z, hdt1);
    }
    const R eta_j = r_fabs(anj.w);
    const R eta_ij = r_div((R)2. * eta_j * eta_i, eta_i + eta_j + (R)1.e-15);
    const R temp0 = cij * eta_ij;
    for (int d = 0; d < D; d++) t[d] = rmul(vi[d] - vj[d], temp0);
  };
  // entry j: its force terms t (0 when it has none), its kernel-sum term; cij is
  // the stored coefficient (read in stage 2, written in stage 1).  Returns
  // whether it counts towards the kernel sum.
  auto entry = [&](int j, R& cij, R* t, R& wt) -> bool {
    bool counts = false;
    t[0] = t[1] = t[2] = 0;
    wt = 0;
    if constexpr (GEO) {
      R dr[3], cg;
      counts = pair(j, dr, cg, wt);
      cij = cg;
      if (STAGE == 1)
        for (int d = 0; d < D; d++) t[d] = rmul(dr[d], cij);
    }
    if (STAGE == 2 && cij != (R)0) visc(j, cij, t);
    return counts;
  };
  const int cnt = w.cnt[i];
  if (ti != SINGULARITY_P) {  // a SINGULARITY particle has no kernel sum and no force
    if constexpr (G == 1) {
      int q = 0;  // entries taken
      auto take = [&](int j, R& cij) {
        R t[3], wt;
        if (entry(j, cij, t, wt)) {
          sum = radd(sum, wt);
          ncount++;
        }
        if (STAGE > 0)
          for (int d = 0; d < D; d++) accum(d, t[d]);
      };
      static_assert(!SPILL, "a spilled particle is taken by a group");
      const long long base = nb_slot(i, 0, w.cap);
      const int* row = w.nbl + base;
      R* crow = w.pc + base;
      // four entries per access: q is a multiple of 4, so row + o and
      // crow + o are 16-byte aligned; entries past cnt inside the group
      // lie within the particle's cap and are ignored (stage 1 stores 0)
      for (; q < cnt; q += 4) {
        const int o = ((q >> 3) << 8) + (q & 7);
        const int4 j4 = LD::ld(reinterpret_cast<const int4*>(row + o));
        const int jj[4] = {j4.x, j4.y, j4.z, j4.w};
        R cc[4] = {0, 0, 0, 0};
        if (STAGE == 2) load4<LD>(crow + o, cc);
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (q + k < cnt) take(jj[k], cc[k]);
        if (STAGE == 1) store4(crow + o, cc);
        for (int d = 0; d < D; d++) flush(d);
      }
    } else {
      // entries q0 .. q0 + kG - 1, this lane's being j (on = false past the end)
      auto chunk = [&](int q0, int j, bool on, R* crow) {
        R t[3] = {0, 0, 0}, wt = 0, cij = 0;
        bool counts = false;
        if (on) {
          if (STAGE == 2 && !SPILL) cij = LD::ld(crow);
          counts = entry(j, cij, t, wt);
          if (STAGE == 1 && !SPILL) *crow = cij;
        }
        if (STAGE > 0)
          for (int d = 0; d < D; d++) gt->term[d][g.gl] = t[d];
        if (STAGE < 2) {
          gt->term[3][g.gl] = wt;
          ncount += __popc(g.ballot(counts));
        }
        __syncwarp(g.mask);
        if constexpr (!F32 && STAGE == 1) {  // plain sums of all four components at once
          if (g.gl < 4) {
            const R* v = gt->term[g.gl];
            R acc = g.gl == 3 ? sum : F[0];
            for (int k = 0; k < kG; k++) acc = acc + v[k];
            if (g.gl == 3) sum = acc;
            else F[0] = acc;
          }
        } else {
          if (STAGE > 0 && g.gl < D) {
            const R* v = gt->term[g.gl];
            for (int k = 0; k < 4; k++) accum(0, v[k]);
            flush(0);
            if (q0 + 4 < cnt) {
              for (int k = 4; k < kG; k++) accum(0, v[k]);
              flush(0);
            }
          }
          if (STAGE < 2 && g.gl == 3)
            for (int k = 0; k < kG; k++) sum = radd(sum, gt->term[3][k]);
        }
        __syncwarp(g.mask);
      };
      if constexpr (!SPILL) {
        const long long base = nb_slot(i, g.gl, w.cap);  // entry q0 + gl at base + 32 q0
        for (int q0 = 0; q0 < cnt; q0 += kG) {
          const bool on = q0 + g.gl < cnt;
          chunk(q0, on ? LD::ld(w.nbl + base + 32 * q0) : 0, on, w.pc + base + 32 * q0);
        }
      } else {
        const PairTest<D, R> pt(c, b.rec, i);
        const SOrigin<D, R> so(c, b.posh[i], b.key ? b.key[i] : 0);
        int held = 0, q0 = 0;
        group_scan<D, R, LD>(c, w, g, gt->rows, i, so, [&](int j, bool in) {
          const bool ok = in && pt.template near<LD>(c, b.rec, j);
          const unsigned m = g.ballot(ok);
          if (ok) gt->vlist[held + __popc(m & g.below)] = j;
          held += __popc(m);
          __syncwarp(g.mask);
          if (held >= kG) {
            chunk(q0, gt->vlist[g.gl], true, nullptr);
            q0 += kG;
            held -= kG;
            const int rest = g.gl < held ? gt->vlist[kG + g.gl] : 0;
            __syncwarp(g.mask);
            if (g.gl < held) gt->vlist[g.gl] = rest;
            __syncwarp(g.mask);
          }
        });
        if (held > 0) chunk(q0, g.gl < held ? gt->vlist[g.gl] : 0, g.gl < held, nullptr);
      }
    }
  }
  if (G > 1) {
    if (STAGE > 0) {
      if constexpr (F32) F[0] = F[0] - Fc[0];
      F[1] = __shfl_sync(g.mask, F[0], 1, kG);
      F[2] = __shfl_sync(g.mask, F[0], 2, kG);
    }
    if (STAGE < 2) sum = __shfl_sync(g.mask, sum, 3, kG);
    if (g.gl != 0) return;
    if (D == 2) F[2] = 0;
  } else if constexpr (F32) {
    for (int d = 0; d < D; d++) F[d] = F[d] - Fc[d];
  }
  if (STAGE < 2) {
    if (ti == REAL_P) {
      if (WEN32) sum = rmul(sum, (R)((float)kern_norm(K_WEN, D) * (D == 3 ? inv_h * inv_h * inv_h : inv_h * inv_h)));
      ncount = cnt;
    }
    if (ncount > 1) sum = (R)1. / radd(sum, (R)1.e-15);
    w.sum[i] = sum;
    if (STAGE == 0) return;
  }
  R a[3] = {0, 0, 0};
  if (ti != SINGULARITY_P) {
    for (int d = 0; d < D; d++) a[d] = STAGE == 1 ? rmul(F[d], -sum) : F[d];
    if (STAGE == 2)
      for (int d = 0; d < D; d++) a[d] = madd(vi[d], pick<R>(c.prm.damp_coeff, c.prm.damp_coeff_f), a[d]);
    if (ti == SURFACE_P || ti == SEGMENT_P) {  // Map_surface_particle_force, :1122-1126
      R nf = dot3<D, R>(a, ni);
      for (int d = 0; d < D; d++) a[d] = madd(-ni[d], nf, a[d]);
    }
  }
  R U = r_sqrt(dot3<D, R>(vi, vi));
  R A = r_sqrt(dot3<D, R>(a, a));
  R ts = (R)0.25 * r_sqrt(h / (A + (R)1.e-15));
  ts = AMIN1(ts, h / (R)40. / (U + (R)1.e-15));
  if (STAGE == 2) {
    R nu_new = pick<R>(c.prm.nu_coeff, c.prm.nu_coeff_f) * h * U;
    ts = AMIN1(ts, (R)0.125 * h * h / radd(nu_new, (R)1.e-15));
    b.nu_next[i] = nu_new;
    b.v1[i] = mk4<R>(vi[0], vi[1], vi[2], U);
    b.a2[i] = mk4<R>(a[0], a[1], a[2], 0);
  } else {
    const R eta = b.nu[i] * rho;
    w.a1[i] = mk4<R>(a[0], a[1], a[2], ti != REAL_P ? -eta : eta);
  }
  my_dt = fmin(my_dt, (double)ts);
  my_v = fmax(my_v, (double)U);
}

template <int STAGE>
__device__ inline void force_reduce(const KCtx& c, double my_dt, double my_v) {
  if (STAGE == 1) block_minmax_to_global(my_dt, my_v, &c.sc->dt1, &c.sc->vmax1);
  if (STAGE == 2) block_minmax_to_global(my_dt, my_v, &c.sc->dt2, &c.sc->vmax2);
}

// KK: the kernel kind fixed at compile time (FP32 Wendland C2), or -1.
// The blockDim.x / G particles from first; those whose list spilled are left to
// k_force_spill.  gt: a GroupTile per group (G = kG).
template <int D, class R, int STAGE, int KK, int G, class LD = LdNC>
__device__ inline void force_block(const KCtx& c, const Buf<R>& b, const Work<R>& w, GroupTile<R>* gt,
                                   long long first) {
  const GroupLanes g;
  double my_dt = 1.e300, my_v = 0.0;
  const long long i = first + threadIdx.x / G;
  if (i < c.n && w.cnt[i] <= w.cap)
    force_particle<D, R, STAGE, KK, G, false, LD>(c, b, w, g, G > 1 ? gt + threadIdx.x / G : nullptr, i, my_dt, my_v);
  __syncwarp();
  force_reduce<STAGE>(c, my_dt, my_v);
}

template <int D, class R, int STAGE, int KK>
__global__ void __launch_bounds__(256, (std::is_same<R, float>::value ? (STAGE == 1 ? MRSPH_FORCE_MIN_BLOCKS : MRSPH_FORCE2_MIN_BLOCKS) : 1)) k_force(KCtx c, Buf<R> b, Work<R> w) {
  chain_wait();
  if (STAGE < 2 && blockIdx.x == 0 && threadIdx.x == 0) accum_pairs_body(c.sc);
  force_block<D, R, STAGE, KK, 1>(c, b, w, nullptr, (long long)blockIdx.x * 256);
}

constexpr int kGroupThreads = 128;
// The force stage of the particles whose list spilled (queued by the list
// pass; grid-stride over groups), re-scanning their cells.
template <int D, class R, int STAGE, int KK, class LD = LdNC>
__device__ inline void force_spill_items(const KCtx& c, const Buf<R>& b, const Work<R>& w, GroupTile<R>* gt,
                                         long long blk, long long nblk) {
  const GroupLanes g;
  double my_dt = 1.e300, my_v = 0.0;
  const long long nq = c.sc->nspill, per = blockDim.x / kG;
  if (blk * per >= nq) return;  // block-uniform: nothing queued for this block
  for (long long t = blk * per + threadIdx.x / kG; t < nq; t += nblk * per) {
    const int i = w.spillq[t];
    if (w.cnt[i] > w.cap)
      force_particle<D, R, STAGE, KK, kG, true, LD>(c, b, w, g, gt + threadIdx.x / kG, i, my_dt, my_v);
  }
  __syncwarp();
  force_reduce<STAGE>(c, my_dt, my_v);
}

template <int D, class R, int STAGE, int KK>
__global__ void __launch_bounds__(kGroupThreads, std::is_same<R, float>::value ? 8 : 1) k_force_group(KCtx c, Buf<R> b, Work<R> w) {
  chain_wait();
  __shared__ GroupTile<R> gt[kGroupThreads / kG];
  if (STAGE < 2 && blockIdx.x == 0 && threadIdx.x == 0) accum_pairs_body(c.sc);
  force_block<D, R, STAGE, KK, kG>(c, b, w, gt, (long long)blockIdx.x * (kGroupThreads / kG));
}

template <int D, class R, int STAGE, int KK>
__global__ void __launch_bounds__(kGroupThreads) k_force_spill(KCtx c, Buf<R> b, Work<R> w) {
  chain_wait();
  __shared__ GroupTile<R> gt[kGroupThreads / kG];
  force_spill_items<D, R, STAGE, KK>(c, b, w, gt, blockIdx.x, gridDim.x);
}

// ----------------------------------------------------------------- taps
template <int D, class R>
__global__ void k_tap(KCtx c, Buf<R> b, Work<R> w, const int* __restrict__ slot_of_id, double* out, int field,
                      int have_work) {
  using P = PosOps<D, R>;
  long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= c.n) return;
  int s = slot_of_id[k];
  double* o3 = out + 3 * k;
  switch (field) {
    case 0: { double x[3]; P::world(c, b.posh[s], b.key ? b.key[s] : 0, x); o3[0] = x[0]; o3[1] = x[1]; o3[2] = x[2]; break; }
    case 1: {  // velocity after the last complete step
      double dt2 = bitsd(c.sc->dt2);
      auto v1 = b.v1[s]; auto a2 = b.a2[s];
      R hdt = (R)(0.5 * dt2);
      o3[0] = (double)(v1.x + a2.x * hdt); o3[1] = (double)(v1.y + a2.y * hdt);
      o3[2] = (D == 3) ? (double)(v1.z + a2.z * hdt) : 0.0;
      break;
    }
    case 2: { auto q = b.nr[s]; o3[0] = q.x; o3[1] = q.y; o3[2] = q.z; break; }
    case 3: { auto q = have_work ? w.a1[s] : mk4<R>(0, 0, 0, 0); o3[0] = q.x; o3[1] = q.y; o3[2] = q.z; break; }
    case 4: { auto q = b.a2[s]; o3[0] = q.x; o3[1] = q.y; o3[2] = q.z; break; }
    case 5: out[k] = (double)b.posh[s].w; break;
    case 6: out[k] = (double)b.phi[s]; break;
    case 7: out[k] = (double)b.curv[s]; break;
    case 8: out[k] = have_work ? (double)w.sum[s] : 0.0; break;
    case 9: out[k] = (double)b.nr[s].w; break;
    case 10: out[k] = (double)b.nu_next[s]; break;
    case 11: out[k] = (double)(b.meta[s] & 0xFF); break;
    case 12: out[k] = (double)(signed char)((b.meta[s] >> 8) & 0xFF); break;
  }
}

// triangulation inputs by particle id; rows translated to ids and sorted
template <int D, class R>
__global__ void k_export_tri(KCtx c, Buf<R> b, Work<R> w, double* __restrict__ xyz, int* __restrict__ type,
                             double* __restrict__ phi, int* __restrict__ rows, int* __restrict__ cnt, int rowcap,
                             unsigned* flags, double* __restrict__ hout, bool sort_rows) {
  using P = PosOps<D, R>;
  long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= c.n) return;
  int s = w.slot_of_id[k];
  double x[3];
  P::world(c, b.posh[s], b.key ? b.key[s] : 0, x);
  xyz[3 * k] = x[0]; xyz[3 * k + 1] = x[1]; xyz[3 * k + 2] = x[2];
  type[k] = b.meta[s] & 0xFF;
  phi[k] = (double)b.phi[s];
  if (hout) hout[k] = (double)b.posh[s].w;
  int m = w.cnt[s];
  if (m > w.cap || m > rowcap) { atomicOr(flags, 4u); m = min(w.cap, rowcap); }
  cnt[k] = m;
  const int* src = w.nbl + nb_slot(s, 0, w.cap);
  int* dst = rows + k * rowcap;
  if (!sort_rows) {
    for (int q = 0; q < m; q++) dst[q] = b.id[src[((q >> 3) << 8) + (q & 7)]];
    return;
  }
  for (int q = 0; q < m; q++) {  // insertion sort by id
    int v = b.id[src[((q >> 3) << 8) + (q & 7)]];
    int p = q;
    while (p > 0 && dst[p - 1] > v) { dst[p] = dst[p - 1]; p--; }
    dst[p] = v;
  }
}

template <int D, class R>
__global__ void k_upload(KCtx c, Buf<R> b, const double* __restrict__ xyz) {
  using P = PosOps<D, R>;
  long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= c.n) return;
  int id = b.id[s];
  double x[3] = {xyz[3 * (long long)id], xyz[3 * (long long)id + 1], xyz[3 * (long long)id + 2]};
  auto p = b.posh[s];
  int key = b.key ? b.key[s] : 0;
  P::set_world(c, p, key, x);
  b.posh[s] = p;
  if (b.key) b.key[s] = key;
}

template <int D, class R>
__global__ void k_set_state(KCtx c, Buf<R> b, const double* __restrict__ in, int has_v, int has_h, int has_nu,
                            int has_level, const int* __restrict__ type, const int* __restrict__ level) {
  using P = PosOps<D, R>;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.n) return;
  const long long n = c.n;
  double x[3] = {in[3 * i], in[3 * i + 1], in[3 * i + 2]};
  typename V4<R>::T p = mk4<R>(0, 0, 0, has_h ? (R)in[9 * n + i] : (R)0);
  int key = 0;
  P::set_world(c, p, key, x);
  b.posh[i] = p;
  if (b.key) b.key[i] = key;
  R v[3] = {0, 0, 0};
  if (has_v) for (int d = 0; d < 3; d++) v[d] = (R)in[3 * n + 3 * i + d];
  b.v1[i] = mk4<R>(v[0], v[1], v[2], 0);
  b.a2[i] = mk4<R>(0, 0, 0, 0);
  R nu = has_nu ? (R)in[6 * n + i] : (R)0;
  b.nu[i] = nu;
  b.nu_next[i] = nu;
  int t = type ? type[i] : REAL_P;
  int e = has_level ? level[i] : 0;
  b.meta[i] = t | ((e & 0xFF) << 8);
  b.id[i] = (int)i;
  b.nr[i] = mk4<R>(0, 0, 0, 0);
  b.phi[i] = 0;
  b.curv[i] = 0;
}

static __global__ void k_iota(int* a, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = (int)i;
}

template <int D, class R>
__global__ void k_sample_points(KCtx c, long long n, const double* __restrict__ xyz, double* out) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double x[3] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
  R phi, nn[3], curv;
  ls_sample<D, R>(c.ls, x, phi, nn, curv);
  out[6 * i + 0] = phi;
  out[6 * i + 1] = nn[0];
  out[6 * i + 2] = nn[1];
  out[6 * i + 3] = nn[2];
  out[6 * i + 4] = curv;
  out[6 * i + 5] = (double)ls_tag<D, R>(c.ls, x);
}

// the same into separate arrays
template <int D, class R>
__global__ void k_sample_arrays(KCtx c, long long n, const double* __restrict__ xyz, double* __restrict__ phi,
                                double* __restrict__ norm, double* __restrict__ curv, int* __restrict__ tag) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x[3] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
  R ph, nn[3], cv;
  ls_sample<D, R>(c.ls, x, ph, nn, cv);
  phi[i] = ph;
  norm[3 * i] = nn[0];
  norm[3 * i + 1] = nn[1];
  norm[3 * i + 2] = nn[2];
  curv[i] = cv;
  tag[i] = ls_tag<D, R>(c.ls, x);
}

// ---------------------------------------------------------------------------
// host engine
// ---------------------------------------------------------------------------
#define MR_CK(call)                                                                     \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) {                                                            \
      err = std::string(#call) + ": " + cudaGetErrorString(e_);                         \
      return MRSPH_ERR_CUDA;                                                            \
    }                                                                                   \
  } while (0)

template <int D, class R>
class Engine : public EngineBase {
  using T4 = typename V4<R>::T;

 public:
  explicit Engine(const EngineConfig& cfg) : cfg_(cfg) {
    kc_.prm = cfg.prm;
    kc_.geo = cfg.geo;
    kc_.ls = cfg.ls;
    kc_.n = 0;
    kc_.sc = nullptr;
    st_ = cfg.stream;
    // FP32 copies of the run parameters, read by the FP32-split kernels
    kc_.prm.cell_ratio_f = (float)kc_.prm.cell_ratio;
    kc_.prm.cutoff_f = (float)kc_.prm.cutoff;
    kc_.prm.cos_thres_f = (float)kc_.prm.cos_thres;
    kc_.prm.nu_coeff_f = (float)kc_.prm.nu_coeff;
    kc_.prm.damp_coeff_f = (float)kc_.prm.damp_coeff;
    kc_.ls.max_phi_f = (float)kc_.ls.max_phi;
    kc_.ls.dl0_f = (float)kc_.ls.dl0;
    kc_.ls.min_dl_f = (float)kc_.ls.min_dl;
    kc_.ls.max_dl_f = (float)kc_.ls.max_dl;
    kc_.ls.middle_dl_f = (float)kc_.ls.middle_dl;
    kc_.ls.max_curv_f = (float)kc_.ls.max_curv;
    kc_.ls.min_curv_f = (float)kc_.ls.min_curv;
    kc_.geo.max_scale_f = (float)kc_.geo.max_scale;
    kc_.geo.ext_f = 0.f;
    for (int d = 0; d < D; d++) kc_.geo.ext_f = std::max(kc_.geo.ext_f, (float)(cfg.prm.box_r[d] - cfg.prm.box_l[d]));
    if (std::is_same<R, float>::value) init_rc_ = anchor_tables();
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev);
    cudaGetLastError();
    if (sms_ < 1) sms_ = 1;
  }
  ~Engine() override {
    release();
    for (void* p : anc_allocs_) cudaFree(p);
  }

  int seed(long long n) override {
    int rc = alloc(n);
    if (rc) return rc;
    MR_CK(cudaMemsetAsync(kc_.sc, 0, sizeof(DevScalars), st_));
    k_seed<D, R><<<grid(n), 256, 0, st_>>>(kc_, buf_[cur_], 1000000u);
    MR_CK(cudaGetLastError());
    return pre_run();
  }

  int set_state(long long n, const mrsph_state_in* s, int pre) override {
    int rc = alloc(n);
    if (rc) return rc;
    std::vector<double> host((size_t)10 * n, 0.0);
    for (long long i = 0; i < 3 * n; i++) host[i] = s->xyz[i];
    if (s->v) for (long long i = 0; i < 3 * n; i++) host[3 * n + i] = s->v[i];
    if (s->nu) for (long long i = 0; i < n; i++) host[6 * n + i] = s->nu[i];
    if (s->h) for (long long i = 0; i < n; i++) host[9 * n + i] = s->h[i];
    double* dbuf = nullptr;
    int* dint = nullptr;
    MR_CK(cudaMalloc(&dbuf, sizeof(double) * 10 * n));
    MR_CK(cudaMalloc(&dint, sizeof(int) * 2 * n));
    MR_CK(cudaMemcpyAsync(dbuf, host.data(), sizeof(double) * 10 * n, cudaMemcpyHostToDevice, st_));
    if (s->type) MR_CK(cudaMemcpyAsync(dint, s->type, sizeof(int) * n, cudaMemcpyHostToDevice, st_));
    if (s->level) MR_CK(cudaMemcpyAsync(dint + n, s->level, sizeof(int) * n, cudaMemcpyHostToDevice, st_));
    MR_CK(cudaMemsetAsync(kc_.sc, 0, sizeof(DevScalars), st_));
    k_set_state<D, R><<<grid(n), 256, 0, st_>>>(kc_, buf_[cur_], dbuf, s->v != nullptr, s->h != nullptr,
                                                 s->nu != nullptr, s->level != nullptr,
                                                 s->type ? dint : nullptr, dint + n);
    MR_CK(cudaGetLastError());
    DevScalars h{};
    h.dt2 = dbits_host(s->dt);
    h.step = (unsigned)s->step;
    MR_CK(cudaMemcpyAsync(kc_.sc, &h, sizeof(h), cudaMemcpyHostToDevice, st_));
    k_iota<<<grid(n), 256, 0, st_>>>(w_.slot_of_id, n);
    MR_CK(cudaStreamSynchronize(st_));
    cudaFree(dbuf);
    cudaFree(dint);
    have_work_ = false;
    if (pre) return pre_run();
    return 0;  // state stays in id order (slot_of_id = identity) until the next step
  }

  int run_phase(int phase) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    int rc = launch_step(phase);
    if (rc) return rc;
    MR_CK(cudaStreamSynchronize(st_));
    MR_CK(cudaGetLastError());
    return 0;
  }

  // Graph replay.  The neighbour-list capacity follows the largest list
  // seen: every 32 steps the device max count is read and the list grown,
  // within a memory budget; particles whose list does not fit are handled by
  // re-scanning their cells in the force kernels.  A state's first step is
  // launched kernel by kernel and settles the capacity before the forces: the
  // re-scan of every particle of a freshly seeded body took longer than the rest
  // of the step, and the step graphs were built twice.
  int step(int nsteps) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    if (nsteps <= 0) return 0;
    for (int k = 0; k < nsteps; k++) {
      if (countdown_ <= 0) {  // the first step of a state
        int rc = launch_step(MRSPH_PHASE_FORCE2, nullptr, true);
        if (rc) return rc;
        countdown_ = 32;
        continue;
      }
      int rc = build_graphs();
      if (rc) return rc;
      MR_CK(cudaGraphLaunch(graphs_[0][cur_], st_));
      cur_ ^= 1;
      have_work_ = true;
      if (--countdown_ <= 0) {
        rc = maybe_grow_cap();
        if (rc) return rc;
        countdown_ = 32;
      }
    }
    return 0;
  }

  // Reads the largest neighbour count of the last step and grows the list
  // capacity (graphs are rebuilt).  Stays with the re-scan fallback when the
  // allocation fails or exceeds the budget (half of the device memory free
  // beside the current lists, at least 48 GB), or when the caller fixed the
  // cap; a growth that falls short raises MRSPH_FLAG_CAPACITY_CLAMPED in the
  // next stats.
  // The form of the passes follows the mean row length seen here.
  // settle: no force has read the lists yet, so those that spill into a larger
  // capacity were no spills.
  int maybe_grow_cap(bool settle = false) {
    DevScalars h;
    MR_CK(cudaMemcpyAsync(&h, kc_.sc, sizeof(h), cudaMemcpyDeviceToHost, st_));
    MR_CK(cudaStreamSynchronize(st_));
    dense_ = (long long)h.pairs > kDenseRow * n_;
    const Forms f = choose_forms(n_, n_);
    if (!(f == alone_)) {
      drop_graphs(0);
      alone_ = forms_ = f;
    }
    const unsigned mc = h.maxcnt;
    if ((int)mc <= w_.cap || cfg_.neighbor_cap > 0) return 0;
    long long want = ((long long)mc * 5 / 4 + 31) / 32 * 32;
    const long long n32 = (n_ + 31) / 32 * 32;  // nb_slot blocks of 32 particles
    const long long per_entry = (long long)(sizeof(int) + sizeof(R)) * n32;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
      cudaGetLastError();
      free_b = 0;
    }
    // the current lists are freed only once the new ones are in place, so the
    // new ones must fit beside them
    const long long avail = (long long)free_b + per_entry * w_.cap;
    const long long budget = std::max(48ll << 30, std::min(avail / 2, (long long)free_b));  // lists + pair coefficients
    long long maxcap = budget / per_entry / 8 * 8;
    if (want > maxcap) {
      want = maxcap;
      cap_clamped_ = true;
    }
    if (want <= w_.cap) return 0;
    int* nb = nullptr;
    R* pc = nullptr;
    cudaError_t e = cudaMalloc(&nb, sizeof(int) * (size_t)want * n32);
    if (e == cudaSuccess) {
      e = cudaMalloc(&pc, sizeof(R) * (size_t)want * n32);
      if (e != cudaSuccess) cudaFree(nb);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      cap_clamped_ = true;
      return 0;
    }
    for (auto& p : allocs_) {
      if (p == w_.nbl) { cudaFree(p); p = nb; }
      else if (p == w_.pc) { cudaFree(p); p = pc; }
    }
    w_.nbl = nb;
    w_.pc = pc;
    w_.cap = (int)want;
    drop_graphs();
    // the lists of the state they belong to, now whole: whoever reads them next
    // (taps, meshes) finds them in the new arrays
    MR_CK(cudaMemsetAsync(&kc_.sc->pairs, 0, sizeof(kc_.sc->pairs), st_));
    MR_CK(cudaMemsetAsync(&kc_.sc->nspill, 0, sizeof(kc_.sc->nspill), st_));
    if (settle) MR_CK(cudaMemcpyAsync(&kc_.sc->flags, &kc_.sc->flags0, sizeof(unsigned), cudaMemcpyDeviceToDevice, st_));
    launch_lists();
    MR_CK(cudaGetLastError());
    MR_CK(cudaStreamSynchronize(st_));  // a batch steps the handle on another stream
    return 0;
  }

  // The step graphs: those of the handle's steps alone, or (set 1) those of its
  // steps beside other handles' with forms of their own.
  int build_graphs(int set = 0) {
    cudaGraphExec_t* const graph_ = graphs_[set];
    for (int p = 0; p < 2; p++) {
      if (!graph_[p]) {
        int saved = cur_;
        cur_ = p;
        MR_CK(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
        forms_ = set ? beside_ : alone_;
        int rc = launch_step(MRSPH_PHASE_FORCE2);
        forms_ = alone_;
        cudaGraph_t g;
        cudaError_t ee = cudaStreamEndCapture(st_, &g);
        cur_ = saved;
        if (rc) return rc;
        if (ee != cudaSuccess) { err = cudaGetErrorString(ee); return MRSPH_ERR_CUDA; }
        cudaError_t ie = cudaGraphInstantiate(&graph_[p], g, 0);
        cudaGraphDestroy(g);
        if (ie != cudaSuccess) { graph_[p] = nullptr; err = cudaGetErrorString(ie); return MRSPH_ERR_CUDA; }
        MR_CK(cudaGraphUpload(graph_[p], st_));  // upload now, not at the first (timed) launch
      }
    }
    return 0;
  }

  void drop_graphs() {
    drop_graphs(0);
    drop_graphs(1);
  }
  void drop_graphs(int set) {
    for (int p = 0; p < 2; p++) {
      cudaGraphExec_t& g = graphs_[set][p];
      if (g) { cudaGraphExecDestroy(g); g = nullptr; }
    }
  }

  // One step of a batch: the step graph of the current parity launched on the
  // handle's stream, without the periodic capacity check (the batch makes it).
  // total: the particles of all handles that step at the same time.
  int step_batched(long long total) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    const int set = graph_set(total);
    int rc = build_graphs(set);
    if (rc) return rc;
    MR_CK(cudaGraphLaunch(graphs_[set][cur_], st_));
    cur_ ^= 1;
    have_work_ = true;
    return 0;
  }

  int prepare_steps(long long total) override { return n_ ? build_graphs(graph_set(total)) : 0; }

  int check_capacity() override { return have_work_ ? maybe_grow_cap() : 0; }

  int stats(mrsph_stats* o) override {
    DevScalars h;
    MR_CK(cudaMemcpyAsync(&h, kc_.sc, sizeof(h), cudaMemcpyDeviceToHost, st_));
    MR_CK(cudaStreamSynchronize(st_));
    // cleared on the engine stream, ordered before the next step's kernels
    MR_CK(cudaMemsetAsync(&kc_.sc->flags, 0, sizeof(unsigned), st_));
    o->dt = bitsd_host(h.dt2);
    o->dt_stage1 = bitsd_host(h.dt1);
    o->max_v = bitsd_host(h.vmax2);
    o->step = h.step;
    o->n = n_;
    o->n_surface = h.nsurf;
    o->pairs = (long long)h.pairs;
    o->pairs_total = (long long)h.pairs_total;
    o->remapped = h.remap;
    o->flags = (int)h.flags | (cap_clamped_ ? MRSPH_FLAG_CAPACITY_CLAMPED : 0);
    cap_clamped_ = false;
    o->num_cell_levels = kc_.geo.ncl;
    o->num_cells = kc_.geo.hoff[kc_.geo.ncl];
    o->max_phi = kc_.ls.max_phi;
    return 0;
  }

  int get_particles(const mrsph_particle_view* v) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    struct F { void* p; int field; int vec; bool isint; };
    F fs[] = {{v->xyz, 0, 1, false}, {v->v, 1, 1, false}, {v->norm, 2, 1, false}, {v->a1, 3, 1, false},
              {v->a2, 4, 1, false}, {v->h, 5, 0, false}, {v->phi, 6, 0, false}, {v->curv, 7, 0, false},
              {v->sum, 8, 0, false}, {v->rho, 9, 0, false}, {v->nu, 10, 0, false}, {v->type, 11, 0, true},
              {v->level, 12, 0, true}};
    std::vector<double> host((size_t)3 * n_);
    for (auto& f : fs) {
      if (!f.p) continue;
      k_tap<D, R><<<grid(n_), 256, 0, st_>>>(kc_, buf_[cur_], w_, w_.slot_of_id, stage_, f.field, have_work_);
      MR_CK(cudaGetLastError());
      size_t cnt = (size_t)(f.vec ? 3 : 1) * n_;
      MR_CK(cudaMemcpyAsync(host.data(), stage_, sizeof(double) * cnt, cudaMemcpyDeviceToHost, st_));
      MR_CK(cudaStreamSynchronize(st_));
      if (f.isint) {
        int* o = (int*)f.p;
        for (size_t k = 0; k < cnt; k++) o[k] = (int)host[k];
      } else {
        std::memcpy(f.p, host.data(), sizeof(double) * cnt);
      }
    }
    return 0;
  }

  int get_cells(int* level_cell, int* sorted_ids) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    std::vector<int> ck(n_), ids(n_);
    MR_CK(cudaMemcpyAsync(ck.data(), buf_[cur_].cellkey, sizeof(int) * n_, cudaMemcpyDeviceToHost, st_));
    MR_CK(cudaMemcpyAsync(ids.data(), buf_[cur_].id, sizeof(int) * n_, cudaMemcpyDeviceToHost, st_));
    MR_CK(cudaStreamSynchronize(st_));
    if (sorted_ids) std::memcpy(sorted_ids, ids.data(), sizeof(int) * n_);
    if (level_cell) {
      for (long long s = 0; s < n_; s++) {
        long long key = ck[s];
        int L = 0;
        while (L + 1 < kc_.geo.ncl && key >= kc_.geo.hoff[L + 1]) L++;
        long long r = key - kc_.geo.hoff[L];  // half cell -> reference cell
        int cx = (int)(r % kc_.geo.hn[L][0]) >> 1;
        r /= kc_.geo.hn[L][0];
        int cy = (int)(r % kc_.geo.hn[L][1]) >> 1;
        int cz = (int)(r / kc_.geo.hn[L][1]) >> 1;
        int* o = level_cell + 4 * (long long)ids[s];
        o[0] = L; o[1] = cx; o[2] = cy; o[3] = cz;
      }
    }
    return 0;
  }

  int get_neighbors(long long* off, int* nb, long long cap, long long* total) override {
    if (!have_work_) { err = "no density phase has run"; return MRSPH_ERR_STATE; }
    std::vector<int> cnt(n_), ids(n_);
    MR_CK(cudaMemcpyAsync(cnt.data(), w_.cnt, sizeof(int) * n_, cudaMemcpyDeviceToHost, st_));
    MR_CK(cudaMemcpyAsync(ids.data(), buf_[cur_].id, sizeof(int) * n_, cudaMemcpyDeviceToHost, st_));
    MR_CK(cudaStreamSynchronize(st_));
    long long tot = 0;
    std::vector<long long> byid_cnt(n_);
    for (long long s = 0; s < n_; s++) {
      if (cnt[s] > w_.cap) { err = "neighbour list spilled; raise neighbor_cap"; return MRSPH_ERR_RANGE; }
      byid_cnt[ids[s]] = cnt[s];
      tot += cnt[s];
    }
    if (total) *total = tot;
    if (!nb) return 0;
    if (cap < tot || !off) { err = "neighbour buffer too small"; return MRSPH_ERR_ARG; }
    const size_t nbl_len = (size_t)w_.cap * ((n_ + 31) / 32 * 32);
    std::vector<int> nbl(nbl_len);
    MR_CK(cudaMemcpy(nbl.data(), w_.nbl, sizeof(int) * nbl_len, cudaMemcpyDeviceToHost));
    off[0] = 0;
    for (long long k = 0; k < n_; k++) off[k + 1] = off[k] + byid_cnt[k];
    for (long long s = 0; s < n_; s++) {
      long long base = off[ids[s]];
      for (int q = 0; q < cnt[s]; q++) nb[base + q] = ids[nbl[nb_slot(s, q, w_.cap)]];
      std::sort(nb + base, nb + base + cnt[s]);
    }
    return 0;
  }

  int upload_positions(const double* xyz) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    MR_CK(cudaMemcpyAsync(stage_, xyz, sizeof(double) * 3 * n_, cudaMemcpyHostToDevice, st_));
    k_upload<D, R><<<grid(n_), 256, 0, st_>>>(kc_, buf_[cur_], stage_);
    MR_CK(cudaGetLastError());
    return 0;
  }

  int download_positions(double* xyz) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    k_tap<D, R><<<grid(n_), 256, 0, st_>>>(kc_, buf_[cur_], w_, w_.slot_of_id, stage_, 0, have_work_);
    MR_CK(cudaGetLastError());
    MR_CK(cudaMemcpyAsync(xyz, stage_, sizeof(double) * 3 * n_, cudaMemcpyDeviceToHost, st_));
    MR_CK(cudaStreamSynchronize(st_));
    return 0;
  }

  int sample(long long n, const double* xyz, double* phi, double* norm, double* curv, int* tag) override {
    // xyz, then the results as the caller's arrays want them: phi, normals, curvature, tags
    double* d = nullptr;
    MR_CK(cudaMalloc(&d, (sizeof(double) * 8 + sizeof(int)) * n));
    double *dphi = d + 3 * n, *dnorm = d + 4 * n, *dcurv = d + 7 * n;
    int* dtag = reinterpret_cast<int*>(d + 8 * n);
    cudaError_t e = cudaMemcpyAsync(d, xyz, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, st_);
    if (e == cudaSuccess) {
      k_sample_arrays<D, R><<<grid(n), 256, 0, st_>>>(kc_, n, d, dphi, dnorm, dcurv, dtag);
      e = cudaGetLastError();
    }
    // up to some 6,000 points through one host buffer: a copy takes 8 us whatever its size
    const size_t all = (sizeof(double) * 5 + sizeof(int)) * n;
    std::vector<char> host(all <= (256 << 10) ? all : 0);
    auto out = [&](void* to, const void* from, size_t bytes) {
      if (!to || e != cudaSuccess) return;
      if (host.empty()) e = copy_home(to, from, bytes, st_);
      else std::memcpy(to, host.data() + ((const char*)from - (const char*)dphi), bytes);
    };
    if (!host.empty() && e == cudaSuccess) {
      e = cudaMemcpyAsync(host.data(), dphi, all, cudaMemcpyDeviceToHost, st_);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
    }
    out(phi, dphi, sizeof(double) * n);
    out(norm, dnorm, sizeof(double) * 3 * n);
    out(curv, dcurv, sizeof(double) * n);
    out(tag, dtag, sizeof(int) * n);
    if (host.empty() && e == cudaSuccess) e = cudaStreamSynchronize(st_);
    cudaFree(d);
    if (e != cudaSuccess) { err = cudaGetErrorString(e); return MRSPH_ERR_CUDA; }
    return 0;
  }

  int sample_device(long long n, const double* d_xyz, double* d_out) override {
    k_sample_points<D, R><<<grid(n), 256, 0, st_>>>(kc_, n, d_xyz, d_out);
    MR_CK(cudaGetLastError());
    return 0;
  }

  cudaStream_t stream() const override { return st_; }
  long long num_particles() const override { return n_; }

  int world_positions(double* d_out) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    k_tap<D, R><<<grid(n_), 256, 0, st_>>>(kc_, buf_[cur_], w_, w_.slot_of_id, d_out, 0, have_work_);
    MR_CK(cudaGetLastError());
    return 0;
  }

  int export_tri(double* d_xyz, int* d_type, double* d_phi, int* d_rows, int* d_cnt, int rowcap,
                 unsigned* d_flags, double* d_h = nullptr, bool sort_rows = true) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    if (!have_work_) { err = "no density phase has run"; return MRSPH_ERR_STATE; }
    k_export_tri<D, R><<<grid(n_), 256, 0, st_>>>(kc_, buf_[cur_], w_, d_xyz, d_type, d_phi, d_rows, d_cnt, rowcap,
                                                   d_flags, d_h, sort_rows);
    MR_CK(cudaGetLastError());
    return 0;
  }

  int neighbor_capacity() const override { return w_.cap; }

  // The batch kernels' view of this handle (FP32-split only).
  int batch_slot(BatchSlot* out) override {
    if (!std::is_same<R, float>::value) { err = "batched kernels take FP32-split handles"; return MRSPH_ERR_ARG; }
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    BatchSlot s{};
    s.c = kc_;
    std::memcpy((void*)&s.buf[0], (const void*)&buf_[0], sizeof(Buf<float>));
    std::memcpy((void*)&s.buf[1], (const void*)&buf_[1], sizeof(Buf<float>));
    std::memcpy((void*)&s.w, (const void*)&w_, sizeof(Work<float>));
    s.w.bcount = s.w.bstart = s.w.order = nullptr;  // the batch's phases do not make the work order
    s.ncells = ncells_;
    s.dim = D;
    s.cur = cur_;
    *out = s;
    return 0;
  }
  // nsteps whole steps ran on this handle's state in a batch launch
  void batch_advance(int nsteps) override {
    cur_ ^= (nsteps & 1);
    have_work_ = true;
  }

 private:
  static unsigned long long dbits_host(double x) { unsigned long long u; std::memcpy(&u, &x, 8); return u; }
  static double bitsd_host(unsigned long long u) { double x; std::memcpy(&x, &u, 8); return x; }
  static int grid(long long n) { return (int)((n + 255) / 256); }
  // grid of the spilled force stages: the queue's length is known on the
  // device only; two blocks per SM at most
  int qgrid() const { return std::max(1, std::min(grid(n_), 2 * sms_)); }

  int pre_run() {
    begin_step(0);
    int rc = run_map_and_bin(MAP_PRE);
    if (rc) return rc;
    // Pre_run (sph_mesh_generation.cpp:1010-1050) leaves v = 0 (Reset_particle_force)
    // and nu = 0 (Set_timestep(2) at v = 0), so the first step's
    // Update_coord_full_step moves nothing; the advection step is set to 0
    Buf<R>& b = buf_[cur_];
    MR_CK(cudaMemsetAsync(b.v1, 0, sizeof(T4) * n_, st_));
    MR_CK(cudaMemsetAsync(b.a2, 0, sizeof(T4) * n_, st_));
    MR_CK(cudaMemsetAsync(b.nu, 0, sizeof(R) * n_, st_));
    MR_CK(cudaMemsetAsync(b.nu_next, 0, sizeof(R) * n_, st_));
    MR_CK(cudaMemsetAsync(&kc_.sc->dt2, 0, sizeof(unsigned long long), st_));
    MR_CK(cudaStreamSynchronize(st_));
    have_work_ = false;
    return 0;
  }

  // map (mode) + counting sort + reorder; swaps cur_.
  int run_map_and_bin(int mode) {
    const long long n = n_;
    launch_chained(k_map<D, R>, grid(n), 256, st_, kc_, buf_[cur_], w_.counts, w_.lhmax, mode, 1000000u);
    MR_CK(cudaGetLastError());
    return bin(1);
  }

  void begin_step(int inc) {
    const long long nl = kc_.geo.nc0 * kc_.geo.ncl;
    launch_chained(k_begin_step, grid(nl), 256, st_, kc_.sc, inc, w_.lhmax, nl);
  }

  int bin(int partial) {
    const long long n = n_;
    cell_scan(w_.counts, w_.cstart, w_.blocksums, ncells_, (int)n, st_);
    cell_scatter(buf_[cur_].cellkey, buf_[cur_].id, w_.counts, w_.cstart, w_.perm, w_.pid, n, st_);
    launch_chained(k_reorder<D, R>, grid(n), 256, st_, buf_[cur_], buf_[cur_ ^ 1], kc_, w_, partial);
    MR_CK(cudaGetLastError());
    cur_ ^= 1;
    return 0;
  }

  Forms choose_forms(long long n, long long total) const {
    return mrsph::choose_forms(D, std::is_same<R, float>::value, kc_.geo.ncl, dense_, n, total);
  }
  // the graphs that a step beside handles of total particles takes
  // (half of their number: two handles of 23,000 take 739 us by the forms of 23,000
  // particles, 827 by those of 46,000)
  int graph_set(long long total) {
    const Forms f = choose_forms(n_, std::max(n_, total / 2));
    if (f == alone_) return 0;
    if (!(f == beside_) && graphs_[1][0]) {
      cudaStreamSynchronize(st_);
      drop_graphs(1);
    }
    beside_ = f;
    return 1;
  }

  int ggrid(int threads) const { return (int)((n_ + threads / kG - 1) / (threads / kG)); }  // kG lanes per particle

  void launch_lists() {
    if constexpr (std::is_same<R, float>::value) {
      const unsigned blocks = (unsigned)((n_ + kDensityThreads - 1) / kDensityThreads);
      if (forms_.list == LIST_LANE) {
        launch_chained(k_density_lane<D>, blocks, kDensityThreads, st_, kc_, buf_[cur_], w_);
        return;
      }
      if constexpr (D == 3) {
        if (forms_.list == LIST_TILE || forms_.list == LIST_BRICK) {
          Work<R> w = w_;
          if (forms_.list == LIST_BRICK) {
            const long long nb = kc_.geo.boff[kc_.geo.ncl];
            int per = 1;  // bricks per warp: 64 warps per SM or more
            while (per < 32 && nb > 64ll * sms_ * 2 * per) per *= 2;
            launch_chained(k_brick_count<D>, grid(nb), 256, st_, kc_, w_.cstart, w_.bcount);
            cell_scan(w_.bcount, w_.bstart, w_.blocksums, nb, (int)n_, st_);
            launch_chained(k_brick_order<D>, grid((nb + per - 1) / per * 32), 256, st_, kc_, w_.cstart, w_.bcount, w_.bstart,
                           w_.order, per);
          } else {
            w.order = w.bstart = nullptr;
          }
          launch_chained(k_density_tile<D>, blocks, kDensityThreads, st_, kc_, buf_[cur_], w);
          return;
        }
      }
    }
    launch_chained(k_density_group<D, R>, ggrid(kDensityThreads), kDensityThreads, st_, kc_, buf_[cur_], w_);
  }

  template <int STAGE, int KK>
  void launch_force_kind() {
    if (forms_.force_group) launch_chained(k_force_group<D, R, STAGE, KK>, ggrid(kGroupThreads), kGroupThreads, st_, kc_, buf_[cur_], w_);
    else launch_chained(k_force<D, R, STAGE, KK>, grid(n_), 256, st_, kc_, buf_[cur_], w_);
    launch_chained(k_force_spill<D, R, STAGE, KK>, qgrid(), kGroupThreads, st_, kc_, buf_[cur_], w_);
  }
  template <int STAGE>
  void launch_force() {
    if (kc_.prm.kernel == K_WEN) launch_force_kind<STAGE, (sizeof(R) == 4 ? K_WEN : -1)>();
    else launch_force_kind<STAGE, -1>();
  }

  // ev (optional, 8 events) brackets the timer phases MRSPH_TIMER_*.
  // settle: the list capacity is made to fit between the lists and the forces
  // (synchronises).
  int launch_step(int phase, cudaEvent_t* ev = nullptr, bool settle = false) {
    const long long n = n_;
    auto mark = [&](int k) { if (ev) cudaEventRecord(ev[k], st_); };
    mark(0);
    begin_step(1);
    launch_chained(k_map<D, R>, grid(n), 256, st_, kc_, buf_[cur_], w_.counts, w_.lhmax, (int)MAP_STEP, 1000000u);
    MR_CK(cudaGetLastError());
    mark(1);
    if (phase < MRSPH_PHASE_BIN) {  // the histogram is not consumed by a scatter: clear it
      MR_CK(cudaMemsetAsync(w_.counts, 0, sizeof(int) * ncells_, st_));
      return 0;
    }
    cell_scan(w_.counts, w_.cstart, w_.blocksums, ncells_, (int)n, st_);
    mark(2);
    cell_scatter(buf_[cur_].cellkey, buf_[cur_].id, w_.counts, w_.cstart, w_.perm, w_.pid, n, st_);
    mark(3);
    launch_chained(k_reorder<D, R>, grid(n), 256, st_, buf_[cur_], buf_[cur_ ^ 1], kc_, w_, phase < MRSPH_PHASE_FORCE2 ? 1 : 0);
    MR_CK(cudaGetLastError());
    cur_ ^= 1;
    mark(4);
    if (phase < MRSPH_PHASE_DENSITY) return 0;
    if (settle) MR_CK(cudaMemcpyAsync(&kc_.sc->flags0, &kc_.sc->flags, sizeof(unsigned), cudaMemcpyDeviceToDevice, st_));
    launch_lists();
    if (settle) {
      int rc = maybe_grow_cap(true);
      if (rc) return rc;
    }
    have_work_ = true;
    mark(5);
    if (phase < MRSPH_PHASE_FORCE1) {
      launch_force<0>();
      return 0;
    }
    launch_force<1>();
    mark(6);
    if (phase < MRSPH_PHASE_FORCE2) return 0;
    launch_force<2>();
    mark(7);
    MR_CK(cudaGetLastError());
    return 0;
  }

 public:
  int step_timed(int nsteps, double* ms) override {
    cudaEvent_t a, b;
    MR_CK(cudaEventCreate(&a));
    MR_CK(cudaEventCreate(&b));
    int rc = 0;
    if (have_work_) rc = maybe_grow_cap();  // settle the list capacity first
    if (!rc) rc = build_graphs();            // instantiate outside the timed region
    if (rc) return rc;
    const int saved = countdown_;
    countdown_ = 1 << 30;                    // no capacity checks while timing
    MR_CK(cudaEventRecord(a, st_));
    rc = step(nsteps);
    MR_CK(cudaEventRecord(b, st_));
    countdown_ = saved;
    MR_CK(cudaEventSynchronize(b));
    float f = 0.f;
    MR_CK(cudaEventElapsedTime(&f, a, b));
    *ms = f;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    return rc;
  }

  int profile_steps(int nsteps, double* phase_ms, int nphase) override {
    if (!n_) { err = "no particles"; return MRSPH_ERR_STATE; }
    cudaEvent_t ev[8];
    for (int k = 0; k < 8; k++) MR_CK(cudaEventCreate(&ev[k]));
    double acc[8] = {0};
    for (int s = 0; s < nsteps; s++) {
      int rc = launch_step(MRSPH_PHASE_FORCE2, ev);
      if (rc) return rc;
      MR_CK(cudaEventSynchronize(ev[7]));
      for (int k = 0; k < 7; k++) {
        float f = 0.f;
        MR_CK(cudaEventElapsedTime(&f, ev[k], ev[k + 1]));
        acc[k] += f;
      }
    }
    for (int k = 0; k < nphase && k < 7; k++) phase_ms[k] = acc[k] / (nsteps > 0 ? nsteps : 1);
    for (int k = 0; k < 8; k++) cudaEventDestroy(ev[k]);
    return 0;
  }

 private:

  // FP32-split level-set location: per level-set level and axis, the
  // package of each anchor cell's lower corner and the corner's FP32 offset
  // inside it (computed here in FP64, once per level set)
  int anchor_tables() {
    const int lm = kc_.geo.ncl - 1;
    for (int l = 0; l < kc_.ls.nls; l++) {
      LsLevel& L = kc_.ls.lv[l];
      for (int d = 0; d < 3; d++) {
        L.anc[d] = nullptr;
        L.dpkg_f[d] = (float)L.dpkg[d];
        L.inv_dpkg_f[d] = (float)L.inv_dpkg[d];
        L.inv_dcell_f[d] = (float)L.inv_dcell[d];
        if (d >= D) continue;
        const int na = kc_.geo.n[lm][d];
        std::vector<int2> t(na);
        for (int k = 0; k < na; k++) {
          const double base = (kc_.geo.box_l[d] - L.box_l[d]) + (double)k * kc_.geo.A[d];
          const double p0 = std::floor(base / L.dpkg[d]);
          const float rem = (float)(base - p0 * L.dpkg[d]);
          t[k].x = (int)p0;
          std::memcpy(&t[k].y, &rem, sizeof(float));
        }
        int2* dv = nullptr;
        if (cudaMalloc(&dv, sizeof(int2) * na) != cudaSuccess) {
          err = "cudaMalloc failed (anchor tables)";
          return MRSPH_ERR_OOM;
        }
        anc_allocs_.push_back(dv);
        // on the engine stream (the kernels that read the table run there) and
        // complete before the host vector goes out of scope
        if (cudaMemcpyAsync(dv, t.data(), sizeof(int2) * na, cudaMemcpyHostToDevice, st_) != cudaSuccess ||
            cudaStreamSynchronize(st_) != cudaSuccess) {
          err = "cudaMemcpy failed (anchor tables)";
          return MRSPH_ERR_CUDA;
        }
        L.anc[d] = dv;
      }
    }
    return 0;
  }

  int alloc(long long n) {
    if (init_rc_) return init_rc_;
    if (n <= 0 || n > (1ll << 30)) { err = "particle count out of range"; return MRSPH_ERR_RANGE; }
    release();
    n_ = n;
    kc_.n = n;
    ncells_ = kc_.geo.hoff[kc_.geo.ncl];
    int cap = cfg_.neighbor_cap > 0 ? (cfg_.neighbor_cap + 7) / 8 * 8 : (D == 2 ? 64 : 192);
    w_.cap = cap;
    auto A = [&](void** p, size_t bytes) -> int {
      cudaError_t e = cudaMalloc(p, bytes);
      if (e != cudaSuccess) { err = std::string("cudaMalloc: ") + cudaGetErrorString(e); return MRSPH_ERR_OOM; }
      allocs_.push_back(*p);
      return 0;
    };
    int rc = 0;
    for (int k = 0; k < 2 && !rc; k++) {
      Buf<R>& b = buf_[k];
      rc |= A((void**)&b.posh, sizeof(T4) * n);
      rc |= A((void**)&b.nr, sizeof(T4) * n);
      rc |= A((void**)&b.v1, sizeof(T4) * n);
      rc |= A((void**)&b.a2, sizeof(T4) * n);
      if (sizeof(R) == 4) rc |= A((void**)&b.key, sizeof(int) * n); else b.key = nullptr;
      rc |= A((void**)&b.meta, sizeof(int) * n);
      rc |= A((void**)&b.id, sizeof(int) * n);
      rc |= A((void**)&b.nu, sizeof(R) * n);
      rc |= A((void**)&b.nu_next, sizeof(R) * n);
      rc |= A((void**)&b.phi, sizeof(R) * n);
      rc |= A((void**)&b.curv, sizeof(R) * n);
      rc |= A((void**)&b.cellkey, sizeof(int) * n);
      rc |= A((void**)&b.rec, sizeof(T4) * 2 * n);
    }
    if (!rc) {
      rc |= A((void**)&w_.sum, sizeof(R) * n);
      rc |= A((void**)&w_.a1, sizeof(T4) * n);
      rc |= A((void**)&w_.cnt, sizeof(int) * n);
      rc |= A((void**)&w_.nbl, sizeof(int) * (size_t)cap * ((n + 31) / 32 * 32));
      rc |= A((void**)&w_.pc, sizeof(R) * (size_t)cap * ((n + 31) / 32 * 32));
      rc |= A((void**)&w_.counts, sizeof(int) * ncells_);
      rc |= A((void**)&w_.lhmax, sizeof(unsigned) * kc_.geo.nc0 * kc_.geo.ncl);
      rc |= A((void**)&w_.rlev, sizeof(float) * kc_.geo.ncl * n);
      rc |= A((void**)&w_.cstart, sizeof(int) * (ncells_ + 1));
      rc |= A((void**)&w_.perm, sizeof(int) * n);
      rc |= A((void**)&w_.pid, sizeof(int) * n);
      rc |= A((void**)&w_.blocksums, sizeof(int) * scan_blocksums_size(ncells_));
      rc |= A((void**)&w_.slot_of_id, sizeof(int) * n);
      rc |= A((void**)&w_.spillq, sizeof(int) * n);
      rc |= A((void**)&stage_, sizeof(double) * 3 * n);
      rc |= A((void**)&kc_.sc, sizeof(DevScalars));
    }
    w_.bcount = w_.bstart = w_.order = nullptr;
    dense_ = false;
    forms_ = alone_ = choose_forms(n, n);
    if (!rc && alone_.list == LIST_BRICK) {
      const long long nb = kc_.geo.boff[kc_.geo.ncl];
      rc |= A((void**)&w_.bcount, sizeof(int) * nb);
      rc |= A((void**)&w_.bstart, sizeof(int) * (nb + 1));
      rc |= A((void**)&w_.order, sizeof(int) * n);
    }
    if (rc) { release(); return rc; }
    MR_CK(cudaMemsetAsync(w_.counts, 0, sizeof(int) * ncells_, st_));
    MR_CK(cudaMemsetAsync(w_.cnt, 0, sizeof(int) * n, st_));
    MR_CK(cudaMemsetAsync(kc_.sc, 0, sizeof(DevScalars), st_));
    cur_ = 0;
    countdown_ = 0;
    return 0;
  }

  void release() {
    drop_graphs();
    for (void* p : allocs_) cudaFree(p);
    allocs_.clear();
    n_ = 0;
    kc_.n = 0;
    kc_.sc = nullptr;
    stage_ = nullptr;
  }

  EngineConfig cfg_;
  KCtx kc_;
  cudaStream_t st_;
  Buf<R> buf_[2]{};
  Work<R> w_{};
  double* stage_ = nullptr;
  long long n_ = 0, ncells_ = 0;
  int cur_ = 0;
  bool have_work_ = false;
  bool dense_ = false;  // rows longer than kDenseRow on average, when the capacity was last checked
  int countdown_ = 0;
  Forms forms_, alone_, beside_;  // those of the launches being made, of steps alone, of graph set 1
  cudaGraphExec_t graphs_[2][2] = {};  // [set][parity]
  std::vector<void*> allocs_;
  std::vector<void*> anc_allocs_;  // anchor tables, kept across re-allocations
  int init_rc_ = 0;
  int sms_ = 1;  // multiprocessors of the engine's device
  bool cap_clamped_ = false;  // a list-capacity growth fell short since the last stats
};

}  // namespace mrsph
