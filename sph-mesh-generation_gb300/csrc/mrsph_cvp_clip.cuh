// mrsph_cvp_clip.cuh — the polygon clip of the CVP faces (mrsph_cvp.cu), kGroup
// lanes per polygon.  Nothing but CUDA's keywords and warp intrinsics is needed,
// so a host compiler can run it against an emulated warp.
#pragma once

namespace mrsph {

constexpr int CVP_MAXV = 64;

// Sutherland-Hodgman clip of polygons by n . x <= d, one polygon per group of
// kGroup lanes, in shared memory (vertex a on lane a mod kGroup): A (nv
// vertices) to B, s the signed distances.  The four groups of a warp call it
// together (nv = 0: nothing to clip).  Vertices leave in the order a
// sequential walk over the edges would write them; those past CVP_MAXV are
// dropped.  Returns the number of vertices written before that limit, or -1
// when no vertex lies outside (B untouched: the polygon stays A).
// One lane per polygon left a warp waiting on a chain of 20 to 30 clips of 4
// to 10 vertices, each some 20 dependent FP64 operations; a group does a clip
// in one vertex's time and keeps the vertices out of local memory.  The
// groups advance in step because an FP64 instruction costs a warp the same 16
// cycles for one group as for four (301,270 points, 128 VPs: 117 us an iteration,
// 130 us when they ran apart; 1,786 us with one lane per pair and no cull).
constexpr int kGroup = 8;
struct Lanes {
  int shift, gl;  // first lane of the group; this lane's index in it
  __device__ Lanes() {
    const int lane = threadIdx.x & 31;
    gl = lane & (kGroup - 1);
    shift = lane - gl;
  }
  __device__ unsigned ballot(bool p) const {
    return (__ballot_sync(0xffffffffu, p) >> shift) & ((1u << kGroup) - 1u);
  }
};

template <class T>
__device__ int gclip(const Lanes& g, const T (*A)[3], int nv, const T* n, T d, T (*B)[3], T* s) {
  bool out = false;
  for (int a = g.gl; a < nv; a += kGroup) {
    T t = n[0] * A[a][0];
    t += n[1] * A[a][1];
    t += n[2] * A[a][2];
    t -= d;
    s[a] = t;
    out = out || !(t <= 0);
  }
  __syncwarp();  // s[a + 1] is another lane's: votes order no memory
  const bool any = g.ballot(out) != 0;
  if (!any) nv = 0;
  int no = 0;
  const unsigned below = (1u << g.gl) - 1u;
  for (int a0 = 0; __any_sync(0xffffffffu, a0 < nv); a0 += kGroup) {
    const int a = a0 + g.gl;
    bool keep = false, cross = false;
    T sa = 0, sb = 0;
    int b = 0;
    if (a < nv) {
      b = a + 1 == nv ? 0 : a + 1;
      sa = s[a];
      sb = s[b];
      keep = sa <= 0;
      cross = keep != (sb <= 0);
    }
    const unsigned km = g.ballot(keep), cm = g.ballot(cross);
    int o = no + __popc(km & below) + __popc(cm & below);
    if (keep) {
      if (o < CVP_MAXV) { B[o][0] = A[a][0]; B[o][1] = A[a][1]; B[o][2] = A[a][2]; }
      o++;
    }
    if (cross && o < CVP_MAXV) {
      const T t = sa / (sa - sb);
      for (int q = 0; q < 3; q++) B[o][q] = A[a][q] + (A[b][q] - A[a][q]) * t;
    }
    no += __popc(km) + __popc(cm);
  }
  __syncwarp();
  return any ? no : -1;
}

}  // namespace mrsph
