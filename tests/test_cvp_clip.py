"""The CVP faces' group clip (csrc/mrsph_cvp_clip.cuh) on an emulated warp (CPU).

CUDA orders no memory across a vote: what a lane writes to shared memory is
another lane's to read only after __syncwarp().  The emulation takes that at its
word.  32 threads run the product's gclip, each on its own copy of the shared
arrays; a vote exchanges the predicates alone, and __syncwarp() hands every
written word to the other lanes.  Chains of clips of four polygons at a time,
of up to 40 vertices, some whole, some cut away, must give the vertices of a
sequential Sutherland-Hodgman walk bit for bit."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sph-mesh-generation_gb300", "csrc")

HARNESS = r'''
#include <barrier>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <thread>
#include <vector>
#define __device__
static thread_local struct { unsigned x; } threadIdx;
static unsigned g_pred[32];
static std::barrier<> g_bar(32);
static unsigned __ballot_sync(unsigned, bool p) {
  g_pred[threadIdx.x] = p;
  g_bar.arrive_and_wait();
  unsigned m = 0;
  for (int l = 0; l < 32; l++) m |= g_pred[l] << l;
  g_bar.arrive_and_wait();
  return m;
}
static bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
static int __popc(unsigned v) { return __builtin_popcount(v); }
static void __syncwarp();
#include "mrsph_cvp_clip.cuh"
using namespace mrsph;

typedef TYPE T;
constexpr int W = 2 * CVP_MAXV * 3 + CVP_MAXV;  // a group's words: A, B, s
static T g_mem[32][W], g_seen[32][W];           // each lane's copy, and as it was at the last barrier
static bool g_race = false;
static void __syncwarp() {
  g_bar.arrive_and_wait();
  if (threadIdx.x % kGroup == 0) {
    const int l0 = threadIdx.x;
    for (int w = 0; w < W; w++) {
      int by = -1;
      for (int l = l0; l < l0 + kGroup; l++)
        if (std::memcmp(&g_mem[l][w], &g_seen[l][w], sizeof(T))) {
          if (by >= 0 && std::memcmp(&g_mem[l][w], &g_mem[by][w], sizeof(T))) g_race = true;
          by = l;
        }
      if (by < 0) continue;
      const T v = g_mem[by][w];
      for (int l = l0; l < l0 + kGroup; l++) g_mem[l][w] = g_seen[l][w] = v;
    }
  }
  g_bar.arrive_and_wait();
}

struct Poly { int nv; T v[CVP_MAXV][3]; };
static void walk(Poly& p, const T* n, T d) {
  Poly o;
  o.nv = 0;
  auto dist = [&](int a) {
    T t = n[0] * p.v[a][0];
    t += n[1] * p.v[a][1];
    t += n[2] * p.v[a][2];
    return t - d;
  };
  for (int a = 0; a < p.nv; a++) {
    const int b = (a + 1) % p.nv;
    const T sa = dist(a), sb = dist(b);
    if (sa <= 0) std::memcpy(o.v[o.nv++], p.v[a], sizeof(p.v[a]));
    if ((sa <= 0) != (sb <= 0)) {
      const T t = sa / (sa - sb);
      for (int q = 0; q < 3; q++) o.v[o.nv][q] = p.v[a][q] + (p.v[b][q] - p.v[a][q]) * t;
      o.nv++;
    }
  }
  p = o;
}

constexpr int NROUND = 12, NCLIP = 12;
static Poly g_in[NROUND][4];
static T g_n[NROUND][NCLIP][4][3], g_d[NROUND][NCLIP][4];
static Poly g_out[NROUND][4];

static void lane(int l) {
  threadIdx.x = l;
  const Lanes g;
  const int grp = l / kGroup;
  for (int r = 0; r < NROUND; r++) {
    T (*A)[3] = reinterpret_cast<T(*)[3]>(g_mem[l]), (*B)[3] = A + CVP_MAXV;
    T* s = g_mem[l] + 2 * CVP_MAXV * 3;
    int nv = g_in[r][grp].nv;
    for (int a = g.gl; a < nv; a += kGroup) std::memcpy(A[a], g_in[r][grp].v[a], sizeof(A[a]));
    __syncwarp();
    for (int c = 0; c < NCLIP; c++) {
      const int no = gclip<T>(g, A, nv, g_n[r][c][grp], g_d[r][c][grp], B, s);
      if (no < 0) continue;
      nv = no;
      std::swap(A, B);
    }
    if (g.gl == 0) {
      g_out[r][grp].nv = nv;
      std::memcpy(g_out[r][grp].v, A, sizeof(T) * 3 * nv);
    }
    __syncwarp();
  }
}

int main() {
  std::mt19937 rng(7);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  const int sizes[] = {4, 3, 8, 9, 7, 16, 17, 40, 12, 31, 32, 5};
  for (int r = 0; r < NROUND; r++)
    for (int g = 0; g < 4; g++) {
      Poly& p = g_in[r][g];
      p.nv = sizes[(r + 3 * g) % 12];
      const double ph = u(rng), tilt = u(rng);
      for (int a = 0; a < p.nv; a++) {  // a convex polygon of a tilted plane
        const double t = 6.283185307179586 * (a + 0.3 * u(rng)) / p.nv + ph;
        p.v[a][0] = (T)std::cos(t);
        p.v[a][1] = (T)std::sin(t);
        p.v[a][2] = (T)(tilt * std::cos(t));
      }
      for (int c = 0; c < NCLIP; c++) {
        for (int q = 0; q < 3; q++) g_n[r][c][g][q] = (T)u(rng);
        g_d[r][c][g] = (T)(g == 3 && c > 8 ? -2.0 : 0.4 + 0.4 * u(rng));  // the last group's polygons are cut away
      }
    }
  std::vector<std::thread> th;
  for (int l = 0; l < 32; l++) th.emplace_back(lane, l);
  for (auto& t : th) t.join();
  int bad = g_race, cut = 0, gone = 0;
  for (int r = 0; r < NROUND; r++)
    for (int g = 0; g < 4; g++) {
      Poly p = g_in[r][g];
      for (int c = 0; c < NCLIP; c++) walk(p, g_n[r][c][g], g_d[r][c][g]);
      cut += p.nv > 0;
      gone += p.nv == 0;
      bad += p.nv != g_out[r][g].nv || std::memcmp(p.v, g_out[r][g].v, sizeof(T) * 3 * p.nv);
    }
  std::printf("%d %d %d\n", bad, cut, gone);
  return 0;
}
'''


@pytest.mark.parametrize("type_", ["float", "double"])
def test_group_clip_with_votes_that_order_no_memory(tmp_path, type_):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "clip.cpp", tmp_path / "clip"
    src.write_text(HARNESS)
    subprocess.run([gxx, "-O1", "-std=c++20", "-ffp-contract=off", "-pthread", "-DTYPE=" + type_, "-I", CSRC, str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300).stdout
    bad, cut, gone = (int(v) for v in out.split())
    assert cut > 10 and gone > 5  # polygons left whole or cut, and polygons clipped away
    assert bad == 0
