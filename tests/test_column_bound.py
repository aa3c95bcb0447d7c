"""The error bounds behind the FP32 and FP64 signs of the cut-cell columns (CPU).

k_vm_columns (csrc/mrsph_levelset.cu) takes the sign of a leaf corner from the
FP32 interpolant beyond 2^-20 M, from the direct FP64 interpolation (vm_point64)
beyond 2^-46 M, and that of a leaf's corner sum beyond 2^-17 M and 2^-44 M, M the
largest |corner| of the sub-cube; the reference's values come from gc_path64.
The product's own FP64 functions and the kernel's FP32 expressions are compiled
for the host and checked against Fractions on seeded corner sets."""
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "sph-mesh-generation_gb300", "csrc", "mrsph_levelset.cu")

HARNESS = r'''
#include "%s"
#include <cstdio>
using namespace mrsph;
static void line(const float* c, int x, int y, float& a, float& e) {
  const float tx = (float)x * 0x1p-6f, ty = (float)y * 0x1p-6f;
  const float v00 = fmaf(tx, c[4] - c[0], c[0]), v01 = fmaf(tx, c[5] - c[1], c[1]);
  const float v10 = fmaf(tx, c[6] - c[2], c[2]), v11 = fmaf(tx, c[7] - c[3], c[3]);
  a = fmaf(ty, v10 - v00, v00);
  e = fmaf(ty, v11 - v01, v01);
}
int main() {
  int ncase;
  if (scanf("%%d", &ncase) != 1) return 1;
  for (int t = 0; t < ncase; t++) {
    double cor[8];
    float c[8];
    int p[3], path[6];
    for (int q = 0; q < 8; q++) { scanf("%%lf", &cor[q]); c[q] = (float)cor[q]; }
    for (int d = 0; d < 3; d++) scanf("%%d", &p[d]);
    for (int l = 0; l < 6; l++)
      path[l] = (((p[0] >> (5 - l)) & 1) << 2) | (((p[1] >> (5 - l)) & 1) << 1) | ((p[2] >> (5 - l)) & 1);
    double leaf[8];
    gc_path64<3>(cor, path, 6, leaf);
    float A[4], E[4];
    for (int u = 0; u < 4; u++) line(c, p[0] + (u >> 1), p[1] + (u & 1), A[u], E[u]);
    for (int q = 0; q < 8; q++) {
      const int u = q >> 1, z = p[2] + (q & 1);
      printf("%%.9g %%.17g %%.17g\n", (double)fmaf((float)z * 0x1p-6f, E[u] - A[u], A[u]),
             vm_point64(cor, 2 * (p[0] + (u >> 1)), 2 * (p[1] + (u & 1)), 2 * z), leaf[q]);
    }
    // rows in y: the lines at x, x + 1 of row y, then those of row y + 1
    const float sA = (A[0] + A[2]) + (A[1] + A[3]), sE = (E[0] + E[2]) + (E[1] + E[3]);
    double s = 0.0;
    for (int q = 0; q < 8; q++) s += leaf[q];
    printf("%%.9g %%.17g %%.17g\n", (double)fmaf(fmaf((float)p[2], 0x1p-6f, 0x1p-7f), sE - sA, sA),
           4.0 * vm_point64(cor, 2 * p[0] + 1, 2 * p[1] + 1, 2 * p[2] + 1), s);
  }
  return 0;
}
'''


def exact_at(cor, x, y, z):
    """The trilinear interpolant at (x, y, z) in 1/128 of the sub-cube."""
    def side(t):
        return (1 - Fraction(t, 128), Fraction(t, 128))

    wx, wy, wz = side(x), side(y), side(z)
    return sum(wx[q >> 2] * wy[(q >> 1) & 1] * wz[q & 1] * cor[q] for q in range(8))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_column_sign_bounds(tmp_path):
    src, exe = tmp_path / "h.cu", tmp_path / "h"
    src.write_text(HARNESS % SRC)
    r = subprocess.run(["nvcc", "-std=c++17", "-O2", "-fmad=false", "-Xcompiler", "-ffp-contract=off",
                        "-gencode", "arch=compute_103a,code=sm_103a", "-I", os.path.dirname(SRC), str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    rng = np.random.default_rng(31)
    g = np.array([(x, y, z) for x in (0, 1) for y in (0, 1) for z in (0, 1)], dtype=float) - 0.5
    cases = []
    for t in range(600):
        scale = 10.0 ** rng.integers(-6, 3)
        p = rng.integers(0, 64, 3)
        if t % 3 == 0:
            node = rng.uniform(-1, 1, 8)
        else:  # a surface; in half of these through the leaf, where the signs are close
            n = rng.normal(size=3)
            node = g @ n + rng.normal(scale=1e-3, size=8)
            if t % 3 == 1:
                node = node - float(exact_at([Fraction(float(v)) for v in node], *(2 * int(k) for k in p)))
        cases.append((node * scale, p))
    inp = f"{len(cases)}\n" + "\n".join(" ".join(repr(float(v)) for v in nd) + " " + " ".join(str(int(c)) for c in p)
                                          for nd, p in cases)
    out = subprocess.run([str(exe)], input=inp, capture_output=True, text=True, check=True).stdout.split()
    vals = np.array(out, dtype=float).reshape(len(cases), 9, 3)
    u32, u64 = Fraction(1, 2 ** 24), Fraction(1, 2 ** 53)
    for (node, p), got in zip(cases, vals):
        cor = [Fraction(float(v)) for v in node]
        M = max(abs(v) for v in cor)
        x, y, z = (int(k) for k in p)
        ex = [exact_at(cor, 2 * (x + (q >> 2)), 2 * (y + ((q >> 1) & 1)), 2 * (z + (q & 1))) for q in range(8)]
        for q in range(8):
            assert abs(Fraction(got[q, 0]) - ex[q]) <= 11 * u32 * M
            assert abs(Fraction(got[q, 1]) - ex[q]) <= 11 * u64 * M
            assert abs(Fraction(got[q, 2]) - ex[q]) <= 18 * u64 * M
        assert abs(Fraction(got[8, 0]) - sum(ex) / 2) <= 60 * u32 * M
        assert abs(Fraction(got[8, 1]) - sum(ex) / 2) <= 44 * u64 * M
        for row, b32, b64 in [(got[q], -20, -46) for q in range(8)] + [(got[8], -17, -44)]:
            if abs(row[0]) > float(M) * 2.0 ** b32:
                assert np.sign(row[0]) == np.sign(row[2])
            if abs(row[1]) > float(M) * 2.0 ** b64:
                assert np.sign(row[1]) == np.sign(row[2])
