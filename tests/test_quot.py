"""The quotient from a shared reciprocal (csrc/mrsph_common.cuh, quot) is within one
unit in the last place of the exact one, for reciprocals a few units off, as
the Wendland gradient forms them (CPU, against Fractions)."""
import math
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sph-mesh-generation_gb300", "csrc")

HARNESS = r'''
#include "mrsph_common.cuh"
#include <cstdio>
int main() {
  double d, h;
  while (scanf("%lf %lf", &d, &h) == 2) {
    const double a2 = h * h * h * (d + 1.e-15), a3 = h * h * (h * h) * (d + 1.e-15);
    printf("%.17g %.17g %.17g\n", mrsph::quot(d, h, 1.0 / h), mrsph::quot(d, h, 1.0 / (a2 * h) * a2),
           mrsph::quot(d, h, 1.0 / (a3 * h) * a3));
  }
  return 0;
}
'''


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_quot_within_one_ulp(tmp_path):
    src, exe = tmp_path / "q.cu", tmp_path / "q"
    src.write_text(HARNESS)
    r = subprocess.run(["nvcc", "-std=c++17", "-O2", "-fmad=false", "-Xcompiler", "-ffp-contract=off",
                        "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    rng = np.random.default_rng(17)
    h = 10.0 ** rng.uniform(-6, 3, 4000)
    d = h * rng.uniform(0.0, 2.6, 4000)
    inp = "\n".join(f"{float(x)!r} {float(y)!r}" for x, y in zip(d, h))
    out = subprocess.run([str(exe)], input=inp, capture_output=True, text=True, check=True).stdout.split()
    for x, y, got in zip(d, h, np.array(out, dtype=float).reshape(-1, 3)):
        exact = Fraction(float(x)) / Fraction(float(y))
        for v in got:
            assert abs(Fraction(float(v)) - exact) <= Fraction(math.ulp(float(v)))
