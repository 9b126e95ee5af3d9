"""The outcome rule of the density-matrix kernels (csrc/dm.cuh, pair_ge)
decides a float pair against 1e-4 as FP64 does, without FP64 instructions.  The
header's own function, compiled for the host (no GPU)."""
import os
import subprocess

import numpy as np

from mentpy_gb300 import build

CSRC = os.path.join(os.path.dirname(os.path.abspath(build.__file__)), "csrc")
PROGRAM = """
#include "dm.cuh"
#include <cstdio>
int main() {
  float v[2];
  while (fread(v, 4, 2, stdin) == 2) putchar(mbqc::pair_ge(make_float2(v[0], v[1]), 1e-4) ? 1 : 0);
}
"""


def _pairs():
    """Renormalised pairs (|lo| <= half an ulp of hi) around the bound."""
    g = np.random.default_rng(5)
    t = 1e-4
    tf = np.float32(t)
    his = [np.float32(0.0), np.float32(1.0), np.float32(-1e-4), np.float32(np.inf), np.float32(np.nan)]
    x = tf
    for _ in range(60):  # 60 floats on each side of the bound (17 of them within 1e-6)
        his.append(x)
        x = np.nextafter(x, np.float32(1))
    x = tf
    for _ in range(60):
        x = np.nextafter(x, np.float32(0))
        his.append(x)
    out = []
    for hi in his:
        los = np.array([0.0], np.float32)
        if np.isfinite(hi) and hi != 0:
            half = float(np.spacing(abs(hi))) / 2
            near = t - float(hi)  # the lo that meets the bound, and its neighbourhood down to 2^-70
            los = [near, -half, half, 0.0, *g.uniform(-half, half, 200)]
            los += [near + s * k * 2.0**e for e in range(-70, -45) for k in (1, 3, 5, 7) for s in (-1, 1)]
            los = np.array([v for v in los if abs(v) <= half], np.float64).astype(np.float32)
            los = np.unique(np.concatenate([los, np.nextafter(los, np.float32(1)), np.nextafter(los, np.float32(-1))]))
            los = los[np.abs(los) <= half]
        out += [(hi, lo) for lo in los]
    return np.array(out, np.float32)


def test_pairs_decide_as_their_fp64_sum(tmp_path):
    src = tmp_path / "bound.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "bound"
    flags = [f for f in build.FLAGS if not f.startswith("-Xptxas")]
    subprocess.run([build.nvcc(), *build.ARCH, *flags, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    pairs = _pairs()
    r = subprocess.run([str(exe)], input=pairs.tobytes(), capture_output=True, check=True)
    got = np.frombuffer(r.stdout, np.uint8).astype(bool)
    want = pairs[:, 0].astype(np.float64) + pairs[:, 1].astype(np.float64) >= 1e-4
    near = np.abs(pairs[:, 0] - np.float32(1e-4)) <= 1e-6 * 1e-4
    assert len(pairs) > 10000 and near.sum() > 1000
    assert 0.2 < want[near].mean() < 0.8
    assert np.array_equal(got, want)
