"""SVGF's values bit for bit, on inputs with general normals, sky, disocclusions and (SPECIAL) infinite, NaN, zero and largest
values of the type: the stored frames are those of the kernels that used the IEEE operators throughout, one tap after the other
(python tests/test_svgf_values_gpu.py FILE stores them). A NaN may carry any payload.

The quotients, reciprocals and roots of quotient.cuh against the operators, by a kernel compiled here: on every mantissa, on the
quotients nearest to a tie (the numerators whose remainder by an odd divisor is next to half of it), and on special operands."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

HERE = os.path.dirname(os.path.abspath(__file__))
GOLDEN = os.path.join(HERE, "golden", "svgf_frames.npz")
SPECIAL = [np.inf, -np.inf, np.nan, 0.0, -0.0, 65504.0, 6e-8]
CONFIGS = {  # width, height, options, special values
    "default": (75, 45, {}, False),
    "three": (64, 40, {"iterations": 3, "taa": 0}, False),
    "sharp": (49, 37, {"iterations": 4, "sigmaN": 48.0, "sigmaZ": 0.25}, False),
    "special": (67, 41, {}, True),
    "sigma0": (33, 21, {"iterations": 2, "sigmaL": 0.0, "sigmaZ": 0.0, "sigmaN": 0.0}, True),
}


def frames(w, h, special, n=7):
    """n G-buffers: three slanted surfaces that slide by whole and broken pixels, sky above, noise on all of it."""
    rng = np.random.default_rng(w * h)
    x, y = np.meshgrid(np.arange(w), np.arange(h))
    for t in range(n):
        obj = np.where(x + 2 * t < w // 3, 0, np.where(x + t < 2 * w // 3, 1, 2))
        nrm = np.stack([0.3 * obj - 0.2, 0.5 + 0 * obj, 1.0 - 0.2 * obj], 2) + 0.05 * rng.standard_normal((h, w, 3))
        nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
        z = np.where(y < 4, -1.0, 3.0 + obj + 0.02 * x + 0.01 * y)
        f = {"radiance": rng.gamma(0.6, 1.5, (h, w, 4)), "material": rng.uniform(0.02, 1.0, (h, w, 4)),
             "emission": rng.gamma(0.2, 0.5, (h, w, 4)), "normalDepth": np.dstack([nrm, z]),
             "motion": np.dstack([1.0 + 0.25 * obj, 0.5 * (obj == 2), 7.0 + obj, z])}
        if special:
            for k in ("radiance", "material", "emission"):
                at = rng.integers(0, f[k].size, 4 * len(SPECIAL))
                f[k].flat[at] = np.tile(SPECIAL, 4)
            f["normalDepth"].flat[4 * rng.integers(0, w * h, 3) + 3] = [np.inf, 0.0, 65504.0]
            f["normalDepth"][5, 5, :3] = 300.0
        with np.errstate(over="ignore"):
            yield {k: v.astype(np.float16) for k, v in f.items()}


def outputs(name):
    from hush_b200 import SVGF

    w, h, options, special = CONFIGS[name]
    s, prev, out = SVGF(0, w, h, options), None, []
    for f in frames(w, h, special):
        d = {k: torch.from_numpy(v).cuda() for k, v in f.items()}
        prev = prev or d
        out.append(s.encode(dict(d, prevNormalDepth=prev["normalDepth"], prevMotion=prev["motion"])).cpu().numpy())
        prev = d
    return np.stack(out)[[0, 2, 6]]


@pytest.mark.parametrize("name", sorted(CONFIGS))
def test_frames_are_the_stored_ones(name):
    want, got = np.load(GOLDEN)[name], outputs(name)
    nan = np.isnan(want)
    assert (np.isnan(got) == nan).all()
    assert ((got.view(np.uint16) == want.view(np.uint16)) | nan).all()


PROBE = r"""
#include <cstdio>
#include "quotient.cuh"
using namespace hush;
__device__ unsigned long long bad[4];
__global__ void mantissas() {  // 2^23 threads
  const unsigned m = blockIdx.x * 256 + threadIdx.x;
  for (unsigned e = 1; e <= 252; e += 7) {
    const float x = __uint_as_float(e << 23 | m);
    if (rcp_rn(x) != __frcp_rn(x) || rcp_rn(-x) != __frcp_rn(-x)) atomicAdd(&bad[0], 1ull);
  }
  for (unsigned e = 26; e < 230; e++) {
    const float x = __uint_as_float(e << 23 | m);
    if (sqrt_rn(x) != __fsqrt_rn(x)) atomicAdd(&bad[1], 1ull);
    if (quot_rn(x, 9.0f, rcp_rn(9.0f)) != __fdiv_rn(x, 9.0f)) atomicAdd(&bad[2], 1ull);
  }
}
__global__ void ties() {  // 2^22 threads: a = ((d +- 1) / 2 + c) 2^-k mod d for the odd d of 24 bits
  const unsigned d = 1u << 23 | 2 * (blockIdx.x * 256 + threadIdx.x) + 1;
  const float D = (float)d, r = rcp_rn(D);
  unsigned long long p = 1;
  for (int k = 1; k <= 25; k++) {
    p = p * ((d + 1ull) / 2) % d;
    for (int c = -2; c <= 2; c++) {
      unsigned long long a = (((d + 1ull) / 2 + c) * p) % d;
      while (a && a < (1u << 23)) a *= 2;
      if (k < 23 || a >= (1u << 24)) continue;
      if (quot_rn((float)a, D, r) != __fdiv_rn((float)a, D)) atomicAdd(&bad[2], 1ull);
    }
  }
}
__global__ void special() {
  const float v[12] = {INFINITY, -INFINITY, NAN, 0.0f, -0.0f, 3e38f, 1e-38f, 1e-44f, 1.0f, -7.0f, 65504.0f, 6e-8f};
  for (int i = 0; i < 12; i++) {
    if (__float_as_uint(sqrt_rn(fmaxf(v[i], 0.0f))) != __float_as_uint(__fsqrt_rn(fmaxf(v[i], 0.0f)))) bad[3]++;
    for (int j = 0; j < 12; j++) {
      if (fabsf(v[j]) > 1e38f && fabsf(v[j]) < INFINITY) continue;  // divisors are below 2^126
      const float3 q = div3(make_float3(v[i], 0.0f, -0.0f), v[j]);
      const float w[3] = {__fdiv_rn(v[i], v[j]), __fdiv_rn(0.0f, v[j]), __fdiv_rn(-0.0f, v[j])}, g[3] = {q.x, q.y, q.z};
      for (int c = 0; c < 3; c++)
        if (__float_as_uint(w[c]) != __float_as_uint(g[c]) && !(w[c] != w[c] && g[c] != g[c]) && !(fabsf(w[c]) < 1e-30f && fabsf(g[c]) < 1e-30f)) bad[3]++;
    }
  }
}
int main() {
  mantissas<<<1 << 15, 256>>>();
  ties<<<1 << 14, 256>>>();
  special<<<1, 1>>>();
  unsigned long long h[4] = {~0ull};
  const cudaError_t e = cudaMemcpyFromSymbol(h, bad, sizeof(h));
  printf("%s %llu %llu %llu %llu\n", cudaGetErrorString(e), h[0], h[1], h[2], h[3]);
  return e != cudaSuccess || h[0] || h[1] || h[2] || h[3];
}
"""


def test_quotients_are_the_operators(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "probe.cu").write_text(PROBE)
    csrc = os.path.join(os.path.dirname(HERE), "hush_b200", "csrc")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-I", csrc, "-gencode", "arch=compute_100a,code=sm_100a", "-o",
                    str(tmp_path / "probe"), str(tmp_path / "probe.cu")], check=True)
    r = subprocess.run([str(tmp_path / "probe")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


if __name__ == "__main__":
    np.savez_compressed(sys.argv[1], **{k: outputs(k) for k in CONFIGS})
