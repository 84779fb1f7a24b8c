"""The fixed-point pass over the alters, checked on the device:
  * gumbel_est is within kGumbelErr = 1.5e-5 of log(-log u);
  * a predictor's terms, added as the pass adds them (signed_fx, mulhi_fx, which is
    at most 3 units of 2^-46 low), are within 3 units per real effect and exact for
    counts, low words of 0 among them;
  * exp_fx is within 3e-15 relatively and one unit of 2^-(44 - sh) of exp;
and the simulator where a ministep repeats its pass with scaled weights (a large
predictor) or leaves the fixed-point range for float64, against the CPU oracle
(identical trajectories, scores within one float32 ulp as tests/test_gpu_parity.py
states and derives)."""
import subprocess

import numpy as np
import pytest

from cusna_gb300 import workloads as WL
from tests.golden.make_golden import run_case
from tests.test_gpu_parity import GpuEngine, assert_parity

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "saom_common.cuh"
using namespace cusna;
struct In { uint64_t th[3], m[2]; int64_t f0, count; int neg[2], sh; uint32_t u; };
struct Out { int64_t f; uint64_t w; float g; double ref; };
__global__ void run(const In *in, const int2 *tab, Out *out, int n) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n) return;
  const In a = in[x];
  int64_t f = a.f0;
  f += signed_fx(a.th[0] >> 2, a.neg[0] ^ 1);
  f += signed_fx(a.th[1] >> 2, a.neg[1] ^ 1);
  f += (int64_t)a.th[2] * a.count;
  f += signed_fx(mulhi_fx(a.th[0], a.m[0]), a.neg[0]);
  f += signed_fx(mulhi_fx(a.th[1], a.m[1]), a.neg[1]);
  f = signed_fx((uint64_t)f, x & 1);
  out[x].f = f;
  out[x].w = exp_fx(f, a.sh, tab);
  out[x].g = gumbel_est(a.u);
  out[x].ref = log(-log(unif01(a.u)));
}
int main() {
  const int n = 1 << 18;
  std::vector<In> in(n);
  std::vector<Out> out(n);
  std::vector<int2> tab(256);
  for (int q = 0; q < 256; ++q) tab[q] = exp_fx_entry(std::exp2(q / 256.0));
  std::mt19937_64 r(7);
  auto theta = [&] { const uint64_t t = r() >> (14 + r() % 8); const int z = r() % 3;
                     return z == 0 ? (uint64_t)0 : (z == 1 ? t >> 32 << 32 : t); };
  for (int x = 0; x < n; ++x) {
    In &a = in[x];
    a.th[0] = theta(); a.th[1] = theta();
    a.th[2] = (uint64_t)((int64_t)(r() >> 17) - (int64_t)(r() >> 17));
    a.m[0] = (1ull << 62) + (r() >> 3) - (r() >> 3); a.m[1] = (1ull << 62) + (r() % 2 ? r() >> 3 : 0);
    a.count = r() % 4; a.f0 = (int64_t)(r() >> 16) - (int64_t)(r() >> 16);
    a.neg[0] = r() & 1; a.neg[1] = r() & 1;
    a.sh = r() % 8 + 16; a.u = x < 2 ? 0u - x : (uint32_t)r();
  }
  In *di; Out *dout; int2 *dt;
  cudaMalloc(&di, n * sizeof(In)); cudaMalloc(&dout, n * sizeof(Out)); cudaMalloc(&dt, 256 * sizeof(int2));
  cudaMemcpy(di, in.data(), n * sizeof(In), cudaMemcpyHostToDevice);
  cudaMemcpy(dt, tab.data(), 256 * sizeof(int2), cudaMemcpyHostToDevice);
  run<<<n / 256, 256>>>(di, dt, dout, n);
  if (cudaMemcpy(out.data(), dout, n * sizeof(Out), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
  int bad_f = 0, bad_w = 0, bad_g = 0;
  for (int x = 0; x < n; ++x) {
    const In &a = in[x];
    // the predictor in 128 bits: th (m - 2^62) / 2^64 per real effect
    __int128 f = a.f0;
    f += (__int128)(int64_t)a.th[2] * a.count;
    for (int q = 0; q < 2; ++q) {
      const __int128 t = (__int128)(int64_t)a.th[q] * (__int128)((int64_t)(a.m[q] - (1ull << 62)));
      f += (a.neg[q] ? -t : t) >> 64;
    }
    if (x & 1) f = -f;
    const __int128 d = f - (__int128)out[x].f;
    if (d > 8 || d < -8) ++bad_f;   // 3 units each, and the roundings of >> 64 and >> 2
    const long double w = expl((long double)out[x].f / 70368744177664.0L) * ldexpl(1.0L, 44 - a.sh);
    const long double e = fabsl((long double)out[x].w - w);
    if (e > 1.0L + 3e-15L * w) ++bad_w;
    if (!(fabs((double)out[x].g - out[x].ref) <= kGumbelErr)) ++bad_g;
  }
  printf("%d %d %d\n", bad_f, bad_w, bad_g);
  return 0;
}
"""


def test_fixed_point_arithmetic_bounds(tmp_path):
    from cusna_gb300.build import ARCH, CSRC, nvcc
    src, exe = tmp_path / "fixed.cu", tmp_path / "fixed"
    src.write_text(PROGRAM)
    subprocess.check_call([nvcc()] + ARCH + ["-O3", "-fmad=false", "-std=c++17", "-I" + CSRC,
                                             str(src), "-o", str(exe)])
    assert subprocess.check_output([str(exe)], text=True).split() == ["0", "0", "0"]


@pytest.mark.parametrize("kind", ["covariate", "structural", "interaction"])
@pytest.mark.parametrize("scale", [6.0, 4e4])
def test_large_predictors_match_the_oracle(gpu_lib, port, kind, scale):
    """scale 6: predictors up to and beyond the sums' room (the pass runs twice); 4e4: beyond
    the fixed-point range (the chain runs in float64)."""
    c = WL.parity_case(kind, seed=2, n=33, M=3)
    c["theta"] = (c["theta"] * scale).astype(np.float32)
    assert_parity(run_case(GpuEngine(), c), run_case(port, c), f"{kind}/scale={scale}")
