"""The fixed-point exponential has no undefined arithmetic: compiled for the host with
traps on signed overflow and on shifts of negative values, over the whole range of
predictors (|f| < 2^14) and of scalings, and within its stated 3e-15 + 2^-62 N (the
rounding of ln2/256, N = f 256/ln2) and one unit of exp."""
import subprocess

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "saom_common.cuh"
using namespace cusna;
int main() {
  std::vector<int2> tab(256);
  for (int q = 0; q < 256; ++q) tab[q] = exp_fx_entry(std::exp2(q / 256.0));
  std::mt19937_64 r(11);
  int bad = 0, seen = 0;
  for (int x = 0; x < (1 << 19); ++x) {
    // |f| from 2^-46 to 2^14, both signs; sh so that the result has 0 to 63 bits
    int64_t f = (int64_t)(r() >> (4 + r() % 60));
    if (x & 1) f = -f;
    const double fr = (double)f / 70368744177664.0, lg = fr / 0.6931471805599453;
    const int sh = (int)std::floor(lg) + 44 - (int)(r() % 62);
    const long double w = expl((long double)f / 70368744177664.0L + (44 - sh) * 0.693147180559945309417L);
    if (w >= 4.6e18L) continue;
    const uint64_t got = exp_fx(f, sh, tab.data());
    const long double err = 3e-15L + fabsl((long double)lg) * 256.0L * 2.2e-19L + 1e-19L * fabsl((long double)sh);
    if (!(fabsl((long double)got - w) <= 1.0L + err * w)) ++bad;
    ++seen;
  }
  printf("%d %d\n", bad, seen > (1 << 18));
  return 0;
}
"""


def test_exponential_has_no_undefined_arithmetic(tmp_path):
    from cusna_gb300.build import ARCH, CSRC, nvcc
    src, exe = tmp_path / "host.cu", tmp_path / "host"
    src.write_text(PROGRAM)
    traps = []
    for flag in ("-fsanitize=signed-integer-overflow", "-fsanitize=shift",
                 "-fsanitize-undefined-trap-on-error"):
        traps += ["-Xcompiler", flag]
    subprocess.check_call([nvcc()] + ARCH + ["-O1", "-std=c++17", "-I" + CSRC] + traps +
                          [str(src), "-o", str(exe)])
    assert subprocess.check_output([str(exe)], text=True).split() == ["0", "1"]
