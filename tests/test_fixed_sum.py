"""Fixed-point sums of doubles (qclojure_gb300/csrc/fixed_sum.cuh), compiled for the host: groups of
1 to 4096 values of both signs, up to 110 bits apart, from the smallest subnormals to 2^1010, and
groups that cancel, against the exact sums in 128-bit integers. Every value loses less than one
unit of the lower integers (2^-88 of the largest value's power of two) and their sum's conversion
half of 2^7; a group with an infinity or NaN gives NaN."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r'''
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "fixed_sum.cuh"

typedef __int128 wide;
struct Sum {
  double hi, lo;
  int E;
};
static Sum fixed(const std::vector<double>& v, const std::vector<int>& flip) {
  uint32_t key = 0;
  for (double x : v) key = std::max(key, qg_fix_key(x));
  const int E = qg_fix_exponent(key);
  int64_t h = 0, l = 0;
  for (size_t i = 0; i < v.size(); ++i) {
    const qg_fixed x = qg_fix(v[i], E, (uint32_t)flip[i]);
    h += x.h;
    l += x.l;
  }
  return Sum{qg_fix_hi(h, E), qg_fix_lo(l, E), E};
}

int main() {
  std::mt19937_64 rng(3);
  long bad = 0;
  for (int rep = 0; rep < 6000; ++rep) {
    const int count = rep % 3 == 0 ? 16 : rep % 3 == 1 ? 1 + (int)(rng() % 4096) : 4096;
    const int unit[4] = {-1074, -60, -900, 900};  // the values are multiples of 2^unit
    const int u = unit[(rep / 3) % 4], widest = 1 + (int)(rng() % 53), spread = (int)(rng() % 58);
    std::vector<double> v;
    std::vector<int> flip;
    wide want = 0;
    for (int i = 0; i < count; ++i) {
      const int64_t m = (int64_t)(rng() >> (64 - (1 + (int)(rng() % widest)))) * (rng() & 1 ? -1 : 1);
      const int shift = (int)(rng() % (spread + 1));
      v.push_back(std::ldexp((double)m, shift + u));
      flip.push_back((int)(rng() & 1));
      want += ((wide)m << shift) * (flip.back() ? -1 : 1);
      if (rep % 5 == 0 && i + 2 < count && rng() % 8) {  // most terms cancel
        v.push_back(v.back());
        flip.push_back(1 - flip.back());
        want -= ((wide)m << shift) * (flip[flip.size() - 2] ? -1 : 1);
        ++i;
      }
    }
    const Sum s = fixed(v, flip);
    const wide got = (wide)std::ldexp(s.hi, -u) + (wide)std::ldexp(s.lo, -u);
    const wide diff = got > want ? got - want : want - got;
    const int low = s.E - 1111 - u;  // the lower integers' unit against the values'
    const double tol = low > 0 ? std::ldexp((double)count + 64, low) : std::ldexp(64.0, low);
    if ((double)diff > tol) {
      if (bad < 5) std::printf("%zu values of unit 2^%d: off by %g, allowed %g\n", v.size(), u, (double)diff, tol);
      ++bad;
    }
  }
  for (double x : {(double)INFINITY, -(double)INFINITY, (double)NAN}) {
    const Sum s = fixed({1.0, x, 0x1p-1074, -2.0}, {0, 1, 0, 1});
    if (!std::isnan(s.hi)) ++bad;
  }
  const Sum z = fixed({0.0, -0.0}, {1, 0});
  if (z.hi != 0 || z.lo != 0) ++bad;
  std::printf(bad ? "MISMATCHES %ld\n" : "ok\n", bad);
  return bad ? 1 : 0;
}
'''


def test_fixed_sums_match_exact_integers(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    src = tmp_path / "fixed_check.cpp"
    exe = tmp_path / "fixed_check"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "qclojure_gb300" / "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip().endswith("ok"), out.stdout
