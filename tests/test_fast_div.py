"""The host-computed multiply-and-shift division by nx (csrc/mp_params.h,
FastDiv) against integer division, over divisors and dividends at the edges
of the range: 0 <= n < 2^31, 1 <= d < 2^31."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))

SOURCE = r"""
#include <cstdio>
#include <initializer_list>
#include "mp_params.h"
int main() {
  const long long top = (1ll << 31) - 1;
  long long bad = 0, seen = 0;
  auto check = [&](long long n, long long d) {
    if (n < 0 || n > top || d < 1 || d > top) return;
    const shield::FastDiv f = shield::fast_div((int)d);
    ++seen;
    if ((long long)(((uint64_t)(uint32_t)n * f.m) >> f.s) != n / d) ++bad;
  };
  auto divisor = [&](long long d) {
    for (long long q : {0ll, 1ll, 2ll, 3ll, top / (d > 0 ? d : 1) - 1, top / (d > 0 ? d : 1)})
      for (int e = -2; e <= 2; ++e) check(q * d + e, d);
    for (long long n = 1; n < top; n = n * 5 / 3 + 1) check(n, d);
    check(top, d);
  };
  for (long long d = 1; d < 5000; ++d) divisor(d);
  for (int b = 12; b <= 31; ++b)
    for (int e = -3; e <= 3; ++e) divisor((1ll << b) + e);
  std::printf("%lld %lld\n", bad, seen);
}
"""


def test_matches_integer_division(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    csrc = os.path.join(os.path.dirname(HERE), "pyshield_b200", "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", csrc, str(src), "-o", str(exe)], check=True)
    bad, seen = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and seen > 100000
