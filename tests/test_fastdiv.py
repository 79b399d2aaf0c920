"""The multiplication that stands in for an index division in the permutation kernels (csrc/fastdiv.cuh), compiled
for the host, against the division itself: divisors and dividends at and beside powers of two, the largest, and a
sweep; multiples of the divisor and their neighbours are where a wrong constant shows."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "ipeps.jl_b200" / "csrc"

PROGRAM = r"""
#include "fastdiv.cuh"
#include <cstdio>
#include <vector>
int main() {
  const uint32_t top = 0x7fffffffu;
  std::vector<uint32_t> ds;
  for (uint32_t d = 1; d <= 3000; ++d) ds.push_back(d);
  for (int b = 11; b < 31; ++b)
    for (int e = -1; e <= 1; ++e) ds.push_back((1u << b) + e);
  ds.push_back(top);
  ds.push_back(top - 1);
  long bad = 0;
  for (uint32_t d : ds) {
    const ipeps::FastDiv f(d);
    auto check = [&](uint64_t n) {
      if (n <= top && f.div(uint32_t(n)) != uint32_t(n) / d) ++bad;
    };
    for (int b = 0; b < 32; ++b)
      for (int e = -1; e <= 1; ++e)
        if ((uint64_t(1) << b) + e <= top) check((uint64_t(1) << b) + e);
    for (uint64_t q = 0; q <= 200; ++q) {
      const uint64_t k = (top / d) * q / 200 * d;
      check(k);
      check(k + 1);
      check(k + d - 1);
      if (k > 0) check(k - 1);
    }
    check(0);
    check(top);
  }
  printf("%ld\n", bad);
  return 0;
}
"""


def test_matches_division(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O2", "-D__host__=", "-D__device__=", "-D__forceinline__=inline",
                    "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "0"
