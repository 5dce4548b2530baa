"""Below 2^24 trial division by the primes up to 31 and strong tests to the first
three bases of the 7-base set decide primality (is_prime_u64, gb_device.cuh):
every odd composite, on the host."""
import shutil
import subprocess

import pytest

_HARNESS = r"""
#include <cstdint>
#include <cstdio>
#include <vector>

static uint64_t power(uint64_t b, uint64_t e, uint64_t n) {
  uint64_t r = 1;
  for (b %= n; e; e >>= 1, b = b * b % n)
    if (e & 1) r = r * b % n;
  return r;
}
static bool strong(uint64_t n, uint64_t a) {
  uint64_t d = n - 1;
  int s = 0;
  for (; !(d & 1); d >>= 1) ++s;
  uint64_t x = power(a, d, n);
  if (x == 1 || x == n - 1) return true;
  for (int i = 1; i < s; ++i)
    if ((x = x * x % n) == n - 1) return true;
  return false;
}
int main() {
  const uint64_t top = 1 << 24;
  std::vector<char> composite(top);
  for (uint64_t i = 3; i * i < top; i += 2)
    if (!composite[i])
      for (uint64_t j = i * i; j < top; j += 2 * i) composite[j] = 1;
  int wrong = 0, bases2 = 0;
  for (uint64_t n = 37 * 37; n < top; n += 2) {
    bool small = false;
    for (int p : {3, 5, 7, 11, 13, 17, 19, 23, 29, 31}) small |= n % p == 0;
    if (small || !composite[n] || !strong(n, 2)) continue;
    bases2 += strong(n, 325);
    wrong += strong(n, 325) && strong(n, 9375);
  }
  std::printf("%d %d\n", wrong, bases2);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_three_bases_decide(tmp_path):
    src, exe = tmp_path / "bases.cpp", tmp_path / "bases"
    src.write_text(_HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", str(exe), str(src)], check=True, capture_output=True, timeout=120)
    wrong, two = map(int, subprocess.run([str(exe)], capture_output=True, text=True, timeout=120).stdout.split())
    assert wrong == 0 and two > 0
