"""The kernels' modular reductions, taken from their sources and compiled for the
host: exact over the whole ranges that their comments state."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "tensorkyber_b200", "csrc")

PRELUDE = r"""
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <initializer_list>
static const int kQ = 3329;
static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b >> 32); }
static inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t sel) {
  const uint64_t v = (uint64_t)b << 32 | a;
  uint32_t r = 0;
  for (int i = 0; i < 4; i++) r |= (uint32_t)(v >> 8 * (sel >> 4 * i & 7) & 255) << 8 * i;
  return r;
}
static inline uint32_t add16x2(uint32_t a, uint32_t b) {
  return ((a + b) & 0xffffu) | (((a >> 16) + (b >> 16)) << 16);
}
"""

MAIN = r"""
#define CHECK(c) do { if (!(c)) { printf("FAIL %s at %lld\n", #c, (long long)s); exit(1); } } while (0)
int main() {
  const uint32_t top = 1u << 26;
  const uint32_t mates[] = {0, 1, 3328, 3329, 12345678, top - 1};
  for (uint32_t s = 0; s < top; s++) {
    const uint32_t r = s % kQ, o = mates[s % 6], m = top - 1 - s;
    CHECK(red_exact_pair(s, m) == (r | (m % kQ) << 16));
    CHECK(red_exact_pair(s, o) == (r | (o % kQ) << 16) && red_exact_pair(o, s) == ((o % kQ) | r << 16));
    if (s + kCentre < top) {
      const int c = (int)r > (kQ - 1) / 2 ? (int)r - kQ : (int)r;
      const int d = (int)(o % kQ) > (kQ - 1) / 2 ? (int)(o % kQ) - kQ : (int)(o % kQ);
      CHECK((int32_t)red_centred(s) == c);
      if (o + kCentre < top)
        CHECK(red_centred_pair(s + kCentre, o + kCentre) ==
              ((uint32_t)(uint16_t)c | (uint32_t)(uint16_t)d << 16));
    }
    if (s < (1u << 25)) {
      const uint32_t l = red_lazy(s);
      CHECK(l % kQ == r && l < (uint32_t)kQ + 11);
      if (s < (1u << 24)) CHECK(l < (uint32_t)kQ + 6);
    }
  }
  for (int s = -(1 << 20) + 1; s < 1 << 20; s++) {
    const int o = s % 2 ? (1 << 20) - 1 : 1 - (1 << 20);
    auto mod = [](int v) { return (uint32_t)((v % kQ + kQ) % kQ); };
    CHECK(reduce_pair((uint32_t)s, (uint32_t)o) == (mod(s) | mod(o) << 16));
    CHECK(reduce_pair((uint32_t)o, (uint32_t)s) == (mod(o) | mod(s) << 16));
  }
  // every quotient of a 32-bit sum, on both sides of its multiple of q
  for (uint64_t j = 0; j * kQ < 1ull << 32; j++)
    for (uint64_t s : {j * kQ, j * kQ + kQ - 1})
      if (s < 1ull << 32) CHECK(red_wide((uint32_t)s) % kQ == s % kQ && red_wide((uint32_t)s) < 4694);
  printf("ok\n");
  return 0;
}
"""


def function(path, name):
    """The definition of a __device__ function, without the device specifiers."""
    with open(os.path.join(CSRC, path)) as f:
        text = f.read()
    m = re.search(rf"^__device__ __forceinline__ (\w+ {name}\(.*?^\}})", text, re.M | re.S)
    return "static inline " + m.group(1) + "\n"


def test_reductions_over_their_ranges(tmp_path):
    with open(os.path.join(CSRC, "tk_ptx.cuh")) as f:
        centre = re.search(r"^constexpr int32_t kCentre = \d+;", f.read(), re.M).group(0)
    src, exe = tmp_path / "r.cpp", tmp_path / "r"
    src.write_text(PRELUDE + centre + "\n" +
                   "".join(function("tk_ptx.cuh", n) for n in ("red_lazy", "red_centred",
                                                               "red_exact_pair", "red_centred_pair")) +
                   function("tk_stages.cuh", "red_wide") + function("tk_pack.cu", "reduce_pair") +
                   MAIN)
    subprocess.run(["g++", "-std=c++17", "-O2", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
