"""The division of the on-chip PLAIN solve (csrc/pf_quotient.cuh), compiled for
the host: by a stored reciprocal and two corrections it must give the bits of the
division.  Every operation in it is an IEEE product, sum or fused multiply-add, so
the host's results are the device's."""
import os
import subprocess

from conftest import ROOT

MAIN = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "pf_quotient.cuh"

static uint64_t state = 88172645463325252ull;
static uint64_t rnd() {
  state ^= state << 13; state ^= state >> 7; state ^= state << 17;
  return state;
}
static double make(uint64_t mantissa, int e, bool neg = false) {
  const uint64_t b = (uint64_t)neg << 63 | (uint64_t)(e + 1023) << 52 | (mantissa & 0xfffffffffffffull);
  double v;
  memcpy(&v, &b, 8);
  return v;
}
static uint64_t bits(double v) {
  uint64_t b;
  memcpy(&b, &v, 8);
  return b;
}
static long bad = 0;
static void check(double r, double d) {
  const double want = d > 0.0 ? r / d : 0.0, got = pf::quotient(r, d, pf::inv_of(d));
  if (bits(want) != bits(got) && !(want != want && got != got) && bad++ < 10)
    printf("r %a d %a: %a, the division gives %a\n", r, d, got, want);
}
int main() {
  // random values, mantissas of few bits and next to 1 and 2 among them
  uint64_t special[12] = {0, 1, 2, 3, 0xfffffffffffffull, 0xffffffffffffeull, 0xffffffffffffdull,
                          0x8000000000000ull, 0x7ffffffffffffull, 0x8000000000001ull, 0x5555555555555ull,
                          0x6a09e667f3bccull};
  for (int i = 0; i < 4000000; ++i) {
    const uint64_t a = rnd(), b = rnd();
    const uint64_t mr = a % 4 == 0 ? special[(a >> 8) % 12] : a >> 12, md = b % 4 == 0 ? special[(b >> 8) % 12] : b >> 12;
    check(make(mr, (int)(rnd() % 1040) - 520, a & 2), make(md, (int)(rnd() % 840) - 420));
    check(make(mr, (int)(rnd() % 60) - 30, a & 2), make(md, (int)(rnd() % 60) - 30));
  }
  // both sides of the ranges' ends, the ends of the exponent range, zeros and the rest
  const double rs[] = {0.0, -0.0, 0x1p-1074, -0x1p-1074, 0x1.8p-1040, 0x1p-1022, 0x1.fffffffffffffp-501, 0x1p-500,
                       0x1.0000000000001p-500, 0x1.fffffffffffffp499, 0x1p500, 0x1.0000000000001p500, 1.0, -3.0,
                       0x1.fffffffffffffp1023, -0x1.fffffffffffffp1023, 1.0 / 0.0 * 1.0, -1.0 / 0.0};
  const double ds[] = {0.0, -1.0, 0x1p-1074, 0x1p-1022, 0x1.fffffffffffffp-401, 0x1p-400, 0x1.0000000000001p-400,
                       0x1.fffffffffffffp399, 0x1p400, 0x1.0000000000001p400, 1.0, 3.0, 0x1.fffffffffffffp-1,
                       0x1.fffffffffffffp1023, 1.0 / 0.0};
  for (double r : rs)
    for (double d : ds) check(r, d);
  for (double d : ds) check(0.0 / 0.0, d);
  printf("%ld differ\n", bad);
  return bad != 0;
}
"""


def test_quotient_gives_the_bits_of_the_division(tmp_path):
    src, exe = tmp_path / "quotient.cpp", tmp_path / "quotient"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I",
                    os.path.join(ROOT, "adaptive-pf-flip_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
