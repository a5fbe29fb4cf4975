"""div_const (csrc/hm_hair_bsdf.cuh): quotient estimate, exact remainder, one
correction is the correctly rounded a / c for every constant it is used with,
for every mantissa of a (two binades; a power of two scales both sides
exactly).  Runs on the host: fmaf is correctly rounded everywhere."""
import re
import subprocess
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "hairmsnn_gb300" / "csrc" / "hm_hair_bsdf.cuh"

PROGRAM = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
int main(void) {
  float c[8];
  int n = 0;
  float ifact = 1.f, i4 = 1.f;
  for (int i = 0; i < 10; ++i) {          /* the Bessel series' divisors */
    if (i > 1) ifact *= (float)i;
    if (i > 2) c[n++] = i4 * (ifact * ifact);
    i4 *= 4.f;
  }
  c[n++] = 1.55f;                         /* the index of refraction */
  for (int k = 0; k < n; ++k) {
    volatile float d = c[k];
    const float y = 1.f / d;
    long bad = 0;
    for (uint32_t m = 0; m < (1u << 24); ++m) {
      const uint32_t bits = (127u << 23) + m;
      float a;
      memcpy(&a, &bits, 4);
      const float q = a * y;
      if (fmaf(fmaf(-d, q, a), y, q) != a / d) ++bad;
    }
    printf("%ld\n", bad);
  }
  return 0;
}
"""


def test_quotients_are_correctly_rounded(tmp_path):
    text = SRC.read_text()
    used = re.findall(r"div_const\(([^;]*)\);", text)
    assert len(used) == 2, used  # the series and the index of refraction: the constants below
    src, exe = tmp_path / "d.c", tmp_path / "d"
    src.write_text(PROGRAM)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", str(src), "-o", str(exe), "-lm"], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert len(out) == 8 and set(out) == {"0"}
