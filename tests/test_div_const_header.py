"""div_const as the header has it, for the constants the header's callers give it.

The bodies of div_const and bessel_i0 are taken from csrc/hm_hair_bsdf.cuh and
compiled for the host (div_const in both its forms, with the device intrinsics'
meaning): bessel_i0 runs once with a div_const that records its divisors, and
for each of them and for the other callers' kEta every mantissa of two binades
must give the correctly rounded quotient (a power of two scales both sides
exactly)."""
import re
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "hairmsnn_gb300" / "csrc"
BSDF, COMMON = (CSRC / "hm_hair_bsdf.cuh").read_text(), (CSRC / "hm_common.cuh").read_text()


def function(text, signature):
    start = text.index(signature)
    at = text.index("{", start)
    depth = 0
    for k in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[start:k + 1]
    raise AssertionError(signature)


def second_arguments(text):
    out = []
    for m in re.finditer(r"\bdiv_const\(", text):
        depth, parts, last = 0, [], m.end()
        for k in range(m.end() - 1, len(text)):
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            if depth == 0 or (depth == 1 and text[k] == ","):
                parts.append(text[last:k].strip())
                last = k + 1
            if depth == 0:
                break
        out.append(parts[1])
    return out


PROGRAM = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#define HM_HD static inline
#define HM_D static inline
%(eta)s
%(sqr)s
static float rec[64];
static int n_rec = 0;
namespace series {
static float div_const(float a, float c) { rec[n_rec++] = c; return a / c; }
%(bessel)s
}
namespace host {
%(div)s
}
#define __CUDA_ARCH__ 1030
#define __fmul_rn(a, b) ((a) * (b))
#define __fmaf_rn fmaf
namespace device {
%(div)s
}
int main() {
  series::bessel_i0(2.f);
  rec[n_rec++] = kEta;
  for (int k = 0; k < n_rec; ++k) {
    volatile float vc = rec[k];
    const float c = vc;
    long bad = 0;
    for (uint32_t m = 0; m < (1u << 24); ++m) {
      const uint32_t bits = (127u << 23) + m;
      float a;
      memcpy(&a, &bits, 4);
      const float q = a / c;
      bad += host::div_const(a, c) != q || device::div_const(a, c) != q;
    }
    printf("%%.9g %%ld\n", c, bad);
  }
}
"""


def test_callers_divide_by_the_checked_constants():
    series = function(BSDF, "HM_D float bessel_i0(float x)")
    rest = BSDF.replace(function(BSDF, "HM_HD float div_const("), "").replace(series, "")
    assert len(second_arguments(series)) == 1
    assert set(second_arguments(rest)) == {"kEta"}
    for path in CSRC.iterdir():
        if path.is_file() and path.name != "hm_hair_bsdf.cuh":
            assert "div_const(" not in path.read_text(), path.name


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    src = PROGRAM % {"eta": re.search(r"constexpr float kEta = [^;]*;", COMMON).group(),
                     "sqr": function(COMMON, "HM_HD float sqr(float v)"),
                     "bessel": function(BSDF, "HM_D float bessel_i0(float x)"),
                     "div": function(BSDF, "HM_HD float div_const(")}
    (d / "d.cpp").write_text(src)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", str(d / "d.cpp"), "-o", str(d / "d"), "-lm"], check=True)
    out = subprocess.run([str(d / "d")], check=True, capture_output=True, text=True).stdout.split()
    return dict(zip(out[0::2], map(int, out[1::2])))


def test_quotients_are_correctly_rounded(results):
    assert len(results) >= 10 and "1.54999995" in results
    assert set(results.values()) == {0}, results
