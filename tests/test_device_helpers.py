"""The device headers' helpers: none is left without a caller, and two of the FP64 kernels' that no other test
restates hold over their whole range, restated in C on the host:

* widen_normal: an f32 widened to f64 on the integer pipe equals the conversion for every zero and normal number (every
  1,021st bit pattern, the ends of the range), and flags exactly the others;
* mag_up: an FP32 number above |v|, or one whose square overflows where |v| is 2^127 or more, infinite or NaN."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "multiq_workbench_gb300" / "csrc"

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
static uint32_t fbits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static uint64_t dbits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
static float ff(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static double fd(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
static double widen_normal(float f, int* odd) {
    const uint32_t u = fbits(f), m = u & 0x7FFFFFFFu;
    *odd |= m - 0x800000u >= 0x7F000000u && m != 0u;
    const uint32_t hi = ((uint32_t)((int32_t)u >> 3) & 0x8FFFFFFFu) + (m ? 0x38000000u : 0u);
    return fd(((uint64_t)hi << 32) | (uint32_t)(u << 29));
}
static float mag_up(double v) {
    int32_t hi = (int32_t)(dbits(v) >> 32) & 0x7fffffff;
    if (hi < 0x38100000) hi = 0x38100000;
    if (hi > 0x47e00000) hi = 0x47e00000;
    return ff((uint32_t)(((hi - 0x38000000) << 3) + 8));
}
static uint64_t st = 88172645463325252ull;
static uint64_t xs(void) { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return st; }
int main(void) {
    unsigned long long bad = 0, n = 0;
    const uint32_t ends[] = {0u, 1u, 0x7FFFFFu, 0x800000u, 0x800001u, 0x7F7FFFFFu, 0x7F800000u, 0x7F800001u, 0x7FFFFFFFu};
    for (uint64_t k = 0; k < 0x100000000ull / 1021 + 18; ++k, ++n) {
        const uint32_t u = k < 18 ? ends[k % 9] | (k < 9 ? 0u : 0x80000000u) : (uint32_t)((k - 18) * 1021);
        const float f = ff(u);
        int odd = 0;
        const double d = widen_normal(f, &odd);
        const int normal = fpclassify(f) == FP_ZERO || fpclassify(f) == FP_NORMAL;
        if (odd != !normal || (normal && dbits(d) != dbits((double)f))) ++bad;
    }
    const double sp[] = {0.0, -0.0, 5e-324, 0x1p-126, 0x1.fffffffffffffp126, 0x1p127, -0x1p127, 1e300, INFINITY, -INFINITY, NAN};
    for (long k = 0; k < 4000011L; ++k, ++n) {
        const double v = k < 11 ? sp[k] : k & 1 ? fd(xs()) : ldexp((double)(int64_t)xs(), (int)(xs() % 240) - 190);
        const float m = mag_up(v);
        if (fabs(v) < 0x1p127 ? !((double)m > fabs(v)) : !isinf(m * m)) ++bad;
    }
    printf("%llu %llu\n", n, bad);
    return 0;
}
"""


def test_every_helper_has_a_caller():
    text = {p.name: p.read_text() for p in CSRC.glob("*") if p.suffix in (".h", ".cu", ".cpp")}
    everything = "\n".join(text.values())
    names = [(f, m) for f, t in text.items() if f.endswith(".h")
             for m in re.findall(r"^(?:__device__ __forceinline__|MQ_HD|MQC_HD|MQG_HD) [\w:]+ (\w+)\(", t, re.M)]
    assert len(names) > 40
    alone = [x for x in names if len(re.findall(rf"\b{x[1]}\b\(", everything)) < 2]
    assert not alone, alone


def test_widen_normal_and_mag_up(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    (tmp_path / "h.c").write_text(SRC)
    subprocess.run([cc, "-O2", "-ffp-contract=off", "-o", str(tmp_path / "h"), str(tmp_path / "h.c"), "-lm"], check=True)
    n, bad = map(int, subprocess.run([str(tmp_path / "h")], check=True, capture_output=True, text=True, timeout=120).stdout.split())
    assert n > 8_000_000 and bad == 0
