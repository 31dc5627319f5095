"""The SpMV's widening of a float from its bits, against the conversion: every exponent, every kind of
mantissa, subnormals, zeros, infinities and NaNs.  The device function's own text, compiled here."""
import os
import re
import subprocess

from conftest import ROOT

HARNESS = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#define __device__
#define __forceinline__ inline
static uint32_t __float_as_uint(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
static double __hiloint2double(int hi, int lo)
{
    const uint64_t u = ((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo;
    double d; memcpy(&d, &u, 8); return d;
}
%s
int main()
{
    long bad = 0, n = 0;
    auto check = [&](uint32_t u) {
        float f; memcpy(&f, &u, 4);
        const double want = (double)f, got = widen(f);
        uint64_t a, b; memcpy(&a, &want, 8); memcpy(&b, &got, 8);
        ++n;
        if (std::isnan(want) ? !std::isnan(got) : a != b) ++bad;
    };
    for (uint32_t sign = 0; sign < 2; ++sign)
        for (uint32_t e = 0; e < 256; ++e) {
            const uint32_t base = sign << 31 | e << 23;
            for (uint32_t m = 0; m < 1u << 23; m += e == 0 || e == 255 ? 1 : 1021) check(base | m);
            for (uint32_t k = 0; k < 23; ++k) { check(base | 1u << k); check(base | ((1u << k) - 1)); check(base | (0x7fffffu & ~(1u << k))); }
            check(base | 0x7fffffu);
        }
    printf("%%ld %%ld\n", bad, n);
    return bad != 0;
}
"""


def test_widen_equals_the_conversion(tmp_path):
    text = open(os.path.join(ROOT, "dumux_gb300", "csrc", "linalg.cu")).read()
    widen = re.search(r"__device__ __forceinline__ double widen\(float f\)\s*\{.*?\n\}", text, re.S).group(0)
    src, exe = tmp_path / "widen.cc", tmp_path / "widen"
    src.write_text(HARNESS % widen)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-o", str(exe), str(src)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout.split()[1]) > 1 << 25
