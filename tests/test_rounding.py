"""The division substitutes of the constraint kernels (csrc/xpbd_round.cuh)
against the division itself, compiled for the host (no GPU)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rlmusclev2_b200" / "csrc"

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include "xpbd_round.cuh"
static float bits(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
// equal, or both not numbers (+0 and -0 are equal)
static bool same(float a, float b) { return a == b || (a != a && b != b); }
static long bad_over(float3 a, float s) {
    const float3 q = xpbd::over(a, s);
    return !same(q.x, a.x / s) + !same(q.y, a.y / s) + !same(q.z, a.z / s);
}
int main() {
    // x / 6: every mantissa, both signs; the error depends on the exponent at the ends of the range only
    long sixths = 0;
    for (int e : {-125, -124, -101, -100, -60, -20, -1, 0, 1, 60, 126, 127})
        for (uint32_t m = 0; m < (1u << 23); ++m)
            for (uint32_t sign = 0; sign < 2; ++sign) {
                const float x = bits(sign << 31 | uint32_t(e + 127) << 23 | m);
                sixths += !same(xpbd::sixth(x), x / 6.f);
            }
    sixths += xpbd::sixth(0.f) != 0.f;
    // a / s: random mantissas, exponents over the whole range, counts and lengths
    std::mt19937_64 g(7);
    long overs = 0;
    auto rnd = [&](int lo, int hi) {
        const uint64_t r = g();
        return bits(uint32_t(r & 1) << 31 | uint32_t(127 + lo + int((r >> 32) % uint64_t(hi - lo + 1))) << 23 |
                    uint32_t(r >> 1 & 0x7fffff));
    };
    for (long k = 0; k < 20000000; ++k) {
        float3 a = make_float3(rnd(-100, 97), rnd(-100, 97), rnd(-100, 97));
        if (k % 16 == 0) a.y = 0.f;
        overs += bad_over(a, k % 2 ? float(1 + g() % 65535) : fabsf(rnd(-20, 62)));
    }
    // what is not finite, and the largest that is
    const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
    const float edge[] = {0.f, -0.f, 1.f, -3e-5f, 0x1p100f, 0x1.fffffep127f, inf, -inf, nan};
    for (float x : edge)
        for (float y : edge)
            for (float z : edge)
                for (float s : {1.f, 3.f, 65535.f, 0x1p63f}) overs += bad_over(make_float3(x, y, z), s);
    std::printf("%ld %ld\n", sixths, overs);
    return 0;
}
"""


def test_substitutes_round_like_the_division(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src, exe = tmp_path / "round.cu", tmp_path / "round"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-march=native,-ffp-contract=off", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", str(CSRC), "-o", str(exe), str(src)], check=True,
                   capture_output=True, text=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out.split() == ["0", "0"], f"x / 6 and a / s that differ: {out}"
