"""The kernels' conversions, sums and comparisons on integers (csrc/tis_fixed.cuh, and to_fix of
csrc/tis_device.cuh), run on the GPU over random values and the edges of their ranges against
the operation each stands for: the same bits everywhere, with the constants tis_create forms."""
import os
import subprocess

import pytest

from tis_gb300 import build

PROGRAM = r"""
#include <cstdio>
#include "tis_fixed.cuh"
using namespace tis;

__device__ inline unsigned long long mix(unsigned long long z)  // splitmix64
{
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
struct Rng {
    unsigned long long s;
    __device__ unsigned long long next() { return mix(s++ * 0x2545f4914f6cdd1dull); }
    __device__ int below(int n) { return (int)(next() % (unsigned)n); }
    __device__ double uniform() { return (double)(next() >> 11) * 0x1p-53; }
    __device__ double sign() { return next() & 1 ? 1.0 : -1.0; }
};
__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b); }
__device__ bool same(float a, float b) { return __float_as_int(a) == __float_as_int(b) || (a != a && b != b); }
__device__ double beside(double x, Rng &g)  // x or up to two units in the last place from it
{
    return __longlong_as_double(__double_as_longlong(x) + (x == 0.0 ? 0 : g.below(5) - 2));
}

// bad[f]: values for which function f differs; used[f]: of them on the integer path
__global__ void check(RepParams R, unsigned long long seed, unsigned long long *bad, unsigned long long *used)
{
    Rng g{mix(seed + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x)};
    for (int it = 0; it < 64; ++it) {
        {  // to_fix: |v| from 2^-40 to the limit, ties, halves, the switch at 2^21, the clamp, NaN and infinities
            const int kind = g.below(6);
            float v = kind == 0   ? (float)(ldexp(1.0 + g.uniform(), g.below(70) - 40))
                      : kind == 1 ? (float)g.below(1 << 20) + 0.5f
                      : kind == 2 ? __uint_as_float(__float_as_uint(2097152.0f) + g.below(9) - 4)
                      : kind == 3 ? __uint_as_float(__float_as_uint(kFixLimit) + g.below(9) - 4)
                      : kind == 4 ? (float)g.below(1 << 21) + (float)ldexp((double)(2 * g.below(8) + 1), -33)
                                  : __uint_as_float(__float_as_uint(0.5f) + g.below(9) - 4);
            if (g.below(64) == 0) v = g.below(2) ? __int_as_float(0x7fc00000) : __int_as_float(0x7f800000);
            if (g.below(2)) v = -v;
            int err = 0;
            const long long got = to_fix(v, err);
            const bool in = fabsf(v) < kFixLimit;
            const float c = v != v ? 0.0f : fminf(fmaxf(v, -kFixLimit), kFixLimit);
            if (got != __float2ll_rn(c * kFixScaleF) || err != (in ? 0 : (int)kErrNonFinite)) atomicAdd(bad + 0, 1ull);
        }
        {  // fix_to_double over and beyond its 53 bits
            const long long v = (long long)(g.next() >> g.below(64)) * (g.below(2) ? 1 : -1) + (g.below(8) ? 0 : g.below(3) - 1);
            if (!same(fix_to_double(v), (double)v)) atomicAdd(bad + 1, 1ull);
        }
        const double L = R.box[0];
        {  // fix_position: the box, its image, small, negative and far coordinates, neighbours of exact multiples
            const int kind = g.below(5);
            double x = kind == 0   ? g.uniform() * 2.0 * L
                       : kind == 1 ? beside((double)(g.next() >> 32) / R.qinv[0], g)
                       : kind == 2 ? ldexp(1.0 + g.uniform(), g.below(90) - 80)
                       : kind == 3 ? beside(2.0 * L, g)
                                   : g.uniform() * 1048576.0;
            if (g.below(4) == 0) x = -x;
            if (fix_position(&R, 0, x) != (int)(unsigned)__double2ll_rd(__dmul_rn(x, R.qinv[0]))) atomicAdd(bad + 2, 1ull);
        }
        // positions: the axis, its ends, powers of two; shifts: up to the largest, tiny, halves of a unit, zero
        const double least = ldexp(1.0, (int)(R.ax[0].lo >> 20) - 1023);
        double x = g.below(3) ? g.uniform() * 1.02 * L : beside(ldexp(1.0, g.below(14) - 12) * 1024.0 * least, g);
        if (g.below(16) == 0) x = g.below(2) ? -x : 0.0;
        const double ulp = __longlong_as_double(__double_as_longlong(fabs(x)) + 1) - fabs(x);
        const int kind = g.below(5);
        double s = kind == 0   ? g.uniform() * least
                   : kind == 1 ? ldexp(1.0 + g.uniform(), -g.below(80)) * least
                   : kind == 2 ? beside(0.5 * ulp * (1 + g.below(8)), g)
                   : kind == 3 ? beside(least, g)
                               : 0.0;
        s *= g.sign();
        {
            Shift<true> sh;
            sh.set(&R, 0, s);
            unsigned long long v;
            if (axis_fix(&R, 0, x, v) && sh.fix[0] != kNoShift) atomicAdd(used + 3, 1ull);
            if (!same(axis_add<true>(&R, 0, x, sh), __dadd_rn(x, s))) atomicAdd(bad + 3, 1ull);
            Shift<false> sf;
            sf.set(&R, 0, s);
            if (!same(axis_add<false>(&R, 0, x, sf), __dadd_rn(x, s))) atomicAdd(bad + 3, 1ull);
        }
        {  // x + (x - o), and the difference in FP32 to a unit of the axis or 2^-23 of it
            const double o = __dsub_rn(x, s), e = __dsub_rn(x, o);
            float a, b, c;
            if (!same(axis_ahead<false, true>(&R, 0, x, o, a), __dadd_rn(x, e))) atomicAdd(bad + 4, 1ull);
            if (!same(axis_ahead<false, false>(&R, 0, x, o, b), __dadd_rn(x, e))) atomicAdd(bad + 4, 1ull);
            if (!same(axis_ahead<true, true>(&R, 0, x, o, c), __dsub_rn(__dmul_rn(2.0, x), o))) atomicAdd(bad + 4, 1ull);
            const double room = (double)R.ax[0].step + ldexp(fabs(e), -23) + 0x1p-126;
            if (!(fabs((double)a - e) <= room && fabs((double)b - e) <= room && fabs((double)c - e) <= room)) atomicAdd(bad + 4, 1ull);
        }
        {  // FP64 to FP32 and back over every exponent, ties of the last place, NaN and infinities
            unsigned long long bits = g.next();
            if (g.below(2)) bits = (bits & 0x800fffffffffffffull) | (unsigned long long)(1023 - 160 + g.below(320)) << 52;
            if (g.below(3) == 0) bits = (bits & ~0x1fffffffull) | 0x10000000ull;  // halfway
            else if (g.below(3) == 0) bits |= 0x1fffffffull;
            const double d = __longlong_as_double((long long)bits);
            if (!same(to_float(d), __double2float_rn(d))) atomicAdd(bad + 5, 1ull);
            const float f = __uint_as_float((unsigned)g.next());
            if (!same(to_double(f), (double)f)) atomicAdd(bad + 6, 1ull);
            // cut towards zero where normal; 0 below 2^-126, at least 2^127 from 2^128 on
            const float cut = cut_to_float(d), rz = __double2float_rz(d);
            const double m = fabs(d);
            if (m < 0x1p-126 ? cut != 0.0f : m < 0x1p127 ? !same(cut, rz) : !(fabsf(cut) >= 0x1p127f)) atomicAdd(bad + 7, 1ull);
            const double p = fabs(d), q = g.below(3) ? fabs(__longlong_as_double((long long)g.next())) : p;
            if (q == q && le_pos(p, q) != (p <= q)) atomicAdd(bad + 8, 1ull);
        }
    }
}

int main(int argc, char **argv)
{
    unsigned long long *d, h[20] = {};
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 1;
    for (int i = 1; i < argc; ++i) {
        RepParams R;
        memset(&R, 0, sizeof R);
        for (int k = 0; k < 3; ++k) set_axis(R, k, atof(argv[i]));
        check<<<64, 256>>>(R, 1000 * (unsigned long long)i, d, d + 10);
    }
    if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    for (int f = 0; f < 9; ++f) printf("%llu ", h[f]);
    printf("%llu\n", h[13]);
    return 0;
}
"""
FUNCTIONS = ["to_fix", "fix_to_double", "fix_position", "axis_add", "axis_ahead", "to_float", "to_double", "cut_to_float", "le_pos"]
BOXES = [51.3, 65.0, 200.0, 250.98, 277.5, 350.0, 501.9, 502.0, 511.9, 512.0, 600.0, 1000.0, 4096.0]


@pytest.mark.gpu
def test_integer_forms_give_the_bits_of_the_fp64_operations(tmp_path):
    src, exe = str(tmp_path / "t.cu"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run([build.NVCC, "-std=c++17", "-O3", "-fmad=false", *build.ARCH, "-I", build.CSRC, src, "-o", exe], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([exe] + [str(b) for b in BOXES], check=True, capture_output=True, text=True).stdout.split()
    assert dict(zip(FUNCTIONS, map(int, out))) == dict.fromkeys(FUNCTIONS, 0)
    assert int(out[-1]) > 64 * 64 * 256 * len(BOXES) // 3  # sums taken by integers


NAN_PROGRAM = r"""
#include <cstdio>
#include "tis_fixed.cuh"

// b[i]: with each b, NaNs of both signs, quiet and signalling, and the one inf - inf gives
__global__ void check(const double *b, int n, double inf, int *le)
{
    const unsigned long long bits[4] = {0x7ff8000000000000ull, 0xfff8000000000000ull, 0x7ff0000000000001ull, 0xffffffffffffffffull};
    for (int i = 0; i < n; ++i) {
        for (int k = 0; k < 4; ++k) *le += tis::le_pos(__longlong_as_double((long long)bits[k]), b[i]);
        *le += tis::le_pos(inf - inf, b[i]);
    }
}

int main()
{
    const double b[6] = {0.0, 4.9e-324, 1.0, 900.0, 1.7976931348623157e308, 1.0 / 0.0};
    double *d;
    int *le, h = -1;
    if (cudaMalloc(&d, sizeof b) != cudaSuccess || cudaMalloc(&le, sizeof h) != cudaSuccess) return 1;
    cudaMemcpy(d, b, sizeof b, cudaMemcpyHostToDevice);
    cudaMemset(le, 0, sizeof h);
    check<<<1, 1>>>(d, 6, 1.0 / 0.0, le);
    if (cudaMemcpy(&h, le, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("%d\n", h);
    return 0;
}
"""


@pytest.mark.gpu
def test_a_distance_that_is_no_number_is_within_no_cutoff(tmp_path):
    src, exe = str(tmp_path / "t.cu"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(NAN_PROGRAM)
    subprocess.run([build.NVCC, "-std=c++17", "-O3", *build.ARCH, "-I", build.CSRC, src, "-o", exe], check=True,
                   capture_output=True, text=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split() == ["0"]
