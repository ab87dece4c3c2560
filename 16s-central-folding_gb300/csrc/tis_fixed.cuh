// Conversions, sums and comparisons of FP64 values on integers, with the results of the FP64
// operations bit for bit: GB300 has 64-bit conversions and FP64 arithmetic at 1/64 of its
// integer rate.  set_axis forms the constants they need; tests/test_device_math.py runs
// every function here, and to_fix, on the GPU against the operation it stands for.
#pragma once
#include <algorithm>
#include <cmath>

#include "tis_device.cuh"

namespace tis {

// the constants of axis k of a box side L (host)
inline void set_axis(RepParams &R, int k, double L)
{
    auto high = [](double v) {
        uint64_t bits;
        memcpy(&bits, &v, 8);
        return (unsigned)(bits >> 32);
    };
    R.box[k] = L;
    R.hbox[k] = 0.5 * L;
    R.qinv[k] = 4294967296.0 / L;
    R.qstep[k] = (float)(L / 4294967296.0);
    int e2l, eq, e;  // 2 L < 2^e2l, qinv < 2^eq, 1.02 L < 2^e
    std::frexp(2.0 * L, &e2l);
    std::frexp(R.qinv[k], &eq);
    std::frexp(1.02 * L, &e);
    R.qx[k].q = (unsigned long long)std::ldexp(R.qinv[k], 64 - eq);
    R.qx[k].hi2l = high(2.0 * L);
    R.qx[k].sh = 1022 + e2l;
    R.qx[k].fb = 64 - eq - e2l - 1;
    R.ax[k].lo = (unsigned)(1023 + e - 10) << 20;
    R.ax[k].span = high(1.01 * L) - R.ax[k].lo;
    R.ax[k].step = std::ldexp(1.0f, e - 40);
    const float u2 = R.ax[k].step * R.ax[k].step;
    R.e2min = std::max(k ? R.e2min : 0.0f, 1.3e11f * u2);
    R.e2pad = std::max(k ? R.e2pad : 1.0e-30f, 1.0e3f * u2);
}

// (double)v by integer operations while v fits the 53 bits of a double's significand
__device__ __forceinline__ double fix_to_double(long long v)
{
    const unsigned long long m = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    if (m >> 53) return (double)v;
    const int z = __clzll((long long)m);  // 11 .. 64
    unsigned long long b = ((m << z) << 1) >> 12;  // the significand below its leading one
    b |= (unsigned long long)(unsigned)(1086 - z) << 52;
    if (m == 0) b = 0;
    return __longlong_as_double((long long)(b | ((unsigned long long)v & 0x8000000000000000ull)));
}

// floor(x qinv) modulo 2^32 of axis c, as __double2ll_rd(x * qinv[c]) gives it.  For
// 0 <= x < 2 L by integers: X = x 2^(63 - B) (2 L <= 2^B) times qinv 2^k, of which the
// high word has fb = k - B - 1 fraction bits (28 to 30).  It lies below the exact product
// by less than 2^-26; the FP64 product is rounded by at most 2^-21, which can only move
// its floor when the fraction lies within 2^-20 of one: those, and other x, take the FP64 form.
__device__ __forceinline__ int fix_position(const RepParams *R, int c, double x)
{
    const int hi = __double2hiint(x);
    if ((unsigned)hi < R->qx[c].hi2l) {
        const int s = R->qx[c].sh - (hi >> 20);
        const unsigned long long m = ((unsigned long long)(unsigned)((hi & 0xfffff) | 0x100000) << 32 | (unsigned)__double2loint(x)) << 10;
        const unsigned long long v = __umul64hi(s < 64 ? m >> s : 0ull, R->qx[c].q);
        const int fb = R->qx[c].fb;
        const unsigned fr = (unsigned)v & ((1u << fb) - 1u);
        if (fr < (1u << fb) - (1u << (fb - 20))) return (int)(unsigned)(v >> fb);
    }
    return (int)(unsigned)__double2ll_rd(x * R->qinv[c]);
}

// Sums of positions by integers, rounded as FP64 rounds them.  Full blocks use them, where
// the FP64 pipe is what the integrator waits for (twelve of its 27 operations per particle
// become some 200 integer instructions, 56 cycles of issue for 192 of the pipe: step of 16
// large replicas 194.1 -> 187.6 us, of 64 replicas 83.1 -> 82.5 us); a handle of few particles
// waits for the chain of one block, which they lengthen (one replica 19.8 -> 20.6 us).
// x in units of 2^(E - 64) (2^E > 1.02 box), exactly, for 2^(E - 10) <= x < 1.01 box
__device__ __forceinline__ bool axis_fix(const RepParams *R, int c, double x, unsigned long long &v)
{
    const unsigned hi = (unsigned)__double2hiint(x), o = hi - R->ax[c].lo;
    v = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | (unsigned)__double2loint(x)) << (((o >> 20) + 2u) & 15u);
    return o < R->ax[c].span;
}

// the double nearest to v units, ties to even, for v >= 2^54
__device__ __forceinline__ double axis_value(const RepParams *R, int c, unsigned long long v)
{
    const unsigned z = (unsigned)__clz((int)(v >> 32));  // 0 .. 9
    const unsigned long long w = v << z;
    const unsigned low = (unsigned)w, up = (low & 0x7ffu) + ((low >> 11) & 1u) > 0x400u;
    return __longlong_as_double((long long)((w >> 11) + ((unsigned long long)(R->ax[c].lo + (8u << 20) - (z << 20)) << 32) + up));
}

// a shift s in the same units, rounded to odd, so that its sum with a position rounds as the
// exact one does; kNoShift when |s| >= 2^(E - 10)
constexpr long long kNoShift = (long long)0x8000000000000000ull;
__device__ __forceinline__ long long shift_fix(const RepParams *R, int c, double s)
{
    const unsigned hi = (unsigned)__double2hiint(s), a = hi & 0x7fffffffu;
    if (a >= R->ax[c].lo) return kNoShift;
    if (s == 0.0) return 0;
    const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | (unsigned)__double2loint(s)) << 1;
    const unsigned r = (R->ax[c].lo >> 20) - 1u - (a >> 20);
    unsigned long long v = r < 64u ? m >> r : 0ull;
    if (r >= 64u || v << r != m) v |= 1ull;
    return (int)hi < 0 ? -(long long)v : (long long)v;
}

// the recentring shift: s, and where positions are summed by integers (I) the same as fix units
template <bool I>
struct Shift {
    double s[3];
    __device__ __forceinline__ void set(const RepParams *, int c, double v) { s[c] = v; }
};
template <>
struct Shift<true> {
    double s[3];
    long long fix[3];
    __device__ __forceinline__ void set(const RepParams *R, int c, double v)
    {
        s[c] = v;
        fix[c] = shift_fix(R, c, v);
    }
};

// x + the shift of axis c
template <bool I>
__device__ __forceinline__ double axis_add(const RepParams *R, int c, double x, const Shift<I> &sh)
{
    if constexpr (!I) return x + sh.s[c];
    else {
        unsigned long long v;
        const long long S = sh.fix[c];
        const bool ok = axis_fix(R, c, x, v) && S != kNoShift;
        v += (unsigned long long)S;
        return ok && v >= (1ull << 54) ? axis_value(R, c, v) : x + sh.s[c];
    }
}

// x as a float, its significand cut to 24 bits (0 below 2^-126, huge from 2^128 on)
__device__ __forceinline__ float cut_to_float(double x)
{
    const int hi = __double2hiint(x), a = hi & 0x7fffffff;
    const int f = __funnelshift_l((unsigned)__double2loint(x), (unsigned)(a - 0x38000000), 3);
    const float m = a < 0x38100000 ? 0.0f : a >= 0x47f00000 ? 3.0e38f : __int_as_float(f);
    return hi < 0 ? -m : m;
}

// x0 + (x0 - o0), the position before the velocity's change; a: x0 - o0 in FP32.  2 x0 - o0
// rounded once, as FP64 mode has it, is also what x0 + (x0 - o0) gives while the difference is
// exact: by integers while both are a usual place and the difference below 2^(E - 10)
template <bool D, bool I>
__device__ __forceinline__ double axis_ahead(const RepParams *R, int c, double x0, double o0, float &a)
{
    if constexpr (I) {
        unsigned long long X, O;
        const bool in = axis_fix(R, c, x0, X) & axis_fix(R, c, o0, O);
        const long long dif = (long long)(X - O);
        X += (unsigned long long)dif;
        if (in && (unsigned long long)(dif + (1ll << 54)) < (1ull << 55) && X >= (1ull << 54)) {
            a = (float)(int)(dif >> 24) * R->ax[c].step;
            return axis_value(R, c, X);
        }
    }
    const double e = x0 - o0;
    a = cut_to_float(e);
    return D ? __dsub_rn(__dmul_rn(2.0, x0), o0) : x0 + e;
}

// a <= b for b >= 0 and an a that is not negative or is NaN, of either sign
__device__ __forceinline__ bool le_pos(double a, double b)
{
    return (unsigned long long)__double_as_longlong(a) <= (unsigned long long)__double_as_longlong(b);
}

// round-to-nearest conversions by integers where both values are normal numbers
__device__ __forceinline__ float to_float(double x)
{
    const int hi = __double2hiint(x), m = hi & 0x7fffffff;
    if ((unsigned)(m - 0x38100000) < 0x0fd00000u) {  // 2^-126 <= |x| < 2^127
        const unsigned lo = (unsigned)__double2loint(x);
        unsigned f = __funnelshift_l(lo, (unsigned)(m - 0x38000000), 3);
        const unsigned rest = lo & 0x1fffffffu;  // below FP32's last place; half of it is 2^28
        f += rest > 0x10000000u || (rest == 0x10000000u && (f & 1u)) ? 1u : 0u;
        return __uint_as_float(f | ((unsigned)hi & 0x80000000u));
    }
    return (float)x;
}
__device__ __forceinline__ double to_double(float x)
{
    const unsigned b = __float_as_uint(x), m = b & 0x7fffffffu;
    if (m - 0x00800000u < 0x7f000000u) return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + 0x38000000u)), (int)(b << 29));
    return (double)x;
}
__device__ __forceinline__ double to_double(double x) { return x; }
template <class T>
__device__ __forceinline__ T to_real(double x)
{
    if constexpr (sizeof(T) == 4) return to_float(x);
    else return x;
}

}  // namespace tis
