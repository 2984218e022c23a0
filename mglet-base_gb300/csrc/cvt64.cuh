// cvt64.cuh -- conversions between FP64 and FP32 as integer arithmetic.
//
// For kernels bound by the FP64 pipe: the rest of a split, x - (double)hi, is an FP64
// subtraction between two conversions, here a few integer instructions.  512 grids of
// 24^3: the divergence 177 -> 125 us; on 448 grids of 16^3 the restriction 24.3 ->
// 22.7, bound_pressure 8.9 -> 8.2.  Kernels bound by the issue of instructions keep the
// casts (the fluxes with a viscosity field: 447 us with casts, 626 with these).  Same
// bits as the casts: values outside the ranges below take them.
#pragma once

namespace mg {

// (float)x, round to nearest even: exponent of x in a normal float's range
__device__ __forceinline__ float cvt_float(double x) {
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    const unsigned e = (h >> 20) & 0x7ffu;
    if (e - 897u <= 253u) {
        unsigned f = __funnelshift_l(l, (h & 0x7fffffffu) - 0x38000000u, 3);
        f += ((l & 0x1fffffffu) + 0x0fffffffu + (f & 1u)) >> 29;   // (a carry goes into the exponent)
        return __uint_as_float(f | (h & 0x80000000u));
    }
    return ((h & 0x7fffffffu) | l) == 0 ? __uint_as_float(h) : (float)x;
}

// (double)x
__device__ __forceinline__ double cvt_double(float x) {
    const unsigned b = __float_as_uint(x), m = b & 0x7fffffffu;
    if (m - 0x00800000u < 0x7f000000u)
        return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + 0x38000000u)), (int)(b << 29));
    return m == 0 ? __hiloint2double((int)b, 0) : (double)x;
}

// hi = (float)x, lo = (float)(x - (double)hi): exponent of x from -74, so that the
// last bit of the rest is a normal float
__device__ __forceinline__ void cvt_split(double x, float& hi, float& lo) {
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    const unsigned e = (h >> 20) & 0x7ffu;
    if (e - 949u <= 200u) {
        unsigned f = __funnelshift_l(l, (h & 0x7fffffffu) - 0x38000000u, 3);
        const unsigned rem = l & 0x1fffffffu, up = (rem + 0x0fffffffu + (f & 1u)) >> 29;
        f += up;
        hi = __uint_as_float(f | (h & 0x80000000u));
        // the signed rest in units of 2^(e - 1023 - 52), rounded once
        const float r = __int2float_rn((int)rem - (int)(up << 29)) * __uint_as_float((e - 948u) << 23);
        lo = h & 0x80000000u ? 0.f - r : r;
        return;
    }
    if (((h & 0x7fffffffu) | l) == 0) {
        hi = __uint_as_float(h);
        lo = 0.f;
        return;
    }
    hi = (float)x;
    lo = (float)(x - (double)hi);
}

}  // namespace mg
