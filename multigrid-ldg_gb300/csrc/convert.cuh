// convert.cuh -- FP32 <-> FP64 conversions on the integer pipes, and sums of
// float pairs.  Only the CUDA intrinsics named here are used, so that the
// functions can be compiled for the host with those defined and checked bit by
// bit.
#pragma once

namespace mg {

// GB300 converts two values per clock and SM (the FP64 pipes), which bounded
// the vector kernels: the direction update of 4.2 million entries took 62 us
// with five conversions and subtractions per entry, against 27 us of HBM
// traffic.

// (double)v: the exponent is rebiased and the mantissa shifted, exact for
// every normal value and zero; others take the conversion
__device__ __forceinline__ double widen(float v) {
    const unsigned u = __float_as_uint(v), e = (u >> 23) & 0xffu;
    const int hi = (int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20)));
    if (e - 1u < 254u) return __hiloint2double(hi, (int)(u << 29));
    return (u << 1) == 0u ? __hiloint2double((int)u, 0) : (double)v;
}
__device__ __forceinline__ double widen(double v) { return v; }

// (float)v, rounded to nearest even; values outside FP32's normal range (and
// non-finite ones) take the conversion
__device__ __forceinline__ float narrow(double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v), mag = u & 0x7fffffffffffffffULL;
    if ((unsigned)(mag >> 52) - 897u >= 253u) return (float)v;
    const unsigned long long r = (mag + 0x0fffffffULL + ((mag >> 29) & 1u)) >> 29;
    return __uint_as_float((unsigned)(r - (896ULL << 23)) | (unsigned)(u >> 32 & 0x80000000u));
}

// v = h + l: h the nearest FP32 value (ties away from zero), l the nearest to
// the rest; the rest is an integer below 2^29 times a power of two, so it
// needs no FP64 operation.  Magnitudes outside 2^-60 .. 2^100 are split with
// conversions.
__device__ __forceinline__ void split_pair(double v, float& h, float& l) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v), mag = u & 0x7fffffffffffffffULL;
    const unsigned e = (unsigned)(mag >> 52), sign = (unsigned)(u >> 32) & 0x80000000u;
    if (e - 963u < 160u) {
        const unsigned long long r = (mag + (1ULL << 28)) & ~((1ULL << 29) - 1);
        const int rest = (int)(long long)(mag - r);
        h = __uint_as_float((unsigned)((r >> 29) - (896ULL << 23)) | sign);
        l = __fmul_rn((float)rest, __uint_as_float(((e - 948u) << 23) | sign));
    } else {
        h = (float)v;
        l = (float)(v - (double)h);
    }
}

// Exact sum of two floats, s + err (Knuth's two-sum).
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
    const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return s;
}

// Sum of float pairs without the FP64 pipes: the two-sum errors of both parts
// are kept, so that the result is the FP64 sum of the pairs up to 2^-72 (a
// plain pair sum would add 2^-48 per term, 1.6 times the error of the
// products themselves for rows of 4 x 6).
struct PairSum {
    float h = 0.f, l = 0.f, w = 0.f;
    __device__ __forceinline__ void add(float ph, float pl) {
        float e, e2, e3;
        h = two_sum(h, ph, e);
        l = two_sum(l, two_sum(e, pl, e2), e3);
        w = __fadd_rn(w, __fadd_rn(e2, e3));
    }
    __device__ __forceinline__ double value() const { return widen(h) + (widen(l) + widen(w)); }
};

}  // namespace mg
