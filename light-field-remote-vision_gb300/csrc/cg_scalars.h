// cg_scalars.h -- scalar arithmetic of the corrected CG (k_cg_strip) that carries more than FP32 on the FP32 pipe: an FP64
// operation of this GPU has a latency of dozens of cycles and holds a narrow pipe 16 cycles a warp, and every block waits
// for these scalars between two iterations. Plain operators, each rounded to nearest, so the host computes the same.
#pragma once

#ifdef __CUDACC__
#define LFRV_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define LFRV_HD inline
#endif

namespace lfrv {

// a / b for positive FP64 a and b, rounded to FP32: the quotient of the rounded operands, corrected by what it leaves of a
// and by the operands' low parts. Within 2^-18 of half a unit in the last place, as the FP64 quotient rounded once; the
// quotient of the rounded operands alone is off by up to one and a half.
LFRV_HD float cg_quotient(double a, double b) {
    const float ah = (float)a, bh = (float)b;
    if (!(ah > 1e-25f && ah < 1e25f && bh > 1e-25f && bh < 1e25f)) return (float)(a / b);
    const float al = (float)(a - (double)ah), bl = (float)(b - (double)bh);
    const float q = ah / bh;
    return fmaf(fmaf(-q, bl, fmaf(-q, bh, ah) + al), 1.0f / bh, q);
}

// An unevaluated sum of two floats, and their addition (Knuth's two-sum; the low part holds the rounding errors).
struct CgSum {
    float hi, lo;
};
LFRV_HD CgSum cg_add(CgSum a, CgSum b) {
    const float s = a.hi + b.hi, t = s - a.hi;
    const float err = (a.hi - (s - t)) + (b.hi - t);
    return {s, (a.lo + b.lo) + err};
}
// The sum: the rounding errors of an infinite one are not numbers, and dropped.
LFRV_HD CgSum cg_result(CgSum a) { return {a.hi, fabsf(a.hi) <= 3.402823466e38f ? a.lo : 0.f}; }

}  // namespace lfrv
