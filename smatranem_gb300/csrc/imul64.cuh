/*
 * FP64 products off the FP64 pipe.
 */
#ifndef SMATRAN_IMUL64_CUH
#define SMATRAN_IMUL64_CUH

#include <cuda_runtime.h>

namespace smat {

/* a b rounded to nearest (ties to even) on the integer pipes: the 53 x 53-bit
 * product of the mantissas, normalised by at most one place, rounded on its
 * low 64 bits; operands and results outside the normal range go through the
 * FP64 unit.  The same bits as a * b.  By itself 2.0 products a clock and SM
 * against the FP64 pipe's 1.7, and beside it 2.7 operations where half are
 * these products (measured): kernels bound by that pipe send their products
 * here and keep it for the additions. */
template <bool NEG = false> /* -a b: the sign bit (a negated double as an operand would cost a DADD) */
__device__ __forceinline__ double imul(double a, double b)
{
    const unsigned ah = (unsigned)__double2hiint(a), bh = (unsigned)__double2hiint(b);
    const unsigned ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
    const unsigned long long ma = ((unsigned long long)((ah & 0xfffffu) | 0x100000u) << 32 | (unsigned)__double2loint(a)) << 11;
    const unsigned long long mb = (unsigned long long)((bh & 0xfffffu) | 0x100000u) << 32 | (unsigned)__double2loint(b);
    unsigned long long hi = __umul64hi(ma, mb), lo = ma * mb; /* hi in [2^51, 2^53) */
    const unsigned up = (unsigned)(hi >> 52);
    const unsigned e = ea + eb - 1024u + up; /* the biased exponent less one: hi's leading bit adds it */
    if (!up) {
        hi = hi << 1 | lo >> 63;
        lo <<= 1;
    }
    const unsigned r = (unsigned)(lo >> 63) & (unsigned)(((lo << 1) != 0) | ((unsigned)hi & 1u));
    const unsigned sign = ((ah ^ bh) & 0x80000000u) ^ (NEG ? 0x80000000u : 0u);
    if (ea - 1u >= 2046u || eb - 1u >= 2046u || e >= 2045u) {
        /* zero times a finite number: fields that no wave has reached yet */
        const bool za = ((ah << 1) | (unsigned)__double2loint(a)) == 0, zb = ((bh << 1) | (unsigned)__double2loint(b)) == 0;
        if ((za && eb != 2047u) || (zb && ea != 2047u)) return __hiloint2double((int)sign, 0);
        return NEG ? -(a * b) : a * b;
    }
    return __longlong_as_double((long long)(((unsigned long long)(sign + (e << 20)) << 32) + hi + r));
}

} // namespace smat

#endif
