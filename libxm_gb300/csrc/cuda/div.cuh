/*
 * FP64 division on the integer and FP32 pipes.
 *
 * GB300's FP64 pipe issues 2 instructions a cycle on each SM; a division
 * there costs about a dozen of them, so that an element-wise division of
 * two arrays runs at an eighth of the memory's rate.  The quotient of two
 * 53-bit significands is a fixed-point problem that the integer pipe (64
 * 32-bit multiply-adds a cycle) solves nearly within the memory's time:
 * xm_div of 71 million elements in 259 blocks 1825 -> 400 us per call
 * (252 us of traffic), of 32448 elements 65 -> 18 us.
 *
 * Method: long division in two digits of 26 bits (Knuth, The Art of
 * Computer Programming 4.3.1, with a precomputed reciprocal).  A 32-bit
 * reciprocal of the divisor comes from the FP32 approximation and one
 * Newton step, and is lowered so that it never exceeds the true one; each
 * digit is then the true one or one below, the running remainder is exact
 * modulo 2^64 and at most twice the divisor, and one conditional step at the
 * end leaves quotient = floor(2^52 a / b) and 0 <= remainder < b.  Rounding
 * to nearest then needs only 2 * remainder > b: a tie would need a divisor
 * with a factor 2^53.  A zero dividend gives its zero directly (the diagonal
 * of an antisymmetric block); subnormal, infinite or NaN operands and
 * results near the ends of the range take the ordinary division.
 */
#ifndef XMG_DIV_CUH
#define XMG_DIV_CUH

#include <stdint.h>
#include <string.h>

namespace xmg {

__host__ __device__ __forceinline__ uint64_t div_bits(double x)
{
#ifdef __CUDA_ARCH__
	return (uint64_t)__double_as_longlong(x);
#else
	uint64_t b;
	memcpy(&b, &x, sizeof b);
	return b;
#endif
}

__host__ __device__ __forceinline__ double div_value(uint64_t b)
{
#ifdef __CUDA_ARCH__
	return __longlong_as_double((long long)b);
#else
	double x;
	memcpy(&x, &b, sizeof x);
	return x;
#endif
}

__host__ __device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
	return __umulhi(a, b);
#else
	return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

/* 1 / y for y in [1, 2) given by its 23 fraction bits, as a 32-bit fixed-
 * point number below 1, to about 2^-22 */
__host__ __device__ __forceinline__ uint32_t recip22(uint32_t frac)
{
	uint32_t u = 0x3f800000u | frac;
#ifdef __CUDA_ARCH__
	u = __float_as_uint(__fdividef(1.0f, __uint_as_float(u)));
#else
	float f;
	memcpy(&f, &u, sizeof f);
	f = 1.0f / f;
	memcpy(&u, &f, sizeof u);
#endif
	/* the approximation may leave [1/2, 1) by its last bit */
	if (u < 0x3f000000u)
		u = 0x3f000000u;
	return u >= 0x3f800000u ? 0xffffffffu : (0x800000u | (u & 0x7fffffu)) << 8;
}

/* x / y; bit for bit the IEEE quotient, rounded to nearest even */
__host__ __device__ __forceinline__ double div_f64(double x, double y)
{
	const uint64_t xb = div_bits(x), yb = div_bits(y);
	const int xe = (int)(xb >> 52) & 0x7ff, ye = (int)(yb >> 52) & 0x7ff;
	const uint64_t M = (1ull << 52) - 1, sign = (xb ^ yb) & (1ull << 63);
	uint64_t a = (xb & M) | (1ull << 52);
	const uint64_t b = (yb & M) | (1ull << 52);
	int e = xe - ye + 1023;

	if ((unsigned)(xe - 1) >= 2046u || (unsigned)(ye - 1) >= 2046u ||
	    e < 2 || e > 2045) {
		if ((xb << 1) == 0 && (unsigned)(ye - 1) < 2046u)
			return div_value(sign);
		return x / y;
	}
	if (a < b) {
		a <<= 1;
		e--;
	}
	/* b <= a < 2 b.  r ~ 2^84 / b: one Newton step (its own error is
	 * below 2^-42 of r; its truncated terms raise r by less than 4 units
	 * and lower it by less than 1), then 5 units lower: never above the
	 * true value, and below it by at most 6 units, 2^-28.4 of it */
	const uint32_t r0 = recip22((uint32_t)(b >> 29) & 0x7fffffu);
	const int32_t t = (int32_t)((1u << 31) - mulhi32((uint32_t)(b >> 21), r0));
	const uint32_t r = r0 - 5u +
	    (uint32_t)(((int64_t)t * (int64_t)(int32_t)(r0 >> 1)) >> 30);
	/* the leading 27 bits of 2^52 a / b, or one less */
	const uint32_t q1 = mulhi32((uint32_t)(a >> 22), r) >> 4;
	const uint64_t rem1 = (a << 26) - (uint64_t)q1 * b;
	/* the next 26 bits (27 where q1 was one less), or one less */
	const uint32_t q2 = mulhi32((uint32_t)(rem1 >> 23), r) >> 3;
	uint64_t rem = (rem1 << 26) - (uint64_t)q2 * b;
	uint64_t q = ((uint64_t)q1 << 26) + q2;
	if (rem >= b) {
		q++;
		rem -= b;
	}
	q += 2 * rem > b;
	/* q's leading bit adds one to the exponent field */
	return div_value(sign | (((uint64_t)(e - 1) << 52) + q));
}

} /* namespace xmg */

#endif
