/* x / 3 without a division: the quotient by the rounded reciprocal,
 * corrected once by its remainder (Markstein's theorem on quotients by a
 * correctly rounded reciprocal). The remainder x - 3q is a small multiple of
 * q's last place, so it is exact down to the subnormal numbers, and the
 * result is x / 3 correctly rounded for every finite x. Infinities, NaN and
 * zeros (and subnormals below 2^-1042, whose quotient is right as it is) have
 * no remainder to correct by: there the quotient is the result. They are told
 * by q's high word: FP64 comparisons cost helium ticks 0.3%, this nothing.
 * Plain C, so that a host program can hold it against the division. */
#ifndef PSG_DIV3_H
#define PSG_DIV3_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define PSG_HD __host__ __device__ __forceinline__
#else
#define PSG_HD static inline
#endif

PSG_HD double psg_div3(double x) {
	const double y = 1.0 / 3.0, q = x * y;
	const double c = fma(fma(-3.0, q, x), y, q);
#ifdef __CUDA_ARCH__
	const uint32_t high = (uint32_t)__double2hiint(q);
#else
	uint64_t w;
	memcpy(&w, &q, 8);
	const uint32_t high = (uint32_t)(w >> 32);
#endif
	/* 1 ... 0x7fefffff: the normal numbers and the larger subnormals */
	return (high & 0x7fffffffu) - 1u < 0x7fefffffu ? c : q;
}

#endif
