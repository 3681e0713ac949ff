/*
 * Arithmetic shortcuts of the shading kernels that give the plain form's
 * result: the sampler's division by a known divisor and the quick cases of
 * the light estimate.  Host + device, so that a CPU test can hold these
 * functions themselves against the plain forms.
 */
#ifndef PSY_SHADE_MATH_H
#define PSY_SHADE_MATH_H

#include "psy_math.h"
#include "psy_libm.cuh"

#if defined(__CUDACC__)
#define PSY_D_NOINLINE static __device__ __noinline__
#else
#define PSY_D_NOINLINE static
#endif

namespace psy {

#define PSY_HPI_D (PSY_PI_D / 2.0)
#define PSY_INV_PI_D (1.0 / PSY_PI_D)

// x divided by d, with recip = floor(2^32 / d), d < 2^16.  The quotient
// x * recip / 2^32 is right or one too small (x * (2^32 - recip * d) < 2^32 *
// d), and the remainder tells which.  (The two hardware-less divisions that a
// digit group took before were most of a sample's instructions.)
struct Division {
	uint32_t q, r;
};
PSY_HD Division divide_by(uint32_t x, uint32_t d, uint32_t recip) {
	Division v;
#if defined(__CUDA_ARCH__)
	v.q = __umulhi(x, recip);
#else
	v.q = (uint32_t)(((uint64_t)x * recip) >> 32);
#endif
	v.r = x - v.q * d;
	if (v.r >= d) {
		v.r -= d;
		++v.q;
	}
	return v;
}

// sphere_lambert (utils/monte_carlo.hpp:207-233) in two parts.
// (The reference takes 1 - x of a float x in double and rounds to float.  The
// double difference is exact but for x below 2^-29 or beyond 2^53, where it
// rounds like the float one, so the float subtraction gives the same bits.)
//
// The cosine tests: |cos a - cos b| <= |a - b|, so where nlcos lies 1e-3 off
// a limit's cosine (0, +-sin r), the angle lies as far off the limit; rsin is
// off sin r by at most 2.5e-4 (the rounding of rcos^2) and the arc cosines
// of the angle tests by less than 1e-6, so both tests agree there.  They
// spare the arc cosines, and where the cap lies wholly above or below the
// horizon (most nodes of a light tree walk) all arc functions.  An nlcos past
// +-1 by rounding (its arc cosine is NaN) takes the angle tests.
enum : int { CAP_ABOVE, CAP_MOSTLY_ABOVE, CAP_MOSTLY_BELOW, CAP_BELOW, CAP_UNSURE };
PSY_HD int cap_case(float nlcos, float rsin2) {
	// (on squares: the margin is far above their rounding)
	const float m = 1e-3f;
	const float c = fabsf(nlcos), in = c + m, out = c - m;
	if (out > 0.0f) {
		if (out * out > rsin2) return c <= 1.0f ? (nlcos > 0.0f ? CAP_ABOVE : CAP_BELOW) : CAP_UNSURE;
		if (in * in < rsin2) return nlcos > 0.0f ? CAP_MOSTLY_ABOVE : CAP_MOSTLY_BELOW;
	}
	return CAP_UNSURE;
}

// What is quick: the estimate of a cap wholly above or below the horizon, or
// (cut: cap_case, else -1) that sphere_lambert_cut has to tell.
struct CapEstimate {
	float est, rsin2;
	int cut;
};
PSY_HD CapEstimate sphere_lambert_quick(float nlcos, float rcos) {
	CapEstimate e;
	e.rsin2 = 1.0f - rcos * rcos;  // (float)(1.0 - (double)..)
	const int c = cap_case(nlcos, e.rsin2);
	e.est = c == CAP_ABOVE ? nlcos * e.rsin2 : 0.0f;
	e.cut = c != CAP_ABOVE && c != CAP_BELOW ? c : -1;
	return e;
}

// A cap that the horizon cuts, or may (c: cap_case).
PSY_D_NOINLINE float sphere_lambert_cut(float nlcos, float rcos, float rsin2, int c) {
	if (c == CAP_UNSURE) {
		const float nl = lm_acosf(nlcos);
		const float r = lm_acosf(rcos);
		if ((double)nl < (PSY_HPI_D - (double)r)) return nlcos * rsin2;
		if ((double)nl < PSY_HPI_D) c = CAP_MOSTLY_ABOVE;
		else if ((double)nl < (PSY_HPI_D + (double)r)) c = CAP_MOSTLY_BELOW;
		else return 0.0f;
	}
	const float nlsin = (float)sqrt(1.0 - (double)(nlcos * nlcos));
	const float rsin = sqrtf(rsin2);
	const float ysin = rcos / nlsin;
	const float ycos2 = 1.0f - ysin * ysin;  // (float)(1.0 - (double)..)
	const float ycos = sqrtf(ycos2);
	const float g = (float)(((((-2.0 * (double)nlsin) * (double)rcos) * (double)ycos) + PSY_HPI_D) -
	                        (double)lm_asinf(ysin) + (double)(ysin * ycos));
	const float h = nlcos * ((ycos * sqrtf(rsin2 - ycos2)) + (rsin2 * lm_asinf(ycos / rsin)));
	if (c == CAP_MOSTLY_ABOVE) return (nlcos * rsin2) + g - h;
	return (float)((double)(g + h) * PSY_INV_PI_D);
}

}  // namespace psy

#endif
