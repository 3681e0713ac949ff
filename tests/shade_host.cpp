// Test harness: the shading shortcuts (shade_math.h) compiled for the host,
// beside the forms that they stand for.
#include "shade_math.h"

using namespace psy;

// x / d and x % d as the sampler takes them
extern "C" void divisions(unsigned n, const uint32_t* x, uint32_t d, uint32_t* q, uint32_t* r) {
	for (unsigned i = 0; i < n; ++i) {
		const Division v = divide_by(x[i], d, (uint32_t)((1ull << 32) / d));
		q[i] = v.q;
		r[i] = v.r;
	}
}

// sphere_lambert as the light tree's walk takes it; cut[i]: the case it came
// to, -1 for the quick ones
extern "C" void lambert(unsigned n, const float* nlcos, const float* rcos, float* out, int* cut) {
	for (unsigned i = 0; i < n; ++i) {
		const CapEstimate e = sphere_lambert_quick(nlcos[i], rcos[i]);
		cut[i] = e.cut;
		out[i] = e.cut < 0 ? e.est : sphere_lambert_cut(nlcos[i], rcos[i], e.rsin2, e.cut);
	}
}

// sphere_lambert with every operation of the reference (utils/monte_carlo.hpp:
// 207-233): arc functions throughout, 1 - x in double
extern "C" void lambert_plain(unsigned n, const float* nlcos_, const float* rcos_, float* out) {
	for (unsigned i = 0; i < n; ++i) {
		const float nlcos = nlcos_[i], rcos = rcos_[i];
		const double hpi = PSY_PI_D / 2.0;
		const float nlsin = (float)sqrt(1.0 - (double)(nlcos * nlcos));
		const float rsin2 = (float)(1.0 - (double)(rcos * rcos));
		const float rsin = sqrtf(rsin2), ysin = rcos / nlsin;
		const float ycos2 = (float)(1.0 - (double)(ysin * ysin));
		const float ycos = sqrtf(ycos2);
		const float g = (float)(((((-2.0 * (double)nlsin) * (double)rcos) * (double)ycos) + hpi) - (double)lm_asinf(ysin) +
		                        (double)(ysin * ycos));
		const float h = nlcos * ((ycos * sqrtf(rsin2 - ycos2)) + (rsin2 * lm_asinf(ycos / rsin)));
		const double nl = (double)lm_acosf(nlcos), r = (double)lm_acosf(rcos);
		out[i] = nl < hpi - r ? nlcos * rsin2
		         : nl < hpi ? (nlcos * rsin2) + g - h
		         : nl < hpi + r ? (float)((double)(g + h) * (1.0 / PSY_PI_D)) : 0.0f;
	}
}

// the place of a time among the samples of a sequence
extern "C" void positions(unsigned n, const float* time, int count, int* first, int* last, float* alpha) {
	for (unsigned i = 0; i < n; ++i) {
		const SeqPos p = seq_pos(time[i], count);
		first[i] = p.i0;
		last[i] = p.single ? p.i0 : p.i0 + 1;
		alpha[i] = p.nalpha;
	}
}
