// Host shim over the column scales of shape_atrophy_gb300/csrc/sa_limb.cuh for the CPU tests.
#include "../shape_atrophy_gb300/csrc/sa_limb.cuh"

// sum of a[k] u[k] with the column scales 2^s[k], as the velocity CG forms it (the row's own scale: own): digits as long as
// the row can take when longer is set; *extra: their extra bits
extern "C" double limb_scaled_dot(const double *a, const double *u, const int *s, int n, int own, int longer, int *extra)
{
	int eA = sa::kLimbNone, eU = 1;
	float top = 0.0f, sum = 0.0f;
	for (int k = 0; k < n; ++k) {
		const int x = sa::limb_scaled_exp(a[k], s[k]), y = sa::fx_exp(__builtin_ldexp(u[k], -s[k]));
		if (x > eA) eA = x;
		if (y > eU) eU = y;
		const float f = sa::limb_float_above(a[k], s[k] + own);
		if (f > top) top = f;
		sum += f;
	}
	*extra = longer && eA < sa::kLimbBad ? sa::limb_extra(top, sum, eA + own) : 0;
	if (eA < sa::kLimbBad) eA -= *extra;
	sa::LimbSum t = sa::limb_zero();
	for (int k = 0; k < n; ++k) {
		int a1 = 0, a0 = 0, u1 = 0, u0 = 0;
		if (eA < sa::kLimbBad) sa::limb_matrix_wide(a[k], eA - s[k], a1, a0);
		sa::limb_vector(__builtin_ldexp(u[k], -s[k]), eU, u1, u0);
		sa::limb_mac(t, a1, a0, u1, u0);
	}
	return sa::limb_scaled_to_double(t, eA, eU);
}

extern "C" float limb_above(double v, int s) { return sa::limb_float_above(v, s); }
