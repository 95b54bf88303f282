// Host shim over shape_atrophy_gb300/csrc/sa_limb.cuh (fixed-point sums of products) for the CPU tests.
#include "../shape_atrophy_gb300/csrc/sa_limb.cuh"

// sum of a[k] u[k] as the kernels form it; the frames are the largest exponent fields of a and of u (eA, eU at least)
extern "C" double limb_dot(const double *a, const double *u, int n, int eA, int eU)
{
	for (int k = 0; k < n; ++k) {
		if (sa::fx_exp(a[k]) > eA) eA = sa::fx_exp(a[k]);
		if (sa::fx_exp(u[k]) > eU) eU = sa::fx_exp(u[k]);
	}
	sa::LimbSum s = sa::limb_zero();
	for (int k = 0; k < n; ++k) {
		int a1 = 0, a0 = 0, u1 = 0, u0 = 0;
		if (eA < 2047) sa::limb_matrix(a[k], eA, a1, a0);
		sa::limb_vector(u[k], eU, u1, u0);
		sa::limb_mac(s, a1, a0, u1, u0);
	}
	return sa::limb_to_double(s, eA, eU);
}

extern "C" int limb_max_terms() { return sa::kLimbMaxTerms; }
