// Host shim over the frames of shape_atrophy_gb300/csrc/sa_limb.cuh for the CPU tests.
#include "../shape_atrophy_gb300/csrc/sa_limb.cuh"

extern "C" int unit_frame(double eps) { return sa::limb_unit_frame(eps); }

// the value of an entry's digits in the frame eA: matrix entry (vec 0) or vector entry (vec 1)
extern "C" double digits_value(double a, int eA, int vec)
{
	int h = 0, l = 0;
	if (vec) sa::limb_vector(a, eA, h, l);
	else sa::limb_matrix(a, eA, h, l);
	return ((double) h * 268435456.0 + (double) l) * __builtin_ldexp(1.0, eA - (vec ? 1078 : 1077));
}
