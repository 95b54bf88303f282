// Host shim over shape_atrophy_gb300/csrc/sa_pairfix.cuh (fixed-point pair terms) for the CPU tests.
#include "../shape_atrophy_gb300/csrc/sa_pairfix.cuh"
#include <cstring>

static const unsigned long long kTab[256] = {SA_PAIR_EXP_TABLE};

// K_c K_d v of a pair with squared distance d2 in widths, directions u, w of length at most 1 and 0 <= v < 1
extern "C" double pair_value(int ck, int dk, double d2, const double *u, const double *w, double v)
{
	unsigned long long b;
	if (ck == 'C') d2 += 1.0;
	std::memcpy(&b, &d2, 8);
	int m, uh[3], ul[3], wh[3], wl[3];
	const unsigned long long k = sa::pair_centre(ck, (unsigned) (b >> 32), (unsigned) b, m, kTab);
	for (int d = 0; d < 3; ++d) { sa::pair_digits(u[d], uh[d], ul[d]); sa::pair_digits(w[d], wh[d], wl[d]); }
	bool neg;
	const unsigned long long a = sa::pair_angle<3>(uh, ul, wh, wl, neg);
	const double t = (double) sa::pair_term(k, m, dk == 'B' ? sa::pair_mulh(a, a) << 1 : a, (unsigned long long) (v * 0x1p63)) * 0x1p-61;
	return neg && dk == 'L' ? -t : t;
}

extern "C" int pair_frame(double n2) { return sa::pair_frame(n2); }

extern "C" double pair_exp(double x)
{
	unsigned long long b;
	std::memcpy(&b, &x, 8);
	int m;
	const unsigned long long e = sa::pair_exp(sa::pair_fix((unsigned) (b >> 32), (unsigned) b), m, kTab);
	return sa::pair_double(e, 63 + m);
}
