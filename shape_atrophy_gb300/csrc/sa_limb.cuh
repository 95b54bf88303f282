// sa_limb.cuh -- FP64 products summed on the integer pipes.
//
// GB300 issues one FP64 multiply-add per warp every 64 clocks on each SM sub-partition (1.60 per clock per SM
// measured), but a multiply-add of 32 x 32 -> 64 bit integers in about four.  A sum of products of
// doubles is therefore formed in fixed point: each factor is cut into signed digits ("limbs") relative to a
// common power of two, the digit products (below 2^57) are added in 64-bit integers, which is exact, and the
// sum is rounded to FP64 once.
//
//   matrix entry a of a row whose largest entry has the exponent field eA: va = rint(a 2^(1077 - eA)), |va| <= 2^55,
//     two digits va = a1 2^28 + a0: exact for entries above a quarter of the row's largest, the others off by at
//     most 2^-56 of twice the largest (one rounding of an FP64 sum over that row costs 2^-53 of the partial sum);
//   vector entry u of a set whose largest entry has the exponent field eU: vu = rint(u 2^(1078 - eU)), |vu| <= 2^56,
//     two digits vu = u1 2^28 + u0: exact for entries above an eighth of the largest, the others off by 2^-57 of
//     twice it;
//   sum va vu = 2^56 S2 + 2^28 S1 + S0, S2 = sum a1 u1, S1 = sum (a1 u0 + a0 u1), S0 = sum a0 u0, nothing dropped.  S1 is
//     formed as M - S2 - S0 from M = sum (a1 + a0)(u1 + u0) (Karatsuba's product), so a product takes three integer
//     multiply-adds, each about four clocks of a sub-partition, and two 32-bit additions.
// Each sum stays below 2^63 for up to kLimbMaxTerms products.  So a product with a vector is as good as FP64's in norm, not
// entry by entry: where a row's terms are 2^-k of its largest entry times the set's largest, it has k bits less.  A frame of 2047 (an Inf or NaN in the row or the set) gives
// NaN.  An entry above its frame has no digits (0 comes out): the caller's frame covers every entry, or the caller looks
// for such entries and gives NaN.
#pragma once
#include "sa_fixsum.cuh"

namespace sa {

constexpr int kLimbMaxTerms = 80;         // products per sum: 80 x 1.5 x 2^56 < 2^63

// the two digits of a matrix entry in the frame of its row's largest exponent field eA
SA_FX_HD void limb_matrix(double a, int eA, int &a1, int &a0)
{
	int e; unsigned long long m; bool neg;
	fx_parts(a, e, m, neg);
	const int d = eA - e;                                     // >= 0 in the frame
	const unsigned long long v = (unsigned) d < 64u ? (((m << 3) >> d) + 1ull) >> 1 : 0ull;
	const long long s = neg ? -(long long) v : (long long) v;
	const long long lo = ((s + (1ll << 27)) & ((1ll << 28) - 1)) - (1ll << 27);
	a1 = (int) ((s - lo) >> 28);
	a0 = (int) lo;
}

// the two digits of a vector entry in the frame of the set's largest exponent field eU
SA_FX_HD void limb_vector(double u, int eU, int &u1, int &u0)
{
	int e; unsigned long long m; bool neg;
	fx_parts(u, e, m, neg);
	const int d = eU - e;                                     // >= 0 in the frame
	const unsigned long long v = (unsigned) d < 64u ? (((m << 4) >> d) + 1ull) >> 1 : 0ull;
	const long long s = neg ? -(long long) v : (long long) v;
	const int lo = (int) (((unsigned) s + (1u << 27)) & ((1u << 28) - 1u)) - (1 << 27);
	u1 = (int) ((s - lo) >> 28);
	u0 = lo;
}

// the frame of a matrix whose off-diagonal entries are 1 at most in size and whose diagonal entries are 1 + eps
inline int limb_unit_frame(double eps)
{
	const int one = fx_exp(1.0), d = fx_exp(1.0 + eps);
	return d > one ? d : one;
}

struct LimbSum { long long s2, sm, s0; };    // S2, M, S0

SA_FX_HD LimbSum limb_zero() { return LimbSum{0ll, 0ll, 0ll}; }

SA_FX_HD void limb_mad(long long &t, int a, int b)
{
#if defined(__CUDA_ARCH__)
	asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(a), "r"(b));
#else
	t += (long long) a * b;
#endif
}

SA_FX_HD void limb_mac(LimbSum &t, int a1, int a0, int u1, int u0)
{
	limb_mad(t.s2, a1, u1);
	limb_mad(t.sm, a1 + a0, u1 + u0);
	limb_mad(t.s0, a0, u0);
}

// v << sh in 128 bits, 0 <= sh < 64
SA_FX_HD Fx fx_shl(long long v, int sh)
{
	return Fx{(unsigned long long) v << sh, sh ? (unsigned long long) (v >> (64 - sh)) : (unsigned long long) (v >> 63)};
}

// the sum as one 128-bit integer
SA_FX_HD Fx limb_fixed(const LimbSum &t)
{
	return fx_add(fx_shl(t.s2, 56), fx_add(fx_shl(t.sm - t.s2 - t.s0, 28), fx_shl(t.s0, 0)));
}

SA_FX_HD double limb_bits(unsigned long long bits)
{
#if defined(__CUDA_ARCH__)
	return __longlong_as_double((long long) bits);
#else
	double d;
	__builtin_memcpy(&d, &bits, 8);
	return d;
#endif
}

// results outside the normal range: |value| = f 2^(top - 1150), bit 127 of f set
SA_FX_HD double limb_edge(Fx f, bool neg, int top)
{
	if (top > 2046) return limb_bits((neg ? 1ull << 63 : 0ull) | (2047ull << 52));
	Fx g{(f.lo >> 1) | (f.hi << 63), f.hi >> 1};              // bit 126: fx_to_double takes signed values
	if (top < -52) return 0.0;                                // below half the smallest subnormal
	const double v = fx_to_double(g, top - 14);
	return neg ? -v : v;
}

// f 2^(em - 1135) (signed f) as a double, rounded to nearest, ties to even.  One copy for all callers on the device:
// the solve kernels run their loop body once per iteration, so its length costs instruction fetches.
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
double limb_round(Fx f, int em)
{
	const bool neg = (long long) f.hi < 0;
	if (neg) f = fx_neg(f);
	int top = em + 15;                                        // exponent field when bit 127 leads
	if (f.hi == 0ull) { f.hi = f.lo; f.lo = 0ull; top -= 64; }
	if (f.hi == 0ull) return 0.0;
	const int z = fx_clz64(f.hi);
	if (z) { f.hi = (f.hi << z) | (f.lo >> (64 - z)); f.lo <<= z; }
	top -= z;
	if (top < 1 || top > 2046) return limb_edge(f, neg, top); // subnormal, or too large
	// 64 leading bits with the rest as a sticky bit, rounded to 53
	const unsigned long long q = f.hi >> 11;
	const unsigned rem = ((unsigned) f.hi & 0x7FFu) | (f.lo ? 1u : 0u);
	const unsigned long long bits = ((unsigned long long) (top - 1) << 52) + q + (rem + (unsigned) (q & 1ull) > 0x400u ? 1ull : 0ull);
	return limb_bits(bits | (neg ? 1ull << 63 : 0ull));
}

// Column scales.  Where columns differ much in size (a stiff layer beside a soft one: rows of A of 10^6 beside 1, u = A^-1 r
// the other way round), one frame for all of u would round the small entries that the large rows multiply.  So each
// column has a power of two, 2^s: the sum is that of (a 2^s)(u 2^-s) and the frames are those of the scaled entries.  The
// matrix's digits are cut from the entries as they are, in the frame eA - s; u comes scaled.
constexpr int kLimbBad = 1 << 14, kLimbNone = -(1 << 14);     // frames of a set with an Inf or NaN, of zeros only

// exponent field of v 2^s
SA_FX_HD int limb_scaled_exp(double v, int s)
{
	unsigned long long b;
#if defined(__CUDA_ARCH__)
	b = (unsigned long long) __double_as_longlong(v);
#else
	__builtin_memcpy(&b, &v, 8);
#endif
	const int e = (int) (b >> 52 & 0x7FFull);
	return e >= 2047 ? kLimbBad : b << 1 ? (e > 1 ? e : 1) + s : kLimbNone;
}

// an FP32 number of at least |v 2^s|, from 2^-126 on: a normal v rounded up (infinite beyond the range)
SA_FX_HD float limb_float_above(double v, int s)
{
	unsigned long long b;
#if defined(__CUDA_ARCH__)
	b = (unsigned long long) __double_as_longlong(v);
#else
	__builtin_memcpy(&b, &v, 8);
#endif
	const int e = (int) (b >> 52 & 0x7FFull) + s - 896;       // FP32 field
	const unsigned m = ((unsigned) (b >> 29) & 0x7FFFFFu) + 1u;
	const unsigned f = e > 253 ? 0x7F800000u : e < 1 ? 0x00800000u : ((unsigned) e << 23) + m;
#if defined(__CUDA_ARCH__)
	return __uint_as_float(f);
#else
	float r;
	__builtin_memcpy(&r, &f, 4);
	return r;
#endif
}

// More bits for a whole row at once: rows of an operator have few large entries, so their digits may be up to 2^4 longer
// than limb_matrix's before a digit sum leaves 63 bits.  The bits that a row can take, from its largest |a 2^s| (top) and the
// sum of them, both 2^x of what they are, and its frame e, x included.  With 80 products of |u1 + u0| <= 1.5 2^28 and
// |a0| <= 2^27, |a1| may sum to 2^33.4 (a1 = a 2^(1049 - e)); a1 + a0 stays a 32-bit number.
constexpr int kLimbExtra = 4;
SA_FX_HD int limb_extra(float top, float sum, int e)
{
	if (e < 1023 - 100 || e > 1023 + 100) return 0;
	const unsigned bits = (unsigned) (127 + 1023 - e) << 23; // 2^(1023 - e)
	float unit;
#if defined(__CUDA_ARCH__)
	unit = __uint_as_float(bits);
#else
	__builtin_memcpy(&unit, &bits, 4);
#endif
	const float t = top * unit, m = sum * unit;              // of |a1|, in units of 2^26
	int g = 0;
	while (g < kLimbExtra && t * (float) (2 << g) <= 29.9f && m * (float) (2 << g) <= 163.0f) ++g;
	return g;
}

// limb_matrix in a frame up to kLimbExtra below the entry's exponent
SA_FX_HD void limb_matrix_wide(double a, int eA, int &a1, int &a0)
{
	int e; unsigned long long m; bool neg;
	fx_parts(a, e, m, neg);
	const int d = eA - e;                                     // >= -kLimbExtra
	const unsigned long long v = d < 0 ? (d >= -kLimbExtra ? m << (2 - d) : 0ull) : d < 64 ? (((m << 3) >> d) + 1ull) >> 1 : 0ull;
	const long long s = neg ? -(long long) v : (long long) v;
	const long long lo = ((s + (1ll << 27)) & ((1ll << 28) - 1)) - (1ll << 27);
	a1 = (int) ((s - lo) >> 28);
	a0 = (int) lo;
}

// the sum as a double, for the frames of the scaled entries
SA_FX_HD double limb_scaled_to_double(const LimbSum &t, int eA, int eU)
{
	if (eA >= kLimbBad || eU >= 2047) return limb_bits(0x7FF8000000000000ull);
	return limb_round(limb_fixed(t), eA + eU - 1020);
}

// the sum as a double, for the matrix frame eA and the vector frame eU
SA_FX_HD double limb_to_double(const LimbSum &t, int eA, int eU)
{
	if (eA >= 2047 || eU >= 2047) return limb_bits(0x7FF8000000000000ull);     // NaN
	return limb_round(limb_fixed(t), eA + eU - 1020);         // value = f 2^(em - 1135), |f| < 2^120
}

}  // namespace sa
