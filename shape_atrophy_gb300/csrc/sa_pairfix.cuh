// sa_pairfix.cuh -- one pair term of the varifold objective on the integer pipes.
//
// K_c(|c_i - c_j| / w) K_d(u_i . u_j) v_j costs 30 FP64 operations for the Matern kernel, at 64 clocks each per warp and
// SM sub-partition.  Only the centre difference and its square (2 D operations) are formed in FP64 here; the root, the
// exponential, the direction product and the three products run in 64-bit fixed point, whose 32 x 32 -> 64 bit
// multiply-adds take about four clocks.  The scales below are powers of two; the numbers give the fraction bits.
//
// Errors, of 400,000 random distances a kernel (an FP64 operation: 2^-53): 'G' 0.5 x 2^-56 of K_c, 'C' 0.04 x 2^-56, 'M'
// 3.4 x 2^-56, on the low side (its last product is cut, 1.2 x 2^-56 on average near r = 0).  The term is rounded to nearest
// at 2^-61 of the frames of its tile's volumes and directions, so a pair whose kernels or volume are tiny beside its tile's
// keeps fewer bits, and none beyond r = 64 for 'M' (K_c < 2^-86) and r = 8 for 'G' (2^-92); 'C' has no such end.
#pragma once
#include "sa_fixsum.cuh"
#include <cmath>

namespace sa {

// 2^(-j/256) 2^63, j = 0 .. 255, rounded to nearest (computed with 60-digit decimal arithmetic)
#define SA_PAIR_EXP_TABLE \
	0x8000000000000000ull, 0x7fa765aca88f6453ull, 0x7f4f08ae3dc7c426ull, 0x7ef6e8da4b544f9aull, \
	0x7e9f06067a4360baull, 0x7e47600890f223deull, 0x7deff6b672f84e24ull, 0x7d98c9e62113e1faull, \
	0x7d41d96db915019dull, 0x7ceb252375c9cf9bull, 0x7c94acddaeea5d3aull, 0x7c3e7072d904a6ceull, \
	0x7be86fb985689ddcull, 0x7b92aa886214411cull, 0x7b3d20b6399fc237ull, 0x7ae7d219f329b948ull, \
	0x7a92be8a92436616ull, 0x7a3de5df36dcfeefull, 0x79e947ef1d320d2dull, 0x7994e4919db5d74eull, \
	0x7940bb9e2cffd89dull, 0x78ecccec5bb84661ull, 0x78991853d684a285ull, 0x78459dac65f45bb5ull, \
	0x77f25ccdee6d7ae6ull, 0x779f559070195e36ull, 0x774c87cc06d1812eull, 0x76f9f358ea0c5249ull, \
	0x76a7980f6cca15c2ull, 0x765575c7fd81d5a0ull, 0x76038c5b260e5eeeull, 0x75b1dba18b9b4c20ull, \
	0x75606373ee921c97ull, 0x750f23ab2a87593eull, 0x74be1c203627c62bull, 0x746d4cac2325a155ull, \
	0x741cb5281e25ee34ull, 0x73cc556d6eadce5full, 0x737c2d55770fe711ull, 0x732c3cb9b459d38bull, \
	0x72dc8373be41a454ull, 0x728d015d47136b40ull, 0x723db6501b9ed447ull, 0x71eea2262324cb0cull, \
	0x719fc4b95f452d29ull, 0x71511de3ebec8913ull, 0x7102ad7fff41e9b4ull, 0x70b47367e994ae92ull, \
	0x70666f76154a7089ull, 0x7018a18506ccf314ull, 0x6fcb096f5c782210ull, 0x6f7da70fce881bf9ull, \
	0x6f307a412f074892ull, 0x6ee382de69bc7bf8ull, 0x6e96c0c284192610ull, 0x6e4a33c89d278e49ull, \
	0x6dfddbcbed791babull, 0x6db1b8a7c714a92bull, 0x6d65ca379564e639ull, 0x6d1a1056dd26c382ull, \
	0x6cce8ae13c57ebdbull, 0x6c8339b26a25494eull, 0x6c381ca636d99642ull, 0x6bed33988bcbfab5ull, \
	0x6ba27e656b4eb57aull, 0x6b57fce8f09dd17full, 0x6b0daeff4fcde703ull, 0x6ac39484d5bae8c5ull, \
	0x6a79ad55e7f6fd10ull, 0x6a2ff94f04b962b0ull, 0x69e6784cc2cd61bdull, 0x699d2a2bd181482aull, \
	0x69540ec8f895722dull, 0x690b2601182b5e56ull, 0x68c26fb128b4cd63ull, 0x6879ebb63ae2edc6ull, \
	0x683199ed779592caull, 0x67e97a341fca775bull, 0x67a18c678c8c8c61ull, 0x6759d0652ee352afull, \
	0x6712460a8fc24072ull, 0x66caed354ff83222ull, 0x6683c5c3281ee6e9ull, 0x663ccf91e88a8873ull, \
	0x65f60a7f79393e2eull, 0x65af7669d9c2cbe4ull, 0x6569132f21483ba7ull, 0x6522e0ad7e639312ull, \
	0x64dcdec3371793d1ull, 0x64970d4ea8bf8766ull, 0x64516c2e47ff1623ull, 0x640bfb40a0b22959ull, \
	0x63c6ba6455dcd8aeull, 0x6381a978219b628full, 0x633cc85ad5122fbdull, 0x62f816eb585de1edull, \
	0x62b39508aa836d6full, 0x626f4291e1603dd5ull, 0x622b1f66299a6599ull, 0x61e72b64c690d8afull, \
	0x61a3666d124bb204ull, 0x615fd05e7d6c83e4ull, 0x611c69188f1eb339ull, 0x60d9307ae507dd9aull, \
	0x6096266533384a2bull, 0x60534ab7441b6546ull, 0x60109d50f86846d8ull, 0x5fce1e124712437cull, \
	0x5f8bccdb3d398841ull, 0x5f49a98bfe1bc11cull, 0x5f07b404c304c9f1ull, 0x5ec5ec25db3f6a41ull, \
	0x5e8451cfac061b5full, 0x5e42e4e2b073d935ull, 0x5e01a53f7974fd86ull, 0x5dc092c6adb825b8ull, \
	0x5d7fad59099f22feull, 0x5d3ef4d75f2ff504ull, 0x5cfe69229605cef5ull, 0x5cbe0a1bab4226dfull, \
	0x5c7dd7a3b17dcf75ull, 0x5c3dd19bd0ba1c1aull, 0x5bfdf7e546520f3eull, 0x5bbe4a6164eb92f4ull, \
	0x5b7ec8f19468bbc9ull, 0x5b3f737751d915c8ull, 0x5b0049d42f6afbb6ull, 0x5ac14be9d45cf869ull, \
	0x5a827999fcef3242ull, 0x5a43d2c67a54e0c0ull, 0x5a05575132a5cc20ull, 0x59c7071c20cfd70cull, \
	0x5988e20954889245ull, 0x594ae7faf23eda52ull, 0x590d18d3330c7f1eull, 0x58cf747464a7f584ull, \
	0x5891fac0e95612c8ull, 0x5854ab9b37dbd1e5ull, 0x581786e5db7022c2ull, 0x57da8c8373adc331ull, \
	0x579dbc56b48521baull, 0x57611642662e4a33ull, 0x57249a29651adc07ull, 0x56e847eea1e80a49ull, \
	0x56ac1f752150a563ull, 0x5670209ffc1f2e82ull, 0x56344b525f1ff495ull, 0x55f89f6f8b133af4ull, \
	0x55bd1cdad49f699cull, 0x5581c377a44346f0ull, 0x5546932976483b15ull, 0x550b8bd3dab49cbdull, \
	0x54d0ad5a753e077cull, 0x5495f7a0fd3bbb8eull, 0x545b6a8b3d990704ull, 0x542105fd14c7b869ull, \
	0x53e6c9da74b29ab5ull, 0x53acb60762affaaeull, 0x5372ca67f774358full, 0x533906e05f045106ull, \
	0x52ff6b54d8a89c75ull, 0x52c5f7a9b6df5b77ull, 0x528cabc35f4f799dull, 0x525387864abb4762ull, \
	0x521a8ad704f3404full, 0x51e1b59a2cc8da3eull, 0x51a907b474015dc9ull, 0x5170810a9f48c7cfull, \
	0x513821818624b40cull, 0x50ffe8fe12e750c4ull, 0x50c7d76542a25b72ull, 0x508fec9c251a267cull, \
	0x50582887dcb8a7e1ull, 0x50208b0d9e8090dfull, 0x4fe91412b2006e83ull, 0x4fb1c37c7145d328ull, \
	0x4f7a993048d088d7ull, 0x4f439513b785cc80ull, 0x4f0cb70c4ea39210ull, 0x4ed5feffb1b3d155ull, \
	0x4e9f6cd3967fdba8ull, 0x4e69006dc503ba65ull, 0x4e32b9b417619617ull, 0x4dfc988c79d52661ull, \
	0x4dc69cdceaa72a9cull, 0x4d90c68b7a20eb1eull, 0x4d5b157e4a7fc325ull, 0x4d25899b8fe8b365ull, \
	0x4cf022c9905bfd32ull, 0x4cbae0eea3a8c63cull, 0x4c85c3f13360c4d5ull, 0x4c50cbb7bacbf4cbull, \
	0x4c1bf828c6dc54b8ull, 0x4be7492af621abd6ull, 0x4bb2bea4f8bd5847ull, 0x4b7e587d905625d1ull, \
	0x4b4a169b900c2d00ull, 0x4b15f8e5dc6cbab0ull, 0x4ae1ff436b663ff7ull, 0x4aae299b443c4a6bull, \
	0x4a7a77d47f7b84b1ull, 0x4a46e9d646edbf6aull, 0x4a137f87d58e025bull, 0x49e038d0777ca5e0ull, \
	0x49ad159789f37496ull, 0x497a15c47b39d53eull, 0x4947393eca98fcd6ull, 0x49147fee085028d6ull, \
	0x48e1e9b9d588e19bull, 0x48af7689e44b44eaull, 0x487d2645f7725895ull, 0x484af8d5e2a06536ull, \
	0x4818ee218a3358eeull, 0x47e70610e3393241ull, 0x47b5408bf36472e2ull, 0x47839d7ad1009a90ull, \
	0x47521cc5a2e6a9e0ull, 0x4720be54a071ad01ull, 0x46ef821011734e6bull, 0x46be67e04e28717cull, \
	0x468d6fadbf2dd4f3ull, 0x465c9960dd74bd4bull, 0x462be4e23237a6efull, 0x45fb521a56ef0042ull, \
	0x45cae0f1f545eb73ull, 0x459a9151c70f0819ull, 0x456a632296394492ull, 0x453a564d3cc4b723ull, \
	0x450a6abaa4b77ecdull, 0x44daa053c812abd2ull, 0x44aaf701b0c72feeull, 0x447b6ead78aad636ull, \
	0x444c0740496d4294ull, 0x441cc0a35c8cf8eaull, 0x43ed9abffb4c6bc9ull, 0x43be957f7ea712b6ull, \
	0x438fb0cb4f468808ull, 0x4360ec8ce577ae44ull, 0x433248adc91fdd02ull, 0x4303c51791b21550ull, \
	0x42d561b3e6243d8aull, 0x42a71e6c7ce464afull, 0x4278fb2b1bce0d15ull, 0x424af7d9981f7e98ull, \
	0x421d1461d66f2023ull, 0x41ef50adcaa0d899ull, 0x41c1aca777db771bull, 0x41942838f07e22a3ull, \
	0x4166c34c5615d0ecull, 0x41397dcbd952c4a6ull, 0x410c57a1b9fe12f6ull, 0x40df50b846ef302bull, \
	0x40b268f9de0183baull, 0x4085a050ec0a036aull, 0x4058f6a7ecccd5b6ull, 0x402c6be96af2fb58ull,

SA_FX_HD unsigned pair_mulhi(unsigned a, unsigned b) { return (unsigned) (((unsigned long long) a * b) >> 32); }

// a b / 2^64, short by at most 3 (the product of the low halves is left out)
SA_FX_HD unsigned long long pair_mulh(unsigned long long a, unsigned long long b)
{
	const unsigned ah = (unsigned) (a >> 32), al = (unsigned) a, bh = (unsigned) (b >> 32), bl = (unsigned) b;
	return (unsigned long long) ah * bh + pair_mulhi(ah, bl) + pair_mulhi(al, bh);
}

// e^-x 2^63 = result 2^-m, x at 57 bits, below 64.  N = 256 x / ln 2 rounded down (or one less), N = 256 m + j,
// r = x - N ln2/256 in [0, 0.0028), e^-r = 1 - p, p = r - r^2 (1/2 - r (1/6 - r (1/24 - r / 120))); the next term is
// 2^-60.  tab: SA_PAIR_EXP_TABLE.
SA_FX_HD unsigned long long pair_exp(unsigned long long x, int &m, const unsigned long long *tab)
{
	const unsigned N = pair_mulhi((unsigned) (x >> 31), 1549082004u) >> 16;
	const unsigned long long r = (x << 15) - N * 12786308645202655659ull;    // 72 bits
	const unsigned rh = (unsigned) (r >> 32);                                // 40 bits
	const unsigned t1 = 2863311531u - pair_mulhi(rh, 2236962u);              // 36 bits
	const unsigned t2 = 2863311531u - (pair_mulhi(rh, t1) >> 10);            // 34 bits
	const unsigned long long h = (1ull << 63) - (((unsigned long long) rh * t2) >> 10);   // 64 bits
	const unsigned long long p = r - (pair_mulh(pair_mulh(r, r), h) >> 8);   // r^2 at 80 bits; p at 72
	const unsigned long long S = tab[N & 255u];
	m = (int) (N >> 8);
	return S - (pair_mulh(S, p) >> 8);
}

constexpr unsigned long long kPairFar = (1ull << 63) - 1ull;   // distances of 64 and more

// a >= 0 at 57 bits (kPairFar from 64 on), hi and lo the words of the double
SA_FX_HD unsigned long long pair_fix(unsigned hi, unsigned lo)
{
	const int e = (int) (hi >> 20) - 1023;
	if (e >= 6) return kPairFar;
	const unsigned long long m = ((unsigned long long) ((hi & 0xfffffu) | 0x100000u) << 32) | lo;
	return e < -58 ? 0ull : (m << 10) >> (5 - e);
}

// sqrt(a) at 57 bits (kPairFar from 64 on), a >= 0: a = A 4^k with A in [1/4, 1), y the FP32 reciprocal root of A;
// s0 = A y to 2^-21, then twice s += (A - s^2) y / 2, whose residual is formed exactly enough in integers
SA_FX_HD unsigned long long pair_sqrt(unsigned hi, unsigned lo)
{
	const int e = (int) (hi >> 20) - 1023, k = (e + 2) >> 1;
	if (k >= 7) return kPairFar;
	if (k < -57) return 0ull;
	const unsigned top = (hi & 0xfffffu) | 0x100000u;
	const unsigned long long A = (((unsigned long long) top << 32) | lo) << (10 + e - 2 * k);     // 62 bits
	const unsigned bits = ((unsigned) (e - 2 * k + 127) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
#ifdef __CUDA_ARCH__
	const float f = __uint_as_float(bits);
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
	const unsigned s0 = __float2uint_rz(f * y * 1073741824.0f) << 1, Y = __float2uint_rz(y * 1073741824.0f);
#else
	float f;
	__builtin_memcpy(&f, &bits, 4);
	const float y = 1.0f / sqrtf(f);
	const unsigned s0 = (unsigned) (f * y * 1073741824.0f) << 1, Y = (unsigned) (y * 1073741824.0f);
#endif
	// s0 at 31 bits (even), Y at 30
	const long long R = (long long) (A - (unsigned long long) s0 * s0);                           // |R| < 2^42
	const int Ys = (int) (Y >> 1), s0h = (int) (s0 >> 1);
	const long long c = ((long long) (int) (R >> 12) * Ys) >> 18;                                 // 62 bits, below 2^41
	const int c1 = (int) (c >> 16), c0 = (int) (c & 0xffff);
	const long long T = (((long long) s0h * c1) >> 13) + (((long long) s0h * c0) >> 29);          // 2 s0 c
	const int R1 = (int) (R - T - (((long long) c1 * c1) >> 30));
	const unsigned long long s = ((unsigned long long) s0 << 31) + c + (((long long) R1 * Ys) >> 30);
	return k == 6 ? s << 1 : s >> (5 - k);
}

// 1 / a at 63 + m bits for a double a >= 1 (0 from 2^62 on): Y the FP32 reciprocal of the significand A in [1, 2), e = 1 - A Y,
// 1 / A = Y (1 + e + e^2); |e| < 2^-21
SA_FX_HD unsigned long long pair_recip(unsigned hi, unsigned lo, int &m)
{
	m = (int) (hi >> 20) - 1023;
	if (m >= 62) return 0ull;
	const unsigned top = (hi & 0xfffffu) | 0x100000u;
	const unsigned long long A = (((unsigned long long) top << 32) | lo) << 10;                   // 62 bits
	const unsigned bits = (127u << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
#ifdef __CUDA_ARCH__
	float y;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(bits)));
	const unsigned Y = __float2uint_rz(y * 536870912.0f) << 1;                                    // 30 bits, even
#else
	float f;
	__builtin_memcpy(&f, &bits, 4);
	const unsigned Y = (unsigned) (1.0f / f * 536870912.0f) << 1;
#endif
	const unsigned long long P = (((A >> 32) * Y) << 2) + (((A & 0xffffffffull) * Y) >> 30);      // A Y at 62 bits
	const long long e = (long long) ((1ull << 62) - P);
	const int eh = (int) (e >> 12);                                                               // 50 bits
	const long long s = e + (((long long) eh * eh) >> 38);
	const long long c = (((s >> 12) * (long long) (int) (Y >> 1)) >> 16) + (((s & 0xfff) * (long long) (int) (Y >> 1)) >> 28);
	return ((unsigned long long) Y << 33) + c;
}

// v 2^-b as a double, v below 2^64; rounded once
SA_FX_HD double pair_double(unsigned long long v, int b)
{
#ifdef __CUDA_ARCH__
	const int n = __clzll((long long) v);
#else
	const int n = v ? __builtin_clzll(v) : 64;
#endif
	if (n == 64 || b > 1000) return 0.0;
	const unsigned long long q = (v << n) >> 10;              // 54 bits
	const unsigned long long r = ((unsigned long long) (1023 + 62 - n - b) << 52) + ((q + 1ull) >> 1);   // the leading bit adds one
#ifdef __CUDA_ARCH__
	return __longlong_as_double((long long) r);
#else
	double d;
	__builtin_memcpy(&d, &r, 8);
	return d;
#endif
}

// K_c at 63 + m bits: 'M' (1 + r) e^-r, 'G' e^-d2, 'C' 1 / a; hi and lo the words of the squared distance d2 in widths ('C': of
// a = 1 + d2)
SA_FX_HD unsigned long long pair_centre(int type, unsigned hi, unsigned lo, int &m, const unsigned long long *tab)
{
	if (type == 'G') return pair_exp(pair_fix(hi, lo), m, tab);
	if (type == 'C') return pair_recip(hi, lo, m);
	const unsigned long long r = pair_sqrt(hi, lo), e = pair_exp(r, m, tab);
	unsigned long long v = pair_mulh(r + (1ull << 57), e);   // 56 bits, below 2^m
	if (m < 7) v <<= 7 - m;
	m = m > 7 ? m - 7 : 0;
	return v;
}

// direction component u 2^-e (the vector at most 1 long) at 61 bits, in two digits of 31
SA_FX_HD void pair_digits(double u, int &h, int &l)
{
	const long long v = (long long) rint(u * 2305843009213693952.0);
	h = (int) (v >> 31);
	l = (int) (v & 0x7fffffff);
}

// |u_i . u_j| at 63 bits, sign apart
template <int D>
SA_FX_HD unsigned long long pair_angle(const int *uh, const int *ul, const int *vh, const int *vl, bool &neg)
{
	long long a = (long long) uh[0] * vh[0], b = (long long) uh[0] * vl[0] + (long long) ul[0] * vh[0];
	for (int d = 1; d < D; ++d) {
		a += (long long) uh[d] * vh[d];
		b += (long long) uh[d] * vl[d] + (long long) ul[d] * vh[d];
	}
	const long long s = (a << 2) + (b >> 29);                // 62 bits: a unit vector's own product may exceed 1
	neg = s < 0;
	return (unsigned long long) (neg ? -s : s) << 1;
}

// K_c K_d v at 61 bits from K_c at 63 + m, K_d and v at 63
SA_FX_HD unsigned long long pair_term(unsigned long long kc, int m, unsigned long long kd, unsigned long long v)
{
	const unsigned long long q = pair_mulh(kc, pair_mulh(kd, v));
	m = m < 63 ? m : 63;
	return (q + ((1ull << m) >> 1)) >> m;
}

// e with |u| <= 2^e (1 + 2^-40), n2 = |u|^2: unit vectors, rounding included, have e = 0
SA_FX_HD int pair_frame(double n2) { return (fx_exp(n2 * (1.0 - 0x1p-40)) - 1021) >> 1; }

}  // namespace sa
