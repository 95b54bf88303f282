// sa_kernel.cu -- RKHS kernel matrix and the K-preconditioned CG of frame mode.
//
// Reference: 2D_frame/computeKernel.cu:7-209 (2D Matern through x^2 K0(x) and
// x K1(x), inc/polybesselk.h:8-99 with the rational-approximation tables of
// inc/besselk.h), 3D_frame/computeKernel.cu:5-153 (closed-form Matern
// n + 1/2), 2D_frame/addEpsIdentity.cu:3-20, and the CG of
// 2D_frame/ipcg.cu:11-100 with ipcgWholeMatrixMultiplication.cu:21-45,
// ipcgSecondMatrixMultiplication.cu:8-24, ipcgKernelMultiplication.cu:5-17.
//
// GB300 changes: scalars and the stopping test stay on the device (the
// reference returns every dot product to the host), and the dense Cholesky
// of K is gone.  The reference needs potrs(K, x0) only for the warm start
// x0 = v_prev; here the solve tracks w = K^{-1} x through the CG recurrences
// (w += alpha K^{-1}d, with K^{-1}d already tracked as KidVec) and starts the
// next step from x0 = K_new w_prev, whose K_new^{-1} x0 = w_prev is known
// exactly.  The converged velocity is the same solution of the same system
// to the CG tolerance.
#include "sa_internal.cuh"
#include "sa_grid.cuh"
#include "sa_limb.cuh"
#include <algorithm>
#include <cmath>

namespace sa {

// rational-approximation coefficients (inc/besselk.h:4-180), same values
__constant__ double cP01[6] = { 2.4708152720399552679e+03,  5.9169059852270512312e+03,
                                4.6850901201934832188e+02,  1.1999463724910714109e+01,
                                1.3166052564989571850e-01,  5.8599221412826100000e-04};
__constant__ double cQ01[3] = { 2.1312714303849120380e+04, -2.4994418972832303646e+02, 1};
__constant__ double cP02[4] = {-4.0320340761145482298e+05, -1.7733784684952985886e+04,
                               -2.9601657892958843866e+02, -1.6414452837299064100e+00};
__constant__ double cQ02[4] = {-1.6128136304458193998e+06,  2.9865713163054025489e+04,
                               -2.5064972445877992730e+02,  1};
__constant__ double cP03[10] = { 1.1600249425076035558e+02,  2.3444738764199315021e+03,
                                 1.8321525870183537725e+04,  7.1557062783764037541e+04,
                                 1.5097646353289914539e+05,  1.7398867902565686251e+05,
                                 1.0577068948034021957e+05,  3.1075408980684392399e+04,
                                 3.6832589957340267940e+03,  1.1394980557384778174e+02};
__constant__ double cQ03[11] = { 9.2556599177304839811e+01,  1.8821890840982713696e+03,
                                 1.4847228371802360957e+04,  5.8824616785857027752e+04,
                                 1.2689839587977598727e+05,  1.5144644673520157801e+05,
                                 9.7418829762268075784e+04,  3.1474655750295278825e+04,
                                 4.4329628889746408858e+03,  2.0013443064949242491e+02, 1};
__constant__ double cP11[6] = {-2.2149374878243304548e+06,  7.1938920065420586101e+05,
                                1.7733324035147015630e+05,  7.1885382604084798576e+03,
                                9.9991373567429309922e+01,  4.8127070456878442310e-01};
__constant__ double cQ11[4] = {-2.2149374878243304548e+06,  3.7264298672067697862e+04,
                               -2.8143915754538725829e+02,  1};
__constant__ double cP12[5] = {-1.3531161492785421328e+06, -1.4758069205414222471e+05,
                               -4.5051623763436087023e+03, -5.3103913335180275253e+01,
                               -2.2795590826955002390e-01};
__constant__ double cQ12[4] = {-2.7062322985570842656e+06,  4.3117653211351080007e+04,
                               -3.0507151578787595807e+02,  1};
__constant__ double cP13[11] = { 2.2196792496874548962e+00,  4.4137176114230414036e+01,
                                 3.4122953486801312910e+02,  1.3319486433183221990e+03,
                                 2.8590657697910288226e+03,  3.4540675585544584407e+03,
                                 2.3123742209168871550e+03,  8.1094256146537402173e+02,
                                 1.3182609918569941308e+02,  7.5584584631176030810e+00,
                                 6.4257745859173138767e-02};
__constant__ double cQ13[10] = { 1.7710478032601086579e+00,  3.4552228452758912848e+01,
                                 2.5951223655579051357e+02,  9.6929165726802648634e+02,
                                 1.9448440788918006154e+03,  2.1181000487171943810e+03,
                                 1.2082692316002348638e+03,  3.3031020088765390854e+02,
                                 3.6001069306861518855e+01,  1};

__device__ __forceinline__ double polyval(int deg, const double *c, double x)
{
	double v = c[deg];
	for (int i = deg - 1; i >= 0; --i) v = v * x + c[i];
	return v;
}

__device__ double p0fcn(double x)
{   // x^2 K0(x): inc/polybesselk.h:17-54
	if (x < DBL_EPSILON || x > 700.0) return 0.0;
	if (x <= 1.0) {
		double xs = x * x, lx = log(x);
		double PQ01 = polyval(5, cP01, xs) / polyval(2, cQ01, xs);
		double PQ02 = polyval(3, cP02, xs) / polyval(3, cQ02, xs);
		return xs * (PQ01 - lx * (xs * PQ02 + 1.0));
	}
	double xi = 1.0 / x;
	return x * sqrt(x) * exp(-x) * (polyval(9, cP03, xi) / polyval(10, cQ03, xi));
}

__device__ double p1fcn(double x)
{   // x K1(x): inc/polybesselk.h:56-99
	if (x < DBL_EPSILON) return 1.0;
	if (x > 700.0) return 0.0;
	if (x <= 1.0) {
		double xs = x * x, lx = log(x);
		double PQ11 = polyval(5, cP11, xs) / polyval(3, cQ11, xs);
		double PQ12 = polyval(4, cP12, xs) / polyval(3, cQ12, xs);
		return PQ11 + xs * lx * PQ12;
	}
	double xi = 1.0 / x;
	return sqrt(x) * exp(-x) * (polyval(10, cP13, xi) / polyval(9, cQ13, xi));
}

template <int D>
__device__ __forceinline__ double kernel_value(int order, double w, double d2)
{
	if (D == 2) {
		if (order == -1) return exp(-(d2 / (w * w)));
		double dij = sqrt(d2) / w, dsq = dij * dij;
		double f1 = p1fcn(dij), f0 = order > 0 ? p0fcn(dij) : 0.0;
		switch (order) {
		case 0: return f1;
		case 1: return 0.5 * (f0 + 2.0 * f1);
		case 2: return (4.0 * f0 + (8.0 + dsq) * f1) / 8.0;
		case 3: return ((24.0 + dsq) * f0 + 8.0 * (6.0 + dsq) * f1) / 48.0;
		default: return (12.0 * (16.0 + dsq) * f0 + (384.0 + dsq * (72.0 + dsq)) * f1) / 384.0;
		}
	}
	if (order == -1) return exp(-(d2 / (w * w)));
	double r = sqrt(d2) / w, ex = exp(-r);
	switch (order) {
	case 0: return ex;
	case 1: return (1.0 + r) * ex;
	case 2: return (3.0 + r * (3.0 + r)) / 3.0 * ex;
	case 3: return (15.0 + r * (15.0 + r * (6.0 + r))) / 15.0 * ex;
	default: return (105.0 + r * (105.0 + r * (45.0 + r * (10.0 + r)))) / 105.0 * ex;
	}
}

// dk/d(d2), the kernel's derivative with respect to the squared distance (discrete adjoint of the frame
// model).  2D Matern through d(x K1)/dx = -x K0 = -p0 / x and d(x^2 K0)/dx = 2 p0 / x - x p1; every order
// but 0 carries a factor x that cancels dx/d(d2) = 1 / (2 w^2 x).  Not called at d2 = 0.
template <int D>
__device__ __forceinline__ double kernel_dvalue(int order, double w, double d2)
{
	if (order == -1) return -exp(-(d2 / (w * w))) / (w * w);
	const double w2 = w * w;
	if (D == 2) {
		double x = sqrt(d2) / w, xs = x * x;
		double f1 = p1fcn(x), f0 = p0fcn(x);
		switch (order) {
		case 0: return -f0 / (2.0 * w2 * xs);
		case 1: return -0.5 * f1 / (2.0 * w2);
		case 2: return -(2.0 * f1 + f0) / (16.0 * w2);
		case 3: return -(4.0 * f0 + (8.0 + xs) * f1) / (96.0 * w2);
		default: return -((24.0 + xs) * f0 + (48.0 + 8.0 * xs) * f1) / (768.0 * w2);
		}
	}
	double r = sqrt(d2) / w, ex = exp(-r);
	switch (order) {
	case 0: return -ex / (2.0 * w2 * r);
	case 1: return -ex / (2.0 * w2);
	case 2: return -(1.0 + r) * ex / (6.0 * w2);
	case 3: return -(3.0 + r * (3.0 + r)) * ex / (30.0 * w2);
	default: return -(15.0 + r * (15.0 + r * (6.0 + r))) * ex / (210.0 * w2);
	}
}

// a_x_i += ldm sum_{j != i} 2 dk/d(d2)(x_i - x_j) sum_d (alpha_id beta_jd + alpha_jd beta_id): the vector-Jacobian
// product of x -> -ldm n^T K(x)^{-1} v with alpha = K^{-1} n, beta = K^{-1} v (nodal vectors, interleaved).
// One thread per node, the other nodes in shared-memory tiles.
template <int D>
__global__ void k_adj_kernel_term(int N, const double *__restrict__ x, const double *__restrict__ alpha,
                                  const double *__restrict__ beta, int order, double w, double ldm,
                                  double *__restrict__ ax)
{
	__shared__ double tx[128 * D], ta[128 * D], tb[128 * D];
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	Vec<D> xi, ai, bi;
	for (int d = 0; d < D; ++d) {
		xi.c[d] = i < N ? x[(long) i * D + d] : 0.0;
		ai.c[d] = i < N ? alpha[(long) i * D + d] : 0.0;
		bi.c[d] = i < N ? beta[(long) i * D + d] : 0.0;
	}
	double acc[D];
	for (int d = 0; d < D; ++d) acc[d] = 0.0;
	for (int j0 = 0; j0 < N; j0 += 128) {
		const int nt = min(128, N - j0);
		__syncthreads();
		for (int t = threadIdx.x; t < nt * D; t += blockDim.x) {
			tx[t] = x[(long) j0 * D + t];
			ta[t] = alpha[(long) j0 * D + t];
			tb[t] = beta[(long) j0 * D + t];
		}
		__syncthreads();
		if (i >= N) continue;
		for (int jj = 0; jj < nt; ++jj) {
			if (j0 + jj == i) continue;
			double d2 = 0.0, ab = 0.0, dx[D];
			for (int d = 0; d < D; ++d) {
				dx[d] = xi.c[d] - tx[jj * D + d];
				d2 += dx[d] * dx[d];
				ab += ai.c[d] * tb[jj * D + d] + ta[jj * D + d] * bi.c[d];
			}
			const double g = 2.0 * kernel_dvalue<D>(order, w, d2) * ab;
			for (int d = 0; d < D; ++d) acc[d] += g * dx[d];
		}
	}
	if (i < N)
		for (int d = 0; d < D; ++d) ax[(long) i * D + d] += ldm * acc[d];
}

template <int D>
void launch_adj_kernel_term(const Model &md, int N, const double *x, const double *alpha, const double *beta,
                            double *ax, cudaStream_t s)
{
	k_adj_kernel_term<D><<<grid_for(N, 128), 128, 0, s>>>(N, x, alpha, beta, md.knlOrder, md.knlWidth, md.ldmWgt, ax);
}

// One RKHS matrix entry k(|q_i - q_j| / w) (without the eps diagonal).  Compiled once, not inlined: the
// stored matrix and the matrix-free products evaluate it with the same instructions, so the compiler's
// multiply-add fusion cannot differ between the two callers and both give the same bits.  Symmetric bit for
// bit: (a - b)^2 = (b - a)^2 exactly.
template <int D>
__device__ __noinline__ double kernel_entry(int order, double w, Vec<D> qi, Vec<D> qj)
{
	double d2 = (qi.c[0] - qj.c[0]) * (qi.c[0] - qj.c[0]);
	for (int d = 1; d < D; ++d) d2 = d2 + (qi.c[d] - qj.c[d]) * (qi.c[d] - qj.c[d]);
	return kernel_value<D>(order, w, d2);
}

// ---------------------------------------------------------------------------
// K-preconditioned CG (reference ipcg) with device scalars
// ---------------------------------------------------------------------------
struct KScal {
	double bSqu, rSqu, rKr, rKrNew, dAd, alpha, beta, tolSqu, ldmWgt;
	int done, code, iters, itrMax;
	unsigned int counter;
	int pad;
};

constexpr int kKBlock = 256;

template <int K>
__device__ __forceinline__ bool kreduce(double (&v)[K], double *part, unsigned int *counter)
{
	__shared__ double sm[K][kKBlock / 32];
	__shared__ bool last;
	int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	for (int k = 0; k < K; ++k)
		for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
	if (lane == 0) for (int k = 0; k < K; ++k) sm[k][wid] = v[k];
	__syncthreads();
	if (threadIdx.x == 0) {
		for (int k = 0; k < K; ++k) {
			double s = 0.0;
			for (int w = 0; w < kKBlock / 32; ++w) s += sm[k][w];
			part[k * gridDim.x + blockIdx.x] = s;
		}
		__threadfence();
		unsigned int t = atomicAdd(counter, 1u);
		last = (t == gridDim.x - 1);
	}
	__syncthreads();
	return last;
}

template <int K>
__device__ __forceinline__ void kfinish(double (&out)[K], const double *part)
{
	int lane = threadIdx.x & 31;
	for (int k = 0; k < K; ++k) {
		double s = 0.0;
		for (int b = lane; b < (int) gridDim.x; b += 32) s += __ldcg(part + k * gridDim.x + b);
		for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
		out[k] = s;
	}
}

// (b, b): zero rhs gives x = 0, w = 0
template <int D>
__global__ void k_kp_bnorm(int N, const double *__restrict__ b, double *part, KScal *sc)
{
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	double v[1] = {0.0};
	if (i < N) for (int d = 0; d < D; ++d) v[0] += b[(long) i * D + d] * b[(long) i * D + d];
	if (!kreduce<1>(v, part, &sc->counter)) return;
	double o[1]; kfinish<1>(o, part);
	if (threadIdx.x == 0) {
		sc->bSqu = o[0];
		if (!isfinite(o[0])) { sc->code = SA_ERR_NONFINITE; sc->done = 1; }
		else if (o[0] == 0.0) sc->done = 2;          // x = 0
		sc->counter = 0;
	}
}

// r = b - (ldm w + Bx0), (r, r)
template <int D>
__global__ void k_kp_init_r(SellOp A, const double *__restrict__ blk, const double *__restrict__ b,
                            const double *__restrict__ x, const double *__restrict__ w, double *__restrict__ r,
                            double *part, KScal *sc)
{
	if (sc->done) return;
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	const int N = A.N;
	double v[1] = {0.0};
	if (i < N) {
		double acc[D];
		sell_row<D, double, double>(A, blk, i, x, acc);
		for (int d = 0; d < D; ++d) {
			long k = (long) i * D + d;
			double Ax = sc->ldmWgt * w[k] + acc[d];
			double rk = 1.0 * b[k] + -1.0 * Ax;
			r[k] = rk;
			v[0] += rk * rk;
		}
	}
	if (!kreduce<1>(v, part, &sc->counter)) return;
	double o[1]; kfinish<1>(o, part);
	if (threadIdx.x == 0) {
		sc->rSqu = o[0];
		if (!isfinite(o[0])) { sc->code = SA_ERR_NONFINITE; sc->done = 1; }
		else if (o[0] < sc->bSqu * sc->tolSqu) sc->done = 1;
		sc->counter = 0;
	}
}

// (r, Kr) after Kr = K r; first = 1: initialise Kid = r, d = Kr; else beta and the d / Kid updates
template <int D>
__global__ void k_kp_rkr(int N, const double *__restrict__ r, const double *__restrict__ Kr, double *part,
                         KScal *sc, int first)
{
	if (sc->done) return;
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	double v[1] = {0.0};
	if (i < N) for (int d = 0; d < D; ++d) v[0] += r[(long) i * D + d] * Kr[(long) i * D + d];
	if (!kreduce<1>(v, part, &sc->counter)) return;
	double o[1]; kfinish<1>(o, part);
	if (threadIdx.x == 0) {
		if (o[0] == 0.0 || !isfinite(o[0])) {
			sc->code = isfinite(o[0]) ? SA_ERR_BREAKDOWN : SA_ERR_NONFINITE;
			sc->done = 1;
		} else if (first) {
			sc->rKr = o[0];
		} else {
			sc->beta = o[0] / sc->rKr;
			sc->rKr = o[0];
		}
		sc->counter = 0;
	}
}

// Kid = r + beta Kid; d = Kr + beta d (first: Kid = r, d = Kr)
template <int D>
__global__ void k_kp_dir(int N, const double *__restrict__ r, const double *__restrict__ Kr, double *__restrict__ Kid,
                         double *__restrict__ dv, const KScal *sc, int first)
{
	if (sc->done) return;
	long k = blockIdx.x * (long) blockDim.x + threadIdx.x;
	if (k >= (long) N * D) return;
	if (first) { Kid[k] = r[k]; dv[k] = Kr[k]; return; }
	double be = sc->beta;
	Kid[k] = 1.0 * r[k] + be * Kid[k];
	dv[k] = 1.0 * Kr[k] + be * dv[k];
}

// Bd = (E + btm P) d; Ad = ldm Kid + Bd; (d, Ad) -> alpha
template <int D>
__global__ void k_kp_ad(SellOp A, const double *__restrict__ blk, const double *__restrict__ dv,
                        const double *__restrict__ Kid, double *__restrict__ Ad, double *part, KScal *sc)
{
	if (sc->done) return;
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	const int N = A.N;
	double v[1] = {0.0};
	if (i < N) {
		double acc[D];
		sell_row<D, double, double>(A, blk, i, dv, acc);
		for (int d = 0; d < D; ++d) {
			long k = (long) i * D + d;
			double a = sc->ldmWgt * Kid[k] + 1.0 * acc[d];
			Ad[k] = a;
			v[0] += dv[k] * a;
		}
	}
	if (!kreduce<1>(v, part, &sc->counter)) return;
	double o[1]; kfinish<1>(o, part);
	if (threadIdx.x == 0) {
		sc->dAd = o[0];
		if (o[0] == 0.0 || !isfinite(o[0])) {
			sc->code = isfinite(o[0]) ? SA_ERR_BREAKDOWN : SA_ERR_NONFINITE;
			sc->done = 1;
		} else sc->alpha = sc->rKr / o[0];
		sc->counter = 0;
	}
}

// x += alpha d; w += alpha Kid; r -= alpha Ad; (r, r) -> stop test
template <int D>
__global__ void k_kp_step(int N, double *__restrict__ x, double *__restrict__ w, double *__restrict__ r,
                          const double *__restrict__ dv, const double *__restrict__ Kid,
                          const double *__restrict__ Ad, double *part, KScal *sc)
{
	if (sc->done) return;
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	double v[1] = {0.0};
	if (i < N) {
		double al = sc->alpha;
		for (int d = 0; d < D; ++d) {
			long k = (long) i * D + d;
			x[k] = 1.0 * x[k] + al * dv[k];
			w[k] = w[k] + al * Kid[k];
			double rk = 1.0 * r[k] + -al * Ad[k];
			r[k] = rk;
			v[0] += rk * rk;
		}
	}
	if (!kreduce<1>(v, part, &sc->counter)) return;
	double o[1]; kfinish<1>(o, part);
	if (threadIdx.x == 0) {
		sc->rSqu = o[0];
		sc->iters += 1;
		if (!isfinite(o[0])) { sc->code = SA_ERR_NONFINITE; sc->done = 1; }
		else if (o[0] < sc->bSqu * sc->tolSqu) sc->done = 1;
		else if (sc->iters >= sc->itrMax) { sc->code = SA_ERR_NOT_CONVERGED; sc->done = 1; }
		sc->counter = 0;
	}
}

__global__ void k_kp_zero(long n, double *x, double *w, const KScal *sc)
{
	if (sc->done != 2) return;
	long k = blockIdx.x * (long) blockDim.x + threadIdx.x;
	if (k < n) { x[k] = 0.0; w[k] = 0.0; }
}

// ---------------------------------------------------------------------------
// Fixed-point products with the RKHS matrix.  The product with D right-hand sides is N^2 D multiply-adds per
// iteration, which the FP64 pipe issues at 1.6 per clock per SM: 37 us of a 69 us iteration on the 3131-node strip, where
// the matrix itself (78 MB) streams from L2 in 5 us.  With the digits below the product takes 20 us there and the
// iteration 37 us.  The entries are therefore kept as two 28-bit digits (the bytes of the double; one frame for all of
// them, the largest entry's, |1 + eps| or 1) and multiplied on the integer pipes (sa_limb.cuh); r is converted once per CTA
// and product into shared memory.  Sums are exact but for 7 bits cut at each flush (2^-96 of the largest product over a row) and rounded once, and the matrix-free form, which converts the same entries on the fly and flushes at
// the same places, gives the same bits.  A far entry is rounded at 2^-55 of the largest, not of itself: in norm the product
// is as good as FP64's, and so are the solves (shells with orders -1 to 4, widths 0.1 to 1 and ldm 1e-3 to 1 against solves
// refined in 113 bits: errors 1.00 times those of FP64 products in the geometric mean).
// What bounds the solve on the strip is latency: issue 33 % of the cycles, integer pipe 30 %, multiply pipe 17 %
// (profiles/k_kpcg_persist_frame_demo_strip.md).
// ---------------------------------------------------------------------------
constexpr int kKpWarps = 16;
constexpr int kKpRows = 8;          // rows of a block: a warp multiplies 8 rows by 4 columns at a time
constexpr int kKpPass = 4;          // row blocks per pass of a CTA
constexpr int kKpLoad = 8;          // loads of a thread in flight (matrix entries, entries of r)
constexpr int kKpFlush = 64;        // products per lane between flushes into 128 bits (kLimbMaxTerms at most)
static_assert(kKpFlush <= kLimbMaxTerms, "digit sums would overflow");

// The stored matrix is tiled: 8 rows x 4 columns per 256 bytes, the tiles of a row block one after the other, so that a
// warp's load is two whole lines and the loads of a batch differ by constants.  Rows and columns past the end hold zero
// entries.
__host__ __device__ __forceinline__ int kernel_tiles(int N) { return (N + 3) / 4; }
__device__ __forceinline__ size_t kernel_place(int N, int i, int j)
{
	return ((size_t) (i / kKpRows) * kernel_tiles(N) + j / 4) * 32 + i % kKpRows + kKpRows * (j % 4);
}

size_t kernel_matrix_entries(int N)
{
	return (size_t) ((N + kKpRows - 1) / kKpRows) * kernel_tiles(N) * 32;
}

// the largest exponent field of a matrix whose entries may exceed 1 (Matern kernels of a width that is not positive: k grows
// with the distance there), into *e
template <int D>
__global__ void k_kernel_frame(int N, const double *__restrict__ x, int order, double w, double eps, int *e)
{
	int top = 1;
	const long pairs = (long) N * N;
	for (long k = blockIdx.x * (long) blockDim.x + threadIdx.x; k < pairs; k += (long) gridDim.x * blockDim.x) {
		const int i = (int) (k / N), j = (int) (k - (long) i * N);
		double v = kernel_entry<D>(order, w, load_node<D>(x, i), load_node<D>(x, j));
		if (i == j) v += eps;
		top = max(top, fx_exp(v));
	}
	top = fx_warp_max(top);
	if ((threadIdx.x & 31) == 0) atomicMax(e, top);
}

// the matrix as digits: one thread per entry on or above the diagonal writes the mirrored entry too (the entries are
// symmetric bit for bit).  An entry above the frame is not finite (nodes that are not, widths that overflow): *over = 2047
// then makes every product NaN.
template <int D>
__global__ void k_kernel_matrix_fix(int N, const double *__restrict__ x, int order, double w, double eps, int eA,
                                    int2 *__restrict__ K, int *over)
{
	const int lane = threadIdx.x & 31, ct = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
	if (ct >= kernel_tiles(N)) return;
	const int j = 4 * ct + lane / kKpRows;
	const int nb = (N + kKpRows - 1) / kKpRows;
	Vec<D> qj;
	for (int d = 0; d < D; ++d) qj.c[d] = j < N ? x[(long) j * D + d] : 0.0;
	for (int b = blockIdx.y; b < nb; b += gridDim.y) {
		const int i = b * kKpRows + lane % kKpRows;
		if (i >= N || j >= N) {
			K[((size_t) b * kernel_tiles(N) + ct) * 32 + lane] = make_int2(0, 0);
			continue;
		}
		if (i > j) continue;
		double v = kernel_entry<D>(order, w, load_node<D>(x, i), qj);
		if (i == j) v += eps;
		if (fx_exp(v) > eA) atomicMax(over, 2047);
		int2 t;
		limb_matrix(v, eA, t.x, t.y);
		K[kernel_place(N, i, j)] = t;
		K[kernel_place(N, j, i)] = t;
	}
}

// a digit sum in 128 bits, moved down to leave room for the sum over up to 2^22 columns of products below 2^111
constexpr int kKpRoom = 7;
__device__ __forceinline__ Fx kernel_fixed(const LimbSum &t)
{
	const Fx f = limb_fixed(t);
	return Fx{(f.lo >> kKpRoom) | (f.hi << (64 - kKpRoom)), (unsigned long long) ((long long) f.hi >> kKpRoom)};
}

__device__ __forceinline__ Fx fx_xor_add(Fx f, int lanes)
{
	return fx_add(f, Fx{__shfl_xor_sync(0xffffffffu, f.lo, lanes), __shfl_xor_sync(0xffffffffu, f.hi, lanes)});
}

template <int D> struct KpSmem {
	Fx seg[kKpPass][kKpWarps][D][kKpRows];
	int e[kKpWarps];
	int bad;                          // an entry evaluated in the product was above the frame
};

// first row block of CTA c: the blocks of kKpRows rows are dealt out evenly and contiguously
__device__ __forceinline__ int kernel_block0(int N, int c, int nctas)
{
	const int nb = (N + kKpRows - 1) / kKpRows;
	return (int) ((long) nb * c / nctas);
}

// Kr = K r for the CTA's row blocks [q0, q1): digits of r in shared memory (dig, at most cap nodes at a time, node by node),
// warp w takes the w-th sixteenth of the columns; lane = row of the block + 8 (column mod 4), so the matrix is read in
// 64-byte pieces and only two lane exchanges per block add the columns.  out(row, component, value) once per
// result by one thread.  Every thread of the CTA calls.
template <int D, bool kFree, typename Out>
__device__ __forceinline__ void kernel_rows(int N, const int2 *__restrict__ K, const double *__restrict__ q, int order,
                                            double kw, double eps, int eA, const double *r, int q0, int q1, int2 *dig,
                                            int cap, KpSmem<D> &sm, Out out)
{
	const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, W = blockDim.x >> 5;
	const int nch = (N + cap - 1) / cap;
	// r (raw, in place of the digits) and its largest exponent.  Each CTA starts at another place: all of them read all of r
	// right after the barrier, and in step they would queue at one L2 slice after the other
	double *raw = reinterpret_cast<double *>(dig);
	int eU = 1;
	{
		const int n = min(N, cap) * D, rot = (int) ((unsigned) n * blockIdx.x / gridDim.x);
		int e = 1;
		for (int t0 = threadIdx.x; t0 < n; t0 += kKpLoad * blockDim.x) {
			double v[kKpLoad];                   // all loads before the first store
#pragma unroll
			for (int u = 0; u < kKpLoad; ++u) {
				const int t = t0 + u * blockDim.x, k = t + rot < n ? t + rot : t + rot - n;
				v[u] = t < n ? __ldcg(r + k) : 0.0;
			}
#pragma unroll
			for (int u = 0; u < kKpLoad; ++u) {
				const int t = t0 + u * blockDim.x, k = t + rot < n ? t + rot : t + rot - n;
				if (t < n) raw[k] = v[u];
				e = max(e, fx_exp(v[u]));
			}
		}
		for (int t = n + threadIdx.x; t < N * D; t += blockDim.x) e = max(e, fx_exp(__ldcg(r + t)));
		e = fx_warp_max(e);
		if (lane == 0) sm.e[wp] = e;
		if (threadIdx.x == 0) sm.bad = 0;
		__syncthreads();
		eU = fx_warp_max(lane < W ? sm.e[lane] : 1);
	}
	for (int p0 = q0; p0 < q1; p0 += kKpPass) {
		const int nb = min(kKpPass, q1 - p0);
		for (int c = 0; c < nch; ++c) {
			const int n0 = c * cap, n = min(N, n0 + cap) - n0;
			if (nch > 1 || p0 == q0) {           // digits of the chunk's nodes
				const bool again = nch > 1 && (c > 0 || p0 > q0);
				if (again) __syncthreads();      // the chunk before has been read
#pragma unroll 2
				for (int t = threadIdx.x; t < n * D; t += blockDim.x) {
					int2 g;
					limb_vector(again ? __ldcg(r + (long) n0 * D + t) : raw[t], eU, g.x, g.y);
					dig[t] = g;
				}
				__syncthreads();
			}
			const int tiles = (n + 3) / 4, t0 = (int) ((unsigned) tiles * wp / W), t1 = (int) ((unsigned) tiles * (wp + 1) / W);
			// batches of kKpLoad tiles, the next batch's entries loaded (also across row blocks) before a batch is used
			const int mb = max(1, (t1 - t0 + kKpLoad - 1) / kKpLoad), full = (t1 - t0) / kKpLoad;
			const int jl = 4 * t0 + (lane >> 3);     // the lane's first column in the chunk
			int2 ka[kKpLoad], kb[kKpLoad];
			auto entries = [&](int b, int t, int2 (&k)[kKpLoad]) {
				if constexpr (kFree) {
					const int i = (p0 + b) * kKpRows + (lane & 7);
					const Vec<D> qi = load_node<D>(q, min(i, N - 1));
#pragma unroll
					for (int u = 0; u < kKpLoad; ++u) {
						const int tile = t0 + kKpLoad * t + u, j = n0 + 4 * tile + (lane >> 3);
						k[u] = make_int2(0, 0);
						if (tile < t1 && i < N && j < N) {
							double v = kernel_entry<D>(order, kw, qi, load_node<D>(q, j));
							if (i == j) v += eps;
							if (fx_exp(v) > eA) sm.bad = 1;
							limb_matrix(v, eA, k[u].x, k[u].y);
						}
					}
				} else {
					const int2 *p = K + ((size_t) (p0 + b) * kernel_tiles(N) + n0 / 4 + t0 + kKpLoad * t) * 32 + lane;
#pragma unroll
					for (int u = 0; u < kKpLoad; ++u) {
						k[u] = make_int2(0, 0);
						if (t < full || t0 + kKpLoad * t + u < t1)
							asm volatile("ld.global.nc.L1::no_allocate.v2.s32 {%0, %1}, [%2];" : "=r"(k[u].x), "=r"(k[u].y) : "l"(p + 32 * u));
					}
				}
			};
			LimbSum acc[D];
			Fx tot[D];
			auto use = [&](int b, int t, const int2 (&k)[kKpLoad]) {
				if (t == 0)
#pragma unroll
					for (int d = 0; d < D; ++d) { tot[d] = fx_zero(); acc[d] = limb_zero(); }
				const int2 *g = dig + (jl + 4 * kKpLoad * t) * D;
				if (t < full) {
#pragma unroll
					for (int u = 0; u < kKpLoad; ++u)
#pragma unroll
						for (int d = 0; d < D; ++d) limb_mac(acc[d], k[u].x, k[u].y, g[4 * u * D + d].x, g[4 * u * D + d].y);
				} else {
					const int rem = t1 - t0 - kKpLoad * full;
#pragma unroll
					for (int u = 0; u < kKpLoad - 1; ++u)
						if (u < rem)                 // the same for the whole warp
#pragma unroll
							for (int d = 0; d < D; ++d) limb_mac(acc[d], k[u].x, k[u].y, g[4 * u * D + d].x, g[4 * u * D + d].y);
				}
				const bool last = t == mb - 1;
				if (last || (t + 1) % (kKpFlush / kKpLoad) == 0)
#pragma unroll
					for (int d = 0; d < D; ++d) { tot[d] = fx_add(tot[d], kernel_fixed(acc[d])); acc[d] = limb_zero(); }
				if (last)
#pragma unroll
					for (int d = 0; d < D; ++d) {
						const Fx s = fx_xor_add(fx_xor_add(tot[d], 8), 16);
						if (lane < kKpRows) sm.seg[b][wp][d][lane] = c == 0 ? s : fx_add(sm.seg[b][wp][d][lane], s);
					}
			};
			int b = 0, t = 0;
			auto next = [&](int &bn, int &tn) { if (++tn == mb) { tn = 0; ++bn; } };
			entries(0, 0, ka);
			while (b < nb) {
				int bn = b, tn = t;
				next(bn, tn);
				if (bn < nb) entries(bn, tn, kb);
				use(b, t, ka);
				b = bn; t = tn;
				if (b >= nb) break;
				next(bn, tn);
				if (bn < nb) entries(bn, tn, ka);
				use(b, t, kb);
				b = bn; t = tn;
			}
		}
		__syncthreads();
		for (int t = threadIdx.x; t < nb * D * kKpRows; t += blockDim.x) {
			const int a = t % kKpRows, d = t / kKpRows % D, b = t / (kKpRows * D), i = (p0 + b) * kKpRows + a;
			Fx s = fx_zero();
#pragma unroll 4
			for (int g = 0; g < kKpWarps; ++g) s = fx_add(s, sm.seg[b][g][d][a]);
			const double v = eU >= 2047 || eA >= 2047 || (kFree && sm.bad) ? limb_bits(0x7FF8000000000000ull) : limb_round(s, eA + eU - 1020 + kKpRoom);
			if (i < N) out(i, d, v);
		}
		__syncthreads();
	}
}

// y = K x, one launch (the products outside the persistent kernel)
template <int D, bool kFree>
__global__ void __launch_bounds__(32 * kKpWarps, 1)
k_kernel_product(int N, const int2 *__restrict__ K, const double *__restrict__ q, int order, double kw, double eps, int frame,
                 const int *over, const double *x, double *y, int cap)
{
	extern __shared__ __align__(16) int2 kdig[];
	__shared__ KpSmem<D> sm;
	const int eA = max(frame, __ldg(over));
	kernel_rows<D, kFree>(N, K, q, order, kw, eps, eA, x, kernel_block0(N, blockIdx.x, gridDim.x),
	                      kernel_block0(N, blockIdx.x + 1, gridDim.x), kdig, cap, sm,
	                      [&](int i, int d, double v) { y[(long) i * D + d] = v; });
}

// ---------------------------------------------------------------------------
// Persistent K-preconditioned CG: one cooperative launch runs all iterations of the loop below (six launches per
// iteration there).  One CTA per SM, kKpWarps warps.  Per iteration three grid-wide exact sums that carry the grid's
// barriers (sum_exchange in sa_grid.cuh; the first iteration, and values that leave their frames, take the partial-sum
// path):
//   A  Kid = r + beta Kid, d = Kr + beta d and Ad = ldm Kid + (E + btm P) d, with (d, Ad) -> alpha.  Eight warps share
//      a slice, each a few of its slots (a row's serial chain of gathers and FP64 operations was 4 us), their partial
//      products added in a fixed order.  A row that gathers a neighbour's d forms it the same way from the
//      neighbour's previous d and Kr (two d buffers alternate), so no barrier separates the direction update from
//      the operator;
//   B  rows: x += alpha d, w += alpha Kid, r -= alpha Ad, with (r, r) -> stop test;
//   C  Kr = K r (kernel_rows), with (r, Kr) -> beta.
// Vectors that other CTAs write during the launch are read with __ldcg (L2), never through the
// incoherent L1.  Iterates, stopping rule and status codes are those of the loop below.
// ---------------------------------------------------------------------------
constexpr int kKpParts = 8;         // warps that share a slice in phase A
constexpr int kKpGroups = kKpWarps / kKpParts;

struct KpVec {
	double *x, *w, *r, *Kr, *Kid, *d0, *d1, *Ad;
};

// sum lines of the three sums (each rotates over three)
struct KpSums { GridBar bar; SumLine line[3][3]; };
static_assert(sizeof(KpSums) <= kGridBarBytes, "sum lines larger than their allocation");

__device__ __forceinline__ double kp_dir(double kr, double dOld, double be, bool first)
{
	return first ? kr : __fma_rn(be, dOld, kr);
}

// One grid sum: v summed over all threads of all CTAs; also the grid's barrier (the CTA's writes are visible to the CTAs that
// passed it).  prev: the sum's value of the iteration before (its frame); slow: no such value yet.  post(sum) runs once per
// CTA, in one thread, before the CTA goes on: scalar FP64 work in every warp would queue at the FP64 pipe.  false: a wait
// gave up.
template <typename Post>
__device__ __forceinline__ bool kp_sum(double v, double prev, bool slow, int which, int turn, KpSums *ks, double *part,
                                       unsigned &target, unsigned (*dig)[kSumWords], int *state, FxScratch &fs, Post post)
{
	const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, W = blockDim.x >> 5, nctas = gridDim.x;
	bool part_path = slow;
	if (!slow) {
		const int frame[1] = {sum_frame(prev)};
		const double t[1] = {v};
		warp_digits<1>(t, frame, dig[wp]);
		__syncthreads();
		if (wp == 0) {
			double o[1];
			bool flag = false;
			__threadfence();
			const bool ok = sum_exchange<1>(dig[0], W, &ks->line[which][turn], nctas, frame, &ks->bar, o, flag);
			if (blockIdx.x == 0 && lane < kSumWords) ks->line[which][turn >= 1 ? turn - 1 : 2].w[lane] = 0ull;
			if (lane == 0) {
				*state = ok ? (flag ? 1 : 0) : 2;
				if (ok && !flag) post(o[0]);
			}
		}
		__syncthreads();
		if (*state == 2) return false;
		part_path = *state == 1;
	}
	if (part_path) {
		double a[1] = {v}, o[1];
		if (!grid_reduce<1, double>(a, o, part + which * nctas, blockIdx.x, nctas, &ks->bar, target, fs)) return false;
		if (threadIdx.x == 0) post(o[0]);
		__syncthreads();
	}
	return true;
}

constexpr int kKpColSlots = 4;      // slots of a warp whose columns are kept in shared memory (one slice per warp)

template <int D, bool kFree>
__global__ void __launch_bounds__(32 * kKpWarps, 1)
k_kpcg_persist(SellOp A, const double *__restrict__ blk, const int2 *__restrict__ K, const double *__restrict__ q,
               int order, double kw, double eps, int frame, const int *over, KpVec v, double *part, KScal *sc, KpSums *ks, int cap)
{
	extern __shared__ __align__(16) int2 kdig[];
	__shared__ FxScratch fs;
	__shared__ KpSmem<D> sm;
	__shared__ unsigned dig[kKpWarps][kSumWords];
	__shared__ double apart[kKpWarps][D][32];
	__shared__ int scol[kKpWarps][kKpColSlots][32];
	__shared__ double rKr, rr, dAd, alpha, be;
	__shared__ int sstate, code, it;
	if (sc->done) return;                       // set before the launch: the same for every CTA
	const int N = A.N, nctas = gridDim.x, lc = blockIdx.x, eA = max(frame, __ldg(over));
	const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
	// rows of phases A and B: 32-row slices dealt round-robin over the CTAs first, so that a small mesh
	// spreads its row work (gathers) over all SMs instead of the first few CTAs
	const int nsl = (N + 31) >> 5, grp = wp / kKpParts, prt = wp - grp * kKpParts;
	const double ldm = sc->ldmWgt;
	if (threadIdx.x == 0) { rKr = sc->rKr; rr = sc->rSqu; dAd = 0.0; be = 0.0; it = sc->iters; code = -1; }
	const double goal = sc->bSqu * sc->tolSqu;
	const int itrMax = sc->itrMax;
	{   // columns of the warp's first slice
		const int sl = blockIdx.x + gridDim.x * grp;
		const int w0 = sl < nsl ? __ldg(A.width + sl) : 0;
		for (int k = prt, t = 0; k < w0 && t < kKpColSlots; k += kKpParts, ++t)
			scol[wp][t][lane] = __ldg(A.col + __ldg(A.off + sl) + lane + 32 * k);
	}
	int turn = 0;
	bool first = true, ok = true;
	unsigned int target = 0;
	const int r0 = kernel_block0(N, lc, nctas), r1 = kernel_block0(N, lc + 1, nctas);       // row blocks of phase C
	double *dOld = v.d0, *dNew = v.d1;
	__syncthreads();
	for (;;) {
		// A: direction, operator, (d, Ad)
		double loc = 0.0;
		for (int s0 = blockIdx.x; s0 < nsl; s0 += gridDim.x * kKpGroups) {
			const int sl = s0 + gridDim.x * grp;
			const double b = be;
			double acc[D];
			for (int c = 0; c < D; ++c) acc[c] = 0.0;
			if (sl < nsl) {
				const int wdt = __ldg(A.width + sl);
				const long base = __ldg(A.off + sl) + lane;
#pragma unroll 2
				for (int k = prt, t = 0; k < wdt; k += kKpParts, ++t) {
					const long idx = base + ((long) k << 5);
					const int j = s0 == (int) blockIdx.x && t < kKpColSlots ? scol[wp][t][lane] : __ldg(A.col + idx);
					double dj[D];
					for (int c = 0; c < D; ++c)
						dj[c] = kp_dir(__ldcg(v.Kr + (long) j * D + c), first ? 0.0 : __ldcg(dOld + (long) j * D + c),
						               b, first);
					double a[D * D];
					load_block<D, double>(blk, A.total, idx, a);
					for (int r = 0; r < D; ++r)
						for (int c = 0; c < D; ++c) acc[r] += a[r * D + c] * dj[c];
				}
			}
			for (int c = 0; c < D; ++c) apart[wp][c][lane] = acc[c];
			// one warp per (group, component): its row's vectors meanwhile, then the parts in order
			const int g = wp / D, c = wp - g * D, slg = s0 + gridDim.x * g, ig = slg * 32 + lane;
			const bool rows = wp < kKpGroups * D && slg < nsl && ig < N;
			const long k = (long) ig * D + c;
			double kid = 0.0, di = 0.0;
			if (rows) {
				const double ri = __ldcg(v.r + k), kr = __ldcg(v.Kr + k);
				const double ko = first ? 0.0 : __ldcg(v.Kid + k), d0 = first ? 0.0 : __ldcg(dOld + k);
				kid = first ? ri : __fma_rn(b, ko, ri);
				di = kp_dir(kr, d0, b, first);
				v.Kid[k] = kid;
				dNew[k] = di;
			}
			__syncthreads();
			if (rows) {
				double t = apart[g * kKpParts][c][lane];
				for (int p = 1; p < kKpParts; ++p) t += apart[g * kKpParts + p][c][lane];
				const double ad = __fma_rn(ldm, kid, t);
				v.Ad[k] = ad;
				loc += di * ad;
			}
			__syncthreads();
		}
		ok = kp_sum(loc, dAd, first, 0, turn, ks, part, target, dig, &sstate, fs, [&](double o) {
			dAd = o;
			if (o == 0.0 || fx_exp(o) >= 2047) code = o == 0.0 ? SA_ERR_BREAKDOWN : SA_ERR_NONFINITE;
			alpha = rKr / o;
		});
		if (!ok || code >= 0) break;
		// B: x, w, r and (r, r), one warp per (slice, component) as they were written in A
		loc = 0.0;
		const double al = alpha;
		for (int s0 = blockIdx.x; s0 < nsl; s0 += gridDim.x * kKpGroups) {
			if (wp >= kKpGroups * D) continue;
			const int g = wp / D, c = wp - g * D, slg = s0 + gridDim.x * g, ig = slg * 32 + lane;
			if (slg >= nsl || ig >= N) continue;
			const long k = (long) ig * D + c;
			const double x0 = v.x[k], d0 = dNew[k], w0 = v.w[k], k0 = v.Kid[k], a0 = v.Ad[k], q0 = __ldcg(v.r + k);
			const double rk = __fma_rn(-al, a0, q0);
			v.r[k] = rk;
			v.x[k] = __fma_rn(al, d0, x0);
			v.w[k] = __fma_rn(al, k0, w0);
			loc += rk * rk;
		}
		ok = kp_sum(loc, rr, false, 1, turn, ks, part, target, dig, &sstate, fs, [&](double o) {
			rr = o;
			const int n = ++it;
			if (fx_exp(o) >= 2047) code = SA_ERR_NONFINITE;
			else if (o < goal) code = SA_OK;
			else if (n >= itrMax) code = SA_ERR_NOT_CONVERGED;
		});
		if (!ok || code >= 0) break;
		// C: Kr = K r over the CTA's rows, (r, Kr)
		loc = 0.0;
		kernel_rows<D, kFree>(N, K, q, order, kw, eps, eA, v.r, r0, r1, kdig, cap, sm, [&](int i, int d, double y) {
			const long k = (long) i * D + d;
			v.Kr[k] = y;
			loc += __ldcg(v.r + k) * y;
		});
		ok = kp_sum(loc, rKr, false, 2, turn, ks, part, target, dig, &sstate, fs, [&](double o) {
			if (o == 0.0 || fx_exp(o) >= 2047) code = o == 0.0 ? SA_ERR_BREAKDOWN : SA_ERR_NONFINITE;
			else { be = o / rKr; rKr = o; }
		});
		if (!ok || code >= 0) break;
		first = false;
		if (++turn == 3) turn = 0;
		double *t = dOld; dOld = dNew; dNew = t;
	}
	if (lc == 0 && threadIdx.x == 0) {
		sc->iters = it; sc->code = ok ? code : SA_ERR_TIMEOUT; sc->rSqu = rr; sc->rKr = rKr; sc->done = 1;
	}
}

static int device_sm_count()
{
	int dev = 0, n = 0;
	SA_CHECK(cudaGetDevice(&dev));
	SA_CHECK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
	return n;
}

// nodes of r whose digits one CTA holds at a time: all of them up to 160 KB
constexpr int kKpDigBytes = 160 * 1024;
template <int D> static int kernel_dig_nodes(int N) { return std::min((N + 3) / 4 * 4, kKpDigBytes / (int) (4 * D * sizeof(int2)) * 4); }

// whether the solves of this mesh can run as the persistent K-PCG
template <int D>
static bool kpcg_can_persist(const Model &md, int N)
{
	if (md.cgKernel == SA_CG_TWO_KERNEL || device_sm_count() > kSumMaxCtas) return false;
	const size_t bytes = sizeof(int2) * (size_t) D * kernel_dig_nodes<D>(N);
	const void *kernel = md.kernelFree ? (const void *) k_kpcg_persist<D, true> : (const void *) k_kpcg_persist<D, false>;
	if (bytes > smem_limit(kernel)) return false;
	int occ = 0;
	const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 32 * kKpWarps, bytes);
	if (e != cudaSuccess) { cudaGetLastError(); return false; }
	return occ >= 1;
}

// one cooperative launch of the persistent K-PCG
template <int D, bool kFree>
static void kpcg_persist_launch(const Mesh &m, const Model &md, const double *blk, const int2 *K, const double *q,
                                double *x, KpcgWork &wk, KScal *sc, cudaStream_t s)
{
	int cap = kernel_dig_nodes<D>(m.N);
	const size_t bytes = sizeof(int2) * (size_t) D * cap;
	const int nctas = device_sm_count();
	KpSums *ks = (KpSums *) wk.bar;
	SA_CHECK(cudaMemsetAsync(ks, 0, sizeof(KpSums), s));
	SellOp A = sell_of(m);
	KpVec v{x, wk.wK, wk.r, wk.Kr, wk.Kid, wk.dv, wk.dv2, wk.Ad};
	int order = md.knlOrder, eA = wk.eA;
	const int *over = wk.over();
	double kw = md.knlWidth, eps = md.knlEps;
	double *part = wk.part;
	void *args[] = {&A, (void *) &blk, (void *) &K, (void *) &q, &order, &kw, &eps, &eA, &over, &v, &part, &sc, &ks, &cap};
	SA_CHECK(cudaLaunchCooperativeKernel((const void *) k_kpcg_persist<D, kFree>, dim3(nctas), dim3(32 * kKpWarps),
	                                     args, bytes, s));
}

// y = K x with the digit matrix, or evaluated on the fly (K null)
template <int D>
static void kernel_product(const Model &md, int N, const int2 *K, const double *q, const KpcgWork &wk, const double *x, double *y,
                           cudaStream_t s)
{
	const int cap = kernel_dig_nodes<D>(N);
	const size_t bytes = sizeof(int2) * (size_t) D * cap;
	const int nctas = std::min(device_sm_count(), (N + kKpRows - 1) / kKpRows);
	auto kernel = K ? k_kernel_product<D, false> : k_kernel_product<D, true>;
	if (bytes > smem_limit((const void *) kernel)) throw CudaError{cudaErrorInvalidValue, "K product: shared memory"};
	kernel<<<nctas, 32 * kKpWarps, bytes, s>>>(N, K, q, md.knlOrder, md.knlWidth, md.knlEps, wk.eA, wk.over(), x, y, cap);
}

template <int D>
void launch_kernel_matrix(const Model &md, int N, const double *x, double *K, KpcgWork &w, cudaStream_t s)
{
	SA_CHECK(cudaMemsetAsync(w.over(), 0, sizeof(int), s));
	w.eA = limb_unit_frame(md.knlEps);
	if (md.knlOrder >= 0 && !(md.knlWidth > 0.0)) {
		k_kernel_frame<D><<<4 * device_sm_count(), 256, 0, s>>>(N, x, md.knlOrder, md.knlWidth, md.knlEps, w.over());
		SA_CHECK(cudaMemcpyAsync(&w.eA, w.over(), sizeof(int), cudaMemcpyDeviceToHost, s));
		SA_CHECK(cudaStreamSynchronize(s));
	}
	if (!K) return;
	dim3 g(grid_for(kernel_tiles(N), 4), std::min((N + kKpRows - 1) / kKpRows, 65535));
	k_kernel_matrix_fix<D><<<g, 128, 0, s>>>(N, x, md.knlOrder, md.knlWidth, md.knlEps, w.eA, (int2 *) (void *) K, w.over());
}

template <int D>
int kpcg(const Mesh &m, const Model &md, const double *blk, const double *K, const double *q, const double *b,
         double *x, KpcgWork &wk, Status *st, int *itersOut, cudaStream_t s)
{
	(void) st;
	int N = m.N;
	long n = (long) N * D;
	int nb = grid_for(N, kKBlock);
	KScal h{};
	h.tolSqu = md.cgTolSqu; h.itrMax = md.cgItrMax; h.ldmWgt = md.ldmWgt;
	KScal *sc = (KScal *) wk.scal;
	SA_CHECK(cudaMemcpyAsync(sc, &h, sizeof(KScal), cudaMemcpyHostToDevice, s));
	const int2 *Kfix = (const int2 *) (const void *) K;
	const bool persist = kpcg_can_persist<D>(md, N);
	auto product = [&](const double *in, double *out) { kernel_product<D>(md, N, Kfix, q, wk, in, out, s); };
	k_kp_bnorm<D><<<nb, kKBlock, 0, s>>>(N, b, wk.part, sc);
	// warm start x0 = K w (w = K^{-1} v of the previous step)
	product(wk.wK, x);
	k_kp_init_r<D><<<nb, kKBlock, 0, s>>>(sell_of(m), blk, b, x, wk.wK, wk.r, wk.part, sc);
	product(wk.r, wk.Kr);
	k_kp_rkr<D><<<nb, kKBlock, 0, s>>>(N, wk.r, wk.Kr, wk.part, sc, 1);
	k_kp_dir<D><<<grid_for(n), kBlock, 0, s>>>(N, wk.r, wk.Kr, wk.Kid, wk.dv, sc, 1);
	SA_CHECK(cudaGetLastError());
	if (persist) {
		if (K) kpcg_persist_launch<D, false>(m, md, blk, Kfix, q, x, wk, sc, s);
		else kpcg_persist_launch<D, true>(m, md, blk, Kfix, q, x, wk, sc, s);
	}
	const int chunk = 8;
	for (int it = 0; !persist && it < md.cgItrMax + chunk; it += chunk) {
		for (int k = 0; k < chunk; ++k) {
			k_kp_ad<D><<<nb, kKBlock, 0, s>>>(sell_of(m), blk, wk.dv, wk.Kid, wk.Ad, wk.part, sc);
			k_kp_step<D><<<nb, kKBlock, 0, s>>>(N, x, wk.wK, wk.r, wk.dv, wk.Kid, wk.Ad, wk.part, sc);
			product(wk.r, wk.Kr);
			k_kp_rkr<D><<<nb, kKBlock, 0, s>>>(N, wk.r, wk.Kr, wk.part, sc, 0);
			k_kp_dir<D><<<grid_for(n), kBlock, 0, s>>>(N, wk.r, wk.Kr, wk.Kid, wk.dv, sc, 0);
		}
		SA_CHECK(cudaGetLastError());
		SA_CHECK(cudaMemcpyAsync(&h, sc, sizeof(KScal), cudaMemcpyDeviceToHost, s));
		SA_CHECK(cudaStreamSynchronize(s));
		if (h.done) break;
	}
	k_kp_zero<<<grid_for(n), kBlock, 0, s>>>(n, x, wk.wK, sc);
	SA_CHECK(cudaMemcpyAsync(&h, sc, sizeof(KScal), cudaMemcpyDeviceToHost, s));
	SA_CHECK(cudaStreamSynchronize(s));
	if (itersOut) *itersOut = h.iters;
	return h.code;
}

template void launch_adj_kernel_term<2>(const Model &, int, const double *, const double *, const double *, double *,
                                        cudaStream_t);
template void launch_adj_kernel_term<3>(const Model &, int, const double *, const double *, const double *, double *,
                                        cudaStream_t);
template void launch_kernel_matrix<2>(const Model &, int, const double *, double *, KpcgWork &, cudaStream_t);
template void launch_kernel_matrix<3>(const Model &, int, const double *, double *, KpcgWork &, cudaStream_t);
template int kpcg<2>(const Mesh &, const Model &, const double *, const double *, const double *, const double *,
                     double *, KpcgWork &, Status *, int *, cudaStream_t);
template int kpcg<3>(const Mesh &, const Model &, const double *, const double *, const double *, const double *,
                     double *, KpcgWork &, Status *, int *, cudaStream_t);

}  // namespace sa
