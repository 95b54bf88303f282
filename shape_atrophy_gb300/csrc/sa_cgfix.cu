// sa_cgfix.cu -- persistent block-Jacobi CG whose matrix products are summed in fixed point.
//
// The FP64 velocity solve of k_cg_persist (sa_cg.cu) is bound by the FP64 pipe: 9 multiply-adds per 3 x 3 block
// at 64 clocks per warp and SM sub-partition, 22 of the 35 us of an iteration on the 92 178-node shell, against
// 6 us for reading the operator (94 MB) from the L2.  Here the products go through the integer pipes
// (sa_limb.cuh), which takes them off the critical path and leaves the loads:
//   * the solve runs on a scaled system (D^-1/2 A D^-1/2, powers of two; see the scales below), so that digits cut relative
//     to a row's and a halo's largest entry lose nothing where soft and stiff materials meet;
//   * the operator is converted once per solve to two digits per entry, of 28 and of up to 32 bits (k_cgfix_operator; the
//     bytes of the FP64 entry).  A slice that fits its warp's ring of slots in shared memory stays there for the whole solve;
//     of larger ones as many slots as fit stay in tensor memory (39 MB over the chip: with the operator, the vectors
//     and u the working set of the shell is 107 MB, beyond what the L2 holds of a cyclic scan), and the rest is
//     streamed by bulk copies into the ring, ahead of its use and across the grid barriers;
//   * the vector u is converted once per CTA and iteration: the distinct nodes a chunk's rows gather (its
//     halo, about 1.7 times its rows in Morton order; in the icosphere's own numbering nearly every slot is a node of
//     its own) are read into shared memory as two 28-bit digits relative to the halo's largest entry, so a
//     slot's gather is six shared-memory words instead of two L2 requests;
//   * the two grid sums of an iteration carry their own barrier (sum_exchange in sa_grid.cuh).
// The shell's iteration takes 21 us here (43 thousand clocks: products 20, vector updates 6, halo 6, the two grid sums 7)
// instead of 35; the 4 096-node annulus, bound by the sums, 8.9 -> 6.3 us; above 92 416 rows (19 slices on each of 152 SMs)
// k_cg_fix_many.  What bounds it is latency: of the shell's solve the warps issue in 36 % of the cycles, the integer pipe is
// busy in 28 %, the multiply pipe in 17 %, the FP64 pipe in 21 %; a waiting warp waits at barriers (grid sums and between
// phases), then on dependent instructions and on shared and global loads (profiles/k_cg_fix.md).
// The recurrences, the reducer warp and the stopping rule are those of k_cg_persist (sa_cg.cu): Chronopoulos-Gear
// in FP64, exact grid sums, bounded waits.
#include "sa_internal.cuh"
#include "sa_grid.cuh"
#include "sa_limb.cuh"
#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

namespace sa {

constexpr int kFixMaxWarps = 20;           // CTA size limit, reducer warp included (as the persistent CG's)
constexpr int kFixMinWarps = 8;            // small solves: warps without rows help to stage the halo
constexpr int kFixMaxParts = 8;            // warps per slice
constexpr int kFixMaxHalo = 8192;          // halo nodes per chunk (shared memory takes about 6000 of them)
constexpr int kFixStagers = 4;             // warps that stage at least, with several chunks per CTA
constexpr int kFixMaxRows = 1 << 20;       // permuted rows whose bit map and prefix counts fit shared memory

// the frame of a row of w 2^s and the exponent s of the row's scale in one word (both within 16 bits)
__host__ __device__ __forceinline__ int row_pack(int e, int s) { return (int) ((unsigned) e << 16 | ((unsigned) s & 0xffffu)); }
__host__ __device__ __forceinline__ int row_frame(int w) { return w >> 16; }
__host__ __device__ __forceinline__ int row_scale(int w) { return (short) w; }

constexpr int kLimbStride = 6;             // words per halo node: three 8-byte bank pairs, odd, so consecutive nodes spread
template <int B> constexpr int fix_u_stride() { return B == 3 ? 4 : 2; }   // doubles per node of the gather copy

// ---------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------
// one CTA per chunk: its rows sorted by length (longest first, ties in Morton order)
__global__ void k_plan_rows(int N, int nchunk, int R, const unsigned long long *__restrict__ keys,
                            const int *__restrict__ rowPtr, int *__restrict__ perm, int *__restrict__ inv,
                            int *__restrict__ width)
{
	extern __shared__ int sh[];
	int *deg = sh, *sorted = sh + R;
	const int c = blockIdx.x, r0 = (int) ((long) c * N / nchunk), n = (int) ((long) (c + 1) * N / nchunk) - r0;
	for (int t = threadIdx.x; t < n; t += blockDim.x) {
		const int i = (int) (keys[r0 + t] & 0xffffffffu);
		deg[t] = rowPtr[i + 1] - rowPtr[i];
	}
	__syncthreads();
	for (int t = threadIdx.x; t < R; t += blockDim.x) {
		if (t >= n) { perm[(long) c * R + t] = -1; continue; }
		const int d = deg[t], i = (int) (keys[r0 + t] & 0xffffffffu);
		int rank = 0;
		for (int q = 0; q < n; ++q) rank += deg[q] > d || (deg[q] == d && q < t);
		perm[(long) c * R + rank] = i;
		inv[i] = c * R + rank;
		sorted[rank] = d;
	}
	__syncthreads();
	for (int q = threadIdx.x; q < R / 32; q += blockDim.x) width[c * (R / 32) + q] = 32 * q < n ? sorted[32 * q] : 0;
}

// first slot of every slice (one CTA); off[ns] = total
__global__ void __launch_bounds__(1024) k_plan_offsets(int ns, const int *__restrict__ width, int *__restrict__ off)
{
	__shared__ int sum[1024];
	const int t = threadIdx.x, per = (ns + 1023) / 1024, a = min(ns, t * per), b = min(ns, a + per);
	int s = 0;
	for (int q = a; q < b; ++q) s += 32 * width[q];
	sum[t] = s;
	__syncthreads();
	for (int h = 1; h < 1024; h <<= 1) {
		const int v = t >= h ? sum[t - h] : 0;
		__syncthreads();
		sum[t] += v;
		__syncthreads();
	}
	int o = sum[t] - s;
	for (int q = a; q < b; ++q) { off[q] = o; o += 32 * width[q]; }
	if (t == 1023) off[ns] = sum[1023];
}

// one CTA per chunk: the distinct columns of its rows (bit map over the permuted rows, prefix counts per word),
// its halo list, and every slot's place in that list (padding slots: place 0, their entries are zero)
__global__ void k_plan_columns(int P, int R, const int *__restrict__ rowPtr, const int *__restrict__ col,
                               const int *__restrict__ perm, const int *__restrict__ inv,
                               const int *__restrict__ width, const int *__restrict__ off, int haloCap,
                               int *__restrict__ halo, int *__restrict__ haloNum, unsigned short *__restrict__ lcol)
{
	extern __shared__ int sh[];
	__shared__ int part[1025];
	const int nw = (P + 31) / 32, c = blockIdx.x, t0 = threadIdx.x, nt = blockDim.x;
	unsigned *bits = (unsigned *) sh;
	unsigned short *pre = (unsigned short *) (sh + nw);
	for (int w = t0; w < nw; w += nt) bits[w] = 0u;
	__syncthreads();
	for (int t = t0; t < R; t += nt) {
		const int i = perm[(long) c * R + t];
		if (i < 0) continue;
		for (int z = rowPtr[i]; z < rowPtr[i + 1]; ++z) {
			const int q = inv[col[z]];
			atomicOr(&bits[q >> 5], 1u << (q & 31));
		}
	}
	__syncthreads();
	const int per = (nw + nt - 1) / nt, a = min(nw, t0 * per), b = min(nw, a + per);
	int s = 0;
	for (int w = a; w < b; ++w) s += __popc(bits[w]);
	part[t0 + 1] = s;
	if (t0 == 0) part[0] = 0;
	__syncthreads();
	if (t0 == 0)
		for (int k = 1; k <= nt; ++k) part[k] += part[k - 1];
	__syncthreads();
	int o = part[t0];
	for (int w = a; w < b; ++w) {
		pre[w] = (unsigned short) min(o, 65535);
		for (unsigned m = bits[w]; m; m &= m - 1u) {
			if (o < haloCap) halo[(long) c * haloCap + o] = 32 * w + __ffs((int) m) - 1;
			++o;
		}
	}
	if (t0 == 0) haloNum[c] = part[nt];
	__syncthreads();
	for (int t = t0; t < R; t += nt) {
		const int i = perm[(long) c * R + t], sl = c * (R / 32) + t / 32, w = width[sl];
		const long base = off[sl] + (t & 31);
		const int z0 = i >= 0 ? rowPtr[i] : 0, len = i >= 0 ? rowPtr[i + 1] - z0 : 0;
		for (int k = 0; k < w; ++k) {
			int h = 0;
			if (k < len) {
				const int q = inv[col[z0 + k]];
				h = pre[q >> 5] + __popc(bits[q >> 5] & ((1u << (q & 31)) - 1u));
			}
			lcol[base + 32L * k] = (unsigned short) h;
		}
	}
}

size_t smem_limit(const void *kernel)
{
	static std::mutex mu;                    // sessions and servers may size launches from several threads
	static std::map<std::pair<int, const void *>, size_t> known;     // the limit belongs to a device's copy of the kernel
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess) {
		cudaGetLastError();
		return 0;
	}
	std::lock_guard<std::mutex> g(mu);
	const auto at = known.find({dev, kernel});
	if (at != known.end()) return at->second;
	int optin = 0;
	cudaFuncAttributes fa;
	size_t want = 0;
	if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
	    cudaFuncGetAttributes(&fa, kernel) == cudaSuccess && (size_t) optin > fa.sharedSizeBytes) {
		want = (size_t) optin - fa.sharedSizeBytes;
		if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) want) == cudaSuccess) {
			known[{dev, kernel}] = want;
			return want;
		}
	}
	cudaGetLastError();                      // not kept: the next call tries again
	return 0;
}

bool cgfix_plan(const Mesh &m, const double *x0soa, int smCount, int maxWarps, CgPlan &p,
                const std::function<void *(size_t)> &alloc, cudaStream_t s)
{
	p = CgPlan();
	const int B = m.dim, ns0 = (m.N + 31) / 32;
	const int cap = std::min(kFixMaxWarps, maxWarps) - 1;
	if (cap < 1 || smCount < 1) return false;
	p.pw = std::max(1, (ns0 + smCount - 1) / smCount);
	p.per = 1;
	p.nchunk = (ns0 + p.pw - 1) / p.pw;
	if (p.pw > cap) {                            // several chunks per CTA, and warps that stage the next chunk
		const int rows = cap - kFixStagers;
		if (rows < 1) return false;
		p.per = (ns0 + rows * smCount - 1) / (rows * smCount);
		p.nchunk = p.per * smCount;
		p.pw = (ns0 + p.nchunk - 1) / p.nchunk;
	}
	for (size_t q = 0; q + 1 < m.slOffHost.size(); ++q)
		p.widest = std::max(p.widest, (m.slOffHost[q + 1] - m.slOffHost[q]) / 32);
	// small chunks: several warps share a slice, two slots or more each (a slot costs one warp about 450 clocks of
	// latency, against 160 of issue; the digit sums are integers, so the split changes no bit)
	p.parts = p.per > 1 ? 1 : std::max(1, std::min({cap / p.pw, kFixMaxParts, (p.widest + 1) / 2}));
	p.warps = p.per > 1 ? cap + 1 : std::max(std::min(kFixMinWarps, maxWarps), p.pw * p.parts + 1);
	p.nslice = p.nchunk * p.pw;
	p.haloCap = std::min(kFixMaxHalo, p.nchunk * 32 * p.pw);
	const int R = 32 * p.pw, P = p.nchunk * R;
	if (P > kFixMaxRows || p.widest * B > kLimbMaxTerms) return false;
	auto get = [&](size_t bytes) { return alloc(std::max<size_t>(bytes, 16)); };
	double *scr = (double *) get(sizeof(double) * morton_order_doubles(B, m.N));
	p.perm = (int *) get(sizeof(int) * (size_t) P);
	p.inv = (int *) get(sizeof(int) * (size_t) m.N);
	p.width = (int *) get(sizeof(int) * (size_t) p.nslice);
	p.off = (int *) get(sizeof(int) * (size_t) (p.nslice + 1));
	p.halo = (int *) get(sizeof(int) * (size_t) p.nchunk * p.haloCap);
	p.haloNum = (int *) get(sizeof(int) * (size_t) p.nchunk);
	if (!scr || !p.perm || !p.inv || !p.width || !p.off || !p.halo || !p.haloNum) return false;
	const unsigned long long *keys = B == 2 ? morton_order<2>(m.N, x0soa, scr, s) : morton_order<3>(m.N, x0soa, scr, s);
	k_plan_rows<<<p.nchunk, 256, 2 * sizeof(int) * R, s>>>(m.N, p.nchunk, R, keys, m.rowPtr, p.perm, p.inv, p.width);
	k_plan_offsets<<<1, 1024, 0, s>>>(p.nslice, p.width, p.off);
	int total = 0;
	SA_CHECK(cudaMemcpyAsync(&total, p.off + p.nslice, sizeof(int), cudaMemcpyDeviceToHost, s));
	SA_CHECK(cudaStreamSynchronize(s));
	p.total = total;
	p.lcol = (unsigned short *) get(sizeof(unsigned short) * (size_t) total);
	p.fix = (int2 *) get(sizeof(int2) * (size_t) total * B * B);
	p.rowExp = (int *) get(sizeof(int) * (size_t) P);
	p.scale = (short *) get(sizeof(short) * (size_t) m.N);
	p.ug = (double *) get(sizeof(double) * (size_t) P * (B == 3 ? fix_u_stride<3>() : fix_u_stride<2>()));
	p.vec = (double *) get(sizeof(double) * (size_t) P * 4 * B);
	if (p.per > 1) p.pinv = (double *) get(sizeof(double) * (size_t) P * B * B);
	if (!p.lcol || !p.fix || !p.rowExp || !p.scale || !p.ug || !p.vec || (p.per > 1 && !p.pinv)) return false;
	const int nw = (P + 31) / 32;
	const size_t sm = sizeof(int) * (size_t) nw + sizeof(unsigned short) * (size_t) (nw + 1);
	if (sm > 48 * 1024 && sm > smem_limit((const void *) k_plan_columns)) return false;
	k_plan_columns<<<p.nchunk, 512, sm, s>>>(P, R, m.rowPtr, m.femVtx + m.Z, p.perm, p.inv, p.width, p.off, p.haloCap,
	                                         p.halo, p.haloNum, p.lcol);
	SA_CHECK(cudaGetLastError());
	std::vector<int> num(p.nchunk);
	SA_CHECK(cudaMemcpyAsync(num.data(), p.haloNum, sizeof(int) * p.nchunk, cudaMemcpyDeviceToHost, s));
	SA_CHECK(cudaStreamSynchronize(s));
	for (int c : num) p.haloMax = std::max(p.haloMax, c);
	p.ok = p.haloMax <= p.haloCap;
	return p.ok;
}

// ---------------------------------------------------------------------------
// Scales of a solve.  With D the block diagonal, the solve runs on D^-1/2 A D^-1/2, whose entries and whose u are alike in
// soft and stiff materials: node i has the scale 2^s, the root of the largest entry of its block inverse to a power of two,
// its u, p and x are over 2^s, its r, s and w times 2^s.  Powers of two, so the FP64 recurrences round as they would
// without; (w, u) and (r, u) do not change, a row's share of (r, r) is taken back by 2^-2s.  With A and u as they are, and one
// frame for a chunk's u, materials 1 : c : 1 on the icosphere-4 shell had errors of 5.1e-9 at c = 10^6 and 3.5e-6 at 10^8
// (2,888 iterations); scaled, and with the operator's longer digits, 6.1e-11 and 6.0e-9 (2,323), as FP64 kernels among
// themselves (9.6e-11, 6.1e-9, 2,345).
// ---------------------------------------------------------------------------
// v 2^s by the exponent field; zeros, subnormal numbers and results outside the normal range by scalbn
__device__ __noinline__ double scale_edge(double v, int s) { return scalbn(v, s); }
__device__ __forceinline__ double scale_pow2(double v, int s)
{
	const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff;
	if (e != 0 && e != 2047 && e + s > 0 && e + s < 2047) return __hiloint2double(hi + s * (1 << 20), __double2loint(v));
	return ((unsigned) hi << 1 | (unsigned) __double2loint(v)) == 0u ? v : scale_edge(v, s);
}

template <int B>
__global__ void k_cgfix_gather_copy(int P, const int *__restrict__ perm, const double *__restrict__ u,
                                    const double *__restrict__ binv, double *__restrict__ ug, short *__restrict__ scale)
{
	const int q = blockIdx.x * blockDim.x + threadIdx.x;
	if (q >= P) return;
	const int i = perm[q];
	int e = 0;
	if (i >= 0)
		for (int t = 0; t < B * B; ++t) e = max(e, fx_exp(__ldg(binv + (long) i * (B * B) + t)));
	const int s = i >= 0 && e < 2047 ? (e - 1023) >> 1 : 0;
	if (i >= 0) scale[i] = (short) s;
	for (int c = 0; c < fix_u_stride<B>(); ++c)
		ug[(long) q * fix_u_stride<B>() + c] = i >= 0 && c < B ? scale_pow2(u[(long) i * B + c], -s) : 0.0;
}

// ---------------------------------------------------------------------------
// operator: the permuted rows' scaled entries as digits, and the row frames.  One warp per slice.
// ---------------------------------------------------------------------------
template <int B>
__global__ void __launch_bounds__(128) k_cgfix_operator(int nslice, SellOp A, const int *__restrict__ rowPtr,
                                                        const double *__restrict__ blk, const int *__restrict__ perm,
                                                        const short *__restrict__ scale,
                                                        const int *__restrict__ width, const int *__restrict__ off,
                                                        int2 *__restrict__ fix, int *__restrict__ rowExp)
{
	const int sl = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
	if (sl >= nslice) return;
	const int i = perm[(long) sl * 32 + lane], w = width[sl];
	const int len = i >= 0 ? rowPtr[i + 1] - rowPtr[i] : 0;
	const long first = i >= 0 ? (long) __ldg(A.off + (i >> 5)) : 0l;
	const double *row = blk + (i >= 0 ? first * (B * B) + (i & 31) : 0l);
	const int *col = A.col + first + (i & 31);
	const int own = i >= 0 ? __ldg(scale + i) : 0;
	// the largest exponent, and the rows' sums of |a 2^s| 2^own (about 1 each) as FP32 numbers that are never too small
	int e = kLimbNone;
	float top = 0.0f, sum[B] = {};               // of the node's B rows, which share a frame
#pragma unroll 2
	for (int k = 0; k < len; ++k) {
		const int s = __ldg(scale + __ldg(col + 32 * k));
#pragma unroll
		for (int t = 0; t < B * B; ++t) {
			const double v = __ldg(row + ((long) k * B * B + t) * 32);
			e = max(e, limb_scaled_exp(v, s));
			const float f = limb_float_above(v, s + own);
			top = fmaxf(top, f);
			sum[t / B] += f;
		}
	}
	for (int r = 1; r < B; ++r) sum[0] = fmaxf(sum[0], sum[r]);
	if (e < kLimbBad) e -= limb_extra(top, sum[0], e + own);
	rowExp[(long) sl * 32 + lane] = row_pack(e < kLimbBad ? e + own : kLimbBad, own);
	int2 *o = fix + (long) off[sl] * (B * B) + lane;
	for (int k = 0; k < w; ++k) {
		const int s = k < len ? __ldg(scale + __ldg(col + 32 * k)) : 0;
		for (int t = 0; t < B * B; ++t) {
			int2 d = make_int2(0, 0);
			if (k < len && e < kLimbBad) limb_matrix_wide(__ldg(row + ((long) k * B * B + t) * 32), e - s, d.x, d.y);
			o[((long) k * B * B + t) * 32] = d;
		}
	}
}

// ---------------------------------------------------------------------------
// the solve
// ---------------------------------------------------------------------------
struct FixArgs {
	int pw, parts, haloCap, haloMax, colMax, stages;
	const int *perm, *width, *off, *halo, *haloNum, *rowExp;
	const unsigned short *lcol;
	const int2 *fix;
	const double *binv, *r0, *u0;
	double *x, *ug, *vec, *part, *pinv;
	CgScal *sc;
	GridSums *gs;
};

// shared memory of one CTA in bytes: operator ring, block inverses, u, ring barriers, the
// other parts' digit sums, halo digits and rows, slot places
template <int B> size_t fix_smem(int pw, int parts, int haloMax, int colMax, int stages)
{
	return (size_t) pw * stages * (256 * B * B + 8) + sizeof(double) * (size_t) pw * 32 * (B * B + B + (parts - 1) * 3 * B) +
	       sizeof(int) * (size_t) haloMax * (kLimbStride + 1) + sizeof(unsigned short) * (size_t) colMax + 16;
}

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned bar)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
	             :: "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// the same with an L2 policy
__device__ __forceinline__ void bulk_load_hint(void *dst, const void *src, unsigned bytes, unsigned bar, unsigned long long policy)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
	             :: "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(bar), "l"(policy) : "memory");
}

__device__ __forceinline__ void ring_load(void *dst, const void *src, unsigned bytes, unsigned bar)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
	bulk_load(dst, src, bytes, bar);
}

constexpr int kRingTries = 1 << 20;        // bounded wait: each try suspends up to a hardware time limit
__device__ __forceinline__ bool ring_wait(unsigned bar, unsigned parity)
{
	for (int n = 0; n < kRingTries; ++n) {
		unsigned ok;
		asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
		             : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
		if (ok) return true;
	}
	return false;
}

// acc += block a (shared memory, [entry][lane]) times the node's digits u
template <int B>
__device__ __forceinline__ void fix_slot_mac(LimbSum (&acc)[B], const int2 *__restrict__ a, const int *__restrict__ u)
{
#pragma unroll
	for (int c = 0; c < B; ++c) {
		const int2 ud = reinterpret_cast<const int2 *>(u)[c];
		const int u1 = ud.x, u0 = ud.y;
#pragma unroll
		for (int r = 0; r < B; ++r) {
			const int2 e = a[(r * B + c) * 32];
			limb_mac(acc[r], e.x, e.y, u1, u0);
		}
	}
}

// Operator slots kept in tensor memory (256 KB per SM, otherwise idle here): warp w of the CTA reaches the 32 lanes
// of its quarter w % 4, one lane per row, 2 B B columns per slot (digits of the block's entries, column by column).
constexpr int kTmemCols = 512;

// slots of one warp in tensor memory: the quarter's columns are shared by (pw + 3) / 4 row warps
template <int B> __host__ __device__ constexpr int tmem_slots(int pw) { return kTmemCols / (2 * B * B * ((pw + 3) / 4)); }

template <int B> __device__ __forceinline__ void tmem_store(unsigned t, const int2 (&e)[B * B])
{
	if constexpr (B == 3)
		asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
		             "tcgen05.st.sync.aligned.32x32b.x2.b32 [%17], {%18, %19};\n"
		             "tcgen05.wait::st.sync.aligned;"
		             :: "r"(t), "r"(e[0].x), "r"(e[0].y), "r"(e[1].x), "r"(e[1].y), "r"(e[2].x), "r"(e[2].y), "r"(e[3].x), "r"(e[3].y),
		                "r"(e[4].x), "r"(e[4].y), "r"(e[5].x), "r"(e[5].y), "r"(e[6].x), "r"(e[6].y), "r"(e[7].x), "r"(e[7].y),
		                "r"(t + 16), "r"(e[8].x), "r"(e[8].y) : "memory");
	else
		asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
		             "tcgen05.wait::st.sync.aligned;"
		             :: "r"(t), "r"(e[0].x), "r"(e[0].y), "r"(e[1].x), "r"(e[1].y), "r"(e[2].x), "r"(e[2].y), "r"(e[3].x), "r"(e[3].y)
		             : "memory");
}

template <int B> __device__ __forceinline__ void tmem_load(unsigned t, int2 (&e)[B * B])
{
	if constexpr (B == 3)
		asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%18];\n"
		             "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%16, %17}, [%19];\n"
		             "tcgen05.wait::ld.sync.aligned;"
		             : "=r"(e[0].x), "=r"(e[0].y), "=r"(e[1].x), "=r"(e[1].y), "=r"(e[2].x), "=r"(e[2].y), "=r"(e[3].x), "=r"(e[3].y),
		               "=r"(e[4].x), "=r"(e[4].y), "=r"(e[5].x), "=r"(e[5].y), "=r"(e[6].x), "=r"(e[6].y), "=r"(e[7].x), "=r"(e[7].y),
		               "=r"(e[8].x), "=r"(e[8].y) : "r"(t), "r"(t + 16));
	else
		asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
		             "tcgen05.wait::ld.sync.aligned;"
		             : "=r"(e[0].x), "=r"(e[0].y), "=r"(e[1].x), "=r"(e[1].y), "=r"(e[2].x), "=r"(e[2].y), "=r"(e[3].x), "=r"(e[3].y)
		             : "r"(t));
}

// acc += the block in e (tensor memory order: column by column) times the node's digits u
template <int B>
__device__ __forceinline__ void tmem_slot_mac(LimbSum (&acc)[B], const int2 (&e)[B * B], const int *__restrict__ u)
{
#pragma unroll
	for (int c = 0; c < B; ++c) {
		const int2 ud = reinterpret_cast<const int2 *>(u)[c];
		const int u1 = ud.x, u0 = ud.y;
#pragma unroll
		for (int r = 0; r < B; ++r) limb_mac(acc[r], e[c * B + r].x, e[c * B + r].y, u1, u0);
	}
}

// a halo node's u, written by other CTAs during the launch: one request, through L2
template <int B> __device__ __forceinline__ void load_halo(const double *p, double (&v)[B])
{
	if constexpr (B == 3) {
		double pad;
		asm volatile("ld.relaxed.gpu.global.v4.f64 {%0, %1, %2, %3}, [%4];"
		             : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(pad) : "l"(p) : "memory");
	} else {
		const double2 t = __ldcg(reinterpret_cast<const double2 *>(p));
		v[0] = t.x;
		v[1] = t.y;
	}
}

// the partial-sum path of a grid sum (no frame yet, or a value out of its frame); called by every thread of every CTA
template <int K>
__device__ __noinline__ bool slow_sum(double a, double b, double *res, double *part, int nctas, GridBar *bar,
                                      unsigned &target, FxScratch &fs)
{
	double v[K], t[K];
	v[0] = a;
	if (K > 1) v[K - 1] = b;
	if (!grid_reduce<K, double>(v, t, part, blockIdx.x, nctas, bar, target, fs)) return false;
	if (threadIdx.x == 0)
		for (int k = 0; k < K; ++k) res[k] = t[k];
	__syncthreads();
	return true;
}

// kStream: the ring does not hold every slot of a slice
template <int B, bool kStream>
__global__ void __launch_bounds__(32 * kFixMaxWarps, 1) k_cg_fix(const FixArgs a)
{
	__shared__ FxScratch fs;
	__shared__ unsigned dig[kFixMaxWarps][kSumWords];
	// the iteration's scalars, written by the reducer warp
	__shared__ double gam, rr, beta, dsub, alpha, delta, two[2];   // dsub = beta * gamma / alphaPrev
	__shared__ double goal;                      // squared residual to reach
	__shared__ int itrMax, stop, broke, iters, gaveUp, slow, sE[32];
	__shared__ unsigned tmemBase;
	extern __shared__ __align__(128) char sdyn[];
	CgScal *sc = a.sc;
	if (sc->done) return;                        // set by k_cg_init: the same for every CTA
	constexpr int S = kLimbStride, U = fix_u_stride<B>(), BB = B * B;
	constexpr unsigned kSlot = 256 * BB;         // bytes of one slot of a slice
	const int nctas = gridDim.x, lc = blockIdx.x, pw = a.pw;
	const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, W = blockDim.x >> 5;
	// warps 0 .. pw - 1 own one slice each; the next pw (parts - 1) warps share their slots; then warps that only stage
	const bool reducer = wp == W - 1, rowWarp = wp < pw, worker = wp < pw * a.parts;
	const int ws = kStream ? wp : wp % pw, part = kStream ? 0 : wp / pw;
	// shared memory: offsets from sdyn
	const int oInv = pw * a.stages * (int) kSlot, oU = oInv + pw * 256 * BB, oBar = oU + pw * 256 * B;
	const int oPart = oBar + 8 * pw * a.stages, oLimb = oPart + (a.parts - 1) * pw * 768 * B, oHalo = oLimb + 4 * a.haloMax * S, oCol = oHalo + 4 * a.haloMax;
	int *slimb = (int *) (sdyn + oLimb), *shalo = (int *) (sdyn + oHalo);
	unsigned short *scol = (unsigned short *) (sdyn + oCol);
	double *su = (double *) (sdyn + oU) + wp * B * 32 + lane;            // row warps only
	char *ring = sdyn + ws * a.stages * (int) kSlot;
	const unsigned mb = smem_addr(sdyn + oBar + 8 * ws * a.stages);
	const int sl = lc * pw + ws, row = sl * 32 + lane;        // permuted row (workers)
	const int i = rowWarp ? __ldg(a.perm + row) : -1;
	const bool own = i >= 0;
	const int wdt = worker ? __ldg(a.width + sl) : 0;
	const int o0 = __ldg(a.off + lc * pw);
	const int o1 = worker ? __ldg(a.off + sl) : o0;
	const char *src = (const char *) a.fix + (size_t) o1 * (8 * BB);
	const unsigned short *mycol = scol + (o1 - o0) + lane;
	const int rowWord = rowWarp ? __ldg(a.rowExp + row) : 0, scl = row_scale(rowWord);
	const int nhalo = __ldg(a.haloNum + lc);
	for (int t = threadIdx.x, n = __ldg(a.off + (lc + 1) * pw) - o0; t < n; t += blockDim.x) scol[t] = __ldg(a.lcol + o0 + t);
	for (int t = threadIdx.x; t < nhalo; t += blockDim.x) shalo[t] = __ldg(a.halo + (long) lc * a.haloCap + t);
	if (threadIdx.x == 0) {
		gam = sc->gam; rr = sc->rr; beta = 0.0; dsub = 0.0; alpha = 1.0; delta = 0.0;
		goal = sc->tolSqu * sc->bb; itrMax = sc->itrMax;
		stop = -1; broke = -1; iters = 0; gaveUp = 0; slow = 0;
	}
	// operator: the warp's last ntm slots in tensor memory (kStream), the others through its ring (all of them at
	// once when they fit: then nothing is loaded again)
	unsigned tmem = 0u;
	int ntm = 0;
	if constexpr (kStream) {
		if (wp == 0) {
			asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(&tmemBase)), "r"(kTmemCols) : "memory");
			asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
		}
		__syncthreads();
		tmem = tmemBase + ((unsigned) (wp & 3) << 21) + (unsigned) ((wp >> 2) * tmem_slots<B>(pw) * 2 * BB);
		ntm = min(tmem_slots<B>(pw), wdt);
		for (int k = 0; k < ntm; ++k) {
			const int2 *g = (const int2 *) (src + (size_t) (wdt - ntm + k) * kSlot) + lane;
			int2 e[BB];
#pragma unroll
			for (int c = 0; c < B; ++c)
#pragma unroll
				for (int r = 0; r < B; ++r) e[c * B + r] = __ldg(g + (r * B + c) * 32);
			tmem_store<B>(tmem + 2 * BB * k, e);
		}
	}
	const int nring = wdt - ntm, nstage = min(a.stages, nring);
	const bool stream = kStream && nstage < nring;
	const int step = kStream ? 1 : a.parts;      // a part's slots: part, part + step, ...
	if (worker && lane == 0) {
		for (int k = part; k < nstage; k += step) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(mb + 8 * k) : "memory");
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
		for (int k = part; k < nstage; k += step) ring_load(ring + k * kSlot, src + (size_t) k * kSlot, kSlot, mb + 8 * k);
	}
	int stage = 0, next = nstage;                // ring place of the next slot used, and the next slot to load
	unsigned parity = 0;
	// x, p, s and r are used only while the reducer waits for the grid: they stay in global memory (L2), which leaves
	// the registers to the digit sums; u and the block inverses in shared memory
	const int vs = nctas * pw * 32 * B, vrow = sl * 32 * B + lane;
	if (rowWarp) {
		double *g = a.vec + vrow;
#pragma unroll
		for (int c = 0; c < B; ++c) {
			const long k = (long) i * B + c;
			g[32 * c] = own ? scale_pow2(a.x[k], -scl) : 0.0;
			g[vs + 32 * c] = g[2 * vs + 32 * c] = 0.0;
			g[3 * vs + 32 * c] = own ? scale_pow2(a.r0[k], scl) : 0.0;
			su[32 * c] = own ? scale_pow2(a.u0[k], -scl) : 0.0;
		}
		double *sbinv = (double *) (sdyn + oInv) + wp * BB * 32 + lane;
		for (int t = 0; t < BB; ++t) sbinv[32 * t] = own ? scale_pow2(__ldg(a.binv + (long) i * BB + t), -2 * scl) : 0.0;
	}
	const int nst = 32 * (W - 1), nSt = reducer ? 0 : nhalo;    // the reducer warp stages nothing
	unsigned target = 0;                         // arrivals of the partial-sum path
	bool pending = false, first = true;
	int line = 0;                                // sum line of the iteration
	__syncthreads();
	if (!stream)
		for (int k = part; k < nstage; k += step)
			if (!ring_wait(mb + 8 * k, 0u)) gaveUp = 1;
	for (;;) {
		// (0) the halo of u as digits in shared memory
		// (raw first, in place, for the largest exponent)
		int e = 1;
#pragma unroll 4
		for (int h = threadIdx.x; h < nSt; h += nst) {
			double v[B];
			load_halo<B>(a.ug + (long) shalo[h] * U, v);
			double *d = reinterpret_cast<double *>(slimb + h * S);
#pragma unroll
			for (int c = 0; c < B; ++c) { d[c] = v[c]; e = max(e, fx_exp(v[c])); }
		}
		e = fx_warp_max(e);
		if (lane == 0) sE[wp] = e;
		__syncthreads();
		const int eU = fx_warp_max(lane < W ? sE[lane] : 1);
#pragma unroll 1
		for (int h = threadIdx.x; h < nSt; h += nst) {
			double *d = reinterpret_cast<double *>(slimb + h * S);
#pragma unroll
			for (int c = 0; c < B; ++c) {
				int2 t;
				limb_vector(d[c], eU, t.x, t.y);
				reinterpret_cast<int2 *>(d)[c] = t;
			}
		}
		__syncthreads();
		// (1) rows: w = A u and (w, u).  Reducer: beta, beta * gamma / alpha and the stopping test of the last update
		double wv[B], rv[B];
		double d1 = 0.0;
#pragma unroll
		for (int c = 0; c < B; ++c) wv[c] = 0.0;
		LimbSum acc[B];
		if (worker) {
#pragma unroll
			for (int c = 0; c < B; ++c) acc[c] = limb_zero();
			if constexpr (kStream) {
				// tensor-memory slots spread between the streamed ones, which evens out the loads
				int kt = 0;
				for (int k = 0; k < nring; ++k) {
					const int *u = slimb + mycol[k << 5] * S;
					if (stream && !ring_wait(mb + 8 * stage, parity)) gaveUp = 1;
					fix_slot_mac<B>(acc, reinterpret_cast<const int2 *>(ring + stage * (int) kSlot) + lane, u);
					if (stream) {
						__syncwarp();            // every lane has read the slot before it is overwritten
						if (lane == 0) ring_load(ring + stage * (int) kSlot, src + next * (int) kSlot, kSlot, mb + 8 * stage);
						if (++next == nring) next = 0;
					}
					if (++stage == nstage) { stage = 0; parity ^= 1u; }
					if (kt < ntm && (kt + 1) * nring <= (k + 1) * ntm) {
						int2 e[BB];
						tmem_load<B>(tmem + 2 * BB * kt, e);
						tmem_slot_mac<B>(acc, e, slimb + mycol[(nring + kt) << 5] * S);
						++kt;
					}
				}
				for (; kt < ntm; ++kt) {
					int2 e[BB];
					tmem_load<B>(tmem + 2 * BB * kt, e);
					tmem_slot_mac<B>(acc, e, slimb + mycol[(nring + kt) << 5] * S);
				}
			} else {
				int k = part;
				for (; k + step < wdt; k += 2 * step) {
					const int *u = slimb + mycol[k << 5] * S, *u2 = slimb + mycol[(k + step) << 5] * S;
					fix_slot_mac<B>(acc, reinterpret_cast<const int2 *>(ring + k * (int) kSlot) + lane, u);
					fix_slot_mac<B>(acc, reinterpret_cast<const int2 *>(ring + (k + step) * (int) kSlot) + lane, u2);
				}
				if (k < wdt)
					fix_slot_mac<B>(acc, reinterpret_cast<const int2 *>(ring + k * (int) kSlot) + lane, slimb + mycol[k << 5] * S);
				if (part > 0) {
					long long *o = (long long *) (sdyn + oPart) + ((part - 1) * pw + ws) * 96 * B + lane;
#pragma unroll
					for (int c = 0; c < B; ++c) {
						o[(3 * c) * 32] = acc[c].s2;
						o[(3 * c + 1) * 32] = acc[c].sm;
						o[(3 * c + 2) * 32] = acc[c].s0;
					}
				}
			}
		}
		if (reducer && pending) {
			// lanes 0 and 1 share one division: g / gamma and g / alpha
			const double g = two[0], q = two[1];
			const double ratio = g / (lane == 1 ? alpha : gam);
			const double ga = __shfl_sync(0xffffffffu, ratio, 1);
			if (lane == 0) {
				beta = ratio;
				dsub = ratio * ga;
				gam = g;
				rr = q;
				const int n = ++iters;
				if (fx_exp(g) >= 2047 || fx_exp(q) >= 2047) stop = SA_ERR_NONFINITE;
				else if (q < goal) stop = SA_OK;
				else if (n >= itrMax) stop = SA_ERR_NOT_CONVERGED;
			}
		}
		if (!kStream && a.parts > 1 && worker)            // the other parts' digit sums (the reducer is not waited for)
			asm volatile("bar.sync 1, %0;" :: "r"(32 * pw * a.parts) : "memory");
		if (rowWarp) {
			for (int q = 1; !kStream && q < a.parts; ++q) {
				const long long *o = (const long long *) (sdyn + oPart) + ((q - 1) * pw + ws) * 96 * B + lane;
#pragma unroll
				for (int c = 0; c < B; ++c) {
					acc[c].s2 += o[(3 * c) * 32];
					acc[c].sm += o[(3 * c + 1) * 32];
					acc[c].s0 += o[(3 * c + 2) * 32];
				}
			}
			if (own) {
#pragma unroll
				for (int c = 0; c < B; ++c) wv[c] = limb_scaled_to_double(acc[c], row_frame(rowWord), eU);
				d1 = wv[0] * su[0];
				for (int c = 1; c < B; ++c) d1 += wv[c] * su[32 * c];
			}
		}
		const int fD[1] = {sum_frame(delta)};
		{
			const double t[1] = {d1};
			if (!first) warp_digits<1>(t, fD, dig[wp]);
		}
		__syncthreads();                         // digits and scalars
		if (stop >= 0) break;
		// (2) reducer: the grid's (w, u) and alpha.  Rows meanwhile: p and s
		if (reducer && !first) {
			double t[1];
			bool flag = false;
			const bool ok = sum_exchange<1>(dig[0], W, &a.gs->delta[line], nctas, fD, &a.gs->bar, t, flag);
			if (lc == 0 && lane < kSumWords) a.gs->delta[line >= 1 ? line - 1 : 2].w[lane] = 0ull;
			if (lane == 0) {
				if (!ok) gaveUp = 1;
				slow = flag ? 1 : 0;
				if (!flag) {
					delta = t[0];
					alpha = gam / (t[0] - dsub);
					// bits, not FP64 compares (64 clocks each): alpha positive and finite, beta finite
					if (__double_as_longlong(alpha) <= 0 || fx_exp(alpha) >= 2047 || fx_exp(beta) >= 2047)
						broke = fx_exp(t[0]) < 2047 ? SA_ERR_BREAKDOWN : SA_ERR_NONFINITE;
				}
			}
		} else if (own) {
			const double be = beta;
			double *g = a.vec + vs + vrow;
#pragma unroll
			for (int c = 0; c < B; ++c) {
				g[32 * c] = su[32 * c] + be * g[32 * c];
				wv[c] = wv[c] + be * g[vs + 32 * c];     // s
				g[vs + 32 * c] = wv[c];
				rv[c] = g[2 * vs + 32 * c];
			}
		}
		__syncthreads();
		if (first || slow) {
			if (!gaveUp && !slow_sum<1>(d1, 0.0, two, a.part, nctas, &a.gs->bar, target, fs)) {
				if (threadIdx.x == 0) gaveUp = 1;
			} else if (threadIdx.x == 0 && !gaveUp) {
				delta = two[0];
				alpha = gam / (delta - dsub);
				if (!(alpha > 0.0) || !isfinite(alpha) || !isfinite(beta))
					broke = isfinite(delta) ? SA_ERR_BREAKDOWN : SA_ERR_NONFINITE;
			}
			__syncthreads();
		}
		if (gaveUp || broke >= 0) break;
		const double al = alpha;
		// (3) rows: r, u and (r, u), (r, r); the reducer adds them over the grid, which also completes u
		double d2[2] = {0.0, 0.0};
		if (own) {
#pragma unroll
			for (int c = 0; c < B; ++c) rv[c] = rv[c] - al * wv[c];
			const double *sbinv = (const double *) (sdyn + oInv) + wp * BB * 32 + lane;
			double uv[B];
#pragma unroll
			for (int r = 0; r < B; ++r) {
				double t = sbinv[32 * (r * B)] * rv[0];
#pragma unroll
				for (int c = 1; c < B; ++c) t += sbinv[32 * (r * B + c)] * rv[c];
				uv[r] = t;
				su[32 * r] = t;
			}
			double2 *o = reinterpret_cast<double2 *>(a.ug + (long) row * U);
			o[0] = make_double2(uv[0], uv[1]);
			if constexpr (B == 3) o[1] = make_double2(uv[2], 0.0);
			d2[0] = rv[0] * uv[0];
			d2[1] = rv[0] * rv[0];
			for (int c = 1; c < B; ++c) { d2[0] += rv[c] * uv[c]; d2[1] += rv[c] * rv[c]; }
		}
		const int fG[2] = {sum_frame(gam), sum_frame(rr)};
		const int fRow[2] = {fG[0], fG[1] + 2 * scl};    // r times 2^s
		warp_digits<2>(d2, fRow, dig[wp]);
		__syncthreads();
		if (reducer) {
			double t[2];
			bool flag = false;
			__threadfence();                     // the CTA's u before its count
			const bool ok = sum_exchange<2>(dig[0], W, &a.gs->gamma[line], nctas, fG, &a.gs->bar, t, flag);
			if (lc == 0 && lane < kSumWords) a.gs->gamma[line >= 1 ? line - 1 : 2].w[lane] = 0ull;
			if (lane == 0) {
				if (!ok) gaveUp = 1;
				slow = flag ? 1 : 0;
				two[0] = t[0];
				two[1] = t[1];
			}
		} else if (own) {
#pragma unroll
			for (int c = 0; c < B; ++c) {                // while the reducer waits
				double *g = a.vec + vrow + 32 * c;
				g[0] = g[0] + al * g[vs];
				g[3 * vs] = rv[c];
			}
		}
		__syncthreads();
		if (gaveUp) break;
		if (slow) {
			if (!slow_sum<2>(d2[0], scalbn(d2[1], -2 * scl), two, a.part + nctas, nctas, &a.gs->bar, target, fs)) {
				if (threadIdx.x == 0) gaveUp = 1;
				__syncthreads();
				break;
			}
		}
		if (++line == 3) line = 0;
		pending = true;
		first = false;
	}
	if (own)
#pragma unroll
		for (int c = 0; c < B; ++c) a.x[(long) i * B + c] = scale_pow2(a.vec[vrow + 32 * c], scl);
	if (stream)                                  // the ring's copies in flight land before the CTA leaves
		for (int k = 0; k < nstage; ++k) {
			ring_wait(mb + 8 * stage, parity);
			if (++stage == nstage) { stage = 0; parity ^= 1u; }
		}
	__syncthreads();
	if constexpr (kStream)
		if (wp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmemBase), "r"(kTmemCols));
	if (lc == 0 && threadIdx.x == 0) {
		sc->iters = iters; sc->code = gaveUp ? SA_ERR_TIMEOUT : max(stop, broke); sc->rr = rr; sc->gam = gam; sc->done = 1;
	}
}

// ---------------------------------------------------------------------------
// The same solve for operators of more than one chunk per CTA (more than 92 416 rows).  The CTA takes its per chunks in
// turn: the row warps multiply one while the staging warps gather and convert the next one's halo.  The warp's operator
// ring, whose slots carry their columns, runs on from chunk to chunk; the last slots of the first chunk's slices stay in
// tensor memory.  x, p, s and r of the rows and their block inverses are in global memory, 32 rows of a component together
// (72 bytes a row in the natural order cost 9 x 32 cache tags per slice, 10k clocks of an iteration).
//
// What bounds it: the operator's bytes.  At 204 810 nodes (3 chunks of 15 slices, 215 MB of entries and columns, 182 of
// them through the ring) 70 of an iteration's 113 thousand clocks are the products, 5.3 TB/s; the rest is the rows' FP64
// (16k), the two grid sums (15k) and the first halo (6k).  A solve of it: 81 us per iteration in the FP64 kernel, 85 with
// each chunk staged by the warps that multiply it, 60 with staging warps and columns in the ring, 55 with the ring's loads
// marked evict-first (a kept first chunk, or two, gave nothing more).
// ---------------------------------------------------------------------------
template <int B>
__global__ void k_cgfix_inverses(int P, const int *__restrict__ perm, const short *__restrict__ scale,
                                 const double *__restrict__ binv, double *__restrict__ out)
{
	const int q = blockIdx.x * blockDim.x + threadIdx.x;
	if (q >= P) return;
	const int i = perm[q];
	for (int t = 0; t < B * B; ++t)
		out[(long) (q >> 5) * (32 * B * B) + 32 * t + (q & 31)] = i >= 0 ? scale_pow2(binv[(long) i * (B * B) + t], -2 * scale[i]) : 0.0;
}

// bytes of a ring slot: entries and columns
template <int B> __host__ __device__ constexpr int many_slot() { return 256 * B * B + 64; }

// shared memory: operator ring and its barriers, two chunks' halo digits, the first chunk's halo rows, columns of the
// slots in tensor memory
template <int B> size_t fix_many_smem(int pw, int haloMax, int stages)
{
	return (size_t) pw * stages * (many_slot<B>() + 8) + sizeof(int) * (size_t) haloMax * (2 * kLimbStride + 1) +
	       (size_t) pw * tmem_slots<B>(pw) * 64 + 16;
}

template <int B>
__global__ void __launch_bounds__(32 * kFixMaxWarps, 1) k_cg_fix_many(const FixArgs a, int per)
{
	__shared__ FxScratch fs;
	__shared__ unsigned dig[kFixMaxWarps][kSumWords];
	__shared__ double gam, rr, beta, dsub, alpha, delta, two[2], goal;
	__shared__ int itrMax, stop, broke, iters, gaveUp, slow, sE[32], sFrame[2];
	__shared__ unsigned tmemBase;
	extern __shared__ __align__(128) char sdyn[];
	CgScal *sc = a.sc;
	if (sc->done) return;
	constexpr int S = kLimbStride, U = fix_u_stride<B>(), BB = B * B;
	constexpr int kSlot = 256 * BB, kRing = many_slot<B>();
	const int nctas = gridDim.x, lc = blockIdx.x, pw = a.pw;
	const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, W = blockDim.x >> 5;
	const bool reducer = wp == W - 1, rowWarp = wp < pw;
	const int oBar = pw * a.stages * kRing, oLimb = oBar + 8 * pw * a.stages, oHalo = oLimb + 8 * a.haloMax * S;
	const int tslots = tmem_slots<B>(pw), oCol = (oHalo + 4 * a.haloMax + 15) & ~15;
	int *slimb = (int *) (sdyn + oLimb), *shalo = (int *) (sdyn + oHalo);
	unsigned short *tcol = (unsigned short *) (sdyn + oCol) + wp * tslots * 32 + lane;
	char *ring = sdyn + wp * a.stages * kRing;
	const unsigned mb = smem_addr(sdyn + oBar + 8 * wp * a.stages);
	const int sl0 = lc * per * pw + wp;          // the warp's slice of chunk j: sl0 + j pw
	const long vs = (long) nctas * per * pw * 32 * B;
	for (int t = threadIdx.x, n = __ldg(a.haloNum + lc * per); t < n; t += blockDim.x)
		shalo[t] = __ldg(a.halo + (long) lc * per * a.haloCap + t);
	if (threadIdx.x == 0) {
		gam = sc->gam; rr = sc->rr; beta = 0.0; dsub = 0.0; alpha = 1.0; delta = 0.0;
		goal = sc->tolSqu * sc->bb; itrMax = sc->itrMax;
		stop = -1; broke = -1; iters = 0; gaveUp = 0; slow = 0;
	}
	if (wp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(&tmemBase)), "r"(kTmemCols) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
	}
	__syncthreads();
	const unsigned tmem = tmemBase + ((unsigned) (wp & 3) << 21) + (unsigned) ((wp >> 2) * tslots * 2 * BB);
	auto slice_width = [&](int j) { return __ldg(a.width + sl0 + j * pw); };
	// slots of chunk j that go through the ring; the others of chunk 0 stay in tensor memory
	const int ntm = rowWarp ? min(tslots, slice_width(0)) : 0;
	auto ring_slots = [&](int j) { return slice_width(j) - (j == 0 ? ntm : 0); };
	if (ntm > 0) {
		const int w0 = ring_slots(0), o = __ldg(a.off + sl0);
		for (int k = 0; k < ntm; ++k) {
			const int2 *g = (const int2 *) ((const char *) a.fix + (size_t) o * (8 * BB) + (size_t) (w0 + k) * kSlot) + lane;
			int2 e[BB];
#pragma unroll
			for (int c = 0; c < B; ++c)
#pragma unroll
				for (int r = 0; r < B; ++r) e[c * B + r] = __ldg(g + (r * B + c) * 32);
			tmem_store<B>(tmem + 2 * BB * k, e);
			tcol[32 * k] = __ldg(a.lcol + o + (w0 + k) * 32 + lane);
		}
	}
	int total = 0;                               // slots through the ring per matvec
	if (rowWarp)
		for (int j = 0; j < per; ++j) total += ring_slots(j);
	const int nstage = min(a.stages, total);
	unsigned long long policy;                   // the operator passes through L2, which keeps u and the rows' vectors
	asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
	int nj = 0, nleft = 0;                       // chunk of the next load, and its slots not asked for yet
	const char *nsrc = nullptr;                  // their entries and columns
	const unsigned short *ncol = nullptr;
	auto open_chunk = [&]() {
		nleft = ring_slots(nj);
		const int o = __ldg(a.off + sl0 + nj * pw);
		nsrc = (const char *) a.fix + (size_t) o * (8 * BB);
		ncol = a.lcol + o;
	};
	auto load_next = [&](int st) {               // every lane keeps the place, lane 0 issues
		while (nleft == 0) { if (++nj == per) nj = 0; open_chunk(); }
		if (lane == 0) {
			const unsigned bar = mb + 8 * st;
			asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"((unsigned) kRing) : "memory");
			bulk_load_hint(ring + st * kRing, nsrc, kSlot, bar, policy);
			bulk_load_hint(ring + st * kRing + kSlot, ncol, 64, bar, policy);
		}
		nsrc += kSlot;
		ncol += 32;
		--nleft;
	};
	if (rowWarp) {
		if (lane == 0) {
			for (int k = 0; k < nstage; ++k) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(mb + 8 * k) : "memory");
			asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
			asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
		}
		__syncwarp();
		open_chunk();
		for (int k = 0; k < nstage; ++k) load_next(k);
		for (int j = 0; j < per; ++j) {
			const int row = (sl0 + j * pw) * 32 + lane, i = __ldg(a.perm + row), scl = row_scale(__ldg(a.rowExp + row));
			double *g = a.vec + (long) (sl0 + j * pw) * 32 * B + lane;
#pragma unroll
			for (int c = 0; c < B; ++c) {
				const long k = (long) i * B + c;
				g[32 * c] = i >= 0 ? scale_pow2(a.x[k], -scl) : 0.0;
				g[vs + 32 * c] = g[2 * vs + 32 * c] = 0.0;
				g[3 * vs + 32 * c] = i >= 0 ? scale_pow2(a.r0[k], scl) : 0.0;
			}
		}
	}
	// stage(): halo values of a chunk into its buffer and the largest exponent; convert(): to digits in the frame e
	auto stage_halo = [&](const int *rows, int nh, int *buf, int t0, int nt) {
		int e = 1;
#pragma unroll 4
		for (int h = t0; h < nh; h += nt) {
			double v[B];
			load_halo<B>(a.ug + (long) rows[h] * U, v);
			double *d = reinterpret_cast<double *>(buf + h * S);
#pragma unroll
			for (int c = 0; c < B; ++c) { d[c] = v[c]; e = max(e, fx_exp(v[c])); }
		}
		e = fx_warp_max(e);
		if (lane == 0) sE[wp] = e;
	};
	auto convert_halo = [&](int nh, int *buf, int e, int t0, int nt) {
#pragma unroll 1
		for (int h = t0; h < nh; h += nt) {
			double *d = reinterpret_cast<double *>(buf + h * S);
#pragma unroll
			for (int c = 0; c < B; ++c) {
				int2 t;
				limb_vector(d[c], e, t.x, t.y);
				reinterpret_cast<int2 *>(d)[c] = t;
			}
		}
	};
	const int nstagers = W - 1 - pw;             // warps pw .. W - 2
	int stage = 0;
	unsigned parity = 0;
	unsigned target = 0;
	bool pending = false, first = true;
	int line = 0;
	__syncthreads();
	for (;;) {
		// (0) the first chunk's halo, by every warp but the reducer, which has the iteration's scalars to finish
		const int nh0 = __ldg(a.haloNum + lc * per);
		if (!reducer) stage_halo(shalo, nh0, slimb, threadIdx.x, 32 * (W - 1));
		else if (pending) {
			// lanes 0 and 1 share one division: g / gamma and g / alpha
			const double g = two[0], q = two[1];
			const double ratio = g / (lane == 1 ? alpha : gam);
			const double ga = __shfl_sync(0xffffffffu, ratio, 1);
			if (lane == 0) {
				beta = ratio;
				dsub = ratio * ga;
				gam = g;
				rr = q;
				const int n = ++iters;
				if (fx_exp(g) >= 2047 || fx_exp(q) >= 2047) stop = SA_ERR_NONFINITE;
				else if (q < goal) stop = SA_OK;
				else if (n >= itrMax) stop = SA_ERR_NOT_CONVERGED;
			}
		}
		__syncthreads();
		if (stop >= 0) break;
		{
			const int e = fx_warp_max(lane < W - 1 ? sE[lane] : 1);
			if (threadIdx.x == 0) sFrame[0] = e;
			if (!reducer) convert_halo(nh0, slimb, e, threadIdx.x, 32 * (W - 1));
		}
		__syncthreads();
		// (1) chunk by chunk: w = A u, (w, u), p and s
		double d1 = 0.0;
		for (int j = 0; j < per; ++j) {
			if (rowWarp) {
				const int sl = sl0 + j * pw, row = sl * 32 + lane, nr = ring_slots(j), nt = j == 0 ? ntm : 0;
				const int *uh = slimb + (j & 1) * a.haloMax * S;
				const bool own = __ldg(a.perm + row) >= 0;
				const int rowWord = __ldg(a.rowExp + row);
				double *g = a.vec + vs + (long) sl * 32 * B + lane;
				double uv[B], pv[B], sv[B];
				load_halo<B>(a.ug + (long) row * U, uv);
#pragma unroll
				for (int c = 0; c < B; ++c) { pv[c] = g[32 * c]; sv[c] = g[vs + 32 * c]; }
				LimbSum acc[B];
#pragma unroll
				for (int c = 0; c < B; ++c) acc[c] = limb_zero();
				int kt = 0;
				for (int k = 0; k < nr; ++k) {
					if (!ring_wait(mb + 8 * stage, parity)) gaveUp = 1;
					const char *slot = ring + stage * kRing;
					const int *u = uh + reinterpret_cast<const unsigned short *>(slot + kSlot)[lane] * S;
					fix_slot_mac<B>(acc, reinterpret_cast<const int2 *>(slot) + lane, u);
					__syncwarp();                // every lane has read the slot before it is overwritten
					load_next(stage);
					if (++stage == nstage) { stage = 0; parity ^= 1u; }
					if (kt < nt && (kt + 1) * nr <= (k + 1) * nt) {
						int2 t[BB];
						tmem_load<B>(tmem + 2 * BB * kt, t);
						tmem_slot_mac<B>(acc, t, uh + tcol[kt << 5] * S);
						++kt;
					}
				}
				for (; kt < nt; ++kt) {
					int2 t[BB];
					tmem_load<B>(tmem + 2 * BB * kt, t);
					tmem_slot_mac<B>(acc, t, uh + tcol[kt << 5] * S);
				}
				if (own) {
					const int eU = sFrame[j & 1];
					const double be = beta;
#pragma unroll
					for (int c = 0; c < B; ++c) {
						const double w = limb_scaled_to_double(acc[c], row_frame(rowWord), eU);
						d1 += w * uv[c];
						g[32 * c] = uv[c] + be * pv[c];
						g[vs + 32 * c] = w + be * sv[c];
					}
				}
			} else if (!reducer && j + 1 < per) {
				const int ch = lc * per + j + 1, nh = __ldg(a.haloNum + ch), t0 = threadIdx.x - 32 * pw;
				int *buf = slimb + ((j + 1) & 1) * a.haloMax * S;
				stage_halo(a.halo + (long) ch * a.haloCap, nh, buf, t0, 32 * nstagers);
				asm volatile("bar.sync 1, %0;" :: "r"(32 * nstagers) : "memory");
				const int e = fx_warp_max(lane < nstagers ? sE[pw + lane] : 1);
				if (t0 == 0) sFrame[(j + 1) & 1] = e;
				convert_halo(nh, buf, e, t0, 32 * nstagers);
			}
			if (j + 1 < per) __syncthreads();    // the next chunk's digits are there, this one's have been read
		}
		const int fD[1] = {sum_frame(delta)};
		{
			const double t[1] = {d1};
			if (!first) warp_digits<1>(t, fD, dig[wp]);
		}
		__syncthreads();
		// (2) reducer: the grid's (w, u) and alpha
		if (reducer && !first) {
			double t[1];
			bool flag = false;
			const bool ok = sum_exchange<1>(dig[0], W, &a.gs->delta[line], nctas, fD, &a.gs->bar, t, flag);
			if (lc == 0 && lane < kSumWords) a.gs->delta[line >= 1 ? line - 1 : 2].w[lane] = 0ull;
			if (lane == 0) {
				if (!ok) gaveUp = 1;
				slow = flag ? 1 : 0;
				if (!flag) {
					delta = t[0];
					alpha = gam / (t[0] - dsub);
					// bits, not FP64 compares (64 clocks each): alpha positive and finite, beta finite
					if (__double_as_longlong(alpha) <= 0 || fx_exp(alpha) >= 2047 || fx_exp(beta) >= 2047)
						broke = fx_exp(t[0]) < 2047 ? SA_ERR_BREAKDOWN : SA_ERR_NONFINITE;
				}
			}
		}
		__syncthreads();
		if (first || slow) {
			if (!gaveUp && !slow_sum<1>(d1, 0.0, two, a.part, nctas, &a.gs->bar, target, fs)) {
				if (threadIdx.x == 0) gaveUp = 1;
			} else if (threadIdx.x == 0 && !gaveUp) {
				delta = two[0];
				alpha = gam / (delta - dsub);
				if (!(alpha > 0.0) || !isfinite(alpha) || !isfinite(beta))
					broke = isfinite(delta) ? SA_ERR_BREAKDOWN : SA_ERR_NONFINITE;
			}
			__syncthreads();
		}
		if (gaveUp || broke >= 0) break;
		const double al = alpha;
		// (3) rows: r, u and (r, u), (r, r); the reducer adds them over the grid, which also completes u
		double d2[2] = {0.0, 0.0};
		if (rowWarp)
#pragma unroll 1
			for (int j = 0; j < per; ++j) {
				const int sl = sl0 + j * pw;
				double *g = a.vec + 2 * vs + (long) sl * 32 * B + lane;
				const double *mi = a.pinv + (long) sl * 32 * BB + lane;
				double rv[B], sv[B], uv[B], m[BB];
				const double back = __hiloint2double((1023 - 2 * row_scale(__ldg(a.rowExp + sl * 32 + lane))) << 20, 0);   // 2^-2s
#pragma unroll
				for (int c = 0; c < B; ++c) { rv[c] = g[vs + 32 * c]; sv[c] = g[32 * c]; }
#pragma unroll
				for (int t = 0; t < BB; ++t) m[t] = __ldg(mi + 32 * t);
#pragma unroll
				for (int c = 0; c < B; ++c) { rv[c] = rv[c] - al * sv[c]; g[vs + 32 * c] = rv[c]; }
#pragma unroll
				for (int r = 0; r < B; ++r) {
					double t = m[r * B] * rv[0];
#pragma unroll
					for (int c = 1; c < B; ++c) t += m[r * B + c] * rv[c];
					uv[r] = t;
				}
				double2 *o = reinterpret_cast<double2 *>(a.ug + (long) (sl * 32 + lane) * U);
				o[0] = make_double2(uv[0], uv[1]);
				if constexpr (B == 3) o[1] = make_double2(uv[2], 0.0);
				double q = rv[0] * rv[0];
				d2[0] += rv[0] * uv[0];
#pragma unroll
				for (int c = 1; c < B; ++c) { d2[0] += rv[c] * uv[c]; q += rv[c] * rv[c]; }
				d2[1] = fma(q, back, d2[1]);
			}
		const int fG[2] = {sum_frame(gam), sum_frame(rr)};
		warp_digits<2>(d2, fG, dig[wp]);
		__syncthreads();
		if (reducer) {
			double t[2];
			bool flag = false;
			__threadfence();                     // the CTA's u before its count
			const bool ok = sum_exchange<2>(dig[0], W, &a.gs->gamma[line], nctas, fG, &a.gs->bar, t, flag);
			if (lc == 0 && lane < kSumWords) a.gs->gamma[line >= 1 ? line - 1 : 2].w[lane] = 0ull;
			if (lane == 0) {
				if (!ok) gaveUp = 1;
				slow = flag ? 1 : 0;
				two[0] = t[0];
				two[1] = t[1];
			}
		} else if (rowWarp) {
#pragma unroll 1
			for (int j = 0; j < per; ++j) {      // while the reducer waits
				double *g = a.vec + (long) (sl0 + j * pw) * 32 * B + lane;
				double xv[B], pv[B];
#pragma unroll
				for (int c = 0; c < B; ++c) { xv[c] = g[32 * c]; pv[c] = g[vs + 32 * c]; }
#pragma unroll
				for (int c = 0; c < B; ++c) g[32 * c] = xv[c] + al * pv[c];
			}
		}
		__syncthreads();
		if (gaveUp) break;
		if (slow) {
			if (!slow_sum<2>(d2[0], d2[1], two, a.part + nctas, nctas, &a.gs->bar, target, fs)) {
				if (threadIdx.x == 0) gaveUp = 1;
				__syncthreads();
				break;
			}
		}
		if (++line == 3) line = 0;
		pending = true;
		first = false;
	}
	if (rowWarp) {
		for (int j = 0; j < per; ++j) {
			const int row = (sl0 + j * pw) * 32 + lane, i = __ldg(a.perm + row), scl = row_scale(__ldg(a.rowExp + row));
			const double *g = a.vec + (long) (sl0 + j * pw) * 32 * B + lane;
			if (i >= 0)
#pragma unroll
				for (int c = 0; c < B; ++c) a.x[(long) i * B + c] = scale_pow2(g[32 * c], scl);
		}
		for (int k = 0; k < nstage; ++k) {       // the ring's copies in flight land before the CTA leaves
			ring_wait(mb + 8 * stage, parity);
			if (++stage == nstage) { stage = 0; parity ^= 1u; }
		}
	}
	__syncthreads();
	if (wp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmemBase), "r"(kTmemCols));
	if (lc == 0 && threadIdx.x == 0) {
		sc->iters = iters; sc->code = gaveUp ? SA_ERR_TIMEOUT : max(stop, broke); sc->rr = rr; sc->gam = gam; sc->done = 1;
	}
}

template <int B>
bool cgfix_run(const Mesh &m, const double *blk, const double *binv, double *x, const double *r, const double *u,
               CgWork &w, cudaEvent_t e0, cudaEvent_t e1, cudaStream_t s)
{
	const CgPlan &p = w.plan;
	if (!p.ok || m.dim != B) return false;
	const int colMax = 32 * p.pw * p.widest;
	const size_t perStage = (size_t) p.pw * (256 * B * B + 8);
	int parts = 1, stages, per = p.per;
	size_t smem;
	const void *kernel;
	if (per > 1) {
		const size_t lim = smem_limit((const void *) k_cg_fix_many<B>), fixed = fix_many_smem<B>(p.pw, p.haloMax, 0);
		const size_t perStage = (size_t) p.pw * (many_slot<B>() + 8);
		if (fixed + 2 * perStage > lim) return false;
		stages = (int) ((lim - fixed) / perStage);
		smem = fix_many_smem<B>(p.pw, p.haloMax, stages);
		kernel = (const void *) k_cg_fix_many<B>;
	} else {
		const size_t lim = std::min(smem_limit((const void *) k_cg_fix<B, false>), smem_limit((const void *) k_cg_fix<B, true>));
		const bool resident = fix_smem<B>(p.pw, p.parts, p.haloMax, colMax, p.widest) <= lim;
		parts = resident ? p.parts : 1;
		const size_t fixed = fix_smem<B>(p.pw, parts, p.haloMax, colMax, 0);
		if (!resident && fixed + 2 * perStage > lim) return false;
		stages = resident ? p.widest : (int) ((lim - fixed) / perStage);
		smem = fix_smem<B>(p.pw, parts, p.haloMax, colMax, stages);
		kernel = resident ? (const void *) k_cg_fix<B, false> : (const void *) k_cg_fix<B, true>;
	}
	const int nctas = p.nchunk / per;
	int occ = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 32 * p.warps, smem) != cudaSuccess) {
		cudaGetLastError();
		return false;
	}
	if (nctas > occ * w.smCount || nctas > kSumMaxCtas) return false;
	const int P = p.nchunk * 32 * p.pw;
	k_cgfix_gather_copy<B><<<grid_for(P), kBlock, 0, s>>>(P, p.perm, u, binv, p.ug, p.scale);
	k_cgfix_operator<B><<<(p.nslice + 3) / 4, 128, 0, s>>>(p.nslice, sell_of(m), m.rowPtr, blk, p.perm, p.scale,
	                                                       p.width, p.off, p.fix, p.rowExp);
	if (per > 1) k_cgfix_inverses<B><<<grid_for(P), kBlock, 0, s>>>(P, p.perm, p.scale, binv, p.pinv);
	SA_CHECK(cudaMemsetAsync(w.bar, 0, sizeof(GridSums), s));
	FixArgs a{p.pw, parts, p.haloCap, p.haloMax, colMax, stages, p.perm, p.width, p.off, p.halo, p.haloNum, p.rowExp, p.lcol, p.fix,
	          binv, r, u, x, p.ug, p.vec, w.part, p.pinv, (CgScal *) w.scal, (GridSums *) w.bar};
	void *args[] = {&a, &per};
	if (e0) SA_CHECK(cudaEventRecord(e0, s));
	SA_CHECK(cudaLaunchCooperativeKernel(kernel, dim3(nctas), dim3(32 * p.warps), args, smem, s));
	if (e1) SA_CHECK(cudaEventRecord(e1, s));
	w.launches += per > 1 ? 4 : 3;
	return true;
}

template bool cgfix_run<2>(const Mesh &, const double *, const double *, double *, const double *, const double *,
                           CgWork &, cudaEvent_t, cudaEvent_t, cudaStream_t);
template bool cgfix_run<3>(const Mesh &, const double *, const double *, double *, const double *, const double *,
                           CgWork &, cudaEvent_t, cudaEvent_t, cudaStream_t);

}  // namespace sa
