// refine.cu -- FP64 kernels of the iterative refinement.
//
//  otf_gemv        y <- beta*y + alpha*A x with A regenerated from the LCG in
//                  FP64 (panel_gemv.hpp:57-180, otf_gemv.cpp:5-131); the
//                  diagonal comes from the FP64 diagonal vector.
//  trsv            x <- L^{-1} x or U^{-1} x with the FP32 LU factors and an
//                  FP64 vector (panel_trsv.hpp:310-758), one persistent
//                  cooperative launch with block-row flags.
//  infnorm, div, axpy   the vector helpers of panel_norm.hpp / panel.hpp.
#include "common.cuh"
#include "internal.h"
#include "tri_inv.cuh"

#include <mutex>

namespace hplai {

namespace {

struct JumpTable64 {
	Coeff p[64];
};

JumpTable64 make_table()
{
	JumpTable64 t;
	Coeff p{kLcgA, kLcgC};
	for (int k = 0; k < 64; ++k) {
		t.p[k] = p;
		p = coeff_mul(p, p);
	}
	return t;
}

const JumpTable64 &table()
{
	static const JumpTable64 t = make_table();
	return t;
}

// max that propagates NaN, so a diverged vector cannot report a finite norm
__device__ __forceinline__ double nan_max(double p, double q) { return (q != q || q > p) ? q : p; }

// *out <- max(*out, the block's largest m); every thread calls it, at most 32
// warps.  Non-negative doubles (and NaN above them) order like their bits.
__device__ __forceinline__ void block_max(double m, double *out)
{
	__shared__ double wm[32];
	for (int o = 16; o; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
	if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
	__syncthreads();
	if (threadIdx.x < 32) {
		m = (threadIdx.x < (blockDim.x + 31) / 32) ? wm[threadIdx.x] : 0.0;
		for (int o = 16; o; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
		if (threadIdx.x == 0)
			atomicMax(reinterpret_cast<unsigned long long *>(out), static_cast<unsigned long long>(__double_as_longlong(m)));
	}
	__syncthreads();
}

// ---------------------------------------------------------------------------
// On-the-fly GEMV: partial sums of GEMV_COLS columns by one of two kernels,
// and the chunks folded by a third, all in a fixed order, so the result does
// not depend on scheduling.
//
// Bound by the integer multiplies of the LCG (three of a 64-bit product, one
// of them wide) together with the FP64 multiply-add, which issue to the same
// port; hence the hardware's 64-bit integer conversion, which has a pipe of
// its own (the conversion through the mantissas of 2^84 and 2^52 costs two
// FP64 additions and was 25 % slower here).
// ---------------------------------------------------------------------------
constexpr int GEMV_THREADS = 256;
constexpr int GEMV_ROWS = 256;
constexpr int GEMV_COLS = 2048;

// The state of row lane's first column, for a warp whose first element is idx0
// and whose rows are `lp` apart; lp becomes the jump by 32 rows.
__device__ __forceinline__ uint64_t row_state(const Coeff *tab, uint64_t idx0, uint64_t state00, Coeff &lp)
{
	uint64_t s = coeff_apply(warp_jump(tab, idx0), state00);
#pragma unroll
	for (int b = 0; b < 5; ++b) {
		if ((threadIdx.x >> b) & 1) s = coeff_apply(lp, s);
		lp = coeff_mul(lp, lp);
	}
	return s;
}

// Large orders: CTA = 256 rows x GEMV_COLS columns, a row per thread with four
// interleaved LCG chains and two FP64 accumulators.
// TRANS: y = A^T x, output i walks column i of A (element (j, i) is state
// j + n*i, so the chain steps by 1 instead of n).  jn: the jump by n.
template <bool TRANS>
__global__ void __launch_bounds__(GEMV_ROWS) otf_rows_kernel(int64_t n, int mb, int nb, double alpha,
	const double *__restrict__ x, uint64_t state00, int with_diag, const double *__restrict__ diag,
	double *__restrict__ part, JumpTable64 tab, Coeff jn, double *norms)
{
	__shared__ __align__(16) double xs[GEMV_COLS];
	__shared__ Coeff stab[64];
	const int t = threadIdx.x, lane = t & 31;
	if (norms && blockIdx.x == 0 && blockIdx.y == 0 && t < 2) norms[t] = 0.0;   // for otf_reduce_kernel
	const int j0 = blockIdx.y * GEMV_COLS;
	const int j1 = min(j0 + GEMV_COLS, nb);
	for (int j = t; j < j1 - j0; j += GEMV_ROWS) xs[j] = x[j0 + j];
	if (t < 64) stab[t] = tab.p[t];
	__syncthreads();
	const int i = blockIdx.x * GEMV_ROWS + t;
	if (i - lane >= mb) return;   // whole warps
	const uint64_t iu = static_cast<uint64_t>(i - lane), ju = static_cast<uint64_t>(j0);
	Coeff lp = TRANS ? jn : stab[0];
	uint64_t s0 = row_state(stab, TRANS ? ju + static_cast<uint64_t>(n) * iu : iu + static_cast<uint64_t>(n) * ju, state00, lp);
	const Coeff jc = TRANS ? stab[0] : jn;
	const Coeff jc4 = coeff_mul(coeff_mul(jc, jc), coeff_mul(jc, jc));
	uint64_t s1 = coeff_apply(jc, s0);
	uint64_t s2 = coeff_apply(jc, s1);
	uint64_t s3 = coeff_apply(jc, s2);
	auto val = [](uint64_t v) { return __ll2double_rn(static_cast<long long>(v)); };
	double a0 = 0.0, a1 = 0.0;
	const int len = j1 - j0;
	const int dj = (with_diag && i >= j0 && i < j1) ? i - j0 : -1;   // diagonal column inside the chunk
	int j = 0;
	if (!__any_sync(0xffffffffu, dj >= 0)) {
		// no diagonal in this chunk for any row of the warp
		for (; j + 3 < len; j += 4) {
			const double2 x01 = *reinterpret_cast<const double2 *>(&xs[j]);
			const double2 x23 = *reinterpret_cast<const double2 *>(&xs[j + 2]);
			a0 = fma(val(s0), x01.x, a0);
			a1 = fma(val(s1), x01.y, a1);
			a0 = fma(val(s2), x23.x, a0);
			a1 = fma(val(s3), x23.y, a1);
			s0 = coeff_apply(jc4, s0);
			s1 = coeff_apply(jc4, s1);
			s2 = coeff_apply(jc4, s2);
			s3 = coeff_apply(jc4, s3);
		}
	} else {
		for (; j + 3 < len; j += 4) {
			const double v0 = j == dj ? 0.0 : val(s0), v1 = j + 1 == dj ? 0.0 : val(s1);
			const double v2 = j + 2 == dj ? 0.0 : val(s2), v3 = j + 3 == dj ? 0.0 : val(s3);
			a0 = fma(v0, xs[j], a0);
			a1 = fma(v1, xs[j + 1], a1);
			a0 = fma(v2, xs[j + 2], a0);
			a1 = fma(v3, xs[j + 3], a1);
			s0 = coeff_apply(jc4, s0);
			s1 = coeff_apply(jc4, s1);
			s2 = coeff_apply(jc4, s2);
			s3 = coeff_apply(jc4, s3);
		}
	}
	for (; j < len; ++j) {
		a0 = fma(j == dj ? 0.0 : val(s0), xs[j], a0);
		s0 = coeff_apply(jc, s0);
	}
	if (i >= mb) return;
	double r = (a0 + a1) * (alpha * kValueScale);
	if (dj >= 0) r = fma(alpha * diag[i], xs[dj], r);
	part[static_cast<int64_t>(blockIdx.y) * mb + i] = r;
}

// Smaller orders, whose rows alone would not fill the GPU: CTA = 64 rows x
// GEMV_COLS columns, divided into eight pieces, a warp each.  A thread walks
// two rows (32 apart, which share the reads of x) across its piece with two
// LCG chains and two FP64 accumulators a row; the pieces are folded in shared
// memory.
template <bool TRANS>
__global__ void __launch_bounds__(GEMV_THREADS) otf_pieces_kernel(int64_t n, int mb, int nb, double alpha,
	const double *__restrict__ x, uint64_t state00, int with_diag, const double *__restrict__ diag,
	double *__restrict__ part, JumpTable64 tab, Coeff jn, double *norms)
{
	constexpr int SPLIT = GEMV_THREADS / 32, R = 64;
	__shared__ __align__(16) double xs[GEMV_COLS];
	__shared__ Coeff stab[64];
	__shared__ double fold[SPLIT * R];
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
	if (norms && blockIdx.x == 0 && blockIdx.y == 0 && t < 2) norms[t] = 0.0;   // for otf_reduce_kernel
	const int j0 = blockIdx.y * GEMV_COLS;
	const int j1 = min(j0 + GEMV_COLS, nb);
	for (int j = t; j < j1 - j0; j += GEMV_THREADS) xs[j] = x[j0 + j];
	if (t < 64) stab[t] = tab.p[t];
	__syncthreads();
	const int iw = blockIdx.x * R;   // rows iw + lane and iw + lane + 32
	const int width = ((j1 - j0 + SPLIT - 1) / SPLIT + 3) & ~3;
	const int p0 = min(warp * width, j1 - j0), p1 = min(p0 + width, j1 - j0);
	double r[2] = {0.0, 0.0};
	// whole warps without columns have nothing to do
	if (p0 < p1) {
		const uint64_t iu = static_cast<uint64_t>(iw), ju = static_cast<uint64_t>(j0 + p0);
		uint64_t s[2][2];   // [row][column parity]
		Coeff lp = TRANS ? jn : stab[0];
		s[0][0] = row_state(stab, TRANS ? ju + static_cast<uint64_t>(n) * iu : iu + static_cast<uint64_t>(n) * ju, state00, lp);
		const Coeff jc = TRANS ? stab[0] : jn;
		const Coeff jc2 = coeff_mul(jc, jc);
		s[1][0] = coeff_apply(lp, s[0][0]);   // 32 rows on
		s[0][1] = coeff_apply(jc, s[0][0]);
		s[1][1] = coeff_apply(jc, s[1][0]);
		auto val = [](uint64_t v) { return __ll2double_rn(static_cast<long long>(v)); };
		double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
		const int len = p1 - p0;
		const double *xp = xs + p0;
		// diagonal columns in the piece
		const int dj0 = with_diag ? iw + lane - j0 - p0 : -1, dj1 = with_diag ? dj0 + 32 : -1;
		int j = 0;
		if (!__any_sync(0xffffffffu, (dj0 >= 0 && dj0 < len) || (dj1 >= 0 && dj1 < len))) {
			// no diagonal in this piece for any row of the warp
#pragma unroll 2
			for (; j + 1 < len; j += 2) {
				const double2 x01 = *reinterpret_cast<const double2 *>(&xp[j]);
#pragma unroll
				for (int q = 0; q < 2; ++q) {
					acc[q][0] = fma(val(s[q][0]), x01.x, acc[q][0]);
					acc[q][1] = fma(val(s[q][1]), x01.y, acc[q][1]);
					s[q][0] = coeff_apply(jc2, s[q][0]);
					s[q][1] = coeff_apply(jc2, s[q][1]);
				}
			}
		} else {
			for (; j + 1 < len; j += 2) {
				const double2 x01 = *reinterpret_cast<const double2 *>(&xp[j]);
#pragma unroll
				for (int q = 0; q < 2; ++q) {
					const int dj = q ? dj1 : dj0;
					const double v0 = j == dj ? 0.0 : val(s[q][0]), v1 = j + 1 == dj ? 0.0 : val(s[q][1]);
					acc[q][0] = fma(v0, x01.x, acc[q][0]);
					acc[q][1] = fma(v1, x01.y, acc[q][1]);
					s[q][0] = coeff_apply(jc2, s[q][0]);
					s[q][1] = coeff_apply(jc2, s[q][1]);
				}
			}
		}
		if (j < len) {
#pragma unroll
			for (int q = 0; q < 2; ++q) {
				const double v = j == (q ? dj1 : dj0) ? 0.0 : val(s[q][0]);
				acc[q][0] = fma(v, xp[j], acc[q][0]);
			}
		}
#pragma unroll
		for (int q = 0; q < 2; ++q) {
			const int dj = q ? dj1 : dj0, i = iw + lane + 32 * q;
			r[q] = (acc[q][0] + acc[q][1]) * (alpha * kValueScale);
			if (dj >= 0 && dj < len && i < mb) r[q] = fma(alpha * diag[i], xp[dj], r[q]);
		}
	}
	fold[warp * R + lane] = r[0];
	fold[warp * R + lane + 32] = r[1];
	__syncthreads();
	for (int e = t; e < R; e += GEMV_THREADS) {
		double v = fold[e];
#pragma unroll
		for (int q = 1; q < SPLIT; ++q) v += fold[q * R + e];
		const int i = blockIdx.x * R + e;
		if (i < mb) part[static_cast<int64_t>(blockIdx.y) * mb + i] = v;
	}
}

// y <- beta y0 + the chunks' sum (y0 may be y).  With `norms` (three doubles,
// the first two zeroed by the kernel before), also max |x_i| and max |y_i|
// into them and *status into the third, for the host to fetch in one copy.
__global__ void __launch_bounds__(256) otf_reduce_kernel(int mb, int nchunks, double beta,
	const double *__restrict__ part, const double *y0, double *y, int overwrite, const double *__restrict__ x,
	double *norms, const uint32_t *status)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	double r = 0.0, xv = 0.0;
	if (i < mb) {
		double s = 0.0;
		for (int c = 0; c < nchunks; ++c) s += part[static_cast<int64_t>(c) * mb + i];
		r = overwrite ? s : fma(beta, y0[i], s);
		y[i] = r;
		if (norms) xv = x[i];
	}
	if (norms) {
		block_max(fabs(xv), norms);
		block_max(fabs(r), norms + 1);
		if (i == 0) norms[2] = status ? static_cast<double>(*status) : 0.0;
	}
}

int otf_launch(int64_t n, int mb, int nb, double alpha, const double *x, double beta, double *y,
	uint64_t state00, int with_diag, const double *diag, void *work, size_t work_bytes, cudaStream_t st,
	bool trans = false, const double *y0 = nullptr, double *norms = nullptr,
	const uint32_t *status = nullptr)
{
	if (mb <= 0) return HPLAI_OK;
	const int nchunks = (nb + GEMV_COLS - 1) / GEMV_COLS;
	if (work_bytes < static_cast<size_t>(nchunks) * mb * sizeof(double)) return HPLAI_EINVAL;
	double *part = static_cast<double *>(work);
	if (nb > 0) {
		const Coeff jn = coeff_pow(static_cast<uint64_t>(n));
		// A row per thread once there are waves enough of such CTAs,
		// else pieces, which spread a small order over the SMs and balance the last
		// wave; for A^T, whose set-up is longer (the lanes' jumps are by n), sooner.
		// Rows / pieces, us: n = 1200 35 / 14.5, 16384 143 / 117, 24576 255 / 249,
		// 32768 426 / 427, 65536 1592 / 1662, 131072 6220 / 6600; A^T 9600 71 / 55,
		// 16384 131 / 123, 20480 183 / 186, 32768 405 / 457, 131072 5950 / 7090.
		const bool wide = static_cast<int64_t>((mb + GEMV_ROWS - 1) / GEMV_ROWS) * nchunks > (trans ? 800 : 2048);
		const dim3 grid((mb + (wide ? GEMV_ROWS : 64) - 1) / (wide ? GEMV_ROWS : 64), nchunks);
		const auto kernel = wide ? (trans ? otf_rows_kernel<true> : otf_rows_kernel<false>)
		                         : (trans ? otf_pieces_kernel<true> : otf_pieces_kernel<false>);
		kernel<<<grid, GEMV_THREADS, 0, st>>>(n, mb, nb, alpha, x, state00, with_diag, diag, part, table(), jn, norms);
		count_launches();
		HPLAI_CUDA_TRY(cudaGetLastError());
	}
	otf_reduce_kernel<<<(mb + 255) / 256, 256, 0, st>>>(mb, nb > 0 ? nchunks : 0, beta, part, y0 ? y0 : y, y,
		beta == 0.0 ? 1 : 0, x, norms, status);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

// ---------------------------------------------------------------------------
// On-the-fly GEMV over Higham's HPL-AI matrix (hmg_gemv_up/low/diag,
// otf_gemv.cpp:133-314): the entries of row i are the lower constants
// fma(ab, j, cl) of the columns j < i, the diagonal d_i and the upper
// constant fma(ab, i, cu) of the row; A^T swaps the two constants.  Same
// CTA shape, accumulators and fixed-order fold as the LCG GEMV.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(GEMV_ROWS) higham_partial_kernel(int n, double alpha, const double *__restrict__ x,
	double ab, double cu, double cl, const double *__restrict__ diag, double *__restrict__ part, double *norms)
{
	if (norms && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) norms[threadIdx.x] = 0.0;   // for otf_reduce_kernel
	__shared__ double xs[GEMV_COLS];
	__shared__ double ls[GEMV_COLS];
	const int j0 = blockIdx.y * GEMV_COLS;
	const int j1 = min(j0 + GEMV_COLS, n);
	for (int j = threadIdx.x; j < j1 - j0; j += GEMV_ROWS) {
		xs[j] = x[j0 + j];
		ls[j] = fma(ab, static_cast<double>(j0 + j), cl);
	}
	__syncthreads();
	const int i = blockIdx.x * GEMV_ROWS + threadIdx.x;
	if (i >= n) return;
	const double up = fma(ab, static_cast<double>(i), cu);
	const int len = j1 - j0;
	double a0 = 0.0, a1 = 0.0;
	int j = 0;
	for (; j + 1 < len; j += 2) {
		const int g = j0 + j;
		const double v0 = g < i ? ls[j] : (g > i ? up : 0.0);
		const double v1 = g + 1 < i ? ls[j + 1] : (g + 1 > i ? up : 0.0);
		a0 = fma(v0, xs[j], a0);
		a1 = fma(v1, xs[j + 1], a1);
	}
	if (j < len) {
		const int g = j0 + j;
		a0 = fma(g < i ? ls[j] : (g > i ? up : 0.0), xs[j], a0);
	}
	double r = (a0 + a1) * alpha;
	if (i >= j0 && i < j1) r = fma(alpha * diag[i], xs[i - j0], r);
	part[static_cast<int64_t>(blockIdx.y) * n + i] = r;
}

// ---------------------------------------------------------------------------
// Triangular solves.  Block rows of TB; CTA c handles block rows c, c+G, ...
// in solve order, accumulating the off-diagonal products as the block
// columns it depends on are published, then applying the FP64 inverse of its
// diagonal block and publishing x for that block.
// Progress is guaranteed because every CTA is resident (cooperative launch)
// and each works through its rows in dependency order.  Every spin is
// bounded; a timeout sets the status word and the kernel returns.
// ---------------------------------------------------------------------------
constexpr int TB = kTriBlock;
constexpr int TRSV_THREADS = kTriThreads;

// Zeroed once by the caller.  `epoch` counts the solves done on this
// workspace; the last CTA of a launch (counted in `done`) advances it.
struct TrsvWork {
	uint32_t epoch;
	uint32_t status;
	uint32_t done;
	uint32_t pad;
	// followed, 16-byte aligned, by the published solution: element j as two
	// 64-bit words, each the launch's epoch (high half) and one half of the
	// double's bits, so that a reader sees value and flag in one load
};

__device__ __forceinline__ void xt_publish(ulonglong2 *p, double v, uint32_t epoch)
{
	const uint64_t e = static_cast<uint64_t>(epoch) << 32;
	const uint64_t lo = e | static_cast<uint32_t>(__double2loint(v)), hi = e | static_cast<uint32_t>(__double2hiint(v));
	asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}

__device__ __forceinline__ ulonglong2 xt_load(const ulonglong2 *p)
{
	ulonglong2 v;
	asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
	return v;
}

__device__ __forceinline__ bool xt_ready(ulonglong2 v, uint32_t epoch)
{
	return static_cast<uint32_t>(v.x >> 32) == epoch && static_cast<uint32_t>(v.y >> 32) == epoch;
}

__device__ __forceinline__ double xt_value(ulonglong2 v)
{
	return __hiloint2double(static_cast<int>(static_cast<uint32_t>(v.y)), static_cast<int>(static_cast<uint32_t>(v.x)));
}

// FP64 inverses of the TB x TB diagonal blocks of the stored factors:
// dinv[(2*r + 0) * TB*TB + c*TB + i] = (L_rr^{-1})[i][c] (unit lower) and
// dinv[(2*r + 1) * TB*TB + c*TB + i] = (U_rr^{-1})[i][c], rows/columns past
// n padded with the identity.  Computed once per factorisation; the
// triangular solves then apply a block as one product.
__global__ void __launch_bounds__(TRSV_THREADS) trsv_dinv_kernel(int n, const float *__restrict__ a, int64_t lda,
	double *__restrict__ dinv, int blk0)
{
	extern __shared__ __align__(16) float dyn_smem[];
	double *X = reinterpret_cast<double *>(dyn_smem);
	const int r = blk0 + blockIdx.x, upper = blockIdx.y;
	const int r0 = r * TB, rows = min(TB, n - r0);
	invert_block(X, a, lda, r0, rows, upper != 0);
	double *out = dinv + (static_cast<int64_t>(2 * r + upper) * TB) * TB;
	for (int e = threadIdx.x; e < TB * TB; e += TRSV_THREADS) {
		const int i = e % TB, c = e / TB;
		out[e] = upper ? X[c * kInvLd + i] : X[i * kInvLd + c];
	}
}

// Copy block (rows r0.., cols c0..) of M into shared memory with cp.async:
// TRANS (M[i][j] = a[i*lda + j]) as blk[i*TB + j], otherwise
// (M[i][j] = a[j*lda + i]) as blk[j*TB + i]; rows >= rows / cols >= cols
// are zero.  vec: 16-byte copies through L2 (a 16-byte aligned, lda % 4 == 0),
// else 4-byte copies.  The matrix is read-only for the whole solve.
template <bool TRANS>
__device__ __forceinline__ void stage_block(float *blk, const float *a, int64_t lda, int r0, int c0, int rows,
	int cols, bool vec)
{
	const int t = threadIdx.x;
	// contiguous index of the stored matrix: rows for M = stored, columns for M^T
	const int ncont = TRANS ? cols : rows, nline = TRANS ? rows : cols;
	if (vec) {
		for (int e = t; e < TB * TB / 4; e += TRSV_THREADS) {
			const int line = e / (TB / 4), g = (e % (TB / 4)) * 4;
			int bytes = (line < nline) ? (ncont - g) * 4 : 0;
			bytes = bytes < 0 ? 0 : (bytes > 16 ? 16 : bytes);
			const float *src = TRANS ? a + static_cast<int64_t>(r0 + (bytes ? line : 0)) * lda + c0 + (bytes ? g : 0)
			                         : a + static_cast<int64_t>(c0 + (bytes ? line : 0)) * lda + r0 + (bytes ? g : 0);
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(blk + line * TB + g)),
				"l"(src), "r"(bytes) : "memory");
		}
	} else {
		for (int e = t; e < TB * TB; e += TRSV_THREADS) {
			const int line = e / TB, g = e % TB;
			const bool in = line < nline && g < ncont;
			const float *src = TRANS ? a + static_cast<int64_t>(r0 + (in ? line : 0)) * lda + c0 + (in ? g : 0)
			                         : a + static_cast<int64_t>(c0 + (in ? line : 0)) * lda + r0 + (in ? g : 0);
			asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(blk + line * TB + g)), "l"(src),
				"r"(in ? 4 : 0) : "memory");
		}
	}
	asm volatile("cp.async.commit_group;" ::: "memory");
}

// x <- T^{-1} x by substitution, T (column-major, TB x TB) and x in shared
// memory: unit LOWER or non-unit upper.  32 rows at a time: the first warp
// solves them, a shuffle and a multiply-add (and a division) per step, and a
// thread per row left applies them.  Ends with a barrier.
template <bool LOWER>
__device__ __noinline__ void substitute_block(const float *T, double *x, int rows)
{
	const int t = threadIdx.x, lane = t & 31;
	for (int k = 0; k < TB / 32; ++k) {
		const int c0 = LOWER ? 32 * k : TB - 32 * (k + 1);
		if (c0 >= rows) continue;
		if (t < 32) {
			const int i = c0 + lane;
			double v = x[i];
			const double d = !LOWER && i < rows ? static_cast<double>(T[i * TB + i]) : 1.0;
			const int w = min(32, rows - c0);
#pragma unroll 4
			for (int q = 0; q < w; ++q) {
				const int j = LOWER ? q : w - 1 - q;
				if (!LOWER && lane == j) v /= d;
				const double xj = __shfl_sync(0xffffffffu, v, j);
				if (LOWER ? lane > j : lane < j) v = fma(-static_cast<double>(T[(c0 + j) * TB + i]), xj, v);
			}
			x[i] = v;
		}
		__syncthreads();
		if (t < TB && (LOWER ? t >= c0 + 32 : t < c0)) {
			double v = x[t];
			for (int j = 0; j < 32; ++j) v = fma(-static_cast<double>(T[(c0 + j) * TB + t]), x[c0 + j], v);
			x[t] = v;
		}
		__syncthreads();
	}
}

// Whether the diagonal block's inverse may be applied: its condition number
// max_i (|T^{-1}| |T| e)_i is at most 32.  Substitution is backward stable for every
// triangle, the product with an explicit inverse only for a well-conditioned one.
// Row by row |b - T x| / (|T| |x| + |b|) over 128 rows, in units of 2^-53, by
// substitution / by the inverse: the factors of dominant matrices (condition 1 to 4)
// 5.9 to 7.6 / 1.0 to 1.4, unit lower entries in (-0.1, 0.1) (condition 40) 2.8 / 1.3,
// (-0.2, 0.2) (170) 2.1 / 2.2, (-0.5, 0.5) (1e4) 1.9 / 82, (-1, 1) (2e9) 1.2 / 1e7.
// inv[q] = T^{-1}[lr][64 grp + q] (NaN and infinities fail the test); part: two rows
// of TB.  The same answer in every thread; ends with a barrier.
__device__ __forceinline__ bool inverse_serves(const double (&inv)[TB / 2], const float *a, int64_t lda, int r0,
	int rows, bool lower, double (*part)[TB])
{
	const int lr = threadIdx.x % TB, grp = threadIdx.x / TB;
	const float *row = a + static_cast<int64_t>(r0 + grp * (TB / 2)) * lda + r0 + lr;
	float sum = 0.f;
#pragma unroll 32
	for (int q = 0; q < TB / 2; ++q) {
		const int j = grp * (TB / 2) + q;
		if (lr < rows && j < rows && (lower ? j < lr : j >= lr)) sum += fabsf(__ldcg(row + static_cast<int64_t>(q) * lda));
	}
	part[grp][lr] = lower && grp == 0 ? 1.0 + sum : sum;
	__syncthreads();
	double c[2] = {0.0, 0.0};
#pragma unroll
	for (int q = 0; q < TB / 2; ++q)
		c[q & 1] = fma(fabs(inv[q]), part[0][grp * (TB / 2) + q] + part[1][grp * (TB / 2) + q], c[q & 1]);
	__syncthreads();
	part[grp][lr] = c[0] + c[1];
	__syncthreads();
	return __syncthreads_and(part[0][lr] + part[1][lr] <= 32.0) != 0;
}

// TRANS: the triangle solved is the transpose of the stored one, M[i][j] =
// a[i*lda + j]: lower = U^T (non-unit), upper = L^T (unit).  Otherwise
// M[i][j] = a[j*lda + i]: lower = L (unit), upper = U (non-unit).
//
// What bounds it: n / 128 dependent steps (a block's x travels to the next
// block row's CTA, is multiplied by one 128 x 128 block and by a diagonal
// inverse), and for large n the one read of the triangle.  So everything a
// step does not need from the step before it happens while it waits:
//  - the off-diagonal blocks stream through three shared-memory buffers, two
//    copies in flight while one block is applied;
//  - x travels as tagged words (xt_publish): one L2 round trip carries value
//    and flag, with no fence on the producer's side and no second load on
//    the consumer's; the words of the next block are requested before the
//    current one is applied;
//  - this thread's 64 entries of the diagonal inverse sit in registers (read
//    from dinv, or, where the caller keeps no inverses (HAVE_INV = false),
//    computed here by invert_block), so the diagonal is one product of four
//    short FMA chains.  Nothing behind a leaf call corrects that product, so
//    without dinv a block that fails inverse_serves is solved by substitution.
// Measured per triangle, before (flag word and fence, 128-step substitution
// without dinv) and now: n = 8192 204 -> 114 us, transposed 590 -> 139;
// n = 65536 2.45 -> 2.13 ms (4.0 TB/s), 131072 8.28 -> 7.70; without dinv
// n = 16384 2370 -> 263 us (256 without the condition numbers; 785 where every
// block is substituted).
template <bool TRANS, bool HAVE_INV>
__global__ void __launch_bounds__(TRSV_THREADS, 1) trsv_kernel(int lower, int n, const float *__restrict__ a,
	int64_t lda, double *x, TrsvWork *w, ulonglong2 *xt, const double *__restrict__ dinv)
{
	extern __shared__ __align__(16) float dyn_smem[];   // three TB x TB blocks
	constexpr int NB = 3;
	const bool vec = ((reinterpret_cast<uintptr_t>(a) & 15u) == 0) && ((lda & 3) == 0);
	__shared__ __align__(16) double xsb[2][TB];   // x of the block columns, alternating
	__shared__ __align__(16) double part[2][TB];  // partial sums of the two column halves
	__shared__ __align__(16) double rhs[TB];

	const uint32_t epoch = *reinterpret_cast<volatile uint32_t *>(&w->epoch) + 1u;
	const int nbt = (n + TB - 1) / TB;
	const int t = threadIdx.x;
	const int lr = t % TB, grp = t / TB;   // row within the block, column half
	const int jb = grp * (TB / 2);
	bool bad = false;

	for (int idx = blockIdx.x; idx < nbt; idx += gridDim.x) {
		const int r = lower ? idx : nbt - 1 - idx;
		const int r0 = r * TB;
		const int rows = min(TB, n - r0);
		const int nblk = lower ? r : nbt - 1 - r;
		int extra = 0;   // 1: the diagonal block is substituted, and staged last (col_of(nblk) == r)
		auto col_of = [&](int q) { return lower ? q : nbt - 1 - q; };
		// the first NB - 1 off-diagonal blocks in flight before anything waits;
		// one copy group per block (empty past the last) keeps the count fixed
		auto stage_q = [&](int q) {
			if (q < nblk + extra) {
				const int cb = col_of(q);
				stage_block<TRANS>(dyn_smem + (q % NB) * TB * TB, a, lda, r0, cb * TB, rows, min(TB, n - cb * TB), vec);
			} else {
				asm volatile("cp.async.commit_group;" ::: "memory");
			}
		};
		// this block's right-hand side (only this CTA writes it, at the end)
		const double xr = (t < rows) ? __ldcg(&x[r0 + t]) : 0.0;
		// dv[q] = M_rr^{-1}[lr][jb + q]
		double dv[TB / 2];
		if (HAVE_INV) {
			const int tri = (lower != 0) == !TRANS ? 0 : 1;   // L for lower / L^T, U for upper / U^T
			const double *dblock = dinv + (static_cast<int64_t>(2 * r + tri) * TB) * TB;
			if (TRANS) {
				const double2 *row = reinterpret_cast<const double2 *>(dblock + static_cast<int64_t>(lr) * TB + jb);
#pragma unroll
				for (int q = 0; q < TB / 4; ++q) {
					const double2 d2 = __ldcg(&row[q]);
					dv[2 * q] = d2.x;
					dv[2 * q + 1] = d2.y;
				}
			} else {
#pragma unroll
				for (int q = 0; q < TB / 2; ++q) dv[q] = __ldcg(&dblock[static_cast<int64_t>(jb + q) * TB + lr]);
			}
		} else if (lower ? nblk <= 1 : nblk == 0 && rows <= 64) {
			// the first blocks have no wait to hide an inverse in, and substitution is
			// shorter where it does not divide or is small (inverse / so: L n = 16
			// 11.6 / 7.3 us, 128 21.7 / 11.9, 256 23.8 / 19.6; U n = 32 13.6 / 9.5, 60 17.7 /
			// 17.9, 128 21.7 / 28)
			extra = 1;
		} else {
			double *X = reinterpret_cast<double *>(dyn_smem);
			invert_block(X, a, lda, r0, rows, lower == 0);
#pragma unroll
			for (int q = 0; q < TB / 2; ++q) dv[q] = lower ? X[lr * kInvLd + jb + q] : X[(jb + q) * kInvLd + lr];
			__syncthreads();
			extra = inverse_serves(dv, a, lda, r0, rows, lower != 0, part) ? 0 : 1;
		}
		double acc4[4] = {0.0, 0.0, 0.0, 0.0};
		// TRANS: warp `wv` takes rows wv, wv + 8, ...; lane takes 4 columns
		double tacc[TB / 8];
#pragma unroll
		for (int q = 0; q < TB / 8; ++q) tacc[q] = 0.0;
		for (int q = 0; q < NB - 1; ++q) stage_q(q);
		ulonglong2 xw = make_ulonglong2(0, 0);
		if (t < TB && nblk > 0) xw = xt_load(xt + static_cast<int64_t>(col_of(0)) * TB + t);
		// Off-diagonal block columns in dependency order, one barrier per block.
		// Before it, the first four warps make sure that x of the block is
		// published and put it in shared memory, and every thread waits for its
		// own copies of the block; after it, the buffer of the previous block
		// receives the block NB - 1 ahead, and the block is applied.
		for (int q = 0; q < nblk; ++q) {
			double *xs = xsb[q & 1];
			if (t < TB) {
				const int j = col_of(q) * TB + t;
				const ulonglong2 *src = xt + j;
				uint64_t t0 = 0;
				for (int it = 0; __any_sync(0xffffffffu, j < n && !xt_ready(xw, epoch)); ++it) {
					// the decision to give up is taken by the whole warp at once
					if ((it & 255) == 0) {
						const uint64_t now = global_ns();
						if (it == 0) t0 = now;
						if (__any_sync(0xffffffffu, now - t0 > kWaitLimitNs)) {
							bad = true;
							break;
						}
					}
					xw = xt_load(src);
				}
				xs[t] = (j < n) ? xt_value(xw) : 0.0;
			}
			// block q has landed (the one after it may still be in flight)
			asm volatile("cp.async.wait_group 1;" ::: "memory");
			bad = __syncthreads_or(bad) != 0;
			if (bad) break;
			stage_q(q + NB - 1);
			if (t < TB && q + 1 < nblk) xw = xt_load(xt + static_cast<int64_t>(col_of(q + 1)) * TB + t);
			const float *cur = dyn_smem + (q % NB) * TB * TB;
			if (TRANS) {
				const int wv = t >> 5, j = 4 * (t & 31);
				const double x0 = xs[j], x1 = xs[j + 1], x2 = xs[j + 2], x3 = xs[j + 3];
#pragma unroll
				for (int qq = 0; qq < TB / 8; ++qq) {
					const int i = wv + 8 * qq;
					const float4 v = *reinterpret_cast<const float4 *>(cur + i * TB + j);
					double s4 = tacc[qq];
					s4 = fma(static_cast<double>(v.x), x0, s4);
					s4 = fma(static_cast<double>(v.y), x1, s4);
					s4 = fma(static_cast<double>(v.z), x2, s4);
					s4 = fma(static_cast<double>(v.w), x3, s4);
					tacc[qq] = s4;
				}
			} else {
				// four independent FMA chains: one chain of 64 dependent FMAs per
				// block left the FP64 pipe waiting on its own latency
#pragma unroll
				for (int k = 0; k < TB / 2; k += 4) {
					const int j = jb + k;
					const double2 x01 = *reinterpret_cast<const double2 *>(&xs[j]);
					const double2 x23 = *reinterpret_cast<const double2 *>(&xs[j + 2]);
					acc4[0] = fma(static_cast<double>(cur[j * TB + lr]), x01.x, acc4[0]);
					acc4[1] = fma(static_cast<double>(cur[(j + 1) * TB + lr]), x01.y, acc4[1]);
					acc4[2] = fma(static_cast<double>(cur[(j + 2) * TB + lr]), x23.x, acc4[2]);
					acc4[3] = fma(static_cast<double>(cur[(j + 3) * TB + lr]), x23.y, acc4[3]);
				}
			}
		}
		if (bad) break;
		if (TRANS) {
			// the 16 rows' sums over 32 lanes: each exchange halves the values a
			// lane holds, in a fixed order
			const int wv = t >> 5, ln = t & 31;
#pragma unroll
			for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
				const bool up = (ln & o) != 0;
#pragma unroll
				for (int q = 0; q < h; ++q) {
					const double send = up ? tacc[q] : tacc[q + h], keep = up ? tacc[q + h] : tacc[q];
					tacc[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
				}
			}
			tacc[0] += __shfl_xor_sync(0xffffffffu, tacc[0], 1);
			const int qq = ((ln >> 4) & 1) * 8 + ((ln >> 3) & 1) * 4 + ((ln >> 2) & 1) * 2 + ((ln >> 1) & 1);
			if ((ln & 1) == 0) {
				part[0][wv + 8 * qq] = tacc[0];
				part[1][wv + 8 * qq] = 0.0;
			}
		} else {
			part[grp][lr] = (acc4[0] + acc4[1]) + (acc4[2] + acc4[3]);
		}
		__syncthreads();
		const double br = (t < rows) ? xr - (part[0][t] + part[1][t]) : 0.0;
		if (t < TB) rhs[t] = br;
		// an infinity or NaN reaches only the rows that depend on it, which the
		// inverse's zeros would not see to
		const bool finite = __syncthreads_and(isfinite(br)) != 0;
		if (!HAVE_INV && (extra || !finite)) {
			float *T = dyn_smem + (nblk % NB) * TB * TB;
			if (!extra) stage_block<false>(T, a, lda, r0, r0, rows, rows, vec);
			asm volatile("cp.async.wait_all;" ::: "memory");
			__syncthreads();
			if (lower)
				substitute_block<true>(T, rhs, rows);
			else
				substitute_block<false>(T, rhs, rows);
			if (t < rows) {
				const double v = rhs[t];
				xt_publish(xt + r0 + t, v, epoch);
				x[r0 + t] = v;
			}
			continue;
		}
		// x_r = M_rr^{-1} rhs
		double v4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
		for (int q = 0; q < TB / 2; q += 4) {
			const double2 y01 = *reinterpret_cast<const double2 *>(&rhs[jb + q]);
			const double2 y23 = *reinterpret_cast<const double2 *>(&rhs[jb + q + 2]);
			v4[0] = fma(dv[q], y01.x, v4[0]);
			v4[1] = fma(dv[q + 1], y01.y, v4[1]);
			v4[2] = fma(dv[q + 2], y23.x, v4[2]);
			v4[3] = fma(dv[q + 3], y23.y, v4[3]);
		}
		part[grp][lr] = (v4[0] + v4[1]) + (v4[2] + v4[3]);
		__syncthreads();
		if (t < rows) {
			const double v = part[0][t] + part[1][t];
			xt_publish(xt + r0 + t, v, epoch);
			x[r0 + t] = v;
		}
	}
	// copies still in flight after a timeout land before the CTA exits
	asm volatile("cp.async.wait_all;" ::: "memory");
	if (t == 0) {
		if (bad) atomicOr(&w->status, 1u);
		// every CTA has read the epoch before it counts itself done
		__threadfence();
		if (atomicAdd(&w->done, 1u) == gridDim.x - 1) {
			w->done = 0;
			w->epoch = epoch;
		}
	}
}

// ---------------------------------------------------------------------------
// Vector helpers.
// ---------------------------------------------------------------------------
__global__ void infnorm_kernel(int n, const double *__restrict__ x, double *out)
{
	double m = 0.0;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = nan_max(m, fabs(x[i]));
	block_max(m, out);
}

// Checksum of the factored matrix (panel_check.hpp:9-65): FP64 sums of
// |a_ij| over the diagonal, the strict upper and the strict lower triangle.
// HBM-bound (4 n^2 bytes read once).  One warp per column, grid-stride over
// columns, two float4 loads in flight per lane where a and lda allow them;
// each CTA writes its three partial sums and one CTA folds them in a fixed
// order, so the result depends on n and the matrix only.
constexpr int kCheckWarps = 8;

int check_blocks(int n)
{
	const int need = (n + kCheckWarps - 1) / kCheckWarps;
	return need < 1184 ? (need > 0 ? need : 1) : 1184;   // 148 SMs x 8 CTAs
}

__device__ __forceinline__ void check_add(float v, int r, int j, double &sd, double &su, double &sl)
{
	const double t = fabs(static_cast<double>(v));
	if (r < j) su += t;
	else if (r == j) sd += t;
	else sl += t;
}

__global__ void __launch_bounds__(kCheckWarps * 32) check_partial_kernel(int n, const float *__restrict__ a,
	int64_t lda, int vec, double *__restrict__ part)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	double sd = 0.0, su = 0.0, sl = 0.0;
	const int n4 = vec ? (n & ~3) : 0;
	for (int j = blockIdx.x * kCheckWarps + warp; j < n; j += gridDim.x * kCheckWarps) {
		const float *col = a + static_cast<int64_t>(j) * lda;
		int i = lane * 4;
		for (; i + 128 < n4; i += 256) {
			const float4 v0 = __ldcs(reinterpret_cast<const float4 *>(col + i));
			const float4 v1 = __ldcs(reinterpret_cast<const float4 *>(col + i + 128));
			check_add(v0.x, i, j, sd, su, sl);
			check_add(v0.y, i + 1, j, sd, su, sl);
			check_add(v0.z, i + 2, j, sd, su, sl);
			check_add(v0.w, i + 3, j, sd, su, sl);
			check_add(v1.x, i + 128, j, sd, su, sl);
			check_add(v1.y, i + 129, j, sd, su, sl);
			check_add(v1.z, i + 130, j, sd, su, sl);
			check_add(v1.w, i + 131, j, sd, su, sl);
		}
		if (i < n4) {
			const float4 v0 = __ldcs(reinterpret_cast<const float4 *>(col + i));
			check_add(v0.x, i, j, sd, su, sl);
			check_add(v0.y, i + 1, j, sd, su, sl);
			check_add(v0.z, i + 2, j, sd, su, sl);
			check_add(v0.w, i + 3, j, sd, su, sl);
		}
		for (int r = n4 + lane; r < n; r += 32) check_add(__ldcs(col + r), r, j, sd, su, sl);
	}
	for (int o = 16; o; o >>= 1) {
		sd += __shfl_xor_sync(0xffffffffu, sd, o);
		su += __shfl_xor_sync(0xffffffffu, su, o);
		sl += __shfl_xor_sync(0xffffffffu, sl, o);
	}
	__shared__ double ws[3][kCheckWarps];
	if (lane == 0) {
		ws[0][warp] = sd;
		ws[1][warp] = su;
		ws[2][warp] = sl;
	}
	__syncthreads();
	if (threadIdx.x < 3) {
		double s = 0.0;
		for (int w = 0; w < kCheckWarps; ++w) s += ws[threadIdx.x][w];
		part[3 * blockIdx.x + threadIdx.x] = s;
	}
}

__global__ void __launch_bounds__(256) check_fold_kernel(int nparts, const double *__restrict__ part, double *sigs)
{
	__shared__ double s[3][256];
	const int t = threadIdx.x;
	double d = 0.0, u = 0.0, l = 0.0;
	for (int p = t; p < nparts; p += 256) {
		d += part[3 * p];
		u += part[3 * p + 1];
		l += part[3 * p + 2];
	}
	s[0][t] = d;
	s[1][t] = u;
	s[2][t] = l;
	for (int o = 128; o; o >>= 1) {
		__syncthreads();
		if (t < o) {
			s[0][t] += s[0][t + o];
			s[1][t] += s[1][t + o];
			s[2][t] += s[2][t + o];
		}
	}
	__syncthreads();
	if (t < 3) sigs[t] = s[t][0];
}

__global__ void div_kernel(int n, const double *__restrict__ num, const double *__restrict__ den, double *out)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) out[i] = num[i] / den[i];
}

__global__ void axpy1_kernel(int n, const double *__restrict__ x, double *y)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) y[i] += x[i];
}

} // namespace

size_t otf_gemv_workspace(int n)
{
	if (n <= 0) return 0;
	const size_t nchunks = (static_cast<size_t>(n) + GEMV_COLS - 1) / GEMV_COLS;
	return nchunks * static_cast<size_t>(n) * sizeof(double);
}

int launch_otf_gemv(int n, double alpha, const double *x, double beta, double *y, uint64_t seed, const double *diag,
	void *work, size_t work_bytes, cudaStream_t st, bool trans, const double *y0, double *norms,
	const uint32_t *status)
{
	return otf_launch(n, n, n, alpha, x, beta, y, state_initial(seed), 1, diag, work, work_bytes, st, trans, y0, norms,
		status);
}

int launch_higham_gemv(int n, double alpha, const double *x, double beta, double *y, double halpha, double hbeta,
	const double *diag, void *work, size_t work_bytes, cudaStream_t st, bool trans, const double *y0, double *norms,
	const uint32_t *status)
{
	if (n <= 0) return HPLAI_OK;
	const int nchunks = (n + GEMV_COLS - 1) / GEMV_COLS;
	if (work_bytes < static_cast<size_t>(nchunks) * n * sizeof(double)) return HPLAI_EINVAL;
	double *part = static_cast<double *>(work);
	const double ab = halpha * hbeta;
	// A: upper constants -beta + ab i, lower -alpha + ab j; A^T the other way round
	const double cu = trans ? -halpha : -hbeta, cl = trans ? -hbeta : -halpha;
	higham_partial_kernel<<<dim3((n + GEMV_ROWS - 1) / GEMV_ROWS, nchunks), GEMV_ROWS, 0, st>>>(n, alpha, x, ab, cu, cl,
		diag, part, norms);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	otf_reduce_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, nchunks, beta, part, y0 ? y0 : y, y, beta == 0.0 ? 1 : 0, x,
		norms, status);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

int launch_otf_gemv_block(int64_t n, int mb, int nb, double alpha, const double *x, double *y, uint64_t state00,
	void *work, size_t work_bytes, cudaStream_t st)
{
	return otf_launch(n, mb, nb, alpha, x, 1.0, y, state00, 0, nullptr, work, work_bytes, st);
}

// header, alignment slack, two 64-bit words per element of the padded solution
size_t trsv_workspace(int n)
{
	const size_t nbt = (static_cast<size_t>(n) + TB - 1) / TB;
	return sizeof(TrsvWork) + 16 + nbt * TB * sizeof(ulonglong2);
}

int launch_trsv(bool lower, int n, const float *a, int64_t lda, double *x, void *work, size_t work_bytes,
	cudaStream_t st, bool trans, const double *dinv)
{
	if (n <= 0) return HPLAI_OK;
	if (!work || work_bytes < trsv_workspace(n)) return HPLAI_EINVAL;
	if (trans && !dinv) return HPLAI_EINVAL;
	constexpr size_t dsmem = sizeof(float) * 3 * TB * TB;
	static_assert(kInvSmem<double> <= dsmem, "the in-kernel inverse shares the block buffers");
	// co-resident CTAs of the cooperative launch on this device
	static DeviceOnce grid_once;
	int max_blocks = 0;
	HPLAI_TRY(grid_once.get([&](int dev, int *v) -> int {
		const void *fns[3] = {reinterpret_cast<const void *>(trsv_kernel<false, false>),
			reinterpret_cast<const void *>(trsv_kernel<false, true>), reinterpret_cast<const void *>(trsv_kernel<true, true>)};
		int least = 1 << 30, sms = 0;
		for (const void *f : fns) {
			int per_sm = 0;
			HPLAI_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(dsmem)));
			HPLAI_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, TRSV_THREADS, dsmem));
			least = per_sm < least ? per_sm : least;
		}
		HPLAI_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
		*v = least * sms;
		return HPLAI_OK;
	}, &max_blocks));
	if (max_blocks <= 0) return HPLAI_EUNSUPPORTED;
	// the transposed solve reads rows of the stored matrix as float4
	if (trans && ((reinterpret_cast<uintptr_t>(a) & 15u) || (lda & 3))) return HPLAI_EINVAL;
	TrsvWork *w = static_cast<TrsvWork *>(work);
	ulonglong2 *xt = reinterpret_cast<ulonglong2 *>((reinterpret_cast<uintptr_t>(w + 1) + 15) & ~static_cast<uintptr_t>(15));
	const int nbt = (n + TB - 1) / TB;
	const int grid = nbt < max_blocks ? nbt : max_blocks;
	int lw = lower ? 1 : 0;
	void *args[] = {(void *)&lw, (void *)&n, (void *)&a, (void *)&lda, (void *)&x, (void *)&w, (void *)&xt, (void *)&dinv};
	const void *fn = trans ? reinterpret_cast<const void *>(trsv_kernel<true, true>)
		: dinv ? reinterpret_cast<const void *>(trsv_kernel<false, true>)
		       : reinterpret_cast<const void *>(trsv_kernel<false, false>);
	HPLAI_CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(TRSV_THREADS), args, dsmem, st));
	count_launches();
	return HPLAI_OK;
}

// Clears the solves' timeout word.
int trsv_status_reset(void *work, cudaStream_t st)
{
	TrsvWork *w = static_cast<TrsvWork *>(work);
	HPLAI_CUDA_TRY(cudaMemsetAsync(&w->status, 0, sizeof(w->status), st));
	return HPLAI_OK;
}

size_t trsv_dinv_doubles(int n)
{
	const size_t nbt = (static_cast<size_t>(n) + TB - 1) / TB;
	return 2 * nbt * TB * TB;
}

int launch_trsv_dinv(int n, const float *a, int64_t lda, double *dinv, cudaStream_t st, int blk0, int nblk)
{
	if (n <= 0) return HPLAI_OK;
	const int nbt = (n + TB - 1) / TB;
	if (nblk < 0) nblk = nbt - blk0;
	if (blk0 < 0 || nblk <= 0 || blk0 + nblk > nbt) return nblk == 0 ? HPLAI_OK : HPLAI_EINVAL;
	static DeviceOnce attr;
	HPLAI_TRY(attr.get([](int, int *) -> int {
		HPLAI_CUDA_TRY(cudaFuncSetAttribute(trsv_dinv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
			static_cast<int>(kInvSmem<double>)));
		return HPLAI_OK;
	}));
	trsv_dinv_kernel<<<dim3(nblk, 2), TRSV_THREADS, kInvSmem<double>, st>>>(n, a, lda, dinv, blk0);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

const uint32_t *trsv_status_word(const void *work) { return &static_cast<const TrsvWork *>(work)->status; }

int launch_infnorm(int n, const double *x, double *out, cudaStream_t st)
{
	HPLAI_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double), st));
	if (n <= 0) return HPLAI_OK;
	int blocks = (n + 255) / 256;
	if (blocks > 1184) blocks = 1184;
	infnorm_kernel<<<blocks, 256, 0, st>>>(n, x, out);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

size_t panel_check_workspace(int n)
{
	return 3 * sizeof(double) * static_cast<size_t>(check_blocks(n));
}

int launch_panel_check(int n, const float *a, int64_t lda, double *sigs, void *work, size_t work_bytes,
	cudaStream_t st)
{
	if (n <= 0) {
		HPLAI_CUDA_TRY(cudaMemsetAsync(sigs, 0, 3 * sizeof(double), st));
		return HPLAI_OK;
	}
	if (work_bytes < panel_check_workspace(n)) return HPLAI_EINVAL;
	const int blocks = check_blocks(n);
	const int vec = (reinterpret_cast<uintptr_t>(a) % 16 == 0 && lda % 4 == 0) ? 1 : 0;
	double *part = static_cast<double *>(work);
	check_partial_kernel<<<blocks, kCheckWarps * 32, 0, st>>>(n, a, lda, vec, part);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	check_fold_kernel<<<1, 256, 0, st>>>(blocks, part, sigs);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

int launch_div(int n, const double *num, const double *den, double *out, cudaStream_t st)
{
	if (n <= 0) return HPLAI_OK;
	div_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, num, den, out);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

int launch_axpy1(int n, const double *x, double *y, cudaStream_t st)
{
	if (n <= 0) return HPLAI_OK;
	axpy1_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, x, y);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free on-the-fly GEMV.
//
// Callers that cannot allocate device memory (code that is handed every
// device buffer by another runtime's allocator and has none of its own, or a
// solve loop that must not call cudaMalloc because it can synchronise the
// device) get the GEMV's partial-sum scratch from this fixed array instead
// of a caller workspace.  It is part of the library image: every GPU that
// loads libhplai holds its 4 MiB until the process exits (beside the 8 MiB of
// the leaf diagonal LU, getrf.cu).  It covers orders
// up to kNoAllocMaxN (ceil(n/2048) * n doubles).  All calls share it.
// ---------------------------------------------------------------------------
constexpr int kNoAllocMaxN = 32768;
constexpr size_t kNoAllocScratchDoubles =
	static_cast<size_t>((kNoAllocMaxN + GEMV_COLS - 1) / GEMV_COLS) * kNoAllocMaxN;
static __device__ __align__(256) double g_gemv_noalloc_scratch[kNoAllocScratchDoubles];

namespace {
std::mutex g_noalloc_mu;
constexpr int kMaxDevices = 64;
void *g_noalloc_addr[kMaxDevices] = {};
} // namespace

// Device address of the scratch array on the current device.  In host code
// the array's name is only a host-side handle, so the address is looked up
// once per device (with that device current) and cached.
static int noalloc_scratch(void **out)
{
	int dev = 0;
	HPLAI_CUDA_TRY(cudaGetDevice(&dev));
	if (dev < 0 || dev >= kMaxDevices) return HPLAI_EUNSUPPORTED;
	std::lock_guard<std::mutex> lk(g_noalloc_mu);
	if (!g_noalloc_addr[dev]) {
		void *p = nullptr;
		const cudaError_t e = cudaGetSymbolAddress(&p, g_gemv_noalloc_scratch);
		if (e != cudaSuccess) {
			set_last_cuda_error(e, "cudaGetSymbolAddress(g_gemv_noalloc_scratch)", __FILE__, __LINE__);
			return HPLAI_ECUDA;
		}
		g_noalloc_addr[dev] = p;
	}
	*out = g_noalloc_addr[dev];
	return HPLAI_OK;
}

} // namespace hplai

extern "C" size_t hplai_otf_gemv_workspace(int n) { return hplai::otf_gemv_workspace(n); }

extern "C" int hplai_otf_gemv(int n, double alpha, const double *x, double beta, double *y, uint64_t seed,
	const double *diag, void *work, size_t work_bytes, void *stream)
{
	if (n <= 0 || !x || !y || !diag || !work) return HPLAI_EINVAL;
	return hplai::launch_otf_gemv(n, alpha, x, beta, y, seed, diag, work, work_bytes, static_cast<cudaStream_t>(stream));
}

extern "C" int hplai_otf_gemv_block(int64_t n, int mb, int nb, double alpha, const double *x, double *y,
	uint64_t state00, void *work, size_t work_bytes, void *stream)
{
	if (n <= 0 || mb < 0 || nb < 0 || !x || !y || !work) return HPLAI_EINVAL;
	return hplai::launch_otf_gemv_block(n, mb, nb, alpha, x, y, state00, work, work_bytes,
		static_cast<cudaStream_t>(stream));
}

extern "C" size_t hplai_trsv_workspace(int n) { return hplai::trsv_workspace(n); }

extern "C" int hplai_trsv_lower(int n, const float *a, int64_t lda, double *x, void *work, size_t work_bytes,
	void *stream)
{
	if (n <= 0 || !a || !x || lda < n) return HPLAI_EINVAL;
	return hplai::launch_trsv(true, n, a, lda, x, work, work_bytes, static_cast<cudaStream_t>(stream));
}

extern "C" int hplai_trsv_upper(int n, const float *a, int64_t lda, double *x, void *work, size_t work_bytes,
	void *stream)
{
	if (n <= 0 || !a || !x || lda < n) return HPLAI_EINVAL;
	return hplai::launch_trsv(false, n, a, lda, x, work, work_bytes, static_cast<cudaStream_t>(stream));
}

extern "C" int hplai_infnorm(int n, const double *x, double *out, void *stream)
{
	if (n < 0 || (!x && n) || !out) return HPLAI_EINVAL;
	return hplai::launch_infnorm(n, x, out, static_cast<cudaStream_t>(stream));
}

extern "C" size_t hplai_panel_check_workspace(int n)
{
	return hplai::panel_check_workspace(n);
}

extern "C" int hplai_panel_check(int n, const float *a, int64_t lda, double *sigs, void *work, size_t work_bytes,
	void *stream)
{
	if (n < 0 || !sigs || (n > 0 && (!a || lda < n || !work))) return HPLAI_EINVAL;
	if (n > 0 && work_bytes < hplai::panel_check_workspace(n)) {
		hplai::set_last_error_message("hplai_panel_check: work is smaller than hplai_panel_check_workspace(n)");
		return HPLAI_EINVAL;
	}
	return hplai::launch_panel_check(n, a, lda, sigs, work, work_bytes, static_cast<cudaStream_t>(stream));
}

extern "C" int hplai_otf_gemv_noalloc(int n, double alpha, const double *x, double beta, double *y, uint64_t seed,
	const double *diag, void *stream)
{
	if (n <= 0 || !x || !y || !diag) return HPLAI_EINVAL;
	if (n > hplai::kNoAllocMaxN) {
		hplai::set_last_error_message("hplai_otf_gemv_noalloc: n exceeds HPLAI_OTF_GEMV_NOALLOC_MAX_N (32768)");
		return HPLAI_EINVAL;
	}
	void *scratch = nullptr;
	HPLAI_TRY(hplai::noalloc_scratch(&scratch));
	// Every partial sum the fold reads is written by this call's first
	// kernel, so the shared array needs no clearing between calls.
	return hplai::launch_otf_gemv(n, alpha, x, beta, y, seed, diag, scratch,
		hplai::kNoAllocScratchDoubles * sizeof(double), static_cast<cudaStream_t>(stream));
}
