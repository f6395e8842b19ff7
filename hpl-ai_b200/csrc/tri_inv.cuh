// tri_inv.cuh -- inverses of 128 x 128 triangular blocks in shared memory: in
// FP64 for the triangular solves of the refinement (refine.cu, batched.cu),
// in FP32 for the panels (tcpanel.cu).
#pragma once

#include "common.cuh"

namespace hplai {

constexpr int kTriBlock = 128;
constexpr int kTriThreads = 256;

// Inverse of one 128 x 128 diagonal block in shared memory (256 threads), R =
// double or float.
// X (row-major, ld kInvLd) becomes T^{-1}, T = L_rr (unit lower) or U_rr^T
// (so X is the transpose of U_rr^{-1}), padded with the identity past `rows`.
// The FP32 factor entries convert exactly.
// The 16 x 16 diagonal blocks are inverted by substitution, one thread per
// row, in registers; then pairs of inverted blocks of h = 16, 32, 64 are
// joined, [A 0; B C]^{-1} = [A^{-1} 0; -C^{-1} B A^{-1}, C^{-1}], as two
// products whose zero triangles are skipped 16 rows (or a column group) at a
// time.  Threads take interleaved rows and columns, so that the operands of a
// warp are 16 neighbouring doubles or a broadcast.  Bound by shared-memory
// reads (two 64-bit ones per four multiply-adds of a product) after the one
// latency of loading the block.  The diagonal blocks of both factors of
// n = 9600: 420 us as one substitution thread per column, 42 us so.
constexpr int kInvLd = kTriBlock + 1;
constexpr int kInvLdW = kTriBlock / 2 + 1;
template <typename R>
constexpr size_t kInvSmem = sizeof(R) * (static_cast<size_t>(kTriBlock) * kInvLd + kTriBlock / 2 * kInvLdW + kTriBlock);

template <typename R, int H>
__device__ __forceinline__ void invert_join(R *X, R *W)
{
	constexpr int TI = 16, NI = H / TI;    // rows ti + 16 a
	constexpr int TJ = H / 4, NJ = 4;      // columns tj + TJ b
	constexpr int per = TI * TJ;           // threads of one pair
	const int t = threadIdx.x;
	const int o = (t / per) * 2 * H;
	const int ti = t % TI, tj = (t % per) / TI;
	R *Wp = W + (t / per) * H;        // pair's columns in W (row i at Wp + i * kInvLdW)
	const R *A = X + o * kInvLd + o, *B = X + (o + H) * kInvLd + o, *C = B + H;
	R acc[NI][NJ];
#pragma unroll
	for (int a = 0; a < NI; ++a)
#pragma unroll
		for (int b = 0; b < NJ; ++b) acc[a][b] = R(0);
	// W = B A^{-1}: column j takes k >= j
#pragma unroll
	for (int s = 0; s < NJ; ++s) {
#pragma unroll 4
		for (int kk = 0; kk < TJ; ++kk) {
			const int k = s * TJ + kk;
			R bv[NI];
#pragma unroll
			for (int a = 0; a < NI; ++a) bv[a] = B[(ti + TI * a) * kInvLd + k];
#pragma unroll
			for (int b = 0; b <= s; ++b) {
				const R av = A[k * kInvLd + tj + TJ * b];
#pragma unroll
				for (int a = 0; a < NI; ++a) acc[a][b] = fma(bv[a], av, acc[a][b]);
			}
		}
	}
#pragma unroll
	for (int a = 0; a < NI; ++a)
#pragma unroll
		for (int b = 0; b < NJ; ++b) {
			Wp[(ti + TI * a) * kInvLdW + tj + TJ * b] = acc[a][b];
			acc[a][b] = R(0);
		}
	__syncthreads();
	// B <- -C^{-1} W: row i takes k <= i
#pragma unroll
	for (int s = 0; s < NI; ++s) {
#pragma unroll 4
		for (int kk = 0; kk < TI; ++kk) {
			const int k = s * TI + kk;
			R wv[NJ];
#pragma unroll
			for (int b = 0; b < NJ; ++b) wv[b] = Wp[k * kInvLdW + tj + TJ * b];
#pragma unroll
			for (int a = s; a < NI; ++a) {
				const R cv = C[(ti + TI * a) * kInvLd + k];
#pragma unroll
				for (int b = 0; b < NJ; ++b) acc[a][b] = fma(-cv, wv[b], acc[a][b]);
			}
		}
	}
	R *Bo = X + (o + H) * kInvLd + o;
#pragma unroll
	for (int a = 0; a < NI; ++a)
#pragma unroll
		for (int b = 0; b < NJ; ++b) Bo[(ti + TI * a) * kInvLd + tj + TJ * b] = acc[a][b];
	__syncthreads();
}

// smem: kInvSmem<R> bytes.  Ends with a barrier.
template <typename R>
__device__ __noinline__ void invert_block(R *smem, const float *__restrict__ a, int64_t lda, int r0, int rows,
	bool upper)
{
	R *X = smem, *W = X + kTriBlock * kInvLd, *rd = W + kTriBlock / 2 * kInvLdW;
	const int t = threadIdx.x;
	// T[i][j] from the stored block, line l (a column), place s in it
	auto put = [&](int l, int s, float f) {
		const int i = upper ? l : s, j = upper ? s : l;
		const bool in = i < rows && j < rows && (upper ? j <= i : j < i);
		X[i * kInvLd + j] = in ? static_cast<R>(f) : (i == j ? R(1) : R(0));
	};
	// every load of the block in flight at once: the latency of memory is paid
	// once and not once per row of threads
	if (rows == kTriBlock && (reinterpret_cast<uintptr_t>(a) & 15u) == 0 && (lda & 3) == 0) {
		const int s = (t % 32) * 4, l0 = t / 32;
		const float *src = a + static_cast<int64_t>(r0 + l0) * lda + r0 + s;
		float4 f[16];
#pragma unroll
		for (int q = 0; q < 16; ++q) f[q] = __ldcg(reinterpret_cast<const float4 *>(src + 8 * q * lda));
#pragma unroll
		for (int q = 0; q < 16; ++q) {
			put(l0 + 8 * q, s, f[q].x);
			put(l0 + 8 * q, s + 1, f[q].y);
			put(l0 + 8 * q, s + 2, f[q].z);
			put(l0 + 8 * q, s + 3, f[q].w);
		}
	} else {
		const int s = t % kTriBlock, l0 = t / kTriBlock;
#pragma unroll 1
		for (int h = 0; h < 4; ++h) {
			float f[16] = {};
			if (32 * h < rows) {
#pragma unroll
				for (int q = 0; q < 16; ++q) {
					const int l = min(l0 + 2 * (16 * h + q), rows - 1);   // put() drops what is past the last
					f[q] = __ldcg(&a[static_cast<int64_t>(r0 + l) * lda + r0 + min(s, rows - 1)]);
				}
			}
#pragma unroll
			for (int q = 0; q < 16; ++q) put(l0 + 2 * (16 * h + q), s, f[q]);
		}
	}
	__syncthreads();
	// v / d is the product with the rounded reciprocal, corrected once by the exact
	// remainder (Markstein, IBM J. Res. Dev. 34, 1990), which shortens the chain of 16
	// steps (a batch of 512 systems 35.8 ms by divisions, 35.3 so).  Where an entry of
	// the diagonal is tiny, huge, infinite or NaN the block divides: a zero over it
	// stays a zero.
	bool ordinary = true;
	if (upper && t < kTriBlock) {
		const R d = X[t * kInvLd + t];
		rd[t] = R(1) / d;
		ordinary = fabs(d) >= R(0x1p-60) && fabs(d) <= R(0x1p+60);
	}
	ordinary = __syncthreads_and(ordinary) != 0;
	R v[16];
	const int b0 = (t / 16) * 16, c = t % 16;
	if (t < kTriBlock) {
		// row c of the block's inverse, from the last column down
#pragma unroll
		for (int i = 0; i < 16; ++i) v[i] = (i == c) ? R(1) : R(0);
#pragma unroll
		for (int j = 15; j >= 0; --j) {
			if (upper) {
				const R d = X[(b0 + j) * kInvLd + b0 + j], y = rd[b0 + j], q = v[j] * y;
				v[j] = ordinary ? fma(fma(-d, q, v[j]), y, q) : v[j] / d;
			}
#pragma unroll
			for (int i = 0; i < j; ++i) v[i] = fma(-X[(b0 + j) * kInvLd + b0 + i], v[j], v[i]);
		}
	}
	__syncthreads();
	if (t < kTriBlock) {
#pragma unroll
		for (int i = 0; i < 16; ++i) X[(b0 + c) * kInvLd + b0 + i] = v[i];
	}
	__syncthreads();
	// rows past `rows` are the identity's: nothing to join there
	if (rows > 16) invert_join<R, 16>(X, W);
	if (rows > 32) invert_join<R, 32>(X, W);
	if (rows > 64) invert_join<R, 64>(X, W);
}

} // namespace hplai
