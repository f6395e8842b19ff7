// panel.cu -- FP32 panel factorisation kernels for the blocked no-pivot LU.
//
//  trsm_kernel      : L panel  A_col <- A_col * U^{-1}, plus its FP16 copy
//                     (update_left_panels + convert_left_panels, panel_trf.hpp:143-157,182-207)
//                     U panel  A_row <- L^{-1} * A_row, plus its FP16 copy, as the
//                     same solve on the transpose
//                     (update_right_panels + convert_right_panels, panel_trf.hpp:158-171,208-233)
//
// Every element receives its updates a_ij <- fma(-l_ik, u_kj, a_ij) in
// increasing k, and the multipliers are formed as a_ik * (1/u_kk), which
// is exactly the operation sequence of the reference's unblocked kernel and
// of netlib strsm (getrf_nopiv.hpp:33-44), so these kernels reproduce a
// sequential FP32 factorisation bit for bit whatever their blocking.
#include "common.cuh"
#include "internal.h"

namespace hplai {


// ---------------------------------------------------------------------------
// Panel TRSM + FP16 copy, one kernel for both panels.
//
// X (m x b) <- X * T^{-1} with T upper triangular (b x b).
//   L panel (update_left_panels):  X = A_col (column-major, X[r][j] at
//            a[j*lda + r]), T = U11 (T[p][j] at t[j*ldt + p]), non-unit.
//   U panel (update_right_panels, UPANEL): L^{-1} A_row = (A_row^T L^{-T})^T, so
//            X = A_row^T (row-major, X[r][j] at a[r*lda + j]) and T = L11^T
//            (T[p][j] = L[j][p] at t[p*ldt + j]), unit diagonal.
// Element (r, j) receives x -= T[p][j] * x[r][p] for p = 0..j-1 in
// increasing p, then x *= 1/T[j][j] when non-unit: netlib strsm's order for
// both (R,U,N,N) and (L,L,N,U), so the result is bit-exact with it.
// hc[(row0 + r)*ldh + j] = half(scale * X[r][j]) in both cases (the L copy is
// row-major; the U copy stores column j of U as row j).
//
// Bound by the chain of 16-column solves, and by FP32 issue and the operands'
// shared-memory reads in the products.  A CTA owns 32 RL rows; a thread holds RL rows (lane,
// lane + 32) of 16 columns (its warp's) of a block of 16 columns per warp in registers.
// Per block: the products with the columns solved before (X and T in chunks
// of 32 p through two or three cp.async stages), then the block's own triangle 16
// columns at a time -- the owning warp solves them in registers and publishes
// them, every later warp applies them (one barrier per 16 columns).  8200 rows,
// b = 512: 124 us a panel (270 with rows staged in shared memory and 4 x 4
// products, two shared-memory reads per four FMAs).
// ---------------------------------------------------------------------------
constexpr int kMicro = 16;
constexpr int kKC = 32;           // p per chunk
constexpr int kLdP = kKC + 4;     // chunk rows that run along p

// NW warps: columns in blocks of 16 per warp, 32 RL rows.
template <int NW, int RL, bool UPANEL>
struct Trsm {
	static constexpr int threads = 32 * NW;
	static constexpr int TB = kMicro * NW;
	static constexpr int R = 32 * RL;
	static constexpr int STAGES = NW == 8 ? 3 : 2;   // two, where three CTAs share an SM
	static constexpr int LDTRI = TB + 4;
	static constexpr int LDX = UPANEL ? kLdP : R + 4;        // X chunk: [r][p] or [p][r]
	static constexpr int LDT = UPANEL ? LDTRI : kLdP;        // T chunk: [p][c] or [c][p]
	static constexpr int XC = (UPANEL ? R : kKC) * LDX;
	static constexpr int TC = (UPANEL ? kKC : TB) * LDT;
	// the chunks belong to the blocks after the first
	static constexpr size_t bytes(int b)
	{
		return sizeof(float) * (TB * LDTRI + TB + 2 * kMicro * R + (b > TB ? STAGES * static_cast<size_t>(XC + TC) : 0));
	}
};

// lines x len floats, line l at src + l * lds, to dst + l * ldd; lines from
// nl on and elements from ne on are zero.
template <int THREADS>
__device__ __forceinline__ void stage_lines(float *dst, int ldd, const float *src, int64_t lds, int lines, int len,
	int nl, int ne, bool vec)
{
	if (vec) {
		const int g4 = len / 4;
		for (int e = threadIdx.x; e < lines * g4; e += THREADS) {
			const int l = e / g4, g = (e % g4) * 4;
			int bytes = l < nl ? (ne - g) * 4 : 0;
			bytes = bytes < 0 ? 0 : (bytes > 16 ? 16 : bytes);
			const float *p = src + (bytes ? static_cast<int64_t>(l) * lds + g : 0);
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + l * ldd + g)), "l"(p),
				"r"(bytes) : "memory");
		}
	} else {
		for (int e = threadIdx.x; e < lines * len; e += THREADS) {
			const int l = e / len, g = e % len;
			if (l < nl && g < ne)
				dst[l * ldd + g] = __ldcg(src + static_cast<int64_t>(l) * lds + g);
			else
				dst[l * ldd + g] = 0.f;
		}
	}
}

template <int NW, int RL, bool UPANEL>
__device__ __forceinline__ void trsm_rows(float *sm, int m, int b, const float *__restrict__ t, int64_t ldt, float *a,
	int64_t lda, __half *__restrict__ hc, int64_t ldh, float scale, int vec_x, int vec_t)
{
	using S = Trsm<NW, RL, UPANEL>;
	constexpr int R = S::R, TB = S::TB, LDTRI = S::LDTRI, THREADS = S::threads, STAGES = S::STAGES;
	constexpr bool UNIT = UPANEL;   // L11^T has a unit diagonal
	float *tri = sm;                      // tri[i * LDTRI + j] = T[j0 + i][j0 + j]
	float *inv = tri + TB * LDTRI;
	float *pub = inv + TB;               // [2][16][R]
	float *chunks = pub + 2 * kMicro * R; // STAGES x (X chunk, T chunk)
	const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
	const int row0 = blockIdx.x * R, rows = min(R, m - row0);
	const int e0 = kMicro * wp;
	for (int j0 = 0; j0 < b; j0 += TB) {
		const int jw = min(TB, b - j0), nc = j0 / kKC;
		auto stage = [&](int q) {
			if (q < nc) {
				float *xc = chunks + (q % STAGES) * (S::XC + S::TC), *tc = xc + S::XC;
				const int p0 = q * kKC;
				if (UPANEL) {
					stage_lines<THREADS>(xc, S::LDX, a + static_cast<int64_t>(row0) * lda + p0, lda, R, kKC, rows, kKC, vec_x != 0);
					stage_lines<THREADS>(tc, S::LDT, t + static_cast<int64_t>(p0) * ldt + j0, ldt, kKC, TB, kKC, jw, vec_t != 0);
				} else {
					stage_lines<THREADS>(xc, S::LDX, a + static_cast<int64_t>(p0) * lda + row0, lda, kKC, R, kKC, rows, vec_x != 0);
					stage_lines<THREADS>(tc, S::LDT, t + static_cast<int64_t>(j0) * ldt + p0, ldt, TB, kKC, jw, kKC, vec_t != 0);
				}
			}
			asm volatile("cp.async.commit_group;" ::: "memory");
		};
		for (int q = 0; q < STAGES - 1; ++q) stage(q);
		// this block's triangle (rows and columns past jw zero) and columns; the
		// loads of each are all in flight together
		if (UPANEL) {
			stage_lines<THREADS>(tri, LDTRI, t + static_cast<int64_t>(j0) * ldt + j0, ldt, TB, TB, jw, jw, vec_t != 0);
			asm volatile("cp.async.commit_group;" ::: "memory");
		} else if (vec_t && jw % 4 == 0) {
			const int c = tid % 32, r4 = (tid / 32) * 4;   // lanes along the columns: rows of T without bank conflicts
			constexpr int G = TB / 32;   // groups of 32 columns
			float4 f[4 * G];
#pragma unroll
			for (int q = 0; q < 4 * G; ++q) {
				const int cc = c + 32 * (q % G), rr = r4 + 4 * NW * (q / G);
				f[q] = make_float4(0.f, 0.f, 0.f, 0.f);
				if (cc < jw && rr < jw)
					f[q] = __ldcg(reinterpret_cast<const float4 *>(t + static_cast<int64_t>(j0 + cc) * ldt + j0 + rr));
			}
#pragma unroll
			for (int q = 0; q < 4 * G; ++q) {
				const int cc = c + 32 * (q % G), rr = r4 + 4 * NW * (q / G);
				tri[rr * LDTRI + cc] = f[q].x;
				tri[(rr + 1) * LDTRI + cc] = f[q].y;
				tri[(rr + 2) * LDTRI + cc] = f[q].z;
				tri[(rr + 3) * LDTRI + cc] = f[q].w;
			}
		} else {
#pragma unroll 16
			for (int e = tid; e < TB * TB; e += THREADS) {
				const int p = e % TB, j = e / TB;
				tri[p * LDTRI + j] = (p < jw && j < jw) ? __ldcg(t + static_cast<int64_t>(j0 + j) * ldt + j0 + p) : 0.f;
			}
		}
		float x[RL][kMicro];
		const bool wide = UPANEL && vec_x && e0 + kMicro <= jw;   // this thread's 16 elements as four float4
#pragma unroll
		for (int r = 0; r < RL; ++r) {
			const int row = lane + 32 * r;
			const float *src = UPANEL ? a + static_cast<int64_t>(row0 + row) * lda + j0 + e0
			                          : a + static_cast<int64_t>(j0 + e0) * lda + row0 + row;
			if (wide) {
#pragma unroll
				for (int g = 0; g < kMicro / 4; ++g) {
					float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
					if (row < rows) v = __ldcg(reinterpret_cast<const float4 *>(src + 4 * g));
					x[r][4 * g] = v.x;
					x[r][4 * g + 1] = v.y;
					x[r][4 * g + 2] = v.z;
					x[r][4 * g + 3] = v.w;
				}
			} else {
#pragma unroll
				for (int c = 0; c < kMicro; ++c)
					x[r][c] = (row < rows && e0 + c < jw) ? __ldcg(src + (UPANEL ? c : static_cast<int64_t>(c) * lda)) : 0.f;
			}
		}
		for (int q = 0; q < nc; ++q) {
			asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
			__syncthreads();   // chunk q is here; everyone is done with the one before it
			stage(q + STAGES - 1);
			const float *xc = chunks + (q % STAGES) * (S::XC + S::TC), *tc = xc + S::XC;
#pragma unroll 2
			for (int p = 0; p < kKC; p += 4) {
				float xp[RL][4];
#pragma unroll
				for (int r = 0; r < RL; ++r) {
					if (UPANEL) {
						const float4 v = *reinterpret_cast<const float4 *>(xc + (lane + 32 * r) * S::LDX + p);
						xp[r][0] = v.x;
						xp[r][1] = v.y;
						xp[r][2] = v.z;
						xp[r][3] = v.w;
					} else {
#pragma unroll
						for (int k = 0; k < 4; ++k) xp[r][k] = xc[(p + k) * S::LDX + lane + 32 * r];
					}
				}
				if (UPANEL) {
#pragma unroll
					for (int k = 0; k < 4; ++k)
#pragma unroll
						for (int g = 0; g < kMicro / 4; ++g) {
							const float4 v = *reinterpret_cast<const float4 *>(tc + (p + k) * S::LDT + e0 + 4 * g);
#pragma unroll
							for (int r = 0; r < RL; ++r) {
								x[r][4 * g] = fmaf(-v.x, xp[r][k], x[r][4 * g]);
								x[r][4 * g + 1] = fmaf(-v.y, xp[r][k], x[r][4 * g + 1]);
								x[r][4 * g + 2] = fmaf(-v.z, xp[r][k], x[r][4 * g + 2]);
								x[r][4 * g + 3] = fmaf(-v.w, xp[r][k], x[r][4 * g + 3]);
							}
						}
				} else {
#pragma unroll
					for (int c = 0; c < kMicro; ++c) {
						const float4 v = *reinterpret_cast<const float4 *>(tc + (e0 + c) * S::LDT + p);
#pragma unroll
						for (int r = 0; r < RL; ++r) {
							x[r][c] = fmaf(-v.x, xp[r][0], x[r][c]);
							x[r][c] = fmaf(-v.y, xp[r][1], x[r][c]);
							x[r][c] = fmaf(-v.z, xp[r][2], x[r][c]);
							x[r][c] = fmaf(-v.w, xp[r][3], x[r][c]);
						}
					}
				}
			}
		}
		asm volatile("cp.async.wait_all;" ::: "memory");
		__syncthreads();   // the triangle is here
		if (!UNIT && tid < TB) inv[tid] = tid < jw ? 1.0f / tri[tid * LDTRI + tid] : 0.f;
		if (!UNIT) __syncthreads();
		const int nmicro = (jw + kMicro - 1) / kMicro;
		for (int oi = 0; oi < nmicro; ++oi) {
			float *const pb = pub + (oi & 1) * kMicro * R + lane;
			if (wp == oi) {
#pragma unroll
				for (int li = 0; li < kMicro; ++li) {
					const int i = kMicro * oi + li;
#pragma unroll
					for (int r = 0; r < RL; ++r) {
						if (!UNIT) x[r][li] *= inv[i];
						pb[li * R + 32 * r] = x[r][li];
					}
					const float4 *row = reinterpret_cast<const float4 *>(tri + i * LDTRI + e0);
#pragma unroll
					for (int g = (li + 1) / 4; g < kMicro / 4; ++g) {
						const float4 v = row[g];
						const float tv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
						for (int h = 0; h < 4; ++h) {
							const int c = 4 * g + h;
							if (c <= li) continue;
#pragma unroll
							for (int r = 0; r < RL; ++r) x[r][c] = fmaf(-tv[h], x[r][li], x[r][c]);
						}
					}
				}
			}
			__syncthreads();
			if (wp > oi) {
#pragma unroll 4
				for (int li = 0; li < kMicro; ++li) {
					float xi[RL];
#pragma unroll
					for (int r = 0; r < RL; ++r) xi[r] = pb[li * R + 32 * r];
					const float4 *row = reinterpret_cast<const float4 *>(tri + (kMicro * oi + li) * LDTRI + e0);
#pragma unroll
					for (int g = 0; g < kMicro / 4; ++g) {
						const float4 v = row[g];
#pragma unroll
						for (int r = 0; r < RL; ++r) {
							x[r][4 * g] = fmaf(-v.x, xi[r], x[r][4 * g]);
							x[r][4 * g + 1] = fmaf(-v.y, xi[r], x[r][4 * g + 1]);
							x[r][4 * g + 2] = fmaf(-v.z, xi[r], x[r][4 * g + 2]);
							x[r][4 * g + 3] = fmaf(-v.w, xi[r], x[r][4 * g + 3]);
						}
					}
				}
			}
		}
#pragma unroll
		for (int r = 0; r < RL; ++r) {
			const int row = lane + 32 * r;
			if (row >= rows) continue;
			float *dst = UPANEL ? a + static_cast<int64_t>(row0 + row) * lda + j0 + e0
			                    : a + static_cast<int64_t>(j0 + e0) * lda + row0 + row;
			if (wide) {
#pragma unroll
				for (int g = 0; g < kMicro / 4; ++g)
					*reinterpret_cast<float4 *>(dst + 4 * g) =
						make_float4(x[r][4 * g], x[r][4 * g + 1], x[r][4 * g + 2], x[r][4 * g + 3]);
			} else {
#pragma unroll
				for (int c = 0; c < kMicro; ++c)
					if (e0 + c < jw) dst[UPANEL ? c : static_cast<int64_t>(c) * lda] = x[r][c];
			}
			if (hc) {
				__half *o = hc + static_cast<int64_t>(row0 + row) * ldh + j0 + e0;
#pragma unroll
				for (int q = 0; q < kMicro / 8; ++q) {
					if (e0 + 8 * q + 8 <= jw) {
						// 8 halves, 16-byte aligned: hc is, ldh and the offset are multiples of 8
						__align__(16) __half h[8];
#pragma unroll
						for (int e = 0; e < 8; ++e) h[e] = __float2half_rn(scale * x[r][8 * q + e]);
						*reinterpret_cast<uint4 *>(o + 8 * q) = *reinterpret_cast<const uint4 *>(h);
					} else {
#pragma unroll
						for (int e = 0; e < 8; ++e)
							if (e0 + 8 * q + e < jw) o[8 * q + e] = __float2half_rn(scale * x[r][8 * q + e]);
					}
				}
			}
		}
		__syncthreads();   // X is in memory for the next block; the triangle is free
	}
}

template <int NW, int RL, bool UPANEL>
__global__ void __launch_bounds__(32 * NW) trsm_kernel(int m, int b, const float *__restrict__ t, int64_t ldt,
	float *a, int64_t lda, __half *__restrict__ hc, int64_t ldh, float scale, int vec_x, int vec_t)
{
	extern __shared__ __align__(16) float sm[];
	trsm_rows<NW, RL, UPANEL>(sm, m, b, t, ldt, a, lda, hc, ldh, scale, vec_x, vec_t);
}

// Both panels of a step in one launch (blockIdx.y = 0: L, 1: U), the
// triangles and panels in one matrix.
constexpr int kPairWarps = 8;
template <int RL>
__global__ void __launch_bounds__(32 * kPairWarps) trsm_pair_kernel(int rem, int b, const float *__restrict__ lu, float *acol,
	float *arow, int64_t lda, __half *__restrict__ lh, __half *__restrict__ uh, int64_t ldh, int vec)
{
	extern __shared__ __align__(16) float sm[];
	if (blockIdx.y == 0)
		trsm_rows<kPairWarps, RL, false>(sm, rem, b, lu, lda, acol, lda, lh, ldh, 1.0f, vec, vec);
	else
		trsm_rows<kPairWarps, RL, true>(sm, rem, b, lu, lda, arow, lda, uh, ldh, 1.0f, vec, vec);
}

template <int NW, int RL, bool UPANEL>
static int trsm_launch(int m, int b, const float *t, int64_t ldt, float *a, int64_t lda, uint16_t *hc, int64_t ldh,
	float scale, cudaStream_t st)
{
	using S = Trsm<NW, RL, UPANEL>;
	static DeviceOnce attr;
	HPLAI_TRY(attr.get([](int, int *) -> int {
		HPLAI_CUDA_TRY(cudaFuncSetAttribute(trsm_kernel<NW, RL, UPANEL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			static_cast<int>(S::bytes(1024))));
		return HPLAI_OK;
	}));
	auto vec = [](const float *p, int64_t ld) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && ld % 4 == 0 ? 1 : 0; };
	trsm_kernel<NW, RL, UPANEL><<<(m + 32 * RL - 1) / (32 * RL), 32 * NW, S::bytes(b), st>>>(m, b, t, ldt, a, lda,
		reinterpret_cast<__half *>(hc), ldh, scale, vec(a, lda), vec(t, ldt));
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

// 64 rows per CTA reuse each triangle read twice; below 74 such CTAs half the
// GPU would idle, and 32 rows per CTA are faster.  Eight warps have the shortest
// chain, but one such CTA fills an SM: past one wave of them (9472 rows) four
// warps, three CTAs an SM, are faster (L panel, four / eight warps: b = 128, 10000
// rows 29 / 35 us, 40000 61 / 87; b = 200, 40000 135 / 177; b = 512, 10000 211 / 238,
// 8200 157 / 123).  A narrower panel has no work for more warps than 16 columns
// each: b = 60, 40000 rows 24 / 49 us, b = 31 two / eight warps 14 / 40.
template <bool UPANEL>
static int trsm_pick(int m, int b, const float *t, int64_t ldt, float *a, int64_t lda, uint16_t *hc, int64_t ldh,
	float scale, cudaStream_t st)
{
	if (b <= 32) {
		if (m > 16000) return trsm_launch<2, 2, UPANEL>(m, b, t, ldt, a, lda, hc, ldh, scale, st);
		return trsm_launch<2, 1, UPANEL>(m, b, t, ldt, a, lda, hc, ldh, scale, st);
	}
	if (m > 64 * (b <= 64 ? 74 : 148)) return trsm_launch<4, 2, UPANEL>(m, b, t, ldt, a, lda, hc, ldh, scale, st);
	if (b <= 64) return trsm_launch<4, 1, UPANEL>(m, b, t, ldt, a, lda, hc, ldh, scale, st);
	if (m > 64 * 74) return trsm_launch<8, 2, UPANEL>(m, b, t, ldt, a, lda, hc, ldh, scale, st);
	return trsm_launch<8, 1, UPANEL>(m, b, t, ldt, a, lda, hc, ldh, scale, st);
}

static bool vec_ok(const uint16_t *hc, int64_t ldh)
{
	return !hc || ((reinterpret_cast<uintptr_t>(hc) & 15u) == 0 && ldh % 8 == 0);
}

int launch_trsm_right_upper(int m, int b, const float *u, int64_t ldu, float *a, int64_t lda, uint16_t *lh,
	int64_t ldh, float scale, cudaStream_t st)
{
	if (m <= 0) return HPLAI_OK;
	if (b <= 0 || b > 1024 || !vec_ok(lh, ldh)) return HPLAI_EINVAL;
	return trsm_pick<false>(m, b, u, ldu, a, lda, lh, ldh, scale, st);
}

int launch_trsm_left_lower(int b, int ncols, const float *l, int64_t ldl, float *a, int64_t lda, uint16_t *uh,
	int64_t ldh, float scale, cudaStream_t st)
{
	if (ncols <= 0) return HPLAI_OK;
	if (b <= 0 || b > 1024 || !vec_ok(uh, ldh)) return HPLAI_EINVAL;
	return trsm_pick<true>(ncols, b, l, ldl, a, lda, uh, ldh, scale, st);
}

template <int RL>
static int pair_launch(int rem, int b, const float *diag, float *acol, float *arow, int64_t lda, uint16_t *lh,
	uint16_t *uh, int64_t ldh, cudaStream_t st)
{
	using SL = Trsm<kPairWarps, RL, false>;
	using SU = Trsm<kPairWarps, RL, true>;
	auto bytes = [](int w) { return SL::bytes(w) > SU::bytes(w) ? SL::bytes(w) : SU::bytes(w); };
	static DeviceOnce attr;
	HPLAI_TRY(attr.get([](int, int *) -> int {
		HPLAI_CUDA_TRY(cudaFuncSetAttribute(trsm_pair_kernel<RL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			static_cast<int>(SL::bytes(1024) > SU::bytes(1024) ? SL::bytes(1024) : SU::bytes(1024))));
		return HPLAI_OK;
	}));
	const int vec = (reinterpret_cast<uintptr_t>(diag) & 15u) == 0 && lda % 4 == 0 && b % 4 == 0 ? 1 : 0;
	trsm_pair_kernel<RL><<<dim3((rem + 32 * RL - 1) / (32 * RL), 2), 32 * kPairWarps, bytes(b), st>>>(rem, b, diag, acol, arow,
		lda, reinterpret_cast<__half *>(lh), reinterpret_cast<__half *>(uh), ldh, vec);
	count_launches();
	HPLAI_CUDA_TRY(cudaGetLastError());
	return HPLAI_OK;
}

int launch_trsm_pair(int rem, int b, const float *diag, float *acol, float *arow, int64_t lda, uint16_t *lh,
	uint16_t *uh, int64_t ldh, cudaStream_t st)
{
	if (rem <= 0) return HPLAI_OK;
	if (b <= 0 || b > 1024 || !vec_ok(lh, ldh) || !vec_ok(uh, ldh)) return HPLAI_EINVAL;
	if (rem > 64 * 74) return pair_launch<2>(rem, b, diag, acol, arow, lda, lh, uh, ldh, st);
	return pair_launch<1>(rem, b, diag, acol, arow, lda, lh, uh, ldh, st);
}

} // namespace hplai

extern "C" int hplai_getrf_nopiv(int b, float *a, int64_t lda, void *stream)
{
	if (!a || lda < b) return HPLAI_EINVAL;
	return hplai::launch_getrf(b, a, lda, static_cast<cudaStream_t>(stream));
}

extern "C" int hplai_trsm_right_upper(int m, int b, const float *u, int64_t ldu, float *a, int64_t lda,
	uint16_t *lh, int64_t ldh, float scale, void *stream)
{
	if (m < 0 || !u || !a || ldu < b || lda < m || (lh && ldh < b)) return HPLAI_EINVAL;
	return hplai::launch_trsm_right_upper(m, b, u, ldu, a, lda, lh, ldh, scale, static_cast<cudaStream_t>(stream));
}

extern "C" int hplai_trsm_left_lower(int b, int ncols, const float *l, int64_t ldl, float *a, int64_t lda,
	uint16_t *uh, int64_t ldh, float scale, void *stream)
{
	if (ncols < 0 || !l || !a || ldl < b || lda < b || (uh && ldh < b)) return HPLAI_EINVAL;
	return hplai::launch_trsm_left_lower(b, ncols, l, ldl, a, lda, uh, ldh, scale, static_cast<cudaStream_t>(stream));
}
