// tile.cuh -- 32 x 32 FP32 tiles in shared memory and the steps of the
// unblocked no-pivot LU on them, a team of four warps per tile (getrf.cu,
// batched.cu).
//
// Each element receives a_ij <- fmaf(-l_ik, u_kj, a_ij) in increasing k,
// multipliers are a_ik * (1/u_kk) and the U tiles use the same unit-lower
// sequence as netlib strsm, so any blocking built from these operations gives
// the bits of the sequential factorisation (getrf_nopiv.hpp:33-44).
//
// A tile's chain of 32 dependent steps is bound by the latency of a step and
// by the rate at which one warp issues (about an instruction in two cycles),
// so the work is divided among four warps, each on its own sub-partition, in
// a way that needs no exchange between warps at a step of the chain:
//  - the factorisation has a row per lane in every warp; warp w keeps the
//    columns w, w + 4, ..., and the four columns of the current panel are kept
//    by all four warps, each carrying out the panel's steps for itself; the
//    next panel's columns go through shared memory, one barrier per four
//    steps;
//  - a solve has eight rows (columns) per warp, four lanes each, a lane with
//    every fourth element; the four lanes share a step by shuffle.
// (One warp per tile: 7,700 cycles for a factorisation, 2,700 to 3,600 for a
// solve, and half as much again beside seven busy warps.)
#pragma once

#include "common.cuh"

namespace hplai {
namespace tile {

constexpr int T = 32;
constexpr int kTeamWarps = 4;
constexpr int kTeam = 32 * kTeamWarps;
constexpr int kPanel = kTeamWarps;            // columns of a panel: one of each warp's
constexpr int kOwn = T / kTeamWarps;          // columns a warp keeps

// A staged tile: column-major, element (i, j) at t[j * kLd + i]; columns of 16
// bytes so that cp.async can fill it.  All lanes reading one element is a
// broadcast, a column of 32 conflict-free.  The solves read a few elements past
// a line (and leave them unused), hence the tail.
constexpr int kLd = 36;
constexpr int kTileFloats = T * kLd + 16;

// A team: its four warps' threads 0 .. 127 and its named barrier.
struct Team {
	int tid, lane, warp, bar;
	__device__ __forceinline__ void sync() const
	{
		asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(kTeam) : "memory");
	}
};

// Tile (rows r0.., cols c0..) -> t, rows >= rv and columns >= cv zero.
// vec: a, lda and r0 allow 16-byte copies (cp.async.cg, L2 only); otherwise
// 4-byte loads through L2.  `threads` threads, this one `tid`; the caller
// waits with stage_wait() and a barrier of those threads.
__device__ __forceinline__ void stage_tile(float *t, const float *a, int64_t lda, int r0, int c0, int rv, int cv,
	bool vec, int tid, int threads)
{
	if (vec) {
		for (int e = tid; e < T * T / 4; e += threads) {
			const int j = e >> 3, g = (e & 7) * 4;
			int bytes = (j < cv) ? (rv - g) * 4 : 0;
			bytes = bytes < 0 ? 0 : (bytes > 16 ? 16 : bytes);
			const float *src = a + static_cast<int64_t>(c0 + (j < cv ? j : 0)) * lda + r0 + (bytes ? g : 0);
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(t + j * kLd + g)), "l"(src),
				"r"(bytes) : "memory");
		}
	} else {
#pragma unroll 8
		for (int e = tid; e < T * T; e += threads) {
			const int i = e & 31, j = e >> 5;
			t[j * kLd + i] = (i < rv && j < cv) ? __ldcg(&a[static_cast<int64_t>(c0 + j) * lda + r0 + i]) : 0.f;
		}
	}
}

__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void store_tile(const float *t, float *a, int64_t lda, int r0, int c0, int rv, int cv,
	int tid, int threads)
{
#pragma unroll 8
	for (int e = tid; e < T * T; e += threads) {
		const int i = e & 31, j = e >> 5;
		if (i < rv && j < cv) a[static_cast<int64_t>(c0 + j) * lda + r0 + i] = t[j * kLd + i];
	}
}

// Exchange buffer of a team: a panel's columns, twice.
constexpr int kXchFloats = 2 * kPanel * kLd;

// Panels p0 .. p1 - 1 of a factorisation, NO columns of this warp after the
// current one (own[0]).  The chain from pivot to pivot is kept to reciprocal,
// multiply, multiply-add: every lane forms the next pivot itself from three
// values that were broadcast while the reciprocal was on its way, by the
// operations that its own lane applies, so the bits are the same.
template <int NO, bool FTZ>
__device__ __forceinline__ void factor_panels(const Team &tm, float (&own)[kOwn], float *d, float *dt, float *xch, int p0,
	int p1, float &least, float &most)
{
	const int lane = tm.lane;
#pragma unroll 1
	for (int p = p0; p < p1; ++p) {
		float *x = xch + (p & 1) * kPanel * kLd + lane;
		x[tm.warp * kLd] = own[0];
		tm.sync();
		float pv[kPanel];
#pragma unroll
		for (int j = 0; j < kPanel; ++j) pv[j] = x[j * kLd];
		const int k0 = kPanel * p;
		float pivot = __shfl_sync(0xffffffffu, pv[0], k0);
#pragma unroll
		for (int i = 0; i < kPanel; ++i) {
			const int k = k0 + i;
			const bool last = i + 1 == kPanel;
			float below = 0.f, right = 0.f, next = 0.f;
			if (!last) {
				below = __shfl_sync(0xffffffffu, pv[i], k + 1);
				right = __shfl_sync(0xffffffffu, pv[i + 1], k);
				next = __shfl_sync(0xffffffffu, pv[i + 1], k + 1);
			}
			float inv;
			if (FTZ) {
				least = fminf(least, fabsf(pivot));
				most = fmaxf(most, fabsf(pivot));
				asm("rcp.rn.ftz.f32 %0, %1;" : "=f"(inv) : "f"(pivot));
			} else {
				inv = 1.0f / pivot;
			}
			const float l = pv[i] * inv;
			if (!last) pivot = fmaf(-(below * inv), right, next);
			const bool active = lane > k;
			if (tm.warp == i) {
				const float e = active ? l : pv[i];
				d[k * kLd + lane] = e;
				dt[lane * kLd + k] = e;
			}
#pragma unroll
			for (int j = i + 1; j < kPanel; ++j) {
				const float u = j == i + 1 ? right : __shfl_sync(0xffffffffu, pv[j], k);
				if (active) pv[j] = fmaf(-l, u, pv[j]);
			}
#pragma unroll
			for (int m = 1; m <= NO; ++m) {
				const float t = fmaf(-l, __shfl_sync(0xffffffffu, own[m], k), own[m]);
				own[last ? m - 1 : m] = active ? t : own[m];
			}
		}
	}
}

// FTZ: the reciprocal flushes subnormal operands and results, which keeps it
// free of branches; for pivots whose reciprocal is a normal number both round
// to nearest, so the result is the same.  False (in every lane and warp: the
// pivots are the same) where one is not.
template <bool FTZ>
__device__ __noinline__ bool factor_team(const Team tm, const float *__restrict__ x, float *__restrict__ d,
	float *__restrict__ dt, float *__restrict__ xch, int kv)
{
	float own[kOwn];
#pragma unroll
	for (int m = 0; m < kOwn; ++m) {
		const int c = tm.warp + 4 * m;
		own[m] = tm.lane == c && c >= kv ? 1.0f : x[c * kLd + tm.lane];
	}
	float least = 1.0f, most = 1.0f;
	factor_panels<7, FTZ>(tm, own, d, dt, xch, 0, 4, least, most);
	factor_panels<3, FTZ>(tm, own, d, dt, xch, 4, 8, least, most);
	tm.sync();
	// 2^-126 .. 2^126: the pivots whose reciprocals are normal
	return !FTZ || (least >= 0x1p-126f && most <= 0x1p126f);
}

// Unblocked LU of the kv x kv tile x (padded to a whole tile with the
// identity); the result to d (column-major) and dt (row by row), neither x.
__device__ __forceinline__ void op_factor(const Team &tm, const float *x, float *d, float *dt, float *xch, int kv)
{
	if (!factor_team<true>(tm, x, d, dt, xch, kv)) factor_team<false>(tm, x, d, dt, xch, kv);
}

// Steps 4 g0 .. 4 g1 - 1 of a solve, NO elements of this lane after the
// current one (v[0]); line k of the triangle is tri[k * kLd ..].
template <int NO, bool LEFT>
__device__ __forceinline__ void solve_steps(float (&v)[kOwn], const float *tri, float *x, int row, int part, float inv,
	int g0, int g1)
{
	const int lane = threadIdx.x & 31;
#pragma unroll 1
	for (int g = g0; g < g1; ++g) {
		const float *line = tri + 4 * g * (kLd + 1) + part;
#pragma unroll
		for (int i = 0; i < 4; ++i, line += kLd) {
			const int k = 4 * g + i;
			const float mine = LEFT ? v[0] * __shfl_sync(0xffffffffu, inv, k) : v[0];
			const float e = __shfl_sync(0xffffffffu, mine, (lane & ~3) | i);
			if (part == i) x[LEFT ? k * kLd + row : row * kLd + k] = e;
			if (i < 3) {
				const float t = fmaf(-e, line[0], v[0]);
				if (part > i) v[0] = t;
			}
#pragma unroll
			for (int m = 1; m <= NO; ++m) v[i == 3 ? m - 1 : m] = fmaf(-e, line[4 * m], v[m]);
		}
	}
}

// The team's tile x, whole triangle tri: LEFT, x <- x U^{-1} with row k of U at
// tri[k * kLd ..]; else x <- L^{-1} x with column k of the unit L there.  A
// row of x (LEFT) or a column per four lanes.  Ends with the team's barrier.
template <bool LEFT>
__device__ __noinline__ void solve_team(const Team tm, float *__restrict__ x, const float *__restrict__ tri)
{
	const int row = 8 * tm.warp + (tm.lane >> 2), part = tm.lane & 3;
	float v[kOwn];
#pragma unroll
	for (int m = 0; m < kOwn; ++m) v[m] = x[LEFT ? (part + 4 * m) * kLd + row : row * kLd + part + 4 * m];
	const float inv = LEFT ? 1.0f / tri[tm.lane * kLd + tm.lane] : 0.f;   // 1/u_kk, lane k's
	__syncwarp();   // the rows of a warp are its own
	solve_steps<7, LEFT>(v, tri, x, row, part, inv, 0, 4);
	solve_steps<3, LEFT>(v, tri, x, row, part, inv, 4, 8);
	tm.sync();
}

// L tile x <- x U^{-1}, U row by row in dt.
__device__ __forceinline__ void op_solve_l(const Team &tm, float *x, const float *dt) { solve_team<true>(tm, x, dt); }

// U tile x <- L^{-1} x, L column by column in d.
__device__ __forceinline__ void op_solve_u(const Team &tm, float *x, const float *d) { solve_team<false>(tm, x, d); }

// Columns 8 warp .. 8 warp + 7 of x -= l u (K = T).  Lane (rg, cg) holds rows
// 4 rg .. 4 rg + 3 of two columns: per four k, four reads of l and two of u
// for 32 multiply-adds.  The caller's barrier follows.
static __device__ __noinline__ void op_update(const Team tm, float *__restrict__ x, const float *__restrict__ l,
	const float *__restrict__ u)
{
	constexpr int NC = 2;
	const int rg = tm.lane & 7, c0 = 8 * tm.warp + (tm.lane >> 3);
	float v[NC][4];
	float *xc = x + c0 * kLd + 4 * rg;
	const float *uc = u + c0 * kLd, *lr = l + 4 * rg;
#pragma unroll
	for (int c = 0; c < NC; ++c) {
		const float4 q = *reinterpret_cast<const float4 *>(xc + 4 * c * kLd);
		v[c][0] = q.x;
		v[c][1] = q.y;
		v[c][2] = q.z;
		v[c][3] = q.w;
	}
#pragma unroll 4
	for (int k = 0; k < T; k += 4) {
		float4 lk[4], uk[NC];
#pragma unroll
		for (int kk = 0; kk < 4; ++kk) lk[kk] = *reinterpret_cast<const float4 *>(lr + (k + kk) * kLd);
#pragma unroll
		for (int c = 0; c < NC; ++c) uk[c] = *reinterpret_cast<const float4 *>(uc + 4 * c * kLd + k);
#pragma unroll
		for (int kk = 0; kk < 4; ++kk)
#pragma unroll
			for (int c = 0; c < NC; ++c) {
				const float m = kk == 0 ? uk[c].x : kk == 1 ? uk[c].y : kk == 2 ? uk[c].z : uk[c].w;
				v[c][0] = fmaf(-lk[kk].x, m, v[c][0]);
				v[c][1] = fmaf(-lk[kk].y, m, v[c][1]);
				v[c][2] = fmaf(-lk[kk].z, m, v[c][2]);
				v[c][3] = fmaf(-lk[kk].w, m, v[c][3]);
			}
	}
#pragma unroll
	for (int c = 0; c < NC; ++c)
		*reinterpret_cast<float4 *>(xc + 4 * c * kLd) = make_float4(v[c][0], v[c][1], v[c][2], v[c][3]);
}

} // namespace tile
} // namespace hplai
