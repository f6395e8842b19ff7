// getrf.cu -- b x b diagonal block LU without pivoting, spread over the GPU.
//
// getrf_nopiv (getrf_nopiv.hpp:30-141) on the diagonal block of each step.
// The block is cut into 32 x 32 tiles that go through the steps of a
// right-looking LU:
//   step r < min(ti, tj):  X -= L(ti, r) U(r, tj)              (trailing update)
//   step r = ti = tj:      X <- LU of X                        (tile factor)
//   step r = tj < ti:      X <- X U(r, r)^{-1}                 (L tile)
//   step r = ti < tj:      X <- L(r, r)^{-1} X  (unit lower)   (U tile)
// A tile that another CTA needs travels through the workspace as tagged words
// (64 bits: an element and the launch's number with the tile's state, handed
// over or final), so that one load carries data and flag: no fence on the
// producer's side, no second round trip on the consumer's.
//
// What bounds it is the diagonal chain, b dependent pivots.  CTA 0 does nothing
// else, and the teams of the other CTAs own every tile that it does not need
// next.  At step r CTA 0 holds the factored tile (r, r), solves L(r+1, r) and
// U(r, r+1) (a team each) while its third team publishes (r, r), updates tile
// (r+1, r+1) and factors it, while the other two publish L(r+1, r) and
// U(r, r+1) and bring in the next step's inputs.  The chain through the
// workers -- (r, r) published, L(r+2, r) solved, tile (r+2, r+1) updated and
// handed back for step r+1 -- is kept to two hops through L2: one team owns
// both (e, e-2) and (e, e-1), and tile (e, e) comes back one update early, the
// last two being applied by CTA 0.  A worker team keeps its tiles in shared
// memory where they fit, so a trailing update reads only its two operands and
// writes nothing until the tile is final or handed over.
// A block within a factorisation, before (a tile per warp, the chain on one
// eight-warp CTA, progress words behind fences) / now: b = 60 29 / 16 us, 240
// 125 / 57, 512 257 / 108, 1024 517 / 226; through the leaf entry point, which
// waits for the status, 512 276 / 125.
// Every wait is on work the producer reaches without waiting on the waiter,
// so the dataflow always completes (all CTAs are resident: cooperative
// launch); every wait is bounded, and a timeout sets the status word and the
// team stops.
//
// Each element receives a_ij <- fmaf(-l_ik, u_kj, a_ij) in increasing k,
// multipliers are a_ik * (1/u_kk) and the U tiles use the same unit-lower
// sequence as netlib strsm: the operation sequence of a sequential FP32
// factorisation, so the result is bit for bit that of the reference's
// unblocked kernel with any blocking (getrf_nopiv.hpp:33-44).
#include "common.cuh"
#include "internal.h"
#include "tile.cuh"

#include <mutex>

namespace hplai {

namespace {

using namespace tile;

constexpr int kTeams = 3;       // teams per CTA
constexpr int kThreads = kTeams * kTeam;
constexpr int kMaxTiles = 32;   // b <= 1024

constexpr int kPairs = T * T / 2;   // two tagged elements are 16 bytes

struct alignas(128) GetrfWork {
	uint32_t status;
	uint32_t pad[31];
	ulonglong2 tiles[kMaxTiles * kMaxTiles][kPairs];
};

// Tags of one launch (epochs count from 1, so none equals the zeroed workspace's).
constexpr uint32_t kHanded = 1, kFinal = 2;

__device__ __forceinline__ void put_tile(const float *t, ulonglong2 *g, uint32_t tag, int tid)
{
	const uint64_t hi = static_cast<uint64_t>(tag) << 32;
#pragma unroll
	for (int q = 0; q < kPairs / kTeam; ++q) {
		const int e = tid + kTeam * q, j = e >> 4, i = (e & 15) * 2;
		const float2 f = *reinterpret_cast<const float2 *>(t + j * kLd + i);
		asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(g + e), "l"(hi | __float_as_uint(f.x)),
			"l"(hi | __float_as_uint(f.y)) : "memory");
	}
}

// One or two tiles (N words a thread) by one team, each thread until its own
// words are there; false on a timeout.  The caller's team barrier follows.
constexpr int kWords = kPairs / kTeam;

template <int N>
__device__ __forceinline__ bool get_words(const ulonglong2 *const (&g)[N], uint32_t tag, int tid, ulonglong2 (&v)[N][kWords])
{
	auto load = [](const ulonglong2 *p) {
		ulonglong2 w;
		asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(p) : "memory");
		return w;
	};
	auto ready = [tag](ulonglong2 w) {
		return static_cast<uint32_t>(w.x >> 32) == tag && static_cast<uint32_t>(w.y >> 32) == tag;
	};
#pragma unroll
	for (int n = 0; n < N; ++n)
#pragma unroll
		for (int q = 0; q < kWords; ++q) v[n][q] = load(g[n] + tid + kTeam * q);
	uint64_t t0 = 0;
	for (int it = 0;; ++it) {
		bool all = true;
#pragma unroll
		for (int n = 0; n < N; ++n)
#pragma unroll
			for (int q = 0; q < kWords; ++q) all = all && ready(v[n][q]);
		if (__all_sync(0xffffffffu, all)) return true;
		// the decision to give up is taken by the whole warp at once
		const uint64_t now = global_ns();
		if (it == 0) t0 = now;
		if (__any_sync(0xffffffffu, now - t0 > kWaitLimitNs)) return false;
		__nanosleep(40);
#pragma unroll
		for (int n = 0; n < N; ++n) {
			// a tile's first word stands for it until it arrives
			if (!ready(v[n][0])) {
				v[n][0] = load(g[n] + tid);
			} else {
#pragma unroll
				for (int q = 1; q < kWords; ++q)
					if (!ready(v[n][q])) v[n][q] = load(g[n] + tid + kTeam * q);
			}
		}
	}
}

__device__ __forceinline__ void keep_words(float *t, const ulonglong2 (&v)[kWords], bool transposed, int tid)
{
#pragma unroll
	for (int q = 0; q < kWords; ++q) {
		const int e = tid + kTeam * q, j = e >> 4, i = (e & 15) * 2;
		const float x = __uint_as_float(static_cast<uint32_t>(v[q].x)), y = __uint_as_float(static_cast<uint32_t>(v[q].y));
		if (transposed) {
			t[i * kLd + j] = x;
			t[(i + 1) * kLd + j] = y;
		} else {
			*reinterpret_cast<float2 *>(t + j * kLd + i) = make_float2(x, y);
		}
	}
}

__device__ __forceinline__ bool get_tile(float *t, const ulonglong2 *g, uint32_t tag, int tid, bool transposed = false)
{
	ulonglong2 v[1][kWords];
	const ulonglong2 *const src[1] = {g};
	const bool ok = get_words<1>(src, tag, tid, v);
	if (ok) keep_words(t, v[0], transposed, tid);
	return ok;
}

__device__ __forceinline__ bool get_tiles(float *t0, const ulonglong2 *g0, float *t1, const ulonglong2 *g1, uint32_t tag,
	int tid)
{
	ulonglong2 v[2][kWords];
	const ulonglong2 *const src[2] = {g0, g1};
	const bool ok = get_words<2>(src, tag, tid, v);
	if (ok) {
		keep_words(t0, v[0], false, tid);
		keep_words(t1, v[1], false, tid);
	}
	return ok;
}

// AND-vote and barrier of the whole CTA (barrier 0).
__device__ __forceinline__ bool all_agree(bool p) { return __syncthreads_and(p) != 0; }

// Tiles of a worker team's shared memory: kRes resident ones, two for a tile
// and its neighbour that have no place there, two for operands.
constexpr int kRes = 11;
constexpr int kTeamTiles = kRes + 4;
constexpr size_t kSmemBytes = static_cast<size_t>(kTeams) * kTeamTiles * kTileFloats * sizeof(float);
constexpr int kMaxUnits = 320;   // of one team: a third of the 959 units of 32 x 32 tiles

// A worker team's unit: a tile, with its neighbour towards the diagonal where it is
// two off it.
struct Unit {
	int m, d, ti, tj, at;   // min(ti, tj), |ti - tj|, the tile, its place in shared memory (-1: none)
	bool left;              // below the diagonal
	__device__ __forceinline__ explicit Unit(uint32_t e)
	    : m(e & 31u), d((e >> 5) & 31u), at(static_cast<int>(e >> 11) - 1), left(((e >> 10) & 1u) != 0)
	{
		ti = left ? m + d : m;
		tj = left ? m : m + d;
	}
	static __device__ __forceinline__ uint32_t pack(int m, int d, bool left)
	{
		return static_cast<uint32_t>(m) | static_cast<uint32_t>(d) << 5 | (left ? 1u << 10 : 0u);
	}
	static __device__ __forceinline__ uint32_t place(uint32_t e, int at) { return e | static_cast<uint32_t>(at + 1) << 11; }
	__device__ __forceinline__ int tiles() const { return d == 2 ? 2 : 1; }
	__device__ __forceinline__ int ti2() const { return left ? ti : ti + 1; }
	__device__ __forceinline__ int tj2() const { return left ? tj + 1 : tj; }
};

__global__ void __launch_bounds__(kThreads) getrf_tiles_kernel(int b, float *a, int64_t lda, GetrfWork *w,
	uint32_t epoch)
{
	extern __shared__ __align__(16) float dyn[];
	__shared__ __align__(16) float xchs[kTeams][kXchFloats];
	__shared__ uint32_t lists[kTeams][kMaxUnits];
	const int team = threadIdx.x / kTeam;
	const Team tm{static_cast<int>(threadIdx.x) % kTeam, static_cast<int>(threadIdx.x) & 31,
		static_cast<int>(threadIdx.x) % kTeam / 32, 1 + team};
	float *const xch = xchs[team];
	const int nt = (b + T - 1) / T;
	const uint32_t handed = epoch * 4u + kHanded, final_tag = epoch * 4u + kFinal;
	auto slot_of = [w, nt](int ti, int tj) { return w->tiles[ti + nt * tj]; };
	const bool vec = ((reinterpret_cast<uintptr_t>(a) & 15u) == 0) && ((lda & 3) == 0);

	if (blockIdx.x == 0) {
		// ---------------- the diagonal chain ----------------
		float *const tile0 = dyn;
		auto tile = [tile0](int i) { return tile0 + i * kTileFloats; };
		float *D = tile(0), *Dt = tile(1);
		float *const Lb[2] = {tile(2), tile(3)}, *const Ub[2] = {tile(4), tile(5)}, *const Xb[2] = {tile(6), tile(7)};
		float *L2 = tile(8), *U2 = tile(9);   // L(r+2, r), U(r, r+2): the last update but one of tile (r+2, r+2)
		const int v0 = min(T, b);
		if (team == 0) {
			stage_tile(Xb[0], a, lda, 0, 0, v0, v0, vec, tm.tid, kTeam);
			stage_wait();
			tm.sync();
			op_factor(tm, Xb[0], D, Dt, xch, v0);
		} else if (nt > 1) {
			// step 0's inputs are the block's own entries
			const int v1 = min(T, b - T);
			if (team == 1) {
				stage_tile(Lb[0], a, lda, T, 0, v1, T, vec, tm.tid, kTeam);
				stage_tile(Ub[0], a, lda, 0, T, T, v1, vec, tm.tid, kTeam);
			} else {
				stage_tile(Xb[1], a, lda, T, T, v1, v1, vec, tm.tid, kTeam);
			}
			stage_wait();
		}
		__syncthreads();
		bool ok = true;
		for (int r = 0; r + 1 < nt; ++r) {
			const int k0 = r * T, r1 = k0 + T, v1 = min(T, b - r1);
			float *Ld = Lb[r & 1], *Ud = Ub[r & 1], *Xd = Xb[(r + 1) & 1];
			if (team == 0) {
				op_solve_l(tm, Ld, Dt);
			} else if (team == 1) {
				op_solve_u(tm, Ud, D);
			} else {
				put_tile(D, slot_of(r, r), final_tag, tm.tid);
				store_tile(D, a, lda, k0, k0, T, T, tm.tid, kTeam);
			}
			__syncthreads();
			// team 0: the next diagonal tile; meanwhile what is final goes out, and
			// step r+1's inputs come in: tile (r+2, r+2) with r updates, L(r+2, r)
			// and U(r, r+2), tiles (r+2, r+1) and (r+1, r+2) with r+1
			const bool more = r + 2 < nt;
			bool mine = true;
			if (team == 0) {
				op_update(tm, Xd, Ld, Ud);
				tm.sync();
				op_factor(tm, Xd, D, Dt, xch, v1);
			} else if (team == 1) {
				put_tile(Ld, slot_of(r + 1, r), final_tag, tm.tid);
				put_tile(Ud, slot_of(r, r + 1), final_tag, tm.tid);
				store_tile(Ld, a, lda, r1, k0, v1, T, tm.tid, kTeam);
				store_tile(Ud, a, lda, k0, r1, T, v1, tm.tid, kTeam);
				if (more)
					mine = get_tiles(Lb[(r + 1) & 1], slot_of(r + 2, r + 1), Ub[(r + 1) & 1], slot_of(r + 1, r + 2), handed,
						tm.tid);
			} else if (more) {
				const int r2 = r1 + T, v2 = min(T, b - r2);
				float *const X2 = Xb[r & 1];
				if (r > 0) {
					mine = get_tile(X2, slot_of(r + 2, r + 2), handed, tm.tid);
				} else {
					stage_tile(X2, a, lda, r2, r2, v2, v2, vec, tm.tid, kTeam);
					stage_wait();
				}
				mine = get_tiles(L2, slot_of(r + 2, r), U2, slot_of(r, r + 2), final_tag, tm.tid) && mine;
				tm.sync();
				op_update(tm, X2, L2, U2);   // its last update but one
			}
			ok = all_agree(mine);
			if (!ok) break;
		}
		if (!ok) {
			if (threadIdx.x == 0) atomicOr(&w->status, 1u);
			return;
		}
		const int r0 = (nt - 1) * T, v = min(T, b - r0);
		store_tile(D, a, lda, r0, r0, v, v, threadIdx.x, kThreads);
		return;
	}

	// ---------------- worker teams ----------------
	// a worker team owns tiles that are two or more off the diagonal, each with its
	// neighbour towards the diagonal if that is one off it, and diagonal tiles from
	// (3, 3) on; team numbers run across the CTAs first, so that the units of a step
	// sit on different SMs
	const int gid = team * (gridDim.x - 1) + (blockIdx.x - 1), nteams = (gridDim.x - 1) * kTeams;
	float *const mem = dyn + team * kTeamTiles * kTileFloats;
	float *const tmp = mem + kRes * kTileFloats, *const tmp2 = tmp + kTileFloats, *const opL = tmp2 + kTileFloats,
	            *const opU = opL + kTileFloats;
	bool ok = true;   // the same in the whole team
	auto rows_of = [b](int ti) { return min(T, b - ti * T); };
	// This team's units in the order of their shells m = min(ti, tj): a unit is
	// final after step m, so the ones left at a step are the end of the list.  A
	// shell has its diagonal tile from 3 on, then (m + d, m) and (m, m + d), d = 2, 3, ..;
	// the units of all shells are dealt to the teams in turn, which shares every
	// step's work evenly whatever the number of teams (dealt column by column, 33
	// teams had a diagonal of 32 tiles each: b = 1024 on 12 SMs 1.40 ms a block, 0.75
	// so).  The list is made once: finding the next unit by divisions at every step
	// took longer than its updates (on 8 SMs 1.58 -> 1.14 ms).
	auto has_diag = [](int m) { return m >= 3 ? 1 : 0; };
	auto count = [&](int m) { return has_diag(m) + 2 * max(nt - m - 2, 0); };
	int units = 0;
	for (int m = 0; m < nt; ++m) units += count(m);
	uint32_t *const list = lists[team];
	const int n = units > gid ? (units - gid + nteams - 1) / nteams : 0;
	for (int i = tm.tid; i < n; i += kTeam) {
		int m = 0, p = gid + i * nteams;
		while (p >= count(m)) p -= count(m++);
		const int d = p < has_diag(m) ? 0 : 2 + (p - has_diag(m)) / 2;
		list[i] = Unit::pack(m, d, (p - has_diag(m)) % 2 == 0);
	}
	tm.sync();
	// places in shared memory for the last tiles: where there are more tiles than
	// places the first units, final soonest, do without
	if (tm.tid == 0)
		for (int i = n - 1, at = kRes; i >= 0; --i) {
			at -= Unit(list[i]).tiles();
			if (at < 0) break;
			list[i] = Unit::place(list[i], at);
		}
	tm.sync();
	auto load = [&](float *t, int ti, int tj) {
		stage_tile(t, a, lda, ti * T, tj * T, rows_of(ti), rows_of(tj), vec, tm.tid, kTeam);
	};
	auto store = [&](const float *t, int ti, int tj) {
		store_tile(t, a, lda, ti * T, tj * T, rows_of(ti), rows_of(tj), tm.tid, kTeam);
	};
	// every warp waits for itself; the barrier that follows makes the outcome the team's
	auto arrived = [&](bool mine) {
		int all;
		asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\t"
		             "selp.s32 %0, 1, 0, q;\n\t}"
		             : "=r"(all) : "r"(mine ? 1 : 0), "r"(tm.bar), "n"(kTeam) : "memory");
		ok = all != 0;
		return ok;
	};
	// X(ti, tj) -= L(ti, r) U(r, tj), an operand that the team already holds
	// given; a resident tile stays where it is unless it is handed over
	auto update = [&](int ti, int tj, int slot, int r, const float *haveL, const float *haveU, bool hand_over) {
		float *x = slot >= 0 ? mem + slot * kTileFloats : tmp2;
		bool mine;
		if (slot < 0) load(x, ti, tj);
		if (haveL)
			mine = get_tile(opU, slot_of(r, tj), final_tag, tm.tid);
		else if (haveU)
			mine = get_tile(opL, slot_of(ti, r), final_tag, tm.tid);
		else
			mine = get_tiles(opL, slot_of(ti, r), opU, slot_of(r, tj), final_tag, tm.tid);
		stage_wait();
		if (!arrived(mine)) return;
		op_update(tm, x, haveL ? haveL : opL, haveU ? haveU : opU);
		tm.sync();   // the operand tiles are free again
		if (hand_over) {
			put_tile(x, slot_of(ti, tj), handed, tm.tid);
		} else if (slot < 0) {
			store(x, ti, tj);
		}
		if (slot < 0) tm.sync();
	};
	for (int i = 0; i < n; ++i) {
		const Unit u(list[i]);
		if (u.at < 0) continue;
		load(mem + u.at * kTileFloats, u.ti, u.tj);
		if (u.d == 2) load(mem + (u.at + 1) * kTileFloats, u.ti2(), u.tj2());
	}
	stage_wait();
	tm.sync();
	for (int r = 0, i0 = 0; r < nt && ok; ++r) {
		// the panel tiles of step r, then the trailing updates
		for (; ok && i0 < n; ++i0) {
			const Unit u(list[i0]);
			if (u.m != r) break;
			if (u.d == 0) continue;
			float *x = u.at >= 0 ? mem + u.at * kTileFloats : tmp;
			const bool left = u.left;
			// L tile X <- X U(r,r)^{-1}, or U tile X <- L(r,r)^{-1} X (tile (r, r) is a whole one)
			if (u.at < 0) load(x, u.ti, u.tj);
			const bool mine = get_tile(opL, slot_of(r, r), final_tag, tm.tid, left);
			stage_wait();
			if (!arrived(mine)) break;
			if (left)
				op_solve_l(tm, x, opL);
			else
				op_solve_u(tm, x, opL);
			put_tile(x, slot_of(u.ti, u.tj), final_tag, tm.tid);
			// its neighbour's last update, and on to the diagonal CTA
			if (u.d == 2)
				update(u.ti2(), u.tj2(), u.at >= 0 ? u.at + 1 : -1, r, left ? x : nullptr, left ? nullptr : x, true);
			store(x, u.ti, u.tj);
			if (u.at < 0) tm.sync();
		}
		for (int i = i0; ok && i < n; ++i) {
			const Unit u(list[i]);
			if (u.d == 0 && u.m < r + 3) continue;   // the diagonal CTA has it
			update(u.ti, u.tj, u.at, r, nullptr, nullptr, u.d == 0 && u.m == r + 3);
			if (ok && u.d == 2) update(u.ti2(), u.tj2(), u.at >= 0 ? u.at + 1 : -1, r, nullptr, nullptr, false);
		}
	}
	if (!ok && tm.tid == 0) atomicOr(&w->status, 1u);
}

std::mutex g_static_mu;
__device__ GetrfWork g_static_work;
uint32_t g_static_epoch = 0;

int max_coresident_ctas()
{
	static DeviceOnce once;
	int n = 0;
	if (once.get([](int dev, int *v) -> int {
		int per_sm = 0, sms = 0;
		HPLAI_CUDA_TRY(cudaFuncSetAttribute(getrf_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
			static_cast<int>(kSmemBytes)));
		HPLAI_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, getrf_tiles_kernel, kThreads,
			kSmemBytes));
		HPLAI_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
		*v = per_sm * sms;
		return HPLAI_OK;
	}, &n) != HPLAI_OK) return 0;
	return n;
}

} // namespace

// a block of order b uses the first nt x nt tiles
size_t getrf_workspace(int b)
{
	const size_t nt = (static_cast<size_t>(b) + T - 1) / T;
	return offsetof(GetrfWork, tiles) + nt * nt * sizeof(ulonglong2) * kPairs;
}

int launch_getrf_tiles(int b, float *a, int64_t lda, void *work, uint32_t *epoch, int max_ctas, cudaStream_t st)
{
	if (b <= 0) return HPLAI_OK;
	if (b > T * kMaxTiles || !a || lda < b || !work || !epoch) return HPLAI_EINVAL;
	const int nt = (b + T - 1) / T;
	// CTA 0: the diagonal chain; then enough worker CTAs for one tile per team
	// (two tiles or fewer to a side leave them nothing to do)
	int grid = 1 + (nt > 2 ? (nt * nt + kTeams - 1) / kTeams : 0);
	const int cap = max_coresident_ctas();
	if (cap < 2) return HPLAI_EUNSUPPORTED;
	if (grid > cap) grid = cap;
	if (max_ctas > 0 && grid > max_ctas) grid = max_ctas < 2 ? 2 : max_ctas;
	if (nt > 2 && grid < 2) grid = 2;
	GetrfWork *w = static_cast<GetrfWork *>(work);
	// tags are epoch * 4 + state: epochs stay below 2^30
	uint32_t ep = ++*epoch;
	if (ep >= (1u << 30)) return HPLAI_EUNSUPPORTED;
	void *args[] = {(void *)&b, (void *)&a, (void *)&lda, (void *)&w, (void *)&ep};
	HPLAI_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(getrf_tiles_kernel), dim3(grid),
		dim3(kThreads), args, kSmemBytes, st));
	count_launches();
	return HPLAI_OK;
}

int getrf_status(void *work, cudaStream_t st, int *status)
{
	uint32_t v = 0;
	GetrfWork *w = static_cast<GetrfWork *>(work);
	HPLAI_CUDA_TRY(cudaMemcpyAsync(&v, &w->status, sizeof(v), cudaMemcpyDeviceToHost, st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	*status = v ? HPLAI_ETIMEOUT : HPLAI_OK;
	return HPLAI_OK;
}

// The leaf entry point's workspace: one per library, calls serialised by
// the host lock (stream order then keeps their flags apart).
int launch_getrf(int b, float *a, int64_t lda, cudaStream_t st)
{
	std::lock_guard<std::mutex> lk(g_static_mu);
	void *w = nullptr;
	HPLAI_CUDA_TRY(cudaGetSymbolAddress(&w, g_static_work));
	HPLAI_TRY(launch_getrf_tiles(b, a, lda, w, &g_static_epoch, 0, st));
	int s = HPLAI_OK;
	HPLAI_TRY(getrf_status(w, st, &s));
	return s;
}

} // namespace hplai
