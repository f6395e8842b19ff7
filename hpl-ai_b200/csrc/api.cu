// api.cu -- the solve context of libhplai: allocation, generation, the
// blocked LU driver and the iterative-refinement driver.
//
// This is the single-GPU collapse of the reference's driver
// (main.cpp:185-488): one n x n FP32 matrix in HBM instead of 2D
// block-cyclic panels, FP16 copies of the current L and U panels instead of
// the broadcast buffers, CUDA streams instead of MPI requests.
#include "common.cuh"
#include "internal.h"

#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>

namespace hplai {

namespace {
std::mutex g_err_mu;
std::string g_err;
std::atomic<unsigned long long> g_launches{0};
} // namespace

void count_launches(int k) { g_launches.fetch_add(static_cast<unsigned long long>(k), std::memory_order_relaxed); }

void set_last_cuda_error(cudaError_t e, const char *what, const char *file, int line)
{
	std::lock_guard<std::mutex> lk(g_err_mu);
	char buf[512];
	std::snprintf(buf, sizeof buf, "%s failed: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
	g_err = buf;
}

void set_last_error_message(const char *msg)
{
	std::lock_guard<std::mutex> lk(g_err_mu);
	g_err = msg;
}

static int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

} // namespace hplai

using namespace hplai;

struct hplai_ctx {
	int n = 0, b = 0, nb = 0, precision = 0;
	unsigned flags = 0;
	int side_sms = 20;   // SMs of the side stream with HPLAI_FLAG_LOOKAHEAD (hplai_autotune sets it)
	int64_t lda = 0, ldh = 0;
	float *A = nullptr;
	// Panel copies for the trailing updates.  A group of `group` consecutive
	// panels (1, 2 with HPLAI_FLAG_GROUP2, 4 with HPLAI_FLAG_GROUP4) updates
	// the trailing matrix in one pass with K = group * b
	// (C -= [L_k .. L_k+g-1] [U_k; ..; U_k+g-1]), which divides the passes over
	// the trailing matrix by the group size.  FP16 group buffers, double
	// buffered (the next group is formed on the side stream while the main
	// stream's update still reads the current one): row i of Lh[q] holds row i
	// of the group's L panels side by side (slot h at column h * ldh, row
	// pitch ldg = gcap * ldh), row j of Uh[q] column j of its U panels (the
	// reference's nbuf = 2 rotating LRPanels, panel.hpp:236-268).
	static constexpr int kMaxGroup = 4;
	int group = 1, gcap = 1;      // panels per update now / that the buffers hold
	int64_t ldg = 0;
	uint16_t *Lh[2] = {nullptr, nullptr}, *Uh[2] = {nullptr, nullptr};
	SchurMaps maps[2][kMaxGroup]; // [buffer][slot]: one panel, K = b
	SchurMaps mapsg[2][2];        // [buffer][0: K = 2b, 1: K = 4b]: the group's slots together
	// precision form: e4m3 group copies with one power-of-two factor per 128
	// rows shared by the group's panels (row pitch ld8g = gcap * ld8), and,
	// for the updates of a group's later blocks by its earlier panels (block
	// e + j receives panels e .. e + j - 1 before it is factored), an e4m3
	// copy of each panel but the group's last (L8s[h], U8s[h] for slot h)
	uint8_t *L8[2] = {nullptr, nullptr}, *U8[2] = {nullptr, nullptr};
	float *sl[2] = {nullptr, nullptr}, *su[2] = {nullptr, nullptr};
	uint8_t *L8s[kMaxGroup - 1] = {}, *U8s[kMaxGroup - 1] = {};
	float *sls[kMaxGroup - 1] = {}, *sus[kMaxGroup - 1] = {};
	unsigned *qbits = nullptr;
	// precision form with FP16 panel products: the e4m3 copies' block maxima,
	// gathered by the panel stores (L and U of the panel's own copy, L and U
	// of the group's shared copy)
	unsigned *qb[4] = {nullptr, nullptr, nullptr, nullptr};
	int64_t ld8 = 0, ld8g = 0;
	// HPLAI_FLAG_FP16_DECK: FP16 trailing-update deck (n x lda halves), holding
	// dscale x (accumulated update)
	uint16_t *deck = nullptr;
	float dscale = 1.f;
	// HPLAI_FLAG_LAZY_A: A is not stored; the deck lives in the upper half of
	// each FP32 column (FP16 element (i, j) at ((uint16_t*)A)[2 lda j + lda + i],
	// FP32 rows lda/2 .. (lda + n)/2), so deck_ld = 2 lda halves; dstage holds
	// a diagonal block's deck while the block is formed over it
	int64_t deck_ld = 0;
	bool deck_aliased = false;
	uint16_t *dstage = nullptr;
	// HPLAI_FLAG_REF_DECK: the reference's `-d` deck (n x lda halves), its
	// FP16 L-panel scale n^0.75 and the lazy-init downscale; regen_a: A is
	// not stored (hplai_generate) and the lazy initialisation regenerates it
	uint16_t *rdeck = nullptr, *rback = nullptr;   // rback: HPLAI_FLAG_REF_BACKBUF
	float rscalea = 1.f, rdownscale = 1.f;
	bool regen_a = false;
	// the matrix family (hplai_set_matrix): the LCG benchmark matrix or
	// Higham's, with its parameters
	int matrix = HPLAI_MATRIX_LCG;
	double h_alpha = 0.0, h_beta = 0.0;
	SchurMaps maps8[2];           // [buffer]: K = b
	SchurMaps maps8g[2][2];       // [buffer][0: K = 2b, 1: K = 4b]
	SchurMaps maps8s[kMaxGroup - 1];   // the single panel copies, K = b
	TcPanels tc;
	float *tcbuf = nullptr;   // phi, plo (n x ldp), the four b x ldp inverse buffers, the inversion work
	double *rhs = nullptr, *d = nullptr, *x = nullptr, *r = nullptr, *scal = nullptr;
	void *gemv_work = nullptr;
	size_t gemv_bytes = 0;
	uint8_t *zeroed = nullptr;    // one allocation, zeroed once: kstatus, trsv_work, getrf_work
	void *trsv_work = nullptr;
	size_t trsv_bytes = 0;
	void *getrf_work = nullptr;   // tagged tiles of the diagonal block LU
	void *check_work = nullptr;   // hplai_checksum: per-CTA partial sums, then the three results
	double *dinv = nullptr;       // FP64 inverses of the factors' 128 x 128 diagonal blocks
	unsigned *kstatus = nullptr;  // timeout words of this context's Schur [0] and panel [1] kernels
	unsigned *f16s = nullptr;     // precision form: triangle maxima [0..1] and inverse scales [2..3]
	uint32_t getrf_epoch = 0;
	cudaStream_t st = nullptr;    // main stream: Schur updates, refinement, everything else
	cudaStream_t st2 = nullptr;   // side stream (high priority): diagonal block + panels
	cudaEvent_t ev_panel = nullptr, ev_next = nullptr;
	std::vector<cudaEvent_t> phase_events;   // PhaseEvents' pool
	// host -> device copies of the matrix streamed behind the factorisation
	// (hplai_solve_host with the FP16 deck): one event per panel's block
	// column and row, created on first use
	cudaStream_t st3 = nullptr;
	std::vector<cudaEvent_t> ev_copy;
	uint64_t seed = 0;
	bool have_inputs = false, factored = false;
	double norma = 0.0, normb = 0.0;
	std::vector<double> log_resid, log_harness;
	double phase_ms[HPLAI_PH_COUNT] = {};
	// hplai_autotune's trials: schedule and factorisation milliseconds
	struct Trial {
		unsigned flags;
		int side_sms;
		double ms;
		int tile_group;
	};
	int tile_group = 0;   // tile rows per group of the Schur kernel's tile order (0: its default)
	int cta_pairs = -1;   // deck updates on CTA pairs: 1 on, 0 off, -1 the library default
	std::vector<Trial> tune_log;
	// GMRES correction: restart length, relative tolerance on the
	// preconditioned residual, basis and scratch (allocated on first use)
	int gm_restart = 30;
	double gm_tol = 1e-12;
	// right (flexible) preconditioning: the basis of A M^{-1}, with the
	// preconditioned vectors z_j = M^{-1} v_j kept (gm_z) so that the
	// correction is Z y -- one application of M^{-1} per inner step and none
	// before or after; left: M^{-1} A, one more application for M^{-1} r
	int gm_right = 1;
	double *gm_v = nullptr;     // n x (gm_restart + 1), ld = gm_ldv
	double *gm_z = nullptr;     // n x gm_restart (right preconditioning), ld = gm_ldv
	double *gm_w = nullptr;     // n
	double *gm_small = nullptr; // part (kDotBlocks x kMaxBasis), H (kMaxBasis^2), tmp, y
	double *rhs2 = nullptr, *x2 = nullptr;   // caller right-hand sides (hplai_solve_rhs / _transpose)
	int64_t gm_ldv = 0;
	int gm_cap = 0;             // restart length gm_v was sized for
	int gm_inner = 0;           // inner steps of the last hplai_refine
};

namespace {

int ctx_free(hplai_ctx *c)
{
	if (!c) return HPLAI_OK;
	cudaFree(c->A);
	for (int i = 0; i < 2; ++i) {
		cudaFree(c->Lh[i]);
		cudaFree(c->Uh[i]);
		cudaFree(c->L8[i]);
		cudaFree(c->U8[i]);
		cudaFree(c->sl[i]);
		cudaFree(c->su[i]);
	}
	for (int h = 0; h < hplai_ctx::kMaxGroup - 1; ++h) {
		cudaFree(c->L8s[h]);
		cudaFree(c->U8s[h]);
		cudaFree(c->sls[h]);
		cudaFree(c->sus[h]);
	}
	cudaFree(c->qbits);
	cudaFree(c->qb[0]);
	if (!c->deck_aliased) cudaFree(c->deck);
	cudaFree(c->dstage);
	cudaFree(c->rdeck);
	cudaFree(c->rback);
	cudaFree(c->tcbuf);
	cudaFree(c->rhs);
	cudaFree(c->d);
	cudaFree(c->x);
	cudaFree(c->r);
	cudaFree(c->scal);
	cudaFree(c->gemv_work);
	cudaFree(c->zeroed);
	cudaFree(c->check_work);
	cudaFree(c->dinv);
	cudaFree(c->f16s);
	cudaFree(c->gm_v);
	cudaFree(c->gm_z);
	cudaFree(c->gm_w);
	cudaFree(c->gm_small);
	cudaFree(c->rhs2);
	cudaFree(c->x2);
	if (c->ev_panel) cudaEventDestroy(c->ev_panel);
	if (c->ev_next) cudaEventDestroy(c->ev_next);
	for (cudaEvent_t e : c->ev_copy) cudaEventDestroy(e);
	for (cudaEvent_t e : c->phase_events) cudaEventDestroy(e);
	if (c->st3) cudaStreamDestroy(c->st3);
	if (c->st) cudaStreamDestroy(c->st);
	if (c->st2) cudaStreamDestroy(c->st2);
	delete c;
	return HPLAI_OK;
}

#define CTX_ALLOC(ptr, bytes)                                                         \
	do {                                                                              \
		cudaError_t e__ = cudaMalloc(reinterpret_cast<void **>(&(ptr)), (bytes));     \
		if (e__ != cudaSuccess) {                                                     \
			set_last_cuda_error(e__, "cudaMalloc(" #ptr ")", __FILE__, __LINE__);     \
			(void)cudaGetLastError();                                                 \
			ctx_free(c);                                                              \
			return HPLAI_ENOMEM;                                                      \
		}                                                                             \
	} while (0)

// Elapsed milliseconds between event pairs recorded around each phase.  The
// events belong to the context and are reused by its next call: an event costs
// the host as much as a launch, and a small solve is bound by its launches.
struct PhaseEvents {
	struct Span {
		int phase;
		cudaEvent_t begin, end;
	};
	std::vector<cudaEvent_t> &pool;
	size_t used = 0;
	std::vector<Span> spans;
	// everything of this call runs on one stream, phase after phase: a phase
	// begins where the last one ended, unless the stream waited in between
	bool chained;
	bool waited = false;
	explicit PhaseEvents(std::vector<cudaEvent_t> &p, bool one_stream = false) : pool(p), chained(one_stream) {}
	int take(cudaEvent_t *e)
	{
		if (used == pool.size()) {
			cudaEvent_t n;
			HPLAI_CUDA_TRY(cudaEventCreate(&n));
			pool.push_back(n);
		}
		*e = pool[used++];
		return HPLAI_OK;
	}
	int record(cudaStream_t st, int ph)
	{
		Span sp{ph, nullptr, nullptr};
		if (chained && !waited && !spans.empty()) {
			sp.begin = spans.back().end;
		} else {
			HPLAI_TRY(take(&sp.begin));
			HPLAI_CUDA_TRY(cudaEventRecord(sp.begin, st));
		}
		waited = false;
		HPLAI_TRY(take(&sp.end));
		spans.push_back(sp);
		return HPLAI_OK;
	}
	int end(cudaStream_t st) { return cudaEventRecord(spans.back().end, st) == cudaSuccess ? HPLAI_OK : HPLAI_ECUDA; }
	// ends the phase and begins the next one on the same stream, nothing between them
	int next(cudaStream_t st, int ph)
	{
		HPLAI_TRY(end(st));
		Span sp{ph, spans.back().end, nullptr};
		HPLAI_TRY(take(&sp.end));
		spans.push_back(sp);
		return HPLAI_OK;
	}
	void collect(double *ms)
	{
		for (const Span &sp : spans) {
			float t = 0.f;
			if (cudaEventElapsedTime(&t, sp.begin, sp.end) == cudaSuccess) ms[sp.phase] += t;
		}
	}
};

int compute_norms(hplai_ctx *c)
{
	HPLAI_TRY(launch_infnorm(c->n, c->rhs, c->scal + 0, c->st));
	HPLAI_TRY(launch_infnorm(c->n, c->d, c->scal + 1, c->st));
	double h[2];
	HPLAI_CUDA_TRY(cudaMemcpyAsync(h, c->scal, sizeof h, cudaMemcpyDeviceToHost, c->st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(c->st));
	c->normb = h[0];
	if (c->matrix == HPLAI_MATRIX_HIGHAM)
		c->norma = higham_norm(c->n, c->h_alpha, c->h_beta);   // higham_infnorm (panel_norm.hpp:86-141)
	else
		c->norma = 2.0 * h[1];   // hpl_infnorm: the diagonal is the off-diagonal row 1-norm
	return HPLAI_OK;
}

// y <- beta y + alpha A x (A^T x with trans), A regenerated in FP64
// (panel_gemv with Matgen<double> or HMGen<double>, panel_gemv.hpp:57-132)
// With y0, beta y0 instead of beta y; with norms, max |x_i|, max |y_i| and the
// triangular solves' timeout word.
int matvec(hplai_ctx *c, double alpha, const double *x, double beta, double *y, cudaStream_t st, bool trans,
	const double *y0 = nullptr, double *norms = nullptr)
{
	if (c->matrix == HPLAI_MATRIX_HIGHAM)
		return launch_higham_gemv(c->n, alpha, x, beta, y, c->h_alpha, c->h_beta, c->d, c->gemv_work, c->gemv_bytes, st,
			trans, y0, norms, trsv_status_word(c->trsv_work));
	return launch_otf_gemv(c->n, alpha, x, beta, y, c->seed, c->d, c->gemv_work, c->gemv_bytes, st, trans, y0, norms,
		trsv_status_word(c->trsv_work));
}

} // namespace

extern "C" const char *hplai_status_string(int status)
{
	switch (status) {
	case HPLAI_OK: return "ok";
	case HPLAI_EINVAL: return "invalid argument";
	case HPLAI_ENOMEM: return "out of memory";
	case HPLAI_ECUDA: return "CUDA error";
	case HPLAI_ENOTCONV: return "refinement did not converge";
	case HPLAI_ETIMEOUT: return "device wait timed out";
	case HPLAI_ESTATE: return "call out of order";
	case HPLAI_EUNSUPPORTED: return "unsupported configuration";
	default: return "unknown status";
	}
}

extern "C" int hplai_version(void) { return HPLAI_VERSION; }

extern "C" unsigned long long hplai_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

extern "C" int hplai_last_error(char *buf, size_t len)
{
	std::lock_guard<std::mutex> lk(g_err_mu);
	if (buf && len) {
		std::strncpy(buf, g_err.c_str(), len - 1);
		buf[len - 1] = 0;
	}
	return HPLAI_OK;
}

extern "C" int hplai_create(hplai_ctx **out, int n, int b, int precision, unsigned flags)
{
	if (!out) return HPLAI_EINVAL;
	*out = nullptr;
	if (n <= 0 || b < 16 || b > 1024 || n % b) return HPLAI_EINVAL;
	if (precision != HPLAI_F32_F16 && precision != HPLAI_F32_F8) return HPLAI_EUNSUPPORTED;
	if ((flags & HPLAI_FLAG_FP16_DECK) && (b % 8)) return HPLAI_EINVAL;
	if ((flags & (HPLAI_FLAG_GROUP2 | HPLAI_FLAG_GROUP4)) && (b % 128)) return HPLAI_EINVAL;
	if ((flags & HPLAI_FLAG_GROUP2) && (flags & HPLAI_FLAG_GROUP4)) return HPLAI_EINVAL;
	if ((flags & HPLAI_FLAG_REF_DECK) && (precision != HPLAI_F32_F16 ||
		(flags & (HPLAI_FLAG_FP16_DECK | HPLAI_FLAG_GROUP2 | HPLAI_FLAG_GROUP4 | HPLAI_FLAG_LOOKAHEAD))))
		return HPLAI_EINVAL;
	if ((flags & HPLAI_FLAG_REF_BACKBUF) && !(flags & HPLAI_FLAG_REF_DECK)) return HPLAI_EINVAL;
	// A regenerated at panel time: the precision form's FP16 panel copies fold it in
	if ((flags & HPLAI_FLAG_LAZY_A) && (!(flags & HPLAI_FLAG_FP16_DECK) || precision != HPLAI_F32_F8 || b % 4 ||
		(flags & (HPLAI_FLAG_SIMT_PANELS | HPLAI_FLAG_REF_DECK))))
		return HPLAI_EINVAL;
	hplai_ctx *c = new hplai_ctx;
	c->n = n;
	c->b = b;
	c->nb = n / b;
	c->precision = precision;
	c->flags = flags;
	// lda padded to 64 floats plus 64 more so that columns do not share a
	// power-of-two stride (the reference's calc_lda_c, panel.hpp:10-18, for HBM).
	c->lda = round_up(n, 64) + 64;
	c->ldh = round_up(b, 64);
	// panel groups need whole 128-byte e4m3 rows and 64-half FP16 rows per
	// panel; buffers for four panels only when asked for (HPLAI_FLAG_GROUP4)
	c->gcap = (b % 128 == 0) ? ((flags & HPLAI_FLAG_GROUP4) ? 4 : 2) : 1;
	c->group = (flags & HPLAI_FLAG_GROUP4) ? 4 : (flags & HPLAI_FLAG_GROUP2) ? 2 : 1;
	c->ldg = c->gcap * c->ldh;
	{
		int lo = 0, hi = 0;
		const cudaError_t e[5] = {cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking),
			cudaDeviceGetStreamPriorityRange(&lo, &hi),
			cudaStreamCreateWithPriority(&c->st2, cudaStreamNonBlocking, hi),
			cudaEventCreateWithFlags(&c->ev_panel, cudaEventDisableTiming),
			cudaEventCreateWithFlags(&c->ev_next, cudaEventDisableTiming)};
		for (cudaError_t ei : e) {
			if (ei != cudaSuccess) {
				set_last_cuda_error(ei, "stream/event creation", __FILE__, __LINE__);
				ctx_free(c);
				return HPLAI_ECUDA;
			}
		}
	}
	CTX_ALLOC(c->A, sizeof(float) * static_cast<size_t>(c->lda) * n);
	for (int i = 0; i < 2; ++i) {
		CTX_ALLOC(c->Lh[i], sizeof(uint16_t) * static_cast<size_t>(c->ldg) * n);
		CTX_ALLOC(c->Uh[i], sizeof(uint16_t) * static_cast<size_t>(c->ldg) * n);
	}
	const int nblk128 = n / 128 + 2;
	if (precision == HPLAI_F32_F8) {
		c->ld8 = round_up(b, 128);
		c->ld8g = c->gcap * c->ld8;
		for (int i = 0; i < 2; ++i) {
			CTX_ALLOC(c->L8[i], static_cast<size_t>(c->ld8g) * n);
			CTX_ALLOC(c->U8[i], static_cast<size_t>(c->ld8g) * n);
			CTX_ALLOC(c->sl[i], sizeof(float) * nblk128);
			CTX_ALLOC(c->su[i], sizeof(float) * nblk128);
		}
		for (int h = 0; h < c->gcap - 1; ++h) {
			CTX_ALLOC(c->L8s[h], static_cast<size_t>(c->ld8) * n);
			CTX_ALLOC(c->U8s[h], static_cast<size_t>(c->ld8) * n);
			CTX_ALLOC(c->sls[h], sizeof(float) * nblk128);
			CTX_ALLOC(c->sus[h], sizeof(float) * nblk128);
		}
		CTX_ALLOC(c->qbits, sizeof(unsigned) * nblk128);
		CTX_ALLOC(c->qb[0], sizeof(unsigned) * 4 * nblk128);
		for (int i = 1; i < 4; ++i) c->qb[i] = c->qb[0] + i * nblk128;
	}
	c->deck_ld = c->lda;
	if (flags & HPLAI_FLAG_LAZY_A) {
		c->deck = reinterpret_cast<uint16_t *>(c->A) + c->lda;
		c->deck_ld = 2 * c->lda;
		c->deck_aliased = true;
		CTX_ALLOC(c->dstage, sizeof(uint16_t) * static_cast<size_t>(b) * b);
		c->dscale = std::ldexp(1.0f, static_cast<int>(std::lround(0.75 * std::log2(static_cast<double>(n)))));
	} else if (flags & HPLAI_FLAG_FP16_DECK) {
		CTX_ALLOC(c->deck, sizeof(uint16_t) * static_cast<size_t>(c->lda) * n);
		// a power of two near n^0.75, the reference's scalea (hpl_rand.hpp:154)
		c->dscale = std::ldexp(1.0f, static_cast<int>(std::lround(0.75 * std::log2(static_cast<double>(n)))));
	}
	if (flags & HPLAI_FLAG_REF_DECK) {
		CTX_ALLOC(c->rdeck, sizeof(uint16_t) * static_cast<size_t>(c->lda) * n);
		if (flags & HPLAI_FLAG_REF_BACKBUF) CTX_ALLOC(c->rback, sizeof(uint16_t) * static_cast<size_t>(c->lda) * n);
		// scalea = sqrt(n sqrt(n)) in FP64, then FP32; downscale = FP32(1 / (scalea * scaleb)), scaleb = 1
		// (hpl_rand.hpp:154-155, panel_trf.hpp:717-719)
		c->rscalea = static_cast<float>(std::sqrt(n * std::sqrt(static_cast<double>(n))));
		c->rdownscale = static_cast<float>(1. / static_cast<double>(c->rscalea * 1.0f));
	}
	const int64_t ldp = round_up(b, 32);
	const size_t tc_elems = static_cast<size_t>(ldp) * (2 * static_cast<size_t>(n) + 4 * static_cast<size_t>(b)) +
		tc_inverse_work_elems(ldp);
	CTX_ALLOC(c->tcbuf, sizeof(float) * tc_elems);
	CTX_ALLOC(c->rhs, sizeof(double) * n);
	CTX_ALLOC(c->d, sizeof(double) * n);
	CTX_ALLOC(c->x, sizeof(double) * n);
	CTX_ALLOC(c->r, sizeof(double) * n);
	CTX_ALLOC(c->scal, sizeof(double) * 8);
	c->gemv_bytes = otf_gemv_workspace(n);
	CTX_ALLOC(c->gemv_work, c->gemv_bytes);
	c->trsv_bytes = trsv_workspace(n);
	const size_t at_trsv = 256, at_getrf = at_trsv + round_up(static_cast<int64_t>(c->trsv_bytes), 256);
	const size_t zeroed_bytes = at_getrf + getrf_workspace(b);
	CTX_ALLOC(c->zeroed, zeroed_bytes);
	c->kstatus = reinterpret_cast<unsigned *>(c->zeroed);
	c->trsv_work = c->zeroed + at_trsv;
	c->getrf_work = c->zeroed + at_getrf;
	CTX_ALLOC(c->check_work, panel_check_workspace(n) + 3 * sizeof(double));
	CTX_ALLOC(c->dinv, sizeof(double) * trsv_dinv_doubles(n));
	CTX_ALLOC(c->f16s, 4 * sizeof(unsigned));
	if (cudaMemset(c->zeroed, 0, zeroed_bytes) != cudaSuccess ||
		cudaMemset(c->tcbuf, 0, sizeof(float) * tc_elems) != cudaSuccess) {
		ctx_free(c);
		return HPLAI_ECUDA;
	}
	int s = HPLAI_OK;
	auto finish = [&](SchurMaps &m) {
		if (s == HPLAI_OK) s = schur_set_cmap(&m, c->A, n, n, c->lda);
		m.status = c->kstatus;
		m.deck_base = c->deck;
		m.deck_ld = c->deck_ld;
	};
	for (int i = 0; i < 2 && s == HPLAI_OK; ++i) {
		for (int h = 0; h < c->gcap && s == HPLAI_OK; ++h) {
			s = schur_make_maps(&c->maps[i][h], c->Lh[i] + h * c->ldh, n, c->ldg, c->Uh[i] + h * c->ldh, n, c->ldg, b);
			finish(c->maps[i][h]);
		}
		for (int g = 0; g < 2 && s == HPLAI_OK; ++g) {
			const int gk = 2 << g;   // panels of the group: 2, 4
			if (gk > c->gcap) break;
			s = schur_make_maps(&c->mapsg[i][g], c->Lh[i], n, c->ldg, c->Uh[i], n, c->ldg, gk * b);
			finish(c->mapsg[i][g]);
		}
		if (s == HPLAI_OK && precision == HPLAI_F32_F8) {
			s = schur_make_maps_fp8(&c->maps8[i], c->L8[i], n, c->ld8g, c->U8[i], n, c->ld8g, b);
			finish(c->maps8[i]);
			for (int g = 0; g < 2 && s == HPLAI_OK; ++g) {
				const int gk = 2 << g;
				if (gk > c->gcap) break;
				s = schur_make_maps_fp8(&c->maps8g[i][g], c->L8[i], n, c->ld8g, c->U8[i], n, c->ld8g, gk * b);
				finish(c->maps8g[i][g]);
			}
		}
	}
	for (int h = 0; h < c->gcap - 1 && s == HPLAI_OK && precision == HPLAI_F32_F8; ++h) {
		s = schur_make_maps_fp8(&c->maps8s[h], c->L8s[h], n, c->ld8, c->U8s[h], n, c->ld8, b);
		finish(c->maps8s[h]);
	}
	if (s == HPLAI_OK) {
		float *base = c->tcbuf;
		const size_t pn = static_cast<size_t>(ldp) * n, pb = static_cast<size_t>(ldp) * b;
		s = tc_panels_make(&c->tc, n, b, base, base + pn, ldp, base + 2 * pn, base + 2 * pn + pb,
			base + 2 * pn + 2 * pb, base + 2 * pn + 3 * pb, base + 2 * pn + 4 * pb);
		c->tc.status = c->kstatus + 1;
		// the precision form's panels only need FP16 accuracy: its Schur operands are e4m3
		if (precision == HPLAI_F32_F8) c->tc.terms = 1;
		c->tc.f16_amax = c->f16s;
		c->tc.f16_oscale = reinterpret_cast<float *>(c->f16s + 2);
	}
	if (s != HPLAI_OK) {
		ctx_free(c);
		return s;
	}
	*out = c;
	return HPLAI_OK;
}

extern "C" int hplai_destroy(hplai_ctx *c) { return ctx_free(c); }

extern "C" int hplai_generate(hplai_ctx *c, uint64_t seed)
{
	if (!c) return HPLAI_EINVAL;
	const int n = c->n;
	// pmatgen (matgen.hpp:7-22): the whole matrix, then the diagonal as the
	// FP32 rounding of the sequential FP64 row sums (which are also d).  The
	// `-d` parity mode stores no A (pmatgen0, main.cpp:260-261): its lazy
	// initialisation regenerates each block when it joins a panel.
	c->regen_a = (c->flags & (HPLAI_FLAG_REF_DECK | HPLAI_FLAG_LAZY_A)) != 0;
	if (c->matrix == HPLAI_MATRIX_HIGHAM) {
		// pmatgen / pdiaggen with HMGen (matgen.hpp:25-77, 227-243); the
		// right-hand side stays the LCG's column n (main.cpp:266)
		HPLAI_TRY(launch_higham_fill(n, c->h_alpha, c->h_beta, c->A, c->lda, c->d, false, c->st));
	} else {
		if (!c->regen_a) HPLAI_TRY(launch_fill(n, 0, 0, n, n, c->A, c->lda, seed, 0, c->st));
		HPLAI_TRY(launch_diag(n, 0, n, c->d, c->regen_a ? nullptr : c->A, c->lda, seed, c->st));
	}
	HPLAI_TRY(launch_rhs(n, c->rhs, seed, c->st));
	c->seed = seed;
	HPLAI_TRY(compute_norms(c));
	c->have_inputs = true;
	c->factored = false;
	return HPLAI_OK;
}

extern "C" int hplai_upload(hplai_ctx *c, const float *a, int64_t lda, const double *rhs, const double *diag,
	uint64_t seed)
{
	if (!c || !a || !rhs || !diag || lda < c->n) return HPLAI_EINVAL;
	if (c->flags & HPLAI_FLAG_LAZY_A) return HPLAI_EUNSUPPORTED;   // the matrix is regenerated, not stored
	const int n = c->n;
	HPLAI_CUDA_TRY(cudaMemcpy2DAsync(c->A, sizeof(float) * c->lda, a, sizeof(float) * lda, sizeof(float) * n, n,
		cudaMemcpyHostToDevice, c->st));
	HPLAI_CUDA_TRY(cudaMemcpyAsync(c->rhs, rhs, sizeof(double) * n, cudaMemcpyHostToDevice, c->st));
	HPLAI_CUDA_TRY(cudaMemcpyAsync(c->d, diag, sizeof(double) * n, cudaMemcpyHostToDevice, c->st));
	c->seed = seed;
	c->regen_a = false;
	HPLAI_TRY(compute_norms(c));
	c->have_inputs = true;
	c->factored = false;
	return HPLAI_OK;
}

namespace {

// The precision form forms its panels on FP16 tensor cores when the store
// epilogue's 16-byte row alignment holds (b a multiple of 4), else in TF32.
bool f16_panel_form(const hplai_ctx *c, bool simt)
{
	return !simt && c->precision == HPLAI_F32_F8 && c->b % 4 == 0;
}

// The plain form's panels by substitution on the CUDA cores, both in one
// launch, while they are small: the tensor-core path's inverses, splits and
// products are seven or more dependent launches that a small panel does not
// fill.  Measured (tensor cores / one launch): b = 60, 600 rows 42 / 11 us,
// 9600 43 / 31, 39960 69 / 86; b = 128, 9600 48 / 45, 19968 56 / 76; b = 256,
// 2304 71 / 36, 9472 79 / 83; b = 512, 1536 104 / 96, 2048 109 / 94, 4608
// 118 / 189.  In wider blocks the substitution's chain alone takes longer:
// b = 640, 640 rows 131 / 137; 768 145 / 189; 1024 178 / 315.
bool pair_panel_form(const hplai_ctx *c, int rem)
{
	return c->precision == HPLAI_F32_F16 && c->b <= 512 && static_cast<int64_t>(rem) * c->b <= 1200000;
}

// Factor the diagonal block of step k and form its two panels with their
// FP16 copies in slot `slot` of group buffer `buf` (getrf_nopiv +
// update_left/right_panels + convert_left/right_panels,
// panel_trf.hpp:143-233).  Precision form: the e4m3 copies for the next
// update that reads this panel -- with one-panel groups this panel's own; in
// a group's earlier slots the panel's single copy, for the updates of the
// group's later blocks; in its last slot the group's shared copy of all its
// panels.
int panel_step(hplai_ctx *c, int k, int buf, int slot, bool simt, int side_ctas, cudaStream_t st, PhaseEvents &pe)
{
	const int n = c->n, b = c->b;
	const int64_t lda = c->lda, ldg = c->ldg;
	const int64_t kb = static_cast<int64_t>(k) * b;
	float *diag = c->A + kb + kb * lda;
	HPLAI_TRY(pe.record(st, HPLAI_PH_DIAG_LU));
	HPLAI_TRY(launch_getrf_tiles(b, diag, lda, c->getrf_work, &c->getrf_epoch, side_ctas, st));
	if (k == c->nb - 1) return pe.end(st);
	HPLAI_TRY(pe.next(st, HPLAI_PH_TRSM_L));
	const int rem = n - static_cast<int>(kb) - b;
	const bool f16_panels = f16_panel_form(c, simt);
	const uint16_t *deck = f16_panels ? c->deck : nullptr;   // folded into the FP16 panel copies
	const float inv_dscale = c->deck ? 1.0f / c->dscale : 0.f;
	uint16_t *lslot = c->Lh[buf] + slot * c->ldh, *uslot = c->Uh[buf] + slot * c->ldh;
	// FP16 panel products: their stores gather the e4m3 copies' block maxima
	// (this panel's own copy; with groups also the group's shared copy, whose
	// blocks start (G - 1 - slot) b below this panel's first row / column)
	const int G = c->group;
	AmaxTargets al, au;
	al.dim = 0;
	au.dim = 1;
	if (f16_panels) {
		const size_t nbw = sizeof(unsigned) * (n / 128 + 2);
		const bool own = G == 1 || slot < G - 1;
		if (own) {
			HPLAI_CUDA_TRY(cudaMemsetAsync(c->qb[0], 0, nbw, st));
			HPLAI_CUDA_TRY(cudaMemsetAsync(c->qb[1], 0, nbw, st));
			al.bits[0] = c->qb[0];
			au.bits[0] = c->qb[1];
		}
		if (G > 1) {
			if (slot == 0) {
				HPLAI_CUDA_TRY(cudaMemsetAsync(c->qb[2], 0, nbw, st));
				HPLAI_CUDA_TRY(cudaMemsetAsync(c->qb[3], 0, nbw, st));
			}
			al.bits[1] = c->qb[2];
			au.bits[1] = c->qb[3];
			al.base[1] = au.base[1] = (G - 1 - slot) * b;
		}
	}
	if (simt) {
		HPLAI_TRY(launch_trsm_right_upper(rem, b, diag, lda, diag + b, lda, lslot + (kb + b) * ldg, ldg, 1.0f, st));
	} else if (f16_panels) {
		// FP16 panel products (the Schur update reads only the e4m3 copies made below)
		HPLAI_TRY(launch_tri_inverses(c->tc, diag, lda, st, false));
		// A not stored: the block column regenerated into the (otherwise unused)
		// TF32 split buffer, column-major with leading dimension n
		const float *src = nullptr;
		if (c->deck_aliased) {
			HPLAI_TRY(launch_fill(n, static_cast<int>(kb) + b, static_cast<int>(kb), rem, b, c->tcbuf, n, c->seed, 0, st));
			src = c->tcbuf;
		}
		HPLAI_TRY(launch_lpanel_f16(c->tc, c->maps[buf][slot], static_cast<int>(kb), rem, c->A, lda, lslot, uslot, ldg,
			deck, c->deck_ld, inv_dscale, side_ctas, st, src, n, &al));
	} else if (pair_panel_form(c, rem)) {
		// both panels and their FP16 copies, timed as TRSM_L
		HPLAI_TRY(launch_trsm_pair(rem, b, diag, diag + b, diag + static_cast<int64_t>(b) * lda, lda, lslot + (kb + b) * ldg,
			uslot + (kb + b) * ldg, ldg, st));
		return pe.end(st);
	} else {
		HPLAI_TRY(launch_tri_inverses(c->tc, diag, lda, st));
		// the precision form's Schur update reads the e4m3 copies only: no FP16 copy
		uint16_t *lh = c->precision == HPLAI_F32_F8 ? nullptr : lslot + (kb + b) * ldg;
		HPLAI_TRY(launch_lpanel_tc(c->tc, rem, diag + b, lda, lh, ldg, 1.0f, side_ctas, st));
	}
	HPLAI_TRY(pe.next(st, HPLAI_PH_TRSM_R));
	if (simt) {
		HPLAI_TRY(launch_trsm_left_lower(b, rem, diag, lda, diag + static_cast<int64_t>(b) * lda, lda,
			uslot + (kb + b) * ldg, ldg, 1.0f, st));
	} else if (f16_panels) {
		// the block row likewise (b x rem, leading dimension the split buffer's ldp)
		const float *src = nullptr;
		const int64_t ldp = (b + 31) / 32 * 32;
		if (c->deck_aliased) {
			HPLAI_TRY(launch_fill(n, static_cast<int>(kb), static_cast<int>(kb) + b, b, rem, c->tcbuf, ldp, c->seed, 0, st));
			src = c->tcbuf;
		}
		HPLAI_TRY(launch_upanel_f16(c->tc, c->maps[buf][slot], static_cast<int>(kb), rem, c->A, lda, uslot, ldg, deck,
			c->deck_ld, inv_dscale, side_ctas, st, src, ldp, &au));
	} else {
		uint16_t *uh = c->precision == HPLAI_F32_F8 ? nullptr : uslot + (kb + b) * ldg;
		HPLAI_TRY(launch_upanel_tc(c->tc, rem, diag + static_cast<int64_t>(b) * lda, lda, uh, ldg, 1.0f, side_ctas, st));
	}
	if (c->precision == HPLAI_F32_F8) {
		// the block maxima: gathered by the FP16 panel stores, else the copy's own pass
		const bool ready = f16_panels;
		unsigned *bl = ready ? c->qb[0] : c->qbits, *bu = ready ? c->qb[1] : c->qbits;
		if (G == 1) {
			HPLAI_TRY(launch_quantize_lpanel(rem, b, diag + b, lda, bl, c->L8[buf] + (kb + b) * c->ld8g, c->ld8g,
				c->sl[buf], st, false, ready));
			HPLAI_TRY(launch_quantize_upanel(rem, b, diag + static_cast<int64_t>(b) * lda, lda, bu,
				c->U8[buf] + (kb + b) * c->ld8g, c->ld8g, c->su[buf], st, false, ready));
		} else if (slot < G - 1) {
			// the panel alone, for the updates of the group's later blocks
			HPLAI_TRY(launch_quantize_lpanel(rem, b, diag + b, lda, bl, c->L8s[slot] + (kb + b) * c->ld8, c->ld8,
				c->sls[slot], st, false, ready));
			HPLAI_TRY(launch_quantize_upanel(rem, b, diag + static_cast<int64_t>(b) * lda, lda, bu,
				c->U8s[slot] + (kb + b) * c->ld8, c->ld8, c->sus[slot], st, false, ready));
		} else {
			// the group's last panel: [L_k-G+1 .. L_k] (rows kb+b.., A columns
			// kb-(G-1)b .. kb+b-1) and [U_k-G+1; ..; U_k] (A rows kb-(G-1)b ..
			// kb+b-1, columns kb+b..) with factors over all the group's panels
			const int64_t back = static_cast<int64_t>(G - 1) * b;
			HPLAI_TRY(launch_quantize_lpanel(rem, G * b, diag + b - back * lda, lda, ready ? c->qb[2] : c->qbits,
				c->L8[buf] + (kb + b) * c->ld8g, c->ld8g, c->sl[buf], st, false, ready));
			HPLAI_TRY(launch_quantize_upanel(rem, G * b, diag - back + static_cast<int64_t>(b) * lda, lda,
				ready ? c->qb[3] : c->qbits, c->U8[buf] + (kb + b) * c->ld8g, c->ld8g, c->su[buf], st, false, ready));
		}
	}
	HPLAI_TRY(pe.end(st));
	return HPLAI_OK;
}

// The operands of one trailing update: FP16 maps, or e4m3 maps with their
// factors (block 0 of sl/su starting at row/column s0).
struct Operands {
	const SchurMaps *m = nullptr;
	bool fp8 = false;
	const float *sl = nullptr, *su = nullptr;
	int s0 = 0;
};

// C -= L U on the rectangle of rows [r0, r1) and columns [c0, c1).
int schur_region(hplai_ctx *c, const Operands &op, int r0, int r1, int c0, int c1, int max_ctas, cudaStream_t st,
	PhaseEvents &pe)
{
	if (r1 <= r0 || c1 <= c0) return HPLAI_OK;
	HPLAI_TRY(pe.record(st, HPLAI_PH_GEMM_UPDATE));
	float *cp = c->A + r0 + static_cast<int64_t>(c0) * c->lda;
	if (c->deck)
		HPLAI_TRY(launch_schur_deck(*op.m, op.fp8, op.sl, op.s0, op.su, op.s0, r0, c0, r1 - r0, c1 - c0, r0, c0,
			c->dscale, max_ctas, st));
	else if (op.fp8)
		HPLAI_TRY(launch_schur_fp8(*op.m, op.sl, op.s0, op.su, op.s0, r0, c0, r1 - r0, c1 - c0, cp, c->lda, r0, c0,
			max_ctas, st));
	else
		HPLAI_TRY(launch_schur(*op.m, r0, c0, r1 - r0, c1 - c0, cp, c->lda, r0, c0, max_ctas, st));
	HPLAI_TRY(pe.end(st));
	return HPLAI_OK;
}

// The operands of the update by the whole group in buffer q whose first
// trailing row/column is e * b.
Operands group_operands(const hplai_ctx *c, int q, int e)
{
	Operands op;
	op.fp8 = c->precision == HPLAI_F32_F8;
	const int g = c->group == 4 ? 1 : 0;
	if (op.fp8) {
		op.m = c->group > 1 ? &c->maps8g[q][g] : &c->maps8[q];
		op.sl = c->sl[q];
		op.su = c->su[q];
		op.s0 = e * c->b;
	} else {
		op.m = c->group > 1 ? &c->mapsg[q][g] : &c->maps[q][0];
	}
	return op;
}

// The operands of the update by one panel of a group alone: the panel in
// slot h of buffer q, of the group whose first block is e (its e4m3 copy's
// rows start below its own block, at (e + h + 1) b).
Operands slot_operands(const hplai_ctx *c, int q, int e, int h)
{
	Operands op;
	op.fp8 = c->precision == HPLAI_F32_F8;
	if (op.fp8) {
		op.m = &c->maps8s[h];
		op.sl = c->sls[h];
		op.su = c->sus[h];
		op.s0 = (e + h + 1) * c->b;
	} else {
		op.m = &c->maps[q][h];
	}
	return op;
}

// Everything block j needs before it is factored, on the side stream: with
// panel groups the updates of the group's block j by the group's earlier
// panels (first .. j-1, each alone); then, with the FP16 deck, the deck folded into the block column and
// row (A + deck / dscale; the FP16 panel copies fold the off-diagonal part
// themselves, so then only the diagonal block).
int prepare_block(hplai_ctx *c, int j, int first, int q, bool simt, int side_ctas, cudaStream_t st, PhaseEvents &pe)
{
	const int n = c->n, b = c->b;
	const int r1 = j * b, r2 = (j + 1) * b;
	// the updates of block j by the group's earlier panels, in panel order
	for (int h = 0; h < j - first; ++h) {
		const Operands op = slot_operands(c, q, first, h);
		HPLAI_TRY(schur_region(c, op, r1, n, r1, r2, side_ctas, st, pe));
		HPLAI_TRY(schur_region(c, op, r1, r2, r2, n, side_ctas, st, pe));
	}
	if (c->deck_aliased) {
		// the diagonal block formed from the LCG and its deck, staged first:
		// near the matrix end its FP32 rows overlay its own deck rows
		HPLAI_TRY(pe.record(st, HPLAI_PH_LAZY_INIT));
		HPLAI_CUDA_TRY(cudaMemcpy2DAsync(c->dstage, sizeof(uint16_t) * b, c->deck + r1 + static_cast<int64_t>(r1) * c->deck_ld,
			sizeof(uint16_t) * c->deck_ld, sizeof(uint16_t) * b, b, cudaMemcpyDeviceToDevice, st));
		HPLAI_TRY(launch_lazy_init(n, r1, r2, r1, r2, c->A, c->lda, c->dstage, nullptr, b, r1, r1, 1.0f / c->dscale,
			c->seed, c->d, true, st));
		HPLAI_TRY(pe.end(st));
	} else if (c->deck && j > 0) {
		HPLAI_TRY(pe.record(st, HPLAI_PH_LAZY_INIT));
		if (f16_panel_form(c, simt)) {
			HPLAI_TRY(launch_deck_apply(r1, r2, r1, r2, c->A, c->lda, c->deck, c->lda, 1.0f / c->dscale, st));
		} else {
			HPLAI_TRY(launch_deck_apply(r1, n, r1, r2, c->A, c->lda, c->deck, c->lda, 1.0f / c->dscale, st));
			HPLAI_TRY(launch_deck_apply(r1, r2, r2, n, c->A, c->lda, c->deck, c->lda, 1.0f / c->dscale, st));
		}
		HPLAI_TRY(pe.end(st));
	}
	return HPLAI_OK;
}

} // namespace

namespace {

// The reference's `-d` LU bit for bit (HPLAI_FLAG_REF_DECK): the steps of
// RDMAPanelLU::run<Matgen, 1, true, false> (panel_trf.hpp:703-856) on one
// stream.  Step k: lazy initialisation of the diagonal block, its LU, lazy
// initialisation + TRSM of the block column (FP16 copy scaled by scalea) and
// of the block row (scale 1), then the FP16-accumulating update of the deck
// by panel k.  Every element sees the updates of the panels before it in
// panel order, as in the reference's split schedule.  With kend < nb the
// last panel's update is not applied (the warm-up, panel_trf.hpp:726).
int factor_refdeck(hplai_ctx *c, int kend)
{
	const int n = c->n, b = c->b, nb = c->nb;
	const int64_t lda = c->lda, ldg = c->ldg;
	cudaStream_t st = c->st;
	for (double &v : c->phase_ms) v = 0.0;
	PhaseEvents pe(c->phase_events);
	HPLAI_CUDA_TRY(cudaMemsetAsync(c->rdeck, 0, sizeof(uint16_t) * static_cast<size_t>(lda) * n, st));
	if (c->rback) HPLAI_CUDA_TRY(cudaMemsetAsync(c->rback, 0, sizeof(uint16_t) * static_cast<size_t>(lda) * n, st));
	HPLAI_CUDA_TRY(cudaMemsetAsync(c->getrf_work, 0, sizeof(uint32_t), st));   // its status word
	// pmatgen0 (matgen.hpp:81-105): the blocks a warm-up leaves unformed hold zero
	if (c->regen_a) HPLAI_CUDA_TRY(cudaMemsetAsync(c->A, 0, sizeof(float) * static_cast<size_t>(lda) * n, st));
	auto lazy = [&](int r0, int r1, int c0, int c1) -> int {
		HPLAI_TRY(pe.record(st, HPLAI_PH_LAZY_INIT));
		HPLAI_TRY(launch_lazy_init(n, r0, r1, c0, c1, c->A, lda, c->rdeck, c->rback, lda, 0, 0, c->rdownscale, c->seed,
			c->d, c->regen_a, st));
		return pe.end(st);
	};
	const int steps = std::min(kend, nb);
	for (int k = 0; k < steps; ++k) {
		const int kb = k * b;
		float *diag = c->A + kb + static_cast<int64_t>(kb) * lda;
		HPLAI_TRY(lazy(kb, kb + b, kb, kb + b));
		HPLAI_TRY(pe.record(st, HPLAI_PH_DIAG_LU));
		HPLAI_TRY(launch_getrf_tiles(b, diag, lda, c->getrf_work, &c->getrf_epoch, 0, st));
		HPLAI_TRY(pe.end(st));
		if (k == nb - 1) break;
		const int rem = n - kb - b;
		uint16_t *lh = c->Lh[0] + static_cast<int64_t>(kb + b) * ldg, *uh = c->Uh[0] + static_cast<int64_t>(kb + b) * ldg;
		HPLAI_TRY(lazy(kb + b, n, kb, kb + b));
		HPLAI_TRY(pe.record(st, HPLAI_PH_TRSM_L));
		HPLAI_TRY(launch_trsm_right_upper(rem, b, diag, lda, diag + b, lda, lh, ldg, c->rscalea, st));
		HPLAI_TRY(pe.end(st));
		HPLAI_TRY(lazy(kb, kb + b, kb + b, n));
		HPLAI_TRY(pe.record(st, HPLAI_PH_TRSM_R));
		HPLAI_TRY(launch_trsm_left_lower(b, rem, diag, lda, diag + static_cast<int64_t>(b) * lda, lda, uh, ldg, 1.0f, st));
		HPLAI_TRY(pe.end(st));
		if (k == kend - 1 && kend < nb) break;
		// BackBuffer::write_back at the end of the reference's iteration k
		// (BB_NCYCLE = 32), before panel k's update, which it applies in k+1
		if (c->rback && k >= 1 && (k - 1) % 32 == 31) {
			HPLAI_TRY(pe.record(st, HPLAI_PH_WRITE_BACK));
			HPLAI_TRY(launch_backbuf_writeback(n, kb + b, c->rdeck, c->rback, lda, st));
			HPLAI_TRY(pe.end(st));
		}
		HPLAI_TRY(pe.record(st, HPLAI_PH_GEMM_UPDATE));
		HPLAI_TRY(launch_hgemm_deck(rem, rem, b, lh, ldg, uh, ldg, c->rdeck + (kb + b) + static_cast<int64_t>(kb + b) * lda,
			lda, st));
		HPLAI_TRY(pe.end(st));
	}
	HPLAI_TRY(pe.record(st, HPLAI_PH_IR_TRSV));
	HPLAI_TRY(launch_trsv_dinv(n, c->A, lda, c->dinv, st));
	HPLAI_TRY(pe.end(st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	pe.collect(c->phase_ms);
	int gs = HPLAI_OK;
	HPLAI_TRY(getrf_status(c->getrf_work, st, &gs));
	HPLAI_TRY(gs);
	c->factored = true;
	return HPLAI_OK;
}

// The factorisation of panels 0 .. kend-1 (kend = nb: the whole LU).  With
// kend < nb (the benchmark warm-up) the updates of panels 0 .. kend-2 are
// applied, as in the reference, whose loop applies panel k-1's update in
// iteration k (RDMAPanelLU::run, panel_trf.hpp:726-850).
int factor_impl(hplai_ctx *c, int kend, const float *host_a = nullptr, int64_t host_lda = 0)
{
	if (!c) return HPLAI_EINVAL;
	if (!c->have_inputs) return HPLAI_ESTATE;
	if (c->flags & HPLAI_FLAG_REF_DECK) return factor_refdeck(c, kend);
	const int n = c->n, b = c->b, nb = c->nb;
	c->group = kend < nb ? 1
		: ((c->flags & HPLAI_FLAG_GROUP4) && c->gcap >= 4) ? 4
		: ((c->flags & HPLAI_FLAG_GROUP2) && c->gcap >= 2) ? 2 : 1;
	const int G = c->group;
	HPLAI_CUDA_TRY(cudaMemsetAsync(c->kstatus, 0, 2 * sizeof(unsigned), c->st));
	if (c->deck_aliased)
		HPLAI_CUDA_TRY(cudaMemset2DAsync(c->deck, sizeof(uint16_t) * c->deck_ld, 0, sizeof(uint16_t) * n, n, c->st));
	else if (c->deck)
		HPLAI_CUDA_TRY(cudaMemsetAsync(c->deck, 0, sizeof(uint16_t) * static_cast<size_t>(c->lda) * n, c->st));
	HPLAI_CUDA_TRY(cudaMemsetAsync(c->getrf_work, 0, sizeof(uint32_t), c->st));   // its status word
	const bool simt = (c->flags & HPLAI_FLAG_SIMT_PANELS) != 0;
	const bool serial = (c->flags & HPLAI_FLAG_LOOKAHEAD) == 0;
	for (double &v : c->phase_ms) v = 0.0;
	PhaseEvents pe(c->phase_events, serial);
	// Right-looking blocked LU without pivoting with look-ahead
	// (panel_lu_async / RDMAPanelLU::run, panel_trf.hpp:434-858), by groups
	// of G panels.  The update by group [s, s+G) of the trailing matrix
	// (rows and columns from e = s+G blocks on) is split into the next
	// group's block columns and rows (first) and the rest (after).  The next
	// group's panels are formed once the first part is done: block by block,
	// the group's second block first receiving its first panel's update.
	// With HPLAI_FLAG_LOOKAHEAD they are formed on the side stream while the
	// main stream applies the rest, which then leaves side_sms SMs to the
	// side stream.  Where nothing overlaps (one stream, or a share above one
	// half) the update is one launch, ahead of the panels: the thin regions
	// fill a fraction of the 128 x 256 tiles.
	cudaStream_t st = c->st, sd = serial ? c->st : c->st2;
	int sms = 148;
	{
		int dev = 0;
		if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	}
	// SMs left to the side stream while it forms the panels of the group
	// starting at block e: a fixed count (side_sms > 0) or, with side_sms < 0,
	// a share of c = -side_sms panels against the remaining trailing blocks,
	// sms * c / (rem / b + c): the panel work grows with rem, the update with
	// rem^2, so the side stream needs more SMs as the matrix shrinks.  With a
	// share above one half nothing overlaps: the update in one launch, then the
	// group's panels on the whole GPU (b % 4 != 0: the panels before the rest of
	// the split update).  0: no overlap.
	auto side_for = [&](int e) -> int {
		if (serial) return 0;
		int side = c->side_sms;
		if (side < 0) {
			const double cp = -side, rb = static_cast<double>(n - e * b) / b;
			side = static_cast<int>(std::lround(sms * cp / (rb + cp)));
			if (side < 8) side = 8;
		}
		return (2 * side > sms) ? 0 : side;
	};
	// With a host source (the FP16 deck form only: the updates go to the deck,
	// so block column and row j of A are first read when panel j is formed)
	// the matrix is copied panel by panel on a copy stream, block column j
	// (rows jb..n) and block row j (columns (j+1)b..n) before event j, and
	// panel j's preparation waits for that event.
	if (host_a) {
		const int64_t lda = c->lda;
		HPLAI_CUDA_TRY(cudaEventRecord(c->ev_next, st));   // the deck's zeroing and the step's inputs
		HPLAI_CUDA_TRY(cudaStreamWaitEvent(c->st3, c->ev_next, 0));
		for (int j = 0; j < nb; ++j) {
			const int64_t jb = static_cast<int64_t>(j) * b;
			HPLAI_CUDA_TRY(cudaMemcpy2DAsync(c->A + jb + jb * lda, sizeof(float) * lda, host_a + jb + jb * host_lda,
				sizeof(float) * host_lda, sizeof(float) * (n - jb), b, cudaMemcpyHostToDevice, c->st3));
			if (jb + b < n)
				HPLAI_CUDA_TRY(cudaMemcpy2DAsync(c->A + jb + (jb + b) * lda, sizeof(float) * lda,
					host_a + jb + (jb + b) * host_lda, sizeof(float) * host_lda, sizeof(float) * b, n - jb - b,
					cudaMemcpyHostToDevice, c->st3));
			HPLAI_CUDA_TRY(cudaEventRecord(c->ev_copy[j], c->st3));
		}
	}
	auto wait_copy = [&](int j) -> int {
		if (host_a) {
			HPLAI_CUDA_TRY(cudaStreamWaitEvent(sd, c->ev_copy[j], 0));
			pe.waited = true;   // the wait for the copy belongs to no phase
		}
		return HPLAI_OK;
	};
	// the side stream starts from the generated matrix: group 0's panels
	HPLAI_CUDA_TRY(cudaEventRecord(c->ev_next, st));
	HPLAI_CUDA_TRY(cudaStreamWaitEvent(sd, c->ev_next, 0));
	for (int j = 0; j < G && j < nb && j < kend; ++j) {
		HPLAI_TRY(wait_copy(j));
		HPLAI_TRY(prepare_block(c, j, 0, 0, simt, 0, sd, pe));
		HPLAI_TRY(panel_step(c, j, 0, j, simt, 0, sd, pe));
	}
	for (int s = 0; s + G < nb && (kend >= nb || s + 1 < kend); s += G) {
		const int q = (s / G) & 1;
		const int e = s + G, ne = std::min(G, nb - e);
		const int r1 = e * b, r2 = (e + ne) * b;
		const Operands op = group_operands(c, q, e);
		const int side = side_for(e);
		const int side_ctas = side, main_ctas = side ? sms - side : 0;
		HPLAI_CUDA_TRY(cudaEventRecord(c->ev_panel, sd));
		HPLAI_CUDA_TRY(cudaStreamWaitEvent(st, c->ev_panel, 0));
		const bool whole = side == 0 && b % 4 == 0;
		if (whole) {
			// nothing to overlap with: the whole trailing matrix in one launch
			// (rows of every region on 16-byte boundaries, so that its elements
			// see the same epilogue as in the split update)
			HPLAI_TRY(schur_region(c, op, r1, n, r1, n, 0, st, pe));
		} else {
			// the next group's block columns (rows r1..n) and block rows (columns r2..n)
			HPLAI_TRY(schur_region(c, op, r1, n, r1, r2, 0, st, pe));
			HPLAI_TRY(schur_region(c, op, r1, r2, r2, n, 0, st, pe));
		}
		HPLAI_CUDA_TRY(cudaEventRecord(c->ev_next, st));
		HPLAI_CUDA_TRY(cudaStreamWaitEvent(sd, c->ev_next, 0));
		for (int j = e; j < e + ne && j < kend; ++j) {
			HPLAI_TRY(wait_copy(j));
			HPLAI_TRY(prepare_block(c, j, e, q ^ 1, simt, side_ctas, sd, pe));
			HPLAI_TRY(panel_step(c, j, q ^ 1, j - e, simt, side_ctas, sd, pe));
		}
		if (!whole && !serial && side == 0) {
			// no overlap for this group: its panels first, on the whole GPU
			HPLAI_CUDA_TRY(cudaEventRecord(c->ev_panel, sd));
			HPLAI_CUDA_TRY(cudaStreamWaitEvent(st, c->ev_panel, 0));
		}
		// the rest of the trailing matrix
		if (!whole) HPLAI_TRY(schur_region(c, op, r2, n, r2, n, main_ctas, st, pe));
	}
	HPLAI_CUDA_TRY(cudaEventRecord(c->ev_panel, sd));
	HPLAI_CUDA_TRY(cudaStreamWaitEvent(st, c->ev_panel, 0));
	// inverses of the factors' 128 x 128 diagonal blocks for the refinement's
	// solves, in one launch of all blocks (0.03 ms at n = 8192, 0.2 at 65536)
	// and not on the chain of the panels
	HPLAI_TRY(pe.record(st, HPLAI_PH_IR_TRSV));
	HPLAI_TRY(launch_trsv_dinv(n, c->A, c->lda, c->dinv, st));
	HPLAI_TRY(pe.end(st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	pe.collect(c->phase_ms);
	{
		unsigned ks[2] = {0, 0};
		HPLAI_CUDA_TRY(cudaMemcpyAsync(ks, c->kstatus, sizeof ks, cudaMemcpyDeviceToHost, st));
		HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
		if (ks[0] || ks[1]) return HPLAI_ETIMEOUT;
	}
	{
		int gs = HPLAI_OK;
		HPLAI_TRY(getrf_status(c->getrf_work, st, &gs));
		HPLAI_TRY(gs);
	}
	c->factored = true;
	return HPLAI_OK;
}

} // namespace

extern "C" int hplai_factor(hplai_ctx *c) { return c ? factor_impl(c, c->nb) : HPLAI_EINVAL; }

extern "C" int hplai_factor_steps(hplai_ctx *c, int steps)
{
	if (!c || steps < 0) return HPLAI_EINVAL;
	return factor_impl(c, std::min(steps, c->nb));
}

extern "C" int hplai_l1est(hplai_ctx *c)
{
	if (!c) return HPLAI_EINVAL;
	if (!c->have_inputs) return HPLAI_ESTATE;
	for (double &v : c->phase_ms) v = 0.0;
	if (c->matrix == HPLAI_MATRIX_HIGHAM) {
		// pmatl1est with HMGen (matgen.hpp:147-192): Higham's matrix is L U with
		// constant strictly triangular parts, so the "approximation" is exact
		HPLAI_TRY(launch_higham_fill(c->n, c->h_alpha, c->h_beta, c->A, c->lda, nullptr, true, c->st));
		HPLAI_TRY(launch_trsv_dinv(c->n, c->A, c->lda, c->dinv, c->st));
		HPLAI_CUDA_TRY(cudaStreamSynchronize(c->st));
		c->factored = true;
		return HPLAI_OK;
	}
	if (c->regen_a) {
		// --l1est stores A even with `-d` (pmatgen, main.cpp:260-263)
		HPLAI_TRY(launch_fill(c->n, 0, 0, c->n, c->n, c->A, c->lda, c->seed, 0, c->st));
		HPLAI_TRY(launch_diag(c->n, 0, c->n, nullptr, c->A, c->lda, c->seed, c->st));
	}
	HPLAI_TRY(launch_l1est(c->n, c->A, c->lda, c->d, c->st));
	HPLAI_TRY(launch_trsv_dinv(c->n, c->A, c->lda, c->dinv, c->st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(c->st));
	c->factored = true;
	return HPLAI_OK;
}

namespace {

int ensure_gmres_buffers(hplai_ctx *c)
{
	const int m = c->gm_restart;
	if (c->gm_v && c->gm_cap >= m) return HPLAI_OK;
	cudaFree(c->gm_v);
	cudaFree(c->gm_z);
	cudaFree(c->gm_w);
	cudaFree(c->gm_small);
	c->gm_v = c->gm_z = c->gm_w = c->gm_small = nullptr;
	c->gm_ldv = round_up(c->n, 32);
	HPLAI_CUDA_TRY(cudaMalloc(&c->gm_v, sizeof(double) * c->gm_ldv * (m + 1)));
	HPLAI_CUDA_TRY(cudaMalloc(&c->gm_z, sizeof(double) * c->gm_ldv * m));
	HPLAI_CUDA_TRY(cudaMalloc(&c->gm_w, sizeof(double) * c->gm_ldv));
	HPLAI_CUDA_TRY(cudaMalloc(&c->gm_small, sizeof(double) * (kDotBlocks * kMaxBasis + kMaxBasis * kMaxBasis +
		2 * kMaxBasis)));
	c->gm_cap = m;
	return HPLAI_OK;
}

// r <- M^{-1} r with M = L U, the FP32 factors applied to an FP64 vector
// (panel_trsvL / panel_trsvU, panel_trsv.hpp:310-758); trans: r <- M^{-T} r,
// U^T first, then L^T.
int apply_lu_inverse(hplai_ctx *c, double *v, PhaseEvents &pe, bool trans)
{
	cudaStream_t st = c->st;
	HPLAI_TRY(pe.record(st, HPLAI_PH_IR_TRSV));
	HPLAI_TRY(launch_trsv(true, c->n, c->A, c->lda, v, c->trsv_work, c->trsv_bytes, st, trans, c->dinv));
	HPLAI_TRY(launch_trsv(false, c->n, c->A, c->lda, v, c->trsv_work, c->trsv_bytes, st, trans, c->dinv));
	HPLAI_TRY(pe.end(st));
	return HPLAI_OK;
}

// The classical correction: x += U^{-1} L^{-1} r (iterative_refinement.hpp:50-53).
int correct_ir(hplai_ctx *c, double *x, PhaseEvents &pe, bool trans)
{
	HPLAI_TRY(apply_lu_inverse(c, c->r, pe, trans));
	HPLAI_TRY(launch_axpy1(c->n, c->r, x, c->st));
	return HPLAI_OK;
}

// The GMRES correction: one cycle of GMRES(m) from d = 0, x += d, either
// right-preconditioned (flexible: A M^{-1} u = r with the vectors
// z_j = M^{-1} v_j kept, d = Z y) or left-preconditioned (M^{-1} A d =
// M^{-1} r).  CGS2 orthogonalisation on the device, Givens rotations and the
// small triangular solve on the host.  Stops at |g_{j+1}| <= tol * beta
// (beta = ||r||_2, or ||M^{-1} r||_2 when left) or after m steps.
int correct_gmres(hplai_ctx *c, double *x, PhaseEvents &pe, int *inner, bool trans)
{
	const int n = c->n, m = c->gm_restart;
	const int64_t ldv = c->gm_ldv;
	cudaStream_t st = c->st;
	double *part = c->gm_small, *H = part + kDotBlocks * kMaxBasis, *tmp = H + kMaxBasis * kMaxBasis,
	       *yd = tmp + kMaxBasis;
	double *V = c->gm_v, *w = c->gm_w, *Z = c->gm_z;
	const bool right = c->gm_right != 0;
	*inner = 0;
	// left: z = M^{-1} r, beta = ||z||, v_0 = z / beta; right: beta = ||r||, v_0 = r / beta
	if (!right) HPLAI_TRY(apply_lu_inverse(c, c->r, pe, trans));
	HPLAI_TRY(launch_dots(n, 1, c->r, ldv, c->r, part, tmp, 2, st));
	HPLAI_TRY(launch_scale(n, c->r, tmp, V, st));
	double beta = 0.0;
	HPLAI_CUDA_TRY(cudaMemcpyAsync(&beta, tmp, sizeof beta, cudaMemcpyDeviceToHost, st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	if (!(beta > 0.0) || !std::isfinite(beta)) return beta == 0.0 ? HPLAI_OK : HPLAI_ENOTCONV;
	std::vector<double> R(static_cast<size_t>(m) * m, 0.0), cs(m), sn(m), g(m + 1, 0.0), h(m + 1);
	g[0] = beta;
	int k = 0;
	for (int j = 0; j < m; ++j) {
		double *vj = V + j * ldv, *vn = V + (j + 1) * ldv, *hc = H + j * kMaxBasis;
		if (right) {
			// z_j = M^{-1} v_j, w = A z_j (A regenerated in FP64)
			double *zj = Z + j * ldv;
			HPLAI_CUDA_TRY(cudaMemcpyAsync(zj, vj, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
			HPLAI_TRY(apply_lu_inverse(c, zj, pe, trans));
			HPLAI_TRY(pe.record(st, HPLAI_PH_IR_GEMV));
			HPLAI_TRY(matvec(c, 1.0, zj, 0.0, w, st, trans));
			HPLAI_TRY(pe.end(st));
		} else {
			// w = M^{-1} A v_j, A regenerated in FP64
			HPLAI_TRY(pe.record(st, HPLAI_PH_IR_GEMV));
			HPLAI_TRY(matvec(c, 1.0, vj, 0.0, w, st, trans));
			HPLAI_TRY(pe.end(st));
			HPLAI_TRY(apply_lu_inverse(c, w, pe, trans));
		}
		// two Gram-Schmidt sweeps against v_0..v_j; ||w|| after the second
		HPLAI_TRY(launch_dots(n, j + 1, V, ldv, w, part, hc, 0, st));
		HPLAI_TRY(launch_gs_update(n, j + 1, V, ldv, hc, w, part, nullptr, st));
		HPLAI_TRY(launch_dots(n, j + 1, V, ldv, w, part, tmp, 0, st));
		HPLAI_TRY(launch_gs_update(n, j + 1, V, ldv, tmp, w, part, hc + j + 1, st));
		HPLAI_TRY(launch_add_small(j + 1, tmp, hc, st));
		HPLAI_TRY(launch_scale(n, w, hc + j + 1, vn, st));
		HPLAI_CUDA_TRY(cudaMemcpyAsync(h.data(), hc, sizeof(double) * (j + 2), cudaMemcpyDeviceToHost, st));
		HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
		++*inner;
		for (int i = 0; i < j; ++i) {
			const double t = cs[i] * h[i] + sn[i] * h[i + 1];
			h[i + 1] = -sn[i] * h[i] + cs[i] * h[i + 1];
			h[i] = t;
		}
		const double rho = std::hypot(h[j], h[j + 1]);
		if (!(rho > 0.0) || !std::isfinite(rho)) break;
		cs[j] = h[j] / rho;
		sn[j] = h[j + 1] / rho;
		h[j] = rho;
		g[j + 1] = -sn[j] * g[j];
		g[j] = cs[j] * g[j];
		for (int i = 0; i <= j; ++i) R[static_cast<size_t>(j) * m + i] = h[i];
		k = j + 1;
		if (std::fabs(g[j + 1]) <= c->gm_tol * beta) break;
	}
	if (k == 0) return HPLAI_ENOTCONV;
	// R y = g, R upper triangular (column j at R[j*m])
	std::vector<double> y(k);
	for (int i = k - 1; i >= 0; --i) {
		double s = g[i];
		for (int j = i + 1; j < k; ++j) s -= R[static_cast<size_t>(j) * m + i] * y[j];
		y[i] = s / R[static_cast<size_t>(i) * m + i];
	}
	HPLAI_CUDA_TRY(cudaMemcpyAsync(yd, y.data(), sizeof(double) * k, cudaMemcpyHostToDevice, st));
	HPLAI_TRY(launch_combine(n, k, right ? Z : V, ldv, yd, x, st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	return HPLAI_OK;
}

} // namespace

extern "C" int hplai_set_gmres(hplai_ctx *c, int restart, double tol)
{
	if (!c || restart < 1 || restart > kMaxBasis - 1 || !(tol > 0.0) || !(tol < 1.0)) return HPLAI_EINVAL;
	c->gm_restart = restart;
	c->gm_tol = tol;
	return HPLAI_OK;
}

extern "C" int hplai_set_gmres_side(hplai_ctx *c, int right)
{
	if (!c || (right != 0 && right != 1)) return HPLAI_EINVAL;
	c->gm_right = right;
	return HPLAI_OK;
}

extern "C" int hplai_get_refine_counts(hplai_ctx *c, int *outer, int *inner)
{
	if (!c) return HPLAI_EINVAL;
	if (outer) *outer = static_cast<int>(c->log_resid.size());
	if (inner) *inner = c->gm_inner;
	return HPLAI_OK;
}

namespace {

// Iterative refinement of op(A) x = rhs (op = identity or transpose) with
// the context's factors: x_0 = rhs ./ diag(A), then residuals with A
// regenerated in FP64 and classical or GMRES corrections until the
// hpl-harness (scaled by ||A||_inf and ||rhs||_inf) is below 16
// (iterative_refinement.hpp:18-57).
int refine_core(hplai_ctx *c, int mode, bool trans, const double *rhs, double normb, double *x, int maxit,
	hplai_ir_errors *err, int *iters)
{
	const int n = c->n;
	cudaStream_t st = c->st;
	c->log_resid.clear();
	c->log_harness.clear();
	c->gm_inner = 0;
	if (err) *err = hplai_ir_errors{-1.0, -1.0};
	if (iters) *iters = 0;
	if (mode == HPLAI_GMRES) HPLAI_TRY(ensure_gmres_buffers(c));
	HPLAI_TRY(trsv_status_reset(c->trsv_work, st));
	PhaseEvents pe(c->phase_events);
	// x_0 = b ./ diag(A)   (iterative_refinement.hpp:31-34)
	HPLAI_TRY(launch_div(n, rhs, c->d, x, st));
	int rc = HPLAI_ENOTCONV;
	bool checked = true;   // the last correction's solves are known to have finished
	for (int it = 0; it < maxit; ++it) {
		// r = b - A x with A regenerated in FP64 (panel_gemv(-1, ..., 1, r)), and
		// ||x||_inf and ||r||_inf from the same pass
		HPLAI_TRY(pe.record(st, HPLAI_PH_IR_GEMV));
		HPLAI_TRY(matvec(c, -1.0, x, 1.0, c->r, st, trans, rhs, c->scal + 2));
		HPLAI_TRY(pe.end(st));
		double h[3];
		HPLAI_CUDA_TRY(cudaMemcpyAsync(h, c->scal + 2, sizeof h, cudaMemcpyDeviceToHost, st));
		HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
		checked = true;
		if (h[2] != 0.0) return HPLAI_ETIMEOUT;   // of the correction before
		const double normx = h[0], normr = h[1];
		// iterative_refinement.hpp:43
		const double hpl = normr / std::fma(c->norma, normx, normb) * 1. / (n * DBL_EPSILON / 2);
		c->log_resid.push_back(normr);
		c->log_harness.push_back(hpl);
		if (iters) *iters = it + 1;
		if (hpl < 16.) {
			if (err) *err = hplai_ir_errors{normr, hpl};
			rc = HPLAI_OK;
			break;
		}
		if (!std::isfinite(hpl)) break;
		checked = false;
		if (mode == HPLAI_IR) {
			HPLAI_TRY(correct_ir(c, x, pe, trans));
		} else {
			int in = 0;
			const int gr = correct_gmres(c, x, pe, &in, trans);
			c->gm_inner += in;
			if (gr != HPLAI_OK) break;
		}
	}
	uint32_t late = 0;
	if (!checked)
		HPLAI_CUDA_TRY(cudaMemcpyAsync(&late, trsv_status_word(c->trsv_work), sizeof late, cudaMemcpyDeviceToHost, st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	if (late) return HPLAI_ETIMEOUT;
	double tmp[HPLAI_PH_COUNT] = {};
	pe.collect(tmp);
	c->phase_ms[HPLAI_PH_IR_GEMV] = tmp[HPLAI_PH_IR_GEMV];
	c->phase_ms[HPLAI_PH_IR_TRSV] = tmp[HPLAI_PH_IR_TRSV];
	return rc;
}

// A solve with a caller's right-hand side (host vectors): rhs -> device,
// refine, x -> host.  Uses the scratch vectors rhs2/x2, not the context's
// own rhs and x.
int solve_vector(hplai_ctx *c, bool trans, const double *b, double *x, int maxit, hplai_ir_errors *err, int *iters)
{
	if (!c || !b || !x || maxit < 0) return HPLAI_EINVAL;
	if (!c->factored) return HPLAI_ESTATE;
	const int n = c->n;
	cudaStream_t st = c->st;
	if (!c->rhs2) {
		HPLAI_CUDA_TRY(cudaMalloc(&c->rhs2, sizeof(double) * n));
		HPLAI_CUDA_TRY(cudaMalloc(&c->x2, sizeof(double) * n));
	}
	HPLAI_CUDA_TRY(cudaMemcpyAsync(c->rhs2, b, sizeof(double) * n, cudaMemcpyHostToDevice, st));
	HPLAI_TRY(launch_infnorm(n, c->rhs2, c->scal + 4, st));
	double normb = 0.0;
	HPLAI_CUDA_TRY(cudaMemcpyAsync(&normb, c->scal + 4, sizeof normb, cudaMemcpyDeviceToHost, st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	const int mode = c->precision == HPLAI_F32_F8 ? HPLAI_GMRES : HPLAI_IR;
	const int rc = refine_core(c, mode, trans, c->rhs2, normb, c->x2, maxit, err, iters);
	if (rc != HPLAI_OK && rc != HPLAI_ENOTCONV) return rc;
	HPLAI_CUDA_TRY(cudaMemcpyAsync(x, c->x2, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	return rc;
}

} // namespace

// Right-hand side `col` of the stream (column n + col), solved with the
// context's factors into x (host, n doubles).  For the batched solver.
int hplai_ctx_solve_stream_rhs(hplai_ctx *c, int col, double *x, int maxit, hplai_ir_errors *err, int *iters)
{
	if (!c || !x || col < 0 || maxit < 0) return HPLAI_EINVAL;
	if (!c->factored) return HPLAI_ESTATE;
	const int n = c->n;
	cudaStream_t st = c->st;
	if (!c->rhs2) {
		HPLAI_CUDA_TRY(cudaMalloc(&c->rhs2, sizeof(double) * n));
		HPLAI_CUDA_TRY(cudaMalloc(&c->x2, sizeof(double) * n));
	}
	const double *rhs = c->rhs;
	double normb = c->normb;
	if (col > 0) {
		HPLAI_TRY(launch_rhs_cols(n, col, 1, c->rhs2, c->seed, st));
		HPLAI_TRY(launch_infnorm(n, c->rhs2, c->scal + 4, st));
		HPLAI_CUDA_TRY(cudaMemcpyAsync(&normb, c->scal + 4, sizeof normb, cudaMemcpyDeviceToHost, st));
		HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
		rhs = c->rhs2;
	}
	const int mode = c->precision == HPLAI_F32_F8 ? HPLAI_GMRES : HPLAI_IR;
	const int rc = refine_core(c, mode, false, rhs, normb, c->x2, maxit, err, iters);
	if (rc != HPLAI_OK && rc != HPLAI_ENOTCONV) return rc;
	HPLAI_CUDA_TRY(cudaMemcpyAsync(x, c->x2, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(st));
	return rc;
}

// The project's own tuner in place of lda_tuner (lda_tuner.hpp:9-45, whose
// call the reference leaves commented out): the factorisation is timed on
// this context (regenerated from `seed` before each trial) under each
// schedule -- one- or two-panel groups (the trailing update's K = b or 2b),
// serial or with look-ahead at several side-stream SM counts -- after one
// discarded warm-up factorisation; the two fastest are timed twice more and
// the one with the lowest median becomes the context's schedule.  Every
// trial is kept for hplai_get_autotune_log.
namespace {

// Every set of Schur maps of the context.
template <class F>
void for_each_maps(hplai_ctx *c, F &&f)
{
	for (int i = 0; i < 2; ++i) {
		for (auto &m : c->maps[i]) f(m);
		for (auto &m : c->mapsg[i]) f(m);
		f(c->maps8[i]);
		for (auto &m : c->maps8g[i]) f(m);
	}
	for (auto &m : c->maps8s) f(m);
}

// The tile order of every Schur launch of the context (trailing updates and
// panel products): groups of `gm` tile rows (0: the kernel's default).
void apply_tile_group(hplai_ctx *c, int gm)
{
	c->tile_group = gm;
	for_each_maps(c, [gm](SchurMaps &m) { m.group_m = gm; });
}

// Deck updates on CTA pairs for every Schur launch of the context (1 on, 0
// off, -1 the library default).
void apply_cta_pairs(hplai_ctx *c, int v)
{
	c->cta_pairs = v;
	for_each_maps(c, [v](SchurMaps &m) { m.pairs = v; });
}

} // namespace

extern "C" int hplai_set_tile_group(hplai_ctx *c, int group_m)
{
	if (!c || group_m < 0 || group_m > 1024) return HPLAI_EINVAL;
	apply_tile_group(c, group_m);
	return HPLAI_OK;
}

extern "C" int hplai_set_cta_pairs(hplai_ctx *c, int on)
{
	if (!c) {
		// the library default, for contexts left at -1 and the leaf calls
		if (on < 0) return HPLAI_EINVAL;
		schur_set_pairs_default(on != 0);
		return HPLAI_OK;
	}
	if (on < -1) return HPLAI_EINVAL;
	apply_cta_pairs(c, on > 0 ? 1 : on);
	return HPLAI_OK;
}

extern "C" int hplai_get_cta_pairs(hplai_ctx *c, int *on)
{
	if (!c || !on) return HPLAI_EINVAL;
	*on = c->cta_pairs;
	return HPLAI_OK;
}

extern "C" int hplai_get_tile_group(hplai_ctx *c, int *group_m)
{
	if (!c || !group_m) return HPLAI_EINVAL;
	*group_m = c->tile_group > 0 ? c->tile_group : 32;
	return HPLAI_OK;
}

extern "C" int hplai_autotune(hplai_ctx *c, uint64_t seed, unsigned *flags_out, int *side_sms_out, double *ms_out)
{
	if (!c) return HPLAI_EINVAL;
	if (c->flags & HPLAI_FLAG_REF_DECK) return HPLAI_EUNSUPPORTED;   // one fixed schedule
	int sms = 148;
	{
		int dev = 0;
		if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	}
	struct Cand {
		unsigned sched;   // HPLAI_FLAG_LOOKAHEAD | HPLAI_FLAG_GROUP2 | HPLAI_FLAG_GROUP4 bits
		int side;
		std::vector<double> ms;
		int tg = 0;       // tile group (0: the kernel's default)
		int pairs = -2;   // deck updates on CTA pairs for the trial (-2: the context's setting)
	};
	std::vector<Cand> cands;
	for (int g : {1, 2, 4}) {
		if (g > c->gcap) break;
		const unsigned gf = g == 4 ? HPLAI_FLAG_GROUP4 : g == 2 ? HPLAI_FLAG_GROUP2 : 0u;
		cands.push_back({gf, 20, {}});
		for (int side : {16, 32})
			if (sms > 2 * side) cands.push_back({gf | HPLAI_FLAG_LOOKAHEAD, side, {}});
		// side-stream share growing as the trailing matrix shrinks (four-panel
		// groups give the side stream twice the panels per update: larger shares)
		static const std::vector<int> shares2 = {8, 16, 24}, shares4 = {16, 20, 24, 28, 32};
		for (int share : (g == 4 ? shares4 : shares2)) cands.push_back({gf | HPLAI_FLAG_LOOKAHEAD, -share, {}});
	}
	const int tg0 = c->tile_group, pairs0 = c->cta_pairs;
	const unsigned sched_bits = HPLAI_FLAG_LOOKAHEAD | HPLAI_FLAG_GROUP2 | HPLAI_FLAG_GROUP4;
	const unsigned flags0 = c->flags, base_flags = c->flags & ~sched_bits;
	const int side0 = c->side_sms;
	cudaEvent_t e0 = nullptr, e1 = nullptr;
	HPLAI_CUDA_TRY(cudaEventCreate(&e0));
	HPLAI_CUDA_TRY(cudaEventCreate(&e1));
	c->tune_log.clear();
	auto trial = [&](const Cand &t, double *ms) -> int {
		c->flags = base_flags | t.sched;
		c->side_sms = t.side;
		apply_tile_group(c, t.tg);
		apply_cta_pairs(c, t.pairs == -2 ? pairs0 : t.pairs);
		HPLAI_TRY(hplai_generate(c, seed));
		HPLAI_CUDA_TRY(cudaEventRecord(e0, c->st));
		HPLAI_TRY(hplai_factor(c));
		HPLAI_CUDA_TRY(cudaEventRecord(e1, c->st));
		HPLAI_CUDA_TRY(cudaEventSynchronize(e1));
		float f = 0.f;
		HPLAI_CUDA_TRY(cudaEventElapsedTime(&f, e0, e1));
		*ms = f;
		c->tune_log.push_back({c->flags | (t.pairs == 1 ? HPLAI_TRIAL_CTA_PAIRS : 0u), t.side, f, t.tg > 0 ? t.tg : 32});
		return HPLAI_OK;
	};
	auto median = [](std::vector<double> v) {
		std::sort(v.begin(), v.end());
		return v[v.size() / 2];
	};
	int rc = HPLAI_OK;
	double warm = 0.0;
	rc = trial(cands[0], &warm);   // discarded: first-touch and module loading
	for (size_t i = 0; i < cands.size() && rc == HPLAI_OK; ++i) {
		double ms = 0.0;
		rc = trial(cands[i], &ms);
		cands[i].ms.push_back(ms);
	}
	if (rc == HPLAI_OK) {
		std::vector<size_t> order(cands.size());
		for (size_t i = 0; i < order.size(); ++i) order[i] = i;
		std::sort(order.begin(), order.end(), [&](size_t a, size_t b) { return cands[a].ms[0] < cands[b].ms[0]; });
		for (size_t r = 0; r < std::min<size_t>(2, order.size()) && rc == HPLAI_OK; ++r)
			for (int rep = 0; rep < 2 && rc == HPLAI_OK; ++rep) {
				double ms = 0.0;
				rc = trial(cands[order[r]], &ms);
				cands[order[r]].ms.push_back(ms);
			}
	}
	size_t pick = 0;
	double best = -1.0;
	for (size_t i = 0; rc == HPLAI_OK && i < cands.size(); ++i) {
		if (cands[i].ms.size() < 3) continue;   // only the re-timed finalists
		const double m = median(cands[i].ms);
		if (best < 0.0 || m < best) {
			best = m;
			pick = i;
		}
	}
	// then the tile order of the chosen schedule: groups of 16 or 64 tile rows
	// instead of 32, kept only when both of their trials beat the schedule's
	// median by half a percent
	int tg_pick = 0;
	for (int tg : {16, 64}) {
		if (rc != HPLAI_OK) break;
		Cand t = cands[pick];
		t.tg = tg;
		double a = 0.0, b2 = 0.0;
		rc = trial(t, &a);
		if (rc == HPLAI_OK) rc = trial(t, &b2);
		if (rc == HPLAI_OK && std::max(a, b2) < 0.995 * best) {
			best = std::max(a, b2);
			tg_pick = tg;
		}
	}
	// then the tile shape of the deck updates with K >= 2048: 256 x 256 tiles
	// on CTA pairs instead of 128 x 256 on single CTAs, by the same rule
	bool pairs_pick = false;
	const bool deck_k2048 = c->deck && (cands[pick].sched & (HPLAI_FLAG_GROUP2 | HPLAI_FLAG_GROUP4)) &&
		(((cands[pick].sched & HPLAI_FLAG_GROUP4) ? 4 : 2) * c->b >= 2048);
	if (rc == HPLAI_OK && deck_k2048) {
		Cand t = cands[pick];
		t.tg = tg_pick;
		t.pairs = 1;
		double a = 0.0, b2 = 0.0;
		rc = trial(t, &a);
		if (rc == HPLAI_OK) rc = trial(t, &b2);
		if (rc == HPLAI_OK && std::max(a, b2) < 0.995 * best) {
			best = std::max(a, b2);
			pairs_pick = true;
		}
	}
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	if (rc != HPLAI_OK) {
		c->flags = flags0;
		c->side_sms = side0;
		apply_tile_group(c, tg0);
		apply_cta_pairs(c, pairs0);
		return rc;
	}
	c->flags = base_flags | cands[pick].sched;
	c->side_sms = cands[pick].side;
	apply_tile_group(c, tg_pick);
	apply_cta_pairs(c, pairs_pick ? 1 : pairs0);
	// the context is left generated and unfactored, as after hplai_generate
	HPLAI_TRY(hplai_generate(c, seed));
	if (flags_out) *flags_out = c->flags;
	if (side_sms_out) *side_sms_out = c->side_sms;
	if (ms_out) *ms_out = best;
	return HPLAI_OK;
}

extern "C" int hplai_set_schedule(hplai_ctx *c, unsigned flags, int side_sms)
{
	const unsigned sched = HPLAI_FLAG_LOOKAHEAD | HPLAI_FLAG_GROUP2 | HPLAI_FLAG_GROUP4;
	if (!c || (flags & ~sched) || side_sms == 0 || side_sms > 64 || side_sms < -256) return HPLAI_EINVAL;
	if ((flags & HPLAI_FLAG_GROUP2) && (flags & HPLAI_FLAG_GROUP4)) return HPLAI_EINVAL;
	if ((flags & HPLAI_FLAG_GROUP2) && c->gcap < 2) return HPLAI_EINVAL;
	if ((flags & HPLAI_FLAG_GROUP4) && c->gcap < 4) return HPLAI_EINVAL;
	if ((c->flags & HPLAI_FLAG_REF_DECK) && flags) return HPLAI_EINVAL;
	c->flags = (c->flags & ~sched) | flags;
	c->side_sms = side_sms;
	return HPLAI_OK;
}

extern "C" int hplai_get_autotune_trials(hplai_ctx *c, unsigned *flags, int *side_sms, int *tile_group, double *ms,
	int cap, int *count)
{
	if (!c || !count || cap < 0) return HPLAI_EINVAL;
	*count = static_cast<int>(c->tune_log.size());
	for (int i = 0; i < cap && i < *count; ++i) {
		if (flags) flags[i] = c->tune_log[i].flags;
		if (side_sms) side_sms[i] = c->tune_log[i].side_sms;
		if (tile_group) tile_group[i] = c->tune_log[i].tile_group;
		if (ms) ms[i] = c->tune_log[i].ms;
	}
	return HPLAI_OK;
}

extern "C" int hplai_higham_params(int n, double cond, double rho, double *alpha, double *beta)
{
	if (!alpha || !beta) return HPLAI_EINVAL;
	const double b = higham_beta(n, cond, rho);
	if (!std::isfinite(b) || !(b > 0.)) return HPLAI_EINVAL;
	*beta = b;
	*alpha = rho * b;
	return HPLAI_OK;
}

extern "C" int hplai_set_matrix(hplai_ctx *c, int kind, double cond, double rho)
{
	if (!c) return HPLAI_EINVAL;
	if (kind == HPLAI_MATRIX_LCG) {
		c->matrix = kind;
	} else if (kind == HPLAI_MATRIX_HIGHAM) {
		// the `-d` parity mode and the lazy form regenerate the LCG matrix at panel time
		if (c->flags & (HPLAI_FLAG_REF_DECK | HPLAI_FLAG_LAZY_A)) return HPLAI_EUNSUPPORTED;
		double a = 0.0, b = 0.0;
		HPLAI_TRY(hplai_higham_params(c->n, cond, rho, &a, &b));
		c->matrix = kind;
		c->h_alpha = a;
		c->h_beta = b;
	} else {
		return HPLAI_EINVAL;
	}
	c->have_inputs = false;
	c->factored = false;
	return HPLAI_OK;
}

extern "C" int hplai_get_autotune_log(hplai_ctx *c, unsigned *flags, int *side_sms, double *ms, int cap, int *count)
{
	if (!c) return HPLAI_EINVAL;
	const int m = static_cast<int>(c->tune_log.size());
	for (int i = 0; i < m && i < cap; ++i) {
		if (flags) flags[i] = c->tune_log[i].flags;
		if (side_sms) side_sms[i] = c->tune_log[i].side_sms;
		if (ms) ms[i] = c->tune_log[i].ms;
	}
	if (count) *count = m;
	return HPLAI_OK;
}

extern "C" int hplai_refine(hplai_ctx *c, int mode, int maxit, hplai_ir_errors *err, int *iters)
{
	if (!c || maxit < 0) return HPLAI_EINVAL;
	if (!c->factored) return HPLAI_ESTATE;
	if (mode != HPLAI_IR && mode != HPLAI_GMRES) return HPLAI_EUNSUPPORTED;
	return refine_core(c, mode, false, c->rhs, c->normb, c->x, maxit, err, iters);
}

extern "C" int hplai_solve_rhs(hplai_ctx *c, const double *b, double *x, int maxit, hplai_ir_errors *err, int *iters)
{
	return solve_vector(c, false, b, x, maxit, err, iters);
}

extern "C" int hplai_solve_transpose(hplai_ctx *c, const double *g, double *lambda, int maxit, hplai_ir_errors *err,
	int *iters)
{
	return solve_vector(c, true, g, lambda, maxit, err, iters);
}

extern "C" int hplai_get_x(hplai_ctx *c, double *x)
{
	if (!c || !x) return HPLAI_EINVAL;
	HPLAI_CUDA_TRY(cudaMemcpyAsync(x, c->x, sizeof(double) * c->n, cudaMemcpyDeviceToHost, c->st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(c->st));
	return HPLAI_OK;
}

extern "C" int hplai_get_lu(hplai_ctx *c, float *a, int64_t lda)
{
	if (!c || !a || lda < c->n) return HPLAI_EINVAL;
	HPLAI_CUDA_TRY(cudaMemcpy2DAsync(a, sizeof(float) * lda, c->A, sizeof(float) * c->lda, sizeof(float) * c->n, c->n,
		cudaMemcpyDeviceToHost, c->st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(c->st));
	return HPLAI_OK;
}

extern "C" int hplai_checksum(hplai_ctx *c, double *sigs)
{
	if (!c || !sigs) return HPLAI_EINVAL;
	double *dsig = static_cast<double *>(c->check_work);
	HPLAI_TRY(launch_panel_check(c->n, c->A, c->lda, dsig, dsig + 3, panel_check_workspace(c->n), c->st));
	HPLAI_CUDA_TRY(cudaMemcpyAsync(sigs, dsig, 3 * sizeof(double), cudaMemcpyDeviceToHost, c->st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(c->st));
	return HPLAI_OK;
}

extern "C" int hplai_get_rhs(hplai_ctx *c, double *rhs)
{
	if (!c || !rhs) return HPLAI_EINVAL;
	HPLAI_CUDA_TRY(cudaMemcpyAsync(rhs, c->rhs, sizeof(double) * c->n, cudaMemcpyDeviceToHost, c->st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(c->st));
	return HPLAI_OK;
}

extern "C" int hplai_get_diag(hplai_ctx *c, double *diag)
{
	if (!c || !diag) return HPLAI_EINVAL;
	HPLAI_CUDA_TRY(cudaMemcpyAsync(diag, c->d, sizeof(double) * c->n, cudaMemcpyDeviceToHost, c->st));
	HPLAI_CUDA_TRY(cudaStreamSynchronize(c->st));
	return HPLAI_OK;
}

extern "C" int hplai_get_ir_log(hplai_ctx *c, double *residual, double *harness, int cap, int *count)
{
	if (!c) return HPLAI_EINVAL;
	const int m = static_cast<int>(c->log_resid.size());
	for (int i = 0; i < m && i < cap; ++i) {
		if (residual) residual[i] = c->log_resid[i];
		if (harness) harness[i] = c->log_harness[i];
	}
	if (count) *count = m;
	return HPLAI_OK;
}

extern "C" int hplai_get_phase_ms(hplai_ctx *c, double *ms, int count)
{
	if (!c || !ms) return HPLAI_EINVAL;
	double total = 0.0;
	for (int i = 0; i < HPLAI_PH_COUNT; ++i)
		if (i != HPLAI_PH_TOTAL) total += c->phase_ms[i];
	for (int i = 0; i < count && i < HPLAI_PH_COUNT; ++i) ms[i] = (i == HPLAI_PH_TOTAL) ? total : c->phase_ms[i];
	return HPLAI_OK;
}

extern "C" void *hplai_get_stream(hplai_ctx *c) { return c ? static_cast<void *>(c->st) : nullptr; }

extern "C" int hplai_get_norms(hplai_ctx *c, double *norma, double *normb)
{
	if (!c) return HPLAI_EINVAL;
	if (norma) *norma = c->norma;
	if (normb) *normb = c->normb;
	return HPLAI_OK;
}

extern "C" int hplai_solve_host(hplai_ctx *c, const float *a, int64_t lda, const double *rhs, const double *diag,
	uint64_t seed, int maxit, double *x, hplai_ir_errors *err, int *iters)
{
	if (!c || !a || !rhs || !diag || !x || lda < c->n) return HPLAI_EINVAL;
	if (c->flags & HPLAI_FLAG_LAZY_A) return HPLAI_EUNSUPPORTED;   // the matrix is regenerated, not stored
	// With the FP16 deck and a page-locked matrix the copy runs behind the
	// factorisation (each panel waits for its own block column and row);
	// otherwise the whole matrix is copied first.
	cudaPointerAttributes pa{};
	const bool pinned = cudaPointerGetAttributes(&pa, a) == cudaSuccess && pa.type == cudaMemoryTypeHost;
	(void)cudaGetLastError();
	if (c->deck && pinned) {
		const int n = c->n;
		if (!c->st3) HPLAI_CUDA_TRY(cudaStreamCreateWithFlags(&c->st3, cudaStreamNonBlocking));
		while (static_cast<int>(c->ev_copy.size()) < c->nb) {
			cudaEvent_t e;
			HPLAI_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
			c->ev_copy.push_back(e);
		}
		HPLAI_CUDA_TRY(cudaMemcpyAsync(c->rhs, rhs, sizeof(double) * n, cudaMemcpyHostToDevice, c->st));
		HPLAI_CUDA_TRY(cudaMemcpyAsync(c->d, diag, sizeof(double) * n, cudaMemcpyHostToDevice, c->st));
		c->seed = seed;
		HPLAI_TRY(compute_norms(c));
		c->have_inputs = true;
		c->factored = false;
		HPLAI_TRY(factor_impl(c, c->nb, a, lda));
	} else {
		HPLAI_TRY(hplai_upload(c, a, lda, rhs, diag, seed));
		HPLAI_TRY(hplai_factor(c));
	}
	const int rc = hplai_refine(c, c->precision == HPLAI_F32_F8 ? HPLAI_GMRES : HPLAI_IR, maxit, err, iters);
	if (rc != HPLAI_OK && rc != HPLAI_ENOTCONV) return rc;
	HPLAI_TRY(hplai_get_x(c, x));
	return rc;
}

extern "C" int hplai_format_report(int n, double seconds, hplai_ir_errors err, char *buf, size_t len)
{
	if (!buf || !len || seconds <= 0.0) return HPLAI_EINVAL;
	// main.cpp:440-452
	const double hplflops = 2. / 3 * n * static_cast<double>(n) * n + 3. / 2 * n * static_cast<double>(n);
	std::snprintf(buf, len, "%.9f sec. %.9f GFlop/s resid = %20.15e hpl-harness = %.9f", seconds,
		hplflops / seconds * 1e-9, err.residual, err.hpl_harness);
	return HPLAI_OK;
}
