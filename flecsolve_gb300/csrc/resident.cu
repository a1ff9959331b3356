// Whole solves in one cooperative launch (resident.cuh): FP64 Jacobi-CG on a
// grid stencil.
//
// The recurrences, the scalar tests and the state a solve leaves behind are
// those of the kernel-per-phase loop (krylov.cu; the reference's cg.hh:43-139).
//
// Bound: the FP64 pipe issues a warp instruction per SM in 19 cycles, and an
// iteration needs 14 per 32 rows (SpMV 7, p'Ap 1, update 5, direction 1).  At
// 77^3 (3,008 rows a CTA) that is 25,000 of the 39,000 cycles an iteration
// takes; the reductions with the CTAs' skew and the scalars take the rest.  At
// 128^2 (128 rows, 11,600 cycles) the two reductions take about 3,500 each, the
// SpMV 1,500 (mostly the packets' latency), the scalars 2,000, update and
// direction 1,500.
#include <cmath>
#include <cstring>

#include "resident.cuh"

namespace fsg {

namespace {

struct ResCg {
	ResGrid<double> A;
	const double *dinv;       // null: no preconditioner
	const double *b;
	double *x, *r, *p, *w;    // global vectors (r, w: used where smem is short)
	ulonglong2 *pk;           // p as packets (PKT)
	KState *st;
	double *hist;
	ResSlots *slots;
	unsigned *err;
	double rtol;
	int maxiter, hist_cap, zero_guess;
	int rows;                 // rows per CTA
	int smem;                 // dynamic shared memory, bytes
	int lost;
};

// PKT: the slice's p fits in shared memory and the other slices read it as
// packets; otherwise p is a global vector and the direction step ends with a
// grid-wide publication.
template<int K, bool GEN, bool PKT>
__global__ void __launch_bounds__(kResThreads, 1)
k_cg_resident(ResCg a) {
	extern __shared__ __align__(16) unsigned char dyn[];
	__shared__ ResShared sh;
	// the solve's scalars, thread 0's (the same in every CTA)
	struct Scalars {
		double tol, tol2, rho, rho_inv, rho_old, pap, rr, rr0, rhs_norm, sol0, beta, xx;
		int it, status, info_iters, flags;
		int turn;  // CTA that keeps the next entry of the history
	};
	__shared__ Scalars z;
	if ((int)blockIdx.x == a.lost)
		return;  // a test of the others' waits
	ResTeam tm;
	tm.init(a.slots, &sh, a.err);
	const int tid = threadIdx.x, nt = blockDim.x;
	const int lo = (int)min((int64_t)blockIdx.x * a.rows, (int64_t)a.A.n);
	const int cnt = (int)min((int64_t)a.rows, (int64_t)a.A.n - lo);
	// the slice's arrays, in order of their accesses per iteration
	ResSmem sm{dyn, a.smem};
	unsigned char *mask = sm.take<unsigned char>(a.rows);
	auto place = [&](double *g) {
		double *q = sm.take<double>(a.rows);
		return q ? q : g;
	};
	double *pl = PKT ? sm.take<double>(a.rows) : a.p + lo;
	double *r = place(a.r + lo), *w = place(a.w + lo);
	double *x = place(a.x + lo);
	double *dv = a.dinv ? sm.take<double>(a.rows) : nullptr;
	const double *dinv = dv ? dv : a.dinv ? a.dinv + lo : nullptr;
	ResRows<double, K, GEN> A;
	A.ld = a.A.ld;
	A.lo = lo;
	A.cnt = cnt;
	A.d[0] = 1;
	A.d[1] = a.A.nx;
	A.d[2] = a.A.nx * a.A.ny;
	A.mask = mask;
	A.G = a.A.S + a.A.ld;
	auto coef = [&](int slot) -> const double * {
		const double *g = a.A.S + (int64_t)slot * a.A.ld + lo;
		double *q = sm.take<double>(a.rows);
		if (q)
			for (int l = tid; l < cnt; l += nt)
				q[l] = g[l];
		return q ? q : g;
	};
	A.D = coef(0);
#pragma unroll
	for (int t = 0; t < K; ++t)
		A.U[t] = coef(1 + t);
	if (GEN)
#pragma unroll
		for (int t = 0; t < K; ++t)
			A.L[t] = coef(1 + K + t);
	for (int l = tid; l < cnt; l += nt) {
		mask[l] = (unsigned char)res_mask<K>(lo + l, a.A.nx, a.A.ny, a.A.nz);
		if (dv)
			dv[l] = a.dinv[lo + l];
	}
	__syncthreads();

	// p of the own row l: to the slice and to the others
	auto put_p = [&](int l, double v) {
		pl[l] = v;
		if constexpr (PKT)
			res_st16(a.pk + (lo + l), (unsigned long long)__double_as_longlong(v), tm.epoch);
	};
	// r = b - A x (b for a zero guess), z = P r, p = z; ||b||, ||x||, ||r||,
	// r'z (cg.hh:55-90)
	double s4[4] = {0.0, 0.0, 0.0, 0.0};
	for (int l = tid; l < cnt; l += nt) {
		const double bi = a.b[lo + l];
		double ri = bi, xi = 0.0;
		if (!a.zero_guess) {
			xi = a.x[lo + l];
			ri = bi - A.template sum<false>(l, a.x + lo, a.x, nullptr, 0, tm);
		}
		const double zi = dinv ? dinv[l] * ri : ri;
		r[l] = ri;
		put_p(l, zi);
		s4[0] = fma(bi, bi, s4[0]);
		s4[1] = fma(xi, xi, s4[1]);
		s4[2] = fma(ri, ri, s4[2]);
		s4[3] = fma(zi, ri, s4[3]);
	}
	unsigned long long tag = tm.epoch;  // of the packets of p
	const double s0 = tm.grid_sum<4, !PKT>(s4);
	if (tid < 128 && (tid & 31) == 0)
		sh.bc[tid >> 5] = s0;
	bool alive = tm.done();
	if (tid == 0) {
		z = Scalars{};
		z.rhs_norm = sqrt(sh.bc[0]);
		if (z.rhs_norm == 0.0)
			z.rhs_norm = 1.0;
		z.tol = a.rtol * z.rhs_norm;
		z.tol2 = res_threshold(z.tol);
		z.sol0 = a.zero_guess ? 0.0 : sh.bc[1];
		z.rr0 = z.rr = sh.bc[2];
		z.rho = z.rho_old = sh.bc[3];
		z.rho_inv = 1.0 / z.rho;
		z.status = FS_STATUS_UNKNOWN;
		if (z.rr <= z.tol2) {
			z.status = FS_CONVERGED_RTOL;
			sh.stop = 1;
		}
		else if (a.maxiter <= 0) {
			z.status = FS_DIVERGED_ITERS;
			sh.stop = 1;
		}
	}
	__syncthreads();
	// x may be a.x itself (no room in shared memory): first written here,
	// after every slice has read its neighbours' rows of the guess
	if (alive)
		for (int l = tid; l < cnt; l += nt)
			x[l] = a.zero_guess ? 0.0 : a.x[lo + l];

	while (alive && !sh.stop) {
		// w = A p, p'Ap -> alpha = rho / p'Ap (cg.hh:94-106)
		double s1[1] = {0.0};
		res_rows<2>(
			cnt, [&](int l) { return A.template sum<PKT>(l, pl, a.p, a.pk, tag, tm); },
			[&](int l, double s) {
				w[l] = s;
				s1[0] = fma(s, pl[l], s1[0]);
			});
		const double pap = tm.grid_sum<1, false>(s1);
		if (tid == 32)
			z.rho_inv = 1.0 / z.rho;  // for beta; this warp has no message to carry
		if (tid == 0) {
			sh.bc[0] = res_divide(z.rho, pap);
			z.pap = pap;
			const long long sign = __double_as_longlong(pap);
			if (!(sign > 0 && sign <= 0x7ff0000000000000ll))  // !(pap > 0)
				z.flags |= KF_NEG_CURVATURE;
		}
		if (!(alive = tm.done()))
			break;
		// x += alpha p, r -= alpha w, z = P r (kept in w), ||r||, r'z
		// (cg.hh:108-123)
		const double alpha = sh.bc[0];
		double s2[2] = {0.0, 0.0};
		struct Row {
			double p, x, w, r, d;
		};
		res_rows<2>(
			cnt, [&](int l) { return Row{pl[l], x[l], w[l], r[l], dinv ? dinv[l] : 1.0}; },
			[&](int l, const Row &t) {
				x[l] = fma(alpha, t.p, t.x);
				const double ri = fma(-alpha, t.w, t.r);
				const double zi = dinv ? t.d * ri : ri;
				r[l] = ri;
				w[l] = zi;
				s2[0] = fma(ri, ri, s2[0]);
				s2[1] = fma(ri, zi, s2[1]);
			});
		const double sum = tm.grid_sum<2, false>(s2);
		if (tid == 32) {
			// beta = rho_new / rho; the reciprocal for the next one follows
			sh.bc[0] = z.beta = res_quotient(sum, z.rho, z.rho_inv);
			z.rho_old = z.rho;
			z.rho = sum;
		}
		if (tid == 0) {
			const double rr = sum;
			const int it = ++z.it;
			z.rr = rr;
			// each CTA keeps every gridDim-th entry of the history, its root
			// taken at the end
			const int turn = z.turn;
			if (it <= a.hist_cap && turn == (int)blockIdx.x)
				a.hist[it - 1] = rr;
			z.turn = turn + 1 < (int)gridDim.x ? turn + 1 : 0;
			const bool finite = res_finite(rr);
			if (!finite)
				z.flags |= KF_NONFINITE;
			if (finite && res_below(rr, z.tol2)) {
				sh.stop = 1;
				z.status = FS_CONVERGED_RTOL;
				z.info_iters = it;
			}
			else if (it >= a.maxiter || !finite) {
				sh.stop = 1;
				z.status = FS_DIVERGED_ITERS;
			}
		}
		if (!(alive = tm.done()))
			break;
		if (sh.stop)
			break;
		// p = beta p + z (cg.hh:124-130), handed to the other slices: they
		// have read the last p, which precedes their message of p'Ap
		const double beta = sh.bc[0];
		tag = tm.epoch;
		res_rows<2>(
			cnt, [&](int l) { return make_double2(pl[l], w[l]); },
			[&](int l, const double2 &t) { put_p(l, fma(beta, t.x, t.y)); });
		if constexpr (PKT) {
			__syncthreads();  // the slice's p, read by its other threads
			res_hold(clock64());
		}
		else {
			const double none[1] = {0.0};
			tm.grid_sum<1, true>(none);
			alive = tm.done();
		}
	}
	// the solution and its norm, the history's roots; the state as the
	// kernel-per-phase loop leaves it
	double sx[1] = {0.0};
	for (int l = tid; l < cnt; l += nt) {
		const double xi = x[l];
		a.x[lo + l] = xi;
		sx[0] = fma(xi, xi, sx[0]);
	}
	if (alive) {
		const double xx = tm.grid_sum<1, false>(sx);
		if (tid == 0)
			z.xx = xx;
		tm.done();
		const int nh = min(z.it, a.hist_cap);
		for (int64_t i = blockIdx.x + (int64_t)tid * gridDim.x; i < nh; i += (int64_t)nt * gridDim.x)
			a.hist[i] = sqrt(a.hist[i]);
	}
	if (blockIdx.x == 0 && tid == 0) {
		KState *st = a.st;
		st->bnorm = st->rhs_norm = z.rhs_norm;
		st->tol = z.tol;
		st->rtol = a.rtol;
		st->sol0 = sqrt(z.sol0);
		st->res0 = sqrt(z.rr0);
		st->res = sqrt(z.rr);
		st->rho = z.rho;
		st->rho_old = z.rho_old;
		st->pAp = z.pap;
		st->beta = z.beta;
		st->aux[2] = sqrt(z.xx);
		st->iter = z.it;
		st->done = 1;
		st->status = z.status;
		st->info_iters = z.info_iters;
		st->flags = z.flags;
		st->maxiter = a.maxiter;
		st->restarts = 0;
		st->hist_cap = a.hist_cap;
		st->nhist = z.it;
	}
	tm.finish();
}

// Rows up to which FP64 CG runs resident.  The gain falls from the launches'
// share of an iteration to the little that the vectors kept in shared memory
// save (us per iteration, kernel per phase -> resident): 18.5 -> 6.4 at 32^2,
// 20.8 -> 5.6 at 128^2, 34.1 -> 12.8 at 512^2, 48 -> 18.8 at 77^3, 57.2 -> 30.5
// at 96^3, 91.1 -> 63.8 at 128^3, 113.3 -> 93.8 at 144^3 (3.0 M rows).
// Beyond, one CTA per SM no longer hides the memory that does not fit.
constexpr int64_t kResCgRows = 3000000;
// Packets are used while the slice's mask and p, r, w and x fit in its shared
// memory (1.0 M rows on 152 SMs); past that the rows a slice needs from others
// are read from the global p through L1, several times each.
constexpr int kResPktArrays = 4;

}  // namespace

// FP64 CG; `taken` = 0 when the solve is not one for the resident kernel
int cg_apply_resident(Solver *s, Vec *b, Vec *x, fs_solve_info *info, int *taken) {
	*taken = 0;
	Ctx *ctx = s->ctx;
	ResCg a{};
	bool gen = false;
	if (s->diag || s->n > kResCgRows || !res_grid<double>(s->A, a.A, gen))
		return FS_OK;
	const int K = s->A->nsym;
	// mask, p, r, w, x, dinv and the diagonals, as far as they fit
	const int per_row = 1 + 8 * (5 + 1 + (gen ? 2 * K : K));
	using Kern = void (*)(ResCg);
	static const Kern kerns[2][2][3] = {
		{{k_cg_resident<1, false, false>, k_cg_resident<2, false, false>, k_cg_resident<3, false, false>},
	     {k_cg_resident<1, false, true>, k_cg_resident<2, false, true>, k_cg_resident<3, false, true>}},
		{{k_cg_resident<1, true, false>, k_cg_resident<2, true, false>, k_cg_resident<3, true, false>},
	     {k_cg_resident<1, true, true>, k_cg_resident<2, true, true>, k_cg_resident<3, true, true>}}};
	const int smem_max = std::min(res_smem_max(ctx, kerns[gen][0][K - 1]),
	                              res_smem_max(ctx, kerns[gen][1][K - 1]));
	const ResShape sh = res_shape(ctx, s->n, per_row, smem_max);
	if (sh.rows > smem_max)
		return FS_OK;
	// packets while the slice's p, r, w and x fit
	const bool pkt = (int64_t)sh.rows * (1 + 8 * kResPktArrays) <= smem_max;
	const Kern kern = kerns[gen][pkt][K - 1];
	if (!res_memory(s, pkt))
		return FS_OK;
	a.pk = pkt ? s->res_pk : nullptr;
	FS_TRY(solver_hist(s, std::max(1, s->set.base.maxiter)));
	a.dinv = s->dinv64();
	a.b = (const double *)b->d;
	a.x = (double *)x->d;
	a.r = s->w64[0];
	a.p = s->w64[1];
	a.w = s->w64[2];
	a.st = s->st;
	a.hist = s->hist;
	a.slots = s->res_slots;
	a.err = ctx->dev_err;
	a.lost = sh.grid > 1 ? s->res_lost - 1 : -1;
	a.rtol = (double)s->set.base.rtol;
	a.maxiter = s->set.base.maxiter;
	a.hist_cap = s->hist_cap;
	a.zero_guess = s->set.base.use_zero_guess != 0;
	a.rows = sh.rows;
	a.smem = sh.smem;
	FS_TRY(res_launch(ctx, kern, sh, a, "resident cg", taken));
	if (!*taken)
		return FS_OK;
	FS_TRY(res_read_state(s));
	const KState &h = *s->hst;
	s->hhist_count = std::min<int64_t>(h.iter, s->hist_cap);
	memset(info, 0, sizeof(*info));
	info->rhs_norm = (float)h.rhs_norm;
	info->sol_norm_initial = (float)h.sol0;
	info->res_norm_initial = (float)h.res0;
	info->sol_norm_final = (float)h.aux[2];
	info->res_norm_final = (float)h.res;
	info->status = h.status;
	info->iters = h.info_iters;
	if (h.iter > 0 && info->iters == 0)
		info->status = FS_DIVERGED_ITERS;  // cg.hh:135-136
	if (h.flags & KF_NONFINITE)
		return set_err(ctx, FS_ERR_NON_FINITE, "CG: non-finite residual norm");
	return FS_OK;
}

// no slot or packet carries the epoch a first launch starts from
static cudaError_t first_epoch(Solver *s, ResSlots *p) {
	return cudaMemsetAsync(&p->epoch, 1, 1, s->ctx->stream);
}

int res_read_state(Solver *s) {
	const int st = read_state(s);
	if (st != FS_OK) {
		cudaStream_t q = s->ctx->stream;
		cudaMemsetAsync(s->res_slots, 0, sizeof(ResSlots), q);
		first_epoch(s, s->res_slots);
		if (s->res_pk)
			cudaMemsetAsync(s->res_pk, 0, (size_t)s->n * sizeof(ulonglong2), q);
		if (s->res_vals)
			cudaMemsetAsync(s->res_vals, 0, s->res_vals_len, q);
		cudaGetLastError();
	}
	return st;
}

bool res_memory(Solver *s, bool packets) {
	// one buffer of zeroes; false (and no error left) when there is no room
	auto get = [&](size_t bytes) -> void * {
		void *p = nullptr;
		if (cudaMalloc(&p, bytes) != cudaSuccess) {
			cudaGetLastError();
			return nullptr;
		}
		s->bufs.push_back(p);
		return cudaMemsetAsync(p, 0, bytes, s->ctx->stream) == cudaSuccess ? p : nullptr;
	};
	if (!s->res_slots) {
		auto *p = (ResSlots *)get(sizeof(ResSlots));
		if (!p || first_epoch(s, p) != cudaSuccess)
			return false;
		s->res_slots = p;
	}
	if (packets && !s->res_pk)
		s->res_pk = (ulonglong2 *)get((size_t)s->n * sizeof(ulonglong2));
	return !packets || s->res_pk;
}

}  // namespace fsg
