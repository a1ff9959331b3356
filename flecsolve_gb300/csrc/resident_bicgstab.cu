// FP64 BiCGSTAB on a grid stencil in one cooperative launch (resident.cuh).
//
// The recurrences, tests and final state are those of the kernel-per-phase
// loop (krylov.cu; the reference's bicgstab.hh:39-187).  Five kernels and four
// reductions an iteration become three reductions: ||s||, which only decides
// the early exit, travels with t't and t's (an early exit has then multiplied
// once in vain).  The SpMV operands P p and P s are formed once per row and
// handed to the other slices as packets, where the gather of the SpMV kernels
// scales every neighbour again: 28 FP64 operations a row and iteration instead
// of 42, at 19 cycles per 32 rows and SM.
#include <cmath>
#include <cstring>

#include "resident.cuh"

namespace fsg {

namespace {

struct ResBi {
	ResGrid<double> A;
	const double *dinv;       // null: no preconditioner
	const double *b;
	double *x, *r, *rt, *p, *v, *t;  // global vectors, used where smem is short
	ulonglong2 *pk;
	KState *st;
	double *hist;
	ResSlots *slots;
	unsigned *err;
	double rtol;
	int maxiter, hist_cap, zero_guess;
	int rows, smem, lost;
};

template<int K, bool GEN>
__global__ void __launch_bounds__(kResThreads, 1)
k_bi_resident(ResBi a) {
	extern __shared__ __align__(16) unsigned char dyn[];
	__shared__ ResShared sh;
	struct Scalars {
		double tol, tol2, rtol2, rho, rho_inv, rho_old, alpha, omega, ao, beta, rr, rr0, ss, rhs_norm,
			sol0, rt_norm, rt_eps, xx;  // tol2, rtol2, rt_eps: res_threshold of the tests
		int it, nhist, status, info_iters, flags, restarts;
		int turn;  // CTA that keeps the next entry of the history
		int what;  // thread 0's verdict: 1 stop, 2 early exit, 3 restart
	};
	__shared__ Scalars z;
	__shared__ ResRows<double, K, GEN> A;
	if ((int)blockIdx.x == a.lost)
		return;  // a test of the others' waits
	ResTeam tm;
	tm.init(a.slots, &sh, a.err);
	const int tid = threadIdx.x, nt = blockDim.x;
	const int lo = (int)min((int64_t)blockIdx.x * a.rows, (int64_t)a.A.n);
	const int cnt = (int)min((int64_t)a.rows, (int64_t)a.A.n - lo);
	ResSmem sm{dyn, a.smem};
	unsigned char *mask = sm.take<unsigned char>(a.rows);
	double *ph = sm.take<double>(a.rows), *sp = sm.take<double>(a.rows);  // P p, P s
	auto place = [&](double *g) {
		double *q = sm.take<double>(a.rows);
		return q ? q : g + lo;
	};
	double *r = place(a.r), *v = place(a.v), *p = place(a.p), *t = place(a.t), *rt = place(a.rt),
	       *x = place(a.x);
	double *dv = a.dinv ? sm.take<double>(a.rows) : nullptr;
	const double *dinv = dv ? dv : a.dinv ? a.dinv + lo : nullptr;
	{
		auto coef = [&](int slot) -> const double * {
			const double *g = a.A.S + (int64_t)slot * a.A.ld + lo;
			double *q = sm.take<double>(a.rows);
			if (q)
				for (int l = tid; l < cnt; l += nt)
					q[l] = g[l];
			return q ? q : g;
		};
		ResRows<double, K, GEN> q;
		q.ld = a.A.ld;
		q.lo = lo;
		q.cnt = cnt;
		q.d[0] = 1;
		q.d[1] = a.A.nx;
		q.d[2] = a.A.nx * a.A.ny;
		q.mask = mask;
		q.G = a.A.S + a.A.ld;
		q.D = coef(0);
#pragma unroll
		for (int k = 0; k < K; ++k)
			q.U[k] = coef(1 + k);
		if (GEN)
#pragma unroll
			for (int k = 0; k < K; ++k)
				q.L[k] = coef(1 + K + k);
		if (tid == 0)
			A = q;
	}
	for (int l = tid; l < cnt; l += nt) {
		mask[l] = (unsigned char)res_mask<K>(lo + l, a.A.nx, a.A.ny, a.A.nz);
		if (dv)
			dv[l] = a.dinv[lo + l];
	}
	__syncthreads();
	auto put = [&](double *own, int l, double q) {
		own[l] = q;
		res_st16(a.pk + (lo + l), res_pack(q), tm.epoch);
	};

	// res = b - A x, r~ = res, p = v = 0 (bicgstab.hh:73-98)
	double s3[3] = {0.0, 0.0, 0.0};
	for (int l = tid; l < cnt; l += nt) {
		const double bi = a.b[lo + l];
		double ri = bi, xi = 0.0;
		if (!a.zero_guess) {
			xi = a.x[lo + l];
			ri = bi - A.template sum<false>(l, a.x + lo, a.x, nullptr, 0, tm);
		}
		r[l] = ri;
		rt[l] = ri;
		p[l] = 0.0;
		v[l] = 0.0;
		s3[0] = fma(bi, bi, s3[0]);
		s3[1] = fma(xi, xi, s3[1]);
		s3[2] = fma(ri, ri, s3[2]);
	}
	const double s0 = tm.grid_sum<3, false>(s3);
	if (tid < 96 && (tid & 31) == 0)
		sh.bc[tid >> 5] = s0;
	bool alive = tm.done();
	if (tid == 0) {
		z = Scalars{};
		z.rhs_norm = sqrt(sh.bc[0]);
		if (z.rhs_norm == 0.0)
			z.rhs_norm = 1.0;
		z.tol = a.rtol * z.rhs_norm;
		z.tol2 = res_threshold(z.tol);
		z.rtol2 = res_threshold(a.rtol);
		z.sol0 = a.zero_guess ? 0.0 : sh.bc[1];
		z.rr0 = z.rr = sh.bc[2];
		z.rt_norm = sqrt(z.rr);
		z.rt_eps = res_threshold(2.220446049250313e-16 * z.rt_norm);
		z.alpha = z.omega = z.ao = 1.0;
		z.rho_old = 2.0;  // std::vector<real> rho{2, 1.0}
		z.rho = z.rr;
		z.beta = (z.rho / z.rho_old) * z.ao;
		z.rho_inv = 1.0 / z.rho;
		z.status = FS_STATUS_UNKNOWN;
		if (z.rr <= z.tol2) {
			z.what = 1;
			z.status = FS_CONVERGED_RTOL;
		}
		else if (a.maxiter <= 0) {
			z.what = 1;
			z.status = FS_DIVERGED_ITERS;
		}
	}
	// x may be a.x itself: first written here, after every slice has read its
	// neighbours' rows of the guess
	if (alive)
		for (int l = tid; l < cnt; l += nt)
			x[l] = a.zero_guess ? 0.0 : a.x[lo + l];
	__syncthreads();
	bool first = true;

	while (alive && z.what != 1) {
		// p = beta (p - omega v) + res (bicgstab.hh:115-122), P p handed out:
		// the others have read the last operand, which precedes their sums
		{
			const double beta = z.beta, om = z.omega;
			res_rows<2>(
				cnt, [&](int l) { return make_double3(p[l], v[l], r[l]); },
				[&](int l, const double3 &q) {
					const double pi = first ? q.z : fma(beta, fma(-om, q.y, q.x), q.z);
					p[l] = pi;
					put(ph, l, dinv ? dinv[l] * pi : pi);
				});
		}
		first = false;
		unsigned long long tag = tm.epoch;
		__syncthreads();
		res_hold(clock64());
		// v = A P p, alpha = rho / r~'v (bicgstab.hh:124-130)
		double s1[1] = {0.0};
		res_rows<2>(
			cnt, [&](int l) { return A.template sum<true>(l, ph, nullptr, a.pk, tag, tm); },
			[&](int l, double q) {
				v[l] = q;
				s1[0] = fma(rt[l], q, s1[0]);
			});
		const double rv = tm.grid_sum<1, false>(s1);
		if (tid == 0) {
			z.alpha = res_divide(z.rho, rv);
			if (!(rv != 0.0)) {
				z.flags |= KF_ALPHA_ZERO;
				z.what = 1;
				z.status = FS_DIVERGED_BREAKDOWN;
			}
		}
		if (tid == 32)
			z.rho_inv = 1.0 / z.rho;
		if (!(alive = tm.done()))
			break;
		if (z.what == 1)
			break;
		// s = res - alpha v (over res), ||s||, P s handed out
		// (bicgstab.hh:132-143)
		double s4[3] = {0.0, 0.0, 0.0};
		{
			const double al = z.alpha;
			res_rows<2>(
				cnt, [&](int l) { return make_double2(r[l], v[l]); },
				[&](int l, const double2 &q) {
					const double si = fma(-al, q.y, q.x);
					r[l] = si;
					put(sp, l, dinv ? dinv[l] * si : si);
					s4[0] = fma(si, si, s4[0]);
				});
		}
		tag = tm.epoch;
		__syncthreads();
		res_hold(clock64());
		// t = A P s, t't, t's (bicgstab.hh:145-151)
		res_rows<2>(
			cnt, [&](int l) { return A.template sum<true>(l, sp, nullptr, a.pk, tag, tm); },
			[&](int l, double q) {
				t[l] = q;
				s4[1] = fma(q, q, s4[1]);
				s4[2] = fma(q, r[l], s4[2]);
			});
		const double u4 = tm.grid_sum<3, false>(s4);
		if (tid < 96 && (tid & 31) == 0)
			sh.bc[tid >> 5] = u4;
		if (!(alive = tm.done()))
			break;
		if (tid == 0) {
			z.ss = sh.bc[0];
			if (z.ss <= z.rtol2) {
				// unscaled early exit (bicgstab.hh:136-142)
				z.what = 2;
				z.info_iters = z.it;
				z.status = FS_CONVERGED_RTOL;
			}
			z.omega = sh.bc[1] == 0.0 ? 0.0 : res_divide(sh.bc[2], sh.bc[1]);
		}
		__syncthreads();
		if (z.what == 2) {
			const double al = z.alpha;
			for (int l = tid; l < cnt; l += nt)
				x[l] = fma(al, ph[l], x[l]);
			break;
		}
		// x += alpha P p + omega P s; res = s - omega t; ||res||, r~'res
		// (bicgstab.hh:153-178)
		double s2[2] = {0.0, 0.0};
		{
			const double al = z.alpha, om = z.omega;
			struct Row {
				double x, p, s, r, t, q;
			};
			res_rows<2>(
				cnt, [&](int l) { return Row{x[l], ph[l], sp[l], r[l], t[l], rt[l]}; },
				[&](int l, const Row &w) {
					x[l] = fma(om, w.s, fma(al, w.p, w.x));
					const double ri = fma(-om, w.t, w.r);
					r[l] = ri;
					s2[0] = fma(ri, ri, s2[0]);
					s2[1] = fma(w.q, ri, s2[1]);
				});
		}
		const double u2 = tm.grid_sum<2, false>(s2);
		if (tid == 64)
			z.ao = z.alpha / z.omega;  // a warp without a message
		if (tid == 32)
			sh.bc[1] = res_quotient(u2, z.rho, z.rho_inv);
		if (tid == 32)
			sh.bc[2] = u2;
		if (tid == 0)
			sh.bc[0] = u2;
		if (!(alive = tm.done()))
			break;
		if (tid == 0) {
			const double rr = sh.bc[0], rho = sh.bc[2];
			const int it = z.it;
			z.beta = sh.bc[1] * z.ao;
			z.rr = rr;
			// each CTA keeps every gridDim-th entry of the history, its root
			// taken at the end
			const int turn = z.turn;
			if (z.nhist < a.hist_cap && turn == (int)blockIdx.x)
				a.hist[z.nhist] = rr;
			z.turn = turn + 1 < (int)gridDim.x ? turn + 1 : 0;
			z.nhist += 1;
			const bool finite = res_finite(rr);
			if (!finite)
				z.flags |= KF_NONFINITE;
			int what = 0;
			if (finite && res_below(rr, z.tol2)) {
				what = 1;
				z.status = FS_CONVERGED_RTOL;
				z.info_iters = it + 1;
			}
			else if (z.omega == 0.0) {
				what = 1;
				z.status = FS_DIVERGED_BREAKDOWN;
				z.info_iters = it + 1;
			}
			z.rho_old = z.rho;
			z.rho = rho;
			z.it = it + 1;
			if (!what) {
				if (it + 1 >= a.maxiter || !finite) {
					what = 1;
					z.status = FS_DIVERGED_ITERS;
				}
				else if (fabs(rho) <= z.rt_eps)
					what = 3;
			}
			z.what = what;
		}
		__syncthreads();
		if (z.what == 3) {
			// restart from the true residual (bicgstab.hh:103-113): r~ = p = res
			for (int l = tid; l < cnt; l += nt)
				put(sp, l, x[l]);
			tag = tm.epoch;
			__syncthreads();
			double q[1] = {0.0};
			for (int l = tid; l < cnt; l += nt) {
				const double ri = a.b[lo + l] - A.template sum<true>(l, sp, nullptr, a.pk, tag, tm);
				r[l] = ri;
				rt[l] = ri;
				p[l] = ri;
				q[0] = fma(ri, ri, q[0]);
			}
			const double rr = tm.grid_sum<1, false>(q);
			if (tid == 0)
				sh.bc[0] = rr;
			if (!(alive = tm.done()))
				break;
			if (tid == 0) {
				const double rs = sh.bc[0];
				z.rr = rs;
				z.rt_norm = sqrt(rs);
				z.rt_eps = res_threshold(2.220446049250313e-16 * z.rt_norm);
				z.rho = rs;
				z.beta = (rs / z.rho_old) * z.ao;
				z.restarts += 1;
				z.it += 1;  // the reference's restart consumes a loop index
				z.what = 0;
				if (z.it >= a.maxiter) {
					z.what = 1;
					z.status = FS_DIVERGED_ITERS;
				}
			}
			__syncthreads();
		}
	}
	__syncthreads();
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
		const int nh = min(z.nhist, a.hist_cap);
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
		st->alpha = z.alpha;
		st->beta = z.beta;
		st->omega = z.omega;
		st->r_tilde_norm = z.rt_norm;
		st->s_norm = sqrt(z.ss);
		st->aux[2] = sqrt(z.xx);
		st->iter = z.it;
		st->done = 1;
		st->status = z.status;
		st->info_iters = z.info_iters;
		st->flags = z.flags;
		st->maxiter = a.maxiter;
		st->restarts = z.restarts;
		st->hist_cap = a.hist_cap;
		st->nhist = z.nhist;
	}
	tm.finish();
}

// Rows up to which FP64 BiCGSTAB runs resident; us an iteration, kernels ->
// resident: 16^3 38.9 -> 12.5, 64^3 52.4 -> 26.3, 96^3 112 -> 77.9, 112^3 (1.4 M
// rows) 163 -> 149; at 128^3 the kernels' 220 are not beaten.
constexpr int64_t kResBiRows = 1500000;

}  // namespace

// FP64 BiCGSTAB (the state is read back); `taken` = 0 when the solve is not
// one for the resident kernel
int bicgstab_apply_resident(Solver *s, Vec *b, Vec *x, int *taken) {
	*taken = 0;
	Ctx *ctx = s->ctx;
	ResBi a{};
	bool gen = false;
	if (s->diag || s->n > kResBiRows || !res_grid<double>(s->A, a.A, gen))
		return FS_OK;
	const int K = s->A->nsym;
	using Kern = void (*)(ResBi);
	static const Kern kerns[2][3] = {
		{k_bi_resident<1, false>, k_bi_resident<2, false>, k_bi_resident<3, false>},
		{k_bi_resident<1, true>, k_bi_resident<2, true>, k_bi_resident<3, true>}};
	const Kern kern = kerns[gen][K - 1];
	const int smem_max = res_smem_max(ctx, kern);
	// mask, P p, P s, six vectors, dinv and the diagonals, as far as they fit
	const int per_row = 1 + 8 * (9 + 1 + (gen ? 2 * K : K));
	const ResShape sh = res_shape(ctx, s->n, per_row, smem_max);
	if ((int64_t)sh.rows * (1 + 16) > smem_max)
		return FS_OK;
	if (!res_memory(s, true))
		return FS_OK;
	FS_TRY(solver_hist(s, std::max(1, s->set.base.maxiter)));
	a.dinv = s->dinv64();
	a.b = (const double *)b->d;
	a.x = (double *)x->d;
	a.r = s->w64[0];
	a.rt = s->w64[1];
	a.p = s->w64[2];
	a.v = s->w64[3];
	a.t = s->w64[5];
	a.pk = s->res_pk;
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
	FS_TRY(res_launch(ctx, kern, sh, a, "resident bicgstab", taken));
	if (!*taken)
		return FS_OK;
	return res_read_state(s);
}

}  // namespace fsg
