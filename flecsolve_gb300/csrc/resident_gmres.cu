// GMRES(m) on a grid stencil in one cooperative launch (resident.cuh), FP64 or
// with an FP32 basis re-anchored on the FP64 residual at every restart.
//
// Orthogonalisation: the delayed CGS2 of gmres_staged.cuh -- column k holds
// the once-orthogonalised candidate u_k; a step forms w = M u_k, all 2 (k + 1)
// dots of w and u_k against the columns in one reduction, and updates q_k and
// u_{k+1}.  As separate kernels a step of a small system costs its launches
// and last-CTA folds: 28 us for the FP32 basis (three kernels), and 120 us for
// the FP64 basis, where modified Gram-Schmidt runs k + 2 reductions.  Here
// (one CTA per SM, its rows of every column in shared memory as far as they
// fit) a step waits for three messages: the packets of u_k's neighbour rows,
// the CTAs' sums on their way to the value's owner, and the owner's total on
// its way back (the 2 (k + 1) values have an owner CTA each, so that a CTA
// reads 2 (k + 1) totals and not all 152 sums of each).  The rotations, the
// residual estimate and the next tentative Hessenberg column, which nothing
// in the step waits for, run in the CTA's last warp (every CTA forms the same
// ones) while the other warps update, multiply and sum; a stop is seen one
// step later, when the columns that the solution needs are still whole.
#include <cmath>
#include <cstring>

#include "resident.cuh"

namespace fsg {

namespace {

constexpr int kRgVals = 2 * kGmDelayedCols;  // values of a step's reduction at most
constexpr int kRgThreads = 512;
constexpr int kRgSeg = 8;  // warps that share a column at most

struct RgSlots {
	ulonglong2 part[2][kRgVals][kResMaxG];  // {sum, epoch << 16 | exponent}
	ulonglong2 total[2][kRgVals];           // {total, epoch}
};

template<class T>
struct ResGm {
	ResGrid<T> A;
	ResGrid<double> A64;
	const T *dinv;            // Jacobi diagonal in T and FP64 (null: none)
	const double *dinv64;
	const double *b;
	double *x, *r64;
	T *V;                     // basis, columns ldv apart
	int64_t ldv;
	ulonglong2 *pk;
	RgSlots *vals;
	ResSlots *slots;
	unsigned *err;
	KState *st;
	double *hist;
	double rtol;
	int maxiter, hist_cap, zero_guess, right, m, mixed;
	int rows, smem, lost;
};

// rows a thread takes at a time in the basis passes: 16 bytes of FP32 rows
template<class T>
struct RgVec;
template<>
struct RgVec<float> {
	static constexpr int W = 4;
	__device__ static void ld(const float *p, float (&o)[4]) {
		const float4 t = *reinterpret_cast<const float4 *>(p);
		o[0] = t.x;
		o[1] = t.y;
		o[2] = t.z;
		o[3] = t.w;
	}
	__device__ static void st(float *p, const float (&o)[4]) {
		*reinterpret_cast<float4 *>(p) = make_float4(o[0], o[1], o[2], o[3]);
	}
};
template<>
struct RgVec<double> {
	static constexpr int W = 1;
	__device__ static void ld(const double *p, double (&o)[1]) { o[0] = *p; }
	__device__ static void st(double *p, const double (&o)[1]) { *p = o[0]; }
};

// A lane's running sum of products: FP64, or FP32 sums of at most 8 terms
// added with two-sum to a pair per row of the 16-byte group
template<class T>
struct RgAcc;
template<>
struct RgAcc<double> {
	double a = 0.0;
	__device__ void add(const double (&x)[1], const double (&y)[1]) { a = fma(x[0], y[0], a); }
	__device__ void flush() {}
	__device__ ResFix sum() const { return res_fix_warp(a); }
};
template<>
struct RgAcc<float> {
	float p[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
	__device__ void add(const float (&x)[4], const float (&y)[4]) {
#pragma unroll
		for (int i = 0; i < 4; ++i)
			p[i] = fmaf(x[i], y[i], p[i]);
	}
	__device__ void flush() {
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			float s, e;
			two_sum(hi[i], p[i], s, e);
			hi[i] = s;
			lo[i] += e;
			p[i] = 0.f;
		}
	}
	__device__ ResFix sum() const {
		const float v[8] = {hi[0], hi[1], hi[2], hi[3], lo[0], lo[1], lo[2], lo[3]};
		return res_fix_warp(v);
	}
};

// the CTA's copy of the small state (the same in every CTA)
struct RgSmall {
	// of the step: the totals, r, 1 / r and tau.  The Hessenberg warp reads them
	// beside the next step's passes; warp 0 writes the next ones after it is
	// through (rg_read_done, rg_read_wait).
	double s[kGmDelayedCols], t[kGmDelayedCols], r, rinv, tau;
	double Hr[kGmDelayedCols * kGmDelayedCols];        // Hessenberg before the rotations
	double H[kGmDelayedCols * kGmDelayedCols];         // and after
	double cs[kGmDelayedCols], sn[kGmDelayedCols], dw[kGmDelayedCols + 1], dy[kGmDelayedCols];
	double bnorm, tol, rhs_norm, sol0, res0, res, beta, xx;
	int k;                                             // finished columns
	int it, nhist, status, info_iters, flags, restarts;
	int stop;                                          // 1: done, 2: the cycle ends
	int flag[2];                                       // the same after a column, by its step's parity
	ResFix seg[kRgVals][kRgSeg];
};

__device__ __forceinline__ void rg_bar(int threads) {
	asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// The Hessenberg warp has read the step's scalars; warp 0, before it writes the
// next ones.  us a step with this / with a slot for each parity of the step: FP64
// 13.7 / 13.9 at 128^2, 13.7 / 14.1 at 64^2, FP32 13.5 / 14.0 at 32^3, 21.3 / 21.1
// at 64^3.
__device__ __forceinline__ void rg_read_done() {
	__threadfence_block();
	asm volatile("bar.arrive 2, 64;" ::: "memory");
}
__device__ __forceinline__ void rg_read_wait() { asm volatile("bar.sync 2, 64;" ::: "memory"); }

// column c of the Hessenberg matrix is final up to the step's s and r:
// rotations, estimate and stop tests (finish_step_warp of gmres.cu on the
// CTA's copy; only CTA 0 writes the history)
__device__ void rg_finish_column(RgSmall &g, int c, double *hist, int hist_cap, int maxiter, int m,
                                 int mixed, int *flag) {
	constexpr int ld = kGmDelayedCols;
	const int lane = threadIdx.x & 31;
	double *col = g.H + ld * c;
	if (lane < c + 1) {
		const double h = g.Hr[lane + ld * c] + g.s[lane];
		g.Hr[lane + ld * c] = h;
		col[lane] = h;
	}
	if (lane == 0) {
		g.Hr[c + 1 + ld * c] = g.r;
		col[c + 1] = g.r;
	}
	__syncwarp();
	double x = col[0];
	for (int i = 0; i < c; ++i) {
		const double y = col[i + 1], cc = g.cs[i], s = g.sn[i];
		const double a = lane == 0 ? cc : -s, b = lane == 0 ? s : cc;
		const double v = a * x + b * y;
		if (lane == 0)
			col[i] = v;
		x = __shfl_sync(0xffffffffu, v, 1);
	}
	if (lane == 0) {
		const double gg = g.r;
		col[c] = x;
		// a column without a remainder takes the identity: its estimate
		// is 0 and not what the cycle before left in dw[c + 1]
		double cc, s;
		if (gg == 0.0) {
			cc = 1.0;
			s = 0.0;
		}
		else if (x == 0.0) {
			cc = 0.0;
			s = gg < 0.0 ? -1.0 : 1.0;
		}
		else {
			const double q = 1.0 / sqrt(x * x + gg * gg);
			cc = fabs(x) * q;
			s = copysign(gg * q, x);
		}
		g.cs[c] = cc;
		g.sn[c] = s;
		col[c] = cc * x + s * gg;
		const double w = g.dw[c];
		g.dw[c] = cc * w;
		g.dw[c + 1] = -s * w;
		const double res = fabs(g.dw[c + 1]);
		g.k = c + 1;
		g.it += 1;
		g.res = res;
		if (blockIdx.x == 0 && g.nhist < hist_cap)
			hist[g.nhist] = res;
		g.nhist += 1;
		if (!isfinite(res))
			g.flags |= KF_NONFINITE;
		int stop = 0;
		if (res < g.tol) {
			// the FP32 estimate is verified on the FP64 residual
			stop = mixed ? 2 : 1;
			g.status = FS_CONVERGED_RTOL;
			g.info_iters = g.it;
		}
		else if (g.it >= maxiter || (g.flags & KF_NONFINITE)) {
			stop = mixed && !(g.flags & KF_NONFINITE) ? 2 : 1;
			g.status = FS_DIVERGED_ITERS;
		}
		else if (g.k == m)
			stop = 2;
		*flag = stop;
	}
	__syncwarp();
}

template<class T, int K, bool GEN>
__global__ void __launch_bounds__(kRgThreads, 1)
k_gm_resident(ResGm<T> a) {
	using VT = RgVec<T>;
	constexpr int W = VT::W;
	extern __shared__ __align__(16) unsigned char dyn[];
	__shared__ ResShared sh;
	__shared__ RgSmall g;
	__shared__ T *col[kGmDelayedCols];    // the slice's rows of each column
	__shared__ T hs[kGmDelayedCols], ht[kGmDelayedCols];
	if ((int)blockIdx.x == a.lost)
		return;  // a test of the others' waits
	ResTeam tm;
	tm.init(a.slots, &sh, a.err);
	const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
	const int nwk = (nt >> 5) - 1, ntk = nwk * 32;  // workers; the last warp keeps the Hessenberg
	const bool worker = wid < nwk;
	const int G = gridDim.x;
	const int lo = (int)min((int64_t)blockIdx.x * a.rows, (int64_t)a.A.n);
	const int cnt = (int)min((int64_t)a.rows, (int64_t)a.A.n - lo);
	const int nch = (cnt + W - 1) / W;    // row groups
	ResSmem sm{dyn, a.smem};
	unsigned char *mask = sm.take<unsigned char>(a.rows);
	T *ph = sm.take<T>(a.rows), *w = sm.take<T>(a.rows);
	for (int j = 0; j <= a.m; ++j) {
		T *q = sm.take<T>(a.rows);
		if (tid == 0)
			col[j] = q ? q : a.V + (int64_t)j * a.ldv + lo;
		if (q)
			for (int l = cnt + tid; l < a.rows; l += nt)
				q[l] = T(0);  // the last row group's tail
	}
	// the operators' addresses in shared memory: in registers they would be
	// spilled around the basis passes
	__shared__ ResRows<T, K, GEN> A;
	__shared__ ResRows<double, K, GEN> A64;
	auto coef = [&](int slot) -> const T * {
		const T *p = a.A.S + (int64_t)slot * a.A.ld + lo;
		T *q = sm.take<T>(a.rows);
		if (q)
			for (int l = tid; l < cnt; l += nt)
				q[l] = p[l];
		return q ? q : p;
	};
	{
		ResRows<T, K, GEN> r;
		ResRows<double, K, GEN> r64;
		r.ld = a.A.ld;
		r64.ld = a.A64.ld;
		r.lo = r64.lo = lo;
		r.cnt = r64.cnt = cnt;
		r.d[0] = r64.d[0] = 1;
		r.d[1] = r64.d[1] = a.A.nx;
		r.d[2] = r64.d[2] = a.A.nx * a.A.ny;
		r.mask = r64.mask = mask;
		r.G = a.A.S + a.A.ld;
		r64.G = a.A64.S + a.A64.ld;
		r.D = coef(0);
		r64.D = a.A64.S + lo;
#pragma unroll
		for (int t = 0; t < K; ++t) {
			r.U[t] = coef(1 + t);
			r64.U[t] = a.A64.S + (int64_t)(1 + t) * a.A64.ld + lo;
		}
		if (GEN)
#pragma unroll
			for (int t = 0; t < K; ++t) {
				r.L[t] = coef(1 + K + t);
				r64.L[t] = a.A64.S + (int64_t)(1 + K + t) * a.A64.ld + lo;
			}
		if (tid == 0) {
			A = r;
			A64 = r64;
		}
	}
	for (int l = tid; l < a.rows; l += nt) {
		if (l < cnt)
			mask[l] = (unsigned char)res_mask<K>(lo + l, a.A.nx, a.A.ny, a.A.nz);
		else
			w[l] = T(0);
	}
	if (tid == 0) {
		g.k = g.it = g.nhist = g.info_iters = g.flags = g.restarts = g.stop = 0;
		g.status = FS_STATUS_UNKNOWN;
		g.res = g.xx = 0.0;
		for (int j = 0; j <= kGmDelayedCols; ++j)
			g.dw[j] = 0.0;
	}
	__syncthreads();
	const T *dinv = a.dinv ? a.dinv + lo : nullptr;
	const double *dinv64 = a.dinv64 ? a.dinv64 + lo : nullptr;

	// r64 = b - A x, or D^-1 of it (left), beta = ||r64||; x's neighbour rows
	// come as packets of `tag`, or x is 0 (first and zero guess)
	auto residual = [&](bool zero, unsigned long long tag) {
		double acc = 0.0;
		for (int l = tid; l < cnt; l += nt) {
			double r = a.b[lo + l];
			if (!zero)
				r -= A64.template sum<true>(l, a.x + lo, nullptr, a.pk, tag, tm);
			if (!a.right && dinv64)
				r = dinv64[l] * r;
			a.r64[lo + l] = r;
			acc = fma(r, r, acc);
		}
		const double v[1] = {acc};
		const double t = tm.grid_sum<1, false>(v);
		if (tid == 0)
			g.beta = sqrt(t);
		return tm.done();
	};
	auto put_x = [&](int l, double v) { res_st16(a.pk + (lo + l), res_pack(v), tm.epoch); };
	// the operand of the next SpMV: P u (right) or u (left)
	auto put_u = [&](int l, T u) {
		const T v = a.right && dinv ? dinv[l] * u : u;
		ph[l] = v;
		res_st16(a.pk + (lo + l), res_pack(v), tm.epoch);
	};

	// ||b||, ||x||
	double s2[2] = {0.0, 0.0};
	for (int l = tid; l < cnt; l += nt) {
		const double bi = a.b[lo + l];
		s2[0] = fma(bi, bi, s2[0]);
		if (a.zero_guess)
			a.x[lo + l] = 0.0;
		else {
			const double xi = a.x[lo + l];
			s2[1] = fma(xi, xi, s2[1]);
			put_x(l, xi);
		}
	}
	unsigned long long tag = tm.epoch;
	{
		const double t = tm.grid_sum<2, false>(s2);
		if (tid == 0) {
			const double bn = sqrt(t);
			g.rhs_norm = bn;
			g.bnorm = bn < 2.220446049250313e-16 ? 1.0 : bn;
			g.tol = a.rtol * g.bnorm;
		}
		if (tid == 32)
			g.sol0 = a.zero_guess ? 0.0 : sqrt(t);
	}
	bool alive = tm.done();
	alive = alive && residual(a.zero_guess, tag);
	if (tid == 0) {
		g.res0 = g.res = g.beta;
		if (g.beta < g.tol) {
			g.status = FS_CONVERGED_RTOL;
			g.stop = 1;
		}
		else if (a.maxiter <= 0) {
			g.status = FS_DIVERGED_ITERS;
			g.stop = 1;
		}
	}
	__syncthreads();

	while (alive && g.stop != 1) {
		// ---- a cycle: column 0 from the residual (gmres.hh:134-139)
		{
			const double inv = 1.0 / g.beta;
			T *c0 = col[0];
			tag = tm.epoch;
			for (int l = tid; l < cnt; l += nt) {
				const T u = (T)(a.r64[lo + l] * inv);
				c0[l] = u;
				put_u(l, u);
			}
			if (tid == 0) {
				g.dw[0] = g.beta;
				g.k = 0;
				g.stop = 0;
				g.flag[0] = g.flag[1] = 0;
			}
		}
		__syncthreads();
		for (int k = 0;; ++k) {
			const bool last = k == a.m;  // u_m's sums alone finish the cycle
			const int nv = last ? k + 1 : 2 * (k + 1);
			++tm.epoch;
			if (worker) {
				if (!last) {
					// w = A P u_k, or D^-1 A u_k
					for (int l = tid; l < cnt; l += ntk) {
						const T v = A.template sum<true>(l, ph, nullptr, a.pk, tag, tm);
						w[l] = !a.right && dinv ? dinv[l] * v : v;
					}
					rg_bar(ntk);
				}
				// the slice's sums u_k . V_j (value j) and w . V_j (value
				// k + 1 + j): a warp a column, several where there are few
				const int nseg = max(1, min(min(kRgSeg, nwk / (k + 1)), (a.rows / W + 31) / 32));
				const T *u = col[k];
				ulonglong2(*part)[kResMaxG] = a.vals->part[tm.epoch & 1];
				for (int jj = wid; jj < (k + 1) * nseg; jj += nwk) {
					const int j = jj / nseg, sg = jj - j * nseg;
					const T *v = col[j];
					RgAcc<T> as, at;
					for (int c0 = sg * 32 + lane; c0 < nch; c0 += 8 * 32 * nseg) {
#pragma unroll
						for (int h = 0; h < 2; ++h) {
							T vv[4][W], uu[4][W], ww[4][W];
#pragma unroll
							for (int q = 0; q < 4; ++q) {
								const int c = c0 + (4 * h + q) * 32 * nseg;
								if (c < nch) {
									VT::ld(v + W * c, vv[q]);
									VT::ld(u + W * c, uu[q]);
									if (!last)
										VT::ld(w + W * c, ww[q]);
								}
							}
#pragma unroll
							for (int q = 0; q < 4; ++q)
								if (c0 + (4 * h + q) * 32 * nseg < nch) {
									as.add(uu[q], vv[q]);
									if (!last)
										at.add(ww[q], vv[q]);
								}
						}
						as.flush();
						at.flush();
					}
					const ResFix fs = as.sum();
					const ResFix ft = last ? ResFix{0, 1} : at.sum();
					if (lane == 0) {
						if (nseg == 1) {
							res_xchg16(&part[j][blockIdx.x], (unsigned long long)fs.q,
							           tm.epoch << 16 | (unsigned long long)fs.e);
							if (!last)
								res_xchg16(&part[k + 1 + j][blockIdx.x], (unsigned long long)ft.q,
								           tm.epoch << 16 | (unsigned long long)ft.e);
						}
						else {
							g.seg[j][sg] = fs;
							g.seg[k + 1 + j][sg] = ft;
						}
					}
				}
				if (nseg > 1) {
					rg_bar(ntk);
					for (int v = wid; v < nv; v += nwk) {
						const ResFix f = res_fix_cta(lane < nseg ? g.seg[v][lane] : ResFix{0, 1});
						if (lane == 0)
							res_xchg16(&part[v][blockIdx.x], (unsigned long long)f.q,
							           tm.epoch << 16 | (unsigned long long)f.e);
					}
				}
				// the values this CTA owns: gather, total, hand back
				for (int i = wid; i * G + (int)blockIdx.x < nv; i += nwk) {
					const int v = i * G + (int)blockIdx.x;
					res_hold(clock64());
					ResFix f[kResMaxG / 32];
					if (!tm.gather(part[v], f) && lane == 0)
						tm.failed();
					const double t = nseg == 1 ? res_fix_grid<kResMaxG / 32, 3>(f)
					                           : res_fix_grid<kResMaxG / 32, 0>(f);
					if (lane == 0)
						res_xchg16(&a.vals->total[tm.epoch & 1][v], res_pack(t), tm.epoch);
				}
				if (wid == 0) {
					// every total; then r = sqrt(u'u - s's), tau = (u'w - s't) / r
					double q[2] = {0.0, 0.0};
					bool here = false;
					res_hold(clock64());
					for (int it = 0; !here && it < kResPolls; ++it) {
						ulonglong2 m[2];
#pragma unroll
						for (int i = 0; i < 2; ++i)
							m[i] = res_ld16(&a.vals->total[tm.epoch & 1][min(lane + i * (k + 1), nv - 1)]);
						here = true;
#pragma unroll
						for (int i = 0; i < 2; ++i) {
							here = here && m[i].y == tm.epoch;
							q[i] = __longlong_as_double((long long)m[i].x);
						}
					}
					if (!__all_sync(0xffffffffu, here) && lane == 0)
						tm.failed();
					const double alpha = __shfl_sync(0xffffffffu, q[0], k);
					const double gamma = __shfl_sync(0xffffffffu, q[1], k);
					double ss = lane < k ? q[0] * q[0] : 0.0, sw = lane < k ? q[0] * q[1] : 0.0;
#pragma unroll
					for (int o = 16; o > 0; o >>= 1) {
						ss += __shfl_xor_sync(0xffffffffu, ss, o);
						sw += __shfl_xor_sync(0xffffffffu, sw, o);
					}
					if (k > 0)
						rg_read_wait();  // (no step precedes the first of a cycle)
					if (lane <= k) {
						g.s[lane] = q[0];
						g.t[lane] = q[1];
						hs[lane] = (T)q[0];
						ht[lane] = (T)q[1];
					}
					const double r = k > 0 ? gm_norm(alpha - ss) : 1.0;
					const double rinv = r != 0.0 ? 1.0 / r : 1.0;
					if (lane == 0) {
						g.r = r;
						g.rinv = rinv;
						g.tau = (gamma - sw) * rinv;
					}
				}
			}
			if (!(alive = tm.done()))
				break;
			// the Hessenberg warp's verdict on column k - 2, formed in the last
			// step (it writes the other parity's flag in this one)
			if (k > 0 && g.flag[(k - 1) & 1]) {
				__syncthreads();
				if (tid == 0)
					g.stop = g.flag[(k - 1) & 1];
				break;
			}
			if (!worker) {
				if (k > 0)
					rg_finish_column(g, k - 1, a.hist, a.hist_cap, a.maxiter, a.m, a.mixed,
					                 &g.flag[k & 1]);
				if (!last && lane <= k) {
					// tentative column k: ([t; tau] - H s) / r over rows 0..k
					double d = 0.0;
					for (int j = 0; j < k; ++j)
						if (j + 1 >= lane)
							d = fma(g.Hr[lane + kGmDelayedCols * j], g.s[j], d);
					g.Hr[lane + kGmDelayedCols * k] = ((lane < k ? g.t[lane] : g.tau) - d) * g.rinv;
				}
				__syncwarp();
				if (!last)
					rg_read_done();
			}
			if (last) {
				__syncthreads();
				if (tid == 0)
					g.stop = g.flag[k & 1];
				break;
			}
			if (worker) {
				// q_k = (u_k - Q s) / r, u_{k+1} = (w - Q t - tau q_k) / r
				T *uk = col[k], *un = col[k + 1];
				const T inv = (T)g.rinv, tau = (T)-g.tau;
				tag = tm.epoch;
				for (int c = tid; c < nch; c += ntk) {
					T q[W], n[W];
					VT::ld(uk + W * c, q);
					VT::ld(w + W * c, n);
					int j = 0;
					for (; j + 4 <= k; j += 4) {
						T v[4][W];
#pragma unroll
						for (int i = 0; i < 4; ++i)
							VT::ld(col[j + i] + W * c, v[i]);
#pragma unroll
						for (int i = 0; i < 4; ++i)
#pragma unroll
							for (int y = 0; y < W; ++y) {
								q[y] = fma(-hs[j + i], v[i][y], q[y]);
								n[y] = fma(-ht[j + i], v[i][y], n[y]);
							}
					}
					for (; j < k; ++j) {
						T v[W];
						VT::ld(col[j] + W * c, v);
#pragma unroll
						for (int y = 0; y < W; ++y) {
							q[y] = fma(-hs[j], v[y], q[y]);
							n[y] = fma(-ht[j], v[y], n[y]);
						}
					}
#pragma unroll
					for (int y = 0; y < W; ++y) {
						if (k > 0)
							q[y] = q[y] * inv;
						n[y] = fma(tau, q[y], n[y]) * inv;
					}
					if (k > 0)
						VT::st(uk + W * c, q);
					VT::st(un + W * c, n);
#pragma unroll
					for (int y = 0; y < W; ++y)
						if (W * c + y < cnt)
							put_u(W * c + y, n[y]);
				}
				rg_bar(ntk);
			}
		}
		if (!alive)
			break;
		__syncthreads();
		// ---- x += P V y (gmres.hh:244-263), y from the back substitution
		const int kk = g.k;
		if (wid == 0 && kk > 0) {
			constexpr int ld = kGmDelayedCols;
			double y = lane < kk ? g.dw[lane] : 0.0;
			const double h = lane < kk ? g.H[lane + ld * lane] : 1.0;
			const double hinv = 1.0 / h;
			for (int i = kk - 1; i >= 0; --i) {
				const double yi = __shfl_sync(0xffffffffu, res_quotient(y, h, hinv), i);
				if (lane == i)
					g.dy[i] = yi;
				if (lane < i)
					y = fma(-g.H[lane + ld * i], yi, y);
			}
		}
		__syncthreads();
		tag = tm.epoch;
		const bool more = a.mixed || g.stop == 2;  // a residual follows
		for (int l = tid; l < cnt; l += nt) {
			double xi = a.x[lo + l];
			if (kk > 0) {
				if (a.right) {
					double z = 0.0;
					for (int j = 0; j < kk; ++j)
						z = fma(g.dy[j], (double)col[j][l], z);
					xi += dinv64 ? dinv64[l] * z : z;
				}
				else
					for (int j = 0; j < kk; ++j)
						xi = fma(g.dy[j], (double)col[j][l], xi);
			}
			a.x[lo + l] = xi;
			if (more)
				put_x(l, xi);
		}
		__syncthreads();
		if (!more)
			break;
		if (!(alive = residual(false, tag)))
			break;
		if (tid == 0) {
			int stop = 2;
			if (a.mixed) {
				// the stopping decision on the FP64 residual
				g.res = g.beta;
				if (!isfinite(g.beta))
					g.flags |= KF_NONFINITE;
				if (g.beta < g.tol) {
					stop = 1;
					g.status = FS_CONVERGED_RTOL;
					g.info_iters = g.it;
				}
				else if (g.it >= a.maxiter || (g.flags & KF_NONFINITE)) {
					stop = 1;
					g.status = FS_DIVERGED_ITERS;
					g.info_iters = 0;
				}
				else {
					g.status = FS_STATUS_UNKNOWN;
					g.info_iters = 0;
				}
			}
			if (stop == 2)
				g.restarts += 1;
			g.stop = stop;
		}
		__syncthreads();
	}
	double xx = 0.0;
	for (int l = tid; l < cnt; l += nt) {
		const double xi = a.x[lo + l];
		xx = fma(xi, xi, xx);
	}
	if (alive) {
		const double v[1] = {xx};
		const double t = tm.grid_sum<1, false>(v);
		if (tid == 0)
			g.xx = t;
		tm.done();
	}
	if (blockIdx.x == 0 && tid == 0) {
		KState *st = a.st;
		st->rhs_norm = g.rhs_norm;
		st->bnorm = g.bnorm;
		st->tol = g.tol;
		st->rtol = a.rtol;
		st->sol0 = g.sol0;
		st->res0 = g.res0;
		st->res = g.res;
		st->aux[2] = sqrt(g.xx);
		st->iter = g.it;
		st->done = 1;
		st->status = g.status;
		st->info_iters = g.info_iters;
		st->flags = g.flags;
		st->maxiter = a.maxiter;
		st->restarts = g.restarts;
		st->hist_cap = a.hist_cap;
		st->nhist = g.nhist;
	}
	tm.finish();
}

// Rows up to which GMRES runs resident, by the basis type.  us a step, kernels
// -> resident.  FP64 (modified Gram-Schmidt in kernels): 128^2 120 -> 13.7,
// 512^2 124 -> 45.7, 64^3 140 -> 46.6, 100^3 237 -> 162.  FP32 (the staged
// passes): 32^3 28.3 -> 13.5, 64^3 32.1 -> 21.3, 96^3 52.9 -> 64.6: past 0.45 M
// rows the columns no longer fit and the tensor copies of the staged passes
// stream them better than this kernel's loads.
template<class T>
constexpr int64_t kResGmRows = sizeof(T) == 8 ? 1000000 : 450000;

}  // namespace

// GMRES with the delayed CGS2; `taken` = 0 when the solve is not one for the
// resident kernel.  s->basis holds min(m, maxiter) + 1 columns of T.
template<class T>
int gmres_apply_resident(Solver *s, Vec *b, Vec *x, int m, bool mixed, int *taken) {
	*taken = 0;
	Ctx *ctx = s->ctx;
	ResGm<T> a{};
	bool gen = false, gen64 = false;
	if (s->diag || m < 1 || m + 1 >= kGmDelayedCols || s->n > kResGmRows<T> ||
	    !(s->set.ortho == FS_ORTHO_DCGS2 || s->set.ortho == FS_ORTHO_AUTO) ||
	    !res_grid<T>(s->A, a.A, gen) || !res_grid<double>(s->A, a.A64, gen64) || gen != gen64)
		return FS_OK;
	const int K = s->A->nsym;
	using Kern = void (*)(ResGm<T>);
	static const Kern kerns[2][3] = {
		{k_gm_resident<T, 1, false>, k_gm_resident<T, 2, false>, k_gm_resident<T, 3, false>},
		{k_gm_resident<T, 1, true>, k_gm_resident<T, 2, true>, k_gm_resident<T, 3, true>}};
	const Kern kern = kerns[gen][K - 1];
	const int smem_max = res_smem_max(ctx, kern);
	// mask, the SpMV's operand and result, the columns and the diagonals
	const int per_row = 1 + (int)sizeof(T) * (2 + m + 1 + 1 + (gen ? 2 * K : K));
	ResShape sh = res_shape(ctx, s->n, per_row, smem_max);
	if ((int64_t)sh.rows * (1 + 2 * (int)sizeof(T)) > smem_max)
		return FS_OK;
	sh.threads = kRgThreads;
	if (!res_memory(s, true))
		return FS_OK;
	if (!s->res_vals) {
		void *p = nullptr;
		if (cudaMalloc(&p, sizeof(RgSlots)) != cudaSuccess) {
			cudaGetLastError();
			return FS_OK;  // no room: the phase kernels
		}
		s->bufs.push_back(p);
		FS_CUDA_TRY(ctx, cudaMemsetAsync(p, 0, sizeof(RgSlots), ctx->stream));
		s->res_vals = p;
		s->res_vals_len = sizeof(RgSlots);
	}
	FS_TRY(solver_hist(s, std::max(1, s->set.base.maxiter)));
	if constexpr (sizeof(T) == 8)
		a.dinv = s->dinv64();
	else
		a.dinv = s->dinv32();
	a.dinv64 = s->dinv64();
	a.b = (const double *)b->d;
	a.x = (double *)x->d;
	a.r64 = s->w64[0];
	a.V = (T *)s->basis;
	a.ldv = (s->n + 31) / 32 * 32;
	a.pk = s->res_pk;
	a.vals = (RgSlots *)s->res_vals;
	a.slots = s->res_slots;
	a.err = ctx->dev_err;
	a.lost = sh.grid > 1 ? s->res_lost - 1 : -1;
	a.st = s->st;
	a.hist = s->hist;
	a.rtol = (double)s->set.base.rtol;
	a.maxiter = s->set.base.maxiter;
	a.hist_cap = s->hist_cap;
	a.zero_guess = s->set.base.use_zero_guess != 0;
	a.right = s->set.pre_side != FS_LEFT;
	a.m = m;
	a.mixed = mixed;
	a.rows = sh.rows;
	a.smem = sh.smem;
	FS_TRY(res_launch(ctx, kern, sh, a, "resident gmres", taken));
	if (!*taken)
		return FS_OK;
	return res_read_state(s);
}

template int gmres_apply_resident<double>(Solver *, Vec *, Vec *, int, bool, int *);
template int gmres_apply_resident<float>(Solver *, Vec *, Vec *, int, bool, int *);

}  // namespace fsg
