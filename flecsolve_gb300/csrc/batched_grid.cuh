// Batched CG on 5-point square grids: every system stays on chip.
//
// A system's rows are dealt to the CTAs of one thread-block cluster in
// contiguous slices (one CTA when the slice limit allows).  In the FP32 phase
// thread t keeps r, x and A p of its rows t, t + NT, ... in registers; the
// direction with s halo rows either side, the three coefficient diagonals and
// D^-1 are in shared memory, 20 bytes a row, so an iteration reads and writes
// nothing beyond the SMs.  The direction's halo is updated by its owner and by
// the neighbour alike, p = z + beta p from the z rows that the owner has pushed
// into the neighbour's shared memory with the residual update; the two sums of
// an iteration are its only cluster barriers.  In the FP64 head p and r are in
// shared memory and A p in registers; the coefficients, D^-1 and x, 48 bytes a
// row, stream from the L2 under the FP64 pipe's seven cycles a row.
//
// The sums run in integers (see resident.cuh): a warp's FP64 instruction holds
// its scheduler for 62 cycles.
//
// Bound: the FP64 pipe in the head (12 operations a row, 6.0 cycles at two a
// cycle and SM; measured 6.9), instruction issue in the FP32 phase (1.0 cycle a
// row), then the sums (about 2,700 cycles each, 1,700 on one CTA).  512 systems
// of side 32..256 at rtol 1e-12, 3.4 G row-iterations in the head and 9.8 G
// after it: 144 ms, of which 73 in the head, 34 in the FP32 loops, 25 in the
// sums, 4 in replacements and 6 % idle SMs, against 234 ms of the general
// kernel, whose vectors and coefficients go through the L2 and the memory 60
// bytes a row and iteration.
#pragma once

#include "resident.cuh"

namespace fsg {

namespace {

// Slice limits.  512 threads with 22 rows each: 66 registers of FP32 vectors
// (44 of A p in the head) of 128, and 20 bytes x 11,264 rows of shared memory.
// Rows without a branch between: the FP32 loops with 2 / 4 take 145.7 / 144.0 ms
// on the 512 systems (one at a time 166), the head's with 2 / 4 take 144 / 153.
constexpr int kBgRows = 22;
constexpr int kBgThreads = 512;
constexpr int kBgG64 = 2, kBgG32 = 4;
constexpr int kBgTeam = 16;  // CTAs per cluster at most (8 are portable)

struct BgShared {
	ResFix part[2][kBgThreads / 32];
	ResFix slots[2][2][kBgTeam];
	double tot[2];      // a sum's values, handed to every thread
	double rho, rz;     // r.z of the direction in use, of the residual
	double thr;         // r.r at which the residual is replaced
	double first[3];    // ||b||, ||x||, ||r|| before the first iteration
	double bc;          // alpha or beta of the head
	float af, bf;
	int act;
};

// f(u) for the rows t + u NT of thread t that the slice has, G of them without
// a branch between while the whole CTA has them
template<int U, class F, int... I>
__device__ __forceinline__ void bg_group(F &f, std::integer_sequence<int, I...>) {
	(f(std::integral_constant<int, U + I>{}), ...);
}
template<int U, class F, int... I>
__device__ __forceinline__ void bg_tail(int cnt, F &f, std::integer_sequence<int, I...>) {
	(((int)threadIdx.x + (U + I) * kBgThreads < cnt ? f(std::integral_constant<int, U + I>{}) : (void)0), ...);
}
template<int G, int U = 0, class F>
__device__ __forceinline__ void bg_rows_do(int cnt, F &&f) {
	if constexpr (U < kBgRows) {
		constexpr int N = U + G <= kBgRows ? G : kBgRows - U;
		if ((U + N) * kBgThreads <= cnt) {
			bg_group<U>(f, std::make_integer_sequence<int, N>{});
			bg_rows_do<G, U + N>(cnt, f);
		}
		else
			bg_tail<U>(cnt, f, std::make_integer_sequence<int, N>{});
	}
}

// floats of dynamic shared memory: p with two halos, the upper diagonals (the
// outer one with a halo of lower partners, the inner one with one row), the
// diagonal, D^-1, z of the halo rows.  The head's doubles (p with two halos,
// r, z of the halo rows) take the same room.
__host__ __device__ inline int64_t bg_smem(int64_t rows, int64_t side) {
	const int64_t f32 = 4 * (5 * rows + 5 * side + 1), f64 = 8 * (2 * rows + 4 * side);
	return ((f32 > f64 ? f32 : f64) + 15) / 16 * 16;
}

// rows per CTA of a system on `team` CTAs
__host__ __device__ inline int64_t bg_rows(int64_t nrow, int team) {
	return team == 1 ? nrow : ((nrow + team - 1) / team + 31) / 32 * 32;
}

__global__ void __launch_bounds__(kBgThreads, 1)
k_batch_grid(BatchArgs a) {
	constexpr int NT = kBgThreads, NW = NT / 32, R = kBgRows;
	extern __shared__ double2 bg_dyn[];
	__shared__ BgShared sh;
	cgrp::cluster_group cl = cgrp::this_cluster();
	const int team = (int)cl.num_blocks(), rank = (int)cl.block_rank();
	const int sys = a.order[a.first + (int)blockIdx.x / team];
	const int64_t R0 = a.off[sys];
	const int nrow = (int)(a.off[sys + 1] - R0);
	const int s = a.side[sys];
	const int chunk = (int)bg_rows(nrow, team);
	const int lo = min(nrow, chunk * rank);  // the slice's first row in the system
	const int cnt = min(nrow - lo, chunk);
	const int64_t g0 = R0 + lo;              // and in the batch
	const int tid = (int)threadIdx.x, lane = tid & 31, wid = tid >> 5;
	int ph = 0;

	// every thread of the team: all that the team wrote before is visible
	auto team_sync = [&]() {
		if (team > 1)
			cl.sync();
		else
			__syncthreads();
	};
	// whether rows u NT .. u NT + NT - 1 hold some that a neighbour needs
	auto edge = [&](int u) { return u * NT < s || u * NT + NT > chunk - s; };
	// The team's sums of up to two values, given by warp; warp k returns value
	// k (the same in each lane and CTA).  A barrier of the team; the caller's
	// next __syncthreads comes before the next sum.
	auto team_sum = [&](auto &f) -> double {
		constexpr int nv = (int)(sizeof(f) / sizeof(ResFix));
#pragma unroll
		for (int k = 0; k < nv; ++k)
			if (lane == 0)
				sh.part[k][wid] = f[k];
		__syncthreads();
		ResFix own{0, 1};
		if (wid < nv) {
			if (lane < NW)
				own = sh.part[wid][lane];
			own = res_fix_cta(own);
			if (team > 1 && lane < team)
				*cl.map_shared_rank(&sh.slots[ph][wid][rank], lane) = own;
		}
		if (team > 1)
			cl.sync();
		double t = 0.0;
		if (wid < nv) {
			if (team > 1) {
				ResFix g[1] = {{0, 1}};
				if (lane < team)
					g[0] = sh.slots[ph][wid][lane];
				t = res_fix_grid<1>(g);
			}
			else
				t = res_fix_value(own);
		}
		ph ^= 1;
		return t;
	};
	// the sums of two doubles a thread, in every thread
	auto sum_all = [&](double v0, double v1, double &t0, double &t1) {
		ResFix f[2] = {res_fix_warp(v0), res_fix_warp(v1)};
		const double t = team_sum(f);
		if (wid < 2 && lane == 0)
			sh.tot[wid] = t;
		__syncthreads();
		t0 = sh.tot[0];
		t1 = sh.tot[1];
		__syncthreads();
	};
	// FP64 row sum of A v on global vectors (rows of the whole system)
	auto row64 = [&](const double *v, int l) -> double {
		const int q = lo + l, ii = q % s;
		const int64_t i = g0 + l;
		double t = 0.0;
		if (q >= s)
			t = fma(a.gu2_64[i - s], v[i - s], t);
		if (ii > 0)
			t = fma(a.gu1_64[i - 1], v[i - 1], t);
		t = fma(a.gd64[i], v[i], t);
		if (ii < s - 1)
			t = fma(a.gu1_64[i], v[i + 1], t);
		if (q < nrow - s)
			t = fma(a.gu2_64[i], v[i + s], t);
		return t;
	};

	// a peer's shared memory may be written once all CTAs of the cluster run
	team_sync();

	// ||b||, ||x||
	double bnorm, res;
	{
		double v0 = 0.0, v1 = 0.0;
		for (int l = tid; l < cnt; l += NT) {
			const double bi = a.b[g0 + l];
			v0 = fma(bi, bi, v0);
			if (a.zero_guess)
				a.x[g0 + l] = 0.0;
			else {
				const double xi = a.x[g0 + l];
				v1 = fma(xi, xi, v1);
			}
		}
		sum_all(v0, v1, v0, v1);
		bnorm = sqrt(v0);
		if (tid == 0) {
			sh.first[0] = bnorm;
			sh.first[1] = sqrt(v1);
		}
	}
	if (bnorm == 0.0)
		bnorm = 1.0;
	const double tol = (double)a.rtol * bnorm;
	int status = FS_DIVERGED_ITERS, iters = 0, outer = 0;
	double bq = 0.0;  //  beta of the direction handed to the FP32 phase
	bool head, handed = false;
	float xr[R];  // the FP32 phase's correction; before it, its first direction
#pragma unroll
	for (int u = 0; u < R; ++u)
		xr[u] = 0.f;

	// ------------------------------------------------------- FP64 head --
	{
		double *P = reinterpret_cast<double *>(bg_dyn);  // rows -s .. chunk + s
		double *Rs = P + chunk + 2 * s, *Z = Rs + chunk;
		double w[R];  // A p, then z
		for (int i = tid; i < 2 * s; i += NT) {
			P[i < s ? i : chunk + i] = 0.0;
			Z[i] = 0.0;
		}
		for (int l = cnt + tid; l < chunk; l += NT)
			P[s + l] = 0.0;  // past the system's last row
		// a neighbour's pushes come after its first sum, whose barrier this
		// CTA reaches after the line above
		auto push = [&](int l, double z) {
			if (l < s && rank > 0)
				*cl.map_shared_rank(&Z[s + l], rank - 1) = z;
			if (l >= chunk - s && rank + 1 < team)
				*cl.map_shared_rank(&Z[l - (chunk - s)], rank + 1) = z;
		};
		team_sync();
		double t0 = 0.0, t1 = 0.0;
		for (int l = tid; l < cnt; l += NT) {
			const double bi = a.b[g0 + l];
			const double ri = a.zero_guess ? bi : bi - row64(a.x, l);
			const double zi = a.dinv64[g0 + l] * ri;
			Rs[l] = ri;
			P[s + l] = zi;
			if (team > 1)
				push(l, zi);
			t0 = fma(ri, ri, t0);
			t1 = fma(ri, zi, t1);
		}
		double rr, rho;
		sum_all(t0, t1, rr, rho);
		res = sqrt(rr);
		if (tid == 0)
			sh.first[2] = res;
		head = res >= tol && a.head > 0.0 && res >= a.head * bnorm && a.maxiter > 0;
		// (a NaN residual takes the FP32 loop's exit, as without a head)
		if (head) {
			const double t_tol = res_threshold(tol), t_head = res_threshold(a.head * bnorm);
			for (int i = tid; i < 2 * s; i += NT)
				P[i < s ? i : chunk + i] = Z[i];
			if (tid == 0)
				sh.rho = rho;
			__syncthreads();
			for (int it = 0; it < a.maxiter; ++it) {
				double q = 0.0;
				bg_rows_do<kBgG64>(cnt, [&](auto uc) {
					constexpr int u = decltype(uc)::value;
					const int l = tid + u * NT;
					// an absent lower partner reads the own row's coefficient
					// and multiplies the halo's zero
					const int64_t i = g0 + l;
					const double c0 = a.gu2_64[lo + l >= s ? i - s : i];
					const double c1 = a.gu1_64[lo + l >= 1 ? i - 1 : i];
					const double c2 = a.gd64[i], c3 = a.gu1_64[i], c4 = a.gu2_64[i];
					const double pc = P[s + l];
					double t = c0 * P[l];
					t = fma(c1, P[s + l - 1], t);
					t = fma(c2, pc, t);
					t = fma(c3, P[s + l + 1], t);
					t = fma(c4, P[2 * s + l], t);
					w[u] = t;
					q = fma(t, pc, q);
				});
				ResFix fq[1] = {res_fix_warp(q)};
				q = team_sum(fq);
				if (tid == 0)
					sh.bc = sh.rho / q;
				__syncthreads();
				const double alpha = sh.bc;
				double u0 = 0.0, u1 = 0.0;
				bg_rows_do<kBgG64>(cnt, [&](auto uc) {
					constexpr int u = decltype(uc)::value;
					const int l = tid + u * NT;
					const double d = a.dinv64[g0 + l], xi = a.x[g0 + l];
					const double ri = fma(-alpha, w[u], Rs[l]);
					Rs[l] = ri;
					const double zi = d * ri;
					w[u] = zi;
					u0 = fma(ri, ri, u0);
					u1 = fma(ri, zi, u1);
					a.x[g0 + l] = fma(alpha, P[s + l], xi);
				});
				if (team > 1)
#pragma unroll
					for (int u = 0; u < R; ++u)
						if (edge(u) && tid + u * NT < cnt)
							push(tid + u * NT, w[u]);
				ResFix f[2] = {res_fix_warp(u0), res_fix_warp(u1)};
				const double t = team_sum(f);
				if (tid == 0)
					sh.tot[0] = t;
				if (tid == 32) {
					sh.bc = t / sh.rho;
					sh.rz = t;
				}
				__syncthreads();
				rr = sh.tot[0];
				iters = it + 1;
				if (rr <= t_tol) {
					status = FS_CONVERGED_RTOL;
					break;
				}
				if (!isfinite(rr) || iters >= a.maxiter)
					break;
				bq = sh.bc;
				if (rr <= t_head) {
					handed = true;
					break;
				}
				bg_rows_do<kBgG64>(cnt, [&](auto uc) {
					constexpr int u = decltype(uc)::value;
					const int l = tid + u * NT;
					P[s + l] = fma(bq, P[s + l], w[u]);
				});
				if (team > 1)
					for (int i = tid; i < 2 * s; i += NT) {
						double *p = P + (i < s ? i : chunk + i);
						*p = fma(bq, *p, Z[i]);
					}
				if (tid == 0)
					sh.rho = sh.rz;
				__syncthreads();
			}
			res = sqrt(rr);
			if (!handed && status != FS_CONVERGED_RTOL)
				iters = a.maxiter;  // stopped by maxiter or a non-finite residual
			// the FP32 phase goes on with p = z + beta p
			if (handed)
#pragma unroll
				for (int u = 0; u < R; ++u) {
					const int l = tid + u * NT;
					if (l < cnt)
						xr[u] = (float)P[s + l];
				}
		}
	}

	// ------------------------------------------------------ FP32 phase --
	if (res < tol)
		status = FS_CONVERGED_RTOL;
	else if (iters < a.maxiter) {
		float *P = reinterpret_cast<float *>(bg_dyn);
		float *U2 = P + chunk + 2 * s, *U1 = U2 + chunk + s, *D = U1 + chunk + 1, *DI = D + chunk;
		float *Z = DI + chunk;
		float r[R], w[R];
		team_sync();  // the head's x, and its last pushes have arrived
		for (int i = tid; i < chunk + s; i += NT) {
			const int q = lo + i - s;  // row of the system
			U2[i] = q >= 0 && q < nrow ? a.gu2_32[R0 + q] : 0.f;
		}
		for (int i = tid; i < chunk + 1; i += NT) {
			const int q = lo + i - 1;
			U1[i] = q >= 0 && q < nrow ? a.gu1_32[R0 + q] : 0.f;
		}
		for (int l = tid; l < cnt; l += NT) {
			D[l] = a.gd32[g0 + l];
			DI[l] = a.dinv32[g0 + l];
		}
		for (int i = tid; i < 2 * s; i += NT) {
			P[i < s ? i : chunk + i] = 0.f;
			Z[i] = 0.f;
		}
		for (int l = cnt + tid; l < chunk; l += NT)
			P[s + l] = 0.f;
		__syncthreads();
		auto push = [&](int l, float z) {
			if (l < s && rank > 0)
				*cl.map_shared_rank(&Z[s + l], rank - 1) = z;
			if (l >= chunk - s && rank + 1 < team)
				*cl.map_shared_rank(&Z[l - (chunk - s)], rank + 1) = z;
		};
		// r = b - A x in FP64, z = D^-1 r; ||r|| and r.z
		double rz;
		auto replace = [&](bool edges) {
			double t0 = 0.0, t1 = 0.0;
#pragma unroll 1
			for (int l = tid; l < cnt; l += NT) {
				const double ri = a.b[g0 + l] - row64(a.x, l);
				const float r32 = (float)ri, z = DI[l] * r32;
				a.r32[g0 + l] = r32;
				if (edges)
					push(l, z);
				t0 = fma(ri, ri, t0);
				t1 = fma((double)r32, (double)z, t1);
			}
#pragma unroll
			for (int u = 0; u < R; ++u) {
				const int l = tid + u * NT;
				r[u] = l < cnt ? a.r32[g0 + l] : 0.f;
				w[u] = l < cnt ? DI[l] * r[u] : 0.f;
			}
			double rr;
			sum_all(t0, t1, rr, rz);
			res = sqrt(rr);
			if (tid == 0)
				sh.thr = fmax(res_threshold(a.delta * res), res_threshold(tol));
		};
		replace(false);
		if (handed) {
			++outer;
			// rz over the r.z before the head's last update
			bq = rz / sh.rho;
		}
		{
			const float bf = (float)bq;
#pragma unroll
			for (int u = 0; u < R; ++u) {
				const int l = tid + u * NT;
				if (l < cnt)
					P[s + l] = fmaf(bf, xr[u], w[u]);
				xr[u] = 0.f;
			}
		}
		team_sync();
		if (tid == 0)
			sh.rz = rz;
		if (team > 1) {
			// the halo from its owners (rows past the system stay 0)
			for (int i = tid; i < s; i += NT) {
				if (rank > 0)
					P[i] = *cl.map_shared_rank(&P[chunk + i], rank - 1);
				if (rank + 1 < team && lo + chunk + i < nrow)
					P[chunk + s + i] = *cl.map_shared_rank(&P[s + i], rank + 1);
			}
		}
		__syncthreads();
		if (res < tol)
			status = FS_CONVERGED_RTOL;
		else
			for (int it = iters; it < a.maxiter; ++it) {
				// w = A p, p . w
				cf32 cq{0.f, 0.f};
				bg_rows_do<kBgG32>(cnt, [&](auto uc) {
					constexpr int u = decltype(uc)::value;
					const int l = tid + u * NT;
					const float pc = P[s + l];
					float t = U2[l] * P[l];
					t = fmaf(U1[l], P[s + l - 1], t);
					t = fmaf(D[l], pc, t);
					t = fmaf(U1[l + 1], P[s + l + 1], t);
					t = fmaf(U2[s + l], P[2 * s + l], t);
					w[u] = t;
					cq.add_prod(t, pc);
				});
				const float vq[2] = {cq.hi, cq.lo};
				ResFix fq[1] = {res_fix_warp(vq)};
				const double q = team_sum(fq);
				if (tid == 0) {
					sh.rho = sh.rz;
					sh.af = res_quotient32(sh.rz, q);
				}
				__syncthreads();
				const float af = sh.af;
				// x += alpha p, r -= alpha w, z = D^-1 r, ||r||^2, r . z
				cf32 c0{0.f, 0.f}, c1{0.f, 0.f};
				bg_rows_do<kBgG32>(cnt, [&](auto uc) {
					constexpr int u = decltype(uc)::value;
					const int l = tid + u * NT;
					xr[u] = fmaf(af, P[s + l], xr[u]);
					r[u] = fmaf(-af, w[u], r[u]);
					w[u] = DI[l] * r[u];
					c0.add_prod(r[u], r[u]);
					c1.add_prod(r[u], w[u]);
				});
				if (team > 1)
#pragma unroll
					for (int u = 0; u < R; ++u)
						if (edge(u) && tid + u * NT < cnt)
							push(tid + u * NT, w[u]);
				const float v0[2] = {c0.hi, c0.lo}, v1[2] = {c1.hi, c1.lo};
				ResFix f[2] = {res_fix_warp(v0), res_fix_warp(v1)};
				const double t = team_sum(f);
				iters = it + 1;
				const bool last = iters >= a.maxiter;
				if (tid == 0) {
					sh.act = t <= sh.thr || last || !isfinite(t);
				}
				if (tid == 32) {
					sh.rz = t;
					sh.bf = res_quotient32(t, sh.rho);
				}
				__syncthreads();
				float bf = sh.bf;
				if (sh.act) {
					// fold the correction and replace r by the FP64 residual
#pragma unroll
					for (int u = 0; u < R; ++u) {
						const int l = tid + u * NT;
						if (l < cnt)
							a.x[g0 + l] += (double)xr[u];
						xr[u] = 0.f;
					}
					team_sync();
					replace(team > 1);
					++outer;
					if (res < tol) {
						status = FS_CONVERGED_RTOL;
						break;
					}
					if (last || !isfinite(res))
						break;
					bf = (float)(rz / sh.rho);
					if (tid == 0)
						sh.rz = rz;
				}
				// p = z + beta p, the halo rows too
				bg_rows_do<kBgG32>(cnt, [&](auto uc) {
					constexpr int u = decltype(uc)::value;
					const int l = tid + u * NT;
					P[s + l] = fmaf(bf, P[s + l], w[u]);
				});
				if (team > 1)
					for (int i = tid; i < 2 * s; i += NT) {
						float *p = P + (i < s ? i : chunk + i);
						*p = fmaf(bf, *p, Z[i]);
					}
				__syncthreads();
			}
	}
	double xx = 0.0, unused;
	for (int l = tid; l < cnt; l += NT) {
		const double xi = a.x[g0 + l];
		xx = fma(xi, xi, xx);
	}
	sum_all(xx, 0.0, xx, unused);
	if (rank == 0 && tid == 0) {
		fs_solve_info inf;
		inf.status = status;
		inf.iters = status == FS_CONVERGED_RTOL ? iters : 0;
		inf.restarts = outer;
		inf.res_norm_initial = (float)sh.first[2];
		inf.res_norm_final = (float)res;
		inf.sol_norm_initial = a.zero_guess ? 0.f : (float)sh.first[1];
		inf.sol_norm_final = (float)sqrt(xx);
		inf.rhs_norm = (float)sh.first[0];
		a.info[sys] = inf;
	}
	// no CTA may leave while a peer can still write its shared memory
	if (team > 1)
		cl.sync();
}

}  // namespace

}  // namespace fsg
