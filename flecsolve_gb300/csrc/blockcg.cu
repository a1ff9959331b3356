// Block Jacobi-PCG (O'Leary, "The block conjugate gradient algorithm and
// related methods", LAA 29, 1980) for S = 16 right-hand sides of one
// operator.  No counterpart in the reference, whose solvers take one
// right-hand side per call (cg.hh:43-139 run 16 times).
//
// X, R, P, Q are N x S row-major (the S values of a row contiguous), so the
// SpMM reads A once for all S columns and gathers one S-value row of P per
// nonzero.  Per iteration:
//   Q = A P,  M = P^T Q                 (SpMM with the Gram product fused)
//   alpha = M^-1 G
//   X += P alpha,  R -= Q alpha,  Z = D^-1 R,  G' = Z^T R, ||R_j||
//   beta = G^-1 G',  P = Z + P beta,  G = G'
// Gram products: each CTA walks 64-row steps; thread (g, a, b) of the 256
// accumulates the 4 x 4 block [4a, 4a+4) x [4b, 4b+4) over the step's rows
// g, g + 16, g + 32, g + 48 (register blocking: 16-byte loads, 16 FMAs per
// pair of loads), adds that step sum to its running sum, and the per-CTA
// sums are folded in a fixed two-level order (groups of 32 CTAs, then the
// groups), so the result is deterministic for a given grid.
//
// Two precisions share the kernels (template V):
//  * FP64 (fs_block_cg_solve): every vector and the matrix in FP64.  On this
//    GPU the FP64 pipe issues about 2 FMA per clock per SM, and an iteration
//    is ~5 N S^2 FMA, so this variant is bound by FP64 issue, not by HBM.
//  * FP32 recurrences with FP64 residual replacement
//    (fs_block_cg_solve_mixed): P, Q, R and a correction to X in FP32, FP32
//    matrix values, tile sums accumulated with compensated (two-sum) FP32
//    additions.  When every unconverged column's recurrence residual has
//    dropped by `delta` since the last replacement, or one of them is below
//    its tolerance, or at maxiter, the correction is folded into the FP64 X
//    and R is replaced by the FP64 residual B - A X (FP64 values).  A column
//    converges only on that FP64 residual (the reference's stopping test,
//    cg.hh:55-60, per column).  The search directions are kept across a
//    replacement (reliable updates, van der Vorst & Ye 2000).
// Columns that converge keep iterating inside the block until all have; the
// block stops when every column has converged or at maxiter.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <type_traits>

#include "solver.cuh"

namespace fsg {
namespace {

constexpr int kS = 16;     // right-hand sides per block
constexpr int kTile = 16;  // rows per tile (kTile * kS = 256 threads)
constexpr int BCG_REPLACE = 1;

struct BcgState {
	double G[kS * kS], Gn[kS * kS], M[kS * kS], alpha[kS * kS], beta[kS * kS];
	double ax[kS * kS];  // FP32 recurrences: coefficients of the pending X += P ax
	double bnorm[kS], rnorm[kS], res0[kS], rlast[kS];
	int conv_iter[kS];
	int iter, done, status, flags, replacements;
};

// running sums: plain FP64, or compensated FP32 (Knuth's two-sum on every
// addition; value = hi + lo)
template<class V>
struct BAcc;
template<>
struct BAcc<double> {
	double s = 0.0;
	__device__ void add(double v) { s += v; }
	__device__ double get() const { return s; }
};
template<>
struct BAcc<float> {
	float hi = 0.f, lo = 0.f;
	__device__ void add(float v) {
		const float s = hi + v;
		const float bp = s - hi;
		lo += (hi - (s - bp)) + (v - bp);
		hi = s;
	}
	__device__ double get() const { return (double)hi + (double)lo; }
};

__device__ __forceinline__ bool bcg_skip(const BcgState *st) {
	return st->done || (st->flags & BCG_REPLACE);
}

// sum over a 16-row tile of a[rr][i] * b[rr][j] (start and replacement
// kernels)
template<class V>
__device__ __forceinline__ V tile_dot(const V (*a)[kS], const V (*b)[kS], int i, int j) {
	V t = 0;
#pragma unroll
	for (int rr = 0; rr < kTile; ++rr)
		t = fma(a[rr][i], b[rr][j], t);
	return t;
}

// The last CTA's fold of the per-CTA partials part[b * stride + t] over the
// grid: eight interleaved running sums (eight loads in flight per thread),
// combined in a fixed order -- deterministic for a given grid.
__device__ __forceinline__ double fold_parts(const double *part, int nb, int stride, int t) {
	double a[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
	for (int b = 0; b < nb; b += 8) {
#pragma unroll
		for (int u = 0; u < 8; ++u)
			if (b + u < nb)
				a[u] += __ldcg(part + (size_t)(b + u) * stride + t);
	}
	return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
}

// Per-CTA partials: one row of kW doubles per CTA (the 16 x 16 Gram entries,
// then up to two 16-value column norms).
constexpr int kW = 256 + 2 * kS;
constexpr int kGroup = 32;  // CTAs per first-level fold group

// Two-level fold of the CTAs' partial rows part[b * kW + t], t < nval: the
// last CTA of each group of kGroup CTAs folds the group's rows (in CTA
// order) into gpart, and the last of those folds the group rows (in group
// order) into res (shared memory).  Returns true in that one CTA.  A fixed
// grouping, so the result is deterministic for a given grid; no CTA waits
// for another.  counters: [0] the groups done, [1 + g] group g's CTAs done.
__device__ bool fold2(const double *part, double *gpart, unsigned *counters, int nval,
                      double *res) {
	__shared__ int s_flag;
	const int G = gridDim.x, g = blockIdx.x / kGroup, ng = (G + kGroup - 1) / kGroup;
	const int b0 = g * kGroup, gsize = min(kGroup, G - b0);
	__threadfence();
	__syncthreads();
	if (threadIdx.x == 0)
		s_flag = atomicAdd(counters + 1 + g, 1u) == (unsigned)(gsize - 1);
	__syncthreads();
	if (!s_flag)
		return false;
	__threadfence();
	for (int t = threadIdx.x; t < nval; t += blockDim.x) {
		double a[4] = {0.0, 0.0, 0.0, 0.0};
		for (int b = 0; b < gsize; b += 16) {
			// sixteen loads in flight
			double v[16];
#pragma unroll
			for (int u = 0; u < 16; ++u)
				v[u] = b + u < gsize ? __ldcg(part + (size_t)(b0 + b + u) * kW + t) : 0.0;
#pragma unroll
			for (int u = 0; u < 16; ++u)
				if (b + u < gsize)
					a[u & 3] += v[u];
		}
		gpart[(size_t)g * kW + t] = (a[0] + a[1]) + (a[2] + a[3]);
	}
	if (threadIdx.x == 0)
		counters[1 + g] = 0;
	__threadfence();
	__syncthreads();
	if (threadIdx.x == 0)
		s_flag = atomicAdd(counters, 1u) == (unsigned)(ng - 1);
	__syncthreads();
	if (!s_flag)
		return false;
	__threadfence();
	for (int t = threadIdx.x; t < nval; t += blockDim.x) {
		double a[4] = {0.0, 0.0, 0.0, 0.0};
		for (int q = 0; q < ng; q += 4) {
#pragma unroll
			for (int u = 0; u < 4; ++u)
				if (q + u < ng)
					a[u] += __ldcg(gpart + (size_t)(q + u) * kW + t);
		}
		res[t] = (a[0] + a[1]) + (a[2] + a[3]);
	}
	if (threadIdx.x == 0)
		counters[0] = 0;
	__syncthreads();
	return true;
}

// X = A^-1 B for the 16 x 16 matrix A with 16 right-hand sides B (both in
// shared memory, row-major, padded rows; B overwritten with the solution):
// Gauss-Jordan elimination with partial pivoting by the first 256 threads of
// the CTA, thread (i, j) holding a_ij and b_ij.  Rows stay in place; the pivot
// of a step is the largest of its column by the upper 32 bits (one redux.sync;
// ties to the first row).  Bound by the chain of 16 steps: a reciprocal (561
// cycles) and three FP64 operations a warp each (19 cycles an SM each), two
// barriers; eliminating both triangles leaves no serial back substitution.
// Every thread of the CTA calls it; returns false (the same in every thread)
// on a zero or NaN pivot.
struct SmallLs {
	double A[kS][kS + 1], B[kS][kS + 1];
	double col[kS], fac[kS], rowa[kS], rowb[kS];
};

__device__ bool small_solve_par(SmallLs &L) {
	const bool act = threadIdx.x < kS * kS;
	const int i = threadIdx.x / kS & (kS - 1), j = threadIdx.x % kS, lane = threadIdx.x & 31;
	double a = L.A[i][j], b = L.B[i][j];
	unsigned used = 0;  // rows that have been pivots
	int mine = 0;       // the step whose pivot row i was
	for (int k = 0; k < kS; ++k) {
		if (act && j == k)
			L.col[i] = a;
		__syncthreads();
		const double v = L.col[lane & (kS - 1)];
		const bool open = lane < kS && !(used >> lane & 1);
		const unsigned key = open ? (unsigned)(__double2hiint(v) & 0x7fffffff) : 0u;
		const unsigned top = __reduce_max_sync(0xffffffffu, key);
		const int p = __ffs(__ballot_sync(0xffffffffu, open && key == top)) - 1;
		const unsigned long long pv = (unsigned long long)__double_as_longlong(L.col[p]) & ~(1ull << 63);
		if (pv == 0 || pv > 0x7ffull << 52)
			return false;
		if (act && i == p) {
			L.rowa[j] = a;
			L.rowb[j] = b;
			mine = k;
		}
		if (threadIdx.x < kS) {
			const double f = v * (1.0 / L.col[p]);
			L.fac[lane] = lane == p ? 0.0 : f;
		}
		used |= 1u << p;
		__syncthreads();
		if (act && i != p) {
			const double f = L.fac[i];
			a = fma(-f, L.rowa[j], a);
			b = fma(-f, L.rowb[j], b);
		}
	}
	// row i holds a single entry, in the column of its step
	__syncthreads();
	if (act && j == mine)
		L.fac[i] = 1.0 / a;
	__syncthreads();
	if (act)
		L.B[mine][j] = b * L.fac[i];
	__syncthreads();
	return true;
}

// beta = G^-1 G', G = G' (all threads of the last CTA); false on breakdown
__device__ bool form_beta(BcgState *st, SmallLs &L) {
	const int i = threadIdx.x / kS, j = threadIdx.x % kS;
	const bool act = threadIdx.x < kS * kS;
	if (act) {
		L.A[i][j] = st->G[threadIdx.x];
		L.B[i][j] = st->Gn[threadIdx.x];
	}
	__syncthreads();
	const bool ok = small_solve_par(L);
	if (act) {
		if (ok)
			st->beta[threadIdx.x] = L.B[i][j];
		st->G[threadIdx.x] = st->Gn[threadIdx.x];
	}
	return ok;
}

// The operator for the block SpMM: a grid stencil in symmetric storage (rows
// addressed by their grid coordinates, every neighbour load independent) or
// the CSR rows.
template<class V>
struct BcgOp {
	const int *rp, *col;
	const V *val;
	const V *S;  // grid: diagonal, upper diagonals (null: CSR)
	int64_t ld;
	int nx, ny, nz, K;
};

// ---------------------------------------------------------------------
// Register-blocked layout of the iteration kernels.  Row phase: a thread
// owns a quad of 4 columns of one row (64 rows per 256-thread step; a warp
// reads 8 rows x 64 contiguous bytes of a block vector with 16-byte loads).
// The 16 x 16 coefficient matrices (alpha, beta) are read 16 bytes at a
// time from shared memory, the step's rows of P / Q / Z / R are staged in
// shared memory (rows padded to kLd values: 16-byte aligned, the 8 rows of a
// warp on distinct banks).  Gram phase: thread (g, a, b) accumulates the 4 x 4
// block [4a, 4a+4) x [4b, 4b+4) of the product over the step rows g, g + 16,
// g + 32, g + 48 (one plain step sum per entry, then a compensated running
// sum); at the end the 16 row groups are folded in a fixed order.
constexpr int kQ = 4;
constexpr int kQRows = 256 / (kS / kQ);  // 64 rows per step
constexpr int kLd = kS + 4;

__device__ __forceinline__ void ld4(const double *p, double (&o)[4]) {
	const double2 t0 = *reinterpret_cast<const double2 *>(p);
	const double2 t1 = *reinterpret_cast<const double2 *>(p + 2);
	o[0] = t0.x;
	o[1] = t0.y;
	o[2] = t1.x;
	o[3] = t1.y;
}
__device__ __forceinline__ void st4(float *p, const float (&o)[4]) {
	*reinterpret_cast<float4 *>(p) = make_float4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ void st4(double *p, const double (&o)[4]) {
	*reinterpret_cast<double2 *>(p) = make_double2(o[0], o[1]);
	*reinterpret_cast<double2 *>(p + 2) = make_double2(o[2], o[3]);
}
template<class V>
__device__ __forceinline__ void ldg4(const V *p, V (&o)[4]) {
	if constexpr (sizeof(V) == 4) {
		const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
		o[0] = t.x;
		o[1] = t.y;
		o[2] = t.z;
		o[3] = t.w;
	}
	else {
		const double2 t0 = __ldg(reinterpret_cast<const double2 *>(p));
		const double2 t1 = __ldg(reinterpret_cast<const double2 *>(p) + 1);
		o[0] = t0.x;
		o[1] = t0.y;
		o[2] = t1.x;
		o[3] = t1.y;
	}
}

// Gram accumulation of one step: m[a'][b'] += sum over the group's rows of
// za[row][4a + a'] * zb[row][4b + b'] (plain step sums, compensated across
// steps)
template<class V>
struct GramAcc {
	BAcc<V> m[kQ][kQ];
	__device__ void step(const V (*za)[kLd], const V (*zb)[kLd], int g, int a, int b) {
		V t[kQ][kQ];
#pragma unroll
		for (int i = 0; i < kQ; ++i)
#pragma unroll
			for (int j = 0; j < kQ; ++j)
				t[i][j] = 0;
#pragma unroll
		for (int rr = 0; rr < kQRows / 16; ++rr) {
			const int row = g + 16 * rr;
			V u[kQ], w[kQ];
			ld4(&za[row][kQ * a], u);
			ld4(&zb[row][kQ * b], w);
#pragma unroll
			for (int i = 0; i < kQ; ++i)
#pragma unroll
				for (int j = 0; j < kQ; ++j)
					t[i][j] = fma(u[i], w[j], t[i][j]);
		}
#pragma unroll
		for (int i = 0; i < kQ; ++i)
#pragma unroll
			for (int j = 0; j < kQ; ++j)
				m[i][j].add(t[i][j]);
	}
	// the CTA's 16 x 16 sums into part row b (entry i * 16 + j); red holds
	// 8 x 256 doubles of shared memory.  Row groups g and g + 1 share a warp
	// (xor-16 shuffle), the 8 warps' sums are then folded in warp order.
	__device__ void to_part(double *part, double (*red)[256], int g, int a, int b) {
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
		__syncthreads();
#pragma unroll
		for (int i = 0; i < kQ; ++i)
#pragma unroll
			for (int j = 0; j < kQ; ++j) {
				double v = m[i][j].get();
				v += __shfl_xor_sync(0xffffffffu, v, 16);
				if (lane < 16)
					red[warp][(kQ * a + i) * kS + kQ * b + j] = v;
			}
		__syncthreads();
		double t = 0.0;
#pragma unroll
		for (int w = 0; w < 8; ++w)
			t += red[w][threadIdx.x];
		part[(size_t)blockIdx.x * kW + threadIdx.x] = t;
	}
};

// q[c] = (A P)[r][4 cq + c], the products in the CSR column order
template<class V>
__device__ __forceinline__ void bcg_row4(const BcgOp<V> &A, const V *__restrict__ P, int r, int cq,
                                         V (&q)[kQ]) {
#pragma unroll
	for (int c = 0; c < kQ; ++c)
		q[c] = 0;
	if (A.S) {
		const int64_t nxy = (int64_t)A.nx * A.ny;
		const int i = r % A.nx;
		const int line = r / A.nx;
		const int jj = A.K >= 2 ? line % A.ny : 0, kk = A.K >= 2 ? line / A.ny : 0;
		// the storage holds K upper diagonals: an absent dimension's (unused)
		// coefficient is read from the diagonal, inside the allocation
		const V *U1 = A.S + A.ld, *U2 = A.K >= 2 ? A.S + 2 * A.ld : A.S,
		        *U3 = A.K >= 3 ? A.S + 3 * A.ld : A.S;
		const bool has[7] = {A.K >= 3 && kk > 0, A.K >= 2 && jj > 0, i > 0, true,
		                     i < A.nx - 1, A.K >= 2 && jj < A.ny - 1, A.K >= 3 && kk < A.nz - 1};
		const int64_t off[7] = {-nxy, -A.nx, -1, 0, 1, A.nx, nxy};
		// all loads issued before any use: an absent neighbour reads row r
		// itself (an L1 hit) and its products are skipped
		V a[7], x[7][kQ];
#pragma unroll
		for (int t = 0; t < 7; ++t) {
			const V *U = t == 3 ? A.S : (t < 3 ? (t == 0 ? U3 : t == 1 ? U2 : U1)
			                                   : (t == 4 ? U1 : t == 5 ? U2 : U3));
			const int64_t c = has[t] ? r + off[t] : r;
			a[t] = __ldg(U + (t < 3 ? c : r));
			ldg4(P + (size_t)c * kS + kQ * cq, x[t]);
		}
#pragma unroll
		for (int t = 0; t < 7; ++t)
			if (has[t])
#pragma unroll
				for (int c = 0; c < kQ; ++c)
					q[c] = fma(a[t], x[t][c], q[c]);
		return;
	}
	const int k0 = __ldg(A.rp + r), k1 = __ldg(A.rp + r + 1);
	for (int k = k0; k < k1; k += 4) {
		// a batch of up to 4 entries: the column ids, then the gathers
		int col[4];
		V a[4];
#pragma unroll
		for (int t = 0; t < 4; ++t) {
			const int kk = k + t < k1 ? k + t : k1 - 1;
			col[t] = __ldg(A.col + kk);
			a[t] = __ldg(A.val + kk);
		}
		V x[4][kQ];
#pragma unroll
		for (int t = 0; t < 4; ++t)
			ldg4(P + (size_t)col[t] * kS + kQ * cq, x[t]);
#pragma unroll
		for (int t = 0; t < 4; ++t)
			if (k + t < k1)
#pragma unroll
				for (int c = 0; c < kQ; ++c)
					q[c] = fma(a[t], x[t][c], q[c]);
	}
}

// (A X)[r][j] in FP64, the products in the CSR column order; on a grid every
// load of the row is independent (two dependent loads a product off one)
__device__ __forceinline__ double bcg_row1(const BcgOp<double> &A, const double *__restrict__ X, int r,
                                           int j) {
	double s = 0.0;
	if (A.S) {
		const int nxy = A.nx * A.ny;
		const int line = r / A.nx, i = r - line * A.nx;
		const int kk = A.K >= 3 ? line / A.ny : 0, jj = A.K >= 2 ? line - kk * A.ny : 0;
		const double *U1 = A.S + A.ld, *U2 = A.K >= 2 ? A.S + 2 * A.ld : A.S,
		             *U3 = A.K >= 3 ? A.S + 3 * A.ld : A.S;
		const bool has[7] = {A.K >= 3 && kk > 0, A.K >= 2 && jj > 0, i > 0, true,
		                     i < A.nx - 1, A.K >= 2 && jj < A.ny - 1, A.K >= 3 && kk < A.nz - 1};
		const int off[7] = {-nxy, -A.nx, -1, 0, 1, A.nx, nxy};
		const double *U[7] = {U3, U2, U1, A.S, U1, U2, U3};
		double a[7], x[7];
#pragma unroll
		for (int t = 0; t < 7; ++t) {
			const int c = has[t] ? r + off[t] : r;  // absent: the row itself, not added
			a[t] = __ldg(U[t] + (t < 3 ? c : r));
			x[t] = __ldg(X + (size_t)c * kS + j);
		}
#pragma unroll
		for (int t = 0; t < 7; ++t)
			if (has[t])
				s = fma(a[t], x[t], s);
		return s;
	}
	for (int k = A.rp[r]; k < A.rp[r + 1]; ++k)
		s = fma(A.val[k], X[(size_t)A.col[k] * kS + j], s);
	return s;
}

// Q = A P and the CTA's part of M = P^T Q; the last CTA forms alpha = M^-1 G
template<class V>
__global__ void __launch_bounds__(256)
k_bcg_spmm(int n, BcgOp<V> A, const V *__restrict__ P, V *__restrict__ Q, BcgState *st,
           double *part, double *gpart, unsigned *counters) {
	__shared__ __align__(16) V sp[kQRows][kLd];
	__shared__ __align__(16) V sq[kQRows][kLd];
	__shared__ double red[8][256];
	__shared__ SmallLs L;
	__shared__ double sres[kW];
	if (bcg_skip(st))
		return;
	const int rs = threadIdx.x >> 2, cq = threadIdx.x & 3;
	const int g = threadIdx.x >> 4, ga = (threadIdx.x >> 2) & 3, gb = threadIdx.x & 3;
	const int nsteps = (n + kQRows - 1) / kQRows;
	GramAcc<V> m;
	for (int t = blockIdx.x; t < nsteps; t += gridDim.x) {
		const int r = t * kQRows + rs;
		V q[kQ], p[kQ];
		if (r < n) {
			bcg_row4(A, P, r, cq, q);
			ldg4(P + (size_t)r * kS + kQ * cq, p);
			st4(Q + (size_t)r * kS + kQ * cq, q);
		}
		else {
#pragma unroll
			for (int c = 0; c < kQ; ++c)
				q[c] = p[c] = 0;
		}
		st4(&sp[rs][kQ * cq], p);
		st4(&sq[rs][kQ * cq], q);
		__syncthreads();
		m.step(sp, sq, g, ga, gb);
		__syncthreads();
	}
	m.to_part(part, red, g, ga, gb);
	if (fold2(part, gpart, counters, 256, sres)) {
		const int tr = threadIdx.x / kS, tj = threadIdx.x % kS;
		const double v = sres[threadIdx.x];
		st->M[threadIdx.x] = v;
		L.A[tr][tj] = v;
		L.B[tr][tj] = st->G[threadIdx.x];
		__syncthreads();
		const bool ok = small_solve_par(L);
		if (ok)
			st->alpha[threadIdx.x] = L.B[tr][tj];
		if (threadIdx.x == 0 && !ok) {
			st->done = 1;
			st->status = FS_DIVERGED_BREAKDOWN;
		}
	}
}

// the scalar part of an update, by the last CTA (Gn and rnorm in place):
// counts the iteration, then
//  * FP64 (delta <= 0): marks the columns below tolerance, stops when all
//    are, else forms beta;
//  * mixed (delta > 0): requests a residual replacement when every
//    unconverged column has dropped by delta since the last one, or one is
//    below tolerance, or at maxiter; else forms beta.
__device__ void update_finish(BcgState *st, SmallLs &L, int &s_beta, double tolf, int maxiter,
                              double delta) {
	__syncthreads();
	if (threadIdx.x < 32) {
		// lane j: column j (the others repeat the last)
		const int lane = threadIdx.x, j = min(lane, kS - 1);
		const int it = st->iter + 1;
		const double rn = st->rnorm[j], bn = st->bnorm[j], rl = st->rlast[j];
		int conv = st->conv_iter[j];
		const bool finite = __all_sync(0xffffffffu, isfinite(rn)), below = rn < tolf * bn;
		bool beta = false;
		__syncwarp();
		if (delta <= 0.0) {
			if (conv == 0 && below) {
				conv = it;
				if (lane < kS)
					st->conv_iter[j] = it;
			}
			const bool all = __all_sync(0xffffffffu, conv != 0);
			beta = !all && finite && it < maxiter;
			if (lane == 0 && !beta) {
				st->done = 1;
				st->status = all ? FS_CONVERGED_RTOL : !finite ? FS_DIVERGED_BREAKDOWN : FS_DIVERGED_ITERS;
			}
		}
		else {
			const bool open = conv == 0;
			const bool dropped = !open || !(rl > 0.0) || rn / rl < delta;
			const bool replace = it >= maxiter || !finite || __any_sync(0xffffffffu, open && below) ||
			                     __all_sync(0xffffffffu, dropped);
			beta = !replace;
			if (lane == 0 && replace)
				st->flags |= BCG_REPLACE;
		}
		if (lane == 0) {
			st->iter = it;
			s_beta = beta;
		}
	}
	__syncthreads();
	if (s_beta && !form_beta(st, L) && threadIdx.x == 0) {
		st->done = 1;
		st->status = FS_DIVERGED_BREAKDOWN;
	}
}

// X += P alpha, R -= Q alpha, Z = D^-1 R; G' = Z^T R and ||R_j||^2 parts,
// then update_finish by the last CTA
template<class V>
__global__ void __launch_bounds__(256)
k_bcg_update(int n, V *__restrict__ X, const V *__restrict__ P, V *__restrict__ R,
             const V *__restrict__ Q, const V *__restrict__ dinv, BcgState *st, double *part,
             double *gpart, unsigned *counters, double tolf, int maxiter, double delta) {
	__shared__ __align__(16) V sa[kS][kLd];
	__shared__ __align__(16) V sp[kQRows][kLd];
	__shared__ __align__(16) V sq[kQRows][kLd];
	__shared__ double red[8][256];
	__shared__ SmallLs L;
	__shared__ int s_beta;
	__shared__ double sres[kW];
	if (bcg_skip(st))
		return;
	{
		const int tr = threadIdx.x / kS, tj = threadIdx.x % kS;
		sa[tr][tj] = (V)st->alpha[threadIdx.x];
	}
	__syncthreads();
	const int rs = threadIdx.x >> 2, cq = threadIdx.x & 3;
	const int g = threadIdx.x >> 4, ga = (threadIdx.x >> 2) & 3, gb = threadIdx.x & 3;
	const int nsteps = (n + kQRows - 1) / kQRows;
	GramAcc<V> gm;
	BAcc<V> nr[kQ];
	for (int t = blockIdx.x; t < nsteps; t += gridDim.x) {
		const int r = t * kQRows + rs;
		V p[kQ], q[kQ], x[kQ], rv[kQ];
		V dr = 0;
		if (r < n) {
			ldg4(P + (size_t)r * kS + kQ * cq, p);
			ldg4(Q + (size_t)r * kS + kQ * cq, q);
			ld4(X + (size_t)r * kS + kQ * cq, x);
			ld4(R + (size_t)r * kS + kQ * cq, rv);
			dr = dinv ? __ldg(dinv + r) : V(1);
		}
		else {
#pragma unroll
			for (int c = 0; c < kQ; ++c)
				p[c] = q[c] = x[c] = rv[c] = 0;
		}
		st4(&sp[rs][kQ * cq], p);
		st4(&sq[rs][kQ * cq], q);
		__syncthreads();
		// x += P[r][:] alpha[:, quad], r -= Q[r][:] alpha[:, quad]
#pragma unroll
		for (int i4 = 0; i4 < kS / kQ; ++i4) {
			V pr[kQ], qr[kQ];
			ld4(&sp[rs][kQ * i4], pr);
			ld4(&sq[rs][kQ * i4], qr);
#pragma unroll
			for (int ii = 0; ii < kQ; ++ii) {
				V al[kQ];
				ld4(&sa[kQ * i4 + ii][kQ * cq], al);
#pragma unroll
				for (int c = 0; c < kQ; ++c) {
					x[c] = fma(pr[ii], al[c], x[c]);
					rv[c] = fma(-qr[ii], al[c], rv[c]);
				}
			}
		}
		V z[kQ];
#pragma unroll
		for (int c = 0; c < kQ; ++c) {
			z[c] = dr * rv[c];
			if (r < n)
				nr[c].add(rv[c] * rv[c]);
		}
		if (r < n) {
			st4(X + (size_t)r * kS + kQ * cq, x);
			st4(R + (size_t)r * kS + kQ * cq, rv);
		}
		else {
#pragma unroll
			for (int c = 0; c < kQ; ++c)
				z[c] = rv[c] = 0;
		}
		__syncthreads();
		// the staged P and Q are consumed: stage Z and R for G' = Z^T R
		st4(&sp[rs][kQ * cq], z);
		st4(&sq[rs][kQ * cq], rv);
		__syncthreads();
		gm.step(sp, sq, g, ga, gb);
		__syncthreads();
	}
	gm.to_part(part, red, g, ga, gb);
	// column norms: this thread's 4 columns, folded over the 64 row slots
	// (in the fold buffer, once every thread has read it)
	double (*cn)[kS] = reinterpret_cast<double (*)[kS]>(&red[0][0]);
	__syncthreads();
#pragma unroll
	for (int c = 0; c < kQ; ++c)
		cn[rs][kQ * cq + c] = nr[c].get();
	__syncthreads();
	if (threadIdx.x < kS) {
		double c = 0.0;
		for (int q = 0; q < kQRows; ++q)
			c += cn[q][threadIdx.x];
		part[(size_t)blockIdx.x * kW + 256 + threadIdx.x] = c;
	}
	if (fold2(part, gpart, counters, 256 + kS, sres)) {
		st->Gn[threadIdx.x] = sres[threadIdx.x];
		if (threadIdx.x < kS)
			st->rnorm[threadIdx.x] = sqrt(sres[256 + threadIdx.x]);
		update_finish(st, L, s_beta, tolf, maxiter, delta);
	}
}

// P = Z + P beta (Z = D^-1 R)
template<class V>
__global__ void __launch_bounds__(256)
k_bcg_dir(int n, V *__restrict__ P, const V *__restrict__ R, const V *__restrict__ dinv,
          const BcgState *st) {
	__shared__ __align__(16) V sb[kS][kLd];
	__shared__ __align__(16) V sp[kQRows][kLd];
	if (bcg_skip(st))
		return;
	{
		const int tr = threadIdx.x / kS, tj = threadIdx.x % kS;
		sb[tr][tj] = (V)st->beta[threadIdx.x];
	}
	const int rs = threadIdx.x >> 2, cq = threadIdx.x & 3;
	const int nsteps = (n + kQRows - 1) / kQRows;
	for (int t = blockIdx.x; t < nsteps; t += gridDim.x) {
		const int r = t * kQRows + rs;
		V p[kQ], pn[kQ];
		if (r < n) {
			ld4(P + (size_t)r * kS + kQ * cq, p);
			ldg4(R + (size_t)r * kS + kQ * cq, pn);
			const V d = dinv ? __ldg(dinv + r) : V(1);
#pragma unroll
			for (int c = 0; c < kQ; ++c)
				pn[c] = d * pn[c];
		}
		else {
#pragma unroll
			for (int c = 0; c < kQ; ++c)
				p[c] = pn[c] = 0;
		}
		__syncthreads();
		st4(&sp[rs][kQ * cq], p);
		__syncthreads();
#pragma unroll
		for (int i4 = 0; i4 < kS / kQ; ++i4) {
			V pr[kQ];
			ld4(&sp[rs][kQ * i4], pr);
#pragma unroll
			for (int ii = 0; ii < kQ; ++ii) {
				V be[kQ];
				ld4(&sb[kQ * i4 + ii][kQ * cq], be);
#pragma unroll
				for (int c = 0; c < kQ; ++c)
					pn[c] = fma(pr[ii], be[c], pn[c]);
			}
		}
		if (r < n)
			st4(P + (size_t)r * kS + kQ * cq, pn);
	}
}

// ---------------------------------------------------------------------
// The iteration kernels of the FP32 recurrences.  A warp takes tiles of 32
// rows by itself: lane (rs, cq) owns the quad cq of rows rs, rs + 8, rs + 16
// and rs + 24, so that the coefficient matrices (alpha, beta), read 16 bytes at
// a time, serve four rows.  A tile's rows are contiguous (2 KB a block
// vector): lane 0 fetches those of the warp's next tiles with bulk copies
// (cp.async.bulk) into a ring of stages of the warp's own, completing on a
// full mbarrier per stage, so the loads in flight cost no registers and only
// __syncwarp orders a tile.  Products of pairs of columns are packed
// (fma.rn.f32x2).
//
// Gram products are symmetric in exact arithmetic (P^T A P, R^T D^-1 R), so
// only the ten 4 x 4 blocks on and above the diagonal are formed, three row
// groups of the tile side by side (30 lanes), plain sums of at most four rows
// added to the running sum with two-sum, and mirrored.
//
// The solution step X += P alpha of an iteration stays pending (st->ax) for
// the direction kernel, which reads P anyway: 10 block vectors an iteration
// instead of 11.
//
// Bound: HBM for the direction kernel; the L2 reads of five row ranges and the
// instructions (some 560 a warp and tile) for the SpMM; HBM and the scalar
// tail for the update.  At 128^3 x 16 they move 302, 402 and 670 MB (45, 60 and
// 100 us at the measured copy rate) and take 112, 110 and 101 us, the two
// reductions' tails (two-level fold, 16 x 16 elimination) about 25 us of the
// first two.  The 64-row steps with three block barriers each that they
// replace took 239, 312 and 96 us.
constexpr int kWRows = 32;              // rows per warp tile
constexpr int kSymBlocks = 10;          // 4 x 4 blocks on and above the diagonal
constexpr int kSymVals = 16 * kSymBlocks;

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
	uint64_t d;
	asm("fma.rn.f32x2 %0, %1, %2, %3;"
	    : "=l"(d)
	    : "l"(*reinterpret_cast<const uint64_t *>(&a)), "l"(*reinterpret_cast<const uint64_t *>(&b)),
	      "l"(*reinterpret_cast<const uint64_t *>(&c)));
	return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
	uint64_t d;
	asm("add.rn.f32x2 %0, %1, %2;"
	    : "=l"(d)
	    : "l"(*reinterpret_cast<const uint64_t *>(&a)), "l"(*reinterpret_cast<const uint64_t *>(&b)));
	return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
	uint64_t d;
	asm("sub.rn.f32x2 %0, %1, %2;"
	    : "=l"(d)
	    : "l"(*reinterpret_cast<const uint64_t *>(&a)), "l"(*reinterpret_cast<const uint64_t *>(&b)));
	return *reinterpret_cast<float2 *>(&d);
}

// compensated running sums of a pair of values (BAcc<float> on both lanes)
struct BAcc2 {
	float2 hi = {0.f, 0.f}, lo = {0.f, 0.f};
	__device__ void add(float2 v) {
		const float2 s = add2(hi, v);
		const float2 bp = sub2(s, hi);
		lo = add2(lo, add2(sub2(hi, sub2(s, bp)), sub2(v, bp)));
		hi = s;
	}
};

// one quad of a row as two pairs
struct Quad {
	float2 a, b;
};
__device__ __forceinline__ Quad ldq(const float *p) {
	const float4 t = *reinterpret_cast<const float4 *>(p);
	return {make_float2(t.x, t.y), make_float2(t.z, t.w)};
}
__device__ __forceinline__ void stq(float *p, Quad q) {
	*reinterpret_cast<float4 *>(p) = make_float4(q.a.x, q.a.y, q.b.x, q.b.y);
}
__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }

// block number -> (block row, block column), a <= b
__device__ __forceinline__ void sym_block(int blk, int &a, int &b) {
	a = blk < 4 ? 0 : blk < 7 ? 1 : blk < 9 ? 2 : 3;
	b = blk - (a == 0 ? 0 : a == 1 ? 3 : a == 2 ? 5 : 6);
}

// the warp's running sums: lane = block + 10 x row group (lanes 30, 31 idle)
struct SymGram {
	BAcc2 m[4][2];
	int a4, b4, g;
	__device__ void init() {
		const int lane = threadIdx.x & 31;
		int a, b;
		sym_block(lane % kSymBlocks, a, b);
		a4 = 4 * a;
		b4 = 4 * b;
		g = lane / kSymBlocks;
	}
	// za^T zb over the tile's 32 rows (16 values each, in shared memory)
	__device__ void tile(const float *za, const float *zb) {
		if (g >= 3)
			return;
#pragma unroll
		for (int h = 0; h < 3; ++h) {
			float2 t[4][2];
#pragma unroll
			for (int i = 0; i < 4; ++i)
				t[i][0] = t[i][1] = make_float2(0.f, 0.f);
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				const int row = g + 3 * (4 * h + q);
				if (row < kWRows) {
					const float4 u = *reinterpret_cast<const float4 *>(za + row * kS + a4);
					const Quad w = ldq(zb + row * kS + b4);
					const float uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
					for (int i = 0; i < 4; ++i) {
						t[i][0] = fma2(dup(uu[i]), w.a, t[i][0]);
						t[i][1] = fma2(dup(uu[i]), w.b, t[i][1]);
					}
				}
			}
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				m[i][0].add(t[i][0]);
				m[i][1].add(t[i][1]);
			}
		}
	}
	// the CTA's sums of its NW warps, in that order (each warp's three row
	// groups merged as compensated pairs), into part[e], e = 16 block + 4 i + j;
	// red: NW x kSymVals doubles
	template<int NW>
	__device__ void to_part(double *part, double *red) {
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
		for (int i = 0; i < 4; ++i)
#pragma unroll
			for (int j = 0; j < 2; ++j) {
				BAcc2 s = m[i][j];
#pragma unroll
				for (int o = 1; o < 3; ++o) {
					const int src = lane + o * kSymBlocks;
					const float2 h = {__shfl_sync(0xffffffffu, m[i][j].hi.x, src),
					                  __shfl_sync(0xffffffffu, m[i][j].hi.y, src)};
					const float2 l = {__shfl_sync(0xffffffffu, m[i][j].lo.x, src),
					                  __shfl_sync(0xffffffffu, m[i][j].lo.y, src)};
					s.add(h);
					s.lo = add2(s.lo, l);
				}
				if (lane < kSymBlocks) {
					double *d = red + (size_t)warp * kSymVals + lane * 16 + 4 * i + 2 * j;
					d[0] = (double)s.hi.x + (double)s.lo.x;
					d[1] = (double)s.hi.y + (double)s.lo.y;
				}
			}
		__syncthreads();
		if (threadIdx.x < kSymVals) {
			double t = 0.0;
#pragma unroll
			for (int w = 0; w < NW; ++w)
				t += red[(size_t)w * kSymVals + threadIdx.x];
			part[threadIdx.x] = t;
		}
	}
};

// entry e of the folded half -> its place(s) in the 16 x 16 matrix
__device__ __forceinline__ double sym_at(const double *res, int i, int j) {
	if (i / 4 > j / 4) {
		const int t = i;
		i = j;
		j = t;
	}
	const int a = i / 4, b = j / 4;
	const int blk = (a == 0 ? 0 : a == 1 ? 3 : a == 2 ? 5 : 6) + b;
	return res[16 * blk + 4 * (i & 3) + (j & 3)];
}


// The stages of one warp: S of BYTES each, filled in turn for the warp's tiles
// t0, t0 + step, ...
template<int S, int BYTES>
struct WarpRing {
	unsigned char *buf;
	unsigned long long *full;  // S barriers
	unsigned *err;
	int issued = 0, used = 0;
	__device__ void init(unsigned char *b, unsigned long long *f, unsigned *e) {
		buf = b;
		full = f;
		err = e;
		if ((threadIdx.x & 31) == 0) {
			for (int s = 0; s < S; ++s)
				mbar_init(&full[s], 1);
			mbar_init_fence();
		}
		__syncwarp();
	}
	// the whole warp, before lane 0 refills a stage: its accesses to the stage
	// precede the copy
	__device__ static void release() {
		asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
		__syncwarp();
	}
	// lane 0: begins the next stage and returns it
	__device__ unsigned char *begin(unsigned bytes) {
		const int s = issued++ % S;
		mbar_arrive_expect_tx(&full[s], bytes);
		return buf + (size_t)s * BYTES;
	}
	__device__ unsigned long long *bar() const { return &full[(issued - 1) % S]; }
	// the whole warp: the next filled stage, null when the wait ran out
	__device__ unsigned char *next() {
		const int s = used % S;
		const bool ok = mbar_wait(&full[s], (unsigned)(used / S & 1));
		++used;
		if (!__all_sync(0xffffffffu, ok)) {
			if ((threadIdx.x & 31) == 0)
				atomicOr(err, 1u);
			return nullptr;
		}
		return buf + (size_t)s * BYTES;
	}
	// lane 0, before the CTA leaves: every copy has landed
	__device__ void drain() {
		for (; used < issued; ++used)
			mbar_wait(&full[used % S], (unsigned)(used / S & 1));
	}
};

constexpr int kTileBytes = kWRows * kS * (int)sizeof(float);  // one block vector's rows of a tile

// SpMM: 16 warps, a stage of P's rows t - 1 .. t + 32 (the tile and a row on
// either side) and the tile's rows at -nx ny, -nx, +nx and +nx ny each; Q's rows
// go over the first of those (a lane reads there only what it overwrites).
// Sixteen warps that take turns hide a tile's loads better than eight with
// two stages do (112 us at 128^3): a tile takes a warp some 560 instructions.
constexpr int kSpWarps = 16, kSpStages = 1;
constexpr int kSpCentre = kTileBytes + 2 * kS * (int)sizeof(float);
constexpr int kSpBytes = kSpCentre + 4 * kTileBytes;
// (off a grid one array each of P's and Q's rows)
template<bool GRID>
constexpr int kSpWarpBytes = GRID ? kSpStages * kSpBytes : 2 * kTileBytes;
template<bool GRID>
constexpr int kSpSmem = kSpWarps * kSpWarpBytes<GRID>;
// update: 16 warps, three stages of Q and R; direction: two of X, P and R
constexpr int kUpWarps = 16, kUpStages = 3, kUpBytes = 2 * kTileBytes;
constexpr int kUpSmem = kUpWarps * kUpStages * kUpBytes;
constexpr int kDirWarps = 16, kDirStages = 2, kDirBytes = 3 * kTileBytes;
constexpr int kDirSmem = kDirWarps * kDirStages * kDirBytes;
static_assert(kSpSmem<false> >= kSpWarps * kSymVals * 8 && kUpSmem >= kUpWarps * kSymVals * 8,
              "the fold fits over the stages");

// Q = A P and M = P^T Q; the last CTA forms alpha = M^-1 G.  GRID: neighbours
// by grid coordinates out of the staged rows; else the CSR rows, P gathered.
template<bool GRID>
__global__ void __launch_bounds__(kSpWarps * 32, 1)
k_bcgf_spmm(int n, BcgOp<float> A, const float *__restrict__ P, float *__restrict__ Q, BcgState *st,
            double *part, double *gpart, unsigned *counters, unsigned *err) {
	extern __shared__ __align__(128) unsigned char dyn[];
	__shared__ unsigned long long full[kSpWarps * kSpStages];
	__shared__ SmallLs L;
	__shared__ double sres[kW];
	pdl_wait();
	pdl_trigger();
	if (bcg_skip(st))
		return;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rs = lane >> 2, cq = lane & 3;
	unsigned char *mine = dyn + warp * kSpWarpBytes<GRID>;
	SymGram m;
	m.init();
	const int ntile = (n + kWRows - 1) / kWRows, step = gridDim.x * kSpWarps;
	const int t0 = blockIdx.x * kSpWarps + warp;
	const int nxy = A.nx * A.ny;
	const int offs[4] = {-nxy, -A.nx, A.nx, nxy};  // the outer neighbours, by stage slot
	if constexpr (GRID) {
		WarpRing<kSpStages, kSpBytes> ring;
		ring.init(mine, full + warp * kSpStages, err);
		// the copies of tile t: row ranges clipped to [0, n)
		auto fetch = [&](int t) {
			const int r0 = t * kWRows, r1 = min(r0 + kWRows, n);
			int lo[5], hi[5], at[5];
			lo[4] = max(r0 - 1, 0);
			hi[4] = min(r1 + 1, n);
			at[4] = (lo[4] - (r0 - 1)) * kS * 4;
			unsigned bytes = (unsigned)(hi[4] - lo[4]) * kS * 4;
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				const bool dim = (q == 1 || q == 2) ? A.K >= 2 : A.K >= 3;
				lo[q] = max(r0 + offs[q], 0);
				hi[q] = dim ? min(r1 + offs[q], n) : 0;
				at[q] = kSpCentre + q * kTileBytes + (lo[q] - (r0 + offs[q])) * kS * 4;
				bytes += hi[q] > lo[q] ? (unsigned)(hi[q] - lo[q]) * kS * 4 : 0u;
			}
			unsigned char *d = ring.begin(bytes);
#pragma unroll
			for (int q = 0; q < 5; ++q)
				if (hi[q] > lo[q])
					bulk_g2s(d + at[q], P + (size_t)lo[q] * kS, (unsigned)(hi[q] - lo[q]) * kS * 4, ring.bar());
		};
		if (lane == 0)
			for (int q = 0; q < kSpStages && t0 + q * step < ntile; ++q)
				fetch(t0 + q * step);
		const float *D = A.S, *U1 = A.S + A.ld;
		const float *U2 = A.K >= 2 ? A.S + 2 * A.ld : A.S, *U3 = A.K >= 3 ? A.S + 3 * A.ld : A.S;
		// one tile ahead, the coefficients of the tile's row `lane`: z-, y-, x-,
		// diagonal, x+, y+, z+; returns which of them the row has
		auto coefs = [&](int t, float (&c)[7]) -> unsigned {
			const int r = t * kWRows + lane;
			unsigned has = 0;
#pragma unroll
			for (int q = 0; q < 7; ++q)
				c[q] = 0.f;
			if (t < ntile && r < n) {
				const int line = r / A.nx, i = r - line * A.nx;
				const int kk = A.K >= 3 ? line / A.ny : 0, jj = A.K >= 2 ? line - kk * A.ny : 0;
				has = 8u | (i > 0 ? 4u : 0u) | (i < A.nx - 1 ? 16u : 0u) |
				      (A.K >= 2 && jj > 0 ? 2u : 0u) | (A.K >= 2 && jj < A.ny - 1 ? 32u : 0u) |
				      (A.K >= 3 && kk > 0 ? 1u : 0u) | (A.K >= 3 && kk < A.nz - 1 ? 64u : 0u);
				const float *at[7] = {U3 + (r - nxy), U2 + (r - A.nx), U1 + (r - 1), D + r, U1 + r, U2 + r, U3 + r};
#pragma unroll
				for (int q = 0; q < 7; ++q)
					if (has >> q & 1)
						c[q] = __ldg(at[q]);
			}
			return has;
		};
		float c[7];
		unsigned has = coefs(t0, c);
		bool alive = true;
		for (int t = t0; t < ntile; t += step) {
			unsigned char *stage = ring.next();
			if (!stage) {
				alive = false;
				break;
			}
			float *ctr = reinterpret_cast<float *>(stage) + kS;  // the tile's rows
			float *out[4];
#pragma unroll
			for (int q = 0; q < 4; ++q)
				out[q] = reinterpret_cast<float *>(stage + kSpCentre + q * kTileBytes);
			float cn[7];
			const unsigned hn = coefs(t + step, cn);
#pragma unroll
			for (int u = 0; u < 4; ++u) {
				const int row = rs + 8 * u, r = t * kWRows + row;
				// row's coefficients sit in lane `row`
				float a[7];
#pragma unroll
				for (int q = 0; q < 7; ++q)
					a[q] = __shfl_sync(0xffffffffu, c[q], row);
				const unsigned h = __shfl_sync(0xffffffffu, has, row);
				Quad s{{0.f, 0.f}, {0.f, 0.f}};
				const float *x[7] = {out[0], out[1], ctr - kS, ctr, ctr + kS, out[2], out[3]};
				if (r < n) {
#pragma unroll
					for (int q = 0; q < 7; ++q)
						if (h >> q & 1) {
							const Quad v = ldq(x[q] + row * kS + kQ * cq);
							s.a = fma2(dup(a[q]), v.a, s.a);
							s.b = fma2(dup(a[q]), v.b, s.b);
						}
					stq(Q + (size_t)r * kS + kQ * cq, s);
				}
				else
					stq(ctr + row * kS + kQ * cq, s);  // no row: zeros for the Gram product
				stq(out[0] + row * kS + kQ * cq, s);
			}
			__syncwarp();
			m.tile(ctr, out[0]);
			ring.release();
			if (lane == 0 && t + kSpStages * step < ntile)
				fetch(t + kSpStages * step);
#pragma unroll
			for (int q = 0; q < 7; ++q)
				c[q] = cn[q];
			has = hn;
		}
		if (lane == 0 && !alive)
			ring.drain();
	}
	else {
		float *sp = reinterpret_cast<float *>(mine), *sq = sp + kWRows * kS;
		for (int t = t0; t < ntile; t += step) {
#pragma unroll
			for (int u = 0; u < 4; ++u) {
				const int r = t * kWRows + rs + 8 * u;
				float q[kQ] = {0.f, 0.f, 0.f, 0.f}, p[kQ] = {0.f, 0.f, 0.f, 0.f};
				if (r < n) {
					bcg_row4(A, P, r, cq, q);
					ldg4(P + (size_t)r * kS + kQ * cq, p);
					st4(Q + (size_t)r * kS + kQ * cq, q);
				}
				st4(sp + (rs + 8 * u) * kS + kQ * cq, p);
				st4(sq + (rs + 8 * u) * kS + kQ * cq, q);
			}
			__syncwarp();
			m.tile(sp, sq);
			__syncwarp();
		}
	}
	__syncthreads();
	m.to_part<kSpWarps>(part + (size_t)blockIdx.x * kW, reinterpret_cast<double *>(dyn));
	if (fold2(part, gpart, counters, kSymVals, sres)) {
		const int tr = threadIdx.x / kS, tj = threadIdx.x % kS;
		const bool act = threadIdx.x < kS * kS;
		if (act) {
			const double v = sym_at(sres, tr, tj);
			st->M[threadIdx.x] = v;
			st->ax[threadIdx.x] = 0.0;  // the direction kernel has applied the last step
			L.A[tr][tj] = v;
			L.B[tr][tj] = st->G[threadIdx.x];
		}
		__syncthreads();
		const bool ok = small_solve_par(L);
		if (act && ok)
			st->alpha[threadIdx.x] = L.B[tr][tj];
		if (threadIdx.x == 0 && !ok) {
			st->done = 1;
			st->status = FS_DIVERGED_BREAKDOWN;
		}
	}
}

// R -= Q alpha, G' = R^T D^-1 R, ||R_j||^2; then the iteration's scalar part
// (update_finish).  The solution step is left pending.
__global__ void __launch_bounds__(kUpWarps * 32, 1)
k_bcgf_update(int n, float *__restrict__ R, const float *__restrict__ Q,
              const float *__restrict__ dinv, BcgState *st, double *part, double *gpart,
              unsigned *counters, double tolf, int maxiter, double delta, unsigned *err) {
	extern __shared__ __align__(128) unsigned char dyn[];
	__shared__ unsigned long long full[kUpWarps * kUpStages];
	__shared__ __align__(16) float sa[kS][kS];
	__shared__ SmallLs L;
	__shared__ int s_beta;
	__shared__ double sres[kW];
	pdl_wait();
	pdl_trigger();
	if (bcg_skip(st))
		return;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rs = lane >> 2, cq = lane & 3;
	WarpRing<kUpStages, kUpBytes> ring;
	ring.init(dyn + warp * kUpStages * kUpBytes, full + warp * kUpStages, err);
	const int ntile = (n + kWRows - 1) / kWRows, step = gridDim.x * kUpWarps;
	const int t0 = blockIdx.x * kUpWarps + warp;
	auto fetch = [&](int t) {
		const unsigned bytes = (unsigned)min(kWRows, n - t * kWRows) * kS * 4;
		unsigned char *d = ring.begin(2 * bytes);
		bulk_g2s(d, Q + (size_t)t * kWRows * kS, bytes, ring.bar());
		bulk_g2s(d + kTileBytes, R + (size_t)t * kWRows * kS, bytes, ring.bar());
	};
	if (lane == 0)
		for (int q = 0; q < kUpStages && t0 + q * step < ntile; ++q)
			fetch(t0 + q * step);
	if (threadIdx.x < kS * kS)
		sa[threadIdx.x / kS][threadIdx.x % kS] = -(float)st->alpha[threadIdx.x];
	__syncthreads();
	SymGram gm;
	gm.init();
	BAcc2 nr[2];
	bool alive = true;
	for (int t = t0; t < ntile; t += step) {
		float d[4];
#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const int r = t * kWRows + rs + 8 * u;
			d[u] = r < n ? (dinv ? __ldg(dinv + r) : 1.f) : 0.f;
		}
		unsigned char *stage = ring.next();
		if (!stage) {
			alive = false;
			break;
		}
		float *s0 = reinterpret_cast<float *>(stage), *s1 = s0 + kWRows * kS;  // Q, R
		Quad rv[4];
#pragma unroll
		for (int u = 0; u < 4; ++u)
			rv[u] = ldq(s1 + (rs + 8 * u) * kS + kQ * cq);
#pragma unroll
		for (int i4 = 0; i4 < 4; ++i4) {
			float4 q[4];
#pragma unroll
			for (int u = 0; u < 4; ++u)
				q[u] = *reinterpret_cast<const float4 *>(s0 + (rs + 8 * u) * kS + 4 * i4);
#pragma unroll
			for (int ii = 0; ii < 4; ++ii) {
				const Quad al = ldq(&sa[4 * i4 + ii][kQ * cq]);
#pragma unroll
				for (int u = 0; u < 4; ++u) {
					const float2 v = dup(ii == 0 ? q[u].x : ii == 1 ? q[u].y : ii == 2 ? q[u].z : q[u].w);
					rv[u].a = fma2(v, al.a, rv[u].a);
					rv[u].b = fma2(v, al.b, rv[u].b);
				}
			}
		}
		__syncwarp();
		// R's rows and D^-1 R over the stage, for the Gram product
#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const int r = t * kWRows + rs + 8 * u;
			if (r < n)
				stq(R + (size_t)r * kS + kQ * cq, rv[u]);
			else
				rv[u] = {{0.f, 0.f}, {0.f, 0.f}};
			nr[0].add(make_float2(rv[u].a.x * rv[u].a.x, rv[u].a.y * rv[u].a.y));
			nr[1].add(make_float2(rv[u].b.x * rv[u].b.x, rv[u].b.y * rv[u].b.y));
			stq(s1 + (rs + 8 * u) * kS + kQ * cq, rv[u]);
			const Quad z{make_float2(d[u] * rv[u].a.x, d[u] * rv[u].a.y),
			             make_float2(d[u] * rv[u].b.x, d[u] * rv[u].b.y)};
			stq(s0 + (rs + 8 * u) * kS + kQ * cq, z);
		}
		__syncwarp();
		gm.tile(s0, s1);
		ring.release();
		if (lane == 0 && t + kUpStages * step < ntile)
			fetch(t + kUpStages * step);
	}
	if (lane == 0 && !alive)
		ring.drain();
	__syncthreads();
	gm.to_part<kUpWarps>(part + (size_t)blockIdx.x * kW, reinterpret_cast<double *>(dyn));
	// column norms: each lane's four columns, over the CTA's row slots
	double (*cn)[kS] = reinterpret_cast<double (*)[kS]>(dyn);
	__syncthreads();
#pragma unroll
	for (int h = 0; h < 2; ++h) {
		cn[warp * 8 + rs][kQ * cq + 2 * h] = (double)nr[h].hi.x + (double)nr[h].lo.x;
		cn[warp * 8 + rs][kQ * cq + 2 * h + 1] = (double)nr[h].hi.y + (double)nr[h].lo.y;
	}
	__syncthreads();
	if (threadIdx.x < kS * kS) {
		// 16 partial sums of a column, then their sum
		double c = 0.0;
		for (int q = threadIdx.x / kS; q < kUpWarps * 8; q += kS)
			c += cn[q][threadIdx.x % kS];
		L.A[threadIdx.x / kS][threadIdx.x % kS] = c;
	}
	__syncthreads();
	if (threadIdx.x < kS) {
		double c = 0.0;
#pragma unroll
		for (int q = 0; q < kS; ++q)
			c += L.A[q][threadIdx.x];
		part[(size_t)blockIdx.x * kW + kSymVals + threadIdx.x] = c;
	}
	if (fold2(part, gpart, counters, kSymVals + kS, sres)) {
		if (threadIdx.x < kS * kS) {
			st->ax[threadIdx.x] = st->alpha[threadIdx.x];
			st->Gn[threadIdx.x] = sym_at(sres, threadIdx.x / kS, threadIdx.x % kS);
		}
		if (threadIdx.x < kS)
			st->rnorm[threadIdx.x] = sqrt(sres[kSymVals + threadIdx.x]);
		update_finish(st, L, s_beta, tolf, maxiter, delta);
	}
}

// X += P ax (the pending solution step), P = D^-1 R + P beta
__global__ void __launch_bounds__(kDirWarps * 32, 1)
k_bcgf_dir(int n, float *__restrict__ X, float *__restrict__ P, const float *__restrict__ R,
           const float *__restrict__ dinv, const BcgState *st, unsigned *err) {
	extern __shared__ __align__(128) unsigned char dyn[];
	__shared__ unsigned long long full[kDirWarps * kDirStages];
	__shared__ __align__(16) float sa[kS][kS], sb[kS][kS];
	pdl_wait();
	pdl_trigger();
	if (bcg_skip(st))
		return;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rs = lane >> 2, cq = lane & 3;
	WarpRing<kDirStages, kDirBytes> ring;
	ring.init(dyn + warp * kDirStages * kDirBytes, full + warp * kDirStages, err);
	const int ntile = (n + kWRows - 1) / kWRows, step = gridDim.x * kDirWarps;
	const int t0 = blockIdx.x * kDirWarps + warp;
	auto fetch = [&](int t) {
		const unsigned bytes = (unsigned)min(kWRows, n - t * kWRows) * kS * 4;
		unsigned char *d = ring.begin(3 * bytes);
		const size_t at = (size_t)t * kWRows * kS;
		bulk_g2s(d, P + at, bytes, ring.bar());
		bulk_g2s(d + kTileBytes, X + at, bytes, ring.bar());
		bulk_g2s(d + 2 * kTileBytes, R + at, bytes, ring.bar());
	};
	if (lane == 0)
		for (int q = 0; q < kDirStages && t0 + q * step < ntile; ++q)
			fetch(t0 + q * step);
	if (threadIdx.x < kS * kS) {
		sa[threadIdx.x / kS][threadIdx.x % kS] = (float)st->ax[threadIdx.x];
		sb[threadIdx.x / kS][threadIdx.x % kS] = (float)st->beta[threadIdx.x];
	}
	__syncthreads();
	bool alive = true;
	for (int t = t0; t < ntile; t += step) {
		float d[4];
#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const int r = t * kWRows + rs + 8 * u;
			d[u] = r < n && dinv ? __ldg(dinv + r) : 1.f;
		}
		unsigned char *stage = ring.next();
		if (!stage) {
			alive = false;
			break;
		}
		const float *s0 = reinterpret_cast<const float *>(stage);  // P, X, R
		Quad x[4], pn[4];
#pragma unroll
		for (int u = 0; u < 4; ++u) {
			x[u] = ldq(s0 + kWRows * kS + (rs + 8 * u) * kS + kQ * cq);
			const Quad rv = ldq(s0 + 2 * kWRows * kS + (rs + 8 * u) * kS + kQ * cq);
			pn[u] = {make_float2(d[u] * rv.a.x, d[u] * rv.a.y), make_float2(d[u] * rv.b.x, d[u] * rv.b.y)};
		}
#pragma unroll
		for (int i4 = 0; i4 < 4; ++i4) {
			float4 p[4];
#pragma unroll
			for (int u = 0; u < 4; ++u)
				p[u] = *reinterpret_cast<const float4 *>(s0 + (rs + 8 * u) * kS + 4 * i4);
#pragma unroll
			for (int ii = 0; ii < 4; ++ii) {
				const Quad al = ldq(&sa[4 * i4 + ii][kQ * cq]), be = ldq(&sb[4 * i4 + ii][kQ * cq]);
#pragma unroll
				for (int u = 0; u < 4; ++u) {
					const float2 v = dup(ii == 0 ? p[u].x : ii == 1 ? p[u].y : ii == 2 ? p[u].z : p[u].w);
					x[u].a = fma2(v, al.a, x[u].a);
					x[u].b = fma2(v, al.b, x[u].b);
					pn[u].a = fma2(v, be.a, pn[u].a);
					pn[u].b = fma2(v, be.b, pn[u].b);
				}
			}
		}
		ring.release();
		if (lane == 0 && t + kDirStages * step < ntile)
			fetch(t + kDirStages * step);
#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const int r = t * kWRows + rs + 8 * u;
			if (r < n) {
				stq(X + (size_t)r * kS + kQ * cq, x[u]);
				stq(P + (size_t)r * kS + kQ * cq, pn[u]);
			}
		}
	}
	if (lane == 0 && !alive)
		ring.drain();
}

// X64 += Xc + P ax, Xc = 0: the fold of the correction with the pending
// solution step; one thread a quad of a row, whose four lanes share its P
__global__ void __launch_bounds__(256)
k_bcgf_fold(int n, double *__restrict__ X, float *__restrict__ Xc, const float *__restrict__ P,
            const BcgState *st) {
	__shared__ __align__(16) float sa[kS][kS];
	sa[threadIdx.x / kS][threadIdx.x % kS] = (float)st->ax[threadIdx.x];
	__syncthreads();
	const int cq = threadIdx.x & 3;
	const bool wide = ((uintptr_t)X & 15) == 0;  // the caller's vector may be a view
	for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 2; r < n;
	     r += ((int64_t)gridDim.x * blockDim.x) >> 2) {
		const size_t at = (size_t)r * kS + kQ * cq;
		Quad x = ldq(Xc + at);
		double x64[kQ];
		if (wide)
			ld4(X + at, x64);
		else
#pragma unroll
			for (int c = 0; c < kQ; ++c)
				x64[c] = X[at + c];
		float4 p[4];
#pragma unroll
		for (int i4 = 0; i4 < 4; ++i4)
			p[i4] = __ldg(reinterpret_cast<const float4 *>(P + (size_t)r * kS) + i4);
#pragma unroll
		for (int i4 = 0; i4 < 4; ++i4) {
			const float pv[4] = {p[i4].x, p[i4].y, p[i4].z, p[i4].w};
#pragma unroll
			for (int ii = 0; ii < 4; ++ii) {
				const Quad al = ldq(&sa[4 * i4 + ii][kQ * cq]);
				x.a = fma2(dup(pv[ii]), al.a, x.a);
				x.b = fma2(dup(pv[ii]), al.b, x.b);
			}
		}
		x64[0] += (double)x.a.x;
		x64[1] += (double)x.a.y;
		x64[2] += (double)x.b.x;
		x64[3] += (double)x.b.y;
		if (wide)
			st4(X + at, x64);
		else
#pragma unroll
			for (int c = 0; c < kQ; ++c)
				X[at + c] = x64[c];
		stq(Xc + at, {{0.f, 0.f}, {0.f, 0.f}});
	}
}
__global__ void k_bcgf_clear_step(BcgState *st) { st->ax[threadIdx.x] = 0.0; }

// R = B - A X (FP64 values; X64 = 0 first for a zero guess), Rv = (V) R,
// P = Z = D^-1 Rv, G = Z^T Rv, ||B_j||, ||R_j||.  Xc, when given, is the FP32
// correction of the mixed variant and is cleared.
template<class V>
__global__ void __launch_bounds__(256)
k_bcg_start(int n, const int *__restrict__ rp, const int *__restrict__ col,
            const double *__restrict__ val, const double *__restrict__ B, double *__restrict__ X,
            V *__restrict__ Xc, V *__restrict__ R, V *__restrict__ P, const V *__restrict__ dinv,
            int zero_guess, BcgState *st, double *part, double *part2, unsigned *counter) {
	__shared__ V sr[kTile][kS], sz[kTile][kS];
	__shared__ double cb[kTile][kS], cr[kTile][kS];
	const int tr = threadIdx.x / kS, tj = threadIdx.x % kS;
	const int ntiles = (n + kTile - 1) / kTile;
	BAcc<V> g;
	double nb = 0.0, nr = 0.0;
	for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
		const int r = t * kTile + tr;
		V rv = 0, z = 0;
		if (r < n) {
			const double bv = B[(size_t)r * kS + tj];
			double ax = 0.0;
			if (zero_guess)
				X[(size_t)r * kS + tj] = 0.0;
			else
				for (int k = rp[r]; k < rp[r + 1]; ++k)
					ax = fma(val[k], X[(size_t)col[k] * kS + tj], ax);
			const double r64 = bv - ax;
			if (Xc)
				Xc[(size_t)r * kS + tj] = V(0);
			rv = (V)r64;
			R[(size_t)r * kS + tj] = rv;
			z = dinv ? dinv[r] * rv : rv;
			P[(size_t)r * kS + tj] = z;
			nb = fma(bv, bv, nb);
			nr = fma(r64, r64, nr);
		}
		sr[tr][tj] = rv;
		sz[tr][tj] = z;
		__syncthreads();
		g.add(tile_dot<V>(sz, sr, tr, tj));
		__syncthreads();
	}
	part[(size_t)blockIdx.x * 256 + threadIdx.x] = g.get();
	cb[tr][tj] = nb;
	cr[tr][tj] = nr;
	__syncthreads();
	if (threadIdx.x < kS) {
		double c1 = 0.0, c2 = 0.0;
		for (int rr = 0; rr < kTile; ++rr) {
			c1 += cb[rr][threadIdx.x];
			c2 += cr[rr][threadIdx.x];
		}
		part2[(size_t)blockIdx.x * 2 * kS + threadIdx.x] = c1;
		part2[(size_t)blockIdx.x * 2 * kS + kS + threadIdx.x] = c2;
	}
	if (last_block(counter)) {
		st->G[threadIdx.x] = fold_parts(part, gridDim.x, 256, threadIdx.x);
		if (threadIdx.x < kS) {
			const double c1 = fold_parts(part2, gridDim.x, 2 * kS, threadIdx.x);
			const double c2 = fold_parts(part2, gridDim.x, 2 * kS, kS + threadIdx.x);
			const double bn = sqrt(c1);
			st->bnorm[threadIdx.x] = bn == 0.0 ? 1.0 : bn;
			st->rnorm[threadIdx.x] = sqrt(c2);
			st->res0[threadIdx.x] = sqrt(c2);
			st->rlast[threadIdx.x] = sqrt(c2);
			st->conv_iter[threadIdx.x] = 0;
		}
		st->ax[threadIdx.x] = 0.0;
		if (threadIdx.x == 0) {
			st->iter = 0;
			st->done = 0;
			st->status = FS_STATUS_UNKNOWN;
			st->flags = 0;
			st->replacements = 0;
			*counter = 0;
		}
	}
}

// mixed: R = (float)(B - A X) with the FP64 values, ||R_j|| in FP64,
// G' = Z^T R; the last CTA decides convergence per column on the FP64
// residual, resets the replacement reference levels and forms beta
__global__ void __launch_bounds__(256)
k_bcg_true_res(int n, BcgOp<double> A, const double *__restrict__ B, const double *__restrict__ X, float *__restrict__ R, const float *__restrict__ dinv,
               BcgState *st, double *part, double *part2, unsigned *counter, double tolf,
               int maxiter) {
	__shared__ float sr[kTile][kS], sz[kTile][kS];
	__shared__ double cr[kTile][kS];
	__shared__ SmallLs L;
	__shared__ int s_beta;
	const int tr = threadIdx.x / kS, tj = threadIdx.x % kS;
	const int ntiles = (n + kTile - 1) / kTile;
	BAcc<float> g;
	double nr = 0.0;
	for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
		const int r = t * kTile + tr;
		float rv = 0.f, z = 0.f;
		if (r < n) {
			const double r64 = B[(size_t)r * kS + tj] - bcg_row1(A, X, r, tj);
			rv = (float)r64;
			R[(size_t)r * kS + tj] = rv;
			z = dinv ? dinv[r] * rv : rv;
			nr = fma(r64, r64, nr);
		}
		sr[tr][tj] = rv;
		sz[tr][tj] = z;
		__syncthreads();
		g.add(tile_dot<float>(sz, sr, tr, tj));
		__syncthreads();
	}
	part[(size_t)blockIdx.x * 256 + threadIdx.x] = g.get();
	cr[tr][tj] = nr;
	__syncthreads();
	if (threadIdx.x < kS) {
		double c = 0.0;
		for (int rr = 0; rr < kTile; ++rr)
			c += cr[rr][threadIdx.x];
		part2[(size_t)blockIdx.x * kS + threadIdx.x] = c;
	}
	if (last_block(counter)) {
		st->Gn[threadIdx.x] = fold_parts(part, gridDim.x, 256, threadIdx.x);
		if (threadIdx.x < kS) {
			const double c = fold_parts(part2, gridDim.x, kS, threadIdx.x);
			st->rnorm[threadIdx.x] = sqrt(c);
			st->rlast[threadIdx.x] = sqrt(c);
		}
		__syncthreads();
		if (threadIdx.x == 0) {
			const int it = st->iter;
			bool all = true, finite = true;
			for (int j = 0; j < kS; ++j) {
				finite = finite && isfinite(st->rnorm[j]);
				if (st->conv_iter[j] == 0 && st->rnorm[j] < tolf * st->bnorm[j])
					st->conv_iter[j] = it > 0 ? it : 1;
				all = all && st->conv_iter[j] != 0;
			}
			st->replacements += 1;
			st->flags &= ~BCG_REPLACE;
			s_beta = 0;
			if (all) {
				st->done = 1;
				st->status = FS_CONVERGED_RTOL;
			}
			else if (!finite) {
				st->done = 1;
				st->status = FS_DIVERGED_BREAKDOWN;
			}
			else if (it >= maxiter) {
				st->done = 1;
				st->status = FS_DIVERGED_ITERS;
			}
			else
				s_beta = 1;
		}
		__syncthreads();
		if (s_beta && !form_beta(st, L) && threadIdx.x == 0) {
			st->done = 1;
			st->status = FS_DIVERGED_BREAKDOWN;
		}
		if (threadIdx.x == 0)
			*counter = 0;
	}
}

struct BcgPlan {
	BcgState *st = nullptr, *hst = nullptr;
	void *work = nullptr;       // P, Q, R (and the FP32 X correction)
	double *part = nullptr;     // per-CTA partial rows (grid x kW) + norm partials
	double *gpart = nullptr;    // per-group partial rows of the two-level fold
	unsigned *counter = nullptr;  // [0] + one per fold group
	int64_t n = 0;
};
std::map<std::pair<const Csr *, bool>, BcgPlan> g_bcg;

template<class V>
int block_cg_run(Ctx *ctx, const fs_krylov_settings *s, Csr *A, bool jac, Vec *B, Vec *X,
                 fs_solve_info *infos) {
	constexpr bool mixed = std::is_same<V, float>::value;
	const int64_t n = A->nrows;
	if (jac)
		FS_TRY(ensure_dinv(A));
	if (mixed)
		FS_TRY(ensure_val32(A));
	BcgPlan &p = g_bcg[std::make_pair((const Csr *)A, mixed)];
	// every kernel on all SMs at its occupancy (resident CTAs per SM), the
	// partials folded in groups of kGroup CTAs
	const int nsteps = (int)((n + kQRows - 1) / kQRows);
	auto grid_of = [&](auto kern) {
		int nb = 0;
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 256, 0) != cudaSuccess || nb < 1)
			nb = 1;
		return std::max(1, std::min(ctx->sms * std::min(nb, 8), nsteps));
	};
	const int G = grid_of(k_bcg_start<V>);
	int Gs, Gu, Gd;  // SpMM, update, direction
	if constexpr (mixed) {
		// one CTA an SM (the stages fill its shared memory)
		const int ntile = (int)((n + kWRows - 1) / kWRows);
		auto tiles = [&](int ctas, int warps) {
			return std::max(1, std::min(ctas, (ntile + warps - 1) / warps));
		};
		Gs = tiles(ctx->sms, kSpWarps);
		Gu = tiles(ctx->sms, kUpWarps);
		Gd = tiles(ctx->sms, kDirWarps);
		FS_CUDA_TRY(ctx, cudaFuncSetAttribute(k_bcgf_spmm<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                      kSpSmem<true>));
		FS_CUDA_TRY(ctx, cudaFuncSetAttribute(k_bcgf_spmm<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                      kSpSmem<false>));
		FS_CUDA_TRY(ctx, cudaFuncSetAttribute(k_bcgf_update, cudaFuncAttributeMaxDynamicSharedMemorySize, kUpSmem));
		FS_CUDA_TRY(ctx, cudaFuncSetAttribute(k_bcgf_dir, cudaFuncAttributeMaxDynamicSharedMemorySize, kDirSmem));
	}
	else {
		Gs = grid_of(k_bcg_spmm<V>);
		Gu = grid_of(k_bcg_update<V>);
		Gd = grid_of(k_bcg_dir<V>);
	}
	const size_t m = (size_t)n * kS;
	if (p.n != n) {
		if (p.work) {
			cudaStreamSynchronize(ctx->stream);
			cudaFree(p.work);
			cudaFree(p.part);
			cudaFree(p.gpart);
			cudaFree(p.counter);
			cudaFree(p.st);
			cudaFreeHost(p.hst);
			p = BcgPlan();
		}
		FS_CUDA_TRY(ctx, cudaMalloc(&p.work, sizeof(V) * (mixed ? 4 : 3) * m));
		FS_CUDA_TRY(ctx, cudaMalloc(&p.part, sizeof(double) * (size_t)ctx->sms * 8 * kW));
		FS_CUDA_TRY(ctx, cudaMalloc(&p.gpart,
		                            sizeof(double) * (size_t)(ctx->sms * 8 / kGroup + 2) * kW));
		const size_t cbytes = sizeof(unsigned) * (size_t)(ctx->sms * 8 / kGroup + 2);
		FS_CUDA_TRY(ctx, cudaMalloc(&p.counter, cbytes));
		FS_CUDA_TRY(ctx, cudaMemset(p.counter, 0, cbytes));
		FS_CUDA_TRY(ctx, fence_setup_copies());
		FS_CUDA_TRY(ctx, cudaMalloc(&p.st, sizeof(BcgState)));
		FS_CUDA_TRY(ctx, cudaMemsetAsync(p.st, 0, sizeof(BcgState), ctx->stream));
		FS_CUDA_TRY(ctx, cudaMallocHost(&p.hst, sizeof(BcgState)));
		p.n = n;
	}
	V *Pm = (V *)p.work, *Qm = Pm + m, *R = Pm + 2 * m;
	V *Xc = mixed ? Pm + 3 * m : nullptr;
	double *part = p.part, *part2 = p.part + (size_t)ctx->sms * 8 * 256;
	const V *dinv = nullptr;
	if (jac)
		dinv = mixed ? (const V *)A->dinv32 : (const V *)A->dinv;
	const V *val = mixed ? (const V *)A->val32 : (const V *)A->val;
	// a grid stencil in symmetric storage: neighbours addressed by the grid
	// coordinates; anything else: the CSR rows
	BcgOp<V> op{A->rowptr, A->col, val, nullptr, 0, 0, 0, 0, 0};
	FS_TRY(ensure_sym(A, mixed));
	const int coding = active_coding(A, mixed);
	if (A->grid_nx > 0 && (coding == kCodingSym || coding == kCodingGrid)) {
		op.S = sym_vals<V>(A);
		op.ld = A->sym_ld;
		op.nx = A->grid_nx;
		op.ny = A->grid_ny;
		op.nz = A->grid_nz;
		op.K = A->nsym;
	}
	BcgOp<double> op64{A->rowptr, A->col, (const double *)A->val, nullptr, 0, 0, 0, 0, 0};
	if constexpr (mixed) {
		// the residual replacement's FP64 operator
		FS_TRY(ensure_sym(A, false));
		const int c64 = active_coding(A, false);
		if (A->grid_nx > 0 && (c64 == kCodingSym || c64 == kCodingGrid)) {
			op64.S = sym_vals<double>(A);
			op64.ld = A->sym_ld;
			op64.nx = A->grid_nx;
			op64.ny = A->grid_ny;
			op64.nz = A->grid_nz;
			op64.K = A->nsym;
		}
	}
	const double *b = (const double *)B->d;
	double *x = (double *)X->d;
	V *xv = mixed ? Xc : (V *)x;
	k_bcg_start<V><<<G, 256, 0, ctx->stream>>>((int)n, A->rowptr, A->col, A->val, b, x, Xc, R, Pm,
	                                           dinv, s->base.use_zero_guess ? 1 : 0, p.st, part,
	                                           part2, p.counter);
	FS_TRY(check_launch(ctx, "block cg start"));
	const double tolf = (double)s->base.rtol;
	const int maxiter = s->base.maxiter;
	const int k = s->k_readback > 0 ? s->k_readback : 16;
	const double delta = mixed ? (s->inner_rtol > 0 ? s->inner_rtol : 0.1) : 0.0;
	auto read_back = [&]() -> int {
		FS_CUDA_TRY(ctx, cudaMemcpyAsync(p.hst, p.st, sizeof(BcgState), cudaMemcpyDeviceToHost,
		                                 ctx->stream));
		return check_device_error(ctx);  // synchronises the stream
	};
	// X += the FP32 correction and its pending step, which are cleared
	auto fold = [&]() -> int {
		if constexpr (mixed) {
			k_bcgf_fold<<<grid_for(ctx, (int64_t)m, 256, 8), 256, 0, ctx->stream>>>((int)n, x, Xc, Pm, p.st);
			FS_TRY(check_launch(ctx, "block cg fold"));
			k_bcgf_clear_step<<<1, kS * kS, 0, ctx->stream>>>(p.st);
			FS_TRY(check_launch(ctx, "block cg fold"));
		}
		return FS_OK;
	};
	FS_TRY(read_back());
	while (!p.hst->done) {
		for (int j = 0; j < k; ++j) {
			if constexpr (mixed) {
				FS_TRY(check_launch_rc(
					ctx,
					op.S ? launch_pdl(ctx->stream, k_bcgf_spmm<true>, Gs, kSpWarps * 32, (size_t)kSpSmem<true>,
				                      (int)n, op, (const float *)Pm, Qm, p.st, part, p.gpart, p.counter,
				                      ctx->dev_err)
						 : launch_pdl(ctx->stream, k_bcgf_spmm<false>, Gs,
				                      kSpWarps * 32, (size_t)kSpSmem<false>, (int)n, op, (const float *)Pm,
				                      Qm, p.st, part, p.gpart, p.counter, ctx->dev_err),
					"block cg spmm"));
				FS_TRY(check_launch_rc(ctx,
				                       launch_pdl(ctx->stream, k_bcgf_update, Gu, kUpWarps * 32,
				                                  (size_t)kUpSmem, (int)n, R, (const float *)Qm, dinv, p.st,
				                                  part, p.gpart, p.counter, tolf, maxiter, delta,
				                                  ctx->dev_err),
				                       "block cg update"));
				FS_TRY(check_launch_rc(ctx,
				                       launch_pdl(ctx->stream, k_bcgf_dir, Gd, kDirWarps * 32,
				                                  (size_t)kDirSmem, (int)n, Xc, Pm, (const float *)R, dinv,
				                                  (const BcgState *)p.st, ctx->dev_err),
				                       "block cg direction"));
			}
			else {
				k_bcg_spmm<V><<<Gs, 256, 0, ctx->stream>>>((int)n, op, Pm, Qm, p.st, part, p.gpart,
				                                          p.counter);
				FS_TRY(check_launch(ctx, "block cg spmm"));
				k_bcg_update<V><<<Gu, 256, 0, ctx->stream>>>((int)n, xv, Pm, R, Qm, dinv, p.st, part,
				                                             p.gpart, p.counter, tolf, maxiter, delta);
				FS_TRY(check_launch(ctx, "block cg update"));
				k_bcg_dir<V><<<Gd, 256, 0, ctx->stream>>>((int)n, Pm, R, dinv, p.st);
				FS_TRY(check_launch(ctx, "block cg direction"));
			}
		}
		FS_TRY(read_back());
		if constexpr (mixed) {
			if (!p.hst->done && (p.hst->flags & BCG_REPLACE)) {
				FS_TRY(fold());
				k_bcg_true_res<<<G, 256, 0, ctx->stream>>>((int)n, op64, b, x, R, dinv, p.st, part, part2,
				                                           p.counter, tolf, maxiter);
				FS_TRY(check_launch(ctx, "block cg true residual"));
				k_bcgf_dir<<<Gd, kDirWarps * 32, kDirSmem, ctx->stream>>>((int)n, Xc, Pm, R, dinv, p.st,
				                                                          ctx->dev_err);
				FS_TRY(check_launch(ctx, "block cg direction"));
				FS_TRY(read_back());
			}
		}
		if (!p.hst->done && p.hst->iter >= maxiter && !(p.hst->flags & BCG_REPLACE))
			break;
	}
	if constexpr (mixed) {
		if (!(p.hst->done && p.hst->status == FS_CONVERGED_RTOL)) {
			// a stop without a final replacement (breakdown): keep the progress
			FS_TRY(fold());
			FS_TRY(read_back());
		}
	}
	const BcgState &hs = *p.hst;
	for (int j = 0; j < kS; ++j) {
		fs_solve_info &inf = infos[j];
		memset(&inf, 0, sizeof inf);
		inf.status = hs.conv_iter[j] ? FS_CONVERGED_RTOL
		                             : (hs.status == FS_DIVERGED_BREAKDOWN ? FS_DIVERGED_BREAKDOWN
		                                                                   : FS_DIVERGED_ITERS);
		inf.iters = hs.conv_iter[j];
		inf.restarts = hs.iter;  // block iterations run
		inf.res_norm_initial = (float)hs.res0[j];
		inf.res_norm_final = (float)hs.rnorm[j];
		inf.rhs_norm = (float)hs.bnorm[j];
	}
	return FS_OK;
}

int block_cg_entry(fs_ctx h, const fs_krylov_settings *s, fs_csr Ah, const fs_precond *Pc, int nrhs,
                   fs_vec bh, fs_vec xh, fs_solve_info *infos, bool mixed) {
	Ctx *ctx = reinterpret_cast<Ctx *>(h);
	Csr *A = reinterpret_cast<Csr *>(Ah);
	Vec *B = reinterpret_cast<Vec *>(bh), *X = reinterpret_cast<Vec *>(xh);
	if (!ok_ctx(ctx) || !ok_csr(A) || !ok_vec(B) || !ok_vec(X) || !s || !infos)
		return FS_ERR_BAD_HANDLE;
	FS_TRY(reject_matrix_free(A, "block_cg_entry"));
	if (nrhs != kS)
		return set_err(ctx, FS_ERR_UNSUPPORTED, "block CG: the library takes %d right-hand sides", kS);
	const int64_t n = A->nrows;
	if (A->nrows != A->ncols || B->n != n * kS || X->n != n * kS || B->dtype != FS_F64 ||
	    X->dtype != FS_F64)
		return set_err(ctx, FS_ERR_SIZE_MISMATCH, "block CG: B and X hold N x %d FP64 row-major", kS);
	if (n == 0)
		return set_err(ctx, FS_ERR_SIZE_MISMATCH, "block CG: empty operator");
	const bool jac = Pc && Pc->kind == FS_PRECOND_JACOBI;
	if (Pc && Pc->kind != FS_PRECOND_NONE && !jac)
		return set_err(ctx, FS_ERR_UNSUPPORTED, "block CG: identity or Jacobi preconditioner");
	if (s->base.maxiter < 1)
		return set_err(ctx, FS_ERR_INVALID_ARG, "block CG: maxiter must be positive");
	cudaSetDevice(ctx->device);
	return mixed ? block_cg_run<float>(ctx, s, A, jac, B, X, infos)
	             : block_cg_run<double>(ctx, s, A, jac, B, X, infos);
}

}  // namespace
}  // namespace fsg

extern "C" FS_API int fs_block_cg_solve(fs_ctx h, const fs_krylov_settings *s, fs_csr A,
                                        const fs_precond *P, int nrhs, fs_vec B, fs_vec X,
                                        fs_solve_info *infos) {
	return fsg::block_cg_entry(h, s, A, P, nrhs, B, X, infos, false);
}

extern "C" FS_API int fs_block_cg_solve_mixed(fs_ctx h, const fs_krylov_settings *s, fs_csr A,
                                              const fs_precond *P, int nrhs, fs_vec B, fs_vec X,
                                              fs_solve_info *infos) {
	return fsg::block_cg_entry(h, s, A, P, nrhs, B, X, infos, true);
}
