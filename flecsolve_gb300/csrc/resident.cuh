// Grid-resident solver kernels: a whole solve (or its iteration loop) in one
// cooperative launch.
//
// A Krylov iteration of a system whose vectors fit in the shared memories and
// the L2 is a chain of short phases separated by reductions.  As separate
// kernels each phase costs its launch, the ramp of its CTAs and a last-CTA
// fold: 20.8 us an iteration for FP64 CG on 16,384 rows, of which the
// arithmetic is under 1 us.  Here one CTA per SM owns a contiguous slice of
// the rows for the whole solve, and the CTAs meet through messages alone:
//
//  * grid_sum, a reduction: every CTA stores one 16-byte message per value,
//    {sum, epoch}, in a slot of its own and reads all slots until they carry
//    the epoch -- one store and one load through the L2, the value and its
//    flag in one access.  Every CTA forms the same sum.  Two slot sets
//    alternate: a CTA overwrites a slot two epochs later, after every CTA has
//    sent the message between, that is, has read the older one.
//  * packets, a vector's neighbour rows: each row of the vector is stored as
//    {value, epoch}, and a slice that needs a row of another one reads it
//    until it carries the epoch.  No fence and no barrier stand between the
//    writer and the reader.
//
// A reader's last look at a packet precedes the writer's next store to it
// without a fence: what it read goes into the sum that the reader then sends,
// and the writer stores again only after it has received that sum (load ->
// arithmetic -> message -> load -> store, each depending on the one before).
// A kernel whose packets did not flow into its next sum would need a fence.
//
// The launch is cooperative, so all CTAs are resident and every wait ends; as
// a guard the waits are bounded all the same (kResPolls reads), after which the
// CTA records an error in the context's device error word and leaves, as do the
// others when their own waits run out.  (The bound is a constant: as a variable
// it costs CG 4 % and the FP32 GMRES 10 %.)  The host then clears all messages
// (res_read_state): CTA 0 may not have stored its last epoch, or a CTA that
// began late may have sent some of an epoch that the next launch would use.
#pragma once

#include <algorithm>
#include <map>
#include <mutex>

#include "solver.cuh"

namespace fsg {

constexpr int kResMaxG = 160;      // CTAs of a resident grid at most
constexpr int kResMaxVals = 4;     // values per grid_sum at most
constexpr int kResThreads = 512;   // threads per CTA at most
constexpr int kResPolls = 1 << 22;  // reads of a wait at most (0.8 s in all)

// ------------------------------------------------ sums in fixed point --
//
// A warp's FP64 instruction occupies its scheduler for 63 cycles on this GPU
// whether or not it depends on the last (measured; 19 cycles an instruction
// an SM with 16 warps), so a tree of shuffles and adds over the warp, the CTA
// and the grid costs more than the messages do: 2,193 cycles of a one-CTA
// sum, of which the message was 600.  The sums therefore run in integers: every
// value is aligned to the largest exponent of its group, its magnitude cut
// into four 23-bit pieces of a 96-bit window, and the pieces are added with
// redux.sync (at most 256 values: 23 + 8 bits).  A value loses only bits
// below 2^-30 of the unit in the last place of the group's largest value, a
// warp's sum is rounded to an eighth of that unit and a CTA's to the unit, so
// the result is at least as accurate as the tree's, and it does not depend on
// the order of the values.  FP32 values lose bits below 2^-29 of the largest
// one's FP32 unit (a double's last bit).

// a group's sum q 2^(e - 1075 - F), F = 3 for a warp, 0 for a CTA; e = 0x7ff:
// some value was not finite, q the union of 1 (+inf), 2 (-inf) and 4 (NaN)
struct ResFix {
	long long q;
	int e;
};

struct ResPieces {
	int p[4];
	__device__ __forceinline__ void clear() {
#pragma unroll
		for (int i = 0; i < 4; ++i)
			p[i] = 0;
	}
	// adds m (m < 2^62; -m when neg) shifted right by d >= 0: the window is
	// m 2^34 / 2^d, its bits 73.., 50.., 27.. and 4.. the pieces
	__device__ __forceinline__ void add(unsigned long long m, int d, bool neg) {
		m <<= 2;
		unsigned w2 = (unsigned)(m >> 32), w1 = (unsigned)m, w0 = 0;
		if (d >= 32) {
			w0 = d < 64 ? w1 : d < 96 ? w2 : 0u;
			w1 = d < 64 ? w2 : 0u;
			w2 = 0;
		}
		const int r = d & 31;
		w0 = __funnelshift_r(w0, w1, r);
		w1 = __funnelshift_r(w1, w2, r);
		w2 >>= r;
		constexpr unsigned M = (1u << 23) - 1;
		const int v[4] = {(int)(w2 >> 9), (int)(__funnelshift_r(w1, w2, 18) & M),
		                  (int)(__funnelshift_r(w0, w1, 27) & M), (int)((w0 >> 4) & M)};
#pragma unroll
		for (int i = 0; i < 4; ++i)
			p[i] += neg ? -v[i] : v[i];
	}
	__device__ __forceinline__ void warp_sum() {
#pragma unroll
		for (int i = 0; i < 4; ++i)
			p[i] = __reduce_add_sync(0xffffffffu, p[i]);
	}
	// the sum as hi 2^16 + lo 2^-30 in the units of m, 0 <= lo < 2^46
	__device__ __forceinline__ void split(long long &hi, long long &lo) const {
		hi = (long long)p[0] * (1 << 23) + p[1];
		lo = (long long)p[2] * (1 << 23) + p[3];
		hi += lo >> 46;
		lo &= (1ll << 46) - 1;
	}
};

__device__ __forceinline__ ResFix res_special(int cls) {
	return {(long long)__reduce_or_sync(0xffffffffu, (unsigned)cls), 0x7ff};
}

// the sum of a warp's 32 doubles, F = 3
__device__ __forceinline__ ResFix res_fix_warp(double v) {
	const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
	int e = (int)(bits >> 52) & 0x7ff;
	unsigned long long m = bits & ((1ull << 52) - 1);
	const bool neg = bits >> 63;
	const int E = __reduce_max_sync(0xffffffffu, max(e, 1));
	if (E == 0x7ff)
		return res_special(e != 0x7ff ? 0 : m ? 4 : neg ? 2 : 1);
	if (e)
		m |= 1ull << 52;
	else
		e = 1;
	ResPieces s;
	s.clear();
	s.add(m, E - e, neg);
	s.warp_sum();
	long long hi, lo;
	s.split(hi, lo);
	return {hi * (1 << 19) + ((lo + (1ll << 26)) >> 27), E};
}

// the sum of the warps' sums (one a lane, {0, 1} in idle lanes), F = 0
__device__ __forceinline__ ResFix res_fix_cta(ResFix f) {
	const int E = __reduce_max_sync(0xffffffffu, f.e);
	if (E == 0x7ff)
		return res_special(f.e == 0x7ff ? (int)f.q : 0);
	ResPieces s;
	s.clear();
	s.add((unsigned long long)(f.q < 0 ? -f.q : f.q), E - f.e, f.q < 0);
	s.warp_sum();
	long long hi, lo;
	s.split(hi, lo);
	return {hi * (1 << 13) + ((lo + (1ll << 32)) >> 33), E};
}

// (hi 2^16 + lo 2^-30) 2^(E - 1075), rounded to nearest (0 <= lo < 2^46).  In
// integers: the conversions, the product and the sum of the FP64 form below
// it take 62 cycles each.
__device__ __forceinline__ double res_fix_double(long long hi, long long lo, int E) {
	const bool neg = hi < 0;
	const unsigned long long l = (unsigned long long)(neg ? -lo & ((1ll << 46) - 1) : lo) << 18;
	const unsigned long long h = (unsigned long long)(neg ? -hi - (lo != 0) : hi);
	const int z = __clzll((long long)h), ex = E - z + 27;
	if (h != 0 && ex > 0 && ex < 0x7fe) {
		const unsigned long long m = z ? h << z | l >> (64 - z) : h, rest = l << z;
		const unsigned r = (unsigned)m & 0x7ff;
		const unsigned long long up = r > 0x400 || (r == 0x400 && ((m & 0x800) || rest));
		return __longlong_as_double((long long)((m >> 11) + ((unsigned long long)(ex - 1) << 52) + up |
		                                        (unsigned long long)neg << 63));
	}
	const double t = fma((double)lo, 0x1p-46, (double)hi);
	const int k = E - 1059;
	if (k >= -1022)
		return t * __longlong_as_double((long long)(k + 1023) << 52);
	return t * 0x1p-600 * __longlong_as_double((long long)(k + 600 + 1023) << 52);
}

// the sum of N doubles a lane over a warp, in every lane
template<int N>
__device__ __forceinline__ double res_warp_sum(const double (&v)[N]) {
	int E = 1;
#pragma unroll
	for (int i = 0; i < N; ++i)
		E = max(E, (int)((unsigned long long)__double_as_longlong(v[i]) >> 52) & 0x7ff);
	E = __reduce_max_sync(0xffffffffu, E);
	if (E == 0x7ff) {
		// not finite: the plain sum has the right infinity or NaN
		double t = 0.0;
#pragma unroll
		for (int i = 0; i < N; ++i)
			t += v[i];
		for (int o = 16; o > 0; o >>= 1)
			t += __shfl_xor_sync(0xffffffffu, t, o);
		return t;
	}
	ResPieces s;
	s.clear();
#pragma unroll
	for (int i = 0; i < N; ++i) {
		const unsigned long long b = (unsigned long long)__double_as_longlong(v[i]);
		const int e = (int)(b >> 52) & 0x7ff;
		s.add((b & ((1ull << 52) - 1)) | (e ? 1ull << 52 : 0ull), E - max(e, 1), b >> 63);
	}
	s.warp_sum();
	long long hi, lo;
	s.split(hi, lo);
	return res_fix_double(hi, lo, E);
}

// the sum of N <= 8 floats a lane over a warp, in every lane: the 24-bit
// mantissas at the largest exponent of the warp with 31 bits below its unit,
// added in 64-bit integers and rounded once
template<int N>
__device__ __forceinline__ double res_warp_sum(const float (&v)[N]) {
	static_assert(N <= 8, "24 + 31 bits, 8 a lane, 32 lanes: below 2^63");
	int E = 1;
#pragma unroll
	for (int i = 0; i < N; ++i)
		E = max(E, (__float_as_int(v[i]) >> 23) & 0xff);
	E = __reduce_max_sync(0xffffffffu, E);
	if (E == 0xff) {
		double t = 0.0;
#pragma unroll
		for (int i = 0; i < N; ++i)
			t += (double)v[i];
		for (int o = 16; o > 0; o >>= 1)
			t += __shfl_xor_sync(0xffffffffu, t, o);
		return t;
	}
	long long q = 0;
#pragma unroll
	for (int i = 0; i < N; ++i) {
		const int b = __float_as_int(v[i]), e = (b >> 23) & 0xff;
		const int m = (b & 0x7fffff) | (e ? 0x800000 : 0);
		const int d = min(E - max(e, 1), 63);
		q += ((long long)(b < 0 ? -m : m) << 31) >> d;
	}
	constexpr long long M = (1ll << 26) - 1;
	const long long p0 = __reduce_add_sync(0xffffffffu, (int)(q & M));
	const long long p1 = __reduce_add_sync(0xffffffffu, (int)(q >> 26 & M));
	const long long p2 = __reduce_add_sync(0xffffffffu, (int)(q >> 52));
	return (double)(p2 * (1ll << 52) + p1 * (1ll << 26) + p0) *
	       __longlong_as_double((long long)(E - 181 + 1023) << 52);
}

// the sum of the CTAs' sums, Q a lane, as a double (the same in every lane)
template<int Q, int F = 0>
__device__ __forceinline__ double res_fix_grid(const ResFix (&f)[Q]) {
	int E = 1;
#pragma unroll
	for (int i = 0; i < Q; ++i)
		E = max(E, f[i].e);
	E = __reduce_max_sync(0xffffffffu, E);
	if (E == 0x7ff) {
		int cls = 0;
#pragma unroll
		for (int i = 0; i < Q; ++i)
			cls |= f[i].e == 0x7ff ? (int)f[i].q : 0;
		const long long q = res_special(cls).q;
		const double inf = __longlong_as_double(0x7ff0000000000000ll);
		return (q & 4) || (q & 3) == 3 ? __longlong_as_double(0x7ff8000000000000ll)
		                               : (q & 1) ? inf : -inf;
	}
	ResPieces s;
	s.clear();
#pragma unroll
	for (int i = 0; i < Q; ++i)
		s.add((unsigned long long)(f[i].q < 0 ? -f[i].q : f[i].q), E - f[i].e, f[i].q < 0);
	s.warp_sum();
	long long hi, lo;
	s.split(hi, lo);
	return res_fix_double(hi, lo, E - F);
}

// a sum's value, F = 0
__device__ __forceinline__ double res_fix_value(ResFix f) {
	if (f.e == 0x7ff) {
		const double inf = __longlong_as_double(0x7ff0000000000000ll);
		return (f.q & 4) || (f.q & 3) == 3 ? __longlong_as_double(0x7ff8000000000000ll)
		                                   : (f.q & 1) ? inf : -inf;
	}
	// q = hi 2^16 + lo 2^-30
	return res_fix_double(f.q >> 16, (f.q & 0xffff) << 30, f.e);
}

// the sum of N <= 8 floats a lane over a warp, F = 3 (29 bits below the unit of
// the largest: 24 + 29 + 8 bits, below 2^62)
template<int N>
__device__ __forceinline__ ResFix res_fix_warp(const float (&v)[N]) {
	static_assert(N <= 8, "");
	int E = 1;
#pragma unroll
	for (int i = 0; i < N; ++i)
		E = max(E, (__float_as_int(v[i]) >> 23) & 0xff);
	E = __reduce_max_sync(0xffffffffu, E);
	if (E == 0xff) {
		int cls = 0;
#pragma unroll
		for (int i = 0; i < N; ++i)
			cls |= isnan(v[i]) ? 4 : isinf(v[i]) ? (v[i] < 0.f ? 2 : 1) : 0;
		return res_special(cls);
	}
	long long q = 0;
#pragma unroll
	for (int i = 0; i < N; ++i) {
		const int b = __float_as_int(v[i]), e = (b >> 23) & 0xff;
		const int m = (b & 0x7fffff) | (e ? 0x800000 : 0);
		const int d = min(E - max(e, 1), 63);
		q += ((long long)(b < 0 ? -m : m) << 29) >> d;
	}
	constexpr long long M = (1ll << 26) - 1;
	const long long p0 = __reduce_add_sync(0xffffffffu, (int)(q & M));
	const long long p1 = __reduce_add_sync(0xffffffffu, (int)(q >> 26 & M));
	const long long p2 = __reduce_add_sync(0xffffffffu, (int)(q >> 52));
	// q 2^(E - 179) = q 2^(e - 1075 - 3)
	return {p2 * (1ll << 52) + p1 * (1ll << 26) + p0, E + 899};
}

// ------------------------------------------------------------ messages --

// device memory of the messages: two sets of kResMaxVals x kResMaxG slots
// {sum, epoch << 16 | exponent}, then the epoch reached by the last launch
struct ResSlots {
	ulonglong2 msg[2][kResMaxVals][kResMaxG];
	unsigned long long epoch;
};

struct ResShared {
	ResFix part[kResMaxVals][kResThreads / 32];
	double bc[8];  // scalars handed from warp 0 to the CTA
	int stop;      // set by warp 0: leave the iteration loop
	int fail;      // a wait ran out
};

__device__ __forceinline__ void res_st16(ulonglong2 *p, unsigned long long a, unsigned long long b) {
	asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
	             "l"(a), "l"(b)
	             : "memory");
}
// the same store as an exchange at the L2: a plain store to a line that other
// SMs are already polling costs them 2,000 to 4,000 cycles (152 CTAs that
// arrive 400 to 1,300 cycles apart: 5,760 cycles a round with st, 3,074 with
// the exchange, 2,419 with the first read held back as well)
__device__ __forceinline__ void res_xchg16(ulonglong2 *p, unsigned long long a, unsigned long long b) {
	asm volatile("{\n .reg .b128 t, u;\n mov.b128 t, {%1, %2};\n"
	             " atom.relaxed.gpu.global.exch.b128 u, [%0], t;\n}\n" ::"l"(p),
	             "l"(a), "l"(b)
	             : "memory");
}
// cycles from a CTA's own message to its first look at the others': about
// what a message takes
constexpr int kResFirstLook = 450;
__device__ __forceinline__ void res_hold(long long since) {
	while (clock64() - since < kResFirstLook) {
	}
}
__device__ __forceinline__ ulonglong2 res_ld16(const ulonglong2 *p) {
	ulonglong2 v;
	asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
	             : "=l"(v.x), "=l"(v.y)
	             : "l"(p)
	             : "memory");
	return v;
}

// A CTA's view of the resident grid
struct ResTeam {
	ResSlots *slots;
	ResShared *sh;
	unsigned *err;
	unsigned long long epoch;  // the same in every thread of the grid

	__device__ void init(ResSlots *s, ResShared *shared, unsigned *e) {
		slots = s;
		sh = shared;
		err = e;
		epoch = *(volatile unsigned long long *)&s->epoch;
		if (threadIdx.x == 0) {
			sh->stop = 0;
			sh->fail = 0;
		}
	}
	__device__ void failed() {
		atomicOr(err, 0x40u);
		*(volatile int *)&sh->fail = 1;
	}

	// One warp: the grid's messages of this epoch, one slot a CTA ({0, 1} past
	// the grid); false in every lane when one did not arrive
	__device__ bool gather(const ulonglong2 *set, ResFix (&f)[kResMaxG / 32]) {
		constexpr int Q = kResMaxG / 32;
		const int lane = threadIdx.x & 31, G = (int)gridDim.x;
		bool here = false;
		for (int it = 0; !here && it < kResPolls; ++it) {
			// every slot of this lane in flight, then the tags
			ulonglong2 m[Q];
#pragma unroll
			for (int q = 0; q < Q; ++q)
				if (q * 32 < G)
					m[q] = res_ld16(&set[min(q * 32 + lane, G - 1)]);
			here = true;
#pragma unroll
			for (int q = 0; q < Q; ++q)
				if (q * 32 < G) {
					here = here && m[q].y >> 16 == epoch;
					f[q] = {(long long)m[q].x, (int)(m[q].y & 0xffff)};
				}
		}
#pragma unroll
		for (int q = 0; q < Q; ++q)
			if (q * 32 + lane >= G)
				f[q] = {0, 1};
		return __all_sync(0xffffffffu, here);
	}

	// Sums NV values over the grid.  Every thread calls it; warp k carries
	// value k through the messages (in parallel: two values take a third
	// longer than one) and has its total in every lane of the returned
	// value.  Thread 32 k then forms the scalars that follow from it, and
	// every thread ends the step with done().  PUB: what the CTAs wrote to
	// global memory before the call is visible to all after done().
	template<int NV, bool PUB>
	__device__ double grid_sum(const double (&v)[NV]) {
		const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
		++epoch;
#pragma unroll
		for (int k = 0; k < NV; ++k) {
			const ResFix f = res_fix_warp(v[k]);
			if (lane == 0)
				sh->part[k][wid] = f;
		}
		__syncthreads();
		if (wid >= NV)
			return 0.0;
		const int nw = (int)blockDim.x >> 5;
		ulonglong2 *set = slots->msg[epoch & 1][wid];
		if (PUB)
			__threadfence();
		ResFix own{0, 1};
		if (lane < nw)
			own = sh->part[wid][lane];
		own = res_fix_cta(own);
		if (lane == 0)
			res_xchg16(&set[blockIdx.x], (unsigned long long)own.q,
			           epoch << 16 | (unsigned long long)own.e);
		res_hold(clock64());
		ResFix f[kResMaxG / 32];
		if (!gather(set, f) && lane == 0)
			failed();
		const double t = res_fix_grid<kResMaxG / 32>(f);
		if (PUB)
			__threadfence();
		return t;
	}
	// ends the step; false when a wait ran out (the same in every thread)
	__device__ bool done() {
		__syncthreads();
		return *(volatile int *)&sh->fail == 0;
	}
	// the last call of a kernel: the next launch goes on from this epoch
	// (past every message and packet of this one, also after a failed wait)
	__device__ void finish() {
		if (blockIdx.x == 0 && threadIdx.x == 0)
			slots->epoch = epoch + 16;
	}
};

// the largest s with sqrt(s) < tol (below 0 when there is none): the stopping
// test on a norm without its square root
__device__ __forceinline__ double res_threshold(double tol) {
	if (!(tol > 0.0))
		return -1.0;
	if (isinf(tol))
		return 1.7976931348623157e308;
	double t = fmin(tol * tol, 1.7976931348623157e308);
	for (int i = 0; i < 8 && t > 0.0 && !(sqrt(t) < tol); ++i)
		t = __longlong_as_double(__double_as_longlong(t) - 1);
	for (int i = 0; i < 8; ++i) {
		const double u = __longlong_as_double(__double_as_longlong(t) + 1);
		if (!(sqrt(u) < tol))
			break;
		t = u;
	}
	return t;
}

__device__ __forceinline__ int res_exponent(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }
__device__ __forceinline__ bool res_finite(double v) { return res_exponent(v) != 0x7ff; }
// s <= t for a sum of squares s that is finite (a comparison is an FP64
// operation; non-negative doubles compare as integers, and a negative t is
// below all of them)
__device__ __forceinline__ bool res_below(double s, double t) {
	return __double_as_longlong(s) <= __double_as_longlong(t);
}

// a / b, correctly rounded, from y = 1 / b correctly rounded (Markstein 1990:
// the residual of a y corrects it); three dependent operations after a is
// known where a division takes 561 cycles.  Outside the range where the
// residual is exact it divides.
__device__ __forceinline__ double res_quotient(double a, double b, double y) {
	const double q = a * y;
	const double r = fma(fma(-q, b, a), y, q);
	const bool safe = (unsigned)(res_exponent(a) - 123) < 1800u && (unsigned)(res_exponent(b) - 123) < 1800u &&
	                  (unsigned)(res_exponent(q) - 123) < 1800u;
	return safe ? r : a / b;
}

// a / b to half a unit in the last place and 2^-36 of one: b's reciprocal from
// the FP32 one of its leading bits (1.5 x 2^-23) and one Newton step (2^-44.8),
// the quotient's residual as above.  Five dependent FP64 operations on the path of a sum that
// everything waits for; the division takes ten.
__device__ __forceinline__ double res_divide(double a, double b) {
	const int ea = res_exponent(a), eb = res_exponent(b), hi = __double2hiint(b);
	if ((unsigned)(ea - 523) >= 1000u || (unsigned)(eb - 523) >= 1000u)
		return a / b;
	const float m = __int_as_float(0x3f800000 | (int)((unsigned)hi << 3 & 0x7fffff) |
	                               (int)((unsigned)__double2loint(b) >> 29));
	const unsigned f = __float_as_uint(__frcp_rn(m));  // 2^-1 .. 1
	const unsigned e = (f >> 23) + (unsigned)(1919 - eb);  // biased; 1 / 2^(eb - 1023)
	const double y0 = __hiloint2double((int)(((unsigned)hi & 0x80000000u) | e << 20 | (f >> 3 & 0xfffffu)),
	                                   (int)(f << 29));
	const double y = fma(fma(-b, y0, 1.0), y0, y0);
	const double q = a * y;
	return fma(fma(-q, b, a), y, q);
}

// a / b rounded to FP32, to half a unit and 2^-40 of the value: the quotient of
// the leading parts, corrected by the residual of both parts (Dekker 1971, "A
// floating-point technique for extending the available precision"), in FP32 on
// the mantissas; 20 short operations where the FP64 division holds the one warp
// that everything waits for 561 cycles
__device__ __forceinline__ float res_quotient32(double a, double b) {
	const long long ua = __double_as_longlong(a), ub = __double_as_longlong(b);
	const int ea = (int)(ua >> 52) & 0x7ff, eb = (int)(ub >> 52) & 0x7ff, e = ea - eb;
	if (ea == 0 || eb == 0 || ea == 0x7ff || eb == 0x7ff || e < -120 || e > 120)
		return (float)(a / b);
	const float ah = __int_as_float(0x3f800000 | ((int)(ua >> 29) & 0x7fffff));
	const float bh = __int_as_float(0x3f800000 | ((int)(ub >> 29) & 0x7fffff));
	const float al = (float)((int)ua & 0x1fffffff) * 0x1p-52f, bl = (float)((int)ub & 0x1fffffff) * 0x1p-52f;
	const float y = __frcp_rn(bh), q = ah * y;
	const float r = fmaf(-q, bh, ah) + fmaf(-q, bl, al);
	const float v = fmaf(r, y, q) * __int_as_float((e + 127) << 23);
	return (ua ^ ub) < 0 ? -v : v;
}

// (double)v of a normal number or zero in integer operations: the conversion
// takes the FP64 pipe as long as an FMA does
__device__ __forceinline__ double widen(float v) {
	const unsigned b = __float_as_uint(v), a = b & 0x7fffffffu;
	return __hiloint2double((int)((a ? (a >> 3) + 0x38000000u : 0u) | (b & 0x80000000u)), (int)(a << 29));
}
__device__ __forceinline__ bool widens(float v) {
	const unsigned a = __float_as_uint(v) & 0x7fffffffu;
	return a - 1u >= 0x7fffffu && a < 0x7f800000u;  // not subnormal, finite
}
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ bool widens(double) { return true; }

// the payload of a packet that had not arrived at the first look (its own
// function: inlined, the loops of a row's neighbours cost the caller spills)
static __device__ __noinline__ unsigned long long res_await(const ulonglong2 *p, unsigned long long tag,
                                                     ResShared *sh, unsigned *err) {
	for (int it = 0; it < kResPolls && !*(volatile int *)&sh->fail; ++it) {
		const ulonglong2 m = res_ld16(p);
		if (m.y == tag)
			return m.x;
	}
	atomicOr(err, 0x40u);
	*(volatile int *)&sh->fail = 1;
	return 0;
}

// a vector entry's packet payload
__device__ __forceinline__ unsigned long long res_pack(double v) {
	return (unsigned long long)__double_as_longlong(v);
}
__device__ __forceinline__ unsigned long long res_pack(float v) { return __float_as_uint(v); }
template<class V>
__device__ __forceinline__ V res_unpack(unsigned long long b) {
	if constexpr (sizeof(V) == 8)
		return __longlong_as_double((long long)b);
	else
		return __uint_as_float((unsigned)b);
}

// Grid-stencil operator of a resident kernel: the symmetric or the general
// grid storage (rows addressed by grid coordinates), K = 1..3 dimensions.
template<class V>
struct ResGrid {
	const V *S;
	int64_t ld;
	int n, nx, ny, nz;
};

// per row, the neighbours inside the grid: bits z-, y-, x-, x+, y+, z+
template<int K>
__device__ __forceinline__ unsigned res_mask(int r, int nx, int ny, int nz) {
	const int line = r / nx, i = r - line * nx;
	const int kk = K >= 3 ? line / ny : 0, j = K >= 2 ? line - kk * ny : 0;
	unsigned m = 0;
	if (K >= 3 && kk > 0)
		m |= 1u;
	if (K >= 2 && j > 0)
		m |= 2u;
	if (i > 0)
		m |= 4u;
	if (i < nx - 1)
		m |= 8u;
	if (K >= 2 && j < ny - 1)
		m |= 16u;
	if (K >= 3 && kk < nz - 1)
		m |= 32u;
	return m;
}

// A slice's operator: the diagonals of the own rows (in shared memory when
// they fit, else global), the global ones for lower partners outside it
template<class V, int K, bool GEN>
struct ResRows {
	const V *D, *U[3], *L[3];  // own rows, indexed from the slice's first row
	const V *G;                // symmetric storage: upper diagonals of all rows
	int64_t ld;
	int lo, cnt, d[3];         // offsets 1, nx, nx ny
	const unsigned char *mask;

	// sum of the own row l over a vector whose own rows are vl (indexed from
	// the slice's first row); rows of other slices come from packets `pk`
	// carrying `tag` (PKT) or from the global vector vg.  The packets of the
	// two outermost neighbours, which most rows of a 2-D or 3-D slice need, are
	// in flight while the others are read; an inner neighbour is outside the
	// slice only near its ends and is awaited where it is added.
	template<bool PKT>
	__device__ __forceinline__ V sum(int l, const V *vl, const V *vg, const ulonglong2 *pk,
	                                 unsigned long long tag, ResTeam &tm) const {
		const unsigned m = mask[l];
		constexpr int O = K - 1;  // outermost dimension
		const bool has_lo = m >> (2 - O) & 1, has_hi = m >> (3 + O) & 1;
		// an absent neighbour reads the own row and its term is not added
		const int jl = has_lo ? l - d[O] : l, jh = has_hi ? l + d[O] : l;
		const bool in_lo = jl >= 0, in_hi = jh < cnt;
		ulonglong2 wl, wh;
		V xl, xh;
		if constexpr (PKT) {
			if (!in_lo)
				wl = res_ld16(pk + (lo + jl));
			if (!in_hi)
				wh = res_ld16(pk + (lo + jh));
		}
		else {
			xl = *(in_lo ? vl + jl : vg + (lo + jl));
			xh = *(in_hi ? vl + jh : vg + (lo + jh));
		}
		auto lower = [&](int e, int j) -> V {  // a(l, l - d[e]), j = l - d[e]
			if constexpr (GEN)
				return L[e][l];
			else
				return *(j >= 0 ? U[e] + j : G + ((int64_t)e * ld + lo + j));
		};
		V x[2 * K + 1], c[2 * K + 1];  // inner neighbours and all coefficients
		c[0] = lower(O, jl);
		c[2 * K] = U[O][l];
#pragma unroll
		for (int t = 1; t < 2 * K; ++t) {
			// t < K: lower neighbour of d[K - 1 - t]; t > K: upper of d[t - K - 1]
			const int e = t < K ? K - 1 - t : t - K - 1;
			const bool has = t == K || (t < K ? m >> (2 - e) & 1 : m >> (3 + e) & 1);
			const int j = t == K || !has ? l : t < K ? l - d[e] : l + d[e];
			const bool in = t == K || (t < K ? j >= 0 : j < cnt);
			if constexpr (PKT) {
				if (in)
					x[t] = vl[j];
				else
					x[t] = res_unpack<V>(res_await(pk + (lo + j), tag, tm.sh, tm.err));
			}
			else
				x[t] = *(in ? vl + j : vg + (lo + j));
			c[t] = t == K ? D[l] : t < K ? lower(e, j) : U[e][l];
		}
		if constexpr (PKT) {
			if (in_lo)
				xl = vl[jl];
			else
				xl = res_unpack<V>(wl.y == tag ? wl.x : res_await(pk + (lo + jl), tag, tm.sh, tm.err));
			if (in_hi)
				xh = vl[jh];
			else
				xh = res_unpack<V>(wh.y == tag ? wh.x : res_await(pk + (lo + jh), tag, tm.sh, tm.err));
		}
		V s = V(0);
		s = has_lo ? fma(c[0], xl, s) : s;
#pragma unroll
		for (int t = 1; t < K; ++t)
			s = (m >> (2 - (K - 1 - t)) & 1) ? fma(c[t], x[t], s) : s;
		s = fma(c[K], x[K], s);
#pragma unroll
		for (int t = K + 1; t < 2 * K; ++t)
			s = (m >> (3 + t - K - 1) & 1) ? fma(c[t], x[t], s) : s;
		s = has_hi ? fma(c[2 * K], xh, s) : s;
		return s;
	}
};

// Hands out the CTA's dynamic shared memory to the slice's arrays in order of
// use until it is full; an array that does not fit stays where it is.
struct ResSmem {
	unsigned char *at;
	int left;
	template<class T>
	__device__ T *take(int count) {
		const int bytes = (count * (int)sizeof(T) + 15) & ~15;
		if (bytes > left)
			return nullptr;
		T *p = reinterpret_cast<T *>(at);
		at += bytes;
		left -= bytes;
		return p;
	}
};

// own rows l = tid, tid + nt, ...: U at a time while there are U, all of
// load(l) before any store(l, value), then one by one
template<int U, class L, class S>
__device__ __forceinline__ void res_rows(int cnt, L &&load, S &&store) {
	using T = decltype(load(0));
	const int nt = (int)blockDim.x;
	int l = (int)threadIdx.x;
	if constexpr (U > 1)
		for (; l + (U - 1) * nt < cnt; l += U * nt) {
			T t[U];
#pragma unroll
			for (int u = 0; u < U; ++u)
				t[u] = load(l + u * nt);
#pragma unroll
			for (int u = 0; u < U; ++u)
				store(l + u * nt, t[u]);
		}
	for (; l < cnt; l += nt) {
		const T t = load(l);
		store(l, t);
	}
}

// ---------------------------------------------------------------- host --

struct ResShape {
	int grid, threads, rows, smem;
};

// One CTA per SM, at least kMinRows rows each (us an iteration of CG at 32^2,
// BiCGSTAB at 16^3 and GMRES at 48^2 with 64 / 128 / 256 / 512 rows: 6.7 / 6.4
// / 6.7 / 7.7, 12.5 / 12.5 / 12.9 / 15.4, 13.5 / 13.5 / 13.1 / 19.6); a thread per row up to
// kResThreads, four warps at least (one per value of a grid_sum); `per_row`
// bytes of shared memory a row, as far as they go.
inline ResShape res_shape(Ctx *ctx, int64_t n, int per_row, int smem_max) {
	constexpr int kMinRows = 128;
	const int64_t cap = std::min(ctx->sms, kResMaxG);
	int64_t g = std::max<int64_t>(1, std::min(cap, (n + kMinRows - 1) / kMinRows));
	int64_t rows = ((n + g - 1) / g + 31) / 32 * 32;
	g = (n + rows - 1) / rows;
	ResShape s;
	s.grid = (int)g;
	s.rows = (int)rows;
	s.threads = (int)std::min<int64_t>(kResThreads, std::max<int64_t>(128, rows));
	// (count * 8 + 15) & ~15 per array: rows is a multiple of 32
	s.smem = (int)std::min<int64_t>(smem_max, rows * per_row);
	return s;
}

// `taken` = 0: the device has no room for every CTA at once (SMs set aside for
// another client), and the caller's phase kernels run instead
template<class Args>
inline int res_launch(Ctx *ctx, void (*kern)(Args), const ResShape &sh, const Args &a, const char *what,
                      int *taken) {
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = dim3((unsigned)sh.grid);
	cfg.blockDim = dim3((unsigned)sh.threads);
	cfg.dynamicSmemBytes = (size_t)sh.smem;
	cfg.stream = ctx->stream;
	cudaLaunchAttribute at[1];
	at[0].id = cudaLaunchAttributeCooperative;
	at[0].val.cooperative = 1;
	cfg.attrs = at;
	cfg.numAttrs = 1;
	const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
	*taken = e != cudaErrorCooperativeLaunchTooLarge;
	if (!*taken) {
		cudaGetLastError();
		return FS_OK;
	}
	return check_launch_rc(ctx, e, what);
}

// dynamic shared memory a resident kernel may use (its static part is taken
// off), set on the kernel once per device; 0 when the device refuses it
template<class Args>
inline int res_smem_max(Ctx *ctx, void (*kern)(Args)) {
	static std::map<std::pair<int, const void *>, int> known;
	static std::mutex mu;
	std::lock_guard<std::mutex> lock(mu);
	const auto key = std::make_pair(ctx->device, (const void *)kern);
	const auto it = known.find(key);
	if (it != known.end())
		return it->second;
	int optin = 0;
	cudaFuncAttributes fa;
	if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) !=
	        cudaSuccess ||
	    cudaFuncGetAttributes(&fa, kern) != cudaSuccess)
		return 0;
	int bytes = std::max(0, (optin - (int)fa.sharedSizeBytes) / 1024 * 1024);
	if (bytes > 0 &&
	    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
		cudaGetLastError();
		bytes = 0;
	}
	known.emplace(key, bytes);
	return bytes;
}

// The operator as a grid stencil in the storage that the SpMV on values of V
// would use; false when it is none
template<class V>
inline bool res_grid(const Csr *A, ResGrid<V> &g, bool &gen) {
	constexpr bool f32 = sizeof(V) == 4;
	if (stores_no_rows(A) || A->view || A->grid_nx <= 0 || A->coding != kCodingGrid ||
	    A->nsym < 1 || A->nsym > 3)
		return false;
	if (f32 ? A->sym32_valid : A->sym64_valid)
		gen = false;
	else if (f32 ? A->gen32_valid : A->gen64_valid)
		gen = true;
	else
		return false;
	if constexpr (f32)
		g.S = gen ? A->gen32 : A->sym32;
	else
		g.S = gen ? A->gen64 : A->sym64;
	g.ld = A->sym_ld;
	g.n = (int)A->nrows;
	g.nx = A->grid_nx;
	g.ny = A->grid_ny;
	g.nz = A->grid_nz;
	return true;
}

// the solver's messages (and row packets), allocated on first use
// (resident.cu); false when there is no memory for them: the caller's phase
// kernels, which need neither, run instead
bool res_memory(Solver *s, bool packets);

// read_state after a resident kernel (resident.cu); clears all messages when a
// wait ran out, so that the solver can be used again
int res_read_state(Solver *s);

}  // namespace fsg
