// The scalar arithmetic of the resident kernels (csrc/resident.cuh) on arrays
// of operands, for tests/test_gpu_resident_math.py: quotients, the threshold of
// the stopping tests and the sums in fixed point.  Every function takes host
// arrays and returns 0 or a CUDA error code.
#include <vector>

#include "resident.cuh"

namespace {

using namespace fsg;

#define API extern "C" __attribute__((visibility("default")))

template<class T>
struct Dev {
	T *p = nullptr;
	size_t n;
	explicit Dev(size_t n_, const T *src = nullptr) : n(n_) {
		if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess)
			p = nullptr;
		else if (src)
			cudaMemcpy(p, src, n * sizeof(T), cudaMemcpyHostToDevice);
	}
	~Dev() { cudaFree(p); }
	int get(T *dst) {
		const cudaError_t e = cudaMemcpy(dst, p, n * sizeof(T), cudaMemcpyDeviceToHost);
		return e == cudaSuccess ? (int)cudaGetLastError() : (int)e;
	}
};

__global__ void k_binary(int op, int n, const double *a, const double *b, double *o) {
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		const double x = a[i], y = b[i];
		o[i] = op == 0   ? res_divide(x, y)
		       : op == 1 ? res_quotient(x, y, 1.0 / y)
		       : op == 2 ? (double)res_quotient32(x, y)
		       : op == 3 ? res_threshold(x)
		       : op == 4 ? (widens((float)x) ? widen((float)x) : (double)(float)x)
		                 : 0.0;
	}
}

__global__ void k_fix_double(int n, const long long *hi, const long long *lo, const int *E, double *o) {
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		o[i] = res_fix_double(hi[i], lo[i], E[i]);
}

// a warp's sum of N values a lane, by block
template<class T, int N>
__global__ void k_warp_sum(const T *v, double *o) {
	T x[N];
	for (int i = 0; i < N; ++i)
		x[i] = v[((size_t)blockIdx.x * 32 + threadIdx.x) * N + i];
	const double t = res_warp_sum<N>(x);
	if (threadIdx.x == 0)
		o[blockIdx.x] = t;
}

// the sum of 512 values a CTA: the warps' parts, then the CTA's
template<class T>
__global__ void k_cta_sum(const T *v, ResFix *o) {
	__shared__ ResFix part[16];
	ResFix f;
	if constexpr (sizeof(T) == 8)
		f = res_fix_warp(v[blockIdx.x * 512 + threadIdx.x]);
	else {
		const T one[1] = {v[blockIdx.x * 512 + threadIdx.x]};
		f = res_fix_warp(one);
	}
	if (threadIdx.x % 32 == 0)
		part[threadIdx.x / 32] = f;
	__syncthreads();
	if (threadIdx.x < 32) {
		const ResFix t = res_fix_cta(threadIdx.x < 16 ? part[threadIdx.x] : ResFix{0, 1});
		if (threadIdx.x == 0)
			o[blockIdx.x] = t;
	}
}
// groups of G <= 160 CTAs' sums, a block each; the value of the first as well
__global__ void k_grid_sum(int G, const ResFix *f, double *o, double *one) {
	ResFix q[kResMaxG / 32];
	for (int i = 0; i < kResMaxG / 32; ++i)
		q[i] = i * 32 + (int)threadIdx.x < G ? f[blockIdx.x * G + i * 32 + threadIdx.x] : ResFix{0, 1};
	const double t = res_fix_grid<kResMaxG / 32>(q);
	if (threadIdx.x == 0) {
		o[blockIdx.x] = t;
		one[blockIdx.x] = res_fix_value(f[blockIdx.x * G]);
	}
}

template<class T>
int cta_grid(int groups, int G, const T *v, double *sum, double *one) {
	Dev<T> d((size_t)groups * G * 512, v);
	Dev<ResFix> f((size_t)groups * G);
	Dev<double> o(groups), p(groups);
	if (!d.p || !f.p || !o.p || !p.p || G > kResMaxG)
		return -1;
	k_cta_sum<T><<<groups * G, 512>>>(d.p, f.p);
	k_grid_sum<<<groups, 32>>>(G, f.p, o.p, p.p);
	const int e = o.get(sum);
	return e ? e : p.get(one);
}

}  // namespace

API int rm_binary(int op, int n, const double *a, const double *b, double *out) {
	Dev<double> da(n, a), db(n, b), o(n);
	if (!da.p || !db.p || !o.p)
		return -1;
	k_binary<<<256, 256>>>(op, n, da.p, db.p, o.p);
	return o.get(out);
}

API int rm_fix_double(int n, const long long *hi, const long long *lo, const int *E, double *out) {
	Dev<long long> h(n, hi), l(n, lo);
	Dev<int> e(n, E);
	Dev<double> o(n);
	if (!h.p || !l.p || !e.p || !o.p)
		return -1;
	k_fix_double<<<256, 256>>>(n, h.p, l.p, e.p, o.p);
	return o.get(out);
}

// groups of 32 x 4 doubles or 32 x 8 floats
API int rm_warp_sum64(int groups, const double *v, double *out) {
	Dev<double> d((size_t)groups * 128, v), o(groups);
	if (!d.p || !o.p)
		return -1;
	k_warp_sum<double, 4><<<groups, 32>>>(d.p, o.p);
	return o.get(out);
}
API int rm_warp_sum32(int groups, const float *v, double *out) {
	Dev<float> d((size_t)groups * 256, v);
	Dev<double> o(groups);
	if (!d.p || !o.p)
		return -1;
	k_warp_sum<float, 8><<<groups, 32>>>(d.p, o.p);
	return o.get(out);
}
// groups of G x 512 values; `one`: the first CTA's sum of each group alone
API int rm_grid_sum64(int groups, int G, const double *v, double *sum, double *one) {
	return cta_grid(groups, G, v, sum, one);
}
API int rm_grid_sum32(int groups, int G, const float *v, double *sum, double *one) {
	return cta_grid(groups, G, v, sum, one);
}
