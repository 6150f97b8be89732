// Hermitian eigen-decomposition of the k x k overlap matrix on the GPU.
//
// Replaces EigenSolver::solve (ZHEEV, eigensolver.hpp:80-84) and the checks
// and scaling of StateSet::orthonormalize (stateset.cpp:155-176): the block
// Jacobi iteration of bjacobi.cu (FP64, every k; up to 4 in one warp) or
// bjacobi32.cu (FP32 states of kBlockJacobi32MinK and more), then the steps of this file: unit columns,
// the ascending sort with the reference's checks, and W = V l^{-1/2}.
//
// FP64 block Jacobi serves small k too: a sweep of k = 200 takes 13 grid-wide
// rounds of 16 x 16 rotations in shared memory, where one grid-wide round per
// k/2 rotations (scalar cyclic Jacobi, 199 rounds of 8.8 us each) took 17.5 ms
// per eigensolve.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>

#include "contract.cuh"
#include "launch.cuh"
#include "../../include/itp2d_gpu.h"

namespace itp2d {

namespace {

// Copy S (k x k) into the padded kp x kp work matrix; V = I.
__global__ void jacobi_init_kernel(const double2* __restrict__ S, int k, int kp, double2* A, double2* V) {
	const long long n = (long long)kp * kp;
	for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
			idx += (long long)gridDim.x * blockDim.x) {
		const int i = (int)(idx / kp), j = (int)(idx % kp);
		A[idx] = (i < k && j < k) ? S[(long long)i * k + j] : make_double2(0.0, 0.0);
		V[idx] = make_double2(i == j ? 1.0 : 0.0, 0.0);
	}
}

// Normalises the first k columns of V in place (removes the norm drift that
// the accumulated rotations leave). 32 columns per CTA, 8 row groups.
// Columns j of V scaled to unit norm: 32 columns per CTA, 32 row groups; the
// row loops are unrolled by 4 so that several loads are in flight per thread.
__global__ void __launch_bounds__(1024) normalize_columns_kernel(double2* V, int k, int kp) {
	__shared__ double part[32][33];
	const int cl = threadIdx.x & 31, rg = threadIdx.x >> 5;
	const int j = blockIdx.x * 32 + cl;
	double sum = 0.0;
	if (j < k) {
#pragma unroll 4
		for (int i = rg; i < kp; i += 32) {
			const double2 v = __ldcg(V + (long long)i * kp + j);
			sum += v.x * v.x + v.y * v.y;
		}
	}
	part[rg][cl] = sum;
	__syncthreads();
	if (rg == 0) {
		double t = 0.0;
		for (int r = 0; r < 32; r++) t += part[r][cl];
		part[0][cl] = t > 0.0 ? 1.0 / sqrt(t) : 1.0;
	}
	__syncthreads();
	const double f = part[0][cl];
	if (j < k) {
#pragma unroll 4
		for (int i = rg; i < kp; i += 32) {
			const long long o = (long long)i * kp + j;
			const double2 v = __ldcg(V + o);
			V[o] = make_double2(v.x * f, v.y * f);
		}
	}
}

// Sort the k eigenvalues ascending (bitonic, one CTA) and run the checks of
// stateset.cpp:158-173 in that order.
__global__ void eig_sort_kernel(const double2* __restrict__ A0, const double2* __restrict__ A1,
		const double2* __restrict__ A2, int k, int kp, const int* counters, int max_sweeps, double* evals, int* perm,
		EigStatus* st, int check) {
	extern __shared__ unsigned char sm[];
	int P = 1;
	while (P < k) P <<= 1;
	double* key = reinterpret_cast<double*>(sm);
	int* idx = reinterpret_cast<int*>(key + P);
	const int which = counters[max_sweeps + 1];
	const double2* A = which == 0 ? A0 : (which == 1 ? A1 : A2);
	for (int i = threadIdx.x; i < P; i += blockDim.x) {
		if (i < k) {
			double v = __ldcg(A + (long long)i * kp + i).x;
			if (v != v) v = -INFINITY;  // NaN sorts first so the check below reports it
			key[i] = v;
		} else {
			key[i] = INFINITY;
		}
		idx[i] = i;
	}
	__syncthreads();
	for (int size = 2; size <= P; size <<= 1) {
		for (int stride = size >> 1; stride > 0; stride >>= 1) {
			for (int i = threadIdx.x; i < P; i += blockDim.x) {
				const int j = i ^ stride;
				if (j > i) {
					const bool up = (i & size) == 0;
					const double ki = key[i], kj = key[j];
					const bool swap = up ? (ki > kj || (ki == kj && idx[i] > idx[j]))
					                     : (ki < kj || (ki == kj && idx[i] < idx[j]));
					if (swap) {
						key[i] = kj;
						key[j] = ki;
						const int t = idx[i];
						idx[i] = idx[j];
						idx[j] = t;
					}
				}
			}
			__syncthreads();
		}
	}
	// the checks in eigenvalue order: the first failing n, found in parallel
	__shared__ int first_bad;
	if (threadIdx.x == 0) first_bad = k;
	__syncthreads();
	for (int i = threadIdx.x; i < k; i += blockDim.x) {
		perm[i] = idx[i];
		const double v = __ldcg(A + (long long)idx[i] * kp + idx[i]).x;
		evals[i] = v;
		if (check && (v <= 0.0 || !(v >= 2.2250738585072014e-308) || isinf(v) || v != v)) atomicMin(&first_bad, i);
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		EigStatus s;
		s.status = ITP2D_OK;
		s.bad_index = -1;
		s.bad_value = 0.0;
		s.pad = 0;
		s.sweeps = counters[max_sweeps];
		if (s.sweeps < 0 && check == 2) {
			s.sweeps = max_sweeps;  // a capped solve: the caller finishes it
		} else if (s.sweeps < 0) {
			s.status = ITP2D_E_EIGENSOLVER;
		} else if (first_bad < k) {
			const int n = first_bad;
			const double v = __ldcg(A + (long long)idx[n] * kp + idx[n]).x;
			s.status = v <= 0.0 ? ITP2D_E_NONPOSITIVE_EIGENVALUE : ITP2D_E_NONNORMAL_EIGENVALUE;
			s.bad_index = n;
			s.bad_value = v;
		}
		*st = s;
	}
}

// S_out[a][b] = (A[p(a)][p(b)] + conj(A[p(b)][p(a)])) / 2 and VT[a][i] =
// V[i][p(a)], p(a) = perm[k - 1 - a]: the overlap of the states rotated onto
// the columns of V, largest eigenvalue (lowest energy) first.
__global__ void eig_cholesky_prep_kernel(const double2* __restrict__ A0, const double2* __restrict__ A1,
		const double2* __restrict__ A2, const double2* __restrict__ V, const int* __restrict__ perm,
		const int* __restrict__ counters, int max_sweeps, int k, int kp, double2* __restrict__ S_out,
		double2* __restrict__ VT) {
	const int which = counters[max_sweeps + 1];
	const double2* A = which == 0 ? A0 : (which == 1 ? A1 : A2);
	const long long n2 = (long long)k * k;
	for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n2;
			idx += (long long)gridDim.x * blockDim.x) {
		const int a = (int)(idx / k), b = (int)(idx % k);
		const int pa = perm[k - 1 - a], pb = perm[k - 1 - b];
		const double2 x = __ldcg(A + (long long)pa * kp + pb), y = __ldcg(A + (long long)pb * kp + pa);
		S_out[idx] = make_double2(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
		VT[idx] = __ldcg(V + (long long)b * kp + pa);
	}
}

// W[i][n] = V[i][perm[n]] / sqrt(l_n) (the zdscal of stateset.cpp:175).
__global__ void build_w_kernel(const double2* __restrict__ V, int k, int kp, const double* __restrict__ evals,
		const int* __restrict__ perm, double2* W) {
	const long long n2 = (long long)k * k;
	for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n2;
			idx += (long long)gridDim.x * blockDim.x) {
		const int i = (int)(idx / k), n = (int)(idx % k);
		const double f = 1.0 / sqrt(evals[n]);
		const double2 v = __ldcg(V + (long long)i * kp + perm[n]);
		W[idx] = make_double2(v.x * f, v.y * f);
	}
}

// W[i][n] = V[i][perm[n]]: the Ritz vectors' coefficients, ascending Ritz values.
__global__ void ritz_w_kernel(const double2* __restrict__ V, int k, int kp, const int* __restrict__ perm, double2* W) {
	const long long n2 = (long long)k * k;
	for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n2;
			idx += (long long)gridDim.x * blockDim.x) {
		const int i = (int)(idx / k), n = (int)(idx % k);
		W[idx] = __ldcg(V + (long long)i * kp + perm[n]);
	}
}

}  // namespace

int eigensolve_exponent(int n, const double* A) {
	double top = 0.0;
	for (int j = 0; j < n; j++)
		for (int i = 0; i <= j; i++) {
			const double* v = A + 2 * ((size_t)j * n + i);
			top = std::max(top, std::max(std::fabs(v[0]), i == j ? 0.0 : std::fabs(v[1])));
		}
	return top > 0.0 && std::isfinite(top) && (top < 0x1p-400 || top > 0x1p400) ? std::ilogb(top) : 0;
}

size_t jacobi_counters(int max_sweeps) { return jacobi_counter_ints(max_sweeps); }

namespace {
std::atomic<int> g_coop_users{0};
std::mutex g_coop_mu;
}  // namespace

void coop_user_enter() { g_coop_users.fetch_add(1); }
void coop_user_leave() { g_coop_users.fetch_sub(1); }

cudaError_t launch_eigensolve(double2* S, int k, JacobiWork& w, double2* W, EigStatus* st, int num_sms,
		cudaStream_t s) {
	cudaError_t e = launch_eigh(S, k, w, st, num_sms, s, 1);
	if (e != cudaSuccess) return e;
	const long long n2 = (long long)k * k;
	const int kp = jacobi_kp(k);
	build_w_kernel<<<(unsigned)std::min<long long>((n2 + 255) / 256, 4096), 256, 0, s>>>(w.V, k, kp, w.evals,
			w.perm, W);
	return cudaGetLastError();
}

cudaError_t launch_ritz(double2* H, int k, JacobiWork& w, double2* W, EigStatus* st, int num_sms, cudaStream_t s) {
	cudaError_t e = launch_eigh(H, k, w, st, num_sms, s, 0);
	if (e != cudaSuccess) return e;
	const long long n2 = (long long)k * k;
	ritz_w_kernel<<<(unsigned)std::min<long long>((n2 + 255) / 256, 4096), 256, 0, s>>>(w.V, k, jacobi_kp(k),
			w.perm, W);
	return cudaGetLastError();
}

cudaError_t launch_eig_cholesky_prep(const JacobiWork& w, int k, double2* S_out, double2* VT, cudaStream_t s) {
	const long long n2 = (long long)k * k;
	eig_cholesky_prep_kernel<<<(unsigned)std::min<long long>((n2 + 255) / 256, 4096), 256, 0, s>>>(w.A0, w.A1, w.A2,
			w.V, w.perm, w.counters, w.max_sweeps, k, jacobi_kp(k), S_out, VT);
	return cudaGetLastError();
}

int jacobi_kp(int k) { return bjacobi_padded(k); }

cudaError_t launch_eigh(double2* S, int k, JacobiWork& w, EigStatus* st, int num_sms, cudaStream_t s, int check) {
	const int kp = jacobi_kp(k);
	const long long n = (long long)kp * kp;
	cudaError_t e = cudaMemsetAsync(w.counters, 0, jacobi_counters(w.max_sweeps) * sizeof(int), s);
	if (e != cudaSuccess) return e;
	// one cooperative kernel at a time while several users share the device:
	// held until the kernel below has finished
	std::unique_lock<std::mutex> serial;
	if (g_coop_users.load() > 1) serial = std::unique_lock<std::mutex>(g_coop_mu);
	if (w.f32.A0 && k >= kBlockJacobi32MinK) {
		e = launch_bjacobi32(S, k, w, num_sms, s);
	} else {
		jacobi_init_kernel<<<(unsigned)std::min<long long>((n + 255) / 256, 4096), 256, 0, s>>>(S, k, kp, w.A0,
				w.V);
		e = launch_bjacobi(w.A0, w.A1, w.A2, w.V, w.Qbuf, k, kp, w.max_sweeps, w.tau_final, w.counters, num_sms, s);
	}
	if (e != cudaSuccess) return e;
	if (serial.owns_lock()) {
		e = cudaStreamSynchronize(s);
		serial.unlock();
		if (e != cudaSuccess) return e;
	}
	normalize_columns_kernel<<<(k + 31) / 32, 1024, 0, s>>>(w.V, k, kp);
	int P = 1;
	while (P < k) P <<= 1;
	const size_t smem = (size_t)P * (sizeof(double) + sizeof(int));
	// up to 16384 keys (the kernel has static shared memory beside them)
	if (smem > 48 * 1024) raise_smem_limit((const void*)eig_sort_kernel, 192 * 1024);
	eig_sort_kernel<<<1, 1024, smem, s>>>(w.A0, w.A1, w.A2, k, kp, w.counters, w.max_sweeps, w.evals, w.perm,
			st, check);
	return cudaGetLastError();
}

}  // namespace itp2d
