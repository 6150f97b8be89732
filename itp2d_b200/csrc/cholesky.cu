// Cholesky (Gram-Schmidt order) orthonormalisation.
//
// With S = Psi^H Psi dx^2 Hermitian positive definite and S = L L^H its
// Cholesky factorisation (L lower triangular, real positive diagonal),
// W = L^{-H} is upper triangular and W^H S W = I: output state n is a
// combination of the input states 0..n only, the result of Gram-Schmidt in
// storage order. The eigendecomposition of the canonical form is replaced by
// about k^3 / 2 complex multiply-adds in three kinds of launches per panel of
// 32 columns:
//
//   1. one CTA factors the diagonal block S_jj = L_jj L_jj^H in shared memory
//      and inverts L_jj;
//   2. the panel below becomes L_21 = A_21 L_jj^{-H}, and the rows of the
//      running inverse X (L X = I, block forward substitution) that belong to
//      this panel become L_jj^{-1} X_j;
//   3. the trailing lower triangle takes A_22 -= L_21 L_21^H and the rows of X
//      below the panel take X_2 -= L_21 X_j (64 x 64 output tiles, FP64).
//
// Finally W[i k + n] = conj(X[n k + i]) for i <= n and 0 below. A pivot that
// is not a positive finite number stops the factorisation with
// ITP2D_E_NONPOSITIVE_EIGENVALUE (bad index = the pivot's row). No reference
// counterpart: the reference orthonormalises canonically (stateset.cpp:136-232).
#include "../../include/itp2d_gpu.h"
#include "contract.cuh"
#include "launch.cuh"

#include <algorithm>

namespace itp2d {

namespace {

constexpr int NB = 32;   // panel width
constexpr int TU = 64;   // trailing-update output tile

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
	return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
	return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// X = I (row-major k x k)
__global__ void chol_identity_kernel(double2* X, int k) {
	const long long n2 = (long long)k * k;
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += (long long)gridDim.x * blockDim.x)
		X[i] = make_double2(i / k == i % k ? 1.0 : 0.0, 0.0);
}

// Step 1: L_jj and L_jj^{-1} of the diagonal block at (j, j); 1024 threads,
// thread (r, c) holding element (r, c) of the block and of its inverse in
// registers. The inverse is built along with the factor (forward substitution
// of the identity: row p of X is final once it is divided by the pivot), two
// barriers per pivot; the thread of the next pivot prepares its reciprocal
// square root right after its update. Latency-bound: a chain of 32 pivots
// (39 us with the inverse substituted afterwards by one thread per column,
// 18 us now).
__global__ void __launch_bounds__(1024) chol_diag_kernel(double2* A, int k, int j, double2* Linv, EigStatus* st) {
	__shared__ double2 lcol[NB], xrow[NB];  // column p of L, row p of X
	__shared__ double s_pivot[2], s_inv[2];
	if (st->status != 0) return;
	const int nb = min(NB, k - j);
	const int r = threadIdx.x / NB, c = threadIdx.x % NB;
	const bool in = r < nb && c <= r;
	double2 l = in ? A[(long long)(j + r) * k + j + c] : make_double2(0.0, 0.0);
	double2 x = make_double2(r == c ? 1.0 : 0.0, 0.0);
	if (threadIdx.x == 0) {
		s_pivot[0] = l.x;
		s_inv[0] = rsqrt(l.x);
	}
	__syncthreads();
	for (int p = 0; p < nb; p++) {
		const double pivot = s_pivot[p & 1], inv = s_inv[p & 1];
		if (!(pivot > 0.0) || !isfinite(pivot)) {
			if (threadIdx.x == 0) {
				st->status = ITP2D_E_NONPOSITIVE_EIGENVALUE;
				st->bad_index = j + p;
				st->bad_value = pivot;
			}
			return;  // every thread read the same pivot: the whole CTA leaves here
		}
		if (c == p && r >= p) {
			l = r == p ? make_double2(pivot * inv, 0.0) : make_double2(l.x * inv, l.y * inv);
			lcol[r] = l;
		}
		if (r == p && c <= p) {
			x = make_double2(x.x * inv, x.y * inv);
			xrow[c] = x;
		}
		__syncthreads();
		if (r > p && r < nb) {
			const double2 lr = lcol[r];
			if (c > p && c <= r) {
				l = csub(l, cmulc(lr, lcol[c]));
				if (r == p + 1) {  // c == r: the next pivot
					s_pivot[r & 1] = l.x;
					s_inv[r & 1] = rsqrt(l.x);
				}
			}
			if (c <= p) x = csub(x, cmul(lr, xrow[c]));
		}
		__syncthreads();
	}
	if (in) A[(long long)(j + r) * k + j + c] = l;
	// zero above the diagonal and beyond nb
	Linv[r * NB + c] = in ? x : make_double2(0.0, 0.0);
}

// Step 2: blocks [0, nrb) turn 32 rows of the panel below the diagonal block
// into L_21 = A_21 L_jj^{-H}; blocks [nrb, ...) turn 32 columns of X's panel
// rows into L_jj^{-1} X_j. 256 threads.
__global__ void __launch_bounds__(256) chol_panel_kernel(double2* A, double2* X, int k, int j, const double2* Linv,
		int nrb, const EigStatus* st) {
	__shared__ double2 Li[NB][NB + 1];
	__shared__ double2 T[NB][NB + 1];
	if (st->status != 0) return;
	const int nb = min(NB, k - j), r0 = j + nb;
	constexpr int NE = NB * NB / 256;  // outputs per thread: rows rr, rr + 8, ...
	if ((int)blockIdx.x < nrb) {
		const int row0 = r0 + NB * blockIdx.x;
		const int rr = threadIdx.x / NB, q = threadIdx.x % NB;
		double2 lv[NE], tv[NE];
#pragma unroll
		for (int e = 0; e < NE; e++) {
			const int row = row0 + rr + 8 * e;
			lv[e] = __ldcg(Linv + threadIdx.x + 256 * e);
			tv[e] = (row < k && q < nb) ? __ldcg(A + (long long)row * k + j + q) : make_double2(0.0, 0.0);
		}
#pragma unroll
		for (int e = 0; e < NE; e++) {
			Li[rr + 8 * e][q] = lv[e];
			T[rr + 8 * e][q] = tv[e];
		}
		__syncthreads();
		// L^{-1} is zero above its diagonal: the sums run over the whole row
		double2 s[NE];
#pragma unroll
		for (int e = 0; e < NE; e++) s[e] = make_double2(0.0, 0.0);
#pragma unroll 8
		for (int p = 0; p < NB; p++) {
			const double2 l = Li[q][p];
#pragma unroll
			for (int e = 0; e < NE; e++) {
				const double2 a = T[rr + 8 * e][p];
				s[e].x += a.x * l.x + a.y * l.y;  // a * conj(l)
				s[e].y += a.y * l.x - a.x * l.y;
			}
		}
#pragma unroll
		for (int e = 0; e < NE; e++) {
			const int row = row0 + rr + 8 * e;
			if (row < k && q < nb) A[(long long)row * k + j + q] = s[e];
		}
		return;
	}
	for (int i = threadIdx.x; i < NB * NB; i += blockDim.x) Li[i / NB][i % NB] = Linv[i];
	const int c0 = NB * (blockIdx.x - nrb);
	if (c0 >= j) {
		// the panel's own columns: X_j = L_jj^{-1} there (identity before)
		for (int i = threadIdx.x; i < NB * NB; i += blockDim.x) {
			const int q = i / NB, cc = i % NB;
			if (q < nb && cc < nb) X[(long long)(j + q) * k + j + cc] = Li[q][cc];
		}
		return;
	}
	const int q0 = threadIdx.x / NB, cc = threadIdx.x % NB;
	double2 tv[NE];
#pragma unroll
	for (int e = 0; e < NE; e++)
		tv[e] = q0 + 8 * e < nb ? __ldcg(X + (long long)(j + q0 + 8 * e) * k + c0 + cc) : make_double2(0.0, 0.0);
#pragma unroll
	for (int e = 0; e < NE; e++) T[q0 + 8 * e][cc] = tv[e];
	__syncthreads();
	double2 s[NE];
#pragma unroll
	for (int e = 0; e < NE; e++) s[e] = make_double2(0.0, 0.0);
#pragma unroll 8
	for (int p = 0; p < NB; p++) {
		const double2 x = T[p][cc];
#pragma unroll
		for (int e = 0; e < NE; e++) {
			const double2 l = Li[q0 + 8 * e][p];
			s[e].x += l.x * x.x - l.y * x.y;
			s[e].y += l.x * x.y + l.y * x.x;
		}
	}
#pragma unroll
	for (int e = 0; e < NE; e++)
		if (q0 + 8 * e < nb) X[(long long)(j + q0 + 8 * e) * k + c0 + cc] = s[e];
}

// Step 3: rows [r0, k) of the trailing part. Column tiles [0, ncx) cover X's
// columns [0, r0) (X_2 -= L_21 X_j); the rest cover A's columns [r0, k)
// aligned with the row tiles (A_22 -= L_21 L_21^H, lower triangle only).
// 256 threads, 4 x 4 outputs each.
__global__ void __launch_bounds__(256, 2) chol_update_kernel(double2* A, double2* X, int k, int j, int ncx,
		const EigStatus* st) {
	extern __shared__ __align__(16) unsigned char smem_raw[];
	double2(*Lt)[NB + 1] = reinterpret_cast<double2(*)[NB + 1]>(smem_raw);             // [TU][NB + 1]
	double2(*Bt)[TU + 1] = reinterpret_cast<double2(*)[TU + 1]>(smem_raw + sizeof(double2) * TU * (NB + 1));
	if (st->status != 0) return;
	const int nb = min(NB, k - j), r0 = j + nb;
	const int rt = blockIdx.y, ct = blockIdx.x;
	const bool xpart = ct < ncx;
	if (!xpart && ct - ncx > rt) return;  // strictly above the diagonal
	const int row0 = r0 + TU * rt;
	const int col0 = xpart ? TU * ct : r0 + TU * (ct - ncx);
	const int col_end = xpart ? r0 : k;
	// every global load of the tile at once, then the shared-memory stores
	constexpr int NL = TU * NB / 256;
	double2 lv[NL], bv[NL];
#pragma unroll
	for (int e = 0; e < NL; e++) {
		const int i = threadIdx.x + 256 * e, rr = i / NB, q = i % NB, row = row0 + rr;
		lv[e] = (row < k && q < nb) ? __ldcg(A + (long long)row * k + j + q) : make_double2(0.0, 0.0);
		if (xpart) {
			const int qq = i / TU, col = col0 + i % TU;
			bv[e] = (qq < nb && col < col_end) ? __ldcg(X + (long long)(j + qq) * k + col) : make_double2(0.0, 0.0);
		} else {
			const int col = col0 + rr;
			bv[e] = (q < nb && col < col_end) ? __ldcg(A + (long long)col * k + j + q) : make_double2(0.0, 0.0);
		}
	}
#pragma unroll
	for (int e = 0; e < NL; e++) {
		const int i = threadIdx.x + 256 * e, rr = i / NB, q = i % NB;
		Lt[rr][q] = lv[e];
		if (xpart) Bt[i / TU][i % TU] = bv[e];
		else Bt[q][rr] = make_double2(bv[e].x, -bv[e].y);
	}
	__syncthreads();
	const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
	double2 acc[4][4];
#pragma unroll
	for (int a = 0; a < 4; a++)
#pragma unroll
		for (int b = 0; b < 4; b++) acc[a][b] = make_double2(0.0, 0.0);
	for (int q = 0; q < nb; q++) {
		double2 l[4], r[4];
#pragma unroll
		for (int a = 0; a < 4; a++) l[a] = Lt[ty + 16 * a][q];
#pragma unroll
		for (int b = 0; b < 4; b++) r[b] = Bt[q][tx + 16 * b];
#pragma unroll
		for (int a = 0; a < 4; a++)
#pragma unroll
			for (int b = 0; b < 4; b++) {
				acc[a][b].x += l[a].x * r[b].x - l[a].y * r[b].y;
				acc[a][b].y += l[a].x * r[b].y + l[a].y * r[b].x;
			}
	}
	double2* out = xpart ? X : A;
	// the old values of two rows of outputs at once (the compiler cannot move a
	// load above an earlier output's store)
#pragma unroll
	for (int a0 = 0; a0 < 4; a0 += 2) {
		double2 old[2][4];
#pragma unroll
		for (int a = 0; a < 2; a++)
#pragma unroll
			for (int b = 0; b < 4; b++) {
				const int row = row0 + ty + 16 * (a0 + a), col = col0 + tx + 16 * b;
				if (row < k && col < col_end && (xpart || col <= row)) old[a][b] = __ldcg(out + (long long)row * k + col);
			}
#pragma unroll
		for (int a = 0; a < 2; a++)
#pragma unroll
			for (int b = 0; b < 4; b++) {
				const int row = row0 + ty + 16 * (a0 + a), col = col0 + tx + 16 * b;
				if (row < k && col < col_end && (xpart || col <= row))
					out[(long long)row * k + col] = csub(old[a][b], acc[a0 + a][b]);
			}
	}
}

// W[i k + n] = conj(X[n k + i]) for i <= n, 0 below (32 x 32 tiles through
// shared memory, coalesced both ways). 32 x 8 threads.
__global__ void chol_w_kernel(const double2* X, int k, double2* W, const EigStatus* st) {
	__shared__ double2 t[32][33];
	if (st->status != 0) return;
	const int bi = blockIdx.y * 32, bn = blockIdx.x * 32;  // W tile rows i, columns n
	for (int yy = threadIdx.y; yy < 32; yy += 8) {
		const int n = bn + yy, i = bi + threadIdx.x;
		t[yy][threadIdx.x] = (n < k && i < k) ? X[(long long)n * k + i] : make_double2(0.0, 0.0);
	}
	__syncthreads();
	for (int yy = threadIdx.y; yy < 32; yy += 8) {
		const int i = bi + yy, n = bn + threadIdx.x;
		if (i >= k || n >= k) continue;
		const double2 x = t[threadIdx.x][yy];
		W[(long long)i * k + n] = i <= n ? make_double2(x.x, -x.y) : make_double2(0.0, 0.0);
	}
}

}  // namespace

size_t cholesky_update_smem() { return sizeof(double2) * (TU * (NB + 1) + NB * (TU + 1)); }

int launch_cholesky_w(const double2* S, int k, double2* A, double2* X, double2* Linv, double2* W, EigStatus* st,
		cudaStream_t s) {
	if (raise_smem_limit((const void*)chol_update_kernel, (int)cholesky_update_smem()) != cudaSuccess)
		return ITP2D_E_CUDA;
	cudaError_t e = cudaMemsetAsync(st, 0, sizeof(EigStatus), s);
	if (e == cudaSuccess) e = cudaMemcpyAsync(A, S, (size_t)k * k * sizeof(double2), cudaMemcpyDeviceToDevice, s);
	if (e != cudaSuccess) return ITP2D_E_CUDA;
	chol_identity_kernel<<<std::min(1184, (int)(((long long)k * k + 255) / 256)), 256, 0, s>>>(X, k);
	for (int j = 0; j < k; j += NB) {
		const int nb = std::min(NB, k - j), r0 = j + nb;
		chol_diag_kernel<<<1, 1024, 0, s>>>(A, k, j, Linv, st);
		const int nrb = (k - r0 + NB - 1) / NB, ncb = (r0 + NB - 1) / NB;
		chol_panel_kernel<<<nrb + ncb, 256, 0, s>>>(A, X, k, j, Linv, nrb, st);
		if (r0 < k) {
			const int nrt = (k - r0 + TU - 1) / TU, ncx = (r0 + TU - 1) / TU;
			chol_update_kernel<<<dim3(ncx + nrt, nrt), 256, cholesky_update_smem(), s>>>(A, X, k, j, ncx, st);
		}
	}
	const int nt = (k + 31) / 32;
	chol_w_kernel<<<dim3(nt, nt), dim3(32, 8), 0, s>>>(X, k, W, st);
	return cudaGetLastError() == cudaSuccess ? ITP2D_OK : ITP2D_E_CUDA;
}

int cholesky_launches(int k) { return 2 + 3 * ((k + NB - 1) / NB); }

}  // namespace itp2d
