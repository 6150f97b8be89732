// One imaginary time step of small square periodic grids in one launch: a state
// stays in shared memory through every row and column pass of a member.
//
// The passes of a step (35 for the 10th order) cost a launch and a round trip
// through L2 each, about 2.6 us at 64 x 64 whatever the work. Here a cluster of
// m / 2 + 1 CTAs takes a state: CTA r runs member m - r and, where that is
// another one, member r, so that every CTA has about as many passes as the
// longest member alone; then the cluster adds the members out of each other's
// shared memory in the order of the passes ((m1 + m2) + m3 ...). A member's
// chain runs on one SM, in stages of 512 threads with a barrier between them: 25
// states of 64 x 64 (FP64, 10th order) take 37 us, in place of 93; two contexts
// that step in turn, each on its own stream, overlap and take 19 us a step. A
// stage of 4096 points takes 1900 cycles: 1270 of shared-memory traffic and 700
// of FP64 work that the barriers keep from overlapping wholly (tables brought into
// L1 ahead, or row stages that wait for their warp alone, changed nothing).
//
// The stages are those of lines.cuh, all in place: an alpha item of row y reads
// and writes the slots [k1][b] of its b, a beta item those of its k1 (rows of A
// runs of BP slots), so a row's points are x = b + B k1 between an alpha stage
// and the next and kx = k1 + A j (j the slot in the run) between a beta stage
// and the next; a column pass, whose arithmetic does not depend on the order of
// the columns, runs over the slots with that kx for its table. Columns use the
// rows b + B k1 in the same way. Odd runs: neither stage has bank conflicts.
#pragma once

#include "lines.cuh"

#include <cooperative_groups.h>

namespace itp2d {

namespace lines {

constexpr int kSmallThreads = 512;

// f(i) for the items i of this thread.
template <int ITEMS, class F>
__device__ __forceinline__ void items(F&& f) {
	for (int i = threadIdx.x; i < ITEMS; i += kSmallThreads) f(i);
	__syncthreads();
}

template <class R, int A, int B>
__global__ void __launch_bounds__(kSmallThreads, 1) small_step_kernel(SmallStepArgs a) {
	namespace cg = cooperative_groups;
	using G = Geo<R, A, B>;
	using T = c2<R>;
	constexpr int N = G::N, BP = G::BP, P = A * BP;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	T* S = reinterpret_cast<T*>(smem_raw);  // [N][A][BP]
	T* xtw = S + N * P;                     // [A][BP]
	T* S2 = xtw + P;                        // [N][N], with a second member
	load_tw<R, G, BP>(xtw, a.tw);
	__syncthreads();
	const int m = a.m, nc = m / 2 + 1, rank = (int)blockIdx.x % nc;
	const long long state = blockIdx.x / nc;
	const T* in = reinterpret_cast<const T*>(a.psi) + state * N * N;

	for (int pick = 0; pick < 2; pick++) {
		// the second member first: its result waits in S2
		const int t = pick ? m - rank : rank;
		if (pick == 0 && (rank == 0 || rank >= m - rank)) continue;
		const SmallMember& mb = a.member[t - 1];
		const R* kx = reinterpret_cast<const R*>(mb.kx);
		const R* vh = reinterpret_cast<const R*>(mb.vh);
		// V / 2 and the forward x transform
		items<N * B>([&](int i) {
			const int y = i / B, b = i % B;
			T v[A];
#pragma unroll
			for (int j = 0; j < A; j++) v[j] = in[y * N + b + B * j];
			if (vh) times<T, A>(v, vh + y * N + b, [](int j) { return B * j; });
			dft<R, A, -1>(v);
			twiddle<R, A, -1, BP>(v, xtw + b);
#pragma unroll
			for (int j = 0; j < A; j++) S[y * P + j * BP + b] = v[j];
		});
		for (int r = 1; r <= t; r++) {
			items<N * A>([&](int i) {
				const int y = i / A, k1 = i % A;
				T* s = S + y * P + k1 * BP;
				T u[B];
#pragma unroll
				for (int j = 0; j < B; j++) u[j] = s[j];
				dft<R, B, -1>(u);
				if (kx) times<T, B>(u, kx + y * N + k1, [](int j) { return A * j; });
#pragma unroll
				for (int j = 0; j < B; j++) s[j] = u[j];
			});
			// column pass: transform pair along y with the kinetic table
			items<N * B>([&](int i) {
				const int b = i / N, c = i % N;
				T* s = S + (c / B) * BP + c % B + b * P;
				T v[A];
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = s[B * j * P];
				dft<R, A, -1>(v);
				twiddle<R, A, -1, BP>(v, xtw + b);
#pragma unroll
				for (int j = 0; j < A; j++) s[B * j * P] = v[j];
			});
			items<N * A>([&](int i) {
				const int k1 = i / N, c = i % N;
				T* s = S + (c / B) * BP + c % B + B * k1 * P;
				T u[B];
#pragma unroll
				for (int j = 0; j < B; j++) u[j] = s[j * P];
				dft<R, B, -1>(u);
				if (mb.kmul) {
					const R* m2 = reinterpret_cast<const R*>(mb.kmul) + k1 * N + c / B + A * (c % B);
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = scale(u[j], m2[A * j * N]);
				} else {
					const R* m1 = reinterpret_cast<const R*>(mb.ky) + k1;
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = scale(u[j], m1[A * j]);
				}
				dft<R, B, 1>(u);
				twiddle<R, B, 1, 1>(u, xtw + k1 * BP);
#pragma unroll
				for (int j = 0; j < B; j++) s[j * P] = u[j];
			});
			items<N * B>([&](int i) {
				const int b = i / N, c = i % N;
				T* s = S + (c / B) * BP + c % B + b * P;
				T v[A];
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = s[B * j * P];
				dft<R, A, 1>(v);
#pragma unroll
				for (int j = 0; j < A; j++) s[B * j * P] = v[j];
			});
			// inverse x transform, V (or c_t V / 2), forward x transform
			items<N * A>([&](int i) {
				const int y = i / A, k1 = i % A;
				T* s = S + y * P + k1 * BP;
				T u[B];
#pragma unroll
				for (int j = 0; j < B; j++) u[j] = s[j];
				if (kx) times<T, B>(u, kx + y * N + k1, [](int j) { return A * j; });
				dft<R, B, 1>(u);
				twiddle<R, B, 1, 1>(u, xtw + k1 * BP);
#pragma unroll
				for (int j = 0; j < B; j++) s[j] = u[j];
			});
			const bool last = r == t;
			const R* mid = reinterpret_cast<const R*>(last ? mb.vp : mb.vsq);
			items<N * B>([&](int i) {
				const int y = i / B, b = i % B;
				T* s = S + y * P + b;
				T v[A];
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = s[j * BP];
				dft<R, A, 1>(v);
				if (mid) times<T, A>(v, mid + y * N + b, [](int j) { return B * j; });
				if (last && pick == 0) {
#pragma unroll
					for (int j = 0; j < A; j++) S2[y * N + b + B * j] = v[j];
					return;
				}
				if (!last) {
					dft<R, A, -1>(v);
					twiddle<R, A, -1, BP>(v, xtw + b);
				}
#pragma unroll
				for (int j = 0; j < A; j++) s[j * BP] = v[j];
			});
		}
	}

	cg::cluster_group cluster = cg::this_cluster();
	cluster.sync();
	T* out = reinterpret_cast<T*>(a.out) + state * N * N;
	for (int i = rank * kSmallThreads + threadIdx.x; i < N * N; i += nc * kSmallThreads) {
		const int y = i / N, x = i % N;
		const int slot = y * P + (x / B) * BP + x % B;
		T sum;
		for (int t = 1; t <= m; t++) {
			// member t is the first one of CTA m - t, or the second one of CTA t
			const bool first = m - t < nc && (m - t == 0 || t >= m - t);
			const T v = first ? cluster.map_shared_rank(S, m - t)[slot] : cluster.map_shared_rank(S2, t)[i];
			sum = t == 1 ? v : add(v, sum);
		}
		out[i] = sum;
	}
	cluster.sync();  // the others may still be reading this CTA's shared memory
}

// Shared memory of a grid of N x N points at m members.
template <class G>
constexpr size_t small_smem(int m) {
	return (size_t)G::ES * ((size_t)(G::N + 1) * G::A * G::BP + (m >= 3 ? G::N * G::N : 0));
}

// Whether one launch beats the passes, both in microseconds of device time. A
// pass takes about 2.5 us plus its traffic at 6 TB/s (L2, at these sizes); a wave
// of clusters 3 us plus, per stage and point, 0.27 ns (FP64) or 0.165 ns (FP32).
// Measured, passes against one launch: FP64 64 x 64, 10th order, 25 states 93
// and 37 us, 800 states 731 and 625; 4th order, 800 states 160 and 179;
// 100 x 100, 4th order, 16 states 26 and 45; FP32 96 x 96, 6th order, 50 states 55
// and 41; 160 x 160, 4th order, 25 states 33 and 69.
template <class G>
bool small_pays(int m, int k) {
	const double points = (double)G::N * G::N;
	const double passes = m * (m + 2) * (2.5 + 2.0 * k * points * G::ES / 6e6);
	// stages of the longest CTA: 6 t + 1 per member t
	const int nc = m / 2 + 1, stages = m >= 3 ? 6 * m + 2 : 6 * m + 1;
	const int at_once = std::max(1, sm_count() / nc);
	const int waves = (k + at_once - 1) / at_once;
	return waves * (3.0 + stages * points * (G::ES == 16 ? 0.27e-3 : 0.165e-3)) < passes;
}

template <class R>
bool small_step(const SmallStepArgs& a, int n, int k, cudaStream_t s) {
	bool done = false;
	for_length<R>(n, [&](auto g) {
		using G = decltype(g);
		if constexpr (small_smem<G>(1) <= kSmemMax) {
			const size_t sm = small_smem<G>(a.m);
			if (sm > kSmemMax || !small_pays<G>(a.m, k)) return;
			const int nc = a.m / 2 + 1;
			auto kernel = small_step_kernel<R, G::A, G::B>;
			cudaError_t e = raise_smem_limit((const void*)kernel);
			cudaLaunchAttribute at[1];
			at[0].id = cudaLaunchAttributeClusterDimension;
			at[0].val.clusterDim.x = nc;
			at[0].val.clusterDim.y = 1;
			at[0].val.clusterDim.z = 1;
			cudaLaunchConfig_t cfg = {};
			cfg.gridDim = dim3((unsigned)(k * nc));
			cfg.blockDim = dim3(kSmallThreads);
			cfg.dynamicSmemBytes = sm;
			cfg.stream = s;
			cfg.attrs = at;
			cfg.numAttrs = 1;
			if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kernel, a);
			done = e == cudaSuccess;
			if (!done) cudaGetLastError();  // refused: the passes run instead, and report what they meet
		}
	});
	return done;
}

}  // namespace lines

}  // namespace itp2d
