// Row and column passes of Dirichlet lines (DST-II forward, DST-III inverse) on
// the two register stages of lines.cuh.
//
// A DST-II of N points is one N-point complex FFT of the reordered line
//   v_n = x_{2n} (2n < N),  v_{N-1-n} = -x_{2n+1}
// followed by a step on the pairs (V_m, V_{N-m}): with w = exp(-i pi / 2N),
// P = w^m V_m and Q = w^{-m} V_{N-m},
//   S_{N-1-m} = P + Q,   S_{m-1} = i (P - Q)   (0 < m < N, m != N/2),
//   S_{N-1} = 2 V_0,     S_{N/2-1} = sqrt(2) V_{N/2},
// and DST-III (2N times its inverse) undoes both steps:
//   V_m = w^{-m} (Y_{N-1-m} - i Y_{m-1}),  V_{N-m} = w^m (Y_{N-1-m} + i Y_{m-1}),
//   V_0 = Y_{N-1},  V_{N/2} = sqrt(2) Y_{N/2-1},  x from the inverse FFT of V.
// (DCT by an N-point FFT, J. Makhoul, IEEE Trans. ASSP 28 (1980) 27; the sine
// transform is the cosine transform of (-1)^j x_j read backwards.)
// The partner of point k1 + A k2 of beta item k1 belongs to beta item A - k1, so
// a thread takes the two items together and the pair step stays in registers:
// a sine pass costs the FFT passes' traffic and exchanges, where the odd
// extension to a 2N-point FFT in shared memory (split.cu, still used for the
// cosine kinds and other lengths) took 48 to 70 us for 64 FP64 states of
// 128 x 128 and these take 11 to 13 us. `ext` is the plan's table exp(-i pi m / 2N).
#pragma once

#include "lines.cuh"

namespace itp2d {

namespace lines {

// Threads per line and work split of the sine passes.
template <class G>
struct Sine {
	static constexpr int A = G::A, B = G::B, N = G::N;
	static constexpr int PAIRS = A % 2 ? (A + 1) / 2 : A / 2;  // beta item pairs; pair 0: items 0 and (A even) A/2
	static constexpr int CNT = PAIRS > B ? PAIRS : B;
	static constexpr int W = G::W;
	static constexpr int COL_THREADS = (CNT * W + 31) / 32 * 32;
	static constexpr int ROW_THREADS = G::ROW_THREADS;
	static constexpr bool WARP_LINE = 32 % CNT == 0;
	static constexpr int LS = CNT == 8 ? (A * G::BP + 15) / 16 * 16 + 8 : A * G::BP;
	// points of a thread's two beta items or its alpha item, and their registers
	static constexpr int POINTS = A > 2 * B ? A : 2 * B;
	static constexpr bool FITS = POINTS * (G::ES / 4) <= 168;
	static constexpr int blocks(int threads) {
		const int n = 65536 / (threads * ((POINTS * (G::ES / 4) + 80 + 7) / 8 * 8));
		return n < 1 ? 1 : n;
	}
};

// Position of the reordered point n, and whether it is negated.
template <int N>
__device__ __forceinline__ int sine_pos(int n) { return 2 * n < N ? 2 * n : 2 * (N - 1 - n) + 1; }
template <int N, class T>
__device__ __forceinline__ T sine_sign(int n, T v) {
	if (2 * n >= N) {
		v.x = -v.x;
		v.y = -v.y;
	}
	return v;
}

// Calls pair(V_m, V_{N-m}, m) for the pairs of a thread's items p and A - p
// (u[0..B) and u[B..2B)), zero(V_0) and half(V_{N/2}) for the points that are
// their own partner.
template <class G, class T, class FP, class FZ, class FH>
__device__ __forceinline__ void sine_pairs(T* u, int p, FP&& pair, FZ&& zero, FH&& half) {
	constexpr int A = G::A, B = G::B;
	if (p == 0) {
		zero(u[0]);
#pragma unroll
		for (int j = 1; j <= (B - 1) / 2; j++) pair(u[j], u[B - j], A * j);
		if (B % 2 == 0) half(u[B / 2]);
		if (A % 2 == 0) {
#pragma unroll
			for (int j = 0; j < B / 2; j++) pair(u[B + j], u[2 * B - 1 - j], A / 2 + A * j);
			if (B % 2) half(u[B + (B - 1) / 2]);
		}
	} else {
#pragma unroll
		for (int j = 0; j < B; j++) pair(u[j], u[2 * B - 1 - j], p + A * j);
	}
}

template <class T>
__device__ __forceinline__ T conj_of(T w) {
	w.y = -w.y;
	return w;
}

// (V_m, V_{N-m}) -> (P + Q, P - Q)
template <class R>
__device__ __forceinline__ void sine_out(c2<R>& a, c2<R>& b, c2<R> w) {
	const c2<R> P = cmul(a, w), Q = cmulc(b, w);
	a = add(P, Q);
	b = sub(P, Q);
}
// (A, iB) -> (V_m, V_{N-m}): w^{-m} (A - iB), w^m (A + iB)
template <class R>
__device__ __forceinline__ void sine_in(c2<R>& a, c2<R>& b, c2<R> w) {
	const c2<R> s = add(a, b), d = sub(a, b);
	a = cmulc(d, w);
	b = cmul(s, w);
}

// Column pass (ColPassArgs, kind 1), tiles as in col_kernel.
template <class R, int A, int B>
__global__ void __launch_bounds__((Sine<Geo<R, A, B>>::COL_THREADS),
		(Sine<Geo<R, A, B>>::blocks(Sine<Geo<R, A, B>>::COL_THREADS))) dst_col_kernel(ColPassArgs a, int k) {
	using G = Geo<R, A, B>;
	using H = Sine<G>;
	using T = c2<R>;
	constexpr int W = G::W, N = G::N;
	constexpr R r2 = (R)1.41421356237309504880;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	T* xtw = reinterpret_cast<T*>(smem_raw);
	load_tw<R, G, B, 2>(xtw, a.lp.fft.tw);
	__syncthreads();
	const int t = threadIdx.x / W, c = threadIdx.x % W;
	T* E = xtw + N + c;
	const bool alpha = t < B, beta = t < H::PAIRS;
	const int i0 = t, i1 = t == 0 ? A / 2 : A - t;  // this thread's beta items
	const bool two = t > 0 || A % 2 == 0;
	const int sx = a.sx;
	const int nct = (sx + W - 1) / W;
	const long long total = (long long)k * nct;
	const R* m2 = reinterpret_cast<const R*>(a.mul2d);
	const R* m1 = reinterpret_cast<const R*>(a.mul1d);
	const T* ext = reinterpret_cast<const T*>(a.lp.ext);
	for (long long tile = blockIdx.x; tile < total; tile += gridDim.x) {
		const int col = (int)(tile % nct) * W + c;
		const bool valid = col < sx;
		T* data = reinterpret_cast<T*>(a.data) + (tile / nct) * a.G + col;
		auto factor = [&](int y) { return m2 ? m2[y * sx + col] : m1[y]; };
		if (a.mode != 2) {
			if (valid && alpha) {
				T v[A];
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = sine_sign<N>(t + B * j, data[sine_pos<N>(t + B * j) * sx]);
				dft<R, A, -1>(v);
				twiddle<R, A, -1, B>(v, xtw + t);
#pragma unroll
				for (int j = 0; j < A; j++) E[(j * B + t) * W] = v[j];
			}
			__syncthreads();
		}
		if (valid && beta) {
			T u[2 * B];
			if (a.mode != 2) {
#pragma unroll
				for (int j = 0; j < B; j++) u[j] = E[(i0 * B + j) * W];
				dft<R, B, -1>(u);
				if (two) {
#pragma unroll
					for (int j = 0; j < B; j++) u[B + j] = E[(i1 * B + j) * W];
					dft<R, B, -1>(u + B);
				}
			}
			if (a.mode == 0) {
				sine_pairs<G>(
						u, t,
						[&](T& p, T& q, int m) {
							const T w = __ldg(ext + m);
							sine_out<R>(p, q, w);
							// times the factors of S_{N-1-m} and S_{m-1} (the i's cancel)
							p = scale(p, factor(N - 1 - m));
							q = scale(q, factor(m - 1));
							const T s = add(p, q), d = sub(p, q);
							p = cmulc(s, w);
							q = cmul(d, w);
						},
						[&](T& z) { z = scale(z, 2 * factor(N - 1)); }, [&](T& h) { h = scale(h, 2 * factor(N / 2 - 1)); });
			} else if (a.mode == 1) {
				sine_pairs<G>(
						u, t,
						[&](T& p, T& q, int m) {
							sine_out<R>(p, q, __ldg(ext + m));
							data[(N - 1 - m) * sx] = p;
							data[(m - 1) * sx] = mk<R>(-q.y, q.x);
						},
						[&](T& z) { data[(N - 1) * sx] = scale(z, (R)2); },
						[&](T& h) { data[(N / 2 - 1) * sx] = scale(h, r2); });
			} else {
				sine_pairs<G>(
						u, t,
						[&](T& p, T& q, int m) {
							p = data[(N - 1 - m) * sx];
							const T y = data[(m - 1) * sx];
							q = mk<R>(-y.y, y.x);
							sine_in<R>(p, q, __ldg(ext + m));
						},
						[&](T& z) { z = data[(N - 1) * sx]; }, [&](T& h) { h = scale(data[(N / 2 - 1) * sx], r2); });
			}
			if (a.mode != 1) {
				dft<R, B, 1>(u);
				twiddle<R, B, 1, 1>(u, xtw + i0 * B);
#pragma unroll
				for (int j = 0; j < B; j++) E[(i0 * B + j) * W] = u[j];
				if (two) {
					dft<R, B, 1>(u + B);
					twiddle<R, B, 1, 1>(u + B, xtw + i1 * B);
#pragma unroll
					for (int j = 0; j < B; j++) E[(i1 * B + j) * W] = u[B + j];
				}
			}
		}
		__syncthreads();
		if (a.mode == 1) continue;
		if (valid && alpha) {
			T v[A];
#pragma unroll
			for (int j = 0; j < A; j++) v[j] = E[(j * B + t) * W];
			dft<R, A, 1>(v);
#pragma unroll
			for (int j = 0; j < A; j++) data[sine_pos<N>(t + B * j) * sx] = sine_sign<N>(t + B * j, v[j]);
		}
		// mode 0: the next tile's first stage writes what the same thread read
		if (a.mode == 2) __syncthreads();
	}
}

// Row pass (RowPassArgs, kind 1), tiles as in row_kernel.
template <class R, int A, int B>
__global__ void __launch_bounds__((Sine<Geo<R, A, B>>::ROW_THREADS),
		(Sine<Geo<R, A, B>>::blocks(Sine<Geo<R, A, B>>::ROW_THREADS))) dst_row_kernel(RowPassArgs a, int k, int lines) {
	using G = Geo<R, A, B>;
	using H = Sine<G>;
	using T = c2<R>;
	constexpr int N = G::N, BP = G::BP;
	constexpr R r2 = (R)1.41421356237309504880;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	T* xtw = reinterpret_cast<T*>(smem_raw);
	load_tw<R, G, BP, 2>(xtw, a.lp.fft.tw);
	__syncthreads();
	const int line = threadIdx.x / H::CNT, t = threadIdx.x - line * H::CNT;
	T* E = xtw + A * BP + line * H::LS;
	const bool alpha = t < B, beta = t < H::PAIRS;
	const int i0 = t, i1 = t == 0 ? A / 2 : A - t;
	const bool two = t > 0 || A % 2 == 0;
	const int ntr = (a.sy + lines - 1) / lines;
	const long long total = (long long)k * ntr;
	const T* ext = reinterpret_cast<const T*>(a.lp.ext);
	for (long long tile = blockIdx.x; tile < total; tile += gridDim.x) {
		const long long state = tile % k;
		const int y = (int)(tile / k) * lines + line;
		const bool valid = line < lines && y < a.sy;
		const long long base = state * a.G + (long long)y * a.sx;
		const T* in = reinterpret_cast<const T*>(a.in) + base;
		T* out = reinterpret_cast<T*>(a.out) + base;
		const T* acc = a.acc ? reinterpret_cast<const T*>(a.acc) + base : nullptr;
		auto table = [&](const void* p) { return p ? reinterpret_cast<const R*>(p) + (long long)y * a.sx : nullptr; };
		const R *mpre = table(a.mul_pre), *mmid = table(a.mul_mid), *mpost = table(a.mul_post);
		if (a.do_inv) {
			if (valid && beta) {
				T u[2 * B];
				auto get = [&](int x) { return mpre ? scale(in[x], mpre[x]) : in[x]; };
				sine_pairs<G>(
						u, t,
						[&](T& p, T& q, int m) {
							p = get(N - 1 - m);
							const T b = get(m - 1);
							q = mk<R>(-b.y, b.x);
							sine_in<R>(p, q, __ldg(ext + m));
						},
						[&](T& z) { z = get(N - 1); }, [&](T& h) { h = scale(get(N / 2 - 1), r2); });
				dft<R, B, 1>(u);
				twiddle<R, B, 1, 1>(u, xtw + i0 * BP);
#pragma unroll
				for (int j = 0; j < B; j++) E[i0 * BP + j] = u[j];
				if (two) {
					dft<R, B, 1>(u + B);
					twiddle<R, B, 1, 1>(u + B, xtw + i1 * BP);
#pragma unroll
					for (int j = 0; j < B; j++) E[i1 * BP + j] = u[B + j];
				}
			}
			stage_sync<H>();
		}
		if (valid && alpha) {
			T v[A];
			if (a.do_inv) {
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = E[j * BP + t];
				dft<R, A, 1>(v);
			} else {
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = sine_sign<N>(t + B * j, in[sine_pos<N>(t + B * j)]);
			}
			if (mmid) times<T, A>(v, mmid, [=](int j) { return sine_pos<N>(t + B * j); });
			if (a.do_fwd) {
				dft<R, A, -1>(v);
				twiddle<R, A, -1, BP>(v, xtw + t);
#pragma unroll
				for (int j = 0; j < A; j++) E[j * BP + t] = v[j];
			} else {
#pragma unroll
				for (int j = 0; j < A; j++) {
					const int x = sine_pos<N>(t + B * j);
					const T z = sine_sign<N>(t + B * j, v[j]);
					out[x] = acc ? add(z, acc[x]) : z;
				}
			}
		}
		stage_sync<H>();
		if (!a.do_fwd) continue;
		if (valid && beta) {
			T u[2 * B];
#pragma unroll
			for (int j = 0; j < B; j++) u[j] = E[i0 * BP + j];
			dft<R, B, -1>(u);
			if (two) {
#pragma unroll
				for (int j = 0; j < B; j++) u[B + j] = E[i1 * BP + j];
				dft<R, B, -1>(u + B);
			}
			auto put = [&](int x, T z) {
				if (mpost) z = scale(z, mpost[x]);
				out[x] = acc ? add(z, acc[x]) : z;
			};
			sine_pairs<G>(
					u, t,
					[&](T& p, T& q, int m) {
						sine_out<R>(p, q, __ldg(ext + m));
						put(N - 1 - m, p);
						put(m - 1, mk<R>(-q.y, q.x));
					},
					[&](T& z) { put(N - 1, scale(z, (R)2)); }, [&](T& h) { put(N / 2 - 1, scale(h, r2)); });
		}
		// the next tile's inverse transform writes what the same thread read; a
		// forward one alone writes other threads' values
		if (!a.do_inv) stage_sync<H>();
	}
}

template <class R>
bool launch_dst_row(const RowPassArgs& a, int k, cudaStream_t s) {
	bool ran = false;
	for_length<R>(a.sx, [&](auto g) {
		using G = decltype(g);
		using H = Sine<G>;
		if constexpr (H::FITS) {
			auto kernel = dst_row_kernel<R, G::A, G::B>;
			const int n = row_lines<H>(a.sy, k);
			const int threads = (n * H::CNT + 31) / 32 * 32;
			const size_t sm = (size_t)(G::A * G::BP + (threads + H::CNT - 1) / H::CNT * H::LS) * G::ES;
			const long long tiles = (long long)k * ((a.sy + n - 1) / n);
			const int grid = grid_for(kernel, threads, sm, tiles);
			kernel<<<grid, threads, sm, s>>>(a, k, n);
			ran = true;
		}
	});
	return ran;
}

template <class R>
bool launch_dst_col(const ColPassArgs& a, int k, cudaStream_t s) {
	bool ran = false;
	for_length<R>(a.sy, [&](auto g) {
		using G = decltype(g);
		using H = Sine<G>;
		if constexpr (H::FITS) {
			auto kernel = dst_col_kernel<R, G::A, G::B>;
			const size_t sm = (size_t)G::N * (1 + G::W) * G::ES;
			const long long tiles = (long long)k * ((a.sx + G::W - 1) / G::W);
			const int grid = grid_for(kernel, H::COL_THREADS, sm, tiles);
			kernel<<<grid, H::COL_THREADS, sm, s>>>(a, k);
			ran = true;
		}
	});
	return ran;
}

}  // namespace lines

}  // namespace itp2d
