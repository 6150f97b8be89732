// Line transforms of N = A * B points in two register stages, and the row,
// column and energy passes built on them.
//
// With n = b + B a and k = k1 + A k2 the DFT of a line factors into
//   Y[b][k1]     = sum_a x[b + B a] w_A^(a k1)        B transforms of length A
//   X[k1 + A k2] = sum_b Y[b][k1] w_N^(b k1) w_B^(b k2)  A transforms of length B
// An "alpha" item b holds the A points b + B a, a "beta" item k1 the B points
// k1 + A k2, both in the registers of one thread; the twiddled values pass
// between them through shared memory at [k1][b]. The inverse transform runs
// the stages the other way round (beta items first), so it starts from the
// points a forward transform ends with: forward, table and inverse (a column
// pass) chain as alpha, beta, alpha, and inverse, table and forward (a row
// pass) as beta, alpha, beta. A chain of two transforms crosses shared memory
// twice, global memory is read and written straight from the registers, and A
// need not be a power of two or a multiple of B: every length with both factors
// among the register transforms below works, where the passes of split.cu
// (Stockham in shared memory, one trip per radix-8 stage) took 59 us for a
// pass over 77 FP32 states of 192 x 160 and these take 9 to 11 us.
//
// Same arithmetic contract as the passes in split.cu: unnormalised transforms
// with FFTW's sign convention (forward exp(-2 pi i jk/N)), tables applied as in
// RowPassArgs / ColPassArgs.
#pragma once

#include "launch.cuh"
#include "split.cuh"

#include <algorithm>
#include <type_traits>
#include <utility>

namespace itp2d {

namespace lines {

// cos and sin of 2 pi j / M, j = 0 .. M - 1, rounded to double.
template <int M> struct Roots;
// clang-format off
template <> struct Roots<3> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[3] = {
				1.0, -0.5, -0.5};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[3] = {
				0.0, 0.8660254037844386, -0.8660254037844386};
		return t[j];
	}
};
template <> struct Roots<5> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[5] = {
				1.0, 0.30901699437494745, -0.8090169943749475, -0.8090169943749475, 0.30901699437494745};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[5] = {
				0.0, 0.9510565162951535, 0.5877852522924731, -0.5877852522924731, -0.9510565162951535};
		return t[j];
	}
};
template <> struct Roots<6> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[6] = {
				1.0, 0.5, -0.5, -1.0, -0.5, 0.5};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[6] = {
				0.0, 0.8660254037844386, 0.8660254037844386, 0.0, -0.8660254037844386, -0.8660254037844386};
		return t[j];
	}
};
template <> struct Roots<8> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[8] = {
				1.0, 0.7071067811865476, 0.0, -0.7071067811865476, -1.0, -0.7071067811865476, 0.0, 0.7071067811865476};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[8] = {
				0.0, 0.7071067811865476, 1.0, 0.7071067811865476, 0.0, -0.7071067811865476, -1.0, -0.7071067811865476};
		return t[j];
	}
};
template <> struct Roots<9> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[9] = {
				1.0, 0.766044443118978, 0.17364817766693036, -0.5, -0.9396926207859084, -0.9396926207859084, -0.5,
				0.17364817766693036, 0.766044443118978};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[9] = {
				0.0, 0.6427876096865394, 0.984807753012208, 0.8660254037844386, 0.3420201433256687, -0.3420201433256687,
				-0.8660254037844386, -0.984807753012208, -0.6427876096865394};
		return t[j];
	}
};
template <> struct Roots<10> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[10] = {
				1.0, 0.8090169943749475, 0.30901699437494745, -0.30901699437494745, -0.8090169943749475, -1.0,
				-0.8090169943749475, -0.30901699437494745, 0.30901699437494745, 0.8090169943749475};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[10] = {
				0.0, 0.5877852522924731, 0.9510565162951535, 0.9510565162951535, 0.5877852522924731, 0.0,
				-0.5877852522924731, -0.9510565162951535, -0.9510565162951535, -0.5877852522924731};
		return t[j];
	}
};
template <> struct Roots<12> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[12] = {
				1.0, 0.8660254037844386, 0.5, 0.0, -0.5, -0.8660254037844386, -1.0, -0.8660254037844386, -0.5, 0.0, 0.5,
				0.8660254037844386};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[12] = {
				0.0, 0.5, 0.8660254037844386, 1.0, 0.8660254037844386, 0.5, 0.0, -0.5, -0.8660254037844386, -1.0,
				-0.8660254037844386, -0.5};
		return t[j];
	}
};
template <> struct Roots<15> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[15] = {
				1.0, 0.9135454576426009, 0.6691306063588582, 0.30901699437494745, -0.10452846326765347, -0.5,
				-0.8090169943749475, -0.9781476007338057, -0.9781476007338057, -0.8090169943749475, -0.5,
				-0.10452846326765347, 0.30901699437494745, 0.6691306063588582, 0.9135454576426009};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[15] = {
				0.0, 0.4067366430758002, 0.7431448254773942, 0.9510565162951535, 0.9945218953682733, 0.8660254037844386,
				0.5877852522924731, 0.20791169081775934, -0.20791169081775934, -0.5877852522924731, -0.8660254037844386,
				-0.9945218953682733, -0.9510565162951535, -0.7431448254773942, -0.4067366430758002};
		return t[j];
	}
};
template <> struct Roots<16> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[16] = {
				1.0, 0.9238795325112867, 0.7071067811865476, 0.3826834323650898, 0.0, -0.3826834323650898,
				-0.7071067811865476, -0.9238795325112867, -1.0, -0.9238795325112867, -0.7071067811865476,
				-0.3826834323650898, 0.0, 0.3826834323650898, 0.7071067811865476, 0.9238795325112867};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[16] = {
				0.0, 0.3826834323650898, 0.7071067811865476, 0.9238795325112867, 1.0, 0.9238795325112867,
				0.7071067811865476, 0.3826834323650898, 0.0, -0.3826834323650898, -0.7071067811865476, -0.9238795325112867,
				-1.0, -0.9238795325112867, -0.7071067811865476, -0.3826834323650898};
		return t[j];
	}
};
template <> struct Roots<18> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[18] = {
				1.0, 0.9396926207859084, 0.766044443118978, 0.5, 0.17364817766693036, -0.17364817766693036, -0.5,
				-0.766044443118978, -0.9396926207859084, -1.0, -0.9396926207859084, -0.766044443118978, -0.5,
				-0.17364817766693036, 0.17364817766693036, 0.5, 0.766044443118978, 0.9396926207859084};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[18] = {
				0.0, 0.3420201433256687, 0.6427876096865394, 0.8660254037844386, 0.984807753012208, 0.984807753012208,
				0.8660254037844386, 0.6427876096865394, 0.3420201433256687, 0.0, -0.3420201433256687, -0.6427876096865394,
				-0.8660254037844386, -0.984807753012208, -0.984807753012208, -0.8660254037844386, -0.6427876096865394,
				-0.3420201433256687};
		return t[j];
	}
};
template <> struct Roots<20> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[20] = {
				1.0, 0.9510565162951535, 0.8090169943749475, 0.5877852522924731, 0.30901699437494745, 0.0,
				-0.30901699437494745, -0.5877852522924731, -0.8090169943749475, -0.9510565162951535, -1.0,
				-0.9510565162951535, -0.8090169943749475, -0.5877852522924731, -0.30901699437494745, 0.0,
				0.30901699437494745, 0.5877852522924731, 0.8090169943749475, 0.9510565162951535};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[20] = {
				0.0, 0.30901699437494745, 0.5877852522924731, 0.8090169943749475, 0.9510565162951535, 1.0,
				0.9510565162951535, 0.8090169943749475, 0.5877852522924731, 0.30901699437494745, 0.0, -0.30901699437494745,
				-0.5877852522924731, -0.8090169943749475, -0.9510565162951535, -1.0, -0.9510565162951535,
				-0.8090169943749475, -0.5877852522924731, -0.30901699437494745};
		return t[j];
	}
};
template <> struct Roots<24> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[24] = {
				1.0, 0.9659258262890683, 0.8660254037844386, 0.7071067811865476, 0.5, 0.25881904510252074, 0.0,
				-0.25881904510252074, -0.5, -0.7071067811865476, -0.8660254037844386, -0.9659258262890683, -1.0,
				-0.9659258262890683, -0.8660254037844386, -0.7071067811865476, -0.5, -0.25881904510252074, 0.0,
				0.25881904510252074, 0.5, 0.7071067811865476, 0.8660254037844386, 0.9659258262890683};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[24] = {
				0.0, 0.25881904510252074, 0.5, 0.7071067811865476, 0.8660254037844386, 0.9659258262890683, 1.0,
				0.9659258262890683, 0.8660254037844386, 0.7071067811865476, 0.5, 0.25881904510252074, 0.0,
				-0.25881904510252074, -0.5, -0.7071067811865476, -0.8660254037844386, -0.9659258262890683, -1.0,
				-0.9659258262890683, -0.8660254037844386, -0.7071067811865476, -0.5, -0.25881904510252074};
		return t[j];
	}
};
template <> struct Roots<25> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[25] = {
				1.0, 0.9685831611286311, 0.8763066800438636, 0.7289686274214116, 0.5358267949789967, 0.30901699437494745,
				0.06279051952931337, -0.18738131458572463, -0.42577929156507266, -0.6374239897486897, -0.8090169943749475,
				-0.9297764858882515, -0.9921147013144779, -0.9921147013144779, -0.9297764858882515, -0.8090169943749475,
				-0.6374239897486897, -0.42577929156507266, -0.18738131458572463, 0.06279051952931337, 0.30901699437494745,
				0.5358267949789967, 0.7289686274214116, 0.8763066800438636, 0.9685831611286311};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[25] = {
				0.0, 0.2486898871648548, 0.48175367410171527, 0.6845471059286887, 0.8443279255020151, 0.9510565162951535,
				0.9980267284282716, 0.9822872507286887, 0.9048270524660196, 0.7705132427757893, 0.5877852522924731,
				0.368124552684678, 0.12533323356430426, -0.12533323356430426, -0.368124552684678, -0.5877852522924731,
				-0.7705132427757893, -0.9048270524660196, -0.9822872507286887, -0.9980267284282716, -0.9510565162951535,
				-0.8443279255020151, -0.6845471059286887, -0.48175367410171527, -0.2486898871648548};
		return t[j];
	}
};
template <> struct Roots<32> {
	static constexpr __host__ __device__ double c(int j) {
		constexpr double t[32] = {
				1.0, 0.9807852804032304, 0.9238795325112867, 0.8314696123025452, 0.7071067811865476, 0.5555702330196022,
				0.3826834323650898, 0.19509032201612828, 0.0, -0.19509032201612828, -0.3826834323650898,
				-0.5555702330196022, -0.7071067811865476, -0.8314696123025452, -0.9238795325112867, -0.9807852804032304,
				-1.0, -0.9807852804032304, -0.9238795325112867, -0.8314696123025452, -0.7071067811865476,
				-0.5555702330196022, -0.3826834323650898, -0.19509032201612828, 0.0, 0.19509032201612828,
				0.3826834323650898, 0.5555702330196022, 0.7071067811865476, 0.8314696123025452, 0.9238795325112867,
				0.9807852804032304};
		return t[j];
	}
	static constexpr __host__ __device__ double s(int j) {
		constexpr double t[32] = {
				0.0, 0.19509032201612828, 0.3826834323650898, 0.5555702330196022, 0.7071067811865476, 0.8314696123025452,
				0.9238795325112867, 0.9807852804032304, 1.0, 0.9807852804032304, 0.9238795325112867, 0.8314696123025452,
				0.7071067811865476, 0.5555702330196022, 0.3826834323650898, 0.19509032201612828, 0.0, -0.19509032201612828,
				-0.3826834323650898, -0.5555702330196022, -0.7071067811865476, -0.8314696123025452, -0.9238795325112867,
				-0.9807852804032304, -1.0, -0.9807852804032304, -0.9238795325112867, -0.8314696123025452,
				-0.7071067811865476, -0.5555702330196022, -0.3826834323650898, -0.19509032201612828};
		return t[j];
	}
};
// clang-format on

// Compile-time loop: f(std::integral_constant<int, I>) for I = 0 .. N-1, so
// that register-array indices inside f are constants.
template <class F, int... I>
__device__ __forceinline__ void sfor_impl(F&& f, std::integer_sequence<int, I...>) {
	(f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void sfor(F&& f) {
	sfor_impl(f, std::make_integer_sequence<int, N>{});
}

// Complex sums and real multiples; FP32 pairs use the packed instructions
// (one issue slot for both parts).
__device__ __forceinline__ float2 f2_of(unsigned long long v) {
	float2 r;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
	return r;
}
__device__ __forceinline__ unsigned long long u_of(float2 v) {
	unsigned long long r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
	return r;
}
__device__ __forceinline__ double2 add(double2 a, double2 b) { return cadd(a, b); }
__device__ __forceinline__ double2 sub(double2 a, double2 b) { return csub(a, b); }
__device__ __forceinline__ double2 scale(double2 a, double s) { return cscale(a, s); }
__device__ __forceinline__ float2 add(float2 a, float2 b) {
	unsigned long long r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(u_of(a)), "l"(u_of(b)));
	return f2_of(r);
}
__device__ __forceinline__ float2 sub(float2 a, float2 b) {
	unsigned long long r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(u_of(b)), "l"(u_of(make_float2(-1.0f, -1.0f))), "l"(u_of(a)));
	return f2_of(r);
}
__device__ __forceinline__ float2 scale(float2 a, float s) {
	unsigned long long r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(u_of(a)), "l"(u_of(make_float2(s, s))));
	return f2_of(r);
}
// a + SIGN i b
template <int SIGN, class T>
__device__ __forceinline__ T add_i(T a, T b) {
	T r;
	if (SIGN > 0) {
		r.x = a.x - b.y;
		r.y = a.y + b.x;
	} else {
		r.x = a.x + b.y;
		r.y = a.y - b.x;
	}
	return r;
}

// First factor of a composite register transform.
constexpr int first_factor(int m) {
	return m == 6 || m == 8 || m == 10 || m == 18 ? 2 : m == 9 || m == 15 || m == 24 ? 3 : m % 4 == 0 ? 4 : 5;
}

// DFT of v[0..M) in place, natural order in and out:
// v[k] = sum_j v[j] exp(SIGN 2 pi i jk / M).
template <class R, int M, int SIGN>
__device__ __forceinline__ void dft(c2<R>* v) {
	using T = c2<R>;
	if constexpr (M == 2) {
		const T a = v[0], b = v[1];
		v[0] = add(a, b);
		v[1] = sub(a, b);
	} else if constexpr (M == 3) {
		constexpr R s3 = (R)0.86602540378443864676;
		const T s = add(v[1], v[2]), d = scale(sub(v[1], v[2]), s3);
		const T m = add(v[0], scale(s, (R)-0.5));
		v[0] = add(v[0], s);
		v[1] = add_i<SIGN>(m, d);
		v[2] = add_i<-SIGN>(m, d);
	} else if constexpr (M == 4) {
		const T t0 = add(v[0], v[2]), t1 = sub(v[0], v[2]), t2 = add(v[1], v[3]), t3 = sub(v[1], v[3]);
		v[0] = add(t0, t2);
		v[1] = add_i<SIGN>(t1, t3);
		v[2] = sub(t0, t2);
		v[3] = add_i<-SIGN>(t1, t3);
	} else if constexpr (M == 5) {
		constexpr R c1 = (R)Roots<5>::c(1), c2_ = (R)Roots<5>::c(2), s1 = (R)Roots<5>::s(1), s2 = (R)Roots<5>::s(2);
		const T a1 = add(v[1], v[4]), b1 = sub(v[1], v[4]), a2 = add(v[2], v[3]), b2 = sub(v[2], v[3]);
		const T m1 = add(v[0], add(scale(a1, c1), scale(a2, c2_)));
		const T m2 = add(v[0], add(scale(a1, c2_), scale(a2, c1)));
		const T d1 = add(scale(b1, s1), scale(b2, s2)), d2 = sub(scale(b1, s2), scale(b2, s1));
		v[0] = add(v[0], add(a1, a2));
		v[1] = add_i<SIGN>(m1, d1);
		v[4] = add_i<-SIGN>(m1, d1);
		v[2] = add_i<SIGN>(m2, d2);
		v[3] = add_i<-SIGN>(m2, d2);
	} else {
		constexpr int P = first_factor(M), Q = M / P;
		T t[M];
		sfor<P>([&](auto q) { sfor<Q>([&](auto i) { t[q * Q + i] = v[P * i + q]; }); });
		sfor<P>([&](auto q) { dft<R, Q, SIGN>(t + q * Q); });
		sfor<Q>([&](auto i) {
			T u[P];
			sfor<P>([&](auto q) {
				constexpr int e = (q * i) % M;
				const T x = t[q * Q + i];
				if constexpr (e == 0) {
					u[q] = x;
				} else if constexpr (4 * e == M) {
					u[q] = cmul_i(x, SIGN);
				} else {
					constexpr R wr = (R)Roots<M>::c(e), wi = (R)(SIGN * Roots<M>::s(e));
					u[q] = cmul(x, mk<R>(wr, wi));
				}
			});
			dft<R, P, SIGN>(u);
			sfor<P>([&](auto k) { v[i + Q * k] = u[k]; });
		});
	}
}

// v[j] *= w_N^(SIGN-signed) [table of forward twiddles, element j at tw[j * ST]], j >= 1.
template <class R, int M, int SIGN, int ST>
__device__ __forceinline__ void twiddle(c2<R>* v, const c2<R>* tw) {
	sfor<M - 1>([&](auto K) {
		constexpr int j = K + 1;
		const c2<R> w = tw[j * ST];
		v[j] = SIGN < 0 ? cmul(v[j], w) : cmulc(v[j], w);
	});
}

// Keeps the loads that follow after the transform that gave v, where v fills
// the registers (FP64, 32 points): hoisted loads would spill.
template <class T, int M>
__device__ __forceinline__ void pin(T* v) {
	if constexpr (sizeof(T) * M >= 512) {
#pragma unroll
		for (int j = 0; j < M; j++) asm volatile("" : "+d"(v[j].x), "+d"(v[j].y)::"memory");
	}
}

// v[j] *= table[at(j)], M elements; long FP64 lines take the table in chunks of
// eight (all loads at once would not fit in registers beside the points).
template <class T, int M, class R, class AT>
__device__ __forceinline__ void times(T* v, const R* table, AT&& at) {
	pin<T, M>(v);
#pragma unroll
	for (int j = 0; j < M; j++) {
		v[j] = scale(v[j], table[at(j)]);
		if (sizeof(T) * M >= 512 && j % 8 == 7) asm volatile("" ::: "memory");
	}
}

// Geometry of lines of N = A * B points in precision R.
template <class R, int A_, int B_>
struct Geo {
	static constexpr int A = A_, B = B_, N = A * B;
	static constexpr int ES = (int)sizeof(c2<R>);
	// threads per line: one per beta item (A), or one per alpha item (B) where
	// that at most halves them (each then takes two beta items)
	static constexpr int CNT = A >= 2 * B ? B : A;
	static constexpr int NB = (A + CNT - 1) / CNT;  // beta items per thread
	// columns per tile: 128 bytes of a row
	static constexpr int W = 128 / ES;
	static constexpr int COL_THREADS = (CNT * W + 31) / 32 * 32;  // whole warps; the last may idle in part
	static constexpr int ROW_THREADS = ES == 16 ? 128 : 256;
	// row exchange area: [k1][b], rows padded to an odd length (conflict-free
	// across both b and k1); lines 8 elements apart modulo 16 where two share a
	// half-warp
	static constexpr int BP = B | 1;
	static constexpr int LS = CNT == 8 ? (A * BP + 15) / 16 * 16 + 8 : A * BP;
	static constexpr bool WARP_LINE = 32 % CNT == 0;  // a line stays inside one warp
	// CTAs per SM for the launch bounds, from the registers a thread needs: its
	// points, their copies in the transforms, addresses (`extra`: what a kernel
	// needs beyond the column pass)
	static constexpr int blocks(int threads, int extra = 0) {
		const int regs = (ES / 4) * A + (ES == 16 ? 56 : 40) + extra;
		const int n = 65536 / (threads * ((regs + 7) / 8 * 8));
		return n < 1 ? 1 : n;
	}
	static constexpr int ROW_BLOCKS = blocks(ROW_THREADS, ES == 16 ? 24 : 0);
	static constexpr int COL_BLOCKS = blocks(COL_THREADS);
	static constexpr int ENERGY_ROW_BLOCKS = blocks(ROW_THREADS, ES == 16 ? 32 : 16);
	static constexpr int ENERGY_COL_BLOCKS = blocks(COL_THREADS, ES == 16 ? 40 : 16);
};

// Forward twiddles w_N^(b k1) at [k1 * LD + b]; tw[ST j] = w_N^j.
template <class R, class G, int LD, int ST = 1>
__device__ __forceinline__ void load_tw(c2<R>* xtw, const void* tw) {
	const c2<R>* g = reinterpret_cast<const c2<R>*>(tw);
	for (int i = threadIdx.x; i < G::N; i += blockDim.x) {
		const int k1 = i / G::B, b = i - k1 * G::B;
		xtw[k1 * LD + b] = g[ST * b * k1];  // b k1 < N
	}
}

// Barrier between the stages of the lines of one CTA.
template <class G>
__device__ __forceinline__ void stage_sync() {
	if constexpr (G::WARP_LINE) __syncwarp();
	else __syncthreads();
}

// Row pass (RowPassArgs): `lines` rows of one state per tile, tiles ordered
// state-fastest, persistent. A pass with one transform is HBM-bound (5.8 to 6
// TB/s from 256 points on, FP32 and FP64), one with two is bound by latency at
// 16 warps per SM (4.1 TB/s at 512 FP32 points; the registers of a thread's 32
// points set the occupancy). Small CTAs (128 threads FP64, 256 FP32): several per
// SM overlap their loads, transforms and stores.
template <class R, int A, int B>
__global__ void __launch_bounds__((Geo<R, A, B>::ROW_THREADS), (Geo<R, A, B>::ROW_BLOCKS))
		row_kernel(RowPassArgs a, int k, int lines) {
	using G = Geo<R, A, B>;
	using T = c2<R>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	T* xtw = reinterpret_cast<T*>(smem_raw);
	load_tw<R, G, G::BP>(xtw, a.lp.fft.tw);
	__syncthreads();
	const int line = threadIdx.x / G::CNT, t = threadIdx.x - line * G::CNT;
	T* E = xtw + A * G::BP + line * G::LS;
	const bool alpha = G::CNT == B || t < B;
	const int sx = a.sx;
	const int ntr = (a.sy + lines - 1) / lines;
	const long long total = (long long)k * ntr;
	const R* mpre = reinterpret_cast<const R*>(a.mul_pre);
	const R* mmid = reinterpret_cast<const R*>(a.mul_mid);
	const R* mpost = reinterpret_cast<const R*>(a.mul_post);
	const T* in = reinterpret_cast<const T*>(a.in);
	T* out = reinterpret_cast<T*>(a.out);
	const T* acc = reinterpret_cast<const T*>(a.acc);
	for (long long tile = blockIdx.x; tile < total; tile += gridDim.x) {
		const long long state = tile % k;
		const int y = (int)(tile / k) * lines + line;
		const bool valid = line < lines && y < a.sy;
		const long long base = state * a.G + (long long)y * sx;
		const int toff = y * sx;
		if (a.do_inv) {
#pragma unroll
			for (int i = 0; i < G::NB; i++) {
				const int k1 = t + G::CNT * i;
				if (valid && (A % G::CNT == 0 || k1 < A)) {
					T u[B];
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = in[base + k1 + A * j];
					if (mpre) times<T, B>(u, mpre + toff + k1, [](int j) { return A * j; });
					dft<R, B, 1>(u);
					twiddle<R, B, 1, 1>(u, xtw + k1 * G::BP);
#pragma unroll
					for (int j = 0; j < B; j++) E[k1 * G::BP + j] = u[j];
				}
			}
			stage_sync<G>();
		}
		if (valid && alpha) {
			T v[A];
			if (a.do_inv) {
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = E[j * G::BP + t];
				dft<R, A, 1>(v);
			} else {
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = in[base + t + B * j];
			}
			if (mmid) times<T, A>(v, mmid + toff + t, [](int j) { return B * j; });
			if (a.do_fwd) {
				dft<R, A, -1>(v);
				twiddle<R, A, -1, G::BP>(v, xtw + t);
#pragma unroll
				for (int j = 0; j < A; j++) E[j * G::BP + t] = v[j];
			} else {
				if (acc) {
					pin<T, A>(v);
#pragma unroll
					for (int j = 0; j < A; j++) v[j] = add(v[j], acc[base + t + B * j]);
				}
#pragma unroll
				for (int j = 0; j < A; j++) out[base + t + B * j] = v[j];
			}
		}
		stage_sync<G>();
		if (!a.do_fwd) continue;
#pragma unroll
		for (int i = 0; i < G::NB; i++) {
			const int k1 = t + G::CNT * i;
			if (valid && (A % G::CNT == 0 || k1 < A)) {
				T u[B];
#pragma unroll
				for (int j = 0; j < B; j++) u[j] = E[k1 * G::BP + j];
				dft<R, B, -1>(u);
				if (mpost) times<T, B>(u, mpost + toff + k1, [](int j) { return A * j; });
				if (acc) {
					pin<T, B>(u);
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = add(u[j], acc[base + k1 + A * j]);
				}
#pragma unroll
				for (int j = 0; j < B; j++) out[base + k1 + A * j] = u[j];
			}
		}
		// the next tile's inverse transform writes what the same thread read; a
		// forward one alone writes other threads' values
		if (!a.do_inv) stage_sync<G>();
	}
}

// Column pass (ColPassArgs), in place: tiles of W columns (128 bytes) x N rows
// of one state; thread (t, c) of a tile works on column c, so every global
// access of a warp covers whole 128-byte row segments, and the exchange area
// [k1][b][column] has no bank conflicts. No staging of the tile in shared memory
// (eight accesses per point before, four now): 60 instructions per point at 512
// FP32 points against 120, 541 -> 287 us for 256 states of 512 x 512 (FP64,
// 256 x 256 x 300: 177 -> 128 us). 64-byte strips (twice the CTAs, half the
// size) were slower: 4.2 against 5.7 TB/s at 256 FP64 points. Bringing the next
// tile in by cp.async during the last stage, or whole tiles by TMA through a
// three-slot ring, did not pay either (FP64, 512 x 512 x 300: propagation
// 4.24 ms here, 5.60 and 5.30 ms): the second and third CTA of an SM hide as much.
template <class R, int A, int B>
__global__ void __launch_bounds__((Geo<R, A, B>::COL_THREADS), (Geo<R, A, B>::COL_BLOCKS))
		col_kernel(ColPassArgs a, int k) {
	using G = Geo<R, A, B>;
	using T = c2<R>;
	constexpr int W = G::W;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	T* xtw = reinterpret_cast<T*>(smem_raw);
	load_tw<R, G, B>(xtw, a.lp.fft.tw);
	__syncthreads();
	const int t = threadIdx.x / W, c = threadIdx.x % W;
	T* E = xtw + G::N + c;
	const bool alpha = G::CNT == B || t < B;
	const bool on = G::COL_THREADS == G::CNT * W || t < G::CNT;
	const int sx = a.sx;
	const int nct = (sx + W - 1) / W;
	const long long total = (long long)k * nct;
	const R* m2 = reinterpret_cast<const R*>(a.mul2d);
	const R* m1 = reinterpret_cast<const R*>(a.mul1d);
	for (long long tile = blockIdx.x; tile < total; tile += gridDim.x) {
		const int col = (int)(tile % nct) * W + c;
		const bool valid = on && col < sx;
		T* data = reinterpret_cast<T*>(a.data) + (tile / nct) * a.G + col;
		if (a.mode != 2) {
			if (valid && alpha) {
				T v[A];
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = data[(t + B * j) * sx];
				dft<R, A, -1>(v);
				twiddle<R, A, -1, B>(v, xtw + t);
#pragma unroll
				for (int j = 0; j < A; j++) E[(j * B + t) * W] = v[j];
			}
			__syncthreads();
		}
#pragma unroll
		for (int i = 0; i < G::NB; i++) {
			const int k1 = t + G::CNT * i;
			if (valid && (A % G::CNT == 0 || k1 < A)) {
				T u[B];
				if (a.mode != 2) {
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = E[(k1 * B + j) * W];
					dft<R, B, -1>(u);
					if (a.mode == 1) {
#pragma unroll
						for (int j = 0; j < B; j++) data[(k1 + A * j) * sx] = u[j];
						continue;
					}
					if (m2) {
#pragma unroll
						for (int j = 0; j < B; j++) u[j] = scale(u[j], m2[(k1 + A * j) * sx + col]);
					} else {
#pragma unroll
						for (int j = 0; j < B; j++) u[j] = scale(u[j], m1[k1 + A * j]);
					}
				} else {
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = data[(k1 + A * j) * sx];
				}
				dft<R, B, 1>(u);
				twiddle<R, B, 1, 1>(u, xtw + k1 * B);
#pragma unroll
				for (int j = 0; j < B; j++) E[(k1 * B + j) * W] = u[j];
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
			for (int j = 0; j < A; j++) data[(t + B * j) * sx] = v[j];
		}
		// mode 0: the next tile's first stage writes what the same thread read
		if (a.mode == 2) __syncthreads();
	}
}

// Energy sums of one element: Re, Im <psi|h>, <h|h>, |h - es psi|^2, <psi|psi>.
template <class T>
__device__ __forceinline__ void esums(double* s, T p, T h, double es) {
	const double pr = p.x, pi = p.y, hr = h.x, hi = h.y;
	s[0] += pr * hr + pi * hi;
	s[1] += pr * hi - pi * hr;
	s[2] += hr * hr + hi * hi;
	const double dr = hr - es * pr, di = hi - es * pi;
	s[3] += dr * dr + di * di;
	s[4] += pr * pr + pi * pi;
}

// Deterministic CTA reduction of the five sums into out[0..5) (threads 0-4);
// red holds 5 doubles per warp. Ends with every warp past its use of red.
__device__ __forceinline__ void reduce5(double* s, double* red, double* out) {
	// (whole warps: the launches round the block size up)
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
	for (int j = 0; j < 5; j++)
		for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
	if (lane == 0)
		for (int j = 0; j < 5; j++) red[warp * 5 + j] = s[j];
	__syncthreads();
	if (threadIdx.x < 5) {
		double v = 0.0;
		for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += red[w * 5 + threadIdx.x];
		out[threadIdx.x] = v;
	}
	__syncthreads();
}

// The elements an alpha item leaves, h = v + add, add = V psi (row pass) or the
// row pass's part (column pass), written to hout and summed against psi. at(j):
// offset of element j; the loads of eight elements are issued together.
template <class R, int A, class AT, class ADD>
__device__ __forceinline__ void energy_tail(c2<R>* v, const c2<R>* psi, c2<R>* hout, bool sums, double es, double* s,
		AT&& at, ADD&& add_of) {
	using T = c2<R>;
	constexpr int EB = 8;
#pragma unroll
	for (int b0 = 0; b0 < A; b0 += EB) {
		T p[EB];
#pragma unroll
		for (int e = 0; e < EB; e++)
			if (b0 + e < A) p[e] = psi[at(b0 + e)];
#pragma unroll
		for (int e = 0; e < EB; e++)
			if (b0 + e < A) v[b0 + e] = add(v[b0 + e], add_of(b0 + e, p[e]));
#pragma unroll
		for (int e = 0; e < EB; e++)
			if (b0 + e < A) {
				if (hout) hout[at(b0 + e)] = v[b0 + e];
				if (sums) esums(s, p[e], v[b0 + e], es);
			}
	}
}

// Energy row pass (EnergyRowArgs): `rows_per_tile` rows of one state per tile,
// sums at [(state * ntiles + tile) * 5]. Persistent, so several CTAs per SM
// keep loads in flight while others transform.
template <class R, int A, int B>
__global__ void __launch_bounds__((Geo<R, A, B>::ROW_THREADS), (Geo<R, A, B>::ENERGY_ROW_BLOCKS))
		energy_row_kernel(EnergyRowArgs a, int k) {
	using G = Geo<R, A, B>;
	using T = c2<R>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	double* red = reinterpret_cast<double*>(smem_raw);  // 5 per warp of 256 threads
	T* xtw = reinterpret_cast<T*>(smem_raw + 5 * 8 * sizeof(double));
	load_tw<R, G, G::BP>(xtw, a.lp.fft.tw);
	__syncthreads();
	const int lines = a.rows_per_tile;
	const int line = threadIdx.x / G::CNT, t = threadIdx.x - line * G::CNT;
	T* E = xtw + A * G::BP + line * G::LS;
	const bool alpha = G::CNT == B || t < B;
	const int sx = a.sx;
	const int ntr = (a.sy + lines - 1) / lines;
	const long long total = (long long)k * ntr;
	const T* src = reinterpret_cast<const T*>(a.src_t);
	const R* tm = reinterpret_cast<const R*>(a.tmul);
	const R* V = reinterpret_cast<const R*>(a.V);
	for (long long tile = blockIdx.x; tile < total; tile += gridDim.x) {
		const long long state = tile % k;
		const int tr = (int)(tile / k);
		const int y = tr * lines + line;
		const bool valid = line < lines && y < a.sy;
		const long long base = state * a.G + (long long)y * sx;
		const int toff = y * sx;
		T v[A];
		if (a.do_fwd) {
			if (valid && alpha) {
#pragma unroll
				for (int j = 0; j < A; j++) v[j] = src[base + t + B * j];
				dft<R, A, -1>(v);
				twiddle<R, A, -1, G::BP>(v, xtw + t);
#pragma unroll
				for (int j = 0; j < A; j++) E[j * G::BP + t] = v[j];
			}
			stage_sync<G>();
		}
#pragma unroll
		for (int i = 0; i < G::NB; i++) {
			const int k1 = t + G::CNT * i;
			if (valid && (A % G::CNT == 0 || k1 < A)) {
				T u[B];
				if (a.do_fwd) {
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = E[k1 * G::BP + j];
					dft<R, B, -1>(u);
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = scale(u[j], tm[toff + k1 + A * j]);
				} else {
#pragma unroll
					for (int j = 0; j < B; j++) u[j] = src[base + k1 + A * j];
				}
				dft<R, B, 1>(u);
				twiddle<R, B, 1, 1>(u, xtw + k1 * G::BP);
#pragma unroll
				for (int j = 0; j < B; j++) E[k1 * G::BP + j] = u[j];
			}
		}
		stage_sync<G>();
		double s[5] = {0, 0, 0, 0, 0};
		if (valid && alpha) {
#pragma unroll
			for (int j = 0; j < A; j++) v[j] = E[j * G::BP + t];
			dft<R, A, 1>(v);
			T* hout = a.h_out ? reinterpret_cast<T*>(a.h_out) + base : nullptr;
			energy_tail<R, A>(
					v, reinterpret_cast<const T*>(a.psi) + base, hout, a.sums != nullptr, a.Eshift ? a.Eshift[state] : 0.0, s,
					[&](int j) { return t + B * j; },
					[&](int j, T p) { return V ? scale(p, V[toff + t + B * j]) : mk<R>(0, 0); });
		}
		if (a.sums) reduce5(s, red, a.sums + ((size_t)state * ntr + tr) * 5);
		else stage_sync<G>();  // the exchange area has been read
	}
}

// Energy column pass (EnergyColArgs), tiles as in col_kernel.
template <class R, int A, int B>
__global__ void __launch_bounds__((Geo<R, A, B>::COL_THREADS), (Geo<R, A, B>::ENERGY_COL_BLOCKS))
		energy_col_kernel(EnergyColArgs a, int k) {
	using G = Geo<R, A, B>;
	using T = c2<R>;
	constexpr int W = G::W;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	double* red = reinterpret_cast<double*>(smem_raw);  // 5 per warp of at most 512 threads
	T* xtw = reinterpret_cast<T*>(smem_raw + 5 * 16 * sizeof(double));
	load_tw<R, G, B>(xtw, a.lp.fft.tw);
	__syncthreads();
	const int t = threadIdx.x / W, c = threadIdx.x % W;
	T* E = xtw + G::N + c;
	const bool alpha = G::CNT == B || t < B;
	const bool on = G::COL_THREADS == G::CNT * W || t < G::CNT;
	const int sx = a.sx;
	const int nct = (sx + W - 1) / W;
	const long long total = (long long)k * nct;
	const R* ty = reinterpret_cast<const R*>(a.ty);
	const T* psi_all = reinterpret_cast<const T*>(a.psi);
	const T* src_all = a.src ? reinterpret_cast<const T*>(a.src) : psi_all;
	for (long long tile = blockIdx.x; tile < total; tile += gridDim.x) {
		const long long state = tile / nct;
		const int ct = (int)(tile % nct);
		const int col = ct * W + c;
		const bool valid = on && col < sx;
		const long long base = state * a.G + col;
		T v[A];
		if (valid && alpha) {
			const T* src = src_all + base;
#pragma unroll
			for (int j = 0; j < A; j++) v[j] = src[(t + B * j) * sx];
			dft<R, A, -1>(v);
			twiddle<R, A, -1, B>(v, xtw + t);
#pragma unroll
			for (int j = 0; j < A; j++) E[(j * B + t) * W] = v[j];
		}
		__syncthreads();
#pragma unroll
		for (int i = 0; i < G::NB; i++) {
			const int k1 = t + G::CNT * i;
			if (valid && (A % G::CNT == 0 || k1 < A)) {
				T u[B];
#pragma unroll
				for (int j = 0; j < B; j++) u[j] = E[(k1 * B + j) * W];
				dft<R, B, -1>(u);
#pragma unroll
				for (int j = 0; j < B; j++) u[j] = scale(u[j], ty[k1 + A * j]);
				dft<R, B, 1>(u);
				twiddle<R, B, 1, 1>(u, xtw + k1 * B);
#pragma unroll
				for (int j = 0; j < B; j++) E[(k1 * B + j) * W] = u[j];
			}
		}
		__syncthreads();
		double s[5] = {0, 0, 0, 0, 0};
		if (valid && alpha) {
#pragma unroll
			for (int j = 0; j < A; j++) v[j] = E[(j * B + t) * W];
			dft<R, A, 1>(v);
			const T* more = reinterpret_cast<const T*>(a.add_in) + base;
			T* hout = a.h_out ? reinterpret_cast<T*>(a.h_out) + base : nullptr;
			energy_tail<R, A>(
					v, psi_all + base, hout, a.sums != nullptr, a.Eshift ? a.Eshift[state] : 0.0, s,
					[&](int j) { return (t + B * j) * sx; }, [&](int j, T) { return more[(t + B * j) * sx]; });
		}
		if (a.sums) reduce5(s, red, a.sums + ((size_t)state * nct + ct) * 5);
	}
}

// Persistent grid: as many CTAs as fit on the device, at most one per tile.
template <class K>
int grid_for(K kernel, int threads, size_t smem, long long tiles) {
	if (smem > 48 * 1024) raise_smem_limit((const void*)kernel);
	const long long resident = resident_ctas((const void*)kernel, threads, smem);
	return (int)std::max(1LL, std::min(resident * sm_count(), tiles));
}

// Rows per tile: a full CTA's worth, fewer where that leaves the device
// without two tiles per SM (down to one warp's worth).
template <class G>
int row_lines(int sy, int k) {
	const int most = std::min(G::ROW_THREADS / G::CNT, sy), least = std::max(1, std::min(most, 32 / G::CNT));
	const long long want = (long long)k * sy / (2 * sm_count());
	return (int)std::max<long long>(least, std::min<long long>(most, want));
}

// f(Geo) for a supported line length (both factors register transforms, the
// larger at most twice the smaller where one exists); false otherwise.
template <class R, class F>
bool for_length(int N, F&& f) {
#define ITP2D_LINE(n, a, b) \
	case n: f(Geo<R, a, b>{}); return true;
	switch (N) {
		ITP2D_LINE(32, 8, 4)
		ITP2D_LINE(36, 6, 6)
		ITP2D_LINE(40, 8, 5)
		ITP2D_LINE(48, 8, 6)
		ITP2D_LINE(60, 10, 6)
		ITP2D_LINE(64, 8, 8)
		ITP2D_LINE(72, 9, 8)
		ITP2D_LINE(80, 10, 8)
		ITP2D_LINE(90, 10, 9)
		ITP2D_LINE(96, 12, 8)
		ITP2D_LINE(100, 10, 10)
		ITP2D_LINE(108, 12, 9)
		ITP2D_LINE(120, 12, 10)
		ITP2D_LINE(128, 16, 8)
		ITP2D_LINE(144, 12, 12)
		ITP2D_LINE(150, 15, 10)
		ITP2D_LINE(160, 16, 10)
		ITP2D_LINE(180, 15, 12)
		ITP2D_LINE(192, 16, 12)
		ITP2D_LINE(200, 20, 10)
		ITP2D_LINE(216, 18, 12)
		ITP2D_LINE(240, 16, 15)
		ITP2D_LINE(256, 16, 16)
		ITP2D_LINE(288, 18, 16)
		ITP2D_LINE(300, 20, 15)
		ITP2D_LINE(320, 20, 16)
		ITP2D_LINE(360, 20, 18)
		ITP2D_LINE(384, 24, 16)
		ITP2D_LINE(400, 20, 20)
		ITP2D_LINE(432, 24, 18)
		ITP2D_LINE(480, 24, 20)
		ITP2D_LINE(500, 25, 20)
		ITP2D_LINE(512, 32, 16)
		ITP2D_LINE(576, 24, 24)
		ITP2D_LINE(640, 32, 20)
		ITP2D_LINE(768, 32, 24)
		ITP2D_LINE(1024, 32, 32)
		default: return false;
	}
#undef ITP2D_LINE
}

}  // namespace lines

}  // namespace itp2d
