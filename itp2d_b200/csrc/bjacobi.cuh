// What the block Jacobi eigensolvers share (bjacobi.cu in double, bjacobi32.cu in
// single precision): pairings, rotations, the sweep of a subproblem in shared
// memory and the items of phase 2. The method is described in bjacobi.cu.
#pragma once

#include "common.cuh"

namespace itp2d {

namespace bj {

constexpr int BS = 16;        // block size
constexpr int MS = 32;        // subproblem size: two blocks
constexpr int NR = MS / 2;    // rotations per inner round
constexpr int LDM = MS + 1;   // row length of M: conflict-free rows and columns
// 512 threads, one CTA per SM: an inner sweep gives its warps separate roles
// (inner_sweep).
constexpr int kThreads = 512;
// Rounds between full inner sweeps (within-block pairs rotated again); every
// 16th round measured best on k = 500 (fewer outer sweeps for little cost).
constexpr int kFullEvery = 16;

// Round-robin pairing of npos positions (circle method): position 0 fixed.
__device__ __forceinline__ int rr_player(int pos, int r, int npos) {
	const int v = pos - 1 + r;  // 0 <= r < npos - 1
	return pos == 0 ? 0 : (v >= npos - 1 ? v - npos + 2 : v + 1);
}

// Global index of local subproblem index i (< 32) for the block pair (P, Q).
__device__ __forceinline__ int gidx(int i, int P, int Q) { return i < BS ? P * BS + i : Q * BS + (i - BS); }

// Reciprocal and reciprocal square root in double precision by Newton-Raphson
// refinement of the single-precision hardware estimates: each step squares the
// relative error (about 1e-7 -> 1e-14 -> below double rounding). Valid for
// positive normal arguments inside the float exponent range, which the
// rotation set-up below guarantees by scaling.
__device__ __forceinline__ double rcp_nr(double x) {
	double y = (double)__frcp_rn((float)x);
	y = y * fma(-x, y, 2.0);
	y = y * fma(-x, y, 2.0);
	return y;
}
__device__ __forceinline__ double rsqrt_nr(double x) {
	double y = (double)rsqrtf((float)x);
	y = y * fma(-0.5 * x * y, y, 1.5);
	y = y * fma(-0.5 * x * y, y, 1.5);
	return y;
}

// A rotation in double precision throughout, for pairs whose exponents leave
// the range of the set-up below: with u = |d| + r and w = 2 r u, cos = u / sqrt(w),
// |sin| = |c| / sqrt(w) and |tau| = |c| / (sqrt(w) + u), d and c scaled by exact
// powers of two (scalbn: the power itself may leave the range where the values
// are subnormal). t: the tangent, 0 where |c| / sqrt(|a b|) is at most tol;
// counted: whether it is above noise; coarse: whether it is above 2^-26.
struct WideRotation {
	double s, tau, er, ei, t;
	bool counted, coarse;
};
static __device__ __noinline__ WideRotation rotation_wide(double a, double b, double cr, double ci, double tol,
		double noise) {
	WideRotation w;
	// the sizes without products of two elements
	const double c = hypot(cr, ci);
	const double scale = sqrt(fabs(a)) * sqrt(fabs(b));
	w.counted = c > noise * scale;
	w.coarse = c > 0x1p-26 * scale;
	w.s = w.tau = w.er = w.ei = w.t = 0.0;
	if (!(c > tol * scale)) return w;
	const double d = 0.5 * (b - a);
	const double ad = fabs(d);
	const double mc = fmax(fabs(cr), fabs(ci));
	const int ex = ilogb(fmax(ad, mc)), exc = ilogb(mc);
	const double dn = scalbn(ad, -ex), crn = scalbn(cr, -ex), cin = scalbn(ci, -ex);
	const double cn2 = crn * crn + cin * cin;
	const double rn2 = dn * dn + cn2;         // [1, 12)
	const double rn = rn2 * rsqrt_nr(rn2);
	const double un = dn + rn;                // [1, 5.5)
	const double wn = 2.0 * rn * un;          // [2, 38)
	const double qn = rsqrt_nr(wn);
	const double cn = sqrt(cn2);
	w.t = cn * rcp_nr(un);
	const double crs = scalbn(cr, -exc), cis = scalbn(ci, -exc);
	const double ec = rsqrt_nr(crs * crs + cis * cis);
	const double sg = d < 0 ? -1.0 : 1.0;
	w.s = sg * cn * qn;
	w.tau = sg * cn * rcp_nr(wn * qn + un);
	w.er = crs * ec;
	w.ei = cis * ec;
	return w;
}

__device__ __forceinline__ float rsqrt_approx(float x) {
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
	float y;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return y;
}

// Whether v >= 0 is between 2^-830 and 2^996 (single precision: 2^-73 and 2^122),
// by its exponent: squares of tol and noise times v stay normal numbers.
__device__ __forceinline__ bool well_inside(double v) {
	return (unsigned)__double2hiint(v) - 0x0C100000u < 0x7E300000u - 0x0C100000u;
}
__device__ __forceinline__ bool well_inside(float v) {
	return __float_as_uint(v) - 0x1B000000u < 0x7C800000u - 0x1B000000u;
}

// Whether c2 / scale2 is above about 2^-52, by exponents (2^-53 to 2^-51).
__device__ __forceinline__ bool above_half_precision(double c2, double scale2) {
	return __double2hiint(c2) - __double2hiint(scale2) > -(52 << 20);
}
__device__ __forceinline__ bool above_half_precision(float, float) { return false; }

// A rotation J = [[cos, s e], [-s conj(e), cos]], cos = 1 - s tau; s = tau = 0
// and e = 1 when the pair is not rotated.
template <class R>
struct Rotation {
	R s, tau, er, ei;
};

// Rotation that (nearly) zeroes c = A_pq of the pair with diagonals a, b. A
// Jacobi rotation has to be unitary to the working precision, but its angle
// need not be exact: the angle comes from single-precision estimates (relative
// error about 1e-7, which leaves 1e-7 |c| in place of the zero, computed by
// rotated_pair), and the unitary is then built from it in precision R:
//   tau = tan(angle / 2) = u (the single-precision value, exactly),
//   sin = 2 u / (1 + u^2), cos = 1 - sin tau = (1 - u^2) / (1 + u^2),
//   e   = c / |c| with |e| corrected to one by the series of (1 - x)^{-1/2}.
// In double precision this replaces a chain of five Newton-refined square roots
// and reciprocals (about 40 dependent operations of 8.5 cycles) by about eight,
// on the critical path of every inner round. Counted rotations (relative size
// above `noise`) and the largest counted tangent accumulate in cnt and tmax. In
// double precision a rotation of a relative size above 2^-26 counts with a tangent
// of at least 2^-28, above the tangent that ends the sweeps by default: it leaves
// 1e-7 of its element, which is more than rounding beside sqrt(|a b|). The tangent
// alone does not say so where the diagonals differ by many decades (1e-9 may go
// with an element as large as sqrt(|a b|)).
template <class R>
__device__ __forceinline__ Rotation<R> make_rotation(R a, R b, R cr, R ci, R tol, R noise, int& cnt, R& tmax) {
	const R c2 = cr * cr + ci * ci;
	const R scale2 = fabs(a) * fabs(b);
	const R d = (R)0.5 * (b - a);
	const R mc = fmax(fabs(cr), fabs(ci));
	bool want = c2 > tol * tol * scale2;
	bool counted = c2 > noise * noise * scale2;
	bool coarse = above_half_precision(c2, scale2);
	// squares and quotients of d and c stay inside the single-precision range
	const bool narrow = mc > (R)1e-18 && mc < (R)1e18 && fabs(d) < (R)1e18;
	const float x = (float)cr, y = (float)ci;
	const float dn = fabsf((float)d);
	const float h2 = x * x + y * y;
	const float ih = rsqrt_approx(h2);
	const float q2 = fmaf(dn, dn, h2);
	const float v = h2 * ih * rcp_approx(fmaf(q2, rsqrt_approx(q2), dn));  // tan = |c| / (|d| + r) in [0, 1]
	const float w = v * v, w2 = w * w, w4 = w2 * w2;
	// tan(angle / 2) = v / (1 + sqrt(1 + w)) and 1 / (1 + u^2) = (1 + 1 / sqrt(1 + w)) / 2
	// from Chebyshev fits on [0, 1] (relative errors 6e-8 and 1.8e-7)
	const float u = v * fmaf(w4, fmaf(w2, fmaf(w, -0.00104739867f, 0.00552987031f), fmaf(w, -0.0140554882f, 0.0248493936f)),
			fmaf(w2, fmaf(w, -0.0385012144f, 0.0624355158f), fmaf(w, -0.124997111f, 0.499999978f)));
	const R q0 = (R)fmaf(w4,
			fmaf(w2, fmaf(w, -0.00630942694f, 0.0319823643f), fmaf(w, -0.0757951591f, 0.118910862f)),
			fmaf(w2, fmaf(w, -0.152307005f, 0.18705187f), fmaf(w, -0.249980073f, 0.999999852f)));
	R t = (R)v;
	const R ud = (R)u;
	const R r1 = fma(-fma(ud, ud, (R)1), q0, (R)1);
	const R inv = fma(q0, fma(r1, r1, r1), q0);  // 1 / (1 + u^2) to r1^3, about 1e-20
	const R e0 = (R)(x * ih), e1 = (R)(y * ih);
	const R dl = fma(-e1, e1, fma(-e0, e0, (R)1));  // 1 - |e|^2, about 1e-7
	const R f = fma(dl, fma(dl, (R)0.375, (R)0.5), (R)1);
	Rotation<R> J;
	J.tau = d < 0 ? -ud : ud;
	J.s = (R)2 * J.tau * inv;
	J.er = e0 * f;
	J.ei = e1 * f;
	// the squares decide where |a b| is well inside the range of R (an element
	// whose square vanishes there is below the threshold)
	if (mc > (R)0 && (!well_inside(scale2) || (want && !narrow))) {
		const WideRotation w = rotation_wide(a, b, cr, ci, tol, noise);
		J.s = (R)w.s;
		J.tau = (R)w.tau;
		J.er = (R)w.er;
		J.ei = (R)w.ei;
		t = (R)w.t;
		want = true;
		counted = w.counted;
		coarse = sizeof(R) == 8 && w.coarse;
	}
	if (!want || t == (R)0) {
		J.s = J.tau = J.ei = (R)0;
		J.er = (R)1;
	} else if (counted) {
		cnt++;
		tmax = fmax(tmax, coarse ? fmax(t, (R)0x1p-28) : t);
	}
	return J;
}

// J^H [[a, c], [conj(c), b]] J: with w = conj(e) c and d = (b - a) / 2 the
// diagonals are a + h and b - h, h = 2 s (s d - cos Re w), and the off-diagonal
// e (Re w - 2 s (s Re w + cos d) + i Im w), which vanishes for the exact angle.
template <class R>
__device__ __forceinline__ void rotated_pair(const Rotation<R>& J, R& a, R& b, R& cr, R& ci) {
	const R cs = fma(-J.s, J.tau, (R)1);
	const R d = (R)0.5 * (b - a);
	const R wr = J.er * cr + J.ei * ci;
	const R wi = J.er * ci - J.ei * cr;
	const R h = (R)2 * J.s * (J.s * d - cs * wr);
	const R g = wr - (R)2 * J.s * (J.s * wr + cs * d);
	a += h;
	b -= h;
	cr = J.er * g - J.ei * wi;
	ci = J.er * wi + J.ei * g;
}

// Element (x, y) of the Hermitian M kept as its upper triangle.
__device__ __forceinline__ int m_at(int x, int y) { return min(x, y) * LDM + max(x, y); }
template <class T>
__device__ __forceinline__ T ld_m(const T* m, int x, int y) {
	T v = m[m_at(x, y)];
	if (x > y) v.y = -v.y;
	return v;
}
template <class T>
__device__ __forceinline__ void st_m(T* m, int x, int y, T v) {
	if (x > y) v.y = -v.y;
	m[m_at(x, y)] = v;
}

// The index of pair position pos in round r of the circle method on MS indices.
__device__ __forceinline__ int circle(int pos, int r) {
	int v = pos - 1 + r;
	if (v >= MS - 1) v -= MS - 1;
	return pos == 0 ? 0 : v + 1;
}

// Rows p, q of J^H X with J = [[c, s e], [-s conj(e), c]] (correction form,
// tau = s / (1 + c)).
template <class R>
__device__ __forceinline__ void rows2(R s, R tau, R er, R ei, R& xpr, R& xpi,
		R& xqr, R& xqi) {
	// yp = xp - s (e xq + tau xp)
	const R ypr = xpr - s * (er * xqr - ei * xqi + tau * xpr);
	const R ypi = xpi - s * (er * xqi + ei * xqr + tau * xpi);
	// yq = xq + s (conj(e) xp - tau xq)
	const R yqr = xqr + s * (er * xpr + ei * xpi - tau * xqr);
	const R yqi = xqi + s * (er * xpi - ei * xpr - tau * xqi);
	xpr = ypr; xpi = ypi; xqr = yqr; xqi = yqi;
}

// Columns s, t of X J (correction form, tau = s / (1 + c)).
template <class R>
__device__ __forceinline__ void cols2(R s, R tau, R er, R ei, R& xsr, R& xsi,
		R& xtr, R& xti) {
	// ys = xs - s (conj(e) xt + tau xs)
	const R ysr = xsr - s * (er * xtr + ei * xti + tau * xsr);
	const R ysi = xsi - s * (er * xti - ei * xtr + tau * xsi);
	// yt = xt + s (e xs - tau xt)
	const R ytr = xtr + s * (er * xsr - ei * xsi - tau * xtr);
	const R yti = xti + s * (er * xsi + ei * xsr - tau * xti);
	xsr = ysr; xsi = ysi; xtr = ytr; xti = yti;
}

// One inner sweep on the MS x MS subproblem in M buffer 0: FULL, MS - 1 rounds
// of NR rotations over all pairs (circle method: pair j is (position j,
// position MS - 1 - j)), or cross, BS rounds (round r pairs j with BS + (j + r)
// % BS). The result is left in M buffer R & 1 (R rounds) and the unitary Q in
// Qg (Q(i, l) at [i * MS + l], transposed with QT). Four groups of warps work
// side by side on round r, one barrier per round:
//  * warp 0 (lane j: pair j) computes rotation r + 1 from M_r and rotation r.
//    The two indices of pair j of round r + 1 sit in two different pairs A, B
//    of round r, so its off-diagonal element is one element of the 2 x 2 block
//    (A, B) rotated by rotation r; its diagonals are lane A's and lane B's,
//    carried in registers.
//  * warps 1, 2, 3 and 5 (one 2 x 2 block of pairs ja < jb per thread, 120 of
//    128) form J^H M J in the other M buffer: the upper triangle only.
//  * warp 4 (lane j: pair j) forms the rotated pairs' own 2 x 2 blocks in double
//    precision (4 % of an eigensolve at k = 200 in place of warp 0 doing it; in
//    single precision warp 0 is 2 % faster with them than without).
//  * warps 6, 7, 9-11 and 13-15 hold Q in registers (lane j: the columns of
//    pair j, four rows per warp) and pass the columns on through shared memory
//    (shuffles of 64-bit values cost four times as much there: 3.7 cycles per
//    32-bit shuffle).
// Warps 8 and 12 stay idle: warp 0 has its scheduler almost to itself, because its
// chain of rotations bounds the round. Before, every warp updating M set up two
// rotations itself, in double precision, and all of M and Q crossed shared
// memory: 2390 cycles per cross round against about 1000 now (FP32 about 700).
// Offsets whose order is known in a cross sweep are formed without comparing
// (with the round counters kept in 32 bits: 8 % of an eigensolve).
// `sh`: m(b), the buffers of M; rst, re, the rotations; xch(), the exchange area
// of the Q warps; cnt and tmax; in double precision mixed (one Q warp notes any
// rotation by more than 2^-20).
template <class R, bool FULL, bool QT, class SH>
__device__ __forceinline__ void inner_sweep(SH& sh, R tol, R noise, c2<R>* Qg) {
	using T = c2<R>;
	constexpr int ROUNDS = FULL ? MS - 1 : BS;
	constexpr bool OWN_PAIRS = sizeof(R) == 4;  // warp 0 stores its pairs' blocks
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	// position of pair index j's second member in round r
	auto second = [](int j, int r) { return FULL ? circle(MS - 1 - j, r) : BS + ((j + r) & (BS - 1)); };
	auto first = [](int j, int r) { return FULL ? circle(j, r) : j; };
	if (warp == 0) {
		const int j = lane & (NR - 1);
		int cnt = 0;
		R tmax = 0.0;
		const int p = first(j, 0), q = second(j, 0);
		R a = sh.m(0)[m_at(p, p)].x, b = sh.m(0)[m_at(q, q)].x;
		T c = ld_m(sh.m(0), p, q);
		Rotation<R> ro = make_rotation<R>(a, b, c.x, c.y, tol, noise, cnt, tmax);
		if (lane < NR) {
			sh.rst[0][j] = mk<R>(ro.s, ro.tau);
			sh.re[0][j] = mk<R>(ro.er, ro.ei);
		}
		// round r + 1's pair j: index 1 of pair A (its first or second member) and
		// of pair B; the other members ride along in the 2 x 2 block
		const int A = FULL ? (j == 0 ? 0 : min(j + 1, NR - 1)) : j;
		const int B = FULL ? (j == 0 ? 1 : j - 1) : ((j + 1) & (NR - 1));
		const bool a_first = !FULL || j < NR - 1, b_first = FULL && j == 0;
		const R sa = a_first ? 1.0 : -1.0, sb = b_first ? 1.0 : -1.0;
		// the block's element offsets and signs of the imaginary parts, formed
		// one round ahead: x and y the indices that meet, xo and yo their partners
		int o11, o21, o12, o22;
		unsigned conj;
		auto block = [&](int r) {
			if constexpr (!FULL) {
				// members below and above BS: the order of all but (xo, y) is known
				const int y = second(B, r), xo = second(A, r);
				o11 = j * LDM + y;
				o21 = m_at(xo, y);
				o12 = m_at(j, B);
				o22 = B * LDM + xo;
				conj = (xo > y ? 2u : 0u) | (j > B ? 4u : 0u) | 8u;
				return;
			}
			const int fa = first(A, r), qa = second(A, r), fb = first(B, r), qb = second(B, r);
			const int x = a_first ? fa : qa, y = b_first ? fb : qb;
			const int xo = a_first ? qa : fa, yo = b_first ? qb : fb;
			o11 = m_at(x, y);
			o21 = m_at(xo, y);
			o12 = m_at(x, yo);
			o22 = m_at(xo, yo);
			conj = (x > y ? 1u : 0u) | (xo > y ? 2u : 0u) | (x > yo ? 4u : 0u) | (xo > yo ? 8u : 0u);
		};
		block(0);
		__syncthreads();
#pragma unroll 1
		for (int r = 0; r < ROUNDS; r++) {
			const int cur = r & 1;
			const T* m = sh.m(cur);
			T* mn = sh.m(cur ^ 1);
			T m11 = m[o11], m21 = m[o21], m12 = m[o12], m22 = m[o22];
			const T ta = sh.rst[cur][A], ea = sh.re[cur][A], tb = sh.rst[cur][B], eb = sh.re[cur][B];
			// the diagonals after rotation r, before the loads are used
			rotated_pair(ro, a, b, c.x, c.y);
			const R ao = a, bo = b;
			if (OWN_PAIRS && lane < NR) {
				const int p = first(j, r), q = second(j, r);
				mn[p * (LDM + 1)] = mk<R>(ao, 0.0);
				mn[q * (LDM + 1)] = mk<R>(bo, 0.0);
				if (FULL) st_m(mn, p, q, c);
				else mn[p * LDM + q] = c;
			}
			if (r + 1 < ROUNDS) {
				if (conj & 1) m11.y = -m11.y;
				if (conj & 2) m21.y = -m21.y;
				if (conj & 4) m12.y = -m12.y;
				if (conj & 8) m22.y = -m22.y;
				// row x of J_A^H M: x - s (e xo + tau x), with s, tau and Im e negated
				// for the second member
				const R s1 = sa * ta.x, t1 = sa * ta.y, e1i = sa * ea.y;
				const R u1r = m11.x - s1 * (ea.x * m21.x - e1i * m21.y + t1 * m11.x);
				const R u1i = m11.y - s1 * (ea.x * m21.y + e1i * m21.x + t1 * m11.y);
				const R u2r = m12.x - s1 * (ea.x * m22.x - e1i * m22.y + t1 * m12.x);
				const R u2i = m12.y - s1 * (ea.x * m22.y + e1i * m22.x + t1 * m12.y);
				// column y of the result times J_B: y - s (conj(e) yo + tau y)
				const R s2 = sb * tb.x, t2 = sb * tb.y, e2i = sb * eb.y;
				c.x = u1r - s2 * (eb.x * u2r + e2i * u2i + t2 * u1r);
				c.y = u1i - s2 * (eb.x * u2i - e2i * u2r + t2 * u1i);
				if (FULL) {
					const R an = __shfl_sync(0xffffffffu, ao, (j + 1) & (NR - 1), NR);
					const R bp = __shfl_sync(0xffffffffu, bo, (j - 1) & (NR - 1), NR);
					a = j == 0 ? ao : (j == NR - 1 ? bo : an);
					b = j == 0 ? an : bp;
				} else {
					b = __shfl_sync(0xffffffffu, bo, (j + 1) & (NR - 1), NR);
				}
				block(r + 1);
				ro = make_rotation<R>(a, b, c.x, c.y, tol, noise, cnt, tmax);
				if (lane < NR) {
					sh.rst[cur ^ 1][j] = mk<R>(ro.s, ro.tau);
					sh.re[cur ^ 1][j] = mk<R>(ro.er, ro.ei);
				}
			}
			__syncthreads();
		}
		if (lane >= NR) {
			cnt = 0;
			tmax = 0.0;
		}
		for (int o = 8; o > 0; o >>= 1) {
			cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
			tmax = fmax(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
		}
		if (lane == 0 && cnt) {
			sh.cnt += cnt;
			const unsigned long long tb = (unsigned long long)__double_as_longlong((double)tmax);
			if (tb > sh.tmax) sh.tmax = tb;
		}
	} else if (warp < 4 || warp == 5) {
		// item (ja, jb), ja < jb, of the NR (NR - 1) / 2
		const int item = (warp < 4 ? warp - 1 : 3) * 32 + lane;
		int ja = 0, jb = 1;
		{
			int left = item;
			while (ja < NR - 1 && left >= NR - 1 - ja) {
				left -= NR - 1 - ja;
				ja++;
			}
			jb = ja + 1 + left;
		}
		const bool on = item < NR * (NR - 1) / 2;
		__syncthreads();
#pragma unroll 1
		for (int r = 0; r < ROUNDS; r++) {
			const int cur = r & 1;
			if (on) {
				const T* m = sh.m(cur);
				T* mn = sh.m(cur ^ 1);
				// offsets of the block's elements, and which are stored conjugated
				const int p = first(ja, r), q = second(ja, r), s = first(jb, r), t = second(jb, r);
				const int ops = FULL ? m_at(p, s) : ja * LDM + jb, opt = FULL ? m_at(p, t) : ja * LDM + t;
				const int oqs = FULL ? m_at(q, s) : jb * LDM + q, oqt = m_at(q, t);
				const bool nps = FULL && p > s, npt = FULL && p > t, nqs = !FULL || q > s, nqt = q > t;
				T ps = m[ops], pt = m[opt], qs = m[oqs], qt = m[oqt];
				if (nps) ps.y = -ps.y;
				if (npt) pt.y = -pt.y;
				if (nqs) qs.y = -qs.y;
				if (nqt) qt.y = -qt.y;
				const T ta = sh.rst[cur][ja], ea = sh.re[cur][ja], tb = sh.rst[cur][jb], eb = sh.re[cur][jb];
				rows2(ta.x, ta.y, ea.x, ea.y, ps.x, ps.y, qs.x, qs.y);
				rows2(ta.x, ta.y, ea.x, ea.y, pt.x, pt.y, qt.x, qt.y);
				cols2(tb.x, tb.y, eb.x, eb.y, ps.x, ps.y, pt.x, pt.y);
				cols2(tb.x, tb.y, eb.x, eb.y, qs.x, qs.y, qt.x, qt.y);
				if (nps) ps.y = -ps.y;
				if (npt) pt.y = -pt.y;
				if (nqs) qs.y = -qs.y;
				if (nqt) qt.y = -qt.y;
				mn[ops] = ps;
				mn[opt] = pt;
				mn[oqs] = qs;
				mn[oqt] = qt;
			}
			__syncthreads();
		}
	} else if ((warp & 3) != 0) {
		// rows i0, i0 + 1 of Q, columns of pair j
		const int w = warp < 8 ? warp - 6 : (warp < 12 ? warp - 7 : warp - 8);
		const int j = lane & (NR - 1);
		const int i0 = 4 * w + 2 * (lane >> 4);
		const int p0 = first(j, 0), q0 = second(j, 0);
		T xp[2], xq[2];
#pragma unroll
		for (int h = 0; h < 2; h++) {
			xp[h] = mk<R>(i0 + h == p0 ? 1.0 : 0.0, 0.0);
			xq[h] = mk<R>(i0 + h == q0 ? 1.0 : 0.0, 0.0);
		}
		bool mixed = false;  // a rotation by more than 2^-20
		// this warp's exchange area: [member][row h][half of the warp][column]
		T* xch = sh.xch() + w * 4 * 2 * NR;
		const int at = (lane >> 4) * NR, own = at + j, up = at + ((j + 1) & (NR - 1)), down = at + ((j - 1) & (NR - 1));
		__syncthreads();
#pragma unroll 1
		for (int r = 0; r < ROUNDS; r++) {
			const T st = sh.rst[r & 1][j], e = sh.re[r & 1][j];
			if constexpr (sizeof(R) == 8) mixed |= (__double2hiint(st.x) & 0x7FFFFFFF) >= (1023 - 20) << 20;
#pragma unroll
			for (int h = 0; h < 2; h++) cols2(st.x, st.y, e.x, e.y, xp[h].x, xp[h].y, xq[h].x, xq[h].y);
			// the columns move on to the lanes of round r + 1's pairs
#pragma unroll
			for (int h = 0; h < 2; h++) {
				xch[32 * h + own] = xq[h];
				if (FULL) xch[64 + 32 * h + own] = xp[h];
			}
			__syncwarp();
#pragma unroll
			for (int h = 0; h < 2; h++) {
				if (FULL) {
					// positions move up by one around the circle, position 0 stays
					const T pn = xch[64 + 32 * h + up];
					const T qn = xch[32 * h + down];
					if (j == NR - 1) xp[h] = xq[h];
					else if (j > 0) xp[h] = pn;
					xq[h] = j == 0 ? pn : qn;
				} else {
					xq[h] = xch[32 * h + up];
				}
			}
			__syncthreads();  // also: the exchange area is free again
		}
		if constexpr (sizeof(R) == 8) {
			if (w == 0 && __any_sync(0xffffffffu, mixed) && lane == 0) sh.mixed = 1;
		}
		// after all rounds the columns are back at their places
#pragma unroll
		for (int h = 0; h < 2; h++) {
			Qg[QT ? p0 * MS + i0 + h : (i0 + h) * MS + p0] = xp[h];
			Qg[QT ? q0 * MS + i0 + h : (i0 + h) * MS + q0] = xq[h];
		}
	} else if (!OWN_PAIRS && warp == 4) {
		const int j = lane & (NR - 1);
		__syncthreads();
#pragma unroll 1
		for (int r = 0; r < ROUNDS; r++) {
			const T* m = sh.m(r & 1);
			T* mn = sh.m((r & 1) ^ 1);
			if (lane < NR) {
				const int p = first(j, r), q = second(j, r), opq = FULL ? m_at(p, q) : p * LDM + q;
				const T st = sh.rst[r & 1][j], e = sh.re[r & 1][j];
				R a = m[p * (LDM + 1)].x, b = m[q * (LDM + 1)].x;
				T c = m[opq];
				if (FULL && p > q) c.y = -c.y;
				rotated_pair(Rotation<R>{st.x, st.y, e.x, e.y}, a, b, c.x, c.y);
				if (FULL && p > q) c.y = -c.y;
				mn[p * (LDM + 1)] = mk<R>(a, 0.0);
				mn[q * (LDM + 1)] = mk<R>(b, 0.0);
				mn[opq] = c;
			}
			__syncthreads();
		}
	} else {
		__syncthreads();
#pragma unroll 1
		for (int r = 0; r < ROUNDS; r++) __syncthreads();
	}
	__syncthreads();
}

// Position of player p in round r of the circle method (inverse of rr_player).
__device__ __forceinline__ int rr_position(int p, int r, int npos) {
	if (p == 0) return 0;
	const int v = p - 1 - r;  // 0 <= r < npos - 1
	return v < 0 ? v + npos : v + 1;
}

// Phase 2 item w of a round: an off-diagonal pair block (jr, jc) of A above the
// diagonal (its mirror image is written with it), or the slab jr of V (32
// rows) for the pair jc.
struct Item {
	int jr, jc;
	bool is_v;
};
__device__ __forceinline__ Item item_of(int w, int np) {
	const int nA2 = np * (np - 1) / 2;
	Item it;
	it.is_v = w >= nA2;
	if (it.is_v) {
		it.jr = (w - nA2) / np;
		it.jc = (w - nA2) % np;
	} else {
		// pair w of the upper triangle jr < jc, by columns
		int jc = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)w)) * 0.5f);
		while (jc * (jc - 1) / 2 > w) jc--;
		while ((jc + 1) * jc / 2 <= w) jc++;
		it.jc = jc;
		it.jr = w - jc * (jc - 1) / 2;
	}
	return it;
}

}  // namespace bj

}  // namespace itp2d
