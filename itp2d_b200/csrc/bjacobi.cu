// Block Jacobi eigensolver of the overlap matrix.
//
// Cyclic two-sided Jacobi (A <- J^H A J, V <- V J) organised for few grid-wide
// rounds: the padded index range is cut into blocks of BS, blocks are paired
// round-robin (k/BS - 1 rounds per sweep), and each round r has two phases:
//   1. one CTA per block pair sweeps the 2BS x 2BS Hermitian subproblem in
//      shared memory with cyclic Jacobi (CTA barriers only), leaving its
//      2BS x 2BS unitary Q_r in global memory and the rotated subproblem as
//      the diagonal pair block of A_r;
//   2. every other 2BS x 2BS block of A_r becomes Q_r^H A_{r-1} Q_r (row and
//      column pairs; the blocks above the diagonal, mirrored) and every slab
//      of 2BS rows of V becomes V Q_r, both as FP64 DMMA products staged in
//      shared memory.
// The phases are pipelined: one grid barrier separates supersteps, and
// superstep t runs phase 1 of round t on one set of CTAs while the others run
// phase 2 of round t - 1. Phase 1 of round t therefore builds its subproblem
// itself: its diagonal blocks are parts of round t - 1's rotated subproblems
// (already in A_{t-1}), and its off-diagonal block (P', Q') is taken from
// Q_a^H A_{t-2}(a, b) Q_b for the round t - 1 pairs a, b that held P' and Q'.
// Three matrix buffers rotate (A_{t-2} read, A_{t-1} completed by phase 2,
// A_t's diagonal pair blocks written by phase 1) and Q alternates between two
// buffers.
// In every 16th round of an outer sweep (starting with the first) every
// subproblem gets one full inner sweep (all pairs of its 2BS indices, so every
// within-block pair is rotated at least once per outer sweep); in the other
// rounds only the BS x BS cross pairs (p in block P, q in block Q) are
// rotated, in BS inner rounds. Over an outer sweep every index pair is thus
// rotated at least once, a block-cyclic ordering of cyclic Jacobi. A rotation is applied when |A_pq| > tol sqrt(|A_pp A_qq|).
// Rotations whose relative off-diagonal |A_pq| / sqrt(|A_pp A_qq|) is at the
// rounding level of the phase-2 products (below 1e-13) do not count against
// convergence; the iteration stops after a sweep whose largest counted
// rotation tangent is below tau_final (3e-9 by default: quadratic convergence
// then leaves off-diagonal elements of order k * 1e-17 relative to the gaps).
#include <cooperative_groups.h>

#include "../../include/itp2d_gpu.h"
#include "contract.cuh"

namespace cg = cooperative_groups;

namespace itp2d {

namespace {

constexpr int BS = 16;        // block size
constexpr int MS = 32;        // subproblem size: two blocks
constexpr int NR = MS / 2;    // rotations per inner round
constexpr int LD = MS + 4;    // padded row length (complex): conflict-free 16-byte DMMA fragments
constexpr int OP = MS * LD;   // elements of one product operand
constexpr int LDM = MS + 1;   // row length of M: conflict-free rows and columns
// 512 threads, one CTA per SM: an inner sweep gives its warps separate roles
// (inner_sweep); the two halves of a phase-2 CTA work on separate products.
constexpr int kThreads = 512;
constexpr double kTauFinal = 3e-9;
// Rounds between full inner sweeps (within-block pairs rotated again); every
// 16th round measured best on k = 500 (fewer outer sweeps for little cost).
constexpr int kFullEvery = 16;
constexpr double kNoiseRel = 1e-13;  // relative off-diagonal treated as rounding noise

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
	asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
			: "+d"(d0), "+d"(d1)
			: "d"(a), "d"(b));
}

// Round-robin pairing of npos positions (circle method): position 0 fixed.
__device__ __forceinline__ int rr_player(int pos, int r, int npos) {
	return pos == 0 ? 0 : ((pos - 1 + r) % (npos - 1)) + 1;
}

// Global index of local subproblem index i (< 64) for the block pair (P, Q).
__device__ __forceinline__ int gidx(int i, int P, int Q) { return i < BS ? P * BS + i : Q * BS + (i - BS); }

struct Shared {
	// phase 1: op[0] and op[1], op[2] formation operands, then the two buffers of
	// the subproblem M (row length LDM); phase 2: half h of the CTA uses op[6h,
	// 6h + 6), two stages of (X, Q_c, Q_r), the next item's copied in while the
	// current one is multiplied
	double2 op[12][OP];
	// rotations of two consecutive inner rounds (round r in buffer r & 1)
	double2 rst[2][NR];                          // (sin, tau), (0, 0): none
	double2 re[2][NR];                           // e = c / |c|
	int next[2];  // phase-2 item of each CTA half
	int cnt;                                     // counted rotations of the current outer sweep
	unsigned long long tmax;                     // largest tangent (bits of a non-negative double)
	// Subproblem buffer b, only the upper triangle (row <= column) in use.
	__device__ double2* m(int b) { return op[3] + b * OP; }
};

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

// Exponent of a positive normal double, and 2^e for -1022 <= e <= 1023, by
// bit manipulation (exact).
__device__ __forceinline__ int exp2i(double x) { return (int)((__double_as_longlong(x) >> 52) & 0x7ff) - 1023; }
__device__ __forceinline__ double pow2i(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

// sin, tau = tan(angle / 2), e and tan of a rotation in double precision
// throughout, for pairs whose exponents leave the range of the single-precision
// set-up below: with u = |d| + r and w = 2 r u, cos = u / sqrt(w), |sin| =
// |c| / sqrt(w) and |tau| = |c| / (sqrt(w) + u), d and c scaled by exact powers
// of two.
__device__ __noinline__ void rotation_wide(double d, double cr, double ci, double& s, double& tau, double& er,
		double& ei, double& t) {
	const double ad = fabs(d);
	const double mc = fmax(fabs(cr), fabs(ci));
	const int ex = ilogb(fmax(ad, mc)), exc = ilogb(mc);
	const double sc = scalbn(1.0, -ex), scc = scalbn(1.0, -exc);
	const double dn = ad * sc, crn = cr * sc, cin = ci * sc;
	const double cn2 = crn * crn + cin * cin;
	const double rn2 = dn * dn + cn2;         // [1, 12)
	const double rn = rn2 * rsqrt_nr(rn2);
	const double un = dn + rn;                // [1, 5.5)
	const double wn = 2.0 * rn * un;          // [2, 38)
	const double qn = rsqrt_nr(wn);
	const double cn = sqrt(cn2);
	t = cn * rcp_nr(un);
	const double crs = cr * scc, cis = ci * scc;
	const double ec = rsqrt_nr(crs * crs + cis * cis);
	const double sg = d < 0 ? -1.0 : 1.0;
	s = sg * cn * qn;
	tau = sg * cn * rcp_nr(wn * qn + un);
	er = crs * ec;
	ei = cis * ec;
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

// A rotation J = [[cos, s e], [-s conj(e), cos]], cos = 1 - s tau; s = tau = 0
// and e = 1 when the pair is not rotated.
struct Rotation {
	double s, tau, er, ei;
};

// Rotation that (nearly) zeroes c = A_pq of the pair with diagonals a, b. A
// Jacobi rotation has to be unitary to double precision, but its angle need
// not be exact: the angle comes from single precision (relative error about
// 1e-7, which leaves 1e-7 |c| in place of the zero, computed by rotated_pair),
// and the unitary is then built from it in double precision:
//   tau = tan(angle / 2) = u (the single-precision value, exactly),
//   sin = 2 u / (1 + u^2), cos = 1 - sin tau = (1 - u^2) / (1 + u^2),
//   e   = c / |c| with |e| corrected to one by the series of (1 - x)^{-1/2}.
// This replaces a chain of five Newton-refined double-precision square roots
// and reciprocals (about 40 dependent operations of 8.5 cycles) by about
// eight, on the critical path of every inner round. Counted rotations and the
// largest counted tangent accumulate in cnt and tmax.
__device__ __forceinline__ Rotation make_rotation(double a, double b, double cr, double ci, double tol, int& cnt,
		double& tmax) {
	const double c2 = cr * cr + ci * ci;
	const double scale2 = fabs(a) * fabs(b);
	const double d = 0.5 * (b - a);
	const double mc = fmax(fabs(cr), fabs(ci));
	const bool want = c2 > 0.0 && c2 > tol * tol * scale2;
	// squares and quotients of d and c stay inside the single-precision range
	const bool narrow = mc > 1e-18 && mc < 1e18 && fabs(d) < 1e18;
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
	const double q0 = (double)fmaf(w4,
			fmaf(w2, fmaf(w, -0.00630942694f, 0.0319823643f), fmaf(w, -0.0757951591f, 0.118910862f)),
			fmaf(w2, fmaf(w, -0.152307005f, 0.18705187f), fmaf(w, -0.249980073f, 0.999999852f)));
	double t = (double)v;
	const double ud = (double)u;
	const double r1 = fma(-fma(ud, ud, 1.0), q0, 1.0);
	const double inv = fma(q0, fma(r1, r1, r1), q0);  // 1 / (1 + u^2) to r1^3, about 1e-20
	const double e0 = (double)(x * ih), e1 = (double)(y * ih);
	const double dl = fma(-e1, e1, fma(-e0, e0, 1.0));  // 1 - |e|^2, about 1e-7
	const double f = fma(dl, fma(dl, 0.375, 0.5), 1.0);
	Rotation R;
	R.tau = d < 0 ? -ud : ud;
	R.s = 2.0 * R.tau * inv;
	R.er = e0 * f;
	R.ei = e1 * f;
	if (want && !narrow) rotation_wide(d, cr, ci, R.s, R.tau, R.er, R.ei, t);
	if (!want || t == 0.0) {
		R.s = R.tau = R.ei = 0.0;
		R.er = 1.0;
	} else if (c2 > kNoiseRel * kNoiseRel * scale2) {
		cnt++;
		tmax = fmax(tmax, t);
	}
	return R;
}

// J^H [[a, c], [conj(c), b]] J: with w = conj(e) c and d = (b - a) / 2 the
// diagonals are a + h and b - h, h = 2 s (s d - cos Re w), and the off-diagonal
// e (Re w - 2 s (s Re w + cos d) + i Im w), which vanishes for the exact angle.
__device__ __forceinline__ void rotated_pair(const Rotation& R, double& a, double& b, double& cr, double& ci) {
	const double cs = fma(-R.s, R.tau, 1.0);
	const double d = 0.5 * (b - a);
	const double wr = R.er * cr + R.ei * ci;
	const double wi = R.er * ci - R.ei * cr;
	const double h = 2.0 * R.s * (R.s * d - cs * wr);
	const double g = wr - 2.0 * R.s * (R.s * wr + cs * d);
	a += h;
	b -= h;
	cr = R.er * g - R.ei * wi;
	ci = R.er * wi + R.ei * g;
}

// Element (x, y) of the Hermitian M kept as its upper triangle.
__device__ __forceinline__ int m_at(int x, int y) { return min(x, y) * LDM + max(x, y); }
__device__ __forceinline__ double2 ld_m(const double2* m, int x, int y) {
	double2 v = m[m_at(x, y)];
	if (x > y) v.y = -v.y;
	return v;
}
__device__ __forceinline__ void st_m(double2* m, int x, int y, double2 v) {
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
__device__ __forceinline__ void rows2(double s, double tau, double er, double ei, double& xpr, double& xpi,
		double& xqr, double& xqi) {
	// yp = xp - s (e xq + tau xp)
	const double ypr = xpr - s * (er * xqr - ei * xqi + tau * xpr);
	const double ypi = xpi - s * (er * xqi + ei * xqr + tau * xpi);
	// yq = xq + s (conj(e) xp - tau xq)
	const double yqr = xqr + s * (er * xpr + ei * xpi - tau * xqr);
	const double yqi = xqi + s * (er * xpi - ei * xpr - tau * xqi);
	xpr = ypr; xpi = ypi; xqr = yqr; xqi = yqi;
}

// Columns s, t of X J (correction form, tau = s / (1 + c)).
__device__ __forceinline__ void cols2(double s, double tau, double er, double ei, double& xsr, double& xsi,
		double& xtr, double& xti) {
	// ys = xs - s (conj(e) xt + tau xs)
	const double ysr = xsr - s * (er * xtr + ei * xti + tau * xsr);
	const double ysi = xsi - s * (er * xti - ei * xtr + tau * xsi);
	// yt = xt + s (e xs - tau xt)
	const double ytr = xtr + s * (er * xsr - ei * xsi - tau * xtr);
	const double yti = xti + s * (er * xsi + ei * xsr - tau * xti);
	xsr = ysr; xsi = ysi; xtr = ytr; xti = yti;
}

// One inner sweep on the MS x MS subproblem in M buffer 0: FULL, MS - 1 rounds
// of NR rotations over all pairs (circle method: pair j is (position j,
// position MS - 1 - j)), or cross, BS rounds (round r pairs j with BS + (j + r)
// % BS). The result is left in M buffer R & 1 (R rounds) and the unitary Q in
// Qg, transposed (Qg[l * MS + i] = Q(i, l)). Three groups of warps work side by side on round r, one barrier per
// round:
//  * warp 0 (lane j: pair j) computes rotation r + 1 from M_r and rotation r.
//    The two indices of pair j of round r + 1 sit in two different pairs A, B
//    of round r, so its off-diagonal element is one element of the 2 x 2 block
//    (A, B) rotated by rotation r; its diagonals are lane A's and lane B's,
//    carried in registers. It also writes the rotated pairs' own 2 x 2 blocks.
//  * warps 1, 2, 3 and 5 (one 2 x 2 block of pairs ja < jb per thread, 120 of
//    128) form J^H M J in the other M buffer: the upper triangle only.
//  * warps 6, 7, 9-11 and 13-15 hold Q in registers (lane j: the columns of
//    pair j, four rows per warp) and pass the columns on through shared memory
//    (shuffles of 64-bit values cost four times as much there: 3.7 cycles per
//    32-bit shuffle).
// Warps 4, 8 and 12 stay idle: warp 0 has its scheduler to itself, because its
// chain of rotations bounds the round. Before, every warp updating M set up two rotations itself,
// in double precision, and all of M and Q crossed shared memory: 2390 cycles
// per cross round against 940 now (1230 per full round).
template <bool FULL>
__device__ __forceinline__ void inner_sweep(Shared& sh, double tol, double2* Qg) {
	constexpr int R = FULL ? MS - 1 : BS;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	// position of pair index j's second member in round r
	auto second = [](int j, int r) { return FULL ? circle(MS - 1 - j, r) : BS + ((j + r) & (BS - 1)); };
	auto first = [](int j, int r) { return FULL ? circle(j, r) : j; };
	if (warp == 0) {
		const int j = lane & (NR - 1);
		int cnt = 0;
		double tmax = 0.0;
		int p = first(j, 0), q = second(j, 0);
		double a = sh.m(0)[m_at(p, p)].x, b = sh.m(0)[m_at(q, q)].x;
		double2 c = ld_m(sh.m(0), p, q);
		Rotation ro = make_rotation(a, b, c.x, c.y, tol, cnt, tmax);
		if (lane < NR) {
			sh.rst[0][j] = make_double2(ro.s, ro.tau);
			sh.re[0][j] = make_double2(ro.er, ro.ei);
		}
		// round r + 1's pair j: index 1 of pair A (its first or second member) and
		// of pair B; the other members ride along in the 2 x 2 block
		const int A = FULL ? (j == 0 ? 0 : min(j + 1, NR - 1)) : j;
		const int B = FULL ? (j == 0 ? 1 : j - 1) : ((j + 1) & (NR - 1));
		const bool a_first = !FULL || j < NR - 1, b_first = FULL && j == 0;
		const double sa = a_first ? 1.0 : -1.0, sb = b_first ? 1.0 : -1.0;
		// the block's element offsets and signs of the imaginary parts, formed
		// one round ahead: x and y the indices that meet, xo and yo their partners
		int x, y, o11, o21, o12, o22;
		unsigned conj;
		auto block = [&](int r) {
			const int fa = first(A, r), qa = second(A, r), fb = first(B, r), qb = second(B, r);
			x = a_first ? fa : qa;
			y = b_first ? fb : qb;
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
		for (int r = 0; r < R; r++) {
			const int cur = r & 1;
			const double2* m = sh.m(cur);
			double2* mn = sh.m(cur ^ 1);
			double2 m11 = m[o11], m21 = m[o21], m12 = m[o12], m22 = m[o22];
			const double2 ta = sh.rst[cur][A], ea = sh.re[cur][A], tb = sh.rst[cur][B], eb = sh.re[cur][B];
			// rotation r's own pair, before the loads are used
			const int po = p, qo = q;
			rotated_pair(ro, a, b, c.x, c.y);
			const double ao = a, bo = b;
			if (lane < NR) {
				mn[m_at(po, po)] = make_double2(ao, 0.0);
				mn[m_at(qo, qo)] = make_double2(bo, 0.0);
				st_m(mn, po, qo, c);
			}
			p = x;
			q = y;
			if (r + 1 < R) {
				if (conj & 1) m11.y = -m11.y;
				if (conj & 2) m21.y = -m21.y;
				if (conj & 4) m12.y = -m12.y;
				if (conj & 8) m22.y = -m22.y;
				// row x of J_A^H M: x - s (e xo + tau x), with s, tau and Im e negated
				// for the second member
				const double s1 = sa * ta.x, t1 = sa * ta.y, e1i = sa * ea.y;
				const double u1r = m11.x - s1 * (ea.x * m21.x - e1i * m21.y + t1 * m11.x);
				const double u1i = m11.y - s1 * (ea.x * m21.y + e1i * m21.x + t1 * m11.y);
				const double u2r = m12.x - s1 * (ea.x * m22.x - e1i * m22.y + t1 * m12.x);
				const double u2i = m12.y - s1 * (ea.x * m22.y + e1i * m22.x + t1 * m12.y);
				// column y of the result times J_B: y - s (conj(e) yo + tau y)
				const double s2 = sb * tb.x, t2 = sb * tb.y, e2i = sb * eb.y;
				c.x = u1r - s2 * (eb.x * u2r + e2i * u2i + t2 * u1r);
				c.y = u1i - s2 * (eb.x * u2i - e2i * u2r + t2 * u1i);
				if (FULL) {
					const double an = __shfl_sync(0xffffffffu, ao, (j + 1) & (NR - 1), NR);
					const double bp = __shfl_sync(0xffffffffu, bo, (j - 1) & (NR - 1), NR);
					a = j == 0 ? ao : (j == NR - 1 ? bo : an);
					b = j == 0 ? an : bp;
				} else {
					b = __shfl_sync(0xffffffffu, bo, (j + 1) & (NR - 1), NR);
				}
				block(r + 1);
				ro = make_rotation(a, b, c.x, c.y, tol, cnt, tmax);
				if (lane < NR) {
					sh.rst[cur ^ 1][j] = make_double2(ro.s, ro.tau);
					sh.re[cur ^ 1][j] = make_double2(ro.er, ro.ei);
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
			const unsigned long long tb = (unsigned long long)__double_as_longlong(tmax);
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
		for (int r = 0; r < R; r++) {
			const int cur = r & 1;
			if (on) {
				const double2* m = sh.m(cur);
				double2* mn = sh.m(cur ^ 1);
				const int p = first(ja, r), q = second(ja, r), s = first(jb, r), t = second(jb, r);
				double2 ps = ld_m(m, p, s), pt = ld_m(m, p, t), qs = ld_m(m, q, s), qt = ld_m(m, q, t);
				const double2 ta = sh.rst[cur][ja], ea = sh.re[cur][ja], tb = sh.rst[cur][jb], eb = sh.re[cur][jb];
				rows2(ta.x, ta.y, ea.x, ea.y, ps.x, ps.y, qs.x, qs.y);
				rows2(ta.x, ta.y, ea.x, ea.y, pt.x, pt.y, qt.x, qt.y);
				cols2(tb.x, tb.y, eb.x, eb.y, ps.x, ps.y, pt.x, pt.y);
				cols2(tb.x, tb.y, eb.x, eb.y, qs.x, qs.y, qt.x, qt.y);
				st_m(mn, p, s, ps);
				st_m(mn, p, t, pt);
				st_m(mn, q, s, qs);
				st_m(mn, q, t, qt);
			}
			__syncthreads();
		}
	} else if ((warp & 3) != 0) {
		// rows i0, i0 + 1 of Q, columns of pair j
		const int w = warp < 8 ? warp - 6 : (warp < 12 ? warp - 7 : warp - 8);
		const int j = lane & (NR - 1);
		const int i0 = 4 * w + 2 * (lane >> 4);
		const int p0 = first(j, 0), q0 = second(j, 0);
		double2 xp[2], xq[2];
#pragma unroll
		for (int h = 0; h < 2; h++) {
			xp[h] = make_double2(i0 + h == p0 ? 1.0 : 0.0, 0.0);
			xq[h] = make_double2(i0 + h == q0 ? 1.0 : 0.0, 0.0);
		}
		// this warp's exchange area: [member][row h][half of the warp][column]
		double2* xch = sh.op[5] + w * 4 * 2 * NR;
		const int at = (lane >> 4) * NR, own = at + j, up = at + ((j + 1) & (NR - 1)), down = at + ((j - 1) & (NR - 1));
		__syncthreads();
#pragma unroll 1
		for (int r = 0; r < R; r++) {
			const double2 st = sh.rst[r & 1][j], e = sh.re[r & 1][j];
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
					const double2 pn = xch[64 + 32 * h + up];
					const double2 qn = xch[32 * h + down];
					if (j == NR - 1) xp[h] = xq[h];
					else if (j > 0) xp[h] = pn;
					xq[h] = j == 0 ? pn : qn;
				} else {
					xq[h] = xch[32 * h + up];
				}
			}
			__syncthreads();  // also: the exchange area is free again
		}
		// after all rounds the columns are back at their places
#pragma unroll
		for (int h = 0; h < 2; h++) {
			Qg[p0 * MS + i0 + h] = xp[h];
			Qg[q0 * MS + i0 + h] = xq[h];
		}
	} else {
		__syncthreads();
#pragma unroll 1
		for (int r = 0; r < R; r++) __syncthreads();
	}
	__syncthreads();
}

// NT adjacent 8 x 8 tiles of the complex product C(i, l) = sum_m A(i, m) B(m, l)
// (32 deep) by one warp with FP64 DMMA, both operands kept with m along their
// rows: A(i, m) at A[i * LD + m] (conjugated with CONJ), B(m, l) at
// B[l * LD + m]. Lane: rows row0 + (lane >> 2), columns col0 + 8 b + 2 (lane & 3)
// + h of accumulator (b, h).
template <int NT, bool CONJ>
__device__ __forceinline__ void ctiles(int lane, const double2* A, const double2* B, int row0, int col0,
		double (&cr)[NT][2], double (&ci)[NT][2]) {
	const double2* a0 = A + (row0 + (lane >> 2)) * LD + (lane & 3);
	const double2* b0 = B + (col0 + (lane >> 2)) * LD + (lane & 3);
#pragma unroll
	for (int b = 0; b < NT; b++) cr[b][0] = cr[b][1] = ci[b][0] = ci[b][1] = 0.0;
#pragma unroll
	for (int kk = 0; kk < MS; kk += 4) {
		double2 a = a0[kk];
		if (CONJ) a.y = -a.y;
#pragma unroll
		for (int b = 0; b < NT; b++) {
			const double2 v = b0[b * 8 * LD + kk];
			dmma(cr[b][0], cr[b][1], a.x, v.x);
			dmma(ci[b][0], ci[b][1], a.x, v.y);
			dmma(cr[b][0], cr[b][1], -a.y, v.y);
			dmma(ci[b][0], ci[b][1], a.y, v.x);
		}
	}
}

// Full 32 x 32 product on one half of the CTA (local warp lw of 8): warp lw
// owns rows (lw >> 1) * 8 .. + 8 and columns (lw & 1) * 16 .. + 16.
template <bool CONJ>
__device__ __forceinline__ void half_gemm(int lt, const double2* A, const double2* B, double (&cr)[2][2],
		double (&ci)[2][2]) {
	const int lane = lt & 31, lw = lt >> 5;
	ctiles<2, CONJ>(lane, A, B, (lw >> 1) * 8, (lw & 1) * 16, cr, ci);
}

// Output coordinates of accumulator (b, h) of half_gemm for local thread lt.
__device__ __forceinline__ void half_rc(int lt, int b, int h, int& row, int& col) {
	const int lane = lt & 31, lw = lt >> 5;
	row = (lw >> 1) * 8 + (lane >> 2);
	col = (lw & 1) * 16 + b * 8 + 2 * (lane & 3) + h;
}

// Barrier of one half of the CTA (named barrier 1 + half, 256 threads).
__device__ __forceinline__ void half_sync(int half) {
	asm volatile("bar.sync %0, %1;\n" ::"r"(1 + half), "r"(kThreads / 2) : "memory");
}

// Position of player p in round r of the circle method (inverse of rr_player).
__device__ __forceinline__ int rr_position(int p, int r, int npos) {
	if (p == 0) return 0;
	const int m = npos - 1;
	return ((p - 1 - r) % m + m) % m + 1;
}

// Phase 1 for pair j of round t (within-sweep round rr): forms the subproblem
// (upper triangle of M buffer 0), sweeps it, stores Q_t and the rotated
// subproblem. prev: A_{t-1} (diagonal pair blocks of round t - 1), prev2:
// A_{t-2}, Qprev: the Q buffer of round t - 1 (t >= 1). For t = 0 the
// subproblem is read from prev = A_{-1}, the initial matrix.
__device__ void phase1_item(Shared& sh, int j, long long t, int rounds, int nb, int np, int kp, double tol,
		const double2* prev, const double2* prev2, const double2* Qprev, double2* Qout, double2* out) {
	const int tid = threadIdx.x;
	const int rr = (int)(t % rounds);
	const int P = rr_player(j, rr, nb), Q = rr_player(nb - 1 - j, rr, nb);
	double2* M = sh.m(0);
	if (t == 0) {
		for (int e = tid; e < MS * MS; e += kThreads) {
			const int i = e / MS, l = e % MS;
			M[i * LDM + l] = __ldcg(prev + (long long)gidx(i, P, Q) * kp + gidx(l, P, Q));
		}
	} else {
		// the round t - 1 pairs (a, b) holding P and Q, and the halves they sit in
		const int ro = (int)((t - 1) % rounds);
		const int posP = rr_position(P, ro, nb), posQ = rr_position(Q, ro, nb);
		const int a = posP < np ? posP : nb - 1 - posP, hP = posP < np ? 0 : 1;
		const int b = posQ < np ? posQ : nb - 1 - posQ, hQ = posQ < np ? 0 : 1;
		const int Pa = rr_player(a, ro, nb), Qa = rr_player(nb - 1 - a, ro, nb);
		const int Pb = rr_player(b, ro, nb), Qb = rr_player(nb - 1 - b, ro, nb);
		// all global loads of the formation at once: A_{t-2}(a, b), Q_a, Q_b
		// and the diagonal blocks (P, P), (Q, Q) of A_{t-1} (kept in registers);
		// then T = A_{t-2}(a, b) Q_b and C = Q_a^H T
		static_assert(MS * MS % kThreads == 0 && 2 * BS * BS % kThreads == 0, "formation tiling");
		constexpr int NL = MS * MS / kThreads, ND = 2 * BS * BS / kThreads;
		double2 la[NL], lqa[NL], lqb[NL], ld[ND];
#pragma unroll
		for (int it = 0; it < NL; it++) {
			const int e = it * kThreads + tid, i = e / MS, l = e % MS;
			la[it] = __ldcg(prev2 + (long long)gidx(i, Pa, Qa) * kp + gidx(l, Pb, Qb));
			lqa[it] = __ldcg(Qprev + (size_t)a * MS * MS + e);
			lqb[it] = __ldcg(Qprev + (size_t)b * MS * MS + e);
		}
#pragma unroll
		for (int it = 0; it < ND; it++) {
			const int e = it * kThreads + tid;
			const int half = e / (BS * BS), i = (e / BS) % BS, l = e % BS;
			const int g0 = (half ? Q : P) * BS;
			ld[it] = __ldcg(prev + (long long)(g0 + i) * kp + g0 + l);
		}
		double2 *X = sh.op[0], *Ta = sh.op[1], *Tb = sh.op[2];
#pragma unroll
		for (int it = 0; it < NL; it++) {
			const int e = it * kThreads + tid, o = (e / MS) * LD + e % MS;
			X[o] = la[it];
			Ta[o] = lqa[it];
			Tb[o] = lqb[it];
		}
		__syncthreads();
		// only the (hP, hQ) quadrant of Q_a^H A_{t-2}(a, b) Q_b enters the
		// subproblem: T^T = Q_b[:, hQ half]^T A_{t-2}(a, b)^T (16 x 32: eight 8 x 8
		// tiles, warps 0-7), then C = Q_a[:, hP half]^H T (16 x 16: four tiles,
		// warps 0-3)
		{
			const int lane = tid & 31, warp = tid >> 5;
			double cr[1][2], ci[1][2];
			if (warp < 8) ctiles<1, false>(lane, Tb + hQ * BS * LD, X, (warp & 1) * 8, (warp >> 1) * 8, cr, ci);
			__syncthreads();
			if (warp < 8)
#pragma unroll
				for (int h = 0; h < 2; h++) {
					const int row = (warp & 1) * 8 + (lane >> 2), col = (warp >> 1) * 8 + 2 * (lane & 3) + h;
					X[row * LD + col] = make_double2(cr[0][h], ci[0][h]);
				}
			__syncthreads();
			if (warp < 4) ctiles<1, true>(lane, Ta + hP * BS * LD, X, (warp >> 1) * 8, (warp & 1) * 8, cr, ci);
			if (warp < 4)
#pragma unroll
				for (int h = 0; h < 2; h++) {
					const int i = (warp >> 1) * 8 + (lane >> 2), l = BS + (warp & 1) * 8 + 2 * (lane & 3) + h;
					M[i * LDM + l] = make_double2(cr[0][h], ci[0][h]);
				}
		}
		// diagonal blocks (P, P) and (Q, Q) of A_{t-1}
#pragma unroll
		for (int it = 0; it < ND; it++) {
			const int e = it * kThreads + tid;
			const int half = e / (BS * BS), i = (e / BS) % BS, l = e % BS;
			M[(half * BS + i) * LDM + half * BS + l] = ld[it];
		}
	}
	__syncthreads();
	double2* Qg = Qout + (size_t)j * MS * MS;
	const bool full = rr % kFullEvery == 0;
	if (full) inner_sweep<true>(sh, tol, Qg);
	else inner_sweep<false>(sh, tol, Qg);
	const int last = full ? (MS - 1) & 1 : BS & 1;
	for (int e = tid; e < MS * MS; e += kThreads) {
		const int i = e / MS, l = e % MS;
		const double2 v = ld_m(sh.m(last), i, l);
		out[(long long)gidx(i, P, Q) * kp + gidx(l, P, Q)] = make_double2(v.x, i == l ? 0.0 : v.y);
	}
	__syncthreads();
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

__device__ __forceinline__ void cp16(double2* dst, const double2* src) {
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
			: "memory");
}

// Starts the copies of an item's operands into stage st (X, Q_c, Q_r) by one
// half of the CTA; one cp.async group per call.
__device__ __forceinline__ void phase2_fetch(double2 (*st)[OP], const Item& it, int lt, int ro, int nb, int kp,
		const double2* src, const double2* V, const double2* Qr) {
	const int Pc = rr_player(it.jc, ro, nb), Qc = rr_player(nb - 1 - it.jc, ro, nb);
	const int Pr = it.is_v ? 2 * it.jr : rr_player(it.jr, ro, nb);
	const int Qr_ = it.is_v ? 2 * it.jr + 1 : rr_player(nb - 1 - it.jr, ro, nb);
	const double2* X = it.is_v ? V : src;
#pragma unroll
	for (int h = 0; h < MS * MS / (kThreads / 2); h++) {
		const int e = h * (kThreads / 2) + lt, i = e / MS, l = e % MS, o = i * LD + l;
		cp16(st[0] + o, X + (long long)gidx(i, Pr, Qr_) * kp + gidx(l, Pc, Qc));
		cp16(st[1] + o, Qr + (size_t)it.jc * MS * MS + e);
		if (!it.is_v) cp16(st[2] + o, Qr + (size_t)it.jr * MS * MS + e);
	}
	asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// The products of an item from stage st, written to dst or V.
__device__ __forceinline__ void phase2_item(double2 (*st)[OP], const Item& it, int half, int lt, int ro, int nb,
		int kp, double2* dst, double2* V) {
	const int Pc = rr_player(it.jc, ro, nb), Qc = rr_player(nb - 1 - it.jc, ro, nb);
	double cr[2][2], ci[2][2];
	if (it.is_v) {
		half_gemm<false>(lt, st[0], st[1], cr, ci);  // V Q_c
#pragma unroll
		for (int b = 0; b < 2; b++)
#pragma unroll
			for (int h = 0; h < 2; h++) {
				int row, col;
				half_rc(lt, b, h, row, col);
				V[(long long)(it.jr * MS + row) * kp + gidx(col, Pc, Qc)] = make_double2(cr[b][h], ci[b][h]);
			}
		return;
	}
	const int Pr = rr_player(it.jr, ro, nb), Qr_ = rr_player(nb - 1 - it.jr, ro, nb);
	half_gemm<false>(lt, st[1], st[0], cr, ci);  // T^T = Q_c^T X^T
	half_sync(half);
#pragma unroll
	for (int b = 0; b < 2; b++)
#pragma unroll
		for (int h = 0; h < 2; h++) {
			int row, col;
			half_rc(lt, b, h, row, col);
			st[0][row * LD + col] = make_double2(cr[b][h], ci[b][h]);
		}
	half_sync(half);
	half_gemm<true>(lt, st[2], st[0], cr, ci);  // Q_r^H T
#pragma unroll
	for (int b = 0; b < 2; b++)
#pragma unroll
		for (int h = 0; h < 2; h++) {
			int row, col;
			half_rc(lt, b, h, row, col);
			const long long gr = gidx(row, Pr, Qr_), gc = gidx(col, Pc, Qc);
			dst[gr * kp + gc] = make_double2(cr[b][h], ci[b][h]);
			dst[gc * kp + gr] = make_double2(cr[b][h], -ci[b][h]);
		}
}

// The items of round ro that one half of the CTA takes: handed out by the
// round's counter, the next one's operands in flight (cp.async, two stages)
// during the products of the current one. Bound: DMMA issue and the operands'
// L2 traffic (48 KB in, 32 KB out per block of A); whole eigensolves, upper
// triangle and copies ahead against all blocks with loads in line: 21.4 -> 17.7
// ms at k = 1000 (9 sweeps), 161 -> 124 ms at k = 2000 (10 sweeps).
__device__ void phase2(Shared& sh, int ro, int nb, int np, int nW, int kp, const double2* src, double2* dst,
		double2* V, const double2* Qr, int* ctr) {
	const int half = threadIdx.x / (kThreads / 2), lt = threadIdx.x & (kThreads / 2 - 1);
	auto take = [&]() {
		if (lt == 0) sh.next[half] = atomicAdd(ctr, 1);
		half_sync(half);
		const int w = sh.next[half];
		half_sync(half);
		return w;
	};
	double2(*st)[OP] = sh.op + 6 * half;
	int w = take(), cur = 0;
	if (w >= nW) return;
	Item it = item_of(w, np);
	phase2_fetch(st, it, lt, ro, nb, kp, src, V, Qr);
	int wn = take();
	while (w < nW) {
		Item nx{};
		if (wn < nW) {
			nx = item_of(wn, np);
			phase2_fetch(st + 3 * (cur ^ 1), nx, lt, ro, nb, kp, src, V, Qr);
			asm volatile("cp.async.wait_group 1;\n" ::: "memory");
		} else {
			asm volatile("cp.async.wait_group 0;\n" ::: "memory");
		}
		half_sync(half);
		// the index after next arrives during the products
		int w2 = nW;
		if (lt == 0 && wn < nW) w2 = atomicAdd(ctr, 1);
		phase2_item(st + 3 * cur, it, half, lt, ro, nb, kp, dst, V);
		if (lt == 0) sh.next[half] = w2;
		half_sync(half);  // the stage is free for the item after next
		it = nx;
		w = wn;
		wn = sh.next[half];
		cur ^= 1;
	}
}

// Buffers: A_r lives in bufs[(r + 1) % 3] (A_{-1} = the input in A0); Q_r in
// Qbuf + (r & 1) * np * MS * MS.
__global__ void __launch_bounds__(kThreads, 1) bjacobi_kernel(double2* A0, double2* A1, double2* A2, double2* V,
		double2* Qbuf, int kp, int max_sweeps, double tol, double tau_final, int* counters,
		unsigned long long* tmax, int* p2ctr) {
	cg::grid_group grid = cg::this_grid();
	extern __shared__ __align__(16) unsigned char smem_raw[];
	Shared& sh = *reinterpret_cast<Shared*>(smem_raw);
	const int tid = threadIdx.x;
	const int nb = kp / BS;
	const int np = nb / 2;
	const int rounds = nb - 1;
	const int nrb = kp / MS;
	const int nW = np * (np - 1) / 2 + nrb * np;
	double2* const bufs[3] = {A0, A1, A2};
	const size_t qstride = (size_t)np * MS * MS;
	// CTAs [0, p1) take phase 1 items, the rest phase 2 items (all CTAs take
	// both kinds when the grid is not larger than the pair count)
	const bool split = (int)gridDim.x > np;
	const int p1 = split ? np : (int)gridDim.x;
	const int p2first = split ? np : 0;
	const int p2count = split ? (int)gridDim.x - np : (int)gridDim.x;
	// with many phase-2 items the phase-1 CTAs take items too once their own
	// subproblems are done (phase 2 is then the longer phase)
	const bool join = split && nW > 8 * p2count;

	if (tid == 0) {
		sh.cnt = 0;
		sh.tmax = 0ULL;
	}
	__syncthreads();

	int sweep = 0;
	bool stop = false, converged = false;
	long long t = 0;
	for (;;) {
		const bool do_p1 = !stop;  // phase 1 of round t
		// round t + 1's item counter (its last use, round t - 3, is complete)
		if (blockIdx.x == 0 && tid == 0) p2ctr[(t + 1) & 3] = 0;
		const bool do_p2 = t >= 1;  // phase 2 of round t - 1
		if (do_p1 && (int)blockIdx.x < p1) {
			const double2* prev = bufs[t % 3];
			const double2* prev2 = bufs[(t + 2) % 3];
			double2* out = bufs[(t + 1) % 3];
			for (int j = blockIdx.x; j < np; j += p1)
				phase1_item(sh, j, t, rounds, nb, np, kp, tol, prev, prev2, Qbuf + ((t + 1) & 1) * qstride,
						Qbuf + (t & 1) * qstride, out);
		}
		if (do_p2 && ((int)blockIdx.x >= p2first || join)) {
			const int ro = (int)((t - 1) % rounds);
			const double2* src = bufs[(t + 2) % 3];
			double2* dst = bufs[t % 3];
			phase2(sh, ro, nb, np, nW, kp, src, dst, V, Qbuf + ((t + 1) & 1) * qstride, p2ctr + ((t - 1) & 3));
		}
		const bool sweep_end = do_p1 && (t % rounds == rounds - 1);
		if (sweep_end && tid == 0) {
			if (sh.cnt) atomicAdd(&counters[sweep], sh.cnt);
			if (sh.tmax) atomicMax(&tmax[sweep], sh.tmax);
			sh.cnt = 0;
			sh.tmax = 0ULL;
		}
		grid.sync();
		if (!do_p1) break;  // that was the last phase 2
		if (sweep_end) {
			// uniform across the grid: the counters are final after grid.sync
			const int cnt = *((volatile int*)&counters[sweep]);
			const double tm = __longlong_as_double((long long)*((volatile unsigned long long*)&tmax[sweep]));
			if (cnt == 0 || tm < tau_final) {
				converged = true;
				stop = true;
			}
			sweep++;
			if (sweep >= max_sweeps) stop = true;
		}
		t++;
	}
	// the last round completed is t - 1; A_{t-1} lives in bufs[t % 3]
	if (blockIdx.x == 0 && tid == 0) {
		counters[max_sweeps] = converged ? sweep : -1;
		counters[max_sweeps + 1] = (int)(t % 3);
	}
}

}  // namespace

int bjacobi_padded(int k) { return ((k + MS - 1) / MS) * MS; }
size_t bjacobi_qbuf_elems(int k) { return 2 * (size_t)(bjacobi_padded(k) / MS) * MS * MS; }

cudaError_t launch_bjacobi(double2* A0, double2* A1, double2* A2, double2* V, double2* Qbuf, int kp,
		int max_sweeps, double tau_final, int* counters, int num_sms, cudaStream_t s) {
	const size_t smem = sizeof(Shared);
	cudaError_t e = cudaFuncSetAttribute(bjacobi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (e != cudaSuccess) return e;
	int per_sm = 0;
	e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bjacobi_kernel, kThreads, smem);
	if (e != cudaSuccess) return e;
	if (per_sm < 1) return cudaErrorLaunchOutOfResources;
	// one CTA per phase-1 pair and one per two phase-2 items, at most one per SM:
	// the grid barrier of a small problem spans few CTAs
	const int np = kp / MS, nW = np * (np - 1) / 2 + np * np;
	const int blocks = std::min(num_sms, np + (nW + 1) / 2);
	double tol = 1e-15;
	if (!(tau_final > 0.0)) tau_final = kTauFinal;
	unsigned long long* tmax = reinterpret_cast<unsigned long long*>(counters + jacobi_tmax_offset(max_sweeps));
	int* p2ctr = counters + jacobi_p2ctr_offset(max_sweeps);
	void* args[] = {&A0, &A1, &A2, &V, &Qbuf, &kp, &max_sweeps, &tol, &tau_final, &counters, &tmax, &p2ctr};
	return cudaLaunchCooperativeKernel((void*)bjacobi_kernel, dim3(blocks), dim3(kThreads), args, smem, s);
}

}  // namespace itp2d
