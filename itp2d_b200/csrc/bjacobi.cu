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
// then leaves off-diagonal elements of order k * 1e-17 relative to the gaps) and
// in which no rotated element was above 1e-8 of sqrt(|A_pp A_qq|). If such a sweep
// turned some pair by more than 2^-20 all the same (one that does not count: equal
// diagonals, an element of rounding size), it takes a second such sweep, or one
// that counts nothing: that rotation may bring back, at full size, an element that
// a counted one has just taken away (clusters of equal eigenvalues: residuals of
// 2e-12 with one such sweep, 1e-15 with two).
#include <cooperative_groups.h>

#include "../../include/itp2d_gpu.h"
#include "bjacobi.cuh"
#include "contract.cuh"

namespace cg = cooperative_groups;

namespace itp2d {

namespace {

using namespace bj;

constexpr int LD = MS + 4;    // padded row length (complex): conflict-free 16-byte DMMA fragments
constexpr int OP = MS * LD;   // elements of one product operand
constexpr double kTauFinal = 3e-9;
constexpr double kNoiseRel = 1e-13;  // relative off-diagonal treated as rounding noise

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
	asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
			: "+d"(d0), "+d"(d1)
			: "d"(a), "d"(b));
}

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
	int mixed;                                   // a rotation by more than 2^-20 in it
	unsigned long long tmax;                     // largest tangent (bits of a non-negative double)
	// Subproblem buffer b, only the upper triangle (row <= column) in use.
	__device__ double2* m(int b) { return op[3] + b * OP; }
	__device__ double2* xch() { return op[5]; }
};

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

// Bit of a sweep's counter beside its counted rotations (fewer than 2^30).
constexpr int kMixed = 1 << 30;

// Whether a sweep with cnt counted rotations and largest tangent tm is the last;
// small: whether the sweep before was below the tolerance too, replaced by this
// one's. A tolerance looser than the default asks for no second sweep.
__device__ __forceinline__ bool last_sweep(int cnt, bool mixed, double tm, double tau_final, bool& small) {
	const bool below = tm < tau_final;
	const bool last = cnt == 0 || (below && (!mixed || small || tau_final > kTauFinal));
	small = below;
	return last;
}

// Phase 1 for pair j of round t (within-sweep round rr): forms the subproblem
// (upper triangle of M buffer 0), sweeps it, stores Q_t and the rotated
// subproblem. prev: A_{t-1} (diagonal pair blocks of round t - 1), prev2:
// A_{t-2}, Qprev: the Q buffer of round t - 1 (t >= 1). For t = 0 the
// subproblem is read from prev = A_{-1}, the initial matrix, and a matrix of one
// pair from prev in every round: phase 1 of round t - 1 left all of it there.
// (Forming its off-diagonal block by products again would put the rounding of the
// large eigenvalues beside the null ones, whose rotations would then never end.)
__device__ void phase1_item(Shared& sh, int j, long long t, int rr, int rounds, int nb, int np, int kp, double tol,
		const double2* prev, const double2* prev2, const double2* Qprev, double2* Qout, double2* out) {
	const int tid = threadIdx.x;
	const int P = rr_player(j, rr, nb), Q = rr_player(nb - 1 - j, rr, nb);
	double2* M = sh.m(0);
	if (t == 0 || np == 1) {
		for (int e = tid; e < MS * MS; e += kThreads) {
			const int i = e / MS, l = e % MS;
			M[i * LDM + l] = __ldcg(prev + (long long)gidx(i, P, Q) * kp + gidx(l, P, Q));
		}
	} else {
		// the round t - 1 pairs (a, b) holding P and Q, and the halves they sit in
		const int ro = rr ? rr - 1 : rounds - 1;
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
	if (full) inner_sweep<double, true, true>(sh, tol, kNoiseRel, Qg);
	else inner_sweep<double, false, true>(sh, tol, kNoiseRel, Qg);
	const int last = full ? (MS - 1) & 1 : BS & 1;
	for (int e = tid; e < MS * MS; e += kThreads) {
		const int i = e / MS, l = e % MS;
		const double2 v = ld_m(sh.m(last), i, l);
		out[(long long)gidx(i, P, Q) * kp + gidx(l, P, Q)] = make_double2(v.x, i == l ? 0.0 : v.y);
	}
	__syncthreads();
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
// ms at k = 1000 (9 sweeps), 161 -> 124 ms at k = 2000 (10 sweeps); the whole
// solves take 16.4 and 112 ms with the cheaper indices of the rounds.
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
		sh.cnt = sh.mixed = 0;
		sh.tmax = 0ULL;
	}
	__syncthreads();

	int sweep = 0;
	bool stop = false, converged = false, small = false;
	// round t, t mod 3 and t mod rounds (64-bit remainders cost 1000 cycles a round)
	long long t = 0;
	int t3 = 0, rr = 0;
	for (;;) {
		const bool do_p1 = !stop;  // phase 1 of round t
		// round t + 1's item counter (its last use, round t - 3, is complete)
		if (blockIdx.x == 0 && tid == 0) p2ctr[(t + 1) & 3] = 0;
		const bool do_p2 = t >= 1;  // phase 2 of round t - 1
		if (do_p1 && (int)blockIdx.x < p1) {
			const double2* prev = bufs[t3];
			const double2* prev2 = bufs[t3 == 0 ? 2 : t3 - 1];
			double2* out = bufs[t3 == 2 ? 0 : t3 + 1];
			for (int j = blockIdx.x; j < np; j += p1)
				phase1_item(sh, j, t, rr, rounds, nb, np, kp, tol, prev, prev2, Qbuf + ((t + 1) & 1) * qstride,
						Qbuf + (t & 1) * qstride, out);
		}
		if (do_p2 && ((int)blockIdx.x >= p2first || join)) {
			const int ro = rr ? rr - 1 : rounds - 1;
			const double2* src = bufs[t3 == 0 ? 2 : t3 - 1];
			double2* dst = bufs[t3];
			phase2(sh, ro, nb, np, nW, kp, src, dst, V, Qbuf + ((t + 1) & 1) * qstride, p2ctr + ((t - 1) & 3));
		}
		const bool sweep_end = do_p1 && rr == rounds - 1;
		if (sweep_end && tid == 0) {
			if (sh.cnt) atomicAdd(&counters[sweep], sh.cnt);
			if (sh.mixed) atomicOr(&counters[sweep], kMixed);
			if (sh.tmax) atomicMax(&tmax[sweep], sh.tmax);
			sh.cnt = sh.mixed = 0;
			sh.tmax = 0ULL;
		}
		grid.sync();
		if (!do_p1) break;  // that was the last phase 2
		if (sweep_end) {
			// uniform across the grid: the counters are final after grid.sync
			const int cnt = *((volatile int*)&counters[sweep]);
			const double tm = __longlong_as_double((long long)*((volatile unsigned long long*)&tmax[sweep]));
			if (last_sweep(cnt & (kMixed - 1), cnt >= kMixed, tm, tau_final, small)) {
				converged = true;
				stop = true;
			}
			sweep++;
			if (sweep >= max_sweeps) stop = true;
		}
		t++;
		t3 = t3 == 2 ? 0 : t3 + 1;
		rr = rr == rounds - 1 ? 0 : rr + 1;
	}
	// the last round completed is t - 1; A_{t-1} lives in bufs[t % 3]
	if (blockIdx.x == 0 && tid == 0) {
		counters[max_sweeps] = converged ? sweep : -1;
		counters[max_sweeps + 1] = (int)(t % 3);
	}
}

// The whole solve of a matrix of at most kTinyN indices by one warp, pair after
// pair (lane i: element i of the two rows and columns that a rotation touches). A
// sweep is 1 to 6 rotations in line here and 31 rounds of 1000 cycles in the
// block kernel, whatever n. Allocation-free eigensolve, n = 1, 2, 3, 4: block
// kernel 101, 139, 169, 188 us, this one 74, 74, 79, 85 (a cooperative kernel of
// one grid-wide round per n / 2 rotations: 82, 85, 161, 184, and 266 against the
// block kernel's 190 at n = 5). A kernel of its own: the same sweep as a branch of
// bjacobi_kernel cost that kernel 7 % of its time at k = 200.
constexpr int kTinyN = 4;
__global__ void __launch_bounds__(32) tiny_jacobi_kernel(double2* A, double2* V, int n, int kp, int max_sweeps,
		double tol, double tau_final, int* counters) {
	__shared__ double2 M[kTinyN * LDM], Q[kTinyN][kTinyN];  // upper triangle; Q(i, l) at [l][i]
	const int i = threadIdx.x;
	for (int e = i; e < n * n; e += 32) {
		const int r = e / n, l = e % n;
		if (r <= l) M[m_at(r, l)] = A[(long long)r * kp + l];
		Q[l][r] = make_double2(r == l ? 1.0 : 0.0, 0.0);
	}
	__syncwarp();
	int sweep = 0;
	bool converged = false, small = false;
	while (!converged && sweep < max_sweeps) {
		int cnt = 0;
		bool mixed = false;
		double tmax = 0.0;
#pragma unroll 1
		for (int p = 0; p + 1 < n; p++)
#pragma unroll 1
			for (int q = p + 1; q < n; q++) {
				double a = M[m_at(p, p)].x, b = M[m_at(q, q)].x;
				double2 c = M[m_at(p, q)];
				const Rotation<double> J = make_rotation<double>(a, b, c.x, c.y, tol, kNoiseRel, cnt, tmax);
				mixed |= fabs(J.s) >= 0x1p-20;
				rotated_pair(J, a, b, c.x, c.y);
				__syncwarp();
				if (i < n) {
					if (i != p && i != q) {
						double2 xp = ld_m(M, p, i), xq = ld_m(M, q, i);
						rows2(J.s, J.tau, J.er, J.ei, xp.x, xp.y, xq.x, xq.y);
						st_m(M, p, i, xp);
						st_m(M, q, i, xq);
					}
					if (i == p) {
						M[m_at(p, p)] = make_double2(a, 0.0);
						M[m_at(q, q)] = make_double2(b, 0.0);
						M[m_at(p, q)] = c;
					}
					double2 vp = Q[p][i], vq = Q[q][i];
					cols2(J.s, J.tau, J.er, J.ei, vp.x, vp.y, vq.x, vq.y);
					Q[p][i] = vp;
					Q[q][i] = vq;
				}
				__syncwarp();
			}
		sweep++;
		converged = last_sweep(cnt, mixed, tmax, tau_final, small);  // the same in every lane
	}
	for (int e = i; e < n * n; e += 32) {
		const int r = e / n, l = e % n;
		A[(long long)r * kp + l] = ld_m(M, r, l);
		V[(long long)r * kp + l] = Q[l][r];
	}
	if (i == 0) {
		counters[max_sweeps] = converged ? sweep : -1;
		counters[max_sweeps + 1] = 0;
	}
}

}  // namespace

int bjacobi_padded(int k) { return ((k + MS - 1) / MS) * MS; }
size_t bjacobi_qbuf_elems(int k) { return 2 * (size_t)(bjacobi_padded(k) / MS) * MS * MS; }

cudaError_t launch_bjacobi(double2* A0, double2* A1, double2* A2, double2* V, double2* Qbuf, int n, int kp,
		int max_sweeps, double tau_final, int* counters, int num_sms, cudaStream_t s) {
	double tol = 1e-15;
	if (!(tau_final > 0.0)) tau_final = kTauFinal;
	if (n <= kTinyN) {
		tiny_jacobi_kernel<<<1, 32, 0, s>>>(A0, V, n, kp, max_sweeps, tol, tau_final, counters);
		return cudaGetLastError();
	}
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
	unsigned long long* tmax = reinterpret_cast<unsigned long long*>(counters + jacobi_tmax_offset(max_sweeps));
	int* p2ctr = counters + jacobi_p2ctr_offset(max_sweeps);
	void* args[] = {&A0, &A1, &A2, &V, &Qbuf, &kp, &max_sweeps, &tol, &tau_final, &counters, &tmax, &p2ctr};
	return cudaLaunchCooperativeKernel((void*)bjacobi_kernel, dim3(blocks), dim3(kThreads), args, smem, s);
}

}  // namespace itp2d
