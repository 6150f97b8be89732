// Single-precision block Jacobi for the overlap matrix of the FP32 form.
//
// The FP32 form's overlap is accurate to about 1e-5 (split-BF16 tensor-core
// contraction) and its eigensolve stops at a largest rotation tangent of 1e-3,
// so FP64 arithmetic buys nothing there. The schedule and the inner sweeps are
// those of bjacobi.cu (in single precision), with block products in FFMA: four
// groups of 128 threads per CTA, each on its own item of phase 2 with the next
// item's operands in flight (cp.async, two stages).
//
// Before, the sweeps kept all of M and Q in shared memory with two barriers
// per full round, every block of A was formed (not the upper triangle only),
// and an item's loads and products came one after the other; whole solves then
// and now: 1.93 and 1.35 ms at k = 256 (8 sweeps), 3.54 and 2.48 ms at k = 500
// (7), 17.0 and 10.4 ms at k = 1000 (8), 120 and 69 ms at k = 2000 (9). At k =
// 500 a round is 11.4 us: about 2 forming the subproblem, 6 in its sweep (the
// rotations and the update of M about as long as each other) and 1.3 in the grid
// barrier.
//
// Accuracy: rotations are unitary to a few FP32 units, so the eigenvector
// matrix is orthonormal to about 1e-6; normalize_columns_kernel (jacobi.cu)
// renormalises its columns in FP64 afterwards. Rotations whose relative
// off-diagonal element is below 1e-7 are not applied, those below 1e-6 do not
// count toward convergence.
#include <cooperative_groups.h>

#include "../../include/itp2d_gpu.h"
#include "bjacobi.cuh"
#include "contract.cuh"

namespace cg = cooperative_groups;

namespace itp2d {

namespace {

using namespace bj;

// Row pitch of the operands: 16-byte rows for cp.async, and column reads of
// eight rows (the mirrored half of a product) spread over the banks.
constexpr int LD = MS + 2;
constexpr int OP = MS * LD;
constexpr int kGroups = 4;
constexpr int kGT = kThreads / kGroups;
constexpr float kSkipRel = 1e-7f;
constexpr float kNoiseRel = 1e-6f;

struct Shared32 {
	// phase 1: op[0..2] formation operands, then two buffers of M and the Q
	// warps' exchange area; phase 2: group g uses op[6 g, 6 g + 6), two stages of
	// (X, Q_c, Q_r), all with element (m, l) at [m * LD + l]
	float2 op[6 * kGroups][OP];
	float2 rst[2][NR];  // (sin, tau), (0, 0): none
	float2 re[2][NR];   // e = c / |c|
	int next[kGroups];  // phase-2 item of each thread group
	int cnt;
	unsigned long long tmax;  // bits of a non-negative double
	__device__ float2* m(int b) { return op[3] + b * OP; }
	__device__ float2* xch() { return op[5]; }
};

// c += a b, c += conj(a) b
template <bool CONJ>
__device__ __forceinline__ void cfma(float2& c, float2 a, float2 b) {
	const float ai = CONJ ? -a.y : a.y;
	c.x = fmaf(a.x, b.x, fmaf(-ai, b.y, c.x));
	c.y = fmaf(a.x, b.y, fmaf(ai, b.x, c.y));
}
__device__ __forceinline__ float4 ld4(const float2* p) { return *reinterpret_cast<const float4*>(p); }

// 32 x 32 products of one thread group: thread lt has rows r0 .. r0 + 3 and
// columns c0 and c0 + 16 (group_at); per step a warp reads its rows by broadcast
// and its columns in whole 128-byte rows.
__device__ __forceinline__ void group_at(int lt, int& r0, int& c0) {
	r0 = 8 * (lt >> 5) + 4 * ((lt >> 4) & 1);
	c0 = lt & 15;
}
// A B
__device__ __forceinline__ void group_ab(const float2* A, const float2* B, int r0, int c0, float2 (&c)[4][2]) {
#pragma unroll
	for (int r = 0; r < 4; r++) c[r][0] = c[r][1] = make_float2(0.f, 0.f);
#pragma unroll 4
	for (int m = 0; m < MS; m += 2) {
		float4 a[4];
		float2 b[2][2];
#pragma unroll
		for (int r = 0; r < 4; r++) a[r] = ld4(A + (r0 + r) * LD + m);
#pragma unroll
		for (int u = 0; u < 2; u++)
#pragma unroll
			for (int q = 0; q < 2; q++) b[u][q] = B[(m + u) * LD + c0 + 16 * q];
#pragma unroll
		for (int r = 0; r < 4; r++)
#pragma unroll
			for (int q = 0; q < 2; q++) {
				cfma<false>(c[r][q], make_float2(a[r].x, a[r].y), b[0][q]);
				cfma<false>(c[r][q], make_float2(a[r].z, a[r].w), b[1][q]);
			}
	}
}
// A^H B
__device__ __forceinline__ void group_ahb(const float2* A, const float2* B, int r0, int c0, float2 (&c)[4][2]) {
#pragma unroll
	for (int r = 0; r < 4; r++) c[r][0] = c[r][1] = make_float2(0.f, 0.f);
#pragma unroll 8
	for (int m = 0; m < MS; m++) {
		const float4 a0 = ld4(A + m * LD + r0), a1 = ld4(A + m * LD + r0 + 2);
		const float2 a[4] = {make_float2(a0.x, a0.y), make_float2(a0.z, a0.w), make_float2(a1.x, a1.y),
				make_float2(a1.z, a1.w)};
		const float2 b[2] = {B[m * LD + c0], B[m * LD + c0 + 16]};
#pragma unroll
		for (int r = 0; r < 4; r++)
#pragma unroll
			for (int q = 0; q < 2; q++) cfma<true>(c[r][q], a[r], b[q]);
	}
}

// Barrier of one thread group (named barrier 1 + g, 128 threads).
__device__ __forceinline__ void group_sync(int g) {
	asm volatile("bar.sync %0, %1;\n" ::"r"(1 + g), "r"(kGT) : "memory");
}

// Phase 1 for pair j of round t (bjacobi.cu phase1_item in FP32; Q is kept as
// Q(i, l) at [i * MS + l] here).
__device__ void phase1_item32(Shared32& sh, int j, long long t, int rr, int rounds, int nb, int np, int kp,
		const float2* prev, const float2* prev2, const float2* Qprev, float2* Qout, float2* out) {
	const int tid = threadIdx.x;
	const int P = rr_player(j, rr, nb), Q = rr_player(nb - 1 - j, rr, nb);
	float2* M = sh.m(0);
	if (t == 0) {
		for (int e = tid; e < MS * MS; e += kThreads) {
			const int i = e / MS, l = e % MS;
			M[i * LDM + l] = __ldcg(prev + (long long)gidx(i, P, Q) * kp + gidx(l, P, Q));
		}
	} else {
		const int ro = rr ? rr - 1 : rounds - 1;
		const int posP = rr_position(P, ro, nb), posQ = rr_position(Q, ro, nb);
		const int a = posP < np ? posP : nb - 1 - posP, hP = posP < np ? 0 : 1;
		const int b = posQ < np ? posQ : nb - 1 - posQ, hQ = posQ < np ? 0 : 1;
		const int Pa = rr_player(a, ro, nb), Qa = rr_player(nb - 1 - a, ro, nb);
		const int Pb = rr_player(b, ro, nb), Qb = rr_player(nb - 1 - b, ro, nb);
		constexpr int NL = MS * MS / kThreads, ND = 2 * BS * BS / kThreads;
		float2 la[NL], lqa[NL], lqb[NL], ldg[ND];
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
			ldg[it] = __ldcg(prev + (long long)(g0 + i) * kp + g0 + l);
		}
		float2 *X = sh.op[0], *Ta = sh.op[1], *Tb = sh.op[2];
#pragma unroll
		for (int it = 0; it < NL; it++) {
			const int e = it * kThreads + tid, o = (e / MS) * LD + e % MS;
			X[o] = la[it];
			Ta[o] = lqa[it];
			Tb[o] = lqb[it];
		}
		__syncthreads();
		// only the (hP, hQ) quadrant of Q_a^H A_{t-2}(a, b) Q_b enters the
		// subproblem: T = A_{t-2}(a, b) Q_b[:, hQ half] (32 x 16, threads [0, 256)
		// two rows each), then C = Q_a[:, hP half]^H T (16 x 16, threads [0, 256))
		const int row = tid >> 4, col = tid & 15;
		if (tid < BS * BS) {
			float2 c0 = make_float2(0.f, 0.f), c1 = c0;
#pragma unroll 8
			for (int m = 0; m < MS; m += 2) {
				const float4 a0 = ld4(X + row * LD + m), a1 = ld4(X + (row + BS) * LD + m);
				const float2 b0 = Tb[m * LD + hQ * BS + col], b1 = Tb[(m + 1) * LD + hQ * BS + col];
				cfma<false>(c0, make_float2(a0.x, a0.y), b0);
				cfma<false>(c1, make_float2(a1.x, a1.y), b0);
				cfma<false>(c0, make_float2(a0.z, a0.w), b1);
				cfma<false>(c1, make_float2(a1.z, a1.w), b1);
			}
			// T beside the other half of Q_b, which nothing reads any more
			float2* T = Tb + (hQ ^ 1) * BS + col;
			T[row * LD] = c0;
			T[(row + BS) * LD] = c1;
		}
		__syncthreads();
		if (tid < BS * BS) {
			const float2* T = Tb + (hQ ^ 1) * BS + col;
			float2 c = make_float2(0.f, 0.f);
#pragma unroll 8
			for (int m = 0; m < MS; m++) cfma<true>(c, Ta[m * LD + hP * BS + row], T[m * LD]);
			M[row * LDM + BS + col] = c;
		}
		// diagonal blocks (P, P) and (Q, Q) of A_{t-1}
#pragma unroll
		for (int it = 0; it < ND; it++) {
			const int e = it * kThreads + tid;
			const int half = e / (BS * BS), i = (e / BS) % BS, l = e % BS;
			M[(half * BS + i) * LDM + half * BS + l] = ldg[it];
		}
	}
	__syncthreads();
	float2* Qg = Qout + (size_t)j * MS * MS;
	const bool full = rr % kFullEvery == 0;
	if (full) inner_sweep<float, true, false>(sh, kSkipRel, kNoiseRel, Qg);
	else inner_sweep<float, false, false>(sh, kSkipRel, kNoiseRel, Qg);
	const int last = full ? (MS - 1) & 1 : BS & 1;
	for (int e = tid; e < MS * MS; e += kThreads) {
		const int i = e / MS, l = e % MS;
		const float2 v = ld_m(sh.m(last), i, l);
		out[(long long)gidx(i, P, Q) * kp + gidx(l, P, Q)] = make_float2(v.x, i == l ? 0.f : v.y);
	}
	__syncthreads();
}

// Starts the copies of an item's operands into stage st by one group.
__device__ __forceinline__ void phase2_fetch32(float2 (*st)[OP], const Item& it, int lt, int ro, int nb, int kp,
		const float2* src, const float2* V, const float2* Qr) {
	const int Pc = rr_player(it.jc, ro, nb), Qc = rr_player(nb - 1 - it.jc, ro, nb);
	const int Pr = it.is_v ? 2 * it.jr : rr_player(it.jr, ro, nb);
	const int Qr_ = it.is_v ? 2 * it.jr + 1 : rr_player(nb - 1 - it.jr, ro, nb);
	const float2* X = it.is_v ? V : src;
	auto cp = [](float2* dst, const float2* s) {
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
				"l"(s) : "memory");
	};
#pragma unroll
	for (int h = 0; h < MS * MS / 2 / kGT; h++) {
		const int e = 2 * (h * kGT + lt), i = e / MS, l = e % MS, o = i * LD + l;
		cp(st[0] + o, X + (long long)gidx(i, Pr, Qr_) * kp + gidx(l, Pc, Qc));
		cp(st[1] + o, Qr + (size_t)it.jc * MS * MS + e);
		if (!it.is_v) cp(st[2] + o, Qr + (size_t)it.jr * MS * MS + e);
	}
	asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// The products of an item from stage st, written to dst or V.
__device__ __forceinline__ void phase2_item32(float2 (*st)[OP], const Item& it, int g, int lt, int ro, int nb, int kp,
		float2* dst, float2* V) {
	const int Pc = rr_player(it.jc, ro, nb), Qc = rr_player(nb - 1 - it.jc, ro, nb);
	int r0, c0;
	group_at(lt, r0, c0);
	float2 c[4][2];
	group_ab(st[0], st[1], r0, c0, c);  // V Q_c, or T = X Q_c
	if (it.is_v) {
#pragma unroll
		for (int r = 0; r < 4; r++)
#pragma unroll
			for (int q = 0; q < 2; q++) V[(long long)(it.jr * MS + r0 + r) * kp + gidx(c0 + 16 * q, Pc, Qc)] = c[r][q];
		return;
	}
	const int Pr = rr_player(it.jr, ro, nb), Qr_ = rr_player(nb - 1 - it.jr, ro, nb);
	group_sync(g);
#pragma unroll
	for (int r = 0; r < 4; r++)
#pragma unroll
		for (int q = 0; q < 2; q++) st[0][(r0 + r) * LD + c0 + 16 * q] = c[r][q];
	group_sync(g);
	group_ahb(st[2], st[0], r0, c0, c);  // Q_r^H T
#pragma unroll
	for (int q = 0; q < 2; q++) {
		const long long gc = gidx(c0 + 16 * q, Pc, Qc), gr = gidx(r0, Pr, Qr_);
#pragma unroll
		for (int r = 0; r < 4; r++) dst[(gr + r) * kp + gc] = c[r][q];
		float4* mirror = reinterpret_cast<float4*>(dst + gc * kp + gr);
		mirror[0] = make_float4(c[0][q].x, -c[0][q].y, c[1][q].x, -c[1][q].y);
		mirror[1] = make_float4(c[2][q].x, -c[2][q].y, c[3][q].x, -c[3][q].y);
	}
}

// The items of round ro that one group takes (phase2 of bjacobi.cu).
__device__ void phase2_32(Shared32& sh, int ro, int nb, int np, int nW, int kp, const float2* src, float2* dst,
		float2* V, const float2* Qr, int* ctr) {
	const int g = threadIdx.x / kGT, lt = threadIdx.x & (kGT - 1);
	auto take = [&]() {
		if (lt == 0) sh.next[g] = atomicAdd(ctr, 1);
		group_sync(g);
		const int w = sh.next[g];
		group_sync(g);
		return w;
	};
	float2(*st)[OP] = sh.op + 6 * g;
	int w = take(), cur = 0;
	if (w >= nW) return;
	Item it = item_of(w, np);
	phase2_fetch32(st, it, lt, ro, nb, kp, src, V, Qr);
	int wn = take();
	while (w < nW) {
		Item nx{};
		if (wn < nW) {
			nx = item_of(wn, np);
			phase2_fetch32(st + 3 * (cur ^ 1), nx, lt, ro, nb, kp, src, V, Qr);
			asm volatile("cp.async.wait_group 1;\n" ::: "memory");
		} else {
			asm volatile("cp.async.wait_group 0;\n" ::: "memory");
		}
		group_sync(g);
		// the index after next arrives during the products
		int w2 = nW;
		if (lt == 0 && wn < nW) w2 = atomicAdd(ctr, 1);
		phase2_item32(st + 3 * cur, it, g, lt, ro, nb, kp, dst, V);
		if (lt == 0) sh.next[g] = w2;
		group_sync(g);  // the stage is free for the item after next
		it = nx;
		w = wn;
		wn = sh.next[g];
		cur ^= 1;
	}
}

// The cooperative solve: bjacobi_kernel of bjacobi.cu in FP32 (one CTA per SM). A_r lives in
// bufs[(r + 1) % 3] (A_{-1} = the input in A0); Q_r in Qbuf + (r & 1) * np * MS^2.
__global__ void __launch_bounds__(kThreads, 1) bjacobi32_kernel(float2* A0, float2* A1, float2* A2, float2* V,
		float2* Qbuf, int kp, int max_sweeps, double tau_final, int* counters, unsigned long long* tmaxg,
		int* p2ctr) {
	cg::grid_group grid = cg::this_grid();
	extern __shared__ __align__(16) unsigned char smem_raw[];
	Shared32& sh = *reinterpret_cast<Shared32*>(smem_raw);
	const int tid = threadIdx.x;
	const int nb = kp / BS;
	const int np = nb / 2;
	const int rounds = nb - 1;
	const int nrb = kp / MS;
	const int nW = np * (np - 1) / 2 + nrb * np;
	float2* const bufs[3] = {A0, A1, A2};
	const size_t qstride = (size_t)np * MS * MS;
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
	// round t, t mod 3 and t mod rounds (64-bit remainders cost 1000 cycles a round)
	long long t = 0;
	int t3 = 0, rr = 0;
	for (;;) {
		const bool do_p1 = !stop;
		// round t + 1's item counter (its last use, round t - 3, is complete)
		if (blockIdx.x == 0 && tid == 0) p2ctr[(t + 1) & 3] = 0;
		const bool do_p2 = t >= 1;
		if (do_p1 && (int)blockIdx.x < p1) {
			const float2* prev = bufs[t3];
			const float2* prev2 = bufs[t3 == 0 ? 2 : t3 - 1];
			float2* out = bufs[t3 == 2 ? 0 : t3 + 1];
			for (int j = blockIdx.x; j < np; j += p1)
				phase1_item32(sh, j, t, rr, rounds, nb, np, kp, prev, prev2, Qbuf + ((t + 1) & 1) * qstride,
						Qbuf + (t & 1) * qstride, out);
		}
		if (do_p2 && ((int)blockIdx.x >= p2first || join)) {
			const int ro = rr ? rr - 1 : rounds - 1;
			const float2* src = bufs[t3 == 0 ? 2 : t3 - 1];
			float2* dst = bufs[t3];
			phase2_32(sh, ro, nb, np, nW, kp, src, dst, V, Qbuf + ((t + 1) & 1) * qstride, p2ctr + ((t - 1) & 3));
		}
		const bool sweep_end = do_p1 && rr == rounds - 1;
		if (sweep_end && tid == 0) {
			if (sh.cnt) atomicAdd(&counters[sweep], sh.cnt);
			if (sh.tmax) atomicMax(&tmaxg[sweep], sh.tmax);
			sh.cnt = 0;
			sh.tmax = 0ULL;
		}
		grid.sync();
		if (!do_p1) break;
		if (sweep_end) {
			const int cnt = *((volatile int*)&counters[sweep]);
			const double tm = __longlong_as_double((long long)*((volatile unsigned long long*)&tmaxg[sweep]));
			if (cnt == 0 || tm < tau_final) {
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
	if (blockIdx.x == 0 && tid == 0) {
		counters[max_sweeps] = converged ? sweep : -1;
		counters[max_sweeps + 1] = (int)(t % 3);
	}
}

// S (k x k, FP64) into the FP32 work matrix A (kp x kp, zero padded) and V = I.
__global__ void narrow_init_kernel(const double2* __restrict__ S, int k, int kp, float2* A, float2* V) {
	const long long n = (long long)kp * kp;
	for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
			idx += (long long)gridDim.x * blockDim.x) {
		const int i = (int)(idx / kp), j = (int)(idx % kp);
		const double2 s = (i < k && j < k) ? S[(long long)i * k + j] : make_double2(0.0, 0.0);
		A[idx] = make_float2((float)s.x, (float)s.y);
		V[idx] = make_float2(i == j ? 1.f : 0.f, 0.f);
	}
}

// The FP32 result widened into the FP64 work matrices the sort and the W build
// read: the diagonal of the final A (all of it with full set) into A0 (whose
// result index becomes 0) and V into the FP64 V.
__global__ void widen_result_kernel(const float2* A0f, const float2* A1f, const float2* A2f, const float2* Vf,
		int kp, int* counters, int max_sweeps, double2* A0, double2* V, int full) {
	const int which = counters[max_sweeps + 1];
	const float2* A = which == 0 ? A0f : (which == 1 ? A1f : A2f);
	const long long n = (long long)kp * kp;
	for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
			idx += (long long)gridDim.x * blockDim.x) {
		const float2 v = Vf[idx];
		V[idx] = make_double2(v.x, v.y);
		const int i = (int)(idx / kp), j = (int)(idx % kp);
		if (full) A0[idx] = make_double2(A[idx].x, i == j ? 0.0 : A[idx].y);
		else if (i == j) A0[idx] = make_double2(A[idx].x, 0.0);
	}
}

__global__ void set_result_index_kernel(int* counters, int max_sweeps) { counters[max_sweeps + 1] = 0; }

}  // namespace

cudaError_t launch_bjacobi32(const double2* S, int k, JacobiWork& w, int num_sms, cudaStream_t s) {
	const int kp = bjacobi_padded(k);
	const long long n = (long long)kp * kp;
	const unsigned gblocks = (unsigned)std::min<long long>((n + 255) / 256, 4096);
	narrow_init_kernel<<<gblocks, 256, 0, s>>>(S, k, kp, w.f32.A0, w.f32.V);
	const size_t smem = sizeof(Shared32);
	cudaError_t e = cudaFuncSetAttribute(bjacobi32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (e != cudaSuccess) return e;
	int per_sm = 0;
	e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bjacobi32_kernel, kThreads, smem);
	if (e != cudaSuccess) return e;
	if (per_sm < 1) return cudaErrorLaunchOutOfResources;
	// one CTA per phase-1 pair and one per four phase-2 items, at most one per SM
	const int np = kp / MS, nW = np * (np - 1) / 2 + np * np;
	const int blocks = std::min(num_sms, np + (nW + kGroups - 1) / kGroups);
	int kpv = kp, ms = w.max_sweeps;
	double tau = w.tau_final > 0.0 ? w.tau_final : 1e-3;
	int* counters = w.counters;
	unsigned long long* tmax = reinterpret_cast<unsigned long long*>(counters + jacobi_tmax_offset(ms));
	float2 *a0 = w.f32.A0, *a1 = w.f32.A1, *a2 = w.f32.A2, *v = w.f32.V, *q = w.f32.Qbuf;
	int* p2ctr = counters + jacobi_p2ctr_offset(ms);
	void* args[] = {&a0, &a1, &a2, &v, &q, &kpv, &ms, &tau, &counters, &tmax, &p2ctr};
	e = cudaLaunchCooperativeKernel((void*)bjacobi32_kernel, dim3(blocks), dim3(kThreads), args, smem, s);
	if (e != cudaSuccess) return e;
	widen_result_kernel<<<gblocks, 256, 0, s>>>(w.f32.A0, w.f32.A1, w.f32.A2, w.f32.V, kp, w.counters, ms, w.A0,
			w.V, w.full_result ? 1 : 0);
	set_result_index_kernel<<<1, 1, 0, s>>>(w.counters, ms);
	return cudaGetLastError();
}

}  // namespace itp2d
