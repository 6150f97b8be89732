// FP64 rotation of the states on the int8 tensor cores (tcgen05.mma
// kind::i8, exact 32-bit integer accumulation in tensor memory):
//
//   out_n[g] = sum_i W[i][n] psi_i[g]                     (stateset.cpp:214-228)
//
// Both operands are split into int8 slices under a power-of-two scale shared
// by a row of the product (the Ozaki scheme): each value x of a row with
// max |x| < 2^e is written x = 2^e sum_s d_s 2^{-7 (s + 1)}, digits d_s in
// [-127, 127] from repeated truncation (v <- 128 v, d = trunc(v), v <- v - d,
// all exact in FP64), kSlices = 8 of them: 56 bits of the row maximum. The
// product of two slices is an exact integer matrix; slice pairs (s, t) with
// s + t = d share the weight 2^{-7 (d + 2)}, so the pairs of one diagonal d
// accumulate into one S32 accumulator (at most 8 x 127^2 x 2k < 2^31 for
// k < 8300 states), and pairs with s + t >= kSlices are dropped (terms below
// 2^-56 of the row maxima; the result agrees with FP64 products to about
// 1e-15 of the largest output of its row). The FP64 result is sum_d 2^{-7 (d + 2)} acc_d,
// times the two row scales.
//
// Operands (K = 2 i + c: state i, component c = re, im):
//   A[n][(i, c)]      = W[i][n].c                      scale per output state n
//   B[2 m][(i, c)]    = (psi_i[g].re, -psi_i[g].im)    real part of out_n[g]
//   B[2 m + 1][(i, c)] = (psi_i[g].im,  psi_i[g].re)   imaginary part
// with g = g0 + m, scale per grid point g (over all states). One MMA of
// M = 128 states, N = 128 columns (64 grid points x re/im), K = 32 (16 states)
// per slice pair. The slices are written once per rotation into the MMA's
// K-major block layout (slice_w_kernel, slice_psi_kernel), so the kernel only
// copies blocks (cp.async.bulk) into a ring of three slots.
//
// Tensor memory holds four 128-column accumulators, so the 8 diagonals run in
// two passes over K: diagonals 0..3 (slices 0..3 copied), then 4..7 (all 8),
// 36 MMAs per step.
// After each pass all threads add their accumulator columns into FP64
// registers. Waits on mbarriers are bounded (tcgen05.cuh).
#include <stdint.h>

#include <algorithm>

#include "../../include/itp2d_gpu.h"
#include "contract.cuh"
#include "launch.cuh"
#include "tcgen05.cuh"

namespace itp2d {

namespace {

using namespace tcg;

constexpr int TM = 128;                     // output states per tile (M)
constexpr int TN = 128;                     // accumulator columns (N): 64 grid points x re/im
constexpr int GT = TN / 2;                  // grid points per tile
constexpr int KS = 16;                      // states per K step (32 int8 K values)
constexpr int kSlices = 8;
constexpr int kBlock = TM * 32;             // 4 KB: one slice of a 128-row x 32-byte block
constexpr int kThreads = 256;
constexpr int kTmemCols = 512;
constexpr int kDiagPerPass = 4;             // 128-column accumulators in tensor memory
static_assert(kDiagPerPass * TN <= kTmemCols, "accumulators");

constexpr int kRing = 3;
constexpr int kSlotBytes = 2 * kSlices * kBlock;  // 64 KB: the A and B slices of one step of pass 1, of two of pass 0

struct OzShared {
	alignas(128) unsigned char ring[kRing * kSlotBytes];
	alignas(8) unsigned long long full[kRing], empty[kRing];
	uint32_t tmem_base;
	int abort, used;
};

// Byte offset of element (row r, K index kk < 32) in a 128 x 32 int8 block:
// core matrix (r / 8, kk / 16) at ((r / 8) * 2 + kk / 16) * 128, rows 16 B apart.
__host__ __device__ __forceinline__ uint32_t kmaj8_off(int r, int kk) {
	return (uint32_t)((((r >> 3) << 1) + (kk >> 4)) * 128 + (r & 7) * 16 + (kk & 15));
}

// Exponent e with m < 2^e (m >= 0; 0 for m = 0, whose digits are all zero),
// at least -1000 so that the scalings below stay normal (a row whose largest
// value is below 2^-1000 keeps fewer digits).
__device__ __forceinline__ int scale_exp(double m) {
	int e = 0;
	if (m > 0.0) frexp(m, &e);  // m = f 2^e, f in [0.5, 1)
	return e < -1000 ? -1000 : e;
}

// 2^p for -1022 <= p <= 1023, from the IEEE-754 bit pattern.
__device__ __forceinline__ double pow2(int p) { return __longlong_as_double((long long)(1023 + p) << 52); }

// The kSlices digits of x 2^{-e} (|x| < 2^e): digits 0-3 in hi, 4-7 in lo, digit
// s of a word's four at byte s mod 4. The digits of repeated truncation are the
// base-128 digits of floor(|x| 2^{56 - e}), each with the sign of x: two products
// by powers of two and one conversion, the rest in integers (eight truncations
// and conversions per value in double precision bounded the slicing kernels
// at 2 to 3 TB/s). -v's digits are neg_digits of v's.
__device__ __forceinline__ uint32_t spread7(uint32_t q) {  // 28 bits -> 4 bytes, most significant digit first
	return ((q >> 21) & 0x7Fu) | ((q >> 6) & 0x7F00u) | ((q << 9) & 0x7F0000u) | ((q << 24) & 0x7F000000u);
}
__device__ __forceinline__ uint32_t neg_digits(uint32_t d) {  // -d in each byte, no borrows between them
	return (0x80808080u - (d & 0x7F7F7F7Fu)) ^ (~d & 0x80808080u);
}
__device__ __forceinline__ uint2 digits(double x, double scale) {  // scale = 2^{-e}
	const unsigned long long q = (unsigned long long)(fabs(x) * scale * 72057594037927936.0);  // 2^56: exact products
	uint32_t hi = spread7((uint32_t)(q >> 28)), lo = spread7((uint32_t)q);
	if (x < 0.0) {
		hi = neg_digits(hi);
		lo = neg_digits(lo);
	}
	return make_uint2(hi, lo);
}
// Transposes the bytes of four words: out[s] holds byte s of w[0..3].
__device__ __forceinline__ void transpose4(const uint32_t* w, uint32_t* out) {
	const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);
	const uint32_t c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);
	out[0] = __byte_perm(a, b, 0x5410);
	out[1] = __byte_perm(a, b, 0x7632);
	out[2] = __byte_perm(c, d, 0x5410);
	out[3] = __byte_perm(c, d, 0x7632);
}

// 16 values' digits (one 16-byte core-matrix row) into the kSlices blocks of one
// step, slice s at blocks + s * stride + off: value j goes to byte j of the row.
__device__ __forceinline__ void put_row16(unsigned char* blocks, int stride, uint32_t off, const uint2* v) {
	uint32_t o[4][kSlices];
#pragma unroll
	for (int q = 0; q < 4; q++) {
		const uint32_t hi[4] = {v[4 * q].x, v[4 * q + 1].x, v[4 * q + 2].x, v[4 * q + 3].x};
		const uint32_t lo[4] = {v[4 * q].y, v[4 * q + 1].y, v[4 * q + 2].y, v[4 * q + 3].y};
		transpose4(hi, o[q]);
		transpose4(lo, o[q] + 4);
	}
#pragma unroll
	for (int s = 0; s < kSlices; s++)
		*reinterpret_cast<uint4*>(blocks + s * stride + off) = make_uint4(o[0][s], o[1][s], o[2][s], o[3][s]);
}

// eA[n] for the rows of A (n < k; W[i][n] over i): 32 columns n per block, 32
// groups of rows i. Rows n >= k (to the tile edge) get 0.
__global__ void __launch_bounds__(1024) w_exp_kernel(const double2* __restrict__ W, int k, int* __restrict__ eA) {
	__shared__ double red[32][33];
	const int c = threadIdx.x & 31, r = threadIdx.x >> 5;
	const int n = blockIdx.x * 32 + c;
	double m = 0.0;
	if (n < k)
#pragma unroll 4
		for (int i = r; i < k; i += 32) {
			const double2 w = W[(size_t)i * k + n];
			m = fmax(m, fmax(fabs(w.x), fabs(w.y)));
		}
	red[r][c] = m;
	__syncthreads();
	if (r) return;
	for (int y = 1; y < 32; y++) m = fmax(m, red[y][c]);
	eA[n] = scale_exp(m);
}

// eB[g] for the grid points (g < G; psi_i[g] over i): one thread per g.
__global__ void psi_exp_kernel(const double2* __restrict__ psi, int k, long long G, long long cols,
		int* __restrict__ eB) {
	const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (g >= cols) return;
	double m = 0.0;
	if (g < G)
		for (int i = 0; i < k; i++) {
			const double2 v = __ldcs(psi + (long long)i * G + g);
			m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
		}
	eB[g] = scale_exp(m);
}

// A slices: block group (n tile nt, step s) at ((nt * ksteps + s) * kSlices)
// * kBlock; thread t of 256 writes row r = t / 2, K half kc = t % 2 (states
// s * 16 + kc * 8 + j / 2, component j % 2, j < 16).
__global__ void slice_w_kernel(const double2* __restrict__ W, int k, int ksteps, const int* __restrict__ eA,
		unsigned char* __restrict__ out) {
	const int nt = blockIdx.x, st = blockIdx.y;
	const int r = threadIdx.x >> 1, kc = threadIdx.x & 1;
	const int n = nt * TM + r;
	const double sc = pow2(-eA[n]);
	uint2 v[16];
#pragma unroll
	for (int j = 0; j < 16; j += 2) {
		const int i = st * KS + kc * 8 + j / 2;
		double2 w = make_double2(0.0, 0.0);
		if (n < k && i < k) w = W[(size_t)i * k + n];
		v[j] = digits(w.x, sc);
		v[j + 1] = digits(w.y, sc);
	}
	put_row16(out + ((size_t)nt * ksteps + st) * kSlices * kBlock, kBlock, kmaj8_off(r, kc * 16), v);
}

// Both B rows 2 m and 2 m + 1 of one half K step (8 complex values): row 2 m is
// (x, sx y) and row 2 m + 1 (y, sy x) per value, sx, sy = 1 or -1
// (NEG_FIRST: sx = -1, else sy = -1), so each component is cut into digits once.
template <bool NEG_FIRST>
__device__ __forceinline__ void put_rows_xy(unsigned char* blocks, int m, int kc, const double2* p, double sc) {
	uint2 a[16], b[16];
#pragma unroll
	for (int j = 0; j < 8; j++) {
		const uint2 x = digits(p[j].x, sc), y = digits(p[j].y, sc);
		const uint2 n = NEG_FIRST ? make_uint2(neg_digits(y.x), neg_digits(y.y)) : make_uint2(neg_digits(x.x), neg_digits(x.y));
		a[2 * j] = x;
		a[2 * j + 1] = NEG_FIRST ? n : y;
		b[2 * j] = y;
		b[2 * j + 1] = NEG_FIRST ? x : n;
	}
	put_row16(blocks, kBlock, kmaj8_off(2 * m, kc * 16), a);
	put_row16(blocks, kBlock, kmaj8_off(2 * m + 1, kc * 16), b);
}

// B slices: block group (grid tile gt, step s) at ((gt * ksteps + s) *
// kSlices) * kBlock. Thread (m, kc) of a block of two steps reads the 8 states
// of its half step at grid point m (64 consecutive points per state row) and
// writes rows 2 m (real: psi.re, -psi.im) and 2 m + 1 (imaginary: psi.im,
// psi.re).
__global__ void __launch_bounds__(256) slice_psi_kernel(const double2* __restrict__ psi, int k, long long G, int ksteps,
		const int* __restrict__ eB, unsigned char* __restrict__ out) {
	const long long gt = blockIdx.x;
	const int m = threadIdx.x & (GT - 1), kc = (threadIdx.x / GT) & 1;
	const int st = blockIdx.y * 2 + threadIdx.x / (2 * GT);
	if (st >= ksteps) return;
	const long long g = gt * GT + m;
	double2 p[8];
#pragma unroll
	for (int j = 0; j < 8; j++) {
		const int i = st * KS + kc * 8 + j;
		p[j] = (i < k && g < G) ? __ldcs(psi + (long long)i * G + g) : make_double2(0.0, 0.0);
	}
	put_rows_xy<true>(out + ((size_t)gt * ksteps + st) * kSlices * kBlock, m, kc, p, pow2(-eB[g]));
}

// Overlap operands. State exponents e[i] (max over the grid of both
// components of psi_i < 2^e[i]; 0 for the padding rows up to the tile edge):
// one block per state.
__global__ void state_exp_kernel(const double2* __restrict__ psi, int k, long long G, int* __restrict__ e) {
	__shared__ double red[32];
	const int i = blockIdx.x;
	double m = 0.0;
	if (i < k)
		for (long long g = threadIdx.x; g < G; g += blockDim.x) {
			const double2 v = __ldcs(psi + (long long)i * G + g);
			m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
		}
	for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
	__syncthreads();
	if (threadIdx.x < 32) {
		m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
		for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
		if (threadIdx.x == 0) e[i] = scale_exp(m);
	}
}

// Slices of the overlap, both operands in one reading of the states.
// A: block group (state tile ti of 128, grid step gs of 16 points) at
// ((ti * gsteps + gs) * kSlices) * kBlock; row r = state ti * 128 + r, K index
// 2 (g - 16 gs) + c: (psi.re, psi.im). B: block group (state tile tj of 64, gs)
// alike; row 2 m = X of state tj * 64 + m (psi.re, psi.im: the real part of the
// overlap), row 2 m + 1 = Y (psi.im, -psi.re: the imaginary part). Row 2 m of B
// holds row r's digits of A. Thread (kc, r) of a block of a grid step and 128
// states takes state ti * 128 + r, grid points 16 gs + 8 kc .. + 7.
__global__ void __launch_bounds__(256) slice_states_kernel(const double2* __restrict__ psi, int k, long long G,
		long long gsteps, int ntj, const int* __restrict__ e, unsigned char* __restrict__ a_out,
		unsigned char* __restrict__ b_out) {
	const int ti = blockIdx.y;
	const long long gs = blockIdx.x;
	const int r = threadIdx.x >> 1, kc = threadIdx.x & 1;
	const int i = ti * TM + r;
	const double sc = pow2(-e[i]);
	uint2 x[16], y[16];
#pragma unroll
	for (int j = 0; j < 8; j++) {
		const long long g = gs * 16 + kc * 8 + j;
		const double2 p = (i < k && g < G) ? __ldcs(psi + (long long)i * G + g) : make_double2(0.0, 0.0);
		x[2 * j] = digits(p.x, sc);
		x[2 * j + 1] = digits(p.y, sc);
		y[2 * j] = x[2 * j + 1];
		y[2 * j + 1] = make_uint2(neg_digits(x[2 * j].x), neg_digits(x[2 * j].y));
	}
	put_row16(a_out + ((size_t)ti * gsteps + gs) * kSlices * kBlock, kBlock, kmaj8_off(r, kc * 16), x);
	const int tj = i / GT, m = i % GT;
	if (tj >= ntj) return;
	unsigned char* b = b_out + ((size_t)tj * gsteps + gs) * kSlices * kBlock;
	put_row16(b, kBlock, kmaj8_off(2 * m, kc * 16), x);
	put_row16(b, kBlock, kmaj8_off(2 * m + 1, kc * 16), y);
}

// The MMAs of one step of pass PASS (diagonals 4 PASS .. 4 PASS + 3): slice pair
// (s, d - s) into accumulator d - 4 PASS; a, b: descriptors of the first slices,
// whose address fields (units of 16 bytes) advance by whole slices. first: the
// step opens its segment (the first pair of each diagonal overwrites its
// accumulator).
template <int PASS>
__device__ __forceinline__ void issue_oz_step(uint32_t tmem, uint64_t a, uint64_t b, bool first) {
	constexpr uint32_t id = idesc_s8(TN);
#pragma unroll
	for (int dd = 0; dd < kDiagPerPass; dd++) {
		constexpr int d0 = PASS * kDiagPerPass;
		const int d = d0 + dd;
#pragma unroll
		for (int s = 0; s <= d; s++)
			umma_i8(tmem + (uint32_t)(dd * TN), a + s * (kBlock >> 4), b + (d - s) * (kBlock >> 4), id,
					(first && s == 0) ? 0u : 1u);
	}
}

// Slices copied for pass p: all slices up to its largest diagonal.
__host__ __device__ constexpr int pass_slices(int pass) { return (pass + 1) * kDiagPerPass; }
static_assert(kSlices == 2 * kDiagPerPass, "two passes");

// A CTA's sequence over K steps [s0, s0 + n) in chunks of L steps: each chunk
// runs pass 0 over its steps, two per ring slot, then pass 1 over the same
// steps, one per slot (the S32 sums of a chunk stay below 2^31); a segment is
// one pass over one chunk, after which the accumulators are added into FP64
// registers. The two passes' slots take about the same MMA time (20 and 26
// MMAs), so the copies run equally far ahead in both: with one step per slot,
// pass 0 (10 MMAs, 640 cycles) waited for its copies.
struct OzSeq {
	int n, L, c0, len, pass, off;
	__device__ OzSeq(int n_, int L_) : n(n_), L(L_), c0(0), len(min(L_, n_)), pass(0), off(0) {}
	__device__ bool done() const { return c0 >= n; }
	__device__ int steps() const { return pass == 0 ? min(2, len - off) : 1; }
	__device__ int slots() const { return pass == 0 ? (len + 1) / 2 : len; }  // of the segment
	__device__ bool closes() const { return off + steps() >= len; }
	__device__ void next() {
		off += steps();
		if (off >= len) next_segment();
	}
	__device__ void next_segment() {
		off = 0;
		if (pass == 0) {
			pass = 1;
		} else {
			pass = 0;
			c0 += len;
			len = min(L, n - c0);
		}
	}
};

// Tensor memory, mbarriers and the abort flag of a CTA (all threads).
__device__ __forceinline__ void oz_setup(OzShared& sh) {
	if (threadIdx.x < 32) tmem_alloc(&sh.tmem_base, kTmemCols);
	if (threadIdx.x == 0) {
		for (int i = 0; i < kRing; i++) {
			mbar_init(smem_u32(&sh.full[i]), 1);
			mbar_init(smem_u32(&sh.empty[i]), 1);
		}
		sh.abort = sh.used = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
}

__device__ __forceinline__ void oz_teardown(OzShared& sh) {
	tc_fence_before();
	__syncthreads();
	if (threadIdx.x < 32) tmem_dealloc(sh.tmem_base, kTmemCols);
}

// The K loop of a CTA (all threads call it). Thread 32 copies the slice blocks
// of a slot's steps (src_a(st), src_b(st): the kSlices blocks of step st) into
// the ring as slots come free; thread 0 issues the MMAs. Two threads, because
// issuing blocks at the tensor pipe's rate (65 cycles per MMA): with the copies
// and their waits in the same thread a third of the tile's time was spent
// between the MMAs (149000 of 229000 cycles issuing at k = 1000). At the end of
// each segment all threads add their 64 accumulator columns (warp w:
// tensor-memory lanes 32 (w % 4) .., columns 64 (w / 4) ..) weighted 2^{-7 d}
// into acc. Returns with sh.abort set if a bounded wait gave up (then acc is
// incomplete). Pairs of CTAs on 256-row tiles (cta_group::2, half the B copies)
// were built and measured slower: 32.1 against 29.6 ms for the rotation of 1000
// states on 512 x 512, 19.7 against 17.9 ms for the overlap.
template <class SrcA, class SrcB>
__device__ __forceinline__ void oz_run(OzShared& sh, int n, int L, SrcA src_a, SrcB src_b, double (&acc)[64],
		int* err) {
	constexpr int S = kRing;
	const int tid = threadIdx.x;
	const uint32_t tmem = sh.tmem_base;
	OzSeq ahead(n, L), seg(n, L);
	int copied = 0, used = 0;  // thread 32: slots filled; all threads: slots consumed
	auto copy = [&]() {
		const int slot = copied % S, ns = ahead.steps(), nsl = pass_slices(ahead.pass);
		const uint32_t fb = smem_u32(&sh.full[slot]);
		const uint32_t dst = smem_u32(sh.ring + slot * kSlotBytes);
		const uint32_t bytes = (uint32_t)(nsl * kBlock);
		mbar_expect_tx(fb, 2 * (uint32_t)ns * bytes);
		for (int j = 0; j < ns; j++) {
			const int st = ahead.c0 + ahead.off + j;
			bulk_copy(dst + j * bytes, src_a(st), bytes, fb);
			bulk_copy(dst + kSlices * kBlock + j * bytes, src_b(st), bytes, fb);
		}
		copied++;
		ahead.next();
	};
#pragma unroll
	for (int j = 0; j < 64; j++) acc[j] = 0.0;
	const int w = tid >> 5;
	const uint32_t trow = tmem + ((uint32_t)((w & 3) * 32) << 16) + (uint32_t)((w >> 2) * 64);
	while (!seg.done()) {
		const int pass = seg.pass;
		const int seg_end = used + seg.slots();
		if (tid == 32 && !sh.abort) {
			// up to the ring's size beyond the segment: the slots its MMAs free
			while (copied < seg_end + S && !ahead.done()) {
				const int pu = copied - S;
				if (pu >= 0 && !mbar_wait(smem_u32(&sh.empty[pu % S]), (uint32_t)((pu / S) & 1))) {
					sh.abort = 1;
					atomicExch(err, ITP2D_E_TIMEOUT);
					break;
				}
				copy();
			}
		}
		if (tid == 0 && !sh.abort) {
			bool ok = true;
			int left = seg.len;  // steps of the segment
			for (int u = used; u < seg_end; u++) {
				const int slot = u % S;
				const uint32_t par = (uint32_t)((u / S) & 1);
				if (!mbar_wait(smem_u32(&sh.full[slot]), par)) {
					ok = false;
					break;
				}
				tc_fence_after();
				const uint32_t base = smem_u32(sh.ring + slot * kSlotBytes);
				const uint64_t a = sdesc(base), b = sdesc(base + kSlices * kBlock);
				if (pass == 0) {
					constexpr int step = kDiagPerPass * kBlock >> 4;
					issue_oz_step<0>(tmem, a, b, u == used);
					if (left >= 2) issue_oz_step<0>(tmem, a + step, b + step, false);
					left -= 2;
				} else {
					issue_oz_step<1>(tmem, a, b, u == used);
				}
				umma_commit(smem_u32(&sh.empty[slot]));
				sh.used = u + 1;
			}
			// the last commit covers every MMA of the segment
			if (!ok || !mbar_wait(smem_u32(&sh.empty[(seg_end - 1) % S]), (uint32_t)(((seg_end - 1) / S) & 1))) {
				sh.abort = 1;
				atomicExch(err, ITP2D_E_TIMEOUT);
			}
		}
		used = seg_end;
		seg.next_segment();
		__syncthreads();
		tc_fence_after();
		if (sh.abort) break;
#pragma unroll
		for (int dd = 0; dd < kDiagPerPass; dd++) {
			const double f = pow2(-7 * (pass * kDiagPerPass + dd));
#pragma unroll
			for (int c = 0; c < 64; c += 32) {
				uint32_t r[32];
				tmem_ld32_raw(trow + (uint32_t)(dd * TN + c), r);
				// exact 32-bit integers to double by their bits: 2^52 + 2^31 + r
				// minus 2^52 + 2^31 (four times the rate of the conversion instruction)
#pragma unroll
				for (int j = 0; j < 32; j++)
					acc[c + j] += (__hiloint2double(0x43300000, (int)(r[j] ^ 0x80000000u)) - 4503601774854144.0) * f;
			}
		}
		tc_fence_before();
		__syncthreads();
		tc_fence_after();
	}
	if (sh.abort && tid == 32) {
		// copies not waited for and the MMAs issued end before the CTA leaves (bounded)
		for (int u = sh.used; u < copied; u++) mbar_wait(smem_u32(&sh.full[u % S]), (uint32_t)((u / S) & 1));
		if (sh.used > 0) mbar_wait(smem_u32(&sh.empty[(sh.used - 1) % S]), (uint32_t)(((sh.used - 1) / S) & 1));
	}
}

__device__ __forceinline__ OzShared& oz_shared() {
	extern __shared__ __align__(128) unsigned char smem_raw[];
	return *reinterpret_cast<OzShared*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
}

// 2^e, also beyond the normal range.
__device__ __forceinline__ double pow2_any(int e) { return e >= -1022 && e <= 1023 ? pow2(e) : ldexp(1.0, e); }

// Rotation tile: states n0 .. n0 + 127 (blockIdx.x), grid points g0 .. g0 + 63
// (blockIdx.y). upper: W is upper triangular (Cholesky), states i >= n0 + 128
// do not contribute. K = 2k stays below 2^31 / (8 127^2) for k < 8300: one
// chunk. The result passes through the ring's memory, so that rows of 64 points
// are written whole (a thread holds 32 points of one state).
__global__ void __launch_bounds__(kThreads, 1) rotate_oz_kernel(const unsigned char* __restrict__ wsl,
		const unsigned char* __restrict__ psl, const int* __restrict__ eA, const int* __restrict__ eB, int k,
		long long G, double2* __restrict__ out, int* err, int upper) {
	OzShared& sh = oz_shared();
	const int n0 = blockIdx.x * TM;
	const long long gt = blockIdx.y;
	const long long g0 = gt * GT;
	const int ksteps = (k + KS - 1) / KS;
	const int nrun = upper ? (min(k, n0 + TM) + KS - 1) / KS : ksteps;
	const unsigned char* ablk = wsl + (size_t)blockIdx.x * ksteps * kSlices * kBlock;
	const unsigned char* bblk = psl + (size_t)gt * ksteps * kSlices * kBlock;
	oz_setup(sh);
	double acc[64];
	oz_run(sh, nrun, nrun, [&](int st) { return ablk + (size_t)st * kSlices * kBlock; },
			[&](int st) { return bblk + (size_t)st * kSlices * kBlock; }, acc, err);
	if (!sh.abort) {
		// row n, grid points g0 + 32 (w / 4) + jj (columns 2 jj, 2 jj + 1: re, im)
		constexpr int P = GT + 1;  // pitch in elements: conflict-free
		static_assert(TM * P * sizeof(double2) <= kRing * kSlotBytes, "staged tile");
		double2* tile = reinterpret_cast<double2*>(sh.ring);
		const int w = threadIdx.x >> 5;
		const int r = (w & 3) * 32 + (threadIdx.x & 31), c0 = (w >> 2) * 32;
		const int ea = eA[n0 + r] - 14;
#pragma unroll
		for (int jj = 0; jj < 32; jj++) {
			const double sc = pow2_any(ea + eB[g0 + c0 + jj]);
			tile[r * P + c0 + jj] = make_double2(acc[2 * jj] * sc, acc[2 * jj + 1] * sc);
		}
		__syncthreads();
		for (int i = threadIdx.x; i < TM * GT; i += kThreads) {
			const int n = n0 + i / GT;
			const long long g = g0 + i % GT;
			if (n < k && g < G) out[(long long)n * G + g] = tile[(i / GT) * P + i % GT];
		}
	}
	oz_teardown(sh);
}

// Overlap tile pair: states i0 .. i0 + 127 (A rows) x states j0 .. j0 + 63 (B:
// X and Y rows), pair index blockIdx.x over the pairs with j0 + 63 >= i0 (the
// upper triangle), grid steps [s0, s0 + n) of split blockIdx.y in chunks of
// kOvChunk steps (2 x 16 x 512 = 16384 K values: 8 x 127^2 x 16384 < 2^31).
// Writes part[split][i][j] = sum over the split's grid points of
// conj(psi_i) psi_j (before dx^2).
constexpr int kOvChunk = 512;
__global__ void __launch_bounds__(kThreads, 1) overlap_oz_kernel(const unsigned char* __restrict__ asl,
		const unsigned char* __restrict__ bsl, const int* __restrict__ e, int k, long long gsteps, int ntj,
		long long split_steps, double2* __restrict__ part, int* err) {
	OzShared& sh = oz_shared();
	int p = blockIdx.x, ti = 0;
	while (p >= ntj - 2 * ti) {
		p -= ntj - 2 * ti;
		ti++;
	}
	const int tj = 2 * ti + p;
	const int i0 = ti * TM, j0 = tj * GT;
	const long long s0 = (long long)blockIdx.y * split_steps;
	const int n = (int)min(split_steps, gsteps - s0);
	const unsigned char* ablk = asl + ((size_t)ti * gsteps + s0) * kSlices * kBlock;
	const unsigned char* bblk = bsl + ((size_t)tj * gsteps + s0) * kSlices * kBlock;
	oz_setup(sh);
	double acc[64];
	oz_run(sh, n, kOvChunk, [&](int st) { return ablk + (size_t)st * kSlices * kBlock; },
			[&](int st) { return bblk + (size_t)st * kSlices * kBlock; }, acc, err);
	if (!sh.abort) {
		const int w = threadIdx.x >> 5;
		const int i = i0 + (w & 3) * 32 + (threadIdx.x & 31);
		if (i < k) {
			const int ei = e[i] - 14;
			double2* dst = part + (size_t)blockIdx.y * k * k + (size_t)i * k;
#pragma unroll
			for (int jj = 0; jj < 32; jj++) {
				const int j = j0 + (w >> 2) * 32 + jj;
				if (j < k) {
					const double sc = pow2_any(ei + e[j]);
					dst[j] = make_double2(acc[2 * jj] * sc, acc[2 * jj + 1] * sc);
				}
			}
		}
	}
	oz_teardown(sh);
}

size_t oz_smem() { return sizeof(OzShared) + 128; }

}  // namespace

bool oz_supported(int k, long long G) { return k >= 2 && k < 8300 && G >= 1; }

size_t oz_w_bytes(int k) {
	return (size_t)((k + TM - 1) / TM) * (size_t)((k + KS - 1) / KS) * kSlices * kBlock;
}

// Slice scratch: the rotation's state slices, or the overlap's A and B
// slices (never needed at the same time).
static size_t ov_rows_bytes(int k, long long G) {
	return (size_t)((k + TM - 1) / TM) * (size_t)((G + 15) / 16) * kSlices * kBlock;
}
static size_t ov_xy_bytes(int k, long long G) {
	return (size_t)((k + GT - 1) / GT) * (size_t)((G + 15) / 16) * kSlices * kBlock;
}

size_t oz_scratch_bytes(int k, long long G) {
	const size_t rot = (size_t)((G + GT - 1) / GT) * (size_t)((k + KS - 1) / KS) * kSlices * kBlock;
	return std::max(rot, ov_rows_bytes(k, G) + ov_xy_bytes(k, G));
}

size_t oz_exp_ints(int k, long long G) {
	return (size_t)((k + TM - 1) / TM) * TM + (size_t)((G + GT - 1) / GT) * GT;
}

static void oz_attributes() {
	raise_smem_limit((const void*)rotate_oz_kernel, (int)oz_smem());
	raise_smem_limit((const void*)overlap_oz_kernel, (int)oz_smem());
}

void launch_rotate_oz(const double2* W, const double2* psi, int k, long long G, unsigned char* wsl,
		unsigned char* scratch, int* ebuf, double2* out, int* err, cudaStream_t s, bool upper) {
	const int nt = (k + TM - 1) / TM, ks = (k + KS - 1) / KS;
	const long long gtiles = (G + GT - 1) / GT;
	int* eA = ebuf;
	int* eB = ebuf + (size_t)nt * TM;
	unsigned char* psl = scratch;
	w_exp_kernel<<<nt * TM / 32, 1024, 0, s>>>(W, k, eA);
	psi_exp_kernel<<<(unsigned)((gtiles * GT + 255) / 256), 256, 0, s>>>(psi, k, G, gtiles * GT, eB);
	slice_w_kernel<<<dim3(nt, ks), 256, 0, s>>>(W, k, ks, eA, wsl);
	slice_psi_kernel<<<dim3((unsigned)gtiles, (ks + 1) / 2), 256, 0, s>>>(psi, k, G, ks, eB, psl);
	oz_attributes();
	rotate_oz_kernel<<<dim3(nt, (unsigned)gtiles), kThreads, oz_smem(), s>>>(wsl, psl, eA, eB, k, G, out, err,
			upper ? 1 : 0);
}

// Tile pairs of the overlap's upper triangle (128 states by 64).
static int overlap_pairs(int k) {
	const int nti = (k + TM - 1) / TM, ntj = (k + GT - 1) / GT;
	int pairs = 0;
	for (int ti = 0; ti < nti; ti++) pairs += ntj - 2 * ti;
	return pairs;
}

int oz_overlap_splits(int k, long long G, int num_sms, int max_splits) {
	const int pairs = overlap_pairs(k);
	const long long gsteps = (G + 15) / 16;
	const int most = (int)std::max(1LL, std::min<long long>(max_splits, gsteps));
	const int lo = std::min(most, std::max(1, (4 * num_sms + pairs - 1) / pairs));
	// the first count up to 4 lo whose last wave of one CTA per SM is 95% full
	int best = lo;
	double best_fill = 0.0;
	for (int ns = lo; ns <= std::min(most, 4 * lo); ns++) {
		const long long ctas = (long long)pairs * ns;
		const double fill = (double)ctas / (double)(((ctas + num_sms - 1) / num_sms) * num_sms);
		if (fill > best_fill + 1e-9) {
			best = ns;
			best_fill = fill;
		}
		if (fill >= 0.95) break;
	}
	return best;
}

void launch_overlap_oz(const double2* psi, int k, long long G, int nsplit, unsigned char* scratch, int* ebuf,
		double2* part, double dx2, double2* S, int* err, cudaStream_t s) {
	const int nti = (k + TM - 1) / TM, ntj = (k + GT - 1) / GT;
	const long long gsteps = (G + 15) / 16;
	unsigned char* asl = scratch;
	unsigned char* bsl = scratch + ov_rows_bytes(k, G);
	state_exp_kernel<<<nti * TM, 256, 0, s>>>(psi, k, G, ebuf);
	slice_states_kernel<<<dim3((unsigned)gsteps, nti), 256, 0, s>>>(psi, k, G, gsteps, ntj, ebuf, asl, bsl);
	const long long split_steps = (gsteps + nsplit - 1) / nsplit;
	const int used = (int)((gsteps + split_steps - 1) / split_steps);
	oz_attributes();
	overlap_oz_kernel<<<dim3(overlap_pairs(k), used), kThreads, oz_smem(), s>>>(asl, bsl, ebuf, k, gsteps, ntj,
			split_steps, part, err);
	launch_overlap_finish(part, k, used, dx2, S, s);
}

int oz_overlap_launches() { return 4; }
int oz_rotate_launches() { return 5; }

}  // namespace itp2d
