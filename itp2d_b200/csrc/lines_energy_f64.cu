// Energy passes of double lines (lines.cuh).
#include "lines.cuh"

namespace itp2d {

// (the FP64 tile for both precisions: an FP32 CTA has at most 128 of the 256
// threads that its kernel is compiled for)
int energy_row_tile_reg(const LinePlan& lp, int sy, int k) {
	int n = 0;
	if (lp.kind == 0)
		lines::for_length<double>(lp.N, [&](auto g) { n = lines::row_lines<decltype(g)>(sy, k); });
	return n;
}

int energy_col_tile_reg(const LinePlan& lp, int elem_bytes) {
	if (lp.kind != 0 || !lines::for_length<double>(lp.N, [](auto) {})) return 0;
	return 128 / elem_bytes;
}

template <>
bool launch_energy_row_reg<double>(const EnergyRowArgs& a, int k, cudaStream_t s) {
	using namespace lines;
	if (a.lp.kind != 0 || a.rows_per_tile == 0 || a.rows_per_tile != energy_row_tile_reg(a.lp, a.sy, k)) return false;
	return for_length<double>(a.sx, [&](auto g) {
		using G = decltype(g);
		auto kernel = energy_row_kernel<double, G::A, G::B>;
		const int n = a.rows_per_tile;
		const int threads = (n * G::CNT + 31) / 32 * 32;
		const size_t sm = (size_t)(G::A * G::BP + (threads + G::CNT - 1) / G::CNT * G::LS) * G::ES + 5 * 8 * sizeof(double);
		const long long tiles = (long long)k * ((a.sy + n - 1) / n);
		const int grid = grid_for(kernel, threads, sm, tiles);
		kernel<<<grid, threads, sm, s>>>(a, k);
	});
}

template <>
bool launch_energy_col_reg<double>(const EnergyColArgs& a, int k, cudaStream_t s) {
	using namespace lines;
	if (a.lp.kind != 0) return false;
	return for_length<double>(a.sy, [&](auto g) {
		using G = decltype(g);
		auto kernel = energy_col_kernel<double, G::A, G::B>;
		const size_t sm = (size_t)G::N * (1 + G::W) * G::ES + 5 * 16 * sizeof(double);
		const long long tiles = (long long)k * ((a.sx + G::W - 1) / G::W);
		const int grid = grid_for(kernel, G::COL_THREADS, sm, tiles);
		kernel<<<grid, G::COL_THREADS, sm, s>>>(a, k);
	});
}

}  // namespace itp2d
