// Row passes of double lines (lines.cuh).
#include "lines.cuh"

namespace itp2d {

template <>
bool launch_row_pass_reg<double>(const RowPassArgs& a, int k, cudaStream_t s) {
	using namespace lines;
	if (a.lp.kind != 0) return false;
	return for_length<double>(a.sx, [&](auto g) {
		using G = decltype(g);
		auto kernel = row_kernel<double, G::A, G::B>;
		const int n = row_lines<G>(a.sy, k);
		const int threads = (n * G::CNT + 31) / 32 * 32;
		const size_t sm = (size_t)(G::A * G::BP + (threads + G::CNT - 1) / G::CNT * G::LS) * G::ES;
		const long long tiles = (long long)k * ((a.sy + n - 1) / n);
		const int grid = grid_for(kernel, threads, sm, tiles);
		kernel<<<grid, threads, sm, s>>>(a, k, n);
	});
}

}  // namespace itp2d
