// Column passes of double lines (lines.cuh).
#include "lines.cuh"

namespace itp2d {

template <>
bool launch_col_pass_reg<double>(const ColPassArgs& a, int k, cudaStream_t s) {
	using namespace lines;
	if (a.lp.kind != 0) return false;
	return for_length<double>(a.sy, [&](auto g) {
		using G = decltype(g);
		auto kernel = col_kernel<double, G::A, G::B>;
		const size_t sm = (size_t)G::N * (1 + G::W) * G::ES;
		const long long tiles = (long long)k * ((a.sx + G::W - 1) / G::W);
		const int grid = grid_for(kernel, G::COL_THREADS, sm, tiles);
		kernel<<<grid, G::COL_THREADS, sm, s>>>(a, k);
	});
}

}  // namespace itp2d
