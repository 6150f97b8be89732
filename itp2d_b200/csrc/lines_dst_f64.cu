// Row and column passes of double Dirichlet lines (lines_dst.cuh).
#include "lines_dst.cuh"

namespace itp2d {

template <>
bool launch_row_pass_sine<double>(const RowPassArgs& a, int k, cudaStream_t s) {
	return a.lp.kind == 1 && lines::launch_dst_row<double>(a, k, s);
}

template <>
bool launch_col_pass_sine<double>(const ColPassArgs& a, int k, cudaStream_t s) {
	return a.lp.kind == 1 && lines::launch_dst_col<double>(a, k, s);
}

}  // namespace itp2d
