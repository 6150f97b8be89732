// One-launch steps of small double grids (lines_small.cuh).
#include "lines_small.cuh"

namespace itp2d {

template <>
bool launch_small_step<double>(const SmallStepArgs& a, int n, int k, cudaStream_t s) {
	return lines::small_step<double>(a, n, k, s);
}

}  // namespace itp2d
