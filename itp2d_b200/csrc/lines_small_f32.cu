// One-launch steps of small float grids (lines_small.cuh).
#include "lines_small.cuh"

namespace itp2d {

template <>
bool launch_small_step<float>(const SmallStepArgs& a, int n, int k, cudaStream_t s) {
	return lines::small_step<float>(a, n, k, s);
}

}  // namespace itp2d
