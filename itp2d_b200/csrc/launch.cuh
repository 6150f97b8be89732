// What launches ask the CUDA runtime about kernels and devices. The answers are
// kept per device, because a process may drive several: a kernel's
// shared-memory limit is an attribute on one device, and so are its occupancy
// and the number of multiprocessors. Failures are returned and not kept.
#pragma once

#include <cuda_runtime_api.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <set>
#include <tuple>
#include <utility>

namespace itp2d {

constexpr int kSmemMax = 227 * 1024;  // dynamic shared memory a CTA can have

// Multiprocessors of the current device (1 where the runtime does not answer).
inline int sm_count() {
	static std::mutex mu;
	static std::map<int, int> known;
	int dev = 0, n = 0;
	if (cudaGetDevice(&dev) != cudaSuccess) return 1;
	std::lock_guard<std::mutex> g(mu);
	const auto it = known.find(dev);
	if (it != known.end()) return it->second;
	if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 1;
	known.emplace(dev, n);
	return n;
}

// Raises the kernel's limit of dynamic shared memory on the current device. The
// limit is shared by every host thread that launches the kernel, so `bytes` has
// to be the same in every call: the most that any launch needs.
inline cudaError_t raise_smem_limit(const void* kernel, int bytes = kSmemMax) {
	static std::mutex mu;
	static std::set<std::pair<const void*, int>> done;
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess) return e;
	std::lock_guard<std::mutex> g(mu);
	if (done.count({kernel, dev})) return cudaSuccess;
	e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
	if (e == cudaSuccess) done.insert({kernel, dev});
	return e;
}

// CTAs of a kernel that fit on an SM of the current device at a launch shape (1
// where the runtime does not answer). Asked for once per device and shape: the
// query costs as much host time as a launch (a solve of 48 states on 96 x 96 takes
// 28.6 ms with a query per launch and 27.5 ms without).
inline int resident_ctas(const void* kernel, int threads, size_t smem) {
	static std::mutex mu;
	static std::map<std::tuple<const void*, int, int, size_t>, int> known;
	int dev = 0, n = 0;
	if (cudaGetDevice(&dev) != cudaSuccess) return 1;
	const auto key = std::make_tuple(kernel, dev, threads, smem);
	std::lock_guard<std::mutex> g(mu);
	const auto it = known.find(key);
	if (it != known.end()) return it->second;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess || n < 1) return 1;
	known.emplace(key, n);
	return n;
}

}  // namespace itp2d
