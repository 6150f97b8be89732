"""The per-device answers of launch.cuh (shared-memory limits, occupancy,
multiprocessor counts), compiled against a stand-in for the CUDA runtime with two
devices: a limit is raised on each device that launches a kernel, answers are
asked for once per device, and a failure is not kept."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cassert>
#include <cstdio>
#include "launch.cuh"

static int device = 0, raised[2] = {0, 0}, limit[2] = {0, 0}, asked[2] = {0, 0}, counted[2] = {0, 0};
static bool refuse = false;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
	if (refuse) return cudaErrorInvalidValue;
	raised[device]++;
	limit[device] = bytes;
	return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* n, cudaDeviceAttr, int dev) {
	if (refuse) return cudaErrorInvalidValue;
	counted[dev]++;
	*n = dev == 0 ? 148 : 100;
	return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
	if (refuse) return cudaErrorInvalidValue;
	asked[device]++;
	*n = device == 0 ? 4 : 3;
	return cudaSuccess;
}
}
#define CHECK(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }

int main() {
	using namespace itp2d;
	const char kernel = 0, other = 0;
	refuse = true;
	CHECK(raise_smem_limit(&kernel) != cudaSuccess);
	CHECK(resident_ctas(&kernel, 128, 1000) == 1 && sm_count() == 1);
	refuse = false;
	for (int pass = 0; pass < 2; pass++)
		for (device = 0; device < 2; device++) {
			CHECK(raise_smem_limit(&kernel) == cudaSuccess);
			CHECK(resident_ctas(&kernel, 128, 1000) == (device == 0 ? 4 : 3));
			CHECK(sm_count() == (device == 0 ? 148 : 100));
		}
	for (device = 0; device < 2; device++)
		CHECK(raised[device] == 1 && limit[device] == kSmemMax && asked[device] == 1 && counted[device] == 1);
	device = 1;
	CHECK(raise_smem_limit(&other, 1024) == cudaSuccess && raised[1] == 2 && limit[1] == 1024);
	CHECK(resident_ctas(&kernel, 256, 1000) == 3 && asked[1] == 2);
	return 0;
}
"""


def test_limits_are_kept_per_device(tmp_path):
    cuda = next((c for c in ("/usr/local/cuda", os.path.dirname(os.path.dirname(shutil.which("nvcc") or "")))
                 if os.path.exists(os.path.join(c, "include", "cuda_runtime_api.h"))), None)
    if not shutil.which("g++") or not cuda:
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "itp2d_b200", "csrc"), "-I",
                    os.path.join(cuda, "include"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
