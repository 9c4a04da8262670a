// root_check.cu - exhaustive check of pair_exact.cuh's square root alone.
//
// risltc_test_root(counts, neg_zero) fills counts[4]:
//   0 lanes of root_from_rsqrt differing from __fsqrt_rn(d) over every finite
//     float d of 2^-76 or more;
//   1 the number of lanes checked there;
//   2 floats of [2^-126, 2^-76) on which it differs;
//   3 the largest of them (as a word; 0: none).
// Returns a cudaError_t.
#include <cuda_runtime.h>

#include "../../risltc_gb300/csrc/cuda/pair_exact.cuh"

namespace {
using namespace risltc;

__device__ float2 root(const PairExact& o, float2 d) {
	return root_from_rsqrt(o, d, make_float2(rsqrt_approx(d.x), rsqrt_approx(d.y)));
}

__global__ void range_kernel(unsigned long long* counts, float neg_zero) {
	const PairExact o{pair(neg_zero)};
	unsigned long long bad = 0, checked = 0;
	for (uint64_t u = kRootMin + blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; u <= kRootMax; u += gridDim.x * blockDim.x) {
		const uint32_t v = kRootMin + (kRootMax - (uint32_t) u);  // the other lane runs from the range's other end
		const float2 d = make_float2(__uint_as_float((uint32_t) u), __uint_as_float(v));
		const float2 s = root(o, d);
		bad += __float_as_uint(s.x) != __float_as_uint(__fsqrt_rn(d.x));
		bad += __float_as_uint(s.y) != __float_as_uint(__fsqrt_rn(d.y));
		checked += 2;
	}
	atomicAdd(counts + 0, bad);
	atomicAdd(counts + 1, checked);
}

__global__ void below_kernel(unsigned long long* counts, float neg_zero) {
	const PairExact o{pair(neg_zero)};
	unsigned long long bad = 0, largest = 0;
	for (uint32_t u = 0x00800000u + blockIdx.x * blockDim.x + threadIdx.x; u < kRootMin; u += gridDim.x * blockDim.x) {
		const float d = __uint_as_float(u);
		if (__float_as_uint(root(o, pair(d)).x) != __float_as_uint(__fsqrt_rn(d))) {
			++bad;
			largest = u;
		}
	}
	atomicAdd(counts + 2, bad);
	atomicMax(counts + 3, largest);
}
}  // namespace

extern "C" int risltc_test_root(unsigned long long* counts, float neg_zero) {
	unsigned long long* d = nullptr;
	cudaError_t e = cudaMalloc(&d, 4 * sizeof(*d));
	if (e != cudaSuccess) return (int) e;
	cudaMemset(d, 0, 4 * sizeof(*d));
	range_kernel<<<2048, 256>>>(d, neg_zero);
	below_kernel<<<2048, 256>>>(d, neg_zero);
	e = cudaMemcpy(counts, d, 4 * sizeof(*d), cudaMemcpyDeviceToHost);
	cudaFree(d);
	return (int) e;
}
