// pair_check.cu - exhaustive check of pair_exact.cuh on this GPU's
// approximation unit.
//
// risltc_test_pairs(counts, neg_zero) fills counts[5]:
//   0 lanes of rsqrt_negated differing from -__frcp_rn(__fsqrt_rn(d)) over
//     every finite float d of 2^-76 or more;
//   1 the number of lanes checked there;
//   2 lanes of edge_fit_negated differing from -__fdiv_rn(a(x), b(x)) over
//     every float x in (0, 1 + 2^-15];
//   3 the number of lanes checked there;
//   4 lanes where PairExact's mul, mul then add, or mul then sub differ
//     bitwise from the separately rounded scalar operations, over 2^28
//     pseudo-random bit patterns with zeros of both signs among them.
// Returns a cudaError_t.
#include <cuda_runtime.h>

#include "../../risltc_gb300/csrc/cuda/pair_exact.cuh"

namespace {
using namespace risltc;

__device__ bool same(float a, float b) {
	return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b));
}

__global__ void root_kernel(unsigned long long* counts, float neg_zero) {
	const PairExact o{pair(neg_zero)};
	unsigned long long bad = 0, checked = 0;
	const uint32_t stride = gridDim.x * blockDim.x;
	for (uint64_t u = kRootMin + blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; u <= kRootMax; u += stride) {
		const uint32_t v = kRootMin + (kRootMax - (uint32_t) u);  // the other lane runs from the range's other end
		const float2 d = make_float2(__uint_as_float((uint32_t) u), __uint_as_float(v));
		const float2 r = rsqrt_negated(o, d);
		bad += !same(r.x, -__frcp_rn(__fsqrt_rn(d.x)));
		bad += !same(r.y, -__frcp_rn(__fsqrt_rn(d.y)));
		checked += 2;
	}
	atomicAdd(counts + 0, bad);
	atomicAdd(counts + 1, checked);
}

__device__ float fit(float x) {
	const float a = __fadd_rn(0.8543985f, __fmul_rn(__fadd_rn(0.4965155f, __fmul_rn(0.0145206f, x)), x));
	const float b = __fadd_rn(3.4175940f, __fmul_rn(__fadd_rn(4.1616724f, x), x));
	return __fdiv_rn(a, b);
}

__global__ void fit_kernel(unsigned long long* counts, float neg_zero) {
	const PairExact o{pair(neg_zero)};
	constexpr uint32_t lo = 1u, hi = 0x3f800100u;
	unsigned long long bad = 0, checked = 0;
	for (uint64_t u = lo + blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; u <= hi; u += gridDim.x * blockDim.x) {
		const float2 x = make_float2(__uint_as_float((uint32_t) u), __uint_as_float(lo + (hi - (uint32_t) u)));
		const float2 r = edge_fit_negated(o, x);
		bad += !same(r.x, -fit(x.x));
		bad += !same(r.y, -fit(x.y));
		checked += 2;
	}
	atomicAdd(counts + 2, bad);
	atomicAdd(counts + 3, checked);
}

__global__ void operation_kernel(unsigned long long* counts, float neg_zero) {
	const PairExact o{pair(neg_zero)};
	unsigned long long bad = 0;
	for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < (1u << 28); u += gridDim.x * blockDim.x) {
		uint32_t w[6], h = u * 2654435761u + 12345u;
		for (int k = 0; k != 6; ++k) {
			h ^= h >> 16;
			h *= 0x85ebca6bu;
			h ^= h >> 13;
			h = h * 0xc2b2ae35u + k;
			w[k] = (h >> 7) % 9u == 0 ? (h & 0x80000000u) : h;
		}
		const float2 a = make_float2(__uint_as_float(w[0]), __uint_as_float(w[1]));
		const float2 b = make_float2(__uint_as_float(w[2]), __uint_as_float(w[3]));
		const float2 c = make_float2(__uint_as_float(w[4]), __uint_as_float(w[5]));
		const float2 m = o.mul(a, b), s = o.add(o.mul(a, b), c), t = o.sub(o.mul(a, b), o.mul(b, c));
		bad += !same(m.x, __fmul_rn(a.x, b.x)) || !same(s.x, __fadd_rn(__fmul_rn(a.x, b.x), c.x)) ||
		       !same(t.x, __fadd_rn(__fmul_rn(a.x, b.x), -__fmul_rn(b.x, c.x)));
		bad += !same(m.y, __fmul_rn(a.y, b.y)) || !same(s.y, __fadd_rn(__fmul_rn(a.y, b.y), c.y)) ||
		       !same(t.y, __fadd_rn(__fmul_rn(a.y, b.y), -__fmul_rn(b.y, c.y)));
	}
	atomicAdd(counts + 4, bad);
}
}  // namespace

extern "C" int risltc_test_pairs(unsigned long long* counts, float neg_zero) {
	unsigned long long* d = nullptr;
	cudaError_t e = cudaMalloc(&d, 5 * sizeof(*d));
	if (e != cudaSuccess) return (int) e;
	cudaMemset(d, 0, 5 * sizeof(*d));
	root_kernel<<<2048, 256>>>(d, neg_zero);
	fit_kernel<<<2048, 256>>>(d, neg_zero);
	operation_kernel<<<2048, 256>>>(d, neg_zero);
	e = cudaMemcpy(counts, d, 5 * sizeof(*d), cudaMemcpyDeviceToHost);
	cudaFree(d);
	return (int) e;
}
