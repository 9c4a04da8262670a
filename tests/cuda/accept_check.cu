// accept_check.cu - reservoir_accepts (ris_binned.cuh) against the comparison
// with the divided weight that it stands for.
//
// risltc_test_accept(counts) fills counts[4]:
//   0 cases of exact numerics in which the two differ, 1 the same of fast
//     numerics, over 2^28 pseudo-random triples (rnd, w, w_sum) with w_sum >= w:
//     rnd 0, 1 and the least multiples of 2^-32 among the drawn ones, weights of
//     every magnitude from the least subnormal to infinity, and sums within a
//     few units of w / rnd;
//   2 of them with a quotient that rounds to 0, 3 accepted ones.
// Returns a cudaError_t.
#include <cuda_runtime.h>

#include "../../risltc_gb300/csrc/cuda/ris_binned.cuh"

namespace {
using namespace risltc;

__global__ void accept_kernel(unsigned long long* counts) {
	unsigned long long exact = 0, fast = 0, zero = 0, accepted = 0;
	for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < (1u << 28); u += gridDim.x * blockDim.x) {
		uint32_t r[4], h = u * 2654435761u + 977u;
		for (int k = 0; k != 4; ++k) {
			h ^= h >> 16;
			h *= 0x85ebca6bu;
			h ^= h >> 13;
			h = h * 0xc2b2ae35u + k;
			r[k] = h ^ (h >> 15);
		}
		const uint32_t kind = r[3] % 8u;
		uint32_t draw = r[0];
		if (kind == 0) draw = 0u;
		if (kind == 1) draw = 0xffffffffu - (r[0] & 255u);
		if (kind == 2) draw = r[0] & 255u;
		const float rnd = __uint2float_rn(draw) * 2.3283064365386962890625e-10f;
		float w = __uint_as_float(r[1] % 0x7f800001u);  // every finite magnitude, and infinity
		if (!(w > 0.0f)) w = 1.0f;
		float w_sum = __uint_as_float(r[2] % 0x7f800001u);
		if ((r[3] >> 3) % 2u && rnd > 0.0f) {
			w_sum = __fdiv_rn(w, rnd);
			if (w_sum < 3e38f) w_sum = __uint_as_float(__float_as_uint(w_sum) + ((r[3] >> 4) % 33u) - 16u);
		}
		if (!(w_sum >= w)) w_sum = w;
		const float q = ExactNumerics::div(w, w_sum);
		const bool want = rnd < q;
		exact += reservoir_accepts<ExactNumerics>(rnd, w, w_sum) != want;
		fast += reservoir_accepts<FastNumerics>(rnd, w, w_sum) != (rnd < FastNumerics::div(w, w_sum));
		zero += q == 0.0f;
		accepted += want;
	}
	atomicAdd(counts + 0, exact);
	atomicAdd(counts + 1, fast);
	atomicAdd(counts + 2, zero);
	atomicAdd(counts + 3, accepted);
}
}  // namespace

extern "C" int risltc_test_accept(unsigned long long* counts) {
	unsigned long long* d = nullptr;
	cudaError_t e = cudaMalloc(&d, 4 * sizeof(*d));
	if (e != cudaSuccess) return (int) e;
	cudaMemset(d, 0, 4 * sizeof(*d));
	accept_kernel<<<2048, 256>>>(d);
	e = cudaMemcpy(counts, d, 4 * sizeof(*d), cudaMemcpyDeviceToHost);
	cudaFree(d);
	return (int) e;
}
